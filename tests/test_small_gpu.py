"""Small calls (one block, start to end) and short batch slices against the oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import _lib, data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1, 2047, 2048, 2049, 4095, 4096, 4097], [4096] * 6, [33] * 40 + [4096]])
@pytest.mark.parametrize("n_low,n_high,ones,compat", [(1, 4, 3, False), (61, 64, 3, True), (509, 8, 3, False),
                                                      (509, 600, 28, False), (8191, 8, 1, True)])
def test_small_calls(gpu, sizes, n_low, n_high, ones, compat):
    masks = qs.generate_hashmask(64, 32, ones, 4, 2)
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, n_high, 32, 1, 64, hash_seed=2654435769, mask_table=masks,
                                      compat_v3=compat)
    orc = oracle.Msws(n_low, n_high, 2654435769, masks, compat_v3=compat)
    q = data.rank_keys(4, 0, 300)
    for i, n in enumerate(sizes):
        keys = data.zipf_keys(n + 1, 300, 1.2, seed=n + i, perm_seed=4)[i & 1:][:n]
        sk.insert(keys)
        orc.insert(keys.cpu().numpy())
    assert np.array_equal(sk.search(q).cpu().numpy(), orc.query(q.cpu().numpy()))
    assert sk.status() == (_lib.QS_ERR_POOL_FULL if orc.pool_full else _lib.QS_OK)
    low, high = sk.tables()
    assert np.array_equal(low, orc.low) and np.array_equal(high, orc.high)
    st = sk.stats()
    assert st["next_level_id"] == orc.next_id and st["dropped_keys"] == orc.dropped


@pytest.mark.parametrize("lengths", [[0, 1, 700, 2048, 2049, 4096], [4096, 4097, 3, 60000, 9, 100]])
@pytest.mark.parametrize("pool", [3, 5000])
def test_graph_batches_with_short_and_long_slices(gpu, lengths, pool):
    n_low = [3, 61, 127, 1021, 509, 4093]
    n_high = [min(n + 2, pool) for n in n_low]
    masks = qs.generate_hashmask(1021, 32, 3, 4, 1)
    b = BatchedSketches(n_low, n_high, seed_rng=3)
    orcs = [oracle.Msws(n_low[s], n_high[s], int(x), masks) for s, x in enumerate(b.seeds())]
    off = np.zeros(7, np.int64)
    off[1:] = np.cumsum(lengths)
    keys = torch.empty(int(off[-1]), dtype=torch.int32, device="cuda")
    offs = torch.from_numpy(off).cuda()
    for call in range(3):
        h = np.concatenate([data.zipf_keys(n, 200, 1.1, seed=10 * call + i, perm_seed=i + 1).cpu().numpy() if n else
                            np.empty(0, np.uint32) for i, n in enumerate(lengths)])
        keys.copy_(torch.from_numpy(h.view(np.int32)))
        b.insert_graph(keys, offs)
        for s in range(6):
            orcs[s].insert(h[off[s]:off[s + 1]])
    full = b.status()
    for s in range(6):
        low, high = b.stream_tables(s)
        assert np.array_equal(low, orcs[s].low) and np.array_equal(high, orcs[s].high), s
    assert full == (_lib.QS_ERR_POOL_FULL if any(o.pool_full for o in orcs) else _lib.QS_OK)
    assert [bool(v & 1) for v in b.stream_status()] == [bool(o.pool_full) for o in orcs]


@pytest.mark.parametrize("streams", [1023, 1024, 1025])
def test_batches_at_the_edge_of_the_one_thread_per_stream_plan(gpu, streams):
    rng = np.random.default_rng(streams)
    lengths = rng.integers(0, 120, streams)
    lengths[[5, streams - 1]] = [9000, 5000]
    n_low = rng.integers(3, 600, streams).tolist()
    b = BatchedSketches(n_low, [n + 2 for n in n_low], seed_rng=3)
    masks = qs.generate_hashmask(1021, 32, 3, 4, 1)
    off = np.zeros(streams + 1, np.int64)
    off[1:] = np.cumsum(lengths)
    h = data.zipf_keys(int(off[-1]), 200, 1.1, seed=4, perm_seed=1).cpu().numpy()
    keys, offs = torch.from_numpy(h.view(np.int32)).cuda(), torch.from_numpy(off).cuda()
    b.insert_graph(keys, offs)
    b.insert(keys, offs)
    got = b.search(keys, offs).cpu().numpy().view(np.uint32)
    assert b.status() == _lib.QS_OK
    for s, seed in enumerate(b.seeds()):
        o = oracle.Msws(n_low[s], n_low[s] + 2, int(seed), masks)
        mine = h[off[s]:off[s + 1]]
        o.insert(np.concatenate([mine, mine]))
        assert np.array_equal(got[off[s]:off[s + 1]], o.query(mine)), s
