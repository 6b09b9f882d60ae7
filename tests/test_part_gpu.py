"""The partitioned insert (large calls with default knobs) against the sequential CPU oracle, at the
edges of its tiles, partitions, mask forms and fallbacks: estimates, tables and allocator bit for
bit."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import _lib, data

pytestmark = pytest.mark.gpu

SEED = 2654435769


def pair(n_low, n_high, masks=None, compat=False, **kw):
    if masks is None:
        masks = qs.generate_hashmask(1021, 32, 3, 4, 1)
    h = masks.size // 4
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, n_high, 32, 1, h, hash_seed=SEED, mask_table=masks, compat_v3=compat, **kw)
    return sk, oracle.Msws(n_low, n_high, SEED, masks, compat_v3=compat)


def compare(sk, orc, pieces, queries, full=False):
    for p in pieces:
        sk.insert(p)
        orc.insert(p.cpu().numpy())
    got = sk.search(queries).cpu().numpy()
    assert sk.status() == (_lib.QS_ERR_POOL_FULL if full else _lib.QS_OK)
    assert np.array_equal(got, orc.query(queries.cpu().numpy()))
    low, high = sk.tables()
    assert np.array_equal(low, orc.low)
    assert np.array_equal(high, orc.high)
    st = sk.stats()
    assert st["next_level_id"] == orc.next_id and st["dropped_keys"] == orc.dropped


@pytest.mark.parametrize("n", [65535, 65536, 65537, 131071, 262144, 524289, 2424831, 2424832, 4194301])
@pytest.mark.parametrize("off", [0, 1])
def test_sizes_at_tile_edges_and_alignments(gpu, n, off):
    sk, orc = pair(16381, 4096)
    keys = data.zipf_keys(n + off, 1 << 15, 1.1, seed=n, perm_seed=7)[off:]
    compare(sk, orc, [keys], data.rank_keys(7, 0, 1 << 15))


@pytest.mark.parametrize("n", [74 * 16384 - 1, 74 * 16384, (3 << 19) - 1, 3 << 19])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_second_call_at_the_edges_of_tile_size_and_heavy_key_sample(gpu, n, off):
    sk, orc = pair(16381, 4096)
    first, keys = data.zipf_keys(5000, 1 << 15, 1.1, seed=n, perm_seed=7), data.zipf_keys(n + off, 1 << 15, 1.1, seed=n, perm_seed=7)
    compare(sk, orc, [first, keys[off:]], data.rank_keys(7, 0, 1 << 15))


@pytest.mark.parametrize("n_low", [449, 512, 513, 2039, 40961, 655359, 655361, 1310719, 1310721])
def test_table_sizes_at_partition_edges(gpu, n_low):
    sk, orc = pair(n_low, 8192)
    keys = data.zipf_keys(1 << 20, 1 << 16, 1.05, seed=n_low, perm_seed=9)
    compare(sk, orc, [keys, keys[: 1 << 19]], data.rank_keys(9, 0, 1 << 16))


@pytest.mark.parametrize("ones,count", [(1, 1021), (2, 64), (3, 1), (3, 2048), (5, 1021), (28, 7)])
@pytest.mark.parametrize("compat", [False, True])
def test_mask_forms(gpu, ones, count, compat):
    masks = qs.generate_hashmask(count, 32, ones, 4, 5)
    sk, orc = pair(8191, 8192, masks, compat)
    keys = data.zipf_keys(700001, 1 << 14, 1.0, seed=ones, perm_seed=3)
    compare(sk, orc, [keys], data.rank_keys(3, 0, 1 << 14))


def test_heavy_key_of_an_unlinked_bucket(gpu):
    # whole tiles of one key that no earlier chunk linked: more records than are sorted, so the
    # switching key is found by bisection; then the same key linked
    sk, orc = pair(16381, 4096)
    uni = data.uniform_keys(1 << 19, seed=3)
    one = torch.full((3 << 20,), 77, dtype=torch.int64, device="cuda").to(torch.uint32)
    two = one.clone().view(torch.int32)
    two[::3] = 12345
    compare(sk, orc, [uni, one, two.view(torch.uint32)], torch.cat([one[:1], two[:1].view(torch.uint32), uni[:4096]]))


@pytest.mark.parametrize("n_high", [8, 300])
def test_pool_runs_out(gpu, n_high):
    sk, orc = pair(8191, n_high)
    keys = data.zipf_keys(3 << 20, 1 << 14, 1.0, seed=12, perm_seed=13)
    compare(sk, orc, [keys], data.rank_keys(13, 0, 1 << 14), full=True)


@pytest.mark.parametrize("compat", [False, True])
def test_more_links_in_a_chunk_than_rows(gpu, compat):
    # one mask for all keys and ~170 keys per bucket: nearly all of 98,299 buckets link in the
    # second chunk, more than a block's accumulators and than the 65,536 rows
    masks = np.full(1021, (1 << 0) | (1 << 5) | (1 << 9), np.uint32).view(np.uint8).copy()
    sk, orc = pair(98299, 98400, masks, compat)
    keys = data.uniform_keys((1 << 18) + (1 << 24), seed=5)
    compare(sk, orc, [keys], keys[: 1 << 20])
    assert orc.next_id - 1025 > 65536


def test_same_result_as_pass_1_in_many_calls(gpu):
    # a caller that fixes a pass-1 knob keeps pass 1: both paths, call after call, give one state
    a, _ = pair(262139, 1 << 14)
    b, _ = pair(262139, 1 << 14, lanes_per_key=4)
    for i, n in enumerate([70001, 300007, 1 << 20, 5 << 20, 65536]):
        keys = data.zipf_keys(n, 1 << 18, 1.2, seed=40 + i, perm_seed=8)
        a.insert(keys)
        b.insert(keys)
        for x, y in zip(a.tables(), b.tables()):
            assert np.array_equal(x, y)
    assert a.stats()["next_level_id"] == b.stats()["next_level_id"] > 1100
