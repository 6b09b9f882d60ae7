"""Chunks of the partitioned insert that link more buckets than there are rows of counts, with pools that
hold all of them, some and few, against the sequential oracle."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import _lib, data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu

ROWS = 65536
MASKS = qs.generate_hashmask(1021, 32, 3, 4, 1)


@pytest.mark.parametrize("n_high", [131100, 90001, 70000, 500])
@pytest.mark.parametrize("compat", [False, True])
@pytest.mark.parametrize("wide", [False, True])
def test_equal_keys_link_together(gpu, n_high, compat, wide):
    # 2^17 keys again and again: the buckets with one of them all cross in the same pass
    n_low = 131071
    masks = qs.generate_hashmask(1021, 32, 5, 4, 1) if wide else MASKS
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, n_high, 32, hash_seed=2654435769, mask_table=masks, compat_v3=compat)
    orc = oracle.Msws(n_low, n_high, 2654435769, masks, compat_v3=compat)
    keys = data.rank_keys(7, 0, 1 << 17).view(torch.int32).repeat(70).view(torch.uint32)
    for _ in range(2):
        sk.insert(keys)
        orc.insert(keys.cpu().numpy())
    for got, want in zip(sk.tables(), (orc.low, orc.high)):
        assert np.array_equal(got, want)
    st = sk.stats()
    assert st["next_level_id"] == orc.next_id and st["dropped_keys"] == orc.dropped
    assert sk.status() == (_lib.QS_ERR_POOL_FULL if orc.pool_full else _lib.QS_OK)
    assert orc.pool_full or orc.next_id - 1025 > ROWS


@pytest.mark.parametrize("pool", [100000, 40000])
@pytest.mark.parametrize("compat", [False, True])
def test_streams_of_a_batch(gpu, pool, compat):
    n_low, n_high = [65521, 65519, 32749], [pool, pool, pool // 2]
    b = BatchedSketches(n_low, n_high, seed_rng=3, compat_v3=compat)
    pieces = [data.rank_keys(5 + s, 0, n).view(torch.int32).repeat(130) for s, n in enumerate(n_low)]
    off = np.zeros(4, np.int64)
    off[1:] = np.cumsum([p.numel() for p in pieces])
    keys = torch.cat(pieces).view(torch.uint32)
    b.insert(keys, torch.from_numpy(off).cuda())
    full, linked = b.status(), 0
    k = keys.cpu().numpy()
    for s, seed in enumerate(b.seeds()):
        orc = oracle.Msws(n_low[s], n_high[s], int(seed), MASKS, compat_v3=compat)
        orc.insert(k[off[s]:off[s + 1]])
        for got, want in zip(b.stream_tables(s), (orc.low, orc.high)):
            assert np.array_equal(got, want)
        assert bool(b.stream_status()[s] & 1) == bool(orc.pool_full)
        linked += orc.next_id - 1025
    assert linked > ROWS or full == _lib.QS_ERR_POOL_FULL
    b.close()
