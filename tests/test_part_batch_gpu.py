"""Batched streams through the partitioned insert: every stream equals the same stream alone (the
oracle), tables, allocators and exhausted pools included."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import _lib, data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu

MASKS = qs.generate_hashmask(1021, 32, 3, 4, 1)


def check(b, streams, n_low, n_high, calls):
    orcs = [oracle.Msws(int(n_low[s]), int(n_high[s]), int(seed), MASKS, compat_v3=b.compat)
            for s, seed in enumerate(b.seeds())]
    for keys, off in calls:
        b.insert(torch.from_numpy(keys).cuda(), torch.from_numpy(off).cuda())
        for s in range(streams):
            orcs[s].insert(keys[off[s]:off[s + 1]])
    full = b.status()
    for s in range(streams):
        low, high = b.stream_tables(s)
        assert np.array_equal(low, orcs[s].low), f"stream {s}: low table"
        assert np.array_equal(high, orcs[s].high), f"stream {s}: high pool"
    assert full == (_lib.QS_ERR_POOL_FULL if any(o.pool_full for o in orcs) else _lib.QS_OK)
    assert [bool(v & 1) for v in b.stream_status()] == [bool(o.pool_full) for o in orcs]


def batch(n_low, n_high, compat=False, **kw):
    b = BatchedSketches(n_low, n_high, seed_rng=3, compat_v3=compat, **kw)
    b.compat = compat
    return b


def draw(lengths, seed, s=1.1, ranks=1 << 14):
    off = np.zeros(len(lengths) + 1, np.int64)
    off[1:] = np.cumsum(lengths)
    keys = np.empty(off[-1], np.uint32)
    for i, n in enumerate(lengths):
        if n:
            keys[off[i]:off[i + 1]] = data.zipf_keys(int(n), ranks, s, seed=seed * 1000 + i, perm_seed=i + 1).cpu().numpy()
    return keys, off


# lengths at the edges of the first round, the tiles and the rule; sketches at the edges of the partitions
LENGTHS = [32767, 32768, 32769, 0, 1, 131072, 131073, 100001, 262144, 600011]
LOWS = [63, 64, 1021, 1024, 1025, 16381, 32749, 131071, 131073, 5003]


@pytest.mark.parametrize("compat", [False, True])
@pytest.mark.parametrize("pool", [4, 100000])
def test_every_stream_equals_itself_alone(gpu, compat, pool):
    n_low = LOWS
    n_high = [min(n + 2, pool) for n in n_low]
    calls = [draw(LENGTHS, 1), draw(LENGTHS[::-1], 2, s=1.3), draw([50000] * 10, 3)]
    check(batch(n_low, n_high, compat), 10, n_low, n_high, calls)


def test_small_windows_and_long_streams(gpu):
    # max_batch 2^14: windows of 2^16 keys, so streams are split over windows
    n_low, n_high = [2039, 8191, 509, 65521], [2041, 8193, 511, 65523]
    check(batch(n_low, n_high, max_batch=1 << 14), 4, n_low, n_high,
          [draw([300007, 70000, 65536, 131073], 5), draw([65537, 0, 200000, 66000], 6)])


def test_more_links_in_a_window_than_rows(gpu):
    masks = np.full(1021, (1 << 0) | (1 << 5) | (1 << 9), np.uint32).view(np.uint8).copy()
    n_low, n_high = [50021, 40009, 1021], [50100, 40100, 1100]
    lengths = [50021 * 165, 40009 * 165, 40000]
    off = np.zeros(4, np.int64)
    off[1:] = np.cumsum(lengths)
    keys = data.uniform_keys(int(off[-1]), seed=9).cpu().numpy()
    p = _lib.qs_batch_params()
    b = batch(n_low, n_high)
    import ctypes
    # the class has no mask_table argument: build the batch through the C ABI
    b.close()
    _lib.lib.qs_batch_params_default(ctypes.byref(p))
    nl, nh = np.array(n_low, np.uint64), np.array(n_high, np.uint64)
    p.n_streams, p.n_low, p.n_high, p.seed_rng = 3, nl.ctypes.data, nh.ctypes.data, 3
    p.mask_table = masks.ctypes.data
    h = ctypes.c_void_p()
    _lib.check(_lib.lib.qs_batch_create(ctypes.byref(p), ctypes.byref(h)), "create")
    b._h, b.n_streams, b.n_low, b.n_high = h, 3, nl, nh
    orcs = [oracle.Msws(n_low[s], n_high[s], int(seed), masks) for s, seed in enumerate(b.seeds())]
    b.insert(torch.from_numpy(keys).cuda(), torch.from_numpy(off).cuda())
    b.sync()
    for s in range(3):
        orcs[s].insert(keys[off[s]:off[s + 1]])
        low, high = b.stream_tables(s)
        assert np.array_equal(low, orcs[s].low) and np.array_equal(high, orcs[s].high)
    assert sum(o.next_id - 1025 for o in orcs) > 65536
