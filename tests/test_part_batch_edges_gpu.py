"""Batched streams at the edges of the partitioned insert's rounds, partition sizes and windows: every
stream's tables equal the oracle's."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu
MASKS = qs.generate_hashmask(1021, 32, 3, 4, 1)


def check(n_low, calls, s=1.0, **kw):
    """Inserts calls (lists of lengths per stream) and compares every stream's tables and allocator."""
    n_high = [n + 2 for n in n_low]
    b = BatchedSketches(n_low, n_high, seed_rng=3, **kw)
    orcs = [oracle.Msws(n_low[i], n_high[i], int(x), MASKS) for i, x in enumerate(b.seeds())]
    for c, lengths in enumerate(calls):
        off = np.zeros(len(n_low) + 1, np.int64)
        off[1:] = np.cumsum(lengths)
        keys = np.concatenate([data.zipf_keys(int(n), 1 << 14, s, seed=97 * c + i, perm_seed=i + 1).cpu().numpy() if n else
                               np.empty(0, np.uint32) for i, n in enumerate(lengths)])
        b.insert(torch.from_numpy(keys).cuda(), torch.from_numpy(off).cuda())
        for i in range(len(n_low)):
            orcs[i].insert(keys[off[i]:off[i + 1]])
    b.sync()
    for i, o in enumerate(orcs):
        low, high = b.stream_tables(i)
        assert np.array_equal(low, o.low) and np.array_equal(high, o.high), i
    b.close()


FIRST, FOLD = 1 << 17, 1 << 15


@pytest.mark.parametrize("s", [0.6, 1.2])
def test_rests_of_a_stream(gpu, s):
    # the rest beyond the first round folded into it (at most 2^15 keys) or not
    lengths = [FIRST - 1, FIRST, FIRST + 1, FIRST + FOLD, FIRST + FOLD + 1, 32768, 0, 32767, 3 * FIRST]
    n_low = [1021, 16381, 65521, 100003, 131071, 32749, 509, 2039, 4093]
    check(n_low, [lengths, lengths[::-1], [FIRST + FOLD] * 9], s)


@pytest.mark.parametrize("n_low", [79, 1021, 1024, 8191, 16384, 30011])
def test_partitions_of_few_keys(gpu, n_low):
    # keys per partition at the lines where partitions double
    check([n_low] * 5, [[32768, 40000, 65535, 65536, 131071], [163840, 32769, 131073, 262144, 500009]])


def test_no_stream_has_a_rest(gpu):
    check([2039, 4093, 8191], [[40000, 50000, 60000], [163840, 131072, 100]])


@pytest.mark.parametrize("max_batch", [1 << 14, 1 << 15, 1 << 16])
def test_small_scratch(gpu, max_batch):
    # first rounds of 2^14, 2^15 and 2^16 keys, rests of more than a window, a large table
    check([2039, 30011, 1048573, 509], [[40960, 40961, 1100003, 36864], [81920, 300007, 0, 32768]], max_batch=max_batch)
