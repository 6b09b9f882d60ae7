"""Calls that take no stream leave nothing in flight, and calls on internal streams start after the
caller's: what follows on another stream sees their results."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu

MASKS = qs.generate_hashmask(1021, 32, 3, 4, 1)


def test_insert_on_a_side_stream_after_the_batch_tuner(gpu):
    # a 400 MB arena: the tuner's last clear is still running when the call below is issued, unless
    # the tuner waits for it
    n_low, n_high = [4194301, 4194301, 2097143], [4096, 4096, 4096]
    b = BatchedSketches(n_low, n_high, seed_rng=3)
    lengths = [30011, 20011, 5003]
    off = np.zeros(4, np.int64)
    off[1:] = np.cumsum(lengths)
    keys = data.zipf_keys(int(off[-1]), 1 << 10, 1.2, seed=4, perm_seed=6)
    offsets, side = torch.from_numpy(off).cuda(), torch.cuda.Stream()
    torch.cuda.synchronize()
    b.autotune(keys, offsets, reps=1)
    b.insert(keys, offsets, total=int(off[-1]), stream=side)
    b.sync(stream=side)
    k = keys.cpu().numpy()
    for s, seed in enumerate(b.seeds()):
        orc = oracle.Msws(n_low[s], n_high[s], int(seed), MASKS)
        orc.insert(k[off[s]:off[s + 1]])
        low, high = b.stream_tables(s)
        assert np.array_equal(low, orc.low) and np.array_equal(high, orc.high)
    b.close()
