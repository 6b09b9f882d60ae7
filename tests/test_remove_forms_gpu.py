"""REMOVE (qs_remove.cu) on both sides of its dispatch lines, by calls that its tiles fill and leave
ragged: tables and counts bit for bit as the oracle's."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data

pytestmark = pytest.mark.gpu
SEED, MASKS = 2654435769, qs.generate_hashmask(1021, 32, 3, 4, 1)
WIDE = qs.generate_hashmask(1021, 32, 6, 4, 1)
BLOCKS = 592  # tiles of n / 592 keys, at least 256 and at most 2048; above 1024 the slots are walked


def stream(n, s, seed):
    k = data.uniform_keys(n, seed=seed) if s == 0 else data.zipf_keys(n, 1 << 16, s, seed=seed, perm_seed=4)
    k.view(torch.int32)[:: max(1, n // 7)] = -1  # the all-ones key, which marks an empty slot
    return k


@pytest.mark.parametrize("n_low", [4091, 4096, 4099, 98303, 98304])
@pytest.mark.parametrize("n", [1, 255, 257, BLOCKS * 256 + 1, BLOCKS * 1024, BLOCKS * 1024 + 1, BLOCKS * 2048 + 77])
@pytest.mark.parametrize("s", [0, 1.1])
def test_msws(gpu, n_low, n, s):
    masks = WIDE if n % 2 else MASKS
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, 2048, 32, hash_seed=SEED, mask_table=masks)
    orc = oracle.Msws(n_low, 2048, SEED, masks)
    ins, rem = stream(1 << 19, s, 5), stream(n, s, 6)
    sk.insert(ins)
    orc.insert(ins.cpu().numpy())
    again = qs.from_snapshot(sk.snapshot())  # does not know its counts: the other subtraction
    orc.remove(rem.cpu().numpy())
    for x in (sk, again):
        x.remove(rem)
        low, high = x.tables()
        assert np.array_equal(low, orc.low) and np.array_equal(high, orc.high)
        assert x.stats()["dropped_keys"] == orc.dropped


@pytest.mark.parametrize("n", [1, 257, BLOCKS * 1024 + 1, BLOCKS * 2048 + 77])
@pytest.mark.parametrize("rows", [1, 5])
def test_count_min(gpu, n, rows):
    sk = qs.Sketch_GPU_Thread(4093, rows, seed_rng=4)
    ref = oracle.CountMin(4093, sk.info()["seeds"])
    ins, rem = stream(1 << 19, 1.1, 5), stream(n, 1.1, 6)
    sk.insert(ins)
    ref.insert(ins.cpu().numpy())
    sk.remove(rem)
    ref.remove(rem.cpu().numpy())
    low, _ = sk.tables()
    assert np.array_equal(low, ref.table)
