"""The partitioned insert on tables at the edges of its partition sizes, and just outside them, against the
oracle; whether a call went through it is read from the launch counts."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data

pytestmark = pytest.mark.gpu
SEED = 2654435769


@pytest.mark.parametrize("n_low,parts", [(496, 0), (497, 32), (512, 32), (513, 33), (1021, 64), (4095, 256), (4096, 128),
                                         (8191, 256), (8192, 128), (16383, 256), (16384, 256), (40959, 640), (40960, 320)])
@pytest.mark.parametrize("s", [0.7, 1.2])
def test_small_tables(gpu, n_low, parts, s):
    masks = qs.generate_hashmask(1021, 32, 3, 4, 1)
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, n_low + 1, 32, hash_seed=SEED, mask_table=masks)
    orc = oracle.Msws(n_low, n_low + 1, SEED, masks)
    for i, n in enumerate([(1 << 18) + 11, 900001, 1 << 18]):
        keys = data.zipf_keys(n, 1 << 16, s, seed=n, perm_seed=9)
        sk.insert(keys)
        orc.insert(keys.cpu().numpy())
    assert (sk.profile()["repair_launches"] == 0) == (parts > 0)
    low, high = sk.tables()
    assert np.array_equal(low, orc.low) and np.array_equal(high, orc.high)
    assert sk.stats()["next_level_id"] == orc.next_id
