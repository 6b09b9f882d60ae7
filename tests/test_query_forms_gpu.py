"""Queries on both sides of the line between the two forms (tables beyond the L2, long calls) against the
oracle."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data

pytestmark = pytest.mark.gpu
SEED = 2654435769


@pytest.mark.parametrize("n_low", [(1 << 22) - 1, 1 << 22])
@pytest.mark.parametrize("ones", [3, 4])
def test_long_queries_of_large_tables(gpu, n_low, ones):
    masks = qs.generate_hashmask(1021, 32, ones, 4, 1)
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, 4096, 32, hash_seed=SEED, mask_table=masks)
    orc = oracle.Msws(n_low, 4096, SEED, masks)
    keys = data.zipf_keys(1 << 20, 1 << 18, 1.0, seed=3, perm_seed=2)
    sk.insert(keys)
    orc.insert(keys.cpu().numpy())
    q = data.zipf_keys((1 << 23) + 1, 1 << 19, 0.8, seed=5, perm_seed=2)
    want = orc.query(q.cpu().numpy())
    for part in (slice(0, 1 << 23), slice(0, (1 << 23) - 1), slice(1, None), slice(0, 1001)):
        assert np.array_equal(sk.search(q[part]).cpu().numpy(), want[part])
