"""qs_clear and qs_batch_clear leave nothing behind, at the edges of the blocks that write the zeros."""
import numpy as np
import pytest
import torch

import qsketch_b200 as qs
from qsketch_b200 import data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_low,n_high", [(1, 2), (1023, 2), (1024, 256), (1025, 257), (5, 1025), (100003, 4099), (2097143, 70001)])
def test_sketch(gpu, n_low, n_high):
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, n_high, 32, hash_seed=2654435769)
    sk.insert(data.uniform_keys(1 << 21, seed=1))
    sk.clear()
    low, high = sk.tables()
    assert not low.any() and not high.any()
    st = sk.stats()
    assert st["next_level_id"] == 1025 and st["status_bits"] == 0 and st["dropped_keys"] == 0


@pytest.mark.parametrize("streams", [1, 700, 3000])
def test_batch(gpu, streams):
    b = BatchedSketches([7] * streams, [2] * streams, seed_rng=3)
    off = torch.arange(0, streams * 900 + 1, 900, dtype=torch.int64, device="cuda")
    keys = data.zipf_keys(streams * 900, 64, 1.0, seed=2, perm_seed=3)
    first = []
    for _ in range(2):
        b.insert(keys, off)
        assert b.stream_status().any()
        first.append(b.search(keys, off).cpu().numpy())
        b.clear()
        assert not b.stream_status().any() and not b.search(keys, off).cpu().numpy().any()
    assert np.array_equal(*first)
    b.close()
