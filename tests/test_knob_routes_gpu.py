"""A caller that fixes a pass-1 knob keeps pass 1 and the replay, whatever the size of its calls."""
import numpy as np
import pytest
import torch

import qsketch_b200 as qs
from qsketch_b200 import data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("knobs", [{}, {"first_chunk": 1 << 16}, {"lanes_per_key": 4}, {"keys_per_tile": 1024},
                                   {"chunk_ramp": False}])
@pytest.mark.parametrize("n", [1000, 1 << 20])
def test_sketch(gpu, knobs, n):
    sk = qs.Sketch_GPU_Sub_Warp_Level(16381, 8, 4096, 32, hash_seed=2654435769, **knobs)
    sk.insert(data.zipf_keys(n, 1 << 12, 1.1, seed=3, perm_seed=4))
    assert (sk.profile()["repair_launches"] > 0) == bool(knobs)


@pytest.mark.parametrize("knobs", [{}, {"class_lanes_per_key": {10: 8}}, {"first_chunk": 1 << 12}, {"lanes_per_key": 2},
                                   {"chunk_ramp": False}])
def test_batch_graph(gpu, knobs):
    b = BatchedSketches([2039] * 8, [64] * 8, seed_rng=3, **knobs)
    off = torch.arange(0, 8 * 2000 + 1, 2000, dtype=torch.int64, device="cuda")
    keys = data.zipf_keys(16000, 100, 1.2, seed=5, perm_seed=6)
    b.insert_graph(keys, off)
    b.sync()
    # the replay counts the calls that found crossed buckets; the one-block insert is not it
    assert (b.profile()["repairs_active"] > 0) == bool(knobs)
    b.close()
