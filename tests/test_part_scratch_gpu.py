"""The scratch of the partitioned insert follows one chunk size, also where the autotuner chose it."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import _lib, autotune, data
from qsketch_b200.batch import BatchedSketches

pytestmark = pytest.mark.gpu


@pytest.fixture
def tuned():
    """tuned(n_low, max_batch): an entry of that chunk size for n_low's size class."""
    def entry(n_low, max_batch):
        best, _ = autotune.autotune(n_low, 4096, data.zipf_keys(1 << 18, 1 << 15, 1.1, seed=1, perm_seed=2), reps=1,
                                    max_batch=max_batch)
        assert best["max_batch"] == max_batch and autotune.lookup(n_low)["max_batch"] == max_batch
    autotune.reset()
    yield entry
    autotune.reset()


def test_batch_windows_fit_the_scratch_of_a_tuned_chunk_size(gpu, tuned):
    n_low, n_high = [16381, 65521, 4093], [4096, 8192, 1024]
    tuned(sum(n_low), 1 << 20)
    p = _lib.qs_batch_params()
    _lib.lib.qs_batch_params_default(ctypes.byref(p))
    nl, nh = np.array(n_low, np.uint64), np.array(n_high, np.uint64)
    p.n_streams, p.n_low, p.n_high, p.seed_rng, p.max_batch = 3, nl.ctypes.data, nh.ctypes.data, 3, 0
    h = ctypes.c_void_p()
    _lib.check(_lib.lib.qs_batch_create(ctypes.byref(p), ctypes.byref(h)), "create")
    b = BatchedSketches.__new__(BatchedSketches)
    b._h, b.n_streams, b.n_low, b.n_high = h, 3, nl, nh
    assert b.info()["max_batch"] == 1 << 20
    # one stream alone, then all together, exceed a window of 4 * 2^20 keys
    lengths = [5000011, 3000017, 300007]
    off = np.zeros(4, np.int64)
    off[1:] = np.cumsum(lengths)
    keys = np.concatenate([data.zipf_keys(n, 1 << 15, 1.0, seed=40 + i, perm_seed=i + 1).cpu().numpy()
                           for i, n in enumerate(lengths)])
    b.insert(torch.from_numpy(keys).cuda(), torch.from_numpy(off).cuda())
    b.sync()
    for s, seed in enumerate(b.seeds()):
        orc = oracle.Msws(n_low[s], n_high[s], int(seed), qs.generate_hashmask(1021, 32, 3, 4, 1))
        orc.insert(keys[off[s]:off[s + 1]])
        low, high = b.stream_tables(s)
        assert np.array_equal(low, orc.low) and np.array_equal(high, orc.high)
    b.close()


@pytest.mark.parametrize("max_batch", [4096, 1 << 20, 1 << 21])
def test_a_tuned_chunk_size_does_not_cut_the_partitioned_chunks(gpu, tuned, max_batch):
    def sketch():
        return qs.Sketch_GPU_Sub_Warp_Level(65521, 8, 8192, 32, hash_seed=2654435769)
    keys = [data.zipf_keys(n, 1 << 16, 1.1, seed=n, perm_seed=3) for n in (9000011, 1 << 22, 70001)]
    plain = sketch()
    tuned(65521, max_batch)
    other = sketch()
    for i, k in enumerate(keys):
        for sk in (plain, other):
            sk.insert(k)
            if i < 2:
                assert sk.profile()["repair_launches"] == 0
    for i in range(2):
        assert np.array_equal(plain.tables()[i], other.tables()[i])
    plain.clear()
    other.clear()
    launches = [sk.profile()["insert_launches"] for sk in (plain, other)]
    for sk in (plain, other):
        sk.insert(keys[0])
    assert plain.profile()["insert_launches"] - launches[0] == other.profile()["insert_launches"] - launches[1]
