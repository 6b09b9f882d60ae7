"""REMOVE of heavy keys (qs_remove): merging within tiles and subtractions that go below zero on the
way, against the oracle."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["msws", "cm", "bucket"])
@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 300001])
def test_remove_heavy_keys_below_zero(gpu, kind, n):
    # a few keys, among them the all-ones key, removed far more often than they were inserted and
    # from many tiles at once: every counter ends at 0 or at its exact difference
    rng = np.random.default_rng(n)
    pool = np.concatenate([rng.integers(0, 1 << 32, 40, dtype=np.uint64).astype(np.uint32), [0xffffffff, 0]]).astype(np.uint32)
    w = 1.0 / np.arange(1, pool.size + 1)
    rng.shuffle(pool)
    ins = pool[rng.choice(pool.size, 200003, p=w / w.sum())]
    rem = pool[rng.choice(pool.size, n)]
    d = lambda a: torch.from_numpy(a).cuda()
    if kind == "msws":
        masks = qs.generate_hashmask(1021, 32, 3, 4, 1)
        sk = qs.Sketch_GPU_Sub_Warp_Level(509, 8, 64, 32, hash_seed=2654435769, mask_table=masks)
        ref = oracle.Msws(509, 64, 2654435769, masks)
    elif kind == "cm":
        sk = qs.Sketch_GPU_Thread(1021, 3, seed_rng=4)
        ref = oracle.CountMin(1021, sk.info()["seeds"])
    else:
        sk = qs.Sketch_GPU_Warp(509, 16, hash_seed=2654435769)
        inf = sk.info()
        ref = oracle.BucketSketch(509, 16, 2654435769, inf["mask_table"])
    sk.insert(d(ins))
    ref.insert(ins)
    for _ in range(3):
        sk.remove(d(rem))
        ref.remove(rem)
        assert np.array_equal(sk.search(d(pool)).cpu().numpy(), ref.query(pool))
    if kind == "msws":
        low, high = sk.tables()
        assert np.array_equal(low, ref.low) and np.array_equal(high, ref.high)
        # a restored sketch does not know how large its counters can be: the other subtraction
        again = qs.from_snapshot(sk.snapshot())
        again.remove(d(rem))
        ref.remove(rem)
        assert np.array_equal(again.search(d(pool)).cpu().numpy(), ref.query(pool))
