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


@pytest.mark.parametrize("side", [False, True])
def test_host_calls_wait_for_device_calls(gpu, side):
    # the clear of a 512 MB sketch takes longer than the copy of a few keys, an insert of 2^24 keys
    # longer than both
    n_low, n_high = 8388593, 1 << 21
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, n_high, 32, hash_seed=2654435769, mask_table=MASKS)
    orc = oracle.Msws(n_low, n_high, 2654435769, MASKS)
    st = torch.cuda.Stream() if side else torch.cuda.current_stream()
    big = data.zipf_keys(1 << 24, 1 << 12, 1.0, seed=8, perm_seed=5)
    few = big[:3001].cpu()
    h = torch.empty(few.numel(), dtype=torch.int32).pin_memory()
    keys = few.view(torch.int32).pin_memory()
    sk.insert_host(keys)
    torch.cuda.synchronize()
    for _ in range(3):
        sk.clear(stream=st)
        sk.insert_host(keys)
        sk.search_host(keys, h)
        assert np.array_equal(h.numpy().view(np.uint32), one_pass(orc, few))
    sk.clear(stream=st)
    sk.insert(big, stream=st)
    sk.search_host(keys, h)
    orc = oracle.Msws(n_low, n_high, 2654435769, MASKS)
    orc.insert(big.cpu().numpy())
    assert np.array_equal(h.numpy().view(np.uint32), orc.query(few.numpy()))
    sk.remove(big, stream=st)
    sk.search_host(keys, h)
    orc.remove(big.cpu().numpy())
    assert np.array_equal(h.numpy().view(np.uint32), orc.query(few.numpy()))


def one_pass(orc, keys):
    """Estimates of `keys` after inserting them once into an empty sketch (computed once)."""
    if not hasattr(orc, "once"):
        orc.insert(keys.numpy())
        orc.once = orc.query(keys.numpy())
    return orc.once
