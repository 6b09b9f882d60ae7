"""REMOVE beside calls recorded into a caller's CUDA graph: replays insert keys that no call counted,
so counters of 2^31 and more must lose their removals like any other."""
import pytest
import torch

import qsketch_b200 as qs

pytestmark = pytest.mark.gpu

PIECE, REPLAYS = 1 << 24, 130  # 2.18e9 occurrences of one key, above 2^31
KEY = 77


def sketch(kind):
    if kind == "msws":
        return qs.Sketch_GPU_Sub_Warp_Level(2039, 8, 64, 32, hash_seed=2654435769)
    return qs.Sketch_GPU_Thread(2039, 3) if kind == "cm" else qs.Sketch_GPU_Warp(2039, 32, hash_seed=2654435769)


def record(fn):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fn()
    return g


@pytest.mark.parametrize("kind", ["msws", "cm", "bucket"])
def test_counters_above_2_31(gpu, kind):
    keys = torch.full((PIECE,), KEY, dtype=torch.int32, device="cuda")
    one = keys[:1].clone()
    sk = sketch(kind)
    sk.insert(keys[:1000])
    sk.remove(keys[:1000])
    taken = record(lambda: sk.remove(keys[:1003]))  # recorded while the counters are small
    taken.replay()
    sk.clear()
    ins = record(lambda: sk.insert(keys))
    sk.clear()
    for _ in range(REPLAYS):
        ins.replay()
    count = PIECE * REPLAYS
    assert int(sk.search(one).to(torch.int64).item()) & 0xffffffff == count
    sk.remove(keys[:5000])
    taken.replay()
    assert int(sk.search(one).to(torch.int64).item()) & 0xffffffff == count - 5000 - 1003
    # a captured clear has cleared nothing: the bound stays unknown
    record(sk.clear)
    sk.remove(keys[:11])
    assert int(sk.search(one).to(torch.int64).item()) & 0xffffffff == count - 5000 - 1003 - 11
