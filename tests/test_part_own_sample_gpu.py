"""Heavy keys of short partitioned calls (sampled by the split's own blocks, warm sketches) against the
oracle: linked and unlinked ones, the all-ones key, ragged tiles, every mask form, and call sizes on
both sides of the tile sizes and of the call-wide sample."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data

pytestmark = pytest.mark.gpu
SEED = 2654435769


def heavy(n, parts, seed):
    """n uniform keys, overwritten by `parts` = [(key, share)] at pseudo-random places."""
    k = data.uniform_keys(n, seed=seed).view(torch.int32)
    g = torch.Generator(device="cuda").manual_seed(seed)
    u, lo = torch.rand(n, generator=g, device="cuda"), 0.0
    for key, share in parts:
        k[(u >= lo) & (u < lo + share)] = key
        lo += share
    return k.view(torch.uint32)


@pytest.mark.parametrize("n", [1 << 18, (1 << 18) + 1, 74 * 16384 - 1, 74 * 16384, (3 << 19) - 1, 3 << 19])
@pytest.mark.parametrize("parts", [[(77, 1.0)], [(-1, 0.6), (5, 0.3)], [(1000 + i, 0.01) for i in range(60)],
                                   [(9, 0.004), (10, 0.02), (11, 0.002)]])
def test_warm_calls(gpu, n, parts):
    masks = qs.generate_hashmask(1021, 32, 3 + n % 2, 4, 1)
    compat = n % 3 == 0
    sk = qs.Sketch_GPU_Sub_Warp_Level(16381, 8, 4096, 32, hash_seed=SEED, mask_table=masks, compat_v3=compat)
    orc = oracle.Msws(16381, 4096, SEED, masks, compat_v3=compat)
    # the first half of the heavy keys is linked when the call comes, the others are not
    warm = heavy(1 << 18, [(k, s / 2) for k, s in parts[: (len(parts) + 1) // 2]], 3)
    keys = heavy(n + 1, parts, n)
    for piece in (warm, keys[1:], keys[:-1]):
        sk.insert(piece)
        orc.insert(piece.cpu().numpy())
    assert sk.profile()["repair_launches"] == 0
    low, high = sk.tables()
    assert np.array_equal(low, orc.low) and np.array_equal(high, orc.high)
    st = sk.stats()
    assert st["next_level_id"] == orc.next_id and st["dropped_keys"] == orc.dropped
