"""The lines that decide a partitioned insert, each met exactly: the shortest calls it takes, the tile
sizes, the sample for heavy keys, the smallest and the largest tables.  Whether a call went through it is read
from the launch counts (the replay has none of its own there)."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data

pytestmark = pytest.mark.gpu
SEED = 2654435769
MASKS = qs.generate_hashmask(1021, 32, 3, 4, 1)
MIN = 1 << 18          # keys of the shortest partitioned call
TILE, SMALL = 16384, 2048
SMALL_MAX = 74 * TILE  # below it a chunk's tiles are small
HOT_MIN = 3 << 19      # from it on the call is sampled by a kernel of its own


def pair(n_low, n_high):
    sk = qs.Sketch_GPU_Sub_Warp_Level(n_low, 8, n_high, 32, hash_seed=SEED, mask_table=MASKS)
    return sk, oracle.Msws(n_low, n_high, SEED, MASKS)


def insert(sk, orc, keys):
    sk.insert(keys)
    orc.insert(keys.cpu().numpy())


def same(sk, orc):
    low, high = sk.tables()
    assert np.array_equal(low, orc.low) and np.array_equal(high, orc.high)
    st = sk.stats()
    assert st["next_level_id"] == orc.next_id and st["dropped_keys"] == orc.dropped


@pytest.mark.parametrize("n", [MIN - 1, MIN, MIN + 1, MIN + SMALL - 1, MIN + SMALL, MIN + SMALL + 1, 3 * MIN - 1, 3 * MIN,
                               3 * MIN + TILE - 1, 3 * MIN + TILE + 1])
@pytest.mark.parametrize("off", [0, 1])
def test_shortest_calls_and_ragged_tiles(gpu, n, off):
    sk, orc = pair(16381, 4096)
    insert(sk, orc, data.zipf_keys(n + off, 1 << 15, 1.1, seed=n, perm_seed=7)[off:])
    assert (sk.profile()["repair_launches"] == 0) == (n >= MIN)
    same(sk, orc)


@pytest.mark.parametrize("n", [SMALL_MAX - 1, SMALL_MAX, SMALL_MAX + 1, HOT_MIN - 1, HOT_MIN, HOT_MIN + 1])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_one_chunk_at_the_tile_and_sample_lines(gpu, n, off):
    # 2^18 keys first: the next call is one chunk of exactly n keys
    sk, orc = pair(16381, 4096)
    insert(sk, orc, data.zipf_keys(MIN, 1 << 15, 1.1, seed=1, perm_seed=7))
    before = sk.profile()["insert_launches"]
    insert(sk, orc, data.zipf_keys(n + off, 1 << 15, 1.1, seed=n, perm_seed=7)[off:])
    p = sk.profile()
    assert p["repair_launches"] == 0 and p["insert_launches"] - before == (4 if n >= HOT_MIN else 3)
    same(sk, orc)


@pytest.mark.parametrize("n_low,parts", [(655359, 640), (655360, 320), (655361, 321), (1310719, 640), (1310720, 640),
                                         (1310721, 641), (2048 * 2048 - 1, 2048), (2048 * 2048, 2048),
                                         (2048 * 2048 + 1, 0)])
def test_large_tables(gpu, n_low, parts):
    sk, orc = pair(n_low, 8192)
    n = n_low + n_low // 2
    keys = data.zipf_keys(n + 3, 1 << 18, 1.05, seed=n_low, perm_seed=9)
    insert(sk, orc, keys[:n])
    assert (sk.profile()["repair_launches"] == 0) == (parts > 0)
    insert(sk, orc, keys[1:n])  # one key short of the rule: pass 1
    assert sk.profile()["repair_launches"] > 0
    insert(sk, orc, keys[3:])
    same(sk, orc)
