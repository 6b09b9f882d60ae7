"""Routed inserts of the learned split through the partitioned path: the exact table plus a plain
sketch fed only the other keys give the same answers."""
import numpy as np
import pytest
import torch

import oracle
import qsketch_b200 as qs
from qsketch_b200 import data
from qsketch_b200.learned import LearnedSketch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,slots,ranks", [(1 << 19, 1 << 10, 1 << 12), ((1 << 20) + 3, 1 << 12, 1 << 15),
                                           ((3 << 20) + 1, 1 << 15, 1 << 17)])
def test_routed_inserts_equal_table_plus_sketch(gpu, n, slots, ranks):
    lk = LearnedSketch(budget_bytes=4 << 20, warmup_keys=1 << 16, table_slots=slots)
    keys = data.zipf_keys(n, ranks, 1.1, seed=n, perm_seed=5)
    admitted = data.rank_keys(5, 0, slots).cpu().numpy()  # more than fit: the table fills up
    lk.admit_keys(admitted)
    lk.insert(keys)
    lk.insert(keys[1:])  # unaligned
    tk, tc, seed = lk.table()
    assert lk.info()["table_fill"] == tk.size > slots // 2
    h = keys.cpu().numpy()
    both = np.concatenate([h, h[1:]])
    inside = np.isin(both, tk)
    u, c = np.unique(both[inside], return_counts=True)
    exact = dict(zip(u.tolist(), c.tolist()))
    assert [exact.get(int(k), 0) for k in tk] == tc.tolist()
    i = lk.info()
    ref = oracle.Msws(int(i["n_low"]), int(i["n_high"]), int(seed), qs.generate_hashmask(1021, 32, 3, 4, 1))
    ref.insert(both[~inside])
    q = data.rank_keys(5, 0, ranks).cpu().numpy()
    want = ref.query(q) + np.array([exact.get(int(k), 0) for k in q], np.uint32)
    assert np.array_equal(lk.search(torch.from_numpy(q).cuda()).cpu().numpy(), want)
