"""The order in which the batched SVD's pair solve rotates its 64 columns (svd.cu,
QuadClass): a step whose groups overlapped would race on the Gram matrix, a pair that no
group holds would never be rotated."""
import numpy as np

from dmrgcc_b200 import capi


def test_solve_groups_cover_every_pair_once():
    steps = capi.svd_solve_groups()
    met = np.zeros((64, 64), dtype=np.int64)
    for groups in steps:
        assert sorted(groups.ravel().tolist()) == list(range(64))  # a step's groups are disjoint
        for g in groups:
            met[np.ix_(g, g)] += 1
    assert np.array_equal(met[np.triu_indices(64, 1)], np.ones(64 * 63 // 2, dtype=np.int64))


def test_solve_groups_hit_distinct_banks():
    # 16 neighbouring threads read the same place of the 16 groups: 8-byte banks are columns mod 16
    for groups in capi.svd_solve_groups():
        for place in groups.T:
            assert len(set((place % 16).tolist())) == 16
