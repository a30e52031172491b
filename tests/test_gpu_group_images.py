"""Periodic neighbour lists of every particle by the group search (70,001 uniform particles):
the reference's image gates against the restatement, the minimum image against the search of
given targets, a warp each, and against brute force; at the slot switches of k, sides as short
as the lists are wide (a particle's own images among its neighbours, groups on both sides of a
half period, images searched with larger offsets than the group's own) and groups on a wall."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import PERIODIC_MIN_IMAGE, KDTree
from tests.helpers import assert_knn_equal, d2_ref, reflect_images, rows_by_id, to_ids

pytestmark = pytest.mark.gpu

N = 70001
CASES = [([1.0, 1.0, 1.0], 31), ([1.0, 1.0, 1.0], 33), ([1.0, 0.25, 2.0], 32),
         ([1.0, 1.0, 0.01], 32), ([1.0, 1.0, 0.01], 64), ([1.0, 1.0, 2e-3], 31),
         ([1.0, 1.0, 1e-6], 16), ([1.0, 0.02, 0.02], 32), ([1.0, 0.01, 0.03], 100)]


def tree(per, seed=17):
    pos = np.random.default_rng(seed).random((N, 3)) * per
    return pos, KDTree(pos, None, np.ones(N), 16, kerntype=0, period=per)


@pytest.mark.parametrize("per,k", CASES)
@pytest.mark.parametrize("method", [0, 1])
def test_reference_gates(gpu, port_built, per, k, method):
    pos, t = tree(per)
    o = oracle.OracleTree(pos, None, np.ones(N), 16, 0, 0, 1000, per, backend="port", nthreads=8)
    nn, d2 = (t.FindNearest if method == 0 else t.FindNearestPos)(k)
    perm = t.GetPerm()
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), *o.knn(k, method),
                     f"method {method}, period {per}", dropped_nearest=method == 0)


@pytest.mark.parametrize("per,k", CASES)
def test_minimum_image(gpu, per, k):
    pos, t = tree(per)
    nn, d2 = t.FindNearest(k, periodic_mode=PERIODIC_MIN_IMAGE)
    targets = np.arange(N, dtype=np.int32)
    tn, td = t.FindNearestTargets(targets, k, periodic_mode=PERIODIC_MIN_IMAGE)
    assert_knn_equal(nn, d2, tn, td, f"period {per}", dropped_nearest=True)
    # and all pairs for some: every image that the search may take, the query itself left out
    x = pos[t.GetPerm()]
    some = np.random.default_rng(3).choice(N, 40, replace=False)
    if min(per) < 0.1:
        return  # with images at the lists' own width the gates decide which are searched
    for i in some:
        d = np.min([d2_ref(q, x) for q in reflect_images(x[i:i + 1], per)[:, 0]], axis=0)
        d[i] = np.inf
        assert np.array_equal(np.sort(d)[:k], d2[i])
