"""Every particle's search on both sides of the lines from which it goes by groups, for even and
for clustered particles (the tree is asked which it holds) and long lists: rows against the
restatement bit-exact, sums to the path's 1e-12."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from tests.helpers import assert_density_close, assert_knn_equal, rows_by_id, to_ids

pytestmark = pytest.mark.gpu


def inputs(kind, n):
    rng = np.random.default_rng(n)
    if kind == "even":
        return rng.random((n, 3)), rng.random(n) + 0.5, rng.normal(size=(n, 3))
    if kind == "same":  # one place for all but a few: every box above them is a point
        pos = np.full((n, 3), 0.5)
        pos[: n // 4] = rng.random((n // 4, 3))
        pos[n // 4:] += rng.random((n - n // 4, 3)) * 1e-9
        return pos, rng.random(n) + 0.5, rng.normal(size=(n, 3))
    pos, mass, vel = syn.clustered_box(n, 1.0, seed=n, nspheres=8, velocities=True)
    return pos, mass, vel


@pytest.mark.parametrize("kind,n,k", [
    ("even", 16383, 32), ("even", 16384, 32), ("clustered", 16384, 32), ("clustered", 49151, 16),
    ("clustered", 49152, 16), ("even", 24577, 33), ("clustered", 98303, 8),
    ("clustered", 98304, 32), ("even", 8191, 100), ("even", 8192, 100), ("clustered", 8193, 65),
    ("same", 20001, 8),
])
def test_without_images(gpu, port_built, kind, n, k):
    pos, mass, vel = inputs(kind, n)
    o = oracle.OracleTree(pos, vel, mass, 16, 0, 0, 1000, None, backend="port", nthreads=16)
    t = KDTree(pos, vel, mass, 16, kerntype=0)
    perm = t.GetPerm()
    nn, d2 = t.FindNearest(k)
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), *o.knn(k, 0), kind)
    assert_density_close(t.CalcDensity(k), o.density(k), "density")
    assert_density_close(t.CalcVelDensity(k // 2, k), o.veldensity(k // 2, k), "veldensity")
    t.close()


@pytest.mark.parametrize("kind,n,k", [
    ("even", 32767, 32), ("even", 32768, 32), ("clustered", 32768, 32), ("clustered", 98304, 32),
    ("even", 65536, 33), ("even", 8192, 64), ("clustered", 8192, 64), ("clustered", 163841, 40),
])
def test_with_images(gpu, port_built, kind, n, k):
    pos, mass, _ = inputs(kind, n)
    per = [1.0, 1.0, 1.0]
    o = oracle.OracleTree(pos, None, mass, 16, 0, 0, 1000, per, backend="port", nthreads=16)
    t = KDTree(pos, None, mass, 16, kerntype=0, period=per)
    perm = t.GetPerm()
    nn, d2 = t.FindNearest(k)
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), *o.knn(k, 0), kind)
    t.close()


@pytest.mark.parametrize("n", [8193, 24577])
def test_velocity_tree(gpu, port_built, n):
    """The same searches over velocities, and many points in velocity space."""
    from nbodylib_gb300.kdtree import TVEL
    rng = np.random.default_rng(n)
    pos, vel = rng.random((n, 3)), rng.normal(size=(n, 3))
    o = oracle.OracleTree(vel, None, np.ones(n), 16, 0, 0, 1000, None, backend="port", nthreads=16)
    t = KDTree(pos, vel, np.ones(n), 16, treetype=TVEL, kerntype=0)
    perm = t.GetPerm()
    nn, d2 = t.FindNearestVel(16)
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), *o.knn(16, 0))
    x = np.repeat(vel[perm], (1 << 17) // n + 1, axis=0) + 1e-4
    nn, d2 = t.FindNearestPoints(x, 8)
    assert_knn_equal(to_ids(nn, perm), d2, *o.knn_pos(x, 8))
    t.close()
