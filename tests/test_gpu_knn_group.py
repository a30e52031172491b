"""The group search (every particle of a tree at once) at the sizes where its groups, buffers
and lists change: neighbour rows against the restatement (bit-exact), densities and velocity
densities against it to the path's 1e-12."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import PERIODIC_MIN_IMAGE, PERIODIC_REF, KDTree
from nbodylib_gb300 import synthetic as syn
from tests.helpers import (assert_density_close, assert_knn_equal, brute_min_image_knn, rows_by_id,
                           to_ids)

pytestmark = pytest.mark.gpu


def inputs(kind, n, seed=11):
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        pos = rng.random((n, 3))
    elif kind == "clustered":  # dense spheres on a sparse background: mixed groups
        pos, _ = syn.clustered_box(n, 1.0, seed=seed, nspheres=7)
    elif kind == "plane":  # no volume: the radius comes from the area
        pos = rng.random((n, 3))
        pos[:, 2] = 0.25
    elif kind == "pairs":  # every particle twice: zero distances
        pos = np.repeat(rng.random(((n + 1) // 2, 3)), 2, axis=0)[:n]
    elif kind == "offset":  # coordinates large against the distances
        pos = 1.0e6 + rng.random((n, 3))
    mass = rng.random(n) + 0.5
    vel = rng.normal(size=(n, 3))
    return pos, mass, vel


CASES = [  # kind, n, bucket, k
    ("uniform", 8, 16, 1), ("uniform", 131, 16, 31), ("uniform", 132, 16, 32),
    ("uniform", 133, 16, 33), ("clustered", 4097, 16, 32), ("clustered", 20011, 16, 32),
    ("clustered", 5003, 1, 7), ("clustered", 5003, 40, 64), ("clustered", 3001, 1000, 40),
    ("clustered", 4099, 16, 65), ("clustered", 4099, 8, 127), ("plane", 3003, 16, 32),
    ("pairs", 2049, 16, 16), ("offset", 6007, 16, 32),
]


@pytest.mark.parametrize("kind,n,b,k", CASES)
def test_every_particle(gpu, port_built, kind, n, b, k):
    pos, mass, vel = inputs(kind, n)
    o = oracle.OracleTree(pos, vel, mass, b, 0, 0, 1000, None, backend="port", nthreads=8)
    t = KDTree(pos, vel, mass, b, kerntype=0)
    perm = t.GetPerm()
    nn, d2 = t.FindNearest(k)
    assert np.all(np.diff(d2, axis=1) >= 0)
    oi, od = o.knn(k, 0)
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), oi, od, kind)
    if k == 1:
        return  # h = 0: no density is defined
    assert_density_close(t.CalcDensity(k), o.density(k), f"density {kind}")
    if kind == "pairs":
        return  # two candidates tie at the k-th place: which one's velocity counts is open
    ns = max(2, k // 2)
    assert_density_close(t.CalcVelDensity(ns, k), o.veldensity(ns, k), f"veldensity {kind}")


# from this many particles on every particle's search goes by groups
LARGE = [("clustered", 32767, 16, 32), ("clustered", 32768, 5, 32), ("uniform", 32771, 1000, 40),
         ("clustered", 40009, 16, 65), ("clustered", 32769, 8, 127), ("plane", 32771, 16, 32),
         ("pairs", 32769, 16, 16), ("offset", 40009, 16, 64)]


@pytest.mark.parametrize("kind,n,b,k", LARGE)
def test_every_particle_large(gpu, port_built, kind, n, b, k):
    test_every_particle(gpu, port_built, kind, n, b, k)


@pytest.mark.parametrize("method,per,k", [(0, [1.0, 1.0, 1.0], 31), (1, [1.0, 1.0, 1.0], 64),
                                          (0, [1.0, 0.25, 2.0], 32)])
def test_periodic_rows_large(gpu, port_built, method, per, k):
    n = 32771
    pos = np.random.default_rng(17).random((n, 3)) * per
    o = oracle.OracleTree(pos, None, np.ones(n), 16, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, None, np.ones(n), 16, kerntype=0, period=per)
    nn, d2 = (t.FindNearest if method == 0 else t.FindNearestPos)(k)
    perm = t.GetPerm()
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), *o.knn(k, method),
                     f"method {method}, period {per}")


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("n,b,k", [(500, 600, 32), (4097, 16, 31), (4097, 16, 32), (9001, 16, 64)])
def test_periodic_rows(gpu, port_built, method, n, b, k):
    """Queries near a wall (image passes), a single leaf (searched without images), and the
    entry that each method leaves out."""
    pos, mass, _ = inputs("uniform", n)
    per = [1.0, 1.0, 1.0]
    o = oracle.OracleTree(pos, None, mass, b, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, None, mass, b, kerntype=0, period=per)
    perm = t.GetPerm()
    nn, d2 = (t.FindNearest if method == 0 else t.FindNearestPos)(k)
    oi, od = o.knn(k, method)
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), oi, od,
                     f"method {method}")


@pytest.mark.parametrize("mode", [PERIODIC_REF, PERIODIC_MIN_IMAGE])
@pytest.mark.parametrize("per", [[1.0, 1.0, 1.0], [1.0, 0.25, 2.0], [1.0, 1.0, 0.01]])
def test_periodic_images(gpu, port_built, mode, per):
    """Short sides (a particle's own images among its neighbours, lists across several walls)
    in both image modes: the squared distances of the reference's search, or of brute force."""
    n, k = 4097, 32
    rng = np.random.default_rng(17)
    pos = rng.random((n, 3)) * per
    o = oracle.OracleTree(pos, None, np.ones(n), 16, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, None, np.ones(n), 16, kerntype=0, period=per)
    nn, d2 = t.FindNearest(k, periodic_mode=mode)
    perm = t.GetPerm()
    got = rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm)
    if mode == PERIODIC_REF:
        assert_knn_equal(*got, *o.knn(k, 0), f"images, period {per}")
    elif min(per) > 0.1:  # every neighbour once: below half the shortest side
        assert_knn_equal(*got, *brute_min_image_knn(pos, per, k), f"minimum image, period {per}")


@pytest.mark.parametrize("n,b,k", [(40, 16, 8), (3001, 1000, 32), (5003, 16, 33), (5003, 1, 64),
                                   (5003, 16, 65), (4099, 16, 127)])
def test_points(gpu, port_built, n, b, k):
    """Points anywhere: on particles (zero distances count), beside them, outside the box."""
    pos, mass, _ = inputs("clustered", n)
    rng = np.random.default_rng(5)
    x = np.concatenate([pos[:101], pos[::-1][:100] + rng.normal(size=(min(n, 100), 3)) * 1e-3,
                        rng.random((99, 3)) * 3.0 - 1.0])
    for per in (None, [1.0, 1.0, 1.0]):
        o = oracle.OracleTree(pos, None, mass, b, 0, 0, 1000, per, backend="port", nthreads=8)
        t = KDTree(pos, None, mass, b, kerntype=0, period=per)
        nn, d2 = t.FindNearestPosPoints(x, k)
        assert np.all(np.diff(d2, axis=1) >= 0)
        oi, od = o.knn_pos(x, k)
        assert_knn_equal(to_ids(nn, t.GetPerm()), d2, oi, od, f"points, period {per}")
