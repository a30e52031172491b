"""Phase-space searches whose metric takes squares to the ends of FP32's range."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300.kdtree import KSPH, TPHS
from tests.helpers import assert_knn_equal, rows_by_id, to_ids

pytestmark = pytest.mark.gpu


def assert_rows_equal(pos, vel, b, k, aniso, rows=slice(None)):
    n = len(pos)
    o = oracle.OracleTree(pos, vel, np.ones(n), b, TPHS, 0, 1000, None, backend="port",
                          nthreads=8, aniso=aniso)
    t = KDTree(pos, vel, np.ones(n), b, treetype=TPHS, kerntype=KSPH, aniso=aniso)
    perm = t.GetPerm()
    nn, d2 = t.FindNearest(k)
    t.close()
    oi, od = o.knn(k, 0)
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm)[rows], rows_by_id(d2, perm)[rows],
                     oi[rows], od[rows])
    return d2


@pytest.mark.parametrize("k", [8, 32, 40])
def test_squares_near_the_largest_float(gpu, port_built, k):
    """Two particles 2e-15 apart in one coordinate weigh it with 2.5e29: the others, at
    2.8e4 to 3.6e4 in it, are at squared distances of 2e38 to 3.3e38 from them."""
    rng = np.random.default_rng(7)
    pos, vel = rng.random((2001, 3)) * 10.0, rng.random((2001, 3)) * 10.0
    pos[:, 0] = rng.uniform(2.8e4, 3.6e4, 2001)
    pos[0, 0], pos[1, 0] = 0.0, 2e-15
    pos[1, 1:], vel[1] = pos[0, 1:] + 0.1, vel[0] + 0.1
    d2 = assert_rows_equal(pos, vel, 16, k, 0)
    assert (d2 == 1e32).sum() >= 2 * (k - 1)  # farther than the searches go


@pytest.mark.parametrize("box", [1e15, 2.5e17])
def test_particles_farther_than_the_search_goes(gpu, port_built, box):
    """Lists start at squared distances of 1e32 and take nothing there or beyond."""
    rng = np.random.default_rng(9)
    d2 = assert_rows_equal(rng.random((3001, 3)) * box, rng.random((3001, 3)), 16, 32, -1)
    assert (d2 == 1e32).any() == (box > 1e17)


@pytest.mark.parametrize("n", [2001, 9001])
def test_queries_without_a_resolved_spacing(gpu, port_built, n):
    """Twelve particles within 1e-16 of one another, whose plain distances FP32 does not
    resolve, take the search of a lane each. (A particle whose nearest they are has a metric
    only if their distances to it do not tie exactly: which one it is taken from is open.)"""
    rng = np.random.default_rng(11)
    pos, vel = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    pos[:12], vel[:12] = rng.normal(size=(12, 3)) * 1e-16, rng.normal(size=(12, 3)) * 1e-16
    x = np.concatenate([pos, vel], axis=1)
    near = [np.partition(((x - y) ** 2).cumsum(axis=1)[:, 5], (1, 2))[1:3] for y in x]
    rows = np.array([a != b for a, b in near])
    assert rows[:12].all() and rows.sum() > n - 5
    for k in (8, 16):
        assert_rows_equal(pos, vel, 16, k, 0, rows)


def test_more_leftovers_than_their_list_holds(gpu, port_built):
    """Two of three particles beside one another at 1e-7 in one coordinate: FP32 resolves none
    of their metrics, and the list of those (an eighth of the particles) is full."""
    n = 12001
    rng = np.random.default_rng(13)
    pos, vel = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    i = np.arange(0, n - 1, 3)
    pos[i + 1] = pos[i] + rng.normal(size=(i.size, 3)) * 0.01
    pos[i + 1, 0] = pos[i, 0] + 1e-7
    vel[i + 1] = vel[i] + rng.normal(size=(i.size, 3)) * 0.01
    assert_rows_equal(pos, vel, 16, 16, 0)
