"""Searches at many points with a small k, where points near one another share a warp: in tree
order, along sightlines, in no order, on flat nodes, with a ragged number of them; rows against
the restatement bit-exact, sums to the path's 1e-12."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from tests.helpers import assert_density_close, assert_knn_equal, to_ids

pytestmark = pytest.mark.gpu

MANY, MORE = (1 << 17) + 11, (1 << 19) + 5  # from which on warps are shared


def points(order, pos, box, nq, rng):
    if order == "tree":
        return np.repeat(pos, nq // len(pos) + 1, axis=0)[:nq] + rng.normal(size=(nq, 3)) * 1e-3
    if order == "lines":
        a, b = rng.random((nq // 1024 + 1, 1, 3)) * box, rng.normal(size=(nq // 1024 + 1, 1, 3))
        return (a + b * np.linspace(0, box, 1024)[None, :, None]).reshape(-1, 3)[:nq]
    return rng.random((nq, 3)) * box


@pytest.mark.parametrize("order", ["tree", "lines", "none"])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nq,k,flat", [(MANY, 1, False), (MANY, 8, False), (MANY, 12, True),
                                       (MORE, 8, False), (MORE, 16, False)])
def test_rows_and_sums(gpu, port_built, order, periodic, nq, k, flat):
    n, rng = 4099, np.random.default_rng(k)
    box = 10.0
    pos, mass, vel = syn.clustered_box(n, box, seed=9, nspheres=6, velocities=True)
    if flat:
        pos[:, 1] = 4.0
    per = [box] * 3 if periodic else None
    o = oracle.OracleTree(pos, vel, mass, 16, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, vel, mass, 16, kerntype=0, period=per)
    perm = t.GetPerm()
    x = points(order, pos[perm], box, nq, rng)
    nn, d2 = t.FindNearestPosPoints(x, k)
    assert_knn_equal(to_ids(nn, perm), d2, *o.knn_pos(x, k), f"{order}, period {per}")
    # the sums of some of the points alone take a warp each (k = 1: h = 0, no sum is defined)
    some = np.sort(rng.choice(nq, 3000, replace=False))
    if k > 1:
        v = rng.normal(size=(nq, 3))
        assert_density_close(t.CalcDensityPosition(x, k)[some], t.CalcDensityPosition(x[some], k))
        ns = max(2, k // 2)
        assert_density_close(t.CalcVelDensityPosition(x, v, ns, k)[some],
                             t.CalcVelDensityPosition(x[some], v[some], ns, k))
        rho = np.asarray(t.CalcDensity(k))
        one, all_ = t.CalcSmoothVelPosition(x[some], k, rho), t.CalcSmoothVelPosition(x, k, rho)
        assert np.abs(all_[some] - one).max() <= 1e-12 * np.abs(one).max()
    t.close()


def test_too_few_neighbours(gpu):
    """Sums at points of a tree with fewer than k particles are refused, rows end with none."""
    from nbodylib_gb300._capi import NbkError
    rng = np.random.default_rng(2)
    t = KDTree(rng.random((9, 3)), None, np.ones(9), 16, kerntype=0)
    x = rng.random((MANY, 3)) * 1e-3
    nn, d2 = t.FindNearestPosPoints(x, 12)
    assert (nn[:, 9:] == -1).all() and (nn[:, :9] >= 0).all() and (d2[:, 9:] == 1e32).all()
    with pytest.raises(NbkError):
        t.CalcDensityPosition(x, 12)
    t.close()
