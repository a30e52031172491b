"""Kernel tables of more cells than 2^20 and 2^21: the cell of every neighbour and with it the
densities and smoothed fields, by the group search (70,001 particles) and the search below it."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from tests.helpers import assert_density_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2001, 70001])
@pytest.mark.parametrize("kernres", [(1 << 20) + 7, 3 << 20, (1 << 22) + 5])
def test_large_tables(gpu, port_built, n, kernres):
    k = 16
    pos, mass, vel = syn.clustered_box(n, 1.0, seed=5, nspheres=7, velocities=True)
    o = oracle.OracleTree(pos, vel, mass, 16, 0, 0, kernres, None, backend="port", nthreads=8)
    t = KDTree(pos, vel, mass, 16, kerntype=0, kernres=kernres)
    rho = o.density(k)
    assert_density_close(t.CalcDensity(k), rho, "density")
    assert_density_close(t.CalcVelDensity(k, k), o.veldensity(k, k), "velocity density")
    # the fields of equal velocities: sums of the same weights, every component the same
    one = KDTree(pos, np.ones((n, 3)), mass, 16, kerntype=0, kernres=kernres)
    coarse = KDTree(pos, np.ones((n, 3)), mass, 16, kerntype=0, kernres=(1 << 20) - 1)
    mean, want = one.CalcSmoothVel(k, rho), coarse.CalcSmoothVel(k, rho)
    # the two tables' interpolations differ by their cells squared: 2^-40 of W and its curvature
    np.testing.assert_allclose(mean, want, rtol=1e-9)
