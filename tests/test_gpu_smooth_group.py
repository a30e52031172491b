"""The smoothing family over rows of the group search (70,001 particles), its row lengths at the
slot switches, against the restatement: 1e-12 of the largest magnitude, as the path's."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from nbodylib_gb300.kdtree import KSPH

pytestmark = pytest.mark.gpu


def close(got, want, what):
    got, want = np.asarray(got).reshape(len(got), -1), np.asarray(want).reshape(len(got), -1)
    worst = np.abs(got - want).max() / np.abs(want).max()
    assert worst <= 1e-12, f"{what}: {worst:.3e}"


@pytest.mark.parametrize("k", [16, 32, 33, 65])
def test_every_particle(gpu, port_built, k):
    pos, mass, vel = syn.clustered_box(70001, 80.0, seed=31 + k, velocities=True)
    # ten particles too close for FP32: the group search leaves them to its list (no two at one
    # place: which of them is the k-th then is open, and the kurtosis subtracts 3 in each term)
    pos[1000:1010] = pos[1000] + np.random.default_rng(k).normal(size=(10, 3)) * 1e-9
    o = oracle.OracleTree(pos, vel, mass, 16, 0, 0, 1000, None, backend="port", nthreads=8)
    t = KDTree(pos, vel, mass, 16, kerntype=KSPH)
    rho = o.density(k)
    mean = o.smooth_vel_moments(0, k, rho)
    disp = o.smooth_vel_moments(1, k, rho, mean).reshape(-1, 9)
    close(t.CalcSmoothVel(k, rho=rho), mean, "CalcSmoothVel")
    close(t.CalcSmoothVelDisp(mean, k, rho=rho), disp, "CalcSmoothVelDisp")
    close(t.CalcSmoothVelSkew(mean, disp, k, rho=rho),
          o.smooth_vel_moments(2, k, rho, mean, disp), "CalcSmoothVelSkew")
    close(t.CalcSmoothVelKurtosis(mean, disp, k, rho=rho),
          o.smooth_vel_moments(3, k, rho, mean, disp), "CalcSmoothVelKurtosis")
    # the same query's value by the search of given targets, a warp each
    every = t.CalcVelDensityWithPhysDensity(k, k, rho=rho)
    targets = np.arange(0, 70001, 7, dtype=np.int32)
    one = t.CalcVelDensityWithPhysDensityParticle(targets, k, k, rho=rho)
    np.testing.assert_allclose(np.asarray(every)[t.GetPerm()[targets]], one, rtol=1e-12)
    t.close()
