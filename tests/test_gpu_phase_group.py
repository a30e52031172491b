"""The phase-space group search (every particle of a TPHS tree) and the launches behind it, at
the sizes and inputs where its parts hand over: buffers of 32, 64 and 128 neighbours, leaves
of one and of many, weights from offsets of 1e-7 (FP32 cannot resolve them), offsets of zero,
weights below one. Rows bit-exact against the restatement, densities to the path's 1e-12."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from nbodylib_gb300.kdtree import KSPH, TPHS
from tests.helpers import assert_density_close, assert_knn_equal, rows_by_id, to_ids

pytestmark = pytest.mark.gpu


def inputs(kind, n, seed=23):
    rng = np.random.default_rng(seed)
    pos, mass, vel = syn.clustered_box(n, 10.0, seed=seed, nspheres=9, velocities=True)
    if kind == "near":  # every third particle beside another one in one coordinate
        i = np.arange(0, n - 1, 3)
        pos[i + 1] = pos[i] + rng.normal(size=(i.size, 3)) * 0.01
        pos[i + 1, 0] = pos[i, 0] + 1e-7
        vel[i + 1] = vel[i] + rng.normal(size=(i.size, 3)) * 0.01
    elif kind == "grid":  # velocities on a lattice: offsets of exactly zero
        vel = np.round(vel * 32.0) / 32.0
    elif kind == "wide":  # offsets above one: weights below one, the reference's pruning shows
        pos = pos * 30.0
    return pos, vel, mass


@pytest.mark.parametrize("kind,n,b,k,aniso", [
    ("box", 36, 16, 8, 0), ("box", 2049, 16, 7, 0), ("box", 4099, 16, 32, -1),
    ("box", 4099, 16, 33, 0), ("box", 3001, 1, 32, 0), ("box", 3001, 300, 40, 0),
    ("box", 3001, 16, 65, 0), ("box", 3001, 8, 127, -1), ("near", 4099, 16, 32, 0),
    ("grid", 3001, 16, 16, 0), ("wide", 4099, 16, 32, 0),
])
def test_every_particle(gpu, port_built, kind, n, b, k, aniso):
    pos, vel, mass = inputs(kind, n)
    o = oracle.OracleTree(pos, vel, mass, b, TPHS, 0, 1000, None, backend="port", nthreads=8,
                          aniso=aniso)
    t = KDTree(pos, vel, mass, b, treetype=TPHS, kerntype=KSPH, aniso=aniso)
    perm = t.GetPerm()
    nn, d2 = t.FindNearest(k)
    oi, od = o.knn(k, 0)
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), oi, od, kind)
    if aniso == 0:
        assert_density_close(t.CalcDensity(k), o.density(k), kind)
