"""Links and balls at scales whose squares leave FP32's range (positions in centimetres or
metres, or very small ones), where FP64 has to decide: the same answers as the restatement's
or brute force, and the same as at scale one."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from nbodylib_gb300.kdtree import FOF3D, FOF6D
from tests.helpers import assert_same_partition, d2_ref, reflect_images

pytestmark = pytest.mark.gpu

SCALES = [1.0, 1e22, 1e18, 3e-16, 1e-20, 1e-22]


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("periodic", [False, True])
def test_fof(gpu, port_built, scale, periodic):
    n, box = 3001, 20.0 * scale
    pos, mass = syn.clustered_box(n, 20.0, seed=3, nspheres=20)
    pos = pos * scale
    per = [box] * 3 if periodic else None
    ll = syn.linking_length(n, box)
    o = oracle.OracleTree(pos, None, mass, 16, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, None, mass, 16, kerntype=0, period=per)
    for got, want in ((t.FOF(ll, 5), o.fof(ll, 5)),
                      (t.FOFCriterion(FOF3D, [0, ll * ll, 0, 0, 0, 0, ll * ll, 0], 5),
                       o.fof_criterion(0, [0, ll * ll, 0, 0, 0, 0, ll * ll, 0], 5))):
        assert got[1] == want[1] > 0
        assert_same_partition(got[0], want[0], f"scale {scale}")


@pytest.mark.parametrize("length,speed", [(1.0, 1.0), (1e22, 1.0), (1e22, 1e7), (1.0, 1e22),
                                          (1e-20, 1.0), (1.0, 1e-20), (1e-20, 1e20)])
@pytest.mark.parametrize("periodic", [False, True])
def test_fof6d(gpu, port_built, length, speed, periodic):
    n = 2001
    pos, mass, vel = syn.clustered_box(n, 20.0, seed=3, nspheres=20, velocities=True)
    pos, vel, box = pos * length, vel * speed, 20.0 * length
    per = [box] * 3 if periodic else None
    ll = syn.linking_length(n, box)
    p = [0, ll * ll, 0, 0, 0, 0, ll * ll, 0.04 * speed * speed]
    o = oracle.OracleTree(pos, vel, mass, 16, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, vel, mass, 16, kerntype=0, period=per)
    g, ng = t.FOFCriterion(FOF6D, p, 5)
    go, ngo = o.fof_criterion(2, p, 5)
    assert ng == ngo > 0
    assert_same_partition(g, go, f"length {length}, speed {speed}")


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("periodic", [False, True])
def test_ball(gpu, scale, periodic):
    """Rows of a few targets, and of all of them in random order (balls all over the box)."""
    n = 5003
    pos, mass = syn.clustered_box(n, 1.0, seed=9, nspheres=6)
    pos = pos * scale
    per = [scale] * 3 if periodic else None
    t = KDTree(pos, None, mass, 16, kerntype=0, period=per)
    tree = pos[t.GetPerm()]
    order = np.random.default_rng(1).permutation(n).astype(np.int32)
    for r in (0.01 * scale, 0.06 * scale):
        off, idx = t.SearchBallPosTagged(order, r * r)
        few, fidx = t.SearchBallPosTagged(order[:3], r * r)
        assert np.array_equal(few, off[:4]) and np.array_equal(fidx, idx[:few[3]])
        for i in range(0, n, 7):
            x = tree[order[i]]
            want = []
            for p, y in enumerate(reflect_images(x[None], per)[:, 0] if periodic else x[None]):
                if p:  # an image is searched when its wall distance is inside the radius
                    s = np.where(x < 0.5 * scale, x, scale - x)[y != x]
                    if not (r * r > (np.abs(s[0]) if s.size == 1 else np.sqrt((s * s).sum())) ** 2):
                        continue
                hit = np.nonzero(d2_ref(y, tree) < r * r)[0]
                want += [j for j in hit if periodic or j != order[i]]
            assert idx[off[i]:off[i + 1]].tolist() == want, (r, i)
