"""SearchBallPosTagged rows: the particles of each ball, in tree order image by image, at the
leaf sizes where a leaf fills part of a half warp, a half warp and more than a warp, for few
queries and many, radii from empty balls to the whole box."""
import numpy as np
import pytest

from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from tests.helpers import d2_ref, reflect_images

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 5003, 40001])
@pytest.mark.parametrize("periodic", [False, True])
def test_order_of_targets(gpu, n, periodic):
    """A target's row does not depend on the targets beside it: a few in random order (balls all
    over the box), all of them in tree order."""
    pos, mass = syn.clustered_box(n, 1.0, seed=4, nspheres=6)
    t = KDTree(pos, None, mass, 16, kerntype=0, period=[1.0, 1.0, 1.0] if periodic else None)
    some = np.random.default_rng(1).permutation(n)[:3000].astype(np.int32)
    for r in (1e-3, 0.02):
        off, idx = t.SearchBallPosTagged(np.arange(n, dtype=np.int32), r * r)
        off2, idx2 = t.SearchBallPosTagged(some, r * r)
        for i, j in enumerate(some):
            assert np.array_equal(idx2[off2[i]:off2[i + 1]], idx[off[j]:off[j + 1]]), (r, j)


@pytest.mark.parametrize("n,b,nq", [(40, 16, 1), (2049, 16, 3), (3001, 5, 700), (3001, 17, 33),
                                    (3001, 100, 64), (5003, 16, 5003)])
@pytest.mark.parametrize("periodic", [False, True])
def test_rows(gpu, n, b, nq, periodic):
    pos, mass = syn.clustered_box(n, 1.0, seed=9, nspheres=6)
    per = [1.0, 1.0, 1.0] if periodic else None
    t = KDTree(pos, None, mass, b, kerntype=0, period=per)
    perm = t.GetPerm()
    tree = pos[perm]
    targets = np.arange(0, n, max(1, n // nq))[:nq].astype(np.int32)
    for r in (1e-6, 0.01, 0.06, 2.0):
        if r == 2.0 and nq > 100:
            continue
        off, idx = t.SearchBallPosTagged(targets, r * r)
        off2, idx2 = t.SearchBallPosTagged(targets, r * r)  # output sized by the first call
        assert np.array_equal(off, off2) and np.array_equal(idx, idx2)
        q = tree[targets]
        imgs = reflect_images(q, [1.0] * 3) if periodic else q[None]
        for i in range(len(targets)):
            want = []
            for p in range(imgs.shape[0]):
                if p:  # an image is searched when its wall distance is inside the radius
                    moved = imgs[p, i] != q[i]
                    s = np.where(q[i] < 0.5, q[i], 1.0 - q[i])[moved]
                    if not (r * r > (np.abs(s[0]) if s.size == 1 else np.sqrt((s * s).sum())) ** 2):
                        continue
                hit = np.nonzero(d2_ref(imgs[p, i], tree) < r * r)[0]
                # the target itself is left out by the search without images only
                want += [j for j in hit if periodic or j != targets[i]]
            got = idx[off[i]:off[i + 1]].tolist()
            assert got == want, (r, i)
