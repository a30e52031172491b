"""FOF and FOF6d at the sizes where the link kernels' queries per warp change, and at leaf sizes
where a leaf fills part of a half warp, a half warp and several: partitions and group counts
identical to the restatement's."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import KDTree
from nbodylib_gb300 import synthetic as syn
from nbodylib_gb300.kdtree import FOF6D
from tests.helpers import assert_same_partition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,b", [(2, 16), (33, 5), (1000, 40), (4863, 16), (9729, 16),
                                 (19457, 17), (40009, 3), (80021, 16)])
@pytest.mark.parametrize("periodic", [False, True])
def test_fof_and_fof6d(gpu, port_built, n, b, periodic):
    box = 20.0
    pos, mass, vel = syn.clustered_box(n, box, seed=n, nspheres=20, velocities=True)
    per = [box] * 3 if periodic else None
    ll = syn.linking_length(n, box)
    o = oracle.OracleTree(pos, vel, mass, b, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, vel, mass, b, kerntype=0, period=per)
    g, ng = t.FOF(ll, 5)
    go, ngo = o.fof(ll, 5)
    assert ng == ngo
    assert_same_partition(g, go, "FOF")
    if n > 20000:
        return  # the restatement's criterion search is slow there
    p = [0, ll * ll, 0, 0, 0, 0, ll * ll, 0.04]
    g, ng = t.FOFCriterion(FOF6D, p, 5)
    go, ngo = o.fof_criterion(2, p, 5)
    assert ng == ngo
    assert_same_partition(g, go, "FOF6d")
