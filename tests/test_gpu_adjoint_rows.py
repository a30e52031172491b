"""The density adjoint where the forward leaves particles without a neighbour row."""
import numpy as np
import pytest

from nbodylib_gb300 import KDTree
from nbodylib_gb300._capi import NbkError

pytestmark = pytest.mark.gpu

NBK_ERR_TOO_FEW = 5


@pytest.mark.parametrize("n,same,k", [(40, 10, 32), (300, 260, 64)])
def test_too_few_neighbours(gpu, n, same, k):
    """Coincident particles have fewer than k neighbours at a non-zero distance: the call is
    refused (its backward has no rows to read for them), and the next one is served."""
    rng = np.random.default_rng(8)
    pos, w = rng.random((n, 3)), rng.normal(size=n)
    few = pos.copy()
    few[:same] = few[0]
    t = KDTree(few, None, np.ones(n), 16, kerntype=0)
    with pytest.raises(NbkError) as e:
        t.DensityAdjoint(k, w)
    assert e.value.status == NBK_ERR_TOO_FEW
    t.close()
    t = KDTree(pos, None, np.ones(n), 16, kerntype=0)
    rho, gp, gm = t.DensityAdjoint(8, w)
    t.close()
    assert (rho > 0).all() and np.isfinite(gp).all() and np.isfinite(gm).all()
