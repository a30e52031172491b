"""Neighbour searches of every particle in boxes where the neighbours lie near or beyond the
distance at which the reference's lists start (squared: 1e32), at the sizes of the group search
and below it: the same rows, and densities refused where a list stays short."""
import numpy as np
import pytest

import oracle
from nbodylib_gb300 import BatchedDensity, KDTree
from nbodylib_gb300._capi import NbkError
from tests.helpers import assert_density_close, assert_knn_equal, rows_by_id, to_ids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3001, 40009])
@pytest.mark.parametrize("box,periodic", [(1e15, False), (1e17, True), (4e17, False),
                                          (4e17, True)])
def test_rows_and_densities(gpu, port_built, n, box, periodic):
    k = 32
    pos = np.random.default_rng(21).random((n, 3)) * box
    per = [box] * 3 if periodic else None
    o = oracle.OracleTree(pos, None, np.ones(n), 16, 0, 0, 1000, per, backend="port", nthreads=8)
    t = KDTree(pos, None, np.ones(n), 16, kerntype=0, period=per)
    nn, d2 = t.FindNearest(k)
    perm = t.GetPerm()
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), *o.knn(k, 0))
    off = np.array([0, n], np.int64)
    batch = BatchedDensity(pos, np.ones(n), off, bucket_size=16)
    try:
        want = o.density(k)  # searched without images: short lists near the walls too
    except RuntimeError:
        with pytest.raises(NbkError):
            t.CalcDensity(k)
        with pytest.raises(NbkError):
            batch.density(k, use_graph=False)
    else:
        assert_density_close(t.CalcDensity(k), want)
        assert_density_close(np.asarray(batch.density(k, use_graph=False)), want)
    batch.close()
    t.close()


@pytest.mark.parametrize("box", [1e-6, 1e-12, 1e-15, 1e-20])
def test_small_boxes(gpu, port_built, box):
    """Distances whose squares fall below FP32's range, one tree and a batch."""
    n, k = 40009, 16
    pos = np.random.default_rng(22).random((n, 3)) * box
    o = oracle.OracleTree(pos, None, np.ones(n), 16, 0, 0, 1000, None, backend="port", nthreads=8)
    t = KDTree(pos, None, np.ones(n), 16, kerntype=0)
    nn, d2 = t.FindNearest(k)
    perm = t.GetPerm()
    assert_knn_equal(rows_by_id(to_ids(nn, perm), perm), rows_by_id(d2, perm), *o.knn(k, 0))
    want = o.density(k)
    assert_density_close(t.CalcDensity(k), want)
    t.close()
    batch = BatchedDensity(pos, np.ones(n), np.array([0, n], np.int64), bucket_size=16)
    assert_density_close(np.asarray(batch.density(k, use_graph=False)), want)
    batch.close()
