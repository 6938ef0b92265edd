"""Lanes a row asked for act in the automatic mode too, where its sync-free sweep serves narrow levels of real rows: the
same bits as the sync-free mode with those lanes."""
import numpy as np
import pytest
import scipy.sparse as sp

from sparsesolv_gb300 import _capi, voxel

pytestmark = pytest.mark.gpu


def scattered(N=16):
    """A curl-curl system in random order, which the tile sweeps do not take, made regular."""
    rp, ci, va, _ = voxel.curl_curl_case(N, 3).assemble()
    A = sp.csr_matrix((va, ci, rp))
    A = sp.csr_matrix(A + 1e-3 * sp.diags(A.diagonal()))
    q = np.random.default_rng(0).permutation(A.shape[0])
    A = sp.csr_matrix(A[q][:, q])
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


@pytest.mark.parametrize("key", [_capi.TUNE_CLUSTER_GROUP, _capi.TUNE_SWEEP_GROUP])
@pytest.mark.parametrize("reciprocal", [1, 0])
def test_handle(gpu, key, reciprocal):
    rp, ci, va = scattered()
    r = np.random.default_rng(1).standard_normal(len(rp) - 1)
    seen = []
    for lanes in (4, 8, 16):
        h, f = _capi.Handle(0), _capi.Handle(0)
        try:
            h.set_tuning(key, lanes)
            f.set_tuning(_capi.TUNE_SWEEP_MODE, 1)
            f.set_tuning(_capi.TUNE_SWEEP_GROUP, lanes)
            z = []
            for hh in (h, f):
                hh.set_tuning(_capi.TUNE_RECIPROCAL_DIAG, reciprocal)
                hh.set_matrix(rp, ci, va)
                hh.factor(1.1)
                z.append(hh.apply_precond(r))
            assert np.array_equal(z[0], z[1])
            seen.append(z[0])
        finally:
            h.close()
            f.close()
    assert not np.array_equal(seen[0], seen[1]) and not np.array_equal(seen[1], seen[2])


@pytest.mark.parametrize("lanes", [4, 16])
def test_internal_batch(gpu, lanes):
    rp, ci, va = scattered()
    n = len(rp) - 1
    B = np.random.default_rng(2).standard_normal((2, n))
    X = []
    for mode in (0, 1):
        h = _capi.Handle(0)
        try:
            h.set_matrix(rp, ci, va)
            o = h.default_options()
            o.accel_factor = 1.1
            o.precondition_type = 0  # IC: SGS solves do not go through the internal batch
            h.set_options(o)
            h.set_tuning(_capi.TUNE_SWEEP_MODE, mode)
            h.set_tuning(_capi.TUNE_BATCH_GROUP, lanes)
            x = np.zeros_like(B)
            assert h.solve_multi(_capi.METHOD_MRTR, B, x, conv=1e-8, max_ite=500)[0]
            X.append(x)
        finally:
            h.close()
    assert np.array_equal(X[0], X[1])
