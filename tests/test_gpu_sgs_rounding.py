"""The Eisenstat sweeps take a row's right-hand side after its sum, in the tile sweeps as in the sync-free ones: on systems
whose sums are exact in any order, one SGS-MRTR iteration gives the same bits through both. Four entries of 2^-54 (2^-53)
beside a right-hand side of 1 are lost one by one where a row starts from it."""
import numpy as np
import pytest

from sparsesolv_gb300 import _capi

pytestmark = pytest.mark.gpu


def backward():
    """u = U^-1 rd: row 0 reads rows 1 to 4."""
    A = np.eye(5)
    A[0, 1:] = A[1:, 0] = -2.0 ** -54
    return A, np.ones(5)


def eisenstat():
    """C^-1 (rd - u): row 4 reads rows 0 to 3, whose values are 2^-26, and rd - u is -1 there through row 5."""
    A = np.eye(6)
    A[4, :4] = A[:4, 4] = -2.0 ** -27
    A[4, 5] = A[5, 4] = -1.0
    b = np.zeros(6)
    b[4] = 1.0
    return A, b


@pytest.mark.parametrize("system", [backward, eisenstat])
def test_one_iteration_has_the_sync_free_sweeps_bits(gpu, system):
    A, b = system()
    n = len(b)
    rows, cols = np.nonzero(A)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    out = []
    for mode in (0, 1):
        h = _capi.Handle(0)
        try:
            h.set_tuning(_capi.TUNE_SWEEP_MODE, mode)
            h.set_tuning(_capi.TUNE_SWEEP_GROUP, 4)
            o = h.default_options()
            o.precondition_type = 1
            o.is_save_residual_log = 1
            h.set_options(o)
            h.set_matrix(rp, cols.astype(np.int32), A[rows, cols])
            x = np.zeros(n)
            h.solve(_capi.METHOD_MRTR, b, x, conv=1e-300, max_ite=1)
            out.append((x, h.residual_log()))
        finally:
            h.close()
    assert np.any(out[0][0] != 0.0)
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
