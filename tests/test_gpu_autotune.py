"""ssg_autotune with the sums kept: results of an untuned run, bit for bit, with either preconditioner, and no schedule that
is slower than the one the handle would have run."""
import numpy as np
import pytest

from sparsesolv_gb300 import _capi, voxel

pytestmark = pytest.mark.gpu


def solves(h, b):
    out = []
    o = h.default_options()
    o.accel_factor = 1.1
    o.is_save_residual_log = 1
    for pre in (0, 1):
        o.precondition_type = pre
        h.set_options(o)
        x = np.zeros_like(b)
        h.solve(_capi.METHOD_MRTR, b, x, conv=1e-6, max_ite=40)
        out += [x, h.residual_log()]
    return out


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("tuning,modes", [
    ({}, (0,)),                                                                      # the automatic mode
    ({_capi.TUNE_CLUSTER_GROUP: 8}, (0,)),
    ({_capi.TUNE_RECIPROCAL_DIAG: 0}, (0, 1, 2, 3)),                                 # no tile sweep
    ({_capi.TUNE_SWEEP_MODE: 1, _capi.TUNE_SWEEP_GROUP: 8}, (0, 1, 2, 3)),
    ({_capi.TUNE_SWEEP_MODE: 2}, (0, 1, 2, 3)),
    ({_capi.TUNE_SWEEP_MODE: 4}, (4,)),
])
def test_kept_sums_keep_the_bits(gpu, cplx, tuning, modes):
    h = _capi.Handle(0)
    try:
        b = h.set_matrix_voxel(voxel.eddy_current_case(14, 4) if cplx else voxel.curl_curl_case(14, 4))
        for k, v in tuning.items():
            h.set_tuning(k, v)
        ref = solves(h, b)
        c = h.autotune(keep_group=True)
        assert c["mode"] in modes and c["ms"] > 0
        got = solves(h, b)
        for r, g in zip(ref, got):
            assert np.array_equal(r, g)
    finally:
        h.close()


def test_a_real_handle_tuned_by_push_takes_a_complex_matrix(gpu):
    """Whatever a real handle's tuning chose, a complex matrix on it solves as on a fresh one with those lanes."""
    h, f = _capi.Handle(0), _capi.Handle(0)
    try:
        h.set_matrix_voxel(voxel.curl_curl_case(8, 4))
        h.autotune()
        h.set_tuning(_capi.TUNE_SWEEP_MODE, 4)
        h.autotune(keep_group=True)
        for hh in (h, f):
            hh.set_tuning(_capi.TUNE_SWEEP_MODE, 0)
            hh.set_tuning(_capi.TUNE_CLUSTER_GROUP, 4)
        case = voxel.eddy_current_case(10, 4)
        b = h.set_matrix_voxel(case)
        f.set_matrix_voxel(case)
        for r, g in zip(solves(h, b), solves(f, b)):
            assert np.array_equal(r, g)
    finally:
        h.close()
        f.close()
