"""The tile sweeps (ss_tile.cu), the automatic choice, where their tiles, groups and rings have edges: one row, one level,
one row a level, ragged rows, more rows than a group, more levels than staged groups, and several tiles.

Real values are summed by age: the apply agrees with the sync-free sweep's at rounding level (two orders of at most 40
products of one size: 40 * 2^-53 a row, amplified through at most the factor's condition; 1e-11 is the bar the other
schedules have). Complex values are summed as the cluster sweep sums them: the same bits, and the same through a solve."""
import numpy as np
import pytest
import scipy.sparse as sp

from sparsesolv_gb300 import _capi, voxel

pytestmark = pytest.mark.gpu


def csr(A):
    A = sp.csr_matrix(A)
    A.sort_indices()
    cplx = np.iscomplexobj(A.data)
    return (A.indptr.astype(np.int32), A.indices.astype(np.int32),
            np.ascontiguousarray(A.data, np.complex128 if cplx else np.float64))


def matrix(name, cplx):
    if name.startswith("voxel"):
        N = int(name[5:])
        rp, ci, va, _ = (voxel.eddy_current_case(N, 3) if cplx else voxel.curl_curl_case(N, 3)).assemble()
        return rp, ci, va
    rng = np.random.default_rng(5)
    if name == "one":
        A = sp.csr_matrix(np.array([[4.0]]))
    elif name == "diagonal":
        A = sp.diags(rng.uniform(0.5, 3.0, 300))
    elif name == "chain":
        n = 1500
        A = sp.diags([-np.ones(n - 1), 2.5 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1])
    elif name == "band40":  # rows of 40 entries below the diagonal, one row a level
        n = 700
        A = sp.diags([np.full(n - k, -0.01) for k in range(1, 41)], list(range(1, 41)))
        A = A + A.T + sp.diags(np.full(n, 3.0))
    else:  # ragged, levels of hundreds of rows
        n = 6000
        S = sp.random(n, n, density=3.0 / n, random_state=np.random.RandomState(3), format="csr")
        S = S + S.T
        A = S + sp.diags(np.asarray(abs(S).sum(axis=1)).ravel() + 1.0)
    if cplx:
        A = sp.csr_matrix(A).astype(np.complex128) + 1j * sp.diags(rng.uniform(0.1, 0.2, A.shape[0]))
    return csr(A)


@pytest.fixture(scope="module")
def handle(gpu):
    h = _capi.Handle(0)
    yield h
    h.close()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("name", ["one", "diagonal", "chain", "band40", "ragged", "voxel5", "voxel9", "voxel24"])
def test_tile_apply(handle, name, cplx):
    rp, ci, va = matrix(name, cplx)
    n = len(rp) - 1
    handle.set_matrix(rp, ci, va)
    handle.factor(1.1)
    rng = np.random.default_rng(1)
    r = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0.0)
    z = handle.apply_precond(r)
    assert np.array_equal(z, handle.apply_precond(r))
    try:
        handle.set_tuning(_capi.TUNE_SWEEP_MODE, 1)
        handle.set_tuning(_capi.TUNE_SWEEP_GROUP, 4)
        ref = handle.apply_precond(r)
    finally:
        handle.set_tuning(_capi.TUNE_SWEEP_MODE, 0)
        handle.set_tuning(_capi.TUNE_SWEEP_GROUP, 0)
    if cplx:
        assert np.array_equal(z, ref)
    else:
        assert np.linalg.norm(z - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("precondition", [0, 1])
def test_complex_solves_keep_the_cluster_sweeps_bits(handle, precondition):
    vox = voxel.eddy_current_case(16, 4)
    b = handle.set_matrix_voxel(vox)
    o = handle.default_options()
    o.accel_factor = 1.1
    o.precondition_type = precondition
    o.is_save_residual_log = 1
    handle.set_options(o)
    x, xc = np.zeros_like(b), np.zeros_like(b)
    try:
        handle.solve(_capi.METHOD_MRTR, b, x, conv=1e-6, max_ite=60)
        log = handle.residual_log()
        handle.set_tuning(_capi.TUNE_SWEEP_MODE, 2)
        handle.solve(_capi.METHOD_MRTR, b, xc, conv=1e-6, max_ite=60)
        assert np.array_equal(log, handle.residual_log()) and np.array_equal(x, xc)
    finally:
        handle.set_tuning(_capi.TUNE_SWEEP_MODE, 0)
        handle.set_options(handle.default_options())
