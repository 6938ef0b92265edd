"""The rules that choose between two kernels (csrc/ss_rules.hpp) against measured times (GB300): the side a rule takes is
never more than a tenth slower than the other."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest
import scipy.sparse as sp

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rules():
    so = os.path.join(tempfile.mkdtemp(prefix="rules"), "librules.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(REPO, "sparsesolv_gb300", "csrc"),
                    "-o", so, os.path.join(REPO, "tests", "cpp", "rules_capi.cpp")], check=True)
    lib = ctypes.CDLL(so)
    lib.rule_sweep_wide_rows.restype = ctypes.c_double
    return lib


# FP32, complex, lanes a row, batch, rows a level, us k_sweep, us k_sweep_wide (forward + backward)
SWEEPS = [
    (0, 0, 8, 1, 12010, 983, 1789), (0, 0, 8, 1, 15980, 1213, 1744), (0, 0, 8, 1, 21005, 1568, 1734),
    (0, 0, 8, 1, 30000, 2170, 1753), (0, 0, 8, 1, 20933, 584, 670), (0, 0, 8, 1, 30018, 802, 693),
    (0, 0, 8, 1, 11997, 605, 1116), (0, 0, 8, 1, 15987, 612, 965),
    (0, 0, 8, 0, 6944, 89, 102), (0, 0, 8, 0, 10288, 102, 106), (0, 0, 8, 0, 14564, 126, 112), (0, 0, 8, 0, 18053, 154, 119),
    (0, 0, 8, 0, 21949, 189, 139), (0, 0, 8, 0, 18182, 98, 77), (0, 0, 8, 0, 11429, 89, 81), (0, 0, 8, 0, 1000000, 347, 144),
    (0, 0, 16, 0, 4678, 301, 385), (0, 0, 16, 0, 7260, 422, 481), (0, 0, 16, 0, 11207, 594, 554), (0, 0, 16, 0, 12766, 447, 392),
    (0, 1, 8, 1, 4523, 1806, 2641), (0, 1, 8, 1, 8995, 2972, 3310), (0, 1, 8, 1, 12010, 3700, 3416),
    (0, 1, 8, 1, 15980, 4664, 3561), (0, 1, 8, 1, 9007, 1398, 2342), (0, 1, 8, 1, 15996, 1731, 1445),
    (0, 1, 8, 0, 10288, 329, 267), (0, 1, 8, 0, 4678, 740, 1060), (0, 1, 4, 0, 10288, 221, 252), (0, 1, 4, 0, 18053, 314, 278),
    (0, 1, 4, 0, 4678, 774, 1335), (0, 1, 16, 0, 4678, 1100, 892), (0, 1, 16, 0, 10288, 594, 341),
    (1, 0, 8, 1, 4523, 305, 492), (1, 0, 8, 1, 6482, 614, 528), (1, 0, 8, 1, 12010, 763, 605), (1, 0, 8, 1, 4542, 129, 185),
    (1, 0, 8, 1, 6517, 210, 200), (1, 0, 8, 1, 20933, 346, 220),
    (1, 1, 8, 1, 8995, 457, 1043), (1, 1, 8, 1, 15980, 716, 970), (1, 1, 8, 1, 20933, 271, 271), (1, 1, 8, 1, 30018, 371, 252),
]


@pytest.mark.parametrize("fp32,cplx,G,batch,width,one,wide", SWEEPS)
def test_sweep_kernel(rules, fp32, cplx, G, batch, width, one, wide):
    takes_wide = width > rules.rule_sweep_wide_rows(fp32, cplx, G, batch)
    assert (wide if takes_wide else one) <= 1.1 * min(one, wide)


@pytest.mark.gpu
@pytest.mark.parametrize("n,cplx", [(22528, False), (22530, False), (16384, True), (16386, True)])
def test_both_sides_of_the_line(gpu, oracle, n, cplx):
    """Two levels of n / 2 rows at 8 lanes a row, at and above the line for one system; a row has one off-diagonal entry
    at most, so the sums agree with the oracle's substitution to a few roundings."""
    from sparsesolv_gb300 import _capi
    rng = np.random.default_rng(n)
    off = np.zeros(n - 1, np.complex128 if cplx else np.float64)
    k = len(off[::2])
    off[::2] = rng.uniform(-0.9, -0.1, k) + (1j * rng.uniform(0.1, 0.3, k) if cplx else 0)
    A = sp.diags([off, rng.uniform(1.5, 2.0, n), off], [-1, 0, 1]).tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    h = _capi.Handle(0)
    try:
        h.set_matrix(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data.astype(off.dtype))
        h.set_tuning(_capi.TUNE_SWEEP_MODE, 1)
        h.set_tuning(_capi.TUNE_SWEEP_GROUP, 8)
        lrp, lci, lval, D = h.factor(1.1)
        r = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)
        z = h.apply_precond(r)
    finally:
        h.close()
    zo = oracle.ic_apply(lrp, lci, lval, D, r)
    assert np.linalg.norm(z - zo) <= 1e-14 * np.linalg.norm(zo)
