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
    (0, 0, 8, 0, 6944, 89, 102), (0, 0, 8, 0, 10288, 102, 106),
    (0, 0, 8, 0, 14564, 126, 112), (0, 0, 8, 0, 18053, 154, 119),
    (0, 0, 8, 0, 21949, 189, 139), (0, 0, 8, 0, 18182, 98, 77),
    (0, 0, 8, 0, 11429, 89, 81), (0, 0, 8, 0, 1000000, 347, 144),
    (0, 0, 16, 0, 4678, 301, 385), (0, 0, 16, 0, 7260, 422, 481),
    (0, 0, 16, 0, 11207, 594, 554), (0, 0, 16, 0, 12766, 447, 392),
    (0, 1, 8, 1, 4523, 1806, 2641), (0, 1, 8, 1, 8995, 2972, 3310), (0, 1, 8, 1, 12010, 3700, 3416),
    (0, 1, 8, 1, 15980, 4664, 3561), (0, 1, 8, 1, 9007, 1398, 2342), (0, 1, 8, 1, 15996, 1731, 1445),
    (0, 1, 8, 0, 10288, 329, 267), (0, 1, 8, 0, 4678, 740, 1060),
    (0, 1, 4, 0, 10288, 221, 252), (0, 1, 4, 0, 18053, 314, 278),
    (0, 1, 4, 0, 4678, 774, 1335), (0, 1, 16, 0, 4678, 1100, 892), (0, 1, 16, 0, 10288, 594, 341),
    (1, 0, 8, 1, 4523, 305, 492), (1, 0, 8, 1, 6482, 614, 528),
    (1, 0, 8, 1, 12010, 763, 605), (1, 0, 8, 1, 4542, 129, 185),
    (1, 0, 8, 1, 6517, 210, 200), (1, 0, 8, 1, 20933, 346, 220),
    (1, 1, 8, 1, 8995, 457, 1043), (1, 1, 8, 1, 15980, 716, 970),
    (1, 1, 8, 1, 20933, 271, 271), (1, 1, 8, 1, 30018, 371, 252),
]


@pytest.mark.parametrize("fp32,cplx,G,batch,width,one,wide", SWEEPS)
def test_sweep_kernel(rules, fp32, cplx, G, batch, width, one, wide):
    takes_wide = width > rules.rule_sweep_wide_rows(fp32, cplx, G, batch)
    assert (wide if takes_wide else one) <= 1.1 * min(one, wide)


# complex, instances, rows, entries and levels of one; us an iteration, persistent and by launches (sync-free sweeps)
ENGINES = [
    (0, 1, 450, 10842, 78, 207, 240), (0, 64, 450, 10842, 78, 213, 265), (0, 256, 450, 10842, 78, 222, 297),
    (0, 1024, 450, 10842, 78, 571, 446), (0, 1, 1176, 31008, 114, 338, 354), (0, 64, 1176, 31008, 114, 344, 388),
    (0, 256, 1176, 31008, 114, 555, 464), (0, 1, 2430, 67350, 150, 498, 479), (0, 64, 2430, 67350, 150, 793, 598),
    (0, 256, 2430, 67350, 150, 840, 690), (0, 1, 7098, 207570, 222, 1137, 661), (0, 64, 7098, 207570, 222, 1883, 856),
    (0, 1, 400, 1920, 39, 55, 147), (0, 64, 400, 1920, 39, 65, 168), (0, 256, 400, 1920, 39, 84, 180),
    (0, 1024, 400, 1920, 39, 217, 314), (0, 1, 2500, 12300, 99, 312, 324), (0, 64, 2500, 12300, 99, 319, 363),
    (0, 256, 2500, 12300, 99, 545, 468), (0, 1024, 2500, 12300, 99, 990, 1190), (0, 1, 10000, 49600, 199, 987, 594),
    (0, 64, 10000, 49600, 199, 1620, 710), (0, 256, 10000, 49600, 199, 1779, 1247), (0, 1, 512, 3200, 22, 50, 125),
    (0, 64, 512, 3200, 22, 59, 137), (0, 256, 512, 3200, 22, 75, 166), (0, 1024, 512, 3200, 22, 206, 348),
    (0, 1, 1728, 11232, 34, 175, 172), (0, 64, 1728, 11232, 34, 175, 193), (0, 256, 1728, 11232, 34, 281, 302),
    (0, 1024, 1728, 11232, 34, 584, 602), (0, 1, 5832, 38880, 52, 499, 232), (0, 64, 5832, 38880, 52, 653, 327),
    (0, 256, 5832, 38880, 52, 907, 662), (0, 1, 500, 1498, 500, 513, 905), (0, 64, 500, 1498, 500, 835, 1139),
    (0, 256, 500, 1498, 500, 861, 1162), (0, 1024, 500, 1498, 500, 1860, 1301), (0, 1, 1176, 31008, 47, 216, 206),
    (0, 64, 1176, 31008, 47, 217, 224), (0, 256, 1176, 31008, 47, 381, 334), (0, 1, 1000, 21952, 64, 178, 244),
    (0, 64, 1000, 21952, 64, 184, 273), (0, 256, 1000, 21952, 64, 301, 327), (0, 1024, 1000, 21952, 64, 568, 646),
    (0, 1, 8000, 195112, 134, 949, 456), (0, 64, 8000, 195112, 134, 1571, 578), (0, 1, 5000, 34982, 17, 374, 139),
    (0, 64, 5000, 34982, 17, 427, 245), (0, 256, 5000, 34982, 17, 686, 392), (0, 1, 1000, 6962, 15, 84, 112),
    (0, 64, 1000, 6962, 15, 88, 129), (0, 256, 1000, 6962, 15, 106, 190), (0, 1024, 1000, 6962, 15, 324, 373),
    (1, 1, 450, 10842, 78, 281, 365), (1, 64, 450, 10842, 78, 288, 406), (1, 256, 450, 10842, 78, 418, 496),
    (1, 1024, 450, 10842, 78, 931, 1163), (1, 1, 2430, 67350, 150, 694, 760), (1, 64, 2430, 67350, 150, 984, 941),
    (1, 256, 2430, 67350, 150, 1152, 1980), (1, 1, 7098, 207570, 222, 1660, 1071),
    (1, 64, 7098, 207570, 222, 2299, 1574), (1, 1, 400, 1920, 39, 90, 218), (1, 64, 400, 1920, 39, 104, 255),
    (1, 256, 400, 1920, 39, 136, 363), (1, 1024, 400, 1920, 39, 389, 830), (1, 1, 2500, 12300, 99, 433, 505),
    (1, 64, 2500, 12300, 99, 445, 627), (1, 256, 2500, 12300, 99, 706, 1368), (1, 1024, 2500, 12300, 99, 1861, 2659),
    (1, 1, 10000, 49600, 199, 1397, 946), (1, 64, 10000, 49600, 199, 1918, 1671),
    (1, 256, 10000, 49600, 199, 2362, 3845), (1, 1, 1728, 11232, 34, 262, 257), (1, 64, 1728, 11232, 34, 264, 415),
    (1, 256, 1728, 11232, 34, 430, 793), (1, 1024, 1728, 11232, 34, 1236, 1502), (1, 1, 5832, 38880, 52, 765, 365),
    (1, 64, 5832, 38880, 52, 1014, 878), (1, 256, 5832, 38880, 52, 1308, 1638), (1, 1, 500, 1498, 500, 833, 1436),
    (1, 64, 500, 1498, 500, 1112, 1697), (1, 256, 500, 1498, 500, 1132, 1739), (1, 1024, 500, 1498, 500, 2648, 2132),
    (1, 1, 1000, 21952, 64, 268, 379), (1, 64, 1000, 21952, 64, 274, 426), (1, 256, 1000, 21952, 64, 437, 759),
    (1, 1024, 1000, 21952, 64, 1168, 2054),
]


def test_batch_engine(rules):
    """Estimates, so a single batch may go the slower way where the two are close: never by more than 40 %, and by 3 % on
    average (persistent everywhere 50 %, launches everywhere 30 %)."""
    loss = []
    for c, count, n, nnz, lev, pers, launches in ENGINES:
        p = rules.rule_batch_persists(*map(ctypes.c_double, (count, n, nnz, lev)), c, 0)
        loss.append((pers if p else launches) / min(pers, launches))
    assert max(loss) <= 1.4 and np.mean(loss) <= 1.03


@pytest.mark.parametrize("c,n,nnz,lev,pers,tiles", [
    # a handle's own batch, whose launches run the tile sweeps: eight right-hand sides, us an iteration
    (0, 450, 10842, 78, 213, 123), (0, 2430, 67350, 150, 502, 235), (0, 7098, 207570, 222, 1469, 300),
    (0, 400, 1920, 39, 63, 92), (0, 512, 3200, 22, 59, 107),
    (0, 2500, 12300, 99, 318, 158), (0, 500, 1498, 500, 816, 406),
    (0, 5832, 38880, 52, 499, 146), (1, 400, 1920, 39, 102, 161),
    (1, 512, 3200, 22, 126, 191), (1, 2500, 12300, 99, 438, 317),
    (1, 10000, 49600, 199, 1458, 493), (1, 500, 1498, 500, 1104, 896), (1, 5832, 38880, 52, 767, 404),
])
def test_batch_engine_beside_the_tile_sweeps(rules, c, n, nnz, lev, pers, tiles):
    p = rules.rule_batch_persists(*map(ctypes.c_double, (8, n, nnz, lev)), c, 1)
    assert (pers if p else tiles) <= 1.1 * min(pers, tiles)


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


@pytest.mark.gpu
@pytest.mark.parametrize("side,count,persists", [(20, 40, True), (100, 4, False)])
def test_automatic_batch_engine(gpu, side, count, persists):
    """Small systems run persistent (one launch for all iterations), few larger ones by launches; the bits are the same."""
    from sparsesolv_gb300 import _capi
    T = sp.diags([-np.ones(side - 1), 2.1 * np.ones(side), -np.ones(side - 1)], [-1, 0, 1])
    A = sp.csr_matrix(sp.kron(T, sp.eye(side)) + sp.kron(sp.eye(side), T))
    A.sort_indices()
    rp, ci, va = A.indptr.astype(np.int32), A.indices.astype(np.int32), np.ascontiguousarray(A.data)
    h = _capi.Handle(0)
    b = _capi.Batch(0)
    try:
        rng = np.random.default_rng(side)
        for _ in range(count):
            b.add(rp, ci, va, rng.standard_normal(len(rp) - 1))

        def run():
            b.start(_capi.METHOD_ICCG, 1.05, conv=1e-8, max_ite=300)
            b.wait()
            before = h.launch_count()
            b.start(_capi.METHOD_ICCG, 1.05, conv=1e-8, max_ite=300)
            b.wait()
            return [b.result(k)[0] for k in range(count)], h.launch_count() - before

        x, launches = run()
        b.set_persistent(0)
        xl, by_launches = run()
        b.set_persistent(1)
        xp, by_persistent = run()
        assert by_persistent < by_launches
        assert launches == (by_persistent if persists else by_launches)
        for k in range(count):
            assert np.array_equal(x[k], xl[k]) and np.array_equal(x[k], xp[k])
    finally:
        b.close()
        h.close()
