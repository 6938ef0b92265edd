"""The tile sweep's schedule (csrc/ss_tile_plan.cpp), checked and emulated on the CPU by tests/cpp/tile_plan_check.cpp:
every read names the value the row needs and is covered by the stage's waits, no ring slot or staged record is reused
before its last reader, no wait can go in a circle, and the emulated sums reproduce a triangular solve. Small rings force
the reuse rules and the far entries that the shipped layout meets only on large systems."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import spsolve_triangular

from sparsesolv_gb300 import voxel

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "sparsesolv_gb300", "csrc")


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(tempfile.mkdtemp(prefix="tileplan"), "libtileplan.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", so,
                    os.path.join(CSRC, "ss_tile_plan.cpp"), os.path.join(REPO, "tests", "cpp", "tile_plan_check.cpp")],
                   check=True)
    lib = ctypes.CDLL(so)
    lib.tile_check.restype = ctypes.c_char_p
    return lib


def _p(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


def irregular(n=3000):
    S = sp.random(n, n, density=5.0 / n, random_state=np.random.RandomState(3), format="csr")
    S = S + S.T
    return sp.csr_matrix(S + sp.diags(np.asarray(abs(S).sum(axis=1)).ravel() + 1.0))


def matrix(name):
    if name.startswith("voxel"):
        rp, ci, va, _ = voxel.curl_curl_case(int(name[5:]), seed=11).assemble()
        va = va.copy()
        va[np.repeat(np.arange(len(rp) - 1), np.diff(rp)) == ci] *= 1.3
        return sp.csr_matrix((va, ci, rp))
    if name == "chain":
        n = 1500
        return sp.diags([-np.ones(n - 1), 2.5 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    if name == "diagonal":
        return sp.diags(np.arange(1.0, 301.0)).tocsr()
    if name == "one":
        return sp.csr_matrix(np.array([[4.0]]))
    if name == "arrow":
        A = sp.lil_matrix((800, 800))
        A.setdiag(2.0)
        A[799, :799] = 1e-3
        A[:799, 799] = 1e-3
        return sp.csr_matrix(A)
    return irregular()


SMALL = (64, 128, 32768)   # own ring, halo ring, staging ring (bytes)


@pytest.mark.parametrize("name", ["voxel8", "voxel13", "irregular", "chain", "arrow", "diagonal", "one"])
@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("T", [0, 1, 7, 40])
@pytest.mark.parametrize("lay", [None, SMALL])
@pytest.mark.parametrize("lanes", [0, 4, 8])
@pytest.mark.parametrize("CS", [1, 8])
def test_tile_plan_checks_and_emulates(lib, oracle, name, lower, T, lay, lanes, CS):
    A = matrix(name)
    A.sort_indices()
    rp, ci = A.indptr.astype(np.int32), A.indices.astype(np.int32)
    n = len(rp) - 1
    trp, tci, tsrc = oracle.triangle(rp, ci, lower)
    level, perm, lptr = oracle.levels(rp, ci, lower)
    nlev = len(lptr) - 1
    level, perm = np.ascontiguousarray(level, np.int32), np.ascontiguousarray(perm, np.int32)
    ipos = np.empty(n, np.int32)
    ipos[perm] = np.arange(n, dtype=np.int32)
    lens = np.diff(trp)[perm]
    prp = np.zeros(n + 1, np.int32)
    np.cumsum(lens, out=prp[1:])
    idx = np.concatenate([np.arange(trp[i], trp[i + 1]) for i in perm])
    pci = np.ascontiguousarray(tci[idx], np.int32)
    val = np.ascontiguousarray(A.data[tsrc][idx], np.float64)
    diag = A.diagonal()
    lvec = np.ascontiguousarray(1.0 / diag[perm])
    r = np.random.default_rng(1).standard_normal(n)
    y = np.full(n, np.nan)
    stats = np.zeros(2, np.int32)
    ring = None if lay is None else np.array(lay, np.int32)
    why = lib.tile_check(n, int(nlev), _p(prp), _p(pci), _p(ipos), _p(level), int(lower), lanes, T, CS, _p(ring), _p(val), _p(lvec),
                         _p(r), _p(y), _p(stats)).decode()
    if "newest dependency left its ring" in why:  # another sweep serves it; never with the shipped rings here
        assert lay is not None and lanes == 0
        return
    if "does not fit the staging ring" in why:  # nor a dense row
        assert name == "arrow"
        return
    assert why == ""
    ref = spsolve_triangular(sp.csr_matrix((A.data[tsrc], tci, trp), shape=(n, n)).tocsr(), r, lower=lower)
    assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref) * max(1.0, np.sqrt(n))
    if lay is not None and name == "voxel13" and T != 40:
        assert stats[1] > 0  # the far path is exercised
