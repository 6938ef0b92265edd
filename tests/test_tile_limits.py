"""Which triangles the tile sweep's plan takes (csrc/ss_tile_plan.cpp): orders that keep a row's dependencies near it, and
not the ones in which tiles mostly read each other, where the sync-free sweep was measured the faster."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest
import scipy.sparse as sp

from sparsesolv_gb300 import voxel

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "sparsesolv_gb300", "csrc")


@pytest.fixture(scope="module")
def lib():
    so = os.path.join(tempfile.mkdtemp(prefix="tilelimits"), "libtilelimits.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", so,
                    os.path.join(CSRC, "ss_tile_plan.cpp"),
                    os.path.join(REPO, "tests", "cpp", "tile_limits_check.cpp")], check=True)
    lib = ctypes.CDLL(so)
    lib.tile_limits_check.restype = ctypes.c_char_p
    return lib


def matrix(name):
    kind, _, order = name.partition(" ")
    if kind.startswith("voxel"):
        rp, ci, va, _ = voxel.curl_curl_case(int(kind[5:]), seed=3).assemble()
        A = sp.csr_matrix((va, ci, rp))
    elif kind.startswith("grid"):  # 7-point
        N = int(kind[4:])
        T = sp.diags([-np.ones(N - 1), 2.1 * np.ones(N), -np.ones(N - 1)], [-1, 0, 1])
        I = sp.eye(N)
        A = sp.csr_matrix(sp.kron(sp.kron(T, I), I) + sp.kron(sp.kron(I, T), I) + sp.kron(sp.kron(I, I), T))
    else:
        n = 20000
        A = sp.csr_matrix(sp.diags([-np.ones(n - 1), 2.5 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1]))
    n = A.shape[0]
    q = np.arange(n)
    if order == "random":
        q = np.random.default_rng(0).permutation(n)
    elif order:  # shuffled within a window of so many rows
        q = np.argsort(q + np.random.default_rng(1).uniform(0, int(order), n))
    A = sp.csr_matrix(A[q][:, q])
    A.sort_indices()
    return A


DEVICE = 284 << 30


def ask(lib, oracle, A, lower, elem, lanes, device_bytes=DEVICE, size=None):
    rp, ci = A.indptr.astype(np.int32), A.indices.astype(np.int32)
    n = len(rp) - 1
    trp, tci, _ = oracle.triangle(rp, ci, lower)
    level, perm, lptr = oracle.levels(rp, ci, lower)
    level, perm = np.ascontiguousarray(level, np.int32), np.ascontiguousarray(perm, np.int32)
    ipos = np.empty(n, np.int32)
    ipos[perm] = np.arange(n, dtype=np.int32)
    lens = np.diff(trp)[perm]
    prp = np.zeros(n + 1, np.int32)
    np.cumsum(lens, out=prp[1:])
    pci = np.ascontiguousarray(tci[np.repeat(trp[:-1][perm] - prp[:-1], lens) + np.arange(prp[-1])], np.int32)
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in (prp, pci, ipos, level)]
    return lib.tile_limits_check(n, len(lptr) - 1, *ptr, int(lower), elem, lanes, ctypes.c_longlong(device_bytes),
                                 size if size is None else ctypes.byref(size)).decode()


# (matrix, lanes a row: 0 real, 4 complex, 8 complex; served by the tile sweep)
@pytest.mark.parametrize("name,lanes,served", [
    ("voxel24", 0, True), ("voxel24", 4, True), ("voxel24", 8, True), ("grid30", 0, True), ("grid30", 4, True),
    ("chain", 0, True), ("chain", 4, True), ("voxel10 random", 0, True), ("voxel12 random", 0, True),
    ("voxel24 500", 0, True), ("voxel24 500", 4, True),
    ("voxel16 random", 0, False), ("voxel24 random", 0, False), ("grid30 random", 0, False),
    ("voxel12 random", 4, False), ("voxel24 random", 4, False), ("voxel24 random", 8, False),
    ("voxel24 6000", 4, False),
])
def test_orders_that_scatter_dependencies_are_refused(lib, oracle, monkeypatch, name, lanes, served):
    A = matrix(name)
    for lower in (True, False):
        got = []
        for threads in ("1", "3", "8"):
            monkeypatch.setenv("SSG_PLAN_THREADS", threads)
            got.append(ask(lib, oracle, A, lower, 16 if lanes else 8, lanes))
        assert got[0] == got[1] == got[2]  # by which limit, too
        assert (got[0] == "") == served, got[0]
        if not served:
            assert "too many" in got[0]


@pytest.mark.parametrize("lanes", [1, 2, 16])
def test_lanes_the_records_cannot_hold_are_refused(lib, oracle, lanes):
    assert "lanes" in ask(lib, oracle, matrix("chain"), True, 16, lanes)


@pytest.mark.parametrize("name,lanes", [("voxel12", 0), ("voxel12", 4), ("chain", 0)])
def test_records_beyond_their_share_of_the_device_are_refused(lib, oracle, monkeypatch, name, lanes):
    """The records may take a sixteenth of the device's memory: at that line the plan is made, a byte below it is not."""
    A = matrix(name)
    size = ctypes.c_longlong(0)
    assert ask(lib, oracle, A, True, 16 if lanes else 8, lanes, size=size) == ""
    for threads in ("1", "8"):
        monkeypatch.setenv("SSG_PLAN_THREADS", threads)
        assert ask(lib, oracle, A, True, 16 if lanes else 8, lanes, 16 * size.value) == ""
        assert ask(lib, oracle, A, True, 16 if lanes else 8, lanes, 16 * size.value - 1) == "records too large"
    csr = (8 + 4 + 8 * (lanes > 0)) * sp.tril(A).nnz
    assert size.value <= 20 * csr  # the inflation the limit is stated with
