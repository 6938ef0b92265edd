"""What the solvers' performance is measured on: whole solves through the entry points a user's program calls.

Every case is a system of the seeded voxel generator (sparsesolv_gb300/voxel.py), in the breadth-first edge order of
the reference's mesh maker: n is about 3 N^3 unknowns with 32 nonzeros a row. One pass is what a time-stepping or
nonlinear FEM program repeats on a mesh it keeps: new values go into the handle, the incomplete factor is rebuilt, the
Krylov iterations run to tolerance and the solution comes back.

``what`` is the kind of work:

* ``solve``   one system, one right-hand side, values and vectors on the device (ssg_update_values_device,
              ssg_solve_device); ``method`` and ``field`` choose the iteration and real or complex values;
* ``multi``   several right-hand sides of one matrix in one call (ssg_solve_multi_device);
* ``mixed``   FP32 inner iterations inside FP64 refinement (precision = mixed);
* ``batch``   many small systems of uneven sizes, several right-hand sides each (ssg_batch_*), host vectors;
* ``new``     the reference's own Python interface on a matrix no handle has seen: SparseMat, a fresh solver, one solve
              with host arrays, so the pattern analysis is paid too.
"""
import math

import numpy as np
import torch

from sparsesolv_gb300 import SparseSolvPy, _capi, voxel

ALPHA = 1.1
MAXIT = 20000
DT = 1.0e-5  # time step of the ``mixed`` cases, s


def listed():
    return [
        # the smallest meshes people debug and teach with: launches and the sweeps' dependency levels are all there is
        {"name": "iccg 10", "what": "solve", "field": "real", "method": "iccg", "N": 10, "conv": 1e-8},
        # the 20^3 static-magnetic model of the project's first workload
        {"name": "iccg 20", "what": "solve", "field": "real", "method": "iccg", "N": 20, "conv": 1e-8},
        # an ordinary mesh, odd size
        {"name": "iccg 41", "what": "solve", "field": "real", "method": "iccg", "N": 41, "conv": 1e-8},
        # the large static-magnetic model: 1.5 M unknowns, the benchmark's workload
        {"name": "iccg 80", "what": "solve", "field": "real", "method": "iccg", "N": 80, "conv": 1e-8},
        # the residual-minimising iteration with the same factor
        {"name": "ic-mrtr 31", "what": "solve", "field": "real", "method": "mrtr", "N": 31, "conv": 1e-8},
        # the default preconditioner of the reference's MRTR: Eisenstat's SGS split, no factor
        {"name": "sgs-mrtr 48", "what": "solve", "field": "real", "method": "sgs", "N": 48, "conv": 1e-8},
        # time-harmonic eddy currents, 0.63 M complex unknowns; 1e-3 is where a frequency sweep or an outer nonlinear
        # loop stops an inner solve, and before the plateau on which these singular systems' iterates turn chaotic
        {"name": "eddy mrtr 60", "what": "solve", "field": "complex", "method": "mrtr", "N": 60, "conv": 1e-3},
        # the same physics with COCG on an ordinary, odd mesh
        {"name": "eddy cocg 33", "what": "solve", "field": "complex", "method": "iccg", "N": 33, "conv": 1e-3},
        # several coils of one device: one matrix, four right-hand sides
        {"name": "coils 36x4", "what": "multi", "field": "real", "method": "iccg", "N": 36, "conv": 1e-8, "rhs": 4},
        # an implicit time step of eddy currents in a conducting background, in mixed precision; the mass term makes the
        # system regular, so the solution is unique and the tolerance fixes its digits
        {"name": "mixed step 44", "what": "mixed", "field": "real", "method": "iccg", "N": 44, "conv": 1e-11},
        # a parameter study: sixteen meshes of 8 to 32 voxels a side, four coil placements each
        {"name": "study 8-32", "what": "batch", "field": "real", "method": "iccg", "lo": 8, "hi": 32, "count": 16,
         "rhs": 4, "conv": 1e-8},
        # a first solve on a new mesh through the drop-in module
        {"name": "new mesh 24", "what": "new", "field": "real", "method": "iccg", "N": 24, "conv": 1e-8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["solve", "solve", "solve", "eddy", "eddy", "multi", "mixed", "batch", "new"])
    if what == "solve":
        method = rng.choice(["iccg", "iccg", "mrtr", "sgs"])
        return {"what": "solve", "field": "real", "method": method, "N": _log_int(rng, 8, 76), "conv": 1e-8}
    if what == "eddy":
        return {"what": "solve", "field": "complex", "method": rng.choice(["mrtr", "iccg"]),
                "N": _log_int(rng, 16, 56), "conv": 1e-3}
    if what == "multi":
        return {"what": "multi", "field": "real", "method": "iccg", "N": _log_int(rng, 10, 40), "conv": 1e-8,
                "rhs": rng.randint(2, 6)}
    if what == "mixed":
        return {"what": "mixed", "field": "real", "method": "iccg", "N": _log_int(rng, 12, 60), "conv": 1e-11}
    if what == "batch":
        hi = rng.choice([12, 16, 24, 32])
        return {"what": "batch", "field": "real", "method": "iccg", "lo": rng.randint(6, 10), "hi": hi,
                "count": rng.randint(6, 24), "rhs": rng.randint(1, 5), "conv": 1e-8}
    return {"what": "new", "field": rng.choice(["real", "real", "complex"]), "method": "iccg",
            "N": _log_int(rng, 16, 32), "conv": 1e-3}


# ---------------------------------------------------------------- systems
def _iron(N):
    # one block on small meshes, three on large ones, as the generator's own workloads have them
    return (1, max(2, (3 * N) // 10)) if N < 32 else (3, max(2, (3 * N) // 20))


def _voxels(case, seed):
    N = case["N"]
    if case["what"] == "mixed":
        c = voxel.curl_curl_case(N, seed, *_iron(N))
        c.conductors = [voxel.Block(0, 0, 0, N, N, N)]
        c.sigma, c.omega = 1.0e7, 1.0 / DT
        return c
    if case["field"] == "complex":
        return voxel.eddy_current_case(N, seed)
    return voxel.curl_curl_case(N, seed, *_iron(N))


def _current(seed):
    """The coil current in A/m^2 (the generator's coils carry 1)."""
    return float(np.random.default_rng(seed + 7919).uniform(0.5, 2.0))


def _system(case, seed):
    """(row_ptr, col, val, b) on the host, assembled on the device."""
    vox = _voxels(case, seed)
    maker = _capi.Handle(0)
    try:
        b = maker.set_matrix_voxel(vox)
        rp, ci, val = maker.get_matrix()
    finally:
        maker.close()
    if case["what"] == "mixed":
        val, b = val.real + val.imag, np.ascontiguousarray(b.real)
    return vox, rp, ci, np.ascontiguousarray(val), b * _current(seed)


def _options(case):
    o = _capi.Handle.default_options()
    o.accel_factor = ALPHA
    o.precondition_type = 1 if case["method"] == "sgs" else 0
    o.is_save_residual_log = 1
    o.precision = _capi.PREC_MIXED if case["what"] == "mixed" else _capi.PREC_FP64
    return o


def _batch_sizes(case):
    """Voxels a side of a batch's systems, N ~ U{lo..hi} (a study's meshes do not change with its geometries)."""
    rng = np.random.default_rng([case["lo"], case["hi"], case["count"]])
    return [int(v) for v in rng.integers(case["lo"], case["hi"] + 1, case["count"])]


def prepare(case, seed):
    what = case["what"]
    if what == "batch":
        batch = _capi.Batch(0)
        rng = np.random.default_rng(seed)
        rhs = []
        for N in _batch_sizes(case):
            vox = voxel.curl_curl_case(N, int(rng.integers(1 << 30)), 1, max(2, N // 4))
            coils = [[voxel.seeded_coil(rng, N)] for _ in range(case["rhs"])]
            rp, ci, val, B = vox.assemble(coils_list=coils)
            rhs.append(np.ascontiguousarray(B * _current(seed)))
            batch.add(rp, ci, val, rhs[-1])
        return {"case": case, "batch": batch, "rhs": rhs}
    vox, rp, ci, val, b = _system(case, seed)
    if what == "new":
        return {"case": case, "csr": (rp, ci, val), "b": b, "x0": np.zeros_like(b)}
    h = _capi.Handle(0)
    h.set_options(_options(case))
    h.set_matrix(rp, ci, val)
    if what == "multi":
        rng = np.random.default_rng(seed + 1)
        more = [vox.rhs([voxel.seeded_coil(rng, case["N"])]) for _ in range(case["rhs"] - 1)]
        b = np.stack([b] + more)
    return {"case": case, "handle": h, "val": torch.from_numpy(val).cuda(), "b": torch.from_numpy(b).cuda()}


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    method = _capi.METHOD_ICCG if case["method"] == "iccg" else _capi.METHOD_MRTR
    if case["what"] == "batch":
        batch = state["batch"]
        for k, B in enumerate(state["rhs"]):
            batch.set_rhs(k, B)
        batch.start(method, ALPHA, conv=case["conv"], max_ite=MAXIT)
        batch.wait()
        return [batch.result(k)[0] for k in range(len(state["rhs"]))]
    if case["what"] == "new":
        cplx = case["field"] == "complex"
        A = (SparseSolvPy.SparseMatC if cplx else SparseSolvPy.SparseMat).from_csr(*state["csr"])
        solver = SparseSolvPy.MatSolverICCG()
        solver.setAccelFactor(ALPHA)
        solve = solver.solve_complex if cplx else solver.solve_real
        return solve(case["conv"], MAXIT, A, state["b"], state["x0"])[1]
    h = state["handle"]
    # torch made the buffers on its own stream, the handle works on its own
    torch.cuda.current_stream().synchronize()
    h.update_values_device(state["val"].data_ptr())
    x = torch.empty_like(state["b"])
    if case["what"] == "multi":
        h.solve_multi_device(method, case["rhs"], state["b"].data_ptr(), x.data_ptr(), conv=case["conv"],
                             max_ite=MAXIT)
    else:
        h.solve_device(method, state["b"].data_ptr(), x.data_ptr(), conv=case["conv"], max_ite=MAXIT)
    return x


# ---------------------------------------------------------------- what a pass cannot do without
def _unknowns(N):
    return 3 * N * (N - 1) ** 2


def _iterations(case, N):
    """About how many iterations the reference's own method takes to the tolerance (counts of the FP64 oracle)."""
    if case["what"] == "mixed":
        return 30
    if case["conv"] > 1e-4:
        return max(8, (0.9 if case["field"] == "complex" else 0.6) * N)
    return 2 + 1.42 * N


def work(case):
    v = 16 if case["field"] == "complex" else 8
    fl = 8 if case["field"] == "complex" else 2
    sizes = [case["N"]] if "N" in case else _batch_sizes(case)
    rhs = case.get("rhs", 1)
    by = ops = 0.0
    for N in sizes:
        n = _unknowns(N)
        nnz, half = 32.4 * n, 16.7 * n
        its = _iterations(case, N)
        # factor: the matrix's lower half in, the factor out; an iteration: the matrix once, the factor twice (or the
        # matrix's two halves), about ten vectors
        vs = 4 if case["what"] == "mixed" else v  # the inner iterations' value size
        by += (4 + v) * nnz + 2 * (4 + v) * half + 2 * v * n * rhs
        by += its * ((4 + vs) * nnz + 2 * (4 + vs) * half + 10 * vs * n * rhs)
        ops += fl * (8.0 * half + rhs * its * (nnz + 2 * half + 8 * n))
    return {"bytes": by, "flops": ops}


# ---------------------------------------------------------------- the same in 64 bits, without the package's solvers
def _plain_factor(n, rp, ci, val, alpha):
    """L (with its pivots on the diagonal) of the shifted IC(0): l_ij = a_ij - sum l_ik l_jk / l_kk on the pattern of A's
    lower half, the diagonal of A multiplied by alpha."""
    rows, dinv = [], [0.0] * n
    val = val.tolist()
    for i in range(n):
        row, full = [], {}
        for k in range(rp[i], rp[i + 1]):
            j = ci[k]
            if j > i:
                break
            s = val[k] if j < i else val[k] * alpha
            if j < i:
                for c, w in rows[j]:
                    if c >= j:
                        break
                    if c in full:
                        s -= full[c] * w * dinv[c]
            else:
                for c, w in row:
                    s -= w * w * dinv[c]
            full[j] = s
            row.append((j, s))
        rows.append(row)
        dinv[i] = 1.0 / row[-1][1]
    return rows


def _plain_cg(A, precond, b, conv, cap):
    x = torch.zeros_like(b)
    r = b.clone()
    z = precond(r)
    p = z.clone()
    rz = torch.sum(r * z)
    bn = float(torch.linalg.vector_norm(b))
    for _ in range(cap):
        ap = A @ p
        a = rz / torch.sum(p * ap)
        x = x + a * p
        r = r - a * ap
        if float(torch.linalg.vector_norm(r)) < conv * bn:
            break
        z = precond(r)
        new = torch.sum(r * z)
        p = z + (new / rz) * p
        rz = new
    return x


def exact(case, seed):
    """``mixed``: the system is regular, so x is A^-1 b (a Jacobi-CG in 64 bits far below the tolerance). Small
    ``iccg`` solves: the same iteration on a factor computed here, with dense triangular solves. The larger and the
    other methods' singular systems have no value that does not depend on the whole iteration."""
    if case["what"] == "mixed":
        _, rp, ci, val, b = _system(case, seed)
        A = torch.sparse_csr_tensor(torch.from_numpy(rp), torch.from_numpy(ci), torch.from_numpy(val)).cuda()
        d = torch.from_numpy(val[np.repeat(np.arange(len(b)), np.diff(rp)) == ci]).cuda()
        return _plain_cg(A, lambda r: r / d, torch.from_numpy(b).cuda(), 1e-15, 600)
    if case["what"] not in ("solve", "new") or case["method"] != "iccg" or case["N"] > 20:
        return None
    _, rp, ci, val, b = _system(case, seed)
    n = len(b)
    L = torch.zeros((n, n), dtype=torch.from_numpy(val).dtype)
    for i, row in enumerate(_plain_factor(n, rp.tolist(), ci.tolist(), val, ALPHA)):
        L[i, [j for j, _ in row]] = torch.tensor([s for _, s in row], dtype=L.dtype)
    L = L.cuda()
    pivots = torch.diagonal(L).clone().unsqueeze(1)
    A = torch.sparse_csr_tensor(torch.from_numpy(rp), torch.from_numpy(ci), torch.from_numpy(val)).cuda()

    def precond(r):
        y = torch.linalg.solve_triangular(L, r.unsqueeze(1), upper=False)
        return torch.linalg.solve_triangular(L.T, y * pivots, upper=True).squeeze(1)

    return _plain_cg(A, precond, torch.from_numpy(b).cuda(), case["conv"], 400)
