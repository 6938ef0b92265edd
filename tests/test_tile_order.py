"""A wait of the tile sweep (csrc/ss_tile.cu) orders memory for the whole warp.

Lane w acquires the progress word of warp w, then every lane reads ring values that any warp wrote. CUDA's vote functions
imply no memory ordering, __syncwarp() does, so it has to stand between the vote and whatever the wait covers. Hardware
that happens to run a converged warp's shared-memory accesses in order hides a missing one: the first test reads the
source, the second repeats sweeps on the GPU."""
import os
import re

import numpy as np
import pytest
import scipy.sparse as sp

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_progress_vote_is_followed_by_a_warp_barrier():
    src = open(os.path.join(REPO, "sparsesolv_gb300", "csrc", "ss_tile.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    body = re.search(r"auto ready = \[&\]\(int og, int h\) \{(.*?)\n        \};", src, re.S).group(1)
    vote = body.index("__all_sync(")
    assert "tl_ld_acquire(" in body[vote:] and "__syncwarp();" in body[vote:]
    # what a wait covers is only looked at through it
    assert len(re.findall(r"tl_ld_acquire\(prog", src)) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("name", ["chain", "voxel24"])
def test_repeated_sweeps_give_the_same_bits(gpu, name, cplx):
    from sparsesolv_gb300 import _capi, voxel
    if name == "chain":  # one row a level: every read is of the newest value of another warp
        n = 1500
        A = sp.diags([-np.ones(n - 1), 2.5 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1], format="csr")
        rp, ci, va = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data + (0.2j if cplx else 0.0)
    else:
        rp, ci, va, _ = (voxel.eddy_current_case(24, 3) if cplx else voxel.curl_curl_case(24, 3)).assemble()
    h = _capi.Handle(0)
    try:
        h.set_matrix(rp, ci, va)
        h.factor(1.1)
        rng = np.random.default_rng(2)
        r = rng.standard_normal(len(rp) - 1) + (1j * rng.standard_normal(len(rp) - 1) if cplx else 0.0)
        z = h.apply_precond(r)
        for _ in range(40):
            assert np.array_equal(z, h.apply_precond(r))
    finally:
        h.close()
