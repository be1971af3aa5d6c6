"""Waits of the resident launches that run out (slices.cuh): the launch gives up
and returns, the solve fails with a message, and the context stays usable.  The
waits are made to run out by a limit of no polls, set on the host."""
import numpy as np
import pytest
import scipy.sparse as sp

from pdal_gb300 import instances as I, lp

MESSAGE = "exchange between the blocks"


def _with_long_rows(m, n, k, seed):
    """random_lp with a dense row and a dense column: pieces in both products."""
    d = I.random_lp(m, n, k, seed=seed)
    rp, ci, v, _ = d.csr()
    rows = np.concatenate([np.repeat(np.arange(m), np.diff(rp)), np.full(n, 5), np.arange(m)])
    cols = np.concatenate([ci, np.arange(n), np.full(m, 11)])
    vals = np.concatenate([v, 0.01 * np.random.default_rng(seed).standard_normal(n + m)])
    A = sp.csr_matrix((vals, (rows, cols)), shape=(m, n))
    A.sum_duplicates()
    d.A = (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, (m, n))
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,precision", [(9000, 21000, 8, "fp64"), (30000, 76000, 8, "fp32_refine")])
def test_barrier_form_with_long_rows_gives_up(lp_lib, m, n, k, precision):
    """The iterations' launch in its barrier form: a warp that gives up on the
    parts of a long row still arrives at its block's barriers, so that the
    block leaves as a whole."""
    d = _with_long_rows(m, n, k, 3)
    p = {"eps": 1e-14, "iteration_limit": 200, "sv_max_iter": 50}
    o = {"precision": precision, "dual_panels": 0}
    # the FP64 form's first resident launch is its power iteration
    fail = {**o, "resident_fail_launch": 2 if precision == "fp64" else 1}
    with pytest.raises(RuntimeError, match=MESSAGE):
        lp.solve(d, p, fail)
    assert lp.solve(d, p, o).iterations == 200


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2000, 5000), (9000, 21000)], ids=["tagged", "barrier"])
@pytest.mark.parametrize("launch", [1, 2], ids=["power", "iterations"])
def test_waits_run_out_and_a_new_solve_succeeds(lp_lib, shape, launch):
    """FP64: the power iteration's launch (the service warp and the warps that
    wait for it in shared memory) and the iterations' launch in both forms."""
    d = I.random_lp(*shape, 8, seed=4)
    p = {"eps": 1e-14, "iteration_limit": 200, "sv_max_iter": 50}
    with pytest.raises(RuntimeError, match=MESSAGE):
        lp.solve(d, p, {"resident_fail_launch": launch})
    assert lp.solve(d, p, {}).iterations == 200


@pytest.mark.gpu
def test_a_session_solves_again_after_a_wait_ran_out(lp_lib):
    """The error of one solve is not the next one's."""
    d = I.random_lp(2000, 5000, 8, seed=4)
    p = {"eps": 1e-14, "iteration_limit": 200, "sv_max_iter": 50}
    s = lp.LPSession(d, p, {"resident_fail_launch": 1})
    with pytest.raises(RuntimeError, match=MESSAGE):
        s.solve()
    again = s.solve()
    s.close()
    assert again.iterations == 200
    assert again.stats["lambda_est"] == lp.solve(d, p, {}).stats["lambda_est"]
