"""Which form the iteration of an LP that fits on the chip takes, and its values on
both sides of the lines."""
import numpy as np
import pytest
import scipy.sparse as sp

from pdal_gb300 import instances as I, lp

P = {"eps": 1e-14, "iteration_limit": 200, "sv_max_iter": 30}


def _options(precision):
    return {"precision": precision, "fp32_switch_tol": 1e-14, "fp32_stall_evals": 0, "dual_panels": 0}


def _dense(m, n):
    """random_lp's data with a dense matrix of unit rows."""
    d = I.random_lp(m, n, 1, seed=3)
    A = sp.csr_matrix(np.random.default_rng(3).standard_normal((m, n)) / np.sqrt(n))
    d.A = (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, (m, n))
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,precision,resident", [
    (2000, 5000, 8, "fp64", True), (2000, 5000, 8, "fp32_refine", True),
    (56000, 140000, 1, "fp64", True),            # fewer nonzeros than rows and columns: up to 150,000
    (80000, 200000, 1, "fp64", False),
    (100000, 290000, 2, "fp64", False),          # many rows, below 600,000
    (50000, 125000, 8, "fp64", True),
    (10000, 25000, 8, "fp32_refine", False),     # FP32 between 100,000 and 630,000
    (50000, 125000, 8, "fp32_refine", True),
    (20000, 50000, 20, "fp32_refine", False),    # fewer rows than lanes
    (30000, 70000, 20, "fp32_refine", False),    # long ones
    (80000, 200000, 8, "fp32_refine", False),    # over 1,500,000
    (280000, 700000, 1, "fp32_refine", False)])
def test_form_by_size_and_shape(lp_lib, m, n, k, precision, resident):
    """The iterations of a block are one launch, or two each."""
    r = lp.solve(I.random_lp(m, n, k, seed=2), P, _options(precision))
    assert r.iterations == 200
    assert (r.stats["kernel_launches"] < 300) == resident


@pytest.mark.gpu
@pytest.mark.parametrize("data", [
    lambda: _dense(40, 1024), lambda: _dense(40, 1025),   # the longest row of a warp, and one in pieces
    lambda: _dense(1025, 30), lambda: _dense(300, 300),
    lambda: I.random_lp(9900, 24800, 8, seed=5),          # just under 200,000 nonzeros
    lambda: I.random_lp(10100, 25300, 8, seed=5),         # just over
    lambda: I.random_lp(12000, 30000, 2, seed=5),         # FP32: plain vectors below 150,000
    lambda: I.transport_lp(30, 31, seed=5)], ids=["row1024", "row1025", "column1025", "dense300", "fp64_tagged",
                                                   "fp64_barrier", "fp32_thin", "transport"])
def test_values_are_those_of_the_launches(lp_lib, data):
    """The forms differ in the order of sums of up to 1,025 terms only: 200
    nonexpansive iterations, at most 200 * 1025 * eps in FP64 and
    sqrt(200 * 1025) * eps in FP32, times 10 for the norm's conditioning.  (The
    estimate of |A|^2 has to have converged for that: after 30 steps it is 5%
    short for two nonzeros per column, and the iteration expands.)"""
    d = data()
    p = {**P, "sv_max_iter": 5000}
    for precision, tol in (("fp64", 5e-10), ("fp32_refine", 6e-4)):
        a = lp.solve(d, p, {**_options(precision), "persistent_loop": 0})
        b = lp.solve(d, p, _options(precision))
        assert a.iterations == b.iterations
        for u, v in ((a.x, b.x), (a.y, b.y)):
            assert np.linalg.norm(u - v) <= tol * (1 + np.linalg.norm(u))


@pytest.mark.gpu
def test_mostly_empty_columns_run_by_launches(lp_lib):
    """6,000 nonzeros in 60,000 columns: a plan of the resident launches would
    list the empty ones too."""
    d = I.random_lp(100, 60000, 1, seed=2)
    rp, ci, v, shape = d.csr()
    A = sp.csr_matrix((v, ci, rp), shape=shape).tocsc()
    A.data[np.repeat(np.arange(shape[1]), np.diff(A.indptr)) >= 6000] = 0.0
    A = A.tocsr()
    A.eliminate_zeros()
    d.A = (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, shape)
    r = lp.solve(d, P, _options("fp64"))
    assert r.iterations == 200 and r.stats["kernel_launches"] > 300
