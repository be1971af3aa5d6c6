"""Resident launches of LPs that fit on the chip (slices.cuh): the sliced plans
on the CPU, and on the GPU the three forms of the iteration and the resident
power iteration against the launches per product."""
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from pdal_gb300 import build, instances as I, lp


def test_sliced_plans_cover_every_nonzero_once(tmp_path):
    exe = tmp_path / "slices_check"
    here = build.ROOT / "tests" / "slices_check.cpp"
    cuda = build._cuda_include()
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", cuda, str(here), str(build.CSRC / "common.cpp"), "-o", str(exe),
                    "-lpthread"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


def _irregular(m, n, k, seed):
    """random_lp with empty rows and columns, a dense row and two dense columns
    (long in the row-block plans)."""
    d = I.random_lp(m, n, k, seed=seed)
    rp, ci, v, _ = d.csr()
    rows = np.repeat(np.arange(m), np.diff(rp))
    keep = ~np.isin(rows, [3, m - 1]) & ~np.isin(ci, [0, 7, n - 2])
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rows[keep], np.full(n // 2, 5), np.arange(0, m, 2), np.arange(1, m, 3)])
    cols = np.concatenate([ci[keep], np.arange(0, n, 2)[:n // 2], np.full((m + 1) // 2, 11), np.full((m + 1) // 3, 12)])
    A = sp.csr_matrix((0.3 * rng.standard_normal(rows.size), (rows, cols)), shape=(m, n))
    A.sum_duplicates()
    d.A = (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, (m, n))
    return d


CASES = {
    "one": lambda: I.random_lp(1, 1, 1, seed=1),
    "tiny": lambda: I.random_lp(17, 33, 3, seed=2),
    "irregular": lambda: _irregular(700, 1500, 6, 3),
    "tagged_largest": lambda: I.random_lp(4500, 11200, 8, seed=4),    # just under 90,000 nonzeros
    "barrier_smallest": lambda: I.random_lp(4500, 11400, 8, seed=5),  # just over
    "irregular_barrier": lambda: _irregular(9000, 21000, 8, 6),
    "fp32_barrier": lambda: I.random_lp(30000, 76000, 8, seed=7),     # over 600,000 nonzeros
}


@pytest.mark.gpu
@pytest.mark.parametrize("protocol", [{}, {"al_lambda": 0.0}, {"sigma_mode": 1}], ids=["default", "lambda0", "sigma"])
@pytest.mark.parametrize("case", CASES)
def test_resident_forms_match_the_launches(lp_lib, case, protocol):
    """200 iterations from the same start.  The forms differ in the order of
    the sums only: a row sum of k terms moves by at most k eps of its absolute
    sum, and the iteration is nonexpansive in its own norm, so 200 iterations
    of rows of up to 1,500 terms stay within 200 * 1500 * eps = 3e-11 (FP64) and
    -- rounding errors adding like a random walk, sqrt(200 * 1500) * eps -- 3e-5
    (FP32) of the iterate, times 10 for the norm's conditioning.  The sigma_max
    estimate is a Rayleigh quotient: its relative error is a few eps."""
    d = CASES[case]()
    p = {"eps": 1e-14, "iteration_limit": 200, "sv_max_iter": 300}
    for precision, tol in (("fp64", 3e-10), ("fp32_refine", 3e-4)):
        o = {**protocol, "precision": precision, "fp32_switch_tol": 1e-14, "fp32_stall_evals": 0, "dual_panels": 0}
        a = lp.solve(d, p, {**o, "persistent_loop": 0})
        b = lp.solve(d, p, o)
        again = lp.solve(d, p, o)
        assert a.status == b.status and a.iterations == b.iterations
        assert a.stats["power_iterations"] == b.stats["power_iterations"]
        assert b.stats["lambda_est"] == pytest.approx(a.stats["lambda_est"], rel=1e-12)
        for u, v in ((a.x, b.x), (a.y, b.y), (a.reduced_cost, b.reduced_cost)):
            assert np.linalg.norm(u - v) <= tol * (1 + np.linalg.norm(u))
        assert np.array_equal(b.x, again.x) and np.array_equal(b.y, again.y)
