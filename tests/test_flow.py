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


def _normals(m):
    """std::normal_distribution over mt19937(1): Marsaglia's polar method on
    pairs of 64-bit uniforms, low word first, the second coordinate's variate
    first."""
    raw = np.random.MT19937()
    raw._legacy_seeding(1)
    w = raw.random_raw(8 * m + 400).astype(np.float64).reshape(-1, 2)
    u = 2.0 * ((w[:, 0] + w[:, 1] * 2.0**32) / 2.0**64) - 1.0
    x, y = u[0::2], u[1::2]
    r2 = x * x + y * y
    x, y, r2 = (a[(r2 <= 1.0) & (r2 > 0.0)] for a in (x, y, r2))
    f = np.sqrt(-2.0 * np.log(r2) / r2)
    return np.stack([y * f, x * f], 1).ravel()[:m]


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 2, 3, 1023, 3000, 20001])
def test_start_vector_of_the_power_iteration(lp_lib, m):
    """One step from the start vector v, scalings off, A = [I | e_i]: the
    quotient is 1 + v_i^2 / |v|^2, for the first, a middle and the last i.
    Rounding: a few eps per variate and sums of m terms in FP64: 1e-12."""
    v = _normals(m)
    for i in {0, m // 2, m - 1}:
        cols = np.concatenate([np.arange(m), [m]])
        rows = np.concatenate([np.arange(m), [i]])
        A = sp.csr_matrix((np.ones(m + 1), (rows, cols)), shape=(m, m + 1))
        d = lp.LPData(np.ones(m + 1), A=A, con_lb=np.zeros(m), con_ub=np.full(m, 5.0), var_lb=np.zeros(m + 1),
                      var_ub=np.full(m + 1, 4.0))
        p = {"eps": 1e-14, "iteration_limit": 1, "sv_max_iter": 1, "l_inf_ruiz_iterations": 0,
             "has_pock_chambolle_alpha": 0}
        g = lp.solve(d, p, {"precision": "fp64"})
        assert g.stats["lambda_est"] == pytest.approx(1.0 + v[i] ** 2 / (v @ v), rel=1e-12)
