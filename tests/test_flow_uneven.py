"""Resident launches of LPs whose rows differ in length: a few rows of some hundred
entries among short ones."""
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from pdal_gb300 import build, instances as I, lp


def test_no_lane_holds_a_long_chain(tmp_path):
    exe = tmp_path / "slices_chain_check"
    here = build.ROOT / "tests" / "slices_chain_check.cpp"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", build._cuda_include(), str(here), str(build.CSRC / "common.cpp"),
                    "-o", str(exe), "-lpthread"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


def _uneven(m, n, k, rows, length, seed):
    """random_lp with `length` more entries in `rows` rows and in one column."""
    d = I.random_lp(m, n, k, seed=seed)
    rp, ci, v, _ = d.csr()
    rng = np.random.default_rng(seed)
    more = rng.choice(m, rows, replace=False)
    r = np.concatenate([np.repeat(np.arange(m), np.diff(rp)), np.repeat(more, length),
                        rng.choice(m, min(length, m), replace=False)])
    c = np.concatenate([ci] + [rng.choice(n, length, replace=False) for _ in more] + [np.full(min(length, m), 11)])
    vals = np.concatenate([v, 0.1 * rng.standard_normal(r.size - v.size)])
    A = sp.csr_matrix((vals, (r, c)), shape=(m, n))
    A.sum_duplicates()
    d.A = (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, (m, n))
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,rows,length", [(1200, 3000, 6, 3, 250), (5000, 10000, 8, 1, 100),
                                               (20000, 50000, 8, 5, 350), (40000, 100000, 8, 20, 1500)])
def test_uneven_rows_match_the_launches(lp_lib, m, n, k, rows, length):
    """200 iterations: the forms differ in the order of the sums only, at most
    200 * 1600 * eps of the iterate in FP64 and sqrt(200 * 1600) * eps in FP32,
    times 10 for the conditioning of its norm."""
    d = _uneven(m, n, k, rows, length, 3)
    p = {"eps": 1e-14, "iteration_limit": 200, "sv_max_iter": 200}
    for precision, tol in (("fp64", 7e-10), ("fp32_refine", 7e-4)):
        o = {"precision": precision, "fp32_switch_tol": 1e-14, "fp32_stall_evals": 0, "dual_panels": 0}
        a = lp.solve(d, p, {**o, "persistent_loop": 0})
        b = lp.solve(d, p, o)
        assert a.iterations == b.iterations
        assert b.stats["lambda_est"] == pytest.approx(a.stats["lambda_est"], rel=1e-12 if precision == "fp64" else 1e-6)
        for u, w in ((a.x, b.x), (a.y, b.y)):
            assert np.linalg.norm(u - w) <= tol * (1 + np.linalg.norm(u))
