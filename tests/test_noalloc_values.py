"""Sizes and special values of the allocation-free evaluation of a point."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from pdal_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("special", [None, "nan_x", "nan_a", "inf_x", "neg_nan"])
@pytest.mark.parametrize("m,n", [(1, 1), (7, 255), (8, 257), (9, 5000), (2049, 300)])
def test_values_match_numpy(lp_lib, m, n, special):
    """Sums of up to 5,000 terms of the same sign pattern in FP64: a relative
    error of 1e-12 of the terms' absolute sum covers any order; the largest
    residual is that of one row of at most 20 terms."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(7 * m + n)
    A = sp.random(m, n, density=min(1.0, 10.0 / n), random_state=rng, format="csr", dtype=np.float64)
    x = rng.standard_normal(n)
    c = rng.standard_normal(n)
    lb, ub = -rng.random(m), rng.random(m)
    lb[::3], ub[1::3] = -np.inf, np.inf
    if special and A.nnz == 0:
        pytest.skip("no entry to carry the value")
    if special in ("nan_x", "inf_x", "neg_nan"):
        x[A.indices[-1]] = {"nan_x": np.nan, "neg_nan": -np.nan, "inf_x": np.inf}[special]
    if special == "nan_a":
        A.data[-1] = np.nan
    d = lambda a, t: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")
    t = [d(A.indptr, torch.int32), d(A.indices, torch.int32), d(A.data, torch.float64)]
    t += [d(a, torch.float64) for a in (lb, ub, c, x)]
    out = torch.full((3,), -1.0, dtype=torch.float64, device="cuda")
    rc = lp_lib.cp_al_gb300_primal_kkt_noalloc(m, n, *(C.c_void_p(a.data_ptr()) for a in (*t, out)), None)
    assert rc == 0, N.last_error(lp_lib)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    with np.errstate(invalid="ignore"):
        s = A @ x
        res = s - np.fmax(lb, np.fmin(s, ub))
        res[np.isnan(s)] = np.nan
        want = [np.sqrt(np.sum(res * res)), np.max(np.abs(res)), np.sum(c * x)]
        scale = [np.linalg.norm(abs(A) @ np.abs(x)), np.max(abs(A) @ np.abs(x)), np.sum(np.abs(c * x))]
    for g, w, k in zip(got, want, scale):
        if np.isfinite(w):
            assert abs(g - w) <= 1e-12 * k
        else:
            assert (np.isnan(g) and np.isnan(w)) or g == w
