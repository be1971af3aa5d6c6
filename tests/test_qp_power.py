"""The power iterations of the QP solver in slices (facp_power.cuh) against the
same ones in the persistent kernel."""
import numpy as np
import pytest
import scipy.sparse as sp

from pdal_gb300 import qp

pytestmark = pytest.mark.gpu


def _qp(m, n, seed, long_rows):
    """Random A and Q, a few rows empty; long_rows stores 97 further entries of
    1e-300 in one row of each, which change no sum and no maximum but send both
    products to the persistent kernel."""
    rng = np.random.default_rng(seed)
    A = sp.random(m, n, density=min(1.0, 4.0 / n), random_state=rng, format="lil")
    B = sp.random(max(n // 2, 1), n, density=min(1.0, 2.0 / n), random_state=rng, format="csr")
    A[0, 0] = 1.0
    Q = (B.T @ B + sp.diags(np.where(np.arange(n) % 5 == 0, 0.0, 0.1))).tolil()
    Q[0, 0] = 1.0
    if long_rows:
        k = np.arange(min(n, 97))
        for M in (A, Q):
            for j in k:
                if M[0, j] == 0.0:
                    M[0, j] = 1e-300
        for j in k:
            if Q[j, 0] == 0.0:
                Q[j, 0] = 1e-300
    return qp.QPData(rng.standard_normal(n), A=A.tocsr(), con_lb=np.zeros(m), con_ub=np.ones(m), var_lb=-np.ones(n),
                     var_ub=np.ones(n), Q=Q.tocsr())


@pytest.mark.parametrize("steps", [1, 7, 5000])
@pytest.mark.parametrize("m,n", [(1, 97), (31, 128), (33, 100), (2048, 2049), (2049, 4100)])
def test_slices_match_the_persistent_kernel(m, n, steps):
    """The quotients are second order in the vectors' rounding, sums of up to
    4,100 terms: 1e-12 relative; the smallest eigenvalue comes from a shift by
    the largest, so 1e-12 of that.  The number of steps is the same unless a
    test falls within rounding of its bound: one step."""
    p = {"iteration_limit": 1, "sv_max_iter": steps}
    a, b = (qp.solve(_qp(m, n, 11 * m + n, lr), p).stats for lr in (True, False))
    assert b["max_singular_value"] == pytest.approx(a["max_singular_value"], rel=1e-12)
    assert b["q_norm"] == pytest.approx(a["q_norm"], rel=1e-12)
    assert b["q_nonconvexity"] == pytest.approx(a["q_nonconvexity"], abs=1e-12 * a["q_norm"])
    assert abs(a["power_iterations_a"] - b["power_iterations_a"]) <= 1
    assert abs(a["power_iterations_q"] - b["power_iterations_q"]) <= 2
