"""Order of the Pock-Chambolle sums of rows longer than a row block."""
import numpy as np
import pytest
import scipy.sparse as sp

from pdal_gb300 import lp


@pytest.mark.gpu
@pytest.mark.parametrize("length", [2049, 5000, 5024])
def test_long_rows_are_summed_in_row_order(lp_lib, length):
    """FP64 form, one Pock-Chambolle pass: the scale of a row of several pieces,
    and of a column of A as long, is the square root of its entries added one
    after the other, bit for bit."""
    rng = np.random.default_rng(length)
    k = length
    A = sp.lil_matrix((k, k + 2))
    A[1, :k] = rng.lognormal(0.0, 3.0, k)
    A[:, k + 1] = rng.lognormal(0.0, 3.0, (k, 1))
    A = A.tocsr()
    d = lp.LPData(np.ones(k + 2), A=A, con_lb=np.zeros(k), con_ub=np.ones(k), var_lb=np.zeros(k + 2),
                  var_ub=np.ones(k + 2))
    p = {"eps": 1e-4, "iteration_limit": 1, "sv_max_iter": 1, "l_inf_ruiz_iterations": 0,
         "has_pock_chambolle_alpha": 1, "pock_chambolle_alpha": 1.0}
    s = lp.LPSession(d, p, {"precision": "fp64"})
    s.solve()
    _, r, c, *_ = s.scaling()
    s.close()
    assert r[1] == np.sqrt(np.add.accumulate(np.abs(A[1].data))[-1])
    assert c[k + 1] == np.sqrt(np.add.accumulate(np.abs(A[:, [k + 1]].toarray().ravel()))[-1])
