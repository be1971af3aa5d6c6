"""Range of the sigma_max estimate of LPs that fit on the chip."""
import numpy as np
import pytest

from pdal_gb300 import instances as I, lp


@pytest.mark.gpu
@pytest.mark.parametrize("options,scales", [({"precision": "fp64"}, (1e-45, 1e-20, 1.0, 1e45)),
                                            ({"precision": "fp32_refine", "power_method": 0}, (1e-8, 1.0, 1e8))],
                         ids=["fp64", "fp32"])
def test_estimate_of_an_unscaled_matrix_is_that_of_the_launches(lp_lib, options, scales):
    """Equilibration off and every entry multiplied by `scale`: the estimate
    takes the square of it, whichever way the products run.  30 steps, none of
    them the last by its residual (tol = 0).  The quotient differs by the order
    of its sums, a few eps: 1e-12 in FP64, 1e-5 in FP32."""
    d = I.random_lp(400, 900, 6, seed=8)
    rp, ci, v, shape = d.csr()
    p = {"l_inf_ruiz_iterations": 0, "has_pock_chambolle_alpha": 0, "bound_objective_rescaling": 0, "sv_max_iter": 30,
         "sv_tol": 0.0}
    tol = 1e-12 if options["precision"] == "fp64" else 1e-5

    def estimate(scale, extra):
        d.A = (rp, ci, np.ascontiguousarray(v * scale), shape)
        s = lp.LPSession(d, p, {**options, **extra})
        _, _, _, *rest = s.scaling()
        s.close()
        return rest[-1] / scale / scale

    plain = estimate(1.0, {"persistent_loop": 0})
    for scale in scales:
        assert estimate(scale, {"persistent_loop": 0}) == pytest.approx(plain, rel=tol)
        assert estimate(scale, {}) == pytest.approx(plain, rel=tol)
