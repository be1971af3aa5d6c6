"""What a session's plan of the resident launches costs."""
import pytest

from pdal_gb300 import instances as I, lp


@pytest.mark.gpu
def test_both_precisions_share_one_plan(lp_lib):
    """FP32_REFINE iterates in both precisions on one sliced plan: it uploads
    what the FP64 form does (a plan of its own is 250 bytes per slice of 32
    rows, here over 60 KB)."""
    d = I.random_lp(2000, 5000, 8, seed=1)
    p = {"eps": 1e-14, "iteration_limit": 200, "sv_max_iter": 20}
    sent = [lp.solve(d, p, {"precision": q, "fp32_switch_tol": 1e-14}).stats["h2d_bytes"]
            for q in ("fp64", "fp32_refine")]
    assert abs(sent[0] - sent[1]) < 4096
