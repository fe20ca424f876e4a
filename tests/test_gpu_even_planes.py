"""Planes at the shared-memory limit of the even form (csrc/even.cu, kEvenSmem).

Half planes of 128x128 points fit in FP32 and not in FP64.  An FP32 loop with some
stages left in FP64 (PYRPA_GB_FP32_STAGES) runs those stages on the same tables, so it
has to take the form that FP64 planes allow.  Against the same call with
PYRPA_GB_EVEN=0; the FP32 tolerance of the other parity tests, 1e-4 of the maximum.
"""
import numpy as np
import pytest

from test_gpu_even import F, close, general, model, step_args  # noqa: F401


@pytest.mark.gpu
@pytest.mark.parametrize("stages", ["vertex", "chi0", "sigma", "chi0,sigma", "chi0,vertex,sigma"])
def test_fp32_stage_lists_at_the_plane_limit(F, monkeypatch, stages):  # noqa: F811
    m = model(1, 128, 128, 1, 8)
    monkeypatch.setenv("PYRPA_GB_FP32_STAGES", stages)
    F.set_precision(32)
    try:
        run = lambda: F.mkself(*step_args(m), scf_loop=1, eps=0.0, pp=0.5, sw_rescale=True)  # noqa: E731
        sg, mu = run()
        gsg, gmu = general(run)
    finally:
        F.set_precision(64)
    close(sg, gsg, 1e-4, 1e-6 * np.abs(gsg).max())
    assert abs(mu - gmu) <= 1e-4
