"""Charge vertices that are singular in 32 bits and not in 64 (csrc/even_impl.cuh,
inverse_as): J next to U / 5, where an eigenvalue 5 J - U of C vanishes.  FP32 cannot
resolve such a matrix (its condition number is above 1e8), but the call is accepted and
returns numbers, as the general form does."""
import numpy as np
import pytest

from oracle import api as O
from test_gpu_even import F, general, model, step_args  # noqa: F401


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(2, 8, 8, 1, 16), (3, 8, 8, 1, 16), (5, 4, 4, 1, 8)])
def test_nearly_singular_charge_vertex_in_32_bits(F, dims):  # noqa: F811
    m = model(*dims)
    olist, site = O.get_chi_orb_list(m["Norb"])
    m["S"], m["C"] = O.gen_SCmatrix(np.asfortranarray(olist), site, 0.4, 0.4 * (0.2 + 1e-9))
    assert 1e8 < np.linalg.cond(m["C"]) < 1e11
    F.set_precision(32)
    try:
        run = lambda: F.mkself(*step_args(m), scf_loop=1, eps=0.0, pp=0.5, sw_rescale=True)[0]  # noqa: E731
        sg, gsg = run(), general(run)
    finally:
        F.set_precision(64)
    assert np.isfinite(sg).all() and np.isfinite(gsg).all()
