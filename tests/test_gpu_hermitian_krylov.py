"""The Arnoldi pass on Hermitian vectors (k_gs_herm, k_scal_herm; double-float and
FP32 operators).

lambda of short passes against the oracle's complex modified Gram-Schmidt in FP64,
for each number of orbitals with a kernel of its own that the oracle does quickly,
vectors shorter than a block, of a length that is no multiple of one, and longer
than one pass over the grid, and a model without the inversion symmetry.  A pass
amplifies the operator's rounding, so the tolerance is the oracle's own: a hundred
times the largest change of its lambda when G moves by the type's rounding (1e-13
and 1e-6, three directions), and that rounding times a hundred.
"""
import numpy as np
import pytest

from oracle import api as O
import _models as M


@pytest.fixture()
def F():
    from pyrpa_gb300 import build, flibs
    if not build.LIB.exists():
        build.build()
    flibs.load_library()
    flibs.set_verbose(0)
    yield flibs
    flibs.set_precision(64)


@pytest.mark.gpu
@pytest.mark.parametrize("bits,unit", [(48, 1e-13), (32, 1e-6)])
@pytest.mark.parametrize("Norb,Nx,Ny,Nw", [(1, 4, 4, 4), (2, 6, 5, 7), (3, 4, 4, 6), (5, 4, 3, 5), (1, 32, 32, 600)])
@pytest.mark.parametrize("m", [1, 2, 5])
def test_lambda_of_short_passes_matches_oracle(F, bits, unit, Norb, Nx, Ny, Nw, m):
    temp = 0.08
    rvec, ham_r = M.random_hoppings(Norb, 11, bandwidth=4.0)
    klist, kmap, invk = O.gen_irr_k_TRS(Nx, Ny, 1)
    hamk = O.gen_ham(klist, ham_r, rvec)
    eig, uni = O.get_eig(hamk)
    olist, site = O.get_chi_orb_list(Norb)
    olist = np.asfortranarray(olist)
    S, C = O.gen_SCmatrix(olist, site, 0.8, 0.1 if Norb > 1 else 0.0)
    G = O.gen_Green0(eig, uni, 0.1, temp, Nw)
    chi, _ = O.get_chi0(S, C, G, olist, kmap, invk, temp, Nx, Ny, 1)
    init = O.get_initial_gap(klist, Norb, 0) + 0.2
    args = (uni, init, S, C, olist, np.ones(Norb), kmap, invk, Nx, Ny, 1, temp, 0)
    _, olam = O.linearized_eliashberg(chi.copy(), G, *args, arnoldi_m=m)
    rng, moved = np.random.default_rng(5), 0.0
    for _ in range(3):
        moved = max(moved, abs(O.linearized_eliashberg(chi.copy(), G * (1 + unit * rng.normal(size=G.shape)), *args,
                                                       arnoldi_m=m)[1] - olam))
    F.set_precision(bits)
    delta, lam = F.linearized_eliashberg(chi.copy(), G, *args, arnoldi_m=m)
    assert abs(lam - olam) <= 100 * (moved + unit)
    # the gap (Norb, Norb, Nw, Nk) is a Hermitian matrix at every point
    assert np.abs(delta - np.conj(np.swapaxes(delta, 0, 1))).max() <= 1e-14 * np.abs(delta).max()
