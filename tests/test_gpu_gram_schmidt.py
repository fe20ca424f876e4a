"""The device-resident orthogonalization of the Arnoldi pass (k_gs_step).

The Hessenberg matrix and the basis of a pass follow the oracle's modified
Gram-Schmidt: lambda of passes of one to six steps (the smallest and odd basis
sizes), on vectors shorter than one launch's threads, of a length that is no
multiple of them, and longer than one pass over the grid.  A pass amplifies
rounding, so the tolerance is the oracle's own: a hundred times the largest change
of its lambda when G moves by 1e-14 (three directions), and 1e-12.
"""
import numpy as np
import pytest

from oracle import api as O
import _models as M


@pytest.fixture(scope="module")
def F():
    from pyrpa_gb300 import build, flibs
    if not build.LIB.exists():
        build.build()
    flibs.load_library()
    flibs.set_verbose(0)
    flibs.set_precision(64)
    return flibs


@pytest.mark.gpu
@pytest.mark.parametrize("Norb,Nx,Ny,Nw", [(1, 4, 4, 4), (2, 6, 5, 7), (1, 32, 32, 600)])
@pytest.mark.parametrize("m", [1, 2, 3, 6])
def test_lambda_of_short_passes_matches_oracle(F, Norb, Nx, Ny, Nw, m):
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
    _, lam = F.linearized_eliashberg(chi.copy(), G, *args, arnoldi_m=m)
    _, olam = O.linearized_eliashberg(chi.copy(), G, *args, arnoldi_m=m)
    rng, moved = np.random.default_rng(5), 0.0
    for _ in range(3):
        moved = max(moved, abs(O.linearized_eliashberg(chi.copy(), G * (1 + 1e-14 * rng.normal(size=G.shape)), *args,
                                                       arnoldi_m=m)[1] - olam))
    assert abs(lam - olam) <= 100 * moved + 1e-12
