"""The chemical-potential search (csrc/mu.cu) against the oracle's.

One FLEX iteration from G0 and the search on its Sigma, on meshes where the search
kernel's point groups and grid can go wrong: fewer points than one block, a count
that is no multiple of the grouped points, more blocks than one, and few Matsubara
frequencies (the digamma tail's recursion below its asymptotic range).  One to
eight orbitals; above five with two sites, whose pair lists stay within the
engine's 32 pairs.  Tolerances of the FLEX parity tests: mu to 1e-8, Sigma to 1e-9.
"""
import numpy as np
import pytest

from oracle import api as O
import _models as M

CASES = [(1, (1,), 4, 4, 1, 3), (1, (1,), 16, 16, 1, 64), (1, (1,), 32, 32, 1, 700), (2, (2,), 5, 5, 1, 13),
         (3, (3,), 8, 8, 1, 20), (4, (4,), 4, 4, 1, 9), (5, (5,), 4, 4, 1, 11), (6, (3, 3), 4, 4, 1, 8),
         (7, (4, 3), 4, 4, 1, 5), (8, (4, 4), 4, 4, 1, 16), (2, (2,), 2, 2, 1, 1)]


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
@pytest.mark.parametrize("Norb,prof,Nx,Ny,Nz,Nw", CASES)
@pytest.mark.parametrize("complex_hop", [False, True])
def test_mu_search_matches_oracle(F, Norb, prof, Nx, Ny, Nz, Nw, complex_hop):
    from pyrpa_gb300 import flibs, models
    temp, fill = 0.1, 0.37 * Norb
    rvec, ham_r = M.random_hoppings(Norb, 7, bandwidth=4.0, complex_hop=complex_hop)
    klist, kmap, invk = O.gen_irr_k_TRS(Nx, Ny, Nz)
    hamk = O.gen_ham(klist, ham_r, rvec)
    eig, uni = O.get_eig(hamk)
    olist, site = flibs.get_chi_orb_list(Norb, prof)
    S, C = O.gen_SCmatrix(olist, site, 0.4, 0.06)
    mu = models.bare_mu(eig, O.gen_kpoint_weight(invk, len(klist)), fill, temp)
    args = (S, C, kmap, invk, olist, hamk, eig, uni, mu, fill, temp, Nw, Nx, Ny, Nz, False, False)
    kw = dict(scf_loop=2, eps=0.0, pp=0.5, sw_rescale=True)
    sg, m = F.mkself(*args, **kw)
    osg, om = O.mkself(*args, **kw)
    assert abs(m - om) <= 1e-8
    assert np.abs(sg - osg).max() <= 1e-9 * np.abs(osg).max() + 2e-9
