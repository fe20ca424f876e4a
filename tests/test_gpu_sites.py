"""Even models with several sites (csrc/even.cuh): the pair lists of sites with up to
four and five orbitals, whose class tables are the largest of the engine (two
four-orbital sites: 32 pairs, 288 classes).

chi0, its Stoner factor and one FLEX iteration against the FP64 oracle, with printing
on and off.  Tolerances are those of the other parity tests: 1e-9 of the maximum plus
2e-9 in FP64, 2e-5 for the factor of an FP32 chi0.  A chi0 beyond the instability is
rescaled to a factor of 1 - 1e-4: its vertex amplifies the 1e-13 that two chi0 differ by
some 1e4 times, which leaves 1e-8 of the largest element of Sigma.
"""
import numpy as np
import pytest

from oracle import api as O
import _models as M

# site profile, Nx, Ny, Nw: from 2^19 mesh points times pair elements on, where get_chi0
# takes the even form
SITES = [((4, 4), 8, 8, 4), ((5, 2, 1), 8, 8, 6), ((4, 3), 8, 8, 8), ((2, 2), 8, 8, 64)]


@pytest.fixture(scope="module")
def F():
    from pyrpa_gb300 import build, flibs
    if not build.LIB.exists():
        build.build()
    flibs.load_library()
    flibs.set_verbose(0)
    flibs.set_precision(64)
    return flibs


def model(F, prof, Nx, Ny, Nw, factor=None, temp=0.1):
    """U chosen for a Stoner factor of chi0 from G0, when given."""
    from pyrpa_gb300 import models
    Norb = sum(prof)
    rvec, ham_r = M.random_hoppings(Norb, 11, bandwidth=4.0)
    klist, kmap, invk = O.gen_irr_k_TRS(Nx, Ny, 1)
    hamk = O.gen_ham(klist, ham_r, rvec)
    eig, uni = O.get_eig(hamk)
    olist, site = F.get_chi_orb_list(Norb, prof)
    S, C = O.gen_SCmatrix(olist, site, 0.4, 0.4 / 6)
    fill = 0.45 * Norb
    mu = models.bare_mu(eig, O.gen_kpoint_weight(invk, len(klist)), fill, temp)
    G = O.gen_Green0(eig, uni, mu, temp, Nw)
    chi, st = O.get_chi0(S, C, G, olist, kmap, invk, temp, Nx, Ny, 1)
    if factor:
        S, C, st = S * (factor / st), C * (factor / st), factor
    step = (S, C, kmap, invk, olist, hamk, eig, uni, mu, fill, temp, Nw, Nx, Ny, 1, False, False)
    return dict(S=S, C=C, G=G, chi=chi, stoner=st, step=step, olist=olist, kmap=kmap, invk=invk, temp=temp,
                mesh=(Nx, Ny, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("prof,Nx,Ny,Nw", SITES)
@pytest.mark.parametrize("verbose", [0, 1])
def test_stoner_factor_of_chi0(F, prof, Nx, Ny, Nw, verbose):
    m = model(F, prof, Nx, Ny, Nw)
    assert 2 * Nx * Ny * Nw * len(m["olist"]) ** 2 >= 2 ** 19
    F.set_verbose(verbose)
    try:
        chi, st = F.get_chi0(m["S"], m["C"], m["G"], m["olist"], m["kmap"], m["invk"], m["temp"], *m["mesh"])
    finally:
        F.set_verbose(0)
    assert abs(st - m["stoner"]) <= 1e-9
    assert np.abs(chi - m["chi"]).max() <= 1e-9 * np.abs(m["chi"]).max() + 2e-9


@pytest.mark.gpu
@pytest.mark.parametrize("prof,Nx,Ny,Nw", SITES)
@pytest.mark.parametrize("factor", [0.7, 1.02])
@pytest.mark.parametrize("verbose", [0, 1])
def test_flex_iteration_matches_oracle(F, prof, Nx, Ny, Nw, factor, verbose):
    """One iteration from G0, below the instability and just beyond it, where the factor
    decides on the rescaling."""
    m = model(F, prof, Nx, Ny, Nw, factor)
    kw = dict(scf_loop=1, eps=0.0, pp=0.5, sw_rescale=True)
    F.set_verbose(verbose)
    try:
        sg, mu = F.mkself(*m["step"], **kw)
    finally:
        F.set_verbose(0)
    assert abs(F.last_stats()["stoner"] - factor) <= 1e-9
    osg, omu = O.mkself(*m["step"], **kw)
    # a shift of Sigma shifts mu by no more
    assert abs(mu - omu) <= (1e-7 if factor < 1 else 1e-8 * np.abs(osg).max() + 1e-7)
    assert np.abs(sg - osg).max() <= (1e-9 if factor < 1 else 1e-8) * np.abs(osg).max() + 2e-9


@pytest.mark.gpu
@pytest.mark.parametrize("prof,Nx,Ny,Nw", SITES)
@pytest.mark.parametrize("bits,tol", [(48, 1e-9), (32, 2e-5)])
def test_stoner_factor_in_other_arithmetics(F, prof, Nx, Ny, Nw, bits, tol):
    m = model(F, prof, Nx, Ny, Nw, 0.7)
    F.set_precision(bits)
    try:
        F.mkself(*m["step"], scf_loop=1, eps=0.0, pp=0.5, sw_rescale=True)
    finally:
        F.set_precision(64)
    assert abs(F.last_stats()["stoner"] - 0.7) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("prof,Nx,Ny,Nw", SITES + [((5,), 8, 8, 8)])
@pytest.mark.parametrize("bits", [64, 32])
def test_results_do_not_depend_on_printing(F, prof, Nx, Ny, Nw, bits):
    """The factor of a chi0 beyond the instability scales chi0, so that another rounding of
    it would reach Sigma: the same bits with printing on and off."""
    m = model(F, prof, Nx, Ny, Nw, 1.2)
    out = []
    for verbose in (0, 1):
        F.set_precision(bits)
        F.set_verbose(verbose)
        try:
            st = F.get_chi0(m["S"], m["C"], m["G"], m["olist"], m["kmap"], m["invk"], m["temp"], *m["mesh"])[1]
            sg, mu = F.mkself(*m["step"], scf_loop=1, eps=0.0, pp=0.5, sw_rescale=True)
        finally:
            F.set_verbose(0)
            F.set_precision(64)
        out.append((st, F.last_stats()["stoner"], mu, sg))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
