"""The even-model form of the convolutions and vertices (csrc/even.cuh).

Models with H(k) = H(k)^T on every k point run chi0, Sigma, the RPA vertices and
the Eliashberg kernel on half the mesh, with half-length time transforms and real
vertex matrices.  Each case here is run in that form and with PYRPA_GB_EVEN=0 (the
general form), and the small ones against the FP64 oracle, on meshes that take each
kernel: sides 16, 32 and 64 (compile-time stages), other, odd and unequal sides,
radices 7, 11 and 13, three dimensions, odd frequency counts, one to five orbitals.

Tolerances are those of the other parity tests: 1e-9 of the maximum plus 2e-9 in
FP64 and double-float (the reference zeroes parts below 1e-9), 2e-5 for chi0 and
1e-4 for Sigma in FP32.
"""
import os

import numpy as np
import pytest

from oracle import api as O
import _models as M

RTOL64, ATOL64 = 1e-9, 2e-9

# Norb, Nx, Ny, Nz, Nw
MESHES = [(1, 16, 16, 1, 32), (2, 32, 32, 1, 24), (3, 8, 8, 1, 30), (2, 5, 7, 1, 9), (2, 12, 10, 1, 16),
          (1, 14, 22, 1, 13), (2, 13, 13, 1, 8), (1, 64, 64, 1, 8), (2, 6, 6, 6, 12), (1, 7, 5, 3, 6),
          (2, 4, 4, 4, 64), (4, 4, 4, 1, 8), (5, 4, 6, 1, 10), (1, 2, 2, 1, 128)]


@pytest.fixture(scope="module")
def F():
    from pyrpa_gb300 import build, flibs
    if not build.LIB.exists():
        build.build()
    flibs.load_library()
    flibs.set_verbose(0)
    flibs.set_precision(64)
    return flibs


def model(Norb, Nx, Ny, Nz, Nw, temp=0.1, seed=3, complex_hop=False):
    from pyrpa_gb300 import models
    dim = 3 if Nz > 1 else 2
    rvec, ham_r = M.random_hoppings(Norb, seed, bandwidth=4.0 if dim == 2 else None, dim=dim, complex_hop=complex_hop)
    klist, kmap, invk = O.gen_irr_k_TRS(Nx, Ny, Nz)
    hamk = O.gen_ham(klist, ham_r, rvec)
    eig, uni = O.get_eig(hamk)
    olist, site = O.get_chi_orb_list(Norb)
    olist = np.asfortranarray(olist)
    S, C = O.gen_SCmatrix(olist, site, 0.4, 0.4 / 6 if Norb > 1 else 0.0)
    fill = 0.45 * Norb
    mu = models.bare_mu(eig, O.gen_kpoint_weight(invk, len(klist)), fill, temp)
    return dict(mesh=(Nx, Ny, Nz), Nw=Nw, temp=temp, fill=fill, mu=mu, klist=klist, kmap=kmap, invk=invk, hamk=hamk,
                eig=eig, uni=uni, olist=olist, S=S, C=C, Norb=Norb)


def close(a, b, rtol=RTOL64, atol=ATOL64):
    a, b = np.asarray(a), np.asarray(b)
    assert a.shape == b.shape
    err, scale = np.abs(a - b).max(), max(np.abs(b).max(), 1e-300)
    assert err <= rtol * scale + atol, f"max |diff| {err:.3e} at scale {scale:.3e}"


def general(fn):
    os.environ["PYRPA_GB_EVEN"] = "0"
    try:
        return fn()
    finally:
        del os.environ["PYRPA_GB_EVEN"]


def step_args(m):
    return (m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"], m["uni"], m["mu"], m["fill"],
            m["temp"], m["Nw"], *m["mesh"], False, False)


def dressed(m):
    """G with a frequency-dependent self-energy, symmetric in its orbitals."""
    No, Nk = m["Norb"], len(m["hamk"])
    w = (2 * np.arange(m["Nw"]) + 1) * np.pi * m["temp"]
    sig = np.zeros((No, No, m["Nw"], Nk), dtype=np.complex128)
    for a in range(No):
        sig[a, a] = (0.2 * (1 + 0.3 * a) / (1j * (w + 0.5)))[:, None] * (1 + 0.1 * np.cos(2 * np.pi * m["klist"][:, 0]))
    return O.gen_green(sig, m["hamk"], m["mu"], m["temp"])


@pytest.mark.gpu
@pytest.mark.parametrize("dims", MESHES + [(2, 16, 16, 1, 64), (1, 64, 64, 1, 64), (3, 12, 10, 1, 40), (2, 6, 6, 6, 80)])
@pytest.mark.parametrize("tail,bits", [(False, 64), (True, 64), (True, 48)])
def test_chi0_matches_oracle_and_general_form(F, dims, tail, bits):
    """get_chi0 takes the even form from 2^19 mesh points times pair elements on (the
    last four meshes); the FP64 tail-corrected entry keeps the general form, the
    double-float one does not."""
    m = model(*dims)
    G = dressed(m)
    if tail:
        args = (m["S"], m["C"], G, m["eig"], m["uni"], m["olist"], m["kmap"], m["invk"], m["mu"], m["temp"], *m["mesh"])
        run, ref = F.get_chi0_tail, O.get_chi0_tail
    else:
        args = (m["S"], m["C"], G, m["olist"], m["kmap"], m["invk"], m["temp"], *m["mesh"])
        run, ref = F.get_chi0, O.get_chi0
    F.set_precision(bits)
    try:
        chi, st = run(*args)
        gchi, gst = general(lambda: run(*args))
    finally:
        F.set_precision(64)
    close(chi, gchi)
    assert abs(st - gst) <= 1e-9
    if chi.size * np.prod(m["mesh"]) < 4e7:
        ochi, ost = ref(*args)
        close(chi, ochi)
        assert abs(st - ost) <= 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("dims", MESHES)
@pytest.mark.parametrize("bits,rtol", [(64, RTOL64), (48, RTOL64), (32, 1e-4)])
def test_flex_iterations_match_general_form(F, dims, bits, rtol):
    m = model(*dims)
    F.set_precision(bits)
    try:
        run = lambda: F.mkself(*step_args(m), scf_loop=2, eps=0.0, pp=0.5, sw_rescale=True, sw_tail=True)  # noqa: E731
        sg, mu = run()
        gsg, gmu = general(run)
    finally:
        F.set_precision(64)
    # two iterations with a chemical potential search between them
    close(sg, gsg, rtol, max(ATOL64, 1e-2 * rtol * np.abs(gsg).max()))
    assert abs(mu - gmu) <= max(1e-7, rtol)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(1, 16, 16, 1, 32), (2, 8, 8, 1, 16), (3, 4, 4, 1, 12), (2, 5, 7, 1, 9), (2, 4, 4, 4, 8)])
def test_mkself_converges_with_oracle(F, dims):
    m = model(*dims)
    kw = dict(eps=1e-6, pp=0.5, sw_rescale=True, sw_tail=True)
    sg, mu = F.mkself(*step_args(m), **kw)
    osg, omu = O.mkself(*step_args(m), **kw)
    assert abs(mu - omu) < 1e-7
    close(sg, osg, 1e-6, 1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(1, 16, 16, 1, 32), (2, 32, 32, 1, 24), (3, 8, 8, 1, 30), (2, 5, 7, 1, 9),
                                  (2, 6, 6, 6, 12), (5, 4, 6, 1, 10)])
@pytest.mark.parametrize("gap_sym", [0, 1])
@pytest.mark.parametrize("bits,rtol", [(64, RTOL64), (3264, 1e-4)])
def test_fused_operator_matches_general_form(F, dims, gap_sym, bits, rtol):
    """One FLEX iteration, then one application of the Eliashberg operator to the
    initial gap (the power method stopped after one step) in the fused call: V_Delta,
    the anomalous function's transforms and the contraction.  The eigenvalue itself
    is not compared, its Krylov space amplifies rounding on weakly paired models."""
    m = model(*dims)
    init = F.get_initial_gap(m["klist"], m["Norb"], gap_sym) + 0.1
    F.set_precision(bits)
    try:
        run = lambda: F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"],  # noqa: E731
                                    m["uni"], init, np.ones(m["Norb"]), m["mu"], m["fill"], m["temp"], m["Nw"],
                                    *m["mesh"], gap_sym, scf_loop=1, eps=1e-12, sw_tail=True, arnoldi_m=0, itemax=1)
        r, g = run(), general(run)
    finally:
        F.set_precision(64)
    close(r["gap"], g["gap"], rtol, max(ATOL64, 1e-2 * rtol * np.abs(g["gap"]).max()))
    assert abs(r["stoner"] - g["stoner"]) <= max(1e-9, rtol)


@pytest.mark.gpu
def test_fp64_pairing_input_keeps_its_bits(F):
    """The FP64 tail-corrected chi0 and lin_eliash take the general form for every
    model: the same bits as with the even form switched off."""
    m = model(2, 32, 32, 1, 64)
    G = dressed(m)
    init = F.get_initial_gap(m["klist"], 2, 0)

    def run():
        chi, st = F.get_chi0_tail(m["S"], m["C"], G, m["eig"], m["uni"], m["olist"], m["kmap"], m["invk"], m["mu"],
                                  m["temp"], *m["mesh"])
        v = chi.copy()
        gap, lam = F.linearized_eliashberg(v, G, m["uni"], init, m["S"], m["C"], m["olist"], np.ones(2), m["kmap"],
                                           m["invk"], *m["mesh"], m["temp"], 0, arnoldi_m=20)
        return chi, v, gap, lam

    for a, b in zip(run(), general(run)):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_broken_symmetry_keeps_the_general_form(F):
    """A G or a Sigma seed without the symmetry, and complex hoppings: the same
    results as with the even form switched off, bit for bit."""
    m = model(2, 32, 32, 1, 24)
    G = dressed(m).copy()
    G[0, 1] *= 1.0 + 1e-6
    args = (m["S"], m["C"], G, m["olist"], m["kmap"], m["invk"], m["temp"], *m["mesh"])
    assert np.array_equal(F.get_chi0(*args)[0], general(lambda: F.get_chi0(*args)[0]))
    mc = model(2, 8, 8, 1, 16, complex_hop=True)
    run = lambda: F.mkself(*step_args(mc), scf_loop=2, eps=0.0, pp=0.5, sw_rescale=True)[0]  # noqa: E731
    assert np.array_equal(run(), general(run))
    seed = F.mkself(*step_args(m), scf_loop=1, eps=0.0, pp=0.5, sw_rescale=True)[0]
    seed[0, 1] *= 1.0 + 1e-6
    init = F.get_initial_gap(m["klist"], 2, 0)
    fused = lambda: F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"],  # noqa: E731
                                  m["uni"], init, np.ones(2), m["mu"], m["fill"], m["temp"], m["Nw"], *m["mesh"], 0,
                                  scf_loop=2, eps=1e-12, arnoldi_m=0, itemax=1, sigma_seed=seed, seed_mu=m["mu"],
                                  seed_mu_old=m["mu"])["sigmak"]
    assert np.array_equal(fused(), general(fused))


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3, 8, 8, 1, 30), (4, 4, 4, 1, 8), (5, 4, 6, 1, 10)])
@pytest.mark.parametrize("size", [0.05, 8.0])
@pytest.mark.parametrize("gap_sym", [0, -1])
def test_pairing_vertex_of_any_matrix(F, dims, size, gap_sym):
    """V_Delta of random matrices with an even model's relations in double-float (the
    pivoted real-basis kernel), far below the instability and far above it.  The
    general form carries 1e-14 too; the worst of some thousand random matrices has a
    condition number of about 1e5, which leaves 1e-8 of the largest element.
    """
    m = model(*dims)
    No, Nk, n = m["Norb"], len(m["hamk"]), m["Norb"] ** 2
    rng = np.random.default_rng(No)
    o = np.asarray(m["olist"])
    at = {(a, b): i for i, (a, b) in enumerate(zip(o[:, 0], o[:, 1]))}
    P = [at[(b, a)] for a, b in zip(o[:, 0], o[:, 1])]
    chi = rng.normal(size=(n, n, m["Nw"], Nk)) + 1j * rng.normal(size=(n, n, m["Nw"], Nk))
    chi[:, :, 0] = chi[:, :, 0].real
    chi = chi + chi.transpose(1, 0, 2, 3)
    chi = np.ascontiguousarray(size * (chi + chi[P][:, P].conj()))
    init = F.get_initial_gap(m["klist"], No, 0) + 0.1
    G = dressed(m)

    def run():
        v = chi.copy()
        F.linearized_eliashberg(v, G, m["uni"], init, m["S"], m["C"], m["olist"], np.ones(No), m["kmap"], m["invk"],
                                *m["mesh"], m["temp"], gap_sym, arnoldi_m=0, itemax=1)
        return v

    F.set_precision(48)
    try:
        v, g = run(), general(run)
    finally:
        F.set_precision(64)
    close(v, g, 1e-8, 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3, 8, 8, 1, 30), (4, 4, 4, 1, 8), (5, 4, 6, 1, 10)])
@pytest.mark.parametrize("factor", [0.5, 3.0, 6.0, 20.0])
def test_fp64_vertex_beyond_the_instability(F, dims, factor):
    """One FP64 iteration without the rescaling, at interactions below and above the
    instability, where S^-1 - chi0 is indefinite and k_vertex_sym may leave matrices to
    the pivoted kernel.  Condition numbers of 1e4 leave 1e-12; the bound is that of the
    other FP64 tests."""
    m = model(*dims)
    m["S"], m["C"] = factor * m["S"], factor * m["C"]
    run = lambda: F.mkself(*step_args(m), scf_loop=1, eps=0.0, pp=0.5, sw_rescale=False, sw_tail=True)[0]  # noqa: E731
    close(run(), general(run))
