"""Which form a call takes, and the even form with several sites.

The other tests compare a call with the same call under PYRPA_GB_EVEN=0, which says
nothing if both are the general form.  The two forms launch different numbers of
kernels, so the counts of the second call of each say whether the even form ran.
Tolerances are those of the other parity tests.
"""
import numpy as np
import pytest

from oracle import api as O
from test_gpu_even import F, close, dressed, general, model, step_args  # noqa: F401


def sites(prof, Nx, Ny, Nz, Nw):
    """model() with the pair list of several sites"""
    m = model(sum(prof), Nx, Ny, Nz, Nw)
    if len(prof) > 1:
        from pyrpa_gb300 import flibs
        m["olist"], site = flibs.get_chi_orb_list(sum(prof), prof)
        m["S"], m["C"] = O.gen_SCmatrix(m["olist"], site, 0.4, 0.4 / 6)
    return m


def counted(F, fn):  # noqa: F811
    """The result and launches of the second call: plans and tables exist by then."""
    fn()
    n = F.kernel_launches()
    r = fn()
    return r, F.kernel_launches() - n


def takes_even_form(F, fn):  # noqa: F811
    return counted(F, fn)[1] != general(lambda: counted(F, fn))[1]


def calls(F, m, G):  # noqa: F811
    """name -> (call, precisions in which an even model takes the even form, and in which not)"""
    init = F.get_initial_gap(m["klist"], m["Norb"], 0) + 0.1
    chi0 = (m["S"], m["C"], G, m["olist"], m["kmap"], m["invk"], m["temp"], *m["mesh"])
    tail = (m["S"], m["C"], G, m["eig"], m["uni"], m["olist"], m["kmap"], m["invk"], m["mu"], m["temp"], *m["mesh"])
    # the entry asks for a chi with an even model's relations to 1e-12, which the zeroing of
    # small parts can break in the general form's
    F.set_precision(48)
    chi = F.get_chi0_tail(*tail)[0]
    F.set_precision(64)

    def lin():
        F.linearized_eliashberg(chi.copy(), G, m["uni"], init, m["S"], m["C"], m["olist"], np.ones(m["Norb"]),
                                m["kmap"], m["invk"], *m["mesh"], m["temp"], 0, arnoldi_m=0, itemax=1)

    return {
        "chi0": (lambda: F.get_chi0(*chi0), (64,), ()),
        "chi0_tail": (lambda: F.get_chi0_tail(*tail), (48,), (64, 32)),
        "mkself": (lambda: F.mkself(*step_args(m), scf_loop=1, eps=0.0, pp=0.5, sw_rescale=True), (64, 48, 32, 3264), ()),
        "flex_eliash": (lambda: F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"],
                                              m["uni"], init, np.ones(m["Norb"]), m["mu"], m["fill"], m["temp"],
                                              m["Nw"], *m["mesh"], 0, scf_loop=1, eps=1e-12, arnoldi_m=0, itemax=1),
                        (64, 3264), ()),
        "lin_eliash": (lin, (32, 3264), (64, 48)),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["chi0", "chi0_tail", "mkself", "flex_eliash", "lin_eliash"])
@pytest.mark.parametrize("symmetric", [True, False])
def test_form_of_each_call(F, name, symmetric):  # noqa: F811
    m = model(2, 32, 32, 1, 64, complex_hop=not symmetric)
    G = dressed(m)
    fn, even, gen = calls(F, m, G)[name]
    try:
        for bits in even + gen:
            F.set_precision(bits)
            assert takes_even_form(F, fn) == (symmetric and bits in even), bits
    finally:
        F.set_precision(64)


@pytest.mark.gpu
@pytest.mark.parametrize("prof,dims", [((2, 2), (8, 8, 1, 64)), ((4, 3), (8, 8, 1, 8)), ((4, 4), (8, 8, 1, 4)),
                                       ((2, 1), (5, 7, 1, 90)), ((2, 2, 1), (4, 4, 4, 8)), ((1, 1), (16, 16, 1, 512))])
@pytest.mark.parametrize("bits,rtol", [(64, 1e-9), (48, 1e-9), (32, 1e-4)])
def test_sites_match_general_form(F, prof, dims, bits, rtol):  # noqa: F811
    """Two FLEX iterations, and one application of the Eliashberg operator (in the
    arithmetics of the fused call)."""
    m = sites(prof, *dims)
    init = F.get_initial_gap(m["klist"], m["Norb"], 0) + 0.1
    F.set_precision(bits)
    try:
        run = lambda: F.mkself(*step_args(m), scf_loop=2, eps=0.0, pp=0.5, sw_rescale=True, sw_tail=True)  # noqa: E731
        ((sg, mu), n), ((gsg, gmu), gn) = counted(F, run), general(lambda: counted(F, run))
        assert n != gn
        close(sg, gsg, rtol, max(2e-9, 1e-2 * rtol * np.abs(gsg).max()))
        assert abs(mu - gmu) <= max(1e-7, rtol)
        F.set_precision(3264 if bits == 32 else 64)
        if bits == 32 and len(m["olist"]) not in (1, 4, 9, 16, 25):
            return  # the mixed call's double-float vertex takes these counts alone
        op = lambda: F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"],  # noqa: E731
                                   m["uni"], init, np.ones(m["Norb"]), m["mu"], m["fill"], m["temp"], m["Nw"],
                                   *m["mesh"], 0, scf_loop=1, eps=1e-12, sw_tail=True, arnoldi_m=0, itemax=1)
        r, g = op(), general(op)
        close(r["gap"], g["gap"], rtol, max(2e-9, 1e-2 * rtol * np.abs(g["gap"]).max()))
    finally:
        F.set_precision(64)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3, 8, 8, 1, 30), (4, 4, 4, 1, 8), (5, 4, 6, 1, 10)])
def test_swept_vertex_leaves_indefinite_matrices(F, dims):  # noqa: F811
    """Below the instability every FP64 vertex is swept; beyond it a few indefinite matrices
    go to the inverse with row pivots (a NumPy model of the sweep finds one or two of 1020,
    80 and 140 at some of these factors), and the results are still those of the general
    form.  Condition numbers up to 1e5 leave 1e-8 of the largest element."""
    m = model(*dims)
    S, C = m["S"], m["C"]
    run = lambda: F.mkself(*step_args(m), scf_loop=1, eps=0.0, pp=0.5, sw_rescale=False)[0]  # noqa: E731
    left = {}
    for factor in (0.5, 1.0, 6.0, 8.0, 10.0, 12.0, 15.0, 30.0):
        m["S"], m["C"] = factor * S, factor * C
        n = F.pivoted_vertices()
        sg = run()
        left[factor] = F.pivoted_vertices() - n
        close(sg, general(run), 1e-8)
    assert left[0.5] == left[1.0] == 0 and sum(left.values()) > 0, left


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3, 8, 8, 1, 30), (4, 4, 4, 1, 8), (5, 4, 6, 1, 10)])
@pytest.mark.parametrize("size", [0.05, 8.0])
@pytest.mark.parametrize("gap_sym", [0, -1])
def test_fp32_pairing_vertex_of_any_matrix(F, dims, size, gap_sym):  # noqa: F811
    """V_Delta of random matrices with an even model's relations through lin_eliash in 32
    bits (the pivoted real-basis kernel for a singlet, the general one for a triplet), far
    below the instability and far above it, against the FP64 general form.  An elimination of n rows in arithmetic of rounding eps
    leaves some n eps kappa of an inverse's largest element; 4 n eps kappa is allowed."""
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

    ref = run()
    F.set_precision(32)
    try:
        v = run()
        assert takes_even_form(F, run) == (gap_sym >= 0)
    finally:
        F.set_precision(64)
    X = chi.transpose(2, 3, 1, 0).reshape(-1, n, n)
    allowed = 0.0
    for c, U, sign in ((1.5 if gap_sym >= 0 else 0.5, m["S"], -1), (0.5, m["C"], 1)):
        A = np.linalg.inv(U.T)[None] + sign * X
        inv = np.linalg.inv(A)
        allowed = allowed + c * np.linalg.cond(A, 1) * np.abs(inv).max(axis=(1, 2))
    err = np.abs(v - ref).transpose(2, 3, 1, 0).reshape(-1, n * n).max(axis=1)
    allowed = 4 * n * 2.0 ** -24 * (allowed + np.abs(m["S"]).max() + np.abs(m["C"]).max())
    assert (err <= allowed).all(), (err / allowed).max()


@pytest.mark.gpu
@pytest.mark.parametrize("dims,bits,tail,even", [
    ((1, 32, 32, 1, 250), 64, False, False), ((1, 32, 32, 1, 256), 64, False, True),
    ((1, 64, 64, 1, 64), 64, False, False), ((1, 64, 64, 1, 250), 64, False, True),
    ((2, 16, 16, 1, 64), 64, False, True),
    ((1, 32, 32, 1, 512), 48, False, False), ((1, 32, 32, 1, 800), 48, False, True),
    ((1, 64, 64, 1, 64), 48, True, False), ((1, 32, 32, 1, 256), 48, True, True),
    ((2, 16, 16, 1, 64), 48, False, True),
    ((1, 32, 32, 1, 1024), 32, False, False), ((1, 32, 32, 1, 2048), 32, False, True),
    ((3, 16, 16, 1, 100), 32, False, False), ((3, 16, 16, 1, 144), 32, False, True),
    ((2, 32, 32, 1, 64), 32, True, False), ((1, 32, 32, 1, 1024), 32, True, True),
    ((4, 8, 8, 1, 15), 32, False, False), ((4, 8, 8, 1, 16), 32, False, True),
    ((2, 64, 64, 1, 32), 32, False, False), ((5, 32, 32, 1, 2), 32, False, True)])
def test_size_from_which_chi0_takes_the_even_form(F, dims, bits, tail, even):  # noqa: F811
    """The even form where it is the faster one (csrc/abi.cu, even_chi0_pays)."""
    m = model(*dims)
    G = dressed(m)
    if tail:
        run = lambda: F.get_chi0_tail(m["S"], m["C"], G, m["eig"], m["uni"], m["olist"], m["kmap"],  # noqa: E731
                                      m["invk"], m["mu"], m["temp"], *m["mesh"])
    else:
        run = lambda: F.get_chi0(m["S"], m["C"], G, m["olist"], m["kmap"], m["invk"], m["temp"], *m["mesh"])  # noqa: E731
    F.set_precision(bits)
    try:
        assert takes_even_form(F, run) == even
        (chi, st), (gchi, gst) = run(), general(run)
    finally:
        F.set_precision(64)
    tol = 2e-5 if bits == 32 else 1e-9
    close(chi, gchi, tol, 2e-9)
    assert abs(st - gst) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(1, 16, 16, 1, 32), (2, 32, 32, 1, 24), (3, 8, 8, 1, 30), (5, 4, 6, 1, 10)])
@pytest.mark.parametrize("bits,rtol", [(64, 1e-9), (3264, 1e-4)])
def test_fused_triplet_matches_general_form(F, dims, bits, rtol):  # noqa: F811
    """One application of the triplet operator in the fused call: the real-basis vertex with
    every element written, and the general form of the rest."""
    m = model(*dims)
    init = F.get_initial_gap(m["klist"], m["Norb"], 0) + 0.1
    F.set_precision(bits)
    try:
        run = lambda: F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"],  # noqa: E731
                                    m["uni"], init, np.ones(m["Norb"]), m["mu"], m["fill"], m["temp"], m["Nw"],
                                    *m["mesh"], -1, scf_loop=1, eps=1e-12, sw_tail=True, arnoldi_m=0, itemax=1)
        r, g = run(), general(run)
    finally:
        F.set_precision(64)
    close(r["gap"], g["gap"], rtol, max(2e-9, 1e-2 * rtol * np.abs(g["gap"]).max()))
