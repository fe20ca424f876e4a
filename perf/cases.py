"""The calls that are timed, through the public entry points of ``pyrpa_gb300.flibs``.

A pyrpa calculation is a chain of library calls on host arrays: chi0 (plain or
with the analytic high-frequency tail), the FLEX self-energy loop, and the
linearized Eliashberg equation on its result.  Each case is one such call, or
the two that a program makes in a row, from the NumPy arrays that the program
has in hand to the NumPy arrays that it gets back.  ``kind``:

  chi0        get_chi0: the bubble of a given G and its Stoner factor
  chi0_tail   get_chi0_tail: the same with the tail correction
  step        mkself with scf_loop=1: one FLEX iteration from G0 (chi0, RPA
              vertices, Sigma, chemical potential), the unit that a run to
              convergence repeats, and the call that the parameter sweep probes
              U_Stoner with
  solve       mkself to a residual
  eliash      get_chi0_tail of a given G, then linearized_eliashberg
  fused       flex_eliash: FLEX to a residual from a coarse-mesh start, then
              the Eliashberg eigenvalue, in one device-resident call

``bits`` is the engine's precision (64, 48 double-float convolutions, 32, 3264
the mixed schedule).  Results of the bulk in 32 bits are kept as complex64, as
a program that asks for 32-bit bulk keeps them.  ``hop`` is the model family:
"sym" H(R) = H(-R) real (orbitals of one parity, the engine's own benchmark
models), "real" real H(R) without inversion (time reversal only), "cplx"
complex H(R) (Hermitian only).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pyrpa_gb300 import flibs as F
from pyrpa_gb300 import models

# fill is electrons per spin and orbital
_BASE = dict(hop="sym", Nz=1, fill=0.45, temp=0.03, tail=False)
# U in units of the bandwidth 4, by orbital count: Stoner factors of 0.7 to 0.8
_U = {1: 0.17, 2: 0.25, 3: 0.11, 4: 0.09, 5: 0.14}


def _case(name, kind, bits, Norb, Nx, Ny, Nw, **more):
    return dict(_BASE, name=name, kind=kind, bits=bits, Norb=Norb, Nx=Nx, Ny=Ny, Nw=Nw, **{"U": _U[Norb], **more})


def listed():
    return [
        # the smallest calls: one orbital on a coarse mesh, bound by latency and launches
        _case("chi0_1orb_16x16_w256", "chi0", 64, 1, 16, 16, 256),
        # the one-orbital square lattice at 32x32x1024, one iteration and to convergence
        _case("step_1orb_32x32_w1024", "step", 64, 1, 32, 32, 1024, temp=0.02),
        _case("solve_1orb_32x32_w1024", "solve", 64, 1, 32, 32, 1024, temp=0.02, eps=1e-6, tail=True),
        # an ordinary susceptibility calculation on a given G
        _case("chi0tail_2orb_32x32_w512", "chi0_tail", 64, 2, 32, 32, 512),
        # odd, ragged mesh and frequency count; time reversal without inversion
        _case("step_2orb_15x21_w300_real", "step", 64, 2, 15, 21, 300, hop="real"),
        # five d orbitals in the default FP64 arithmetic, what an unchanged main.py runs
        _case("step_5orb_32x32_w512", "step", 64, 5, 32, 32, 512),
        # five orbitals on the production mesh in 32-bit bulk: the largest call
        _case("step_5orb_64x64_w1024_fp32", "step", 32, 5, 64, 64, 1024, temp=0.02),
        # a cubic three-orbital lattice with double-float convolutions, radix-3 axes
        _case("step_3orb_12x12x12_w512_df", "step", 48, 3, 12, 12, 512, Nz=12, tail=True),
        # three orbitals without inversion in 32-bit bulk
        _case("step_3orb_32x32_w512_real_fp32", "step", 32, 3, 32, 32, 512, hop="real"),
        # one instance of a parameter sweep in the mixed schedule
        _case("solve_3orb_32x32_w512_mixed", "solve", 3264, 3, 32, 32, 512, eps=1e-4),
        # pairing on a given G: chi0 and the Eliashberg eigenvalue in FP64
        _case("eliash_2orb_32x32_w256", "eliash", 64, 2, 32, 32, 256),
        # the fast form of the headline calculation (five orbitals, warm start, Sigma and lambda)
        _case("fused_5orb_32x32_w256_mixed", "fused", 3264, 5, 32, 32, 256, eps=1e-4, tail=True,
              fill=0.6, U=0.3, temp=0.02),
    ]


def _size(c):
    return c["Nx"] * c["Ny"] * c["Nz"] * c["Nw"] * c["Norb"] ** 4


def _smooth(n):
    """The largest length not above n that the engine transforms (primes up to 13)."""
    while True:
        r = n
        for p in (2, 3, 5, 7, 11, 13):
            while r % p == 0:
                r //= p
        if r == 1:
            return n
        n -= 1


def draw(rng):
    """Another case of the same ranges: every kind, one to five orbitals,
    square, rectangular and cubic meshes with odd sides among them, 64 to 1024
    frequencies, each arithmetic; most models have H(R) = H(-R)."""
    while True:
        kind = rng.choice(["chi0", "chi0_tail", "step", "step", "step", "solve", "eliash", "fused"])
        bits = {"chi0": [64], "chi0_tail": [64, 48], "step": [64, 48, 32], "solve": [64, 3264], "eliash": [64],
                "fused": [3264]}[kind]
        c = dict(_BASE, kind=kind, bits=rng.choice(bits), Norb=rng.randint(1, 5),
                 Nw=_smooth(round(math.exp(rng.uniform(math.log(64), math.log(1024))))),
                 temp=round(rng.uniform(0.02, 0.05), 4), hop=rng.choice(["sym", "sym", "sym", "real", "cplx"]))
        c["U"] = round(_U[c["Norb"]] * rng.uniform(0.6, 1.0), 4)
        c["Nx"] = c["Ny"] = rng.choice([8, 12, 16, 24, 32, 32, 48, 64])
        if rng.random() < 0.3:
            c["Nx"], c["Ny"] = _smooth(rng.randint(7, 40)), _smooth(rng.randint(7, 40))
            if c["Nx"] % 2 > c["Ny"] % 2:  # the k list is defined for an even Nx with an odd Ny only
                c["Nx"], c["Ny"] = c["Ny"], c["Nx"]
        elif rng.random() < 0.2:
            c["Nx"] = c["Ny"] = c["Nz"] = rng.choice([6, 8, 10, 12, 16])
        if kind in ("step", "solve"):
            c["tail"] = rng.random() < 0.5
        if kind in ("solve", "fused"):
            c["hop"], c["eps"] = "sym", 1e-6 if c["bits"] == 64 else 1e-4
        if kind == "fused":  # the coarse start halves each side and the frequency count
            c["fill"], c["tail"] = 0.6, True
            for axis in ("Nx", "Ny", "Nw"):
                c[axis] = 2 * _smooth(c[axis] // 2)
        if kind == "eliash":
            c["hop"] = "sym"
        # no more work than the listed cases of the kind
        cap = {"chi0": 16 * 2 ** 19, "chi0_tail": 16 * 2 ** 19, "step": 625 * 2 ** (19 if c["bits"] == 64 else 21),
               "solve": 81 * 2 ** 19 if c["bits"] == 3264 else 2 ** 20, "eliash": 16 * 2 ** 18,
               "fused": 625 * 2 ** 18}[kind]
        if _size(c) <= cap:
            return c


# ------------------------------------------------------------------- inputs
def _hoppings(c, rng):
    """Seeded hoppings: the fixed model of this orbital count with every
    amplitude moved by a few per cent."""
    No, dim = c["Norb"], 3 if c["Nz"] > 1 else 2
    if No == 1 and dim == 2:
        rvec, ham = models.square_t_tprime(0.5, -0.125)
    else:
        shells = [(1, 0, 0), (1, 1, 0)] + ([(2, 0, 0)] if dim == 2 else [])
        rvec, ham = models.seeded_hoppings(No, 4, shells, dim=dim, bandwidth=4.0)
    index = {tuple(int(v) for v in r): i for i, r in enumerate(rvec)}
    ham = ham.copy()
    for r, i in index.items():
        j = index[tuple(-v for v in r)]
        if j < i:
            continue
        noise = rng.normal(0.0, 0.02, (No, No))
        move = 1.0 + 0.5 * (noise + noise.T)
        odd = np.zeros((No, No), dtype=np.complex128)
        if i != j and c["hop"] != "sym":  # an s-p like hybridization, odd in R
            a = rng.normal(0.0, 0.08, (No, No))
            odd = (a - a.T).astype(np.complex128)
        if i != j and c["hop"] == "cplx":
            a = rng.normal(0.0, 0.05, (No, No))
            odd = odd + 1j * (a + a.T)
        ham[i] = ham[i] * move + odd
        if j != i:
            ham[j] = ham[j] * move + np.conj(odd).T
    return rvec, ham


def prepare(case, seed):
    c = dict(case)
    rng = np.random.default_rng(seed)
    F.set_verbose(0)
    F.set_precision(64)
    No, mesh = c["Norb"], (c["Nx"], c["Ny"], c["Nz"])
    rvec, ham_r = _hoppings(c, rng)
    klist, kmap, invk = F.gen_irr_k_TRS(*mesh)
    hamk = F.gen_ham(klist, ham_r, rvec)
    eig, uni = F.get_eig(hamk)
    olist, site = F.get_chi_orb_list(No)
    U = 4.0 * c["U"]
    S, C = F.gen_SCmatrix(olist, site, U, U / 6.0 if No > 1 else 0.0)
    fill = c["fill"] * No * (1.0 + 0.02 * float(rng.uniform(-1.0, 1.0)))
    mu = models.bare_mu(eig, F.gen_kpoint_weight(invk, len(klist)), fill, c["temp"])
    s = dict(c=c, mesh=mesh, kmap=kmap, invk=invk, hamk=hamk, eig=eig, uni=uni, olist=olist, S=S, C=C, mu=mu,
             fill=fill, plist=np.ones(No), init=F.get_initial_gap(klist, No, 1 if No == 1 else 0))
    if c["kind"] in ("chi0", "chi0_tail", "eliash"):
        # G with a self-energy of Fermi-liquid form, as a converged run leaves it
        w = (2 * np.arange(c["Nw"]) + 1) * np.pi * c["temp"]
        sig = np.zeros((No, No, c["Nw"], len(klist)), dtype=np.complex128)
        for a in range(No):
            amp, gam = 0.15 * (1.0 + 0.2 * float(rng.uniform())), 0.6 + 0.2 * float(rng.uniform())
            sig[a, a] = (amp / (1j * (w + gam)))[:, None]
        s["G"] = F.gen_green(sig, hamk, mu, c["temp"])
    return s


def run(s):
    c = s["c"]
    F.set_precision(c["bits"])
    kind, mesh, temp = c["kind"], s["mesh"], c["temp"]
    if kind == "chi0":
        return F.get_chi0(s["S"], s["C"], s["G"], s["olist"], s["kmap"], s["invk"], temp, *mesh)
    if kind == "chi0_tail":
        return F.get_chi0_tail(s["S"], s["C"], s["G"], s["eig"], s["uni"], s["olist"], s["kmap"], s["invk"], s["mu"],
                               temp, *mesh)
    if kind in ("step", "solve"):
        loop = dict(scf_loop=1, eps=0.0) if kind == "step" else dict(scf_loop=300, eps=c["eps"])
        sigma, mu = F.mkself(s["S"], s["C"], s["kmap"], s["invk"], s["olist"], s["hamk"], s["eig"], s["uni"], s["mu"],
                             s["fill"], temp, c["Nw"], *mesh, False, False, pp=0.5, sw_rescale=True, sw_tail=c["tail"],
                             **loop)
        return _kept(sigma, c["bits"]), mu
    gap_sym = 1 if c["Norb"] == 1 else 0
    if kind == "eliash":
        F.set_arnoldi_tol(1e-8)
        chi, stoner = F.get_chi0_tail(s["S"], s["C"], s["G"], s["eig"], s["uni"], s["olist"], s["kmap"], s["invk"],
                                      s["mu"], temp, *mesh)
        gap, lam = F.linearized_eliashberg(chi, s["G"], s["uni"], s["init"], s["S"], s["C"], s["olist"], s["plist"],
                                           s["kmap"], s["invk"], *mesh, temp, gap_sym, arnoldi_m=20)
        return chi, stoner, gap, lam
    F.set_arnoldi_tol(1e-8)
    r = F.flex_eliash(s["S"], s["C"], s["kmap"], s["invk"], s["olist"], s["hamk"], s["eig"], s["uni"], s["init"],
                      s["plist"], s["mu"], s["fill"], temp, c["Nw"], *mesh, gap_sym, eps=c["eps"], pp=0.5,
                      sw_rescale=True, sw_tail=True, arnoldi_m=20, coarse=(2, 2))
    return _kept(r["sigmak"], c["bits"]), r["mu"], _kept(r["gap"], c["bits"]), r["lam"], r["stoner"]


def _kept(a, bits):
    """Results of 32-bit bulk arithmetic, stored in 32 bits."""
    return torch.from_numpy(a).to(torch.complex64) if bits in (32, 3264) else a


# --------------------------------------------------------------------- work
def work(case):
    """Each input and output array once; the operations of the transforms
    (5 n log2 n a complex transform of the padded grid, one per distinct
    element) and of the two inverses of each vertex matrix, of one iteration
    for a loop (its iteration count is the model's)."""
    c = case
    No, Nw, n = c["Norb"], c["Nw"], c["Nx"] * c["Ny"] * c["Nz"]
    Nk, Nchi = F.irr_k_count(c["Nx"], c["Ny"], c["Nz"]), No * No
    K, P = Nk * Nw, 2 * n * Nw
    el = 8 if c["bits"] in (32, 3264) else 16
    fft = 5.0 * P * math.log2(P)
    pairs = (No ** 4 + 3 * No * No) // 4
    model = 16 * Nk * No * No * 2 + 8 * Nk * No + 48 * n
    chi0_flops = fft * (pairs + No * No) + 8.0 * P * pairs
    if c["kind"] in ("chi0", "chi0_tail"):
        return {"bytes": float(model + 16 * K * (No * No + Nchi * Nchi)), "flops": chi0_flops}
    vertex = 16.0 * K * Nchi ** 3
    if c["kind"] == "eliash":
        return {"bytes": float(model + 16 * K * (2 * No * No + 2 * Nchi * Nchi)),
                "flops": chi0_flops + vertex + fft * pairs + 20 * (2 * fft * No * No + 8.0 * P * Nchi * Nchi)}
    step = chi0_flops + vertex + fft * (pairs + No * No) + 8.0 * P * Nchi * Nchi
    out = el * K * No * No
    if c["kind"] == "fused":
        return {"bytes": float(model + 2 * out), "flops": step + chi0_flops + vertex +
                20 * (2 * fft * No * No + 8.0 * P * Nchi * Nchi)}
    return {"bytes": float(model + out), "flops": step}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """chi0 and one FLEX iteration in plain 64-bit torch, written from the
    definitions; None for the loops, the eigenvalue problem and the sizes that
    would take long."""
    c = dict(case)
    if c["kind"] not in ("chi0", "step") or c["tail"] or _size(c) > 625 * 2 ** 19:
        return None
    s = prepare(case, seed)
    dev = "cuda"
    No, Nw, T, (Nx, Ny, Nz) = c["Norb"], c["Nw"], c["temp"], s["mesh"]
    Nk, Nchi, n = s["hamk"].shape[0], No * No, Nx * Ny * Nz
    kx, ky, kz = (torch.as_tensor(s["kmap"][:, i], device=dev) for i in range(3))
    ki = torch.as_tensor(s["invk"][:, 0] - 1, device=dev)
    at = (kx * Ny + ky) * Nz + kz  # cell of each full point
    cell, flag = torch.empty(n, dtype=torch.int64, device=dev), torch.empty(n, dtype=torch.bool, device=dev)
    cell[at] = ki
    flag[at] = torch.as_tensor(s["invk"][:, 1] != 0, device=dev)
    first = torch.full((Nk,), -1, dtype=torch.int64, device=dev)
    first[cell[~flag]] = torch.nonzero(~flag)[:, 0]
    w = (2 * torch.arange(Nw, device=dev, dtype=torch.float64) + 1) * math.pi * T
    if "G" in s:
        G = torch.as_tensor(s["G"], device=dev).permute(1, 0, 2, 3)  # [a, b, w, k]
    else:
        e, U = torch.as_tensor(s["eig"], device=dev), torch.as_tensor(s["uni"], device=dev)  # U[k, band, orbital]
        z = torch.complex(torch.full_like(w, s["mu"]), w)
        G = torch.einsum("kna,knb,wkn->abwk", U, U.conj(), 1.0 / (z[:, None, None] - e[None]))
    neg = torch.arange(Nw - 1, -1, -1, device=dev)

    def on_grid(pos, pos_t, negative, negative_t):
        """[2Nw, Nx, Ny, Nz] from the values at k and (transposed) at -k."""
        up = torch.where(flag, pos_t[:, cell], pos[:, cell])
        down = torch.where(flag, negative_t[:, cell], negative[:, cell])
        return torch.fft.fftn(torch.cat([up, down]).reshape(2 * Nw, Nx, Ny, Nz))

    Gh = [[on_grid(G[a, b], G[b, a], G[b, a][neg].conj(), G[a, b][neg].conj()) for b in range(No)] for a in range(No)]

    def mirrored(a):
        return torch.roll(torch.flip(a, (0, 1, 2, 3)), (1, 1, 1, 1), (0, 1, 2, 3))

    def irreducible(a):
        return torch.fft.ifftn(a).reshape(2 * Nw, n)[:Nw][:, first]

    def zeroed(a):
        re, im = a.real, a.imag
        return torch.complex(torch.where(re.abs() < 1e-9, 0.0, re), torch.where(im.abs() < 1e-9, 0.0, im))

    o1, o2 = [int(v) - 1 for v in s["olist"][:, 0]], [int(v) - 1 for v in s["olist"][:, 1]]
    pair = {(o1[i], o2[i]): i for i in range(Nchi)}
    chi = torch.zeros((Nchi, Nchi, Nw, Nk), dtype=torch.complex128, device=dev)  # [l, m, w, k] = element (m, l)
    done = set()
    for l in range(Nchi):
        for m in range(Nchi):
            if (l, m) in done:
                continue
            v = zeroed(irreducible(-Gh[o1[l]][o1[m]] * mirrored(Gh[o2[m]][o2[l]])) * (T / n))
            # the exchange partner chi_1234 = conj chi_4321
            l2, m2 = pair[(o2[m], o1[m])], pair[(o2[l], o1[l])]
            if (l2, m2) == (l, m):
                v = v.conj()
            chi[l, m] = v
            if (l2, m2) != (l, m):
                chi[l2, m2] = v.conj()
            done |= {(l, m), (l2, m2)}
    S = torch.as_tensor(s["S"].T.copy(), device=dev, dtype=torch.complex128)
    C = torch.as_tensor(s["C"].T.copy(), device=dev, dtype=torch.complex128)
    X = chi.permute(2, 3, 1, 0)  # [w, k, m, l]
    x0 = X[0]
    stoner = torch.linalg.eigvals((x0 @ S).cpu()).real.max().item()
    if c["kind"] == "chi0":
        return chi.cpu().numpy(), stoner
    if stoner >= 1.0:
        X = X * ((1.0 - 1.0e-4) / stoner)
    one, V = torch.eye(Nchi, device=dev, dtype=torch.complex128), torch.empty_like(chi)
    for j in range(0, Nw, 32):
        XS, XC = X[j:j + 32] @ S, X[j:j + 32] @ C
        v = (1.5 * S - 0.5 * C) + 1.5 * (S @ torch.linalg.solve(one - XS, XS)) \
            + 0.5 * (C @ torch.linalg.solve(one + XC, XC)) - 0.25 * ((S + C) @ (XS + XC))
        V[:, :, j:j + 32] = v.permute(3, 2, 0, 1)
    stat = (1.5 * S - 0.5 * C).real.cpu()
    sig = torch.zeros((No, No, Nw, Nk), dtype=torch.complex128, device=dev)  # [b, a, w, k]
    for b in range(No):
        for a in range(No):
            acc = 0.0
            for l in (i for i in range(Nchi) if o1[i] == b):
                for m in (i for i in range(Nchi) if o1[i] == a):
                    p, q = V[l, m], V[m, l]
                    fixed = torch.full((1, Nk), float(stat[m, l]), dtype=torch.complex128, device=dev)
                    down, down_t = (torch.cat([fixed, x[1:][torch.arange(Nw - 2, -1, -1, device=dev)].conj()])
                                    for x in (q, p))
                    acc = acc + on_grid(p, q, down, down_t) * Gh[o2[m]][o2[l]]
            sig[b, a] = zeroed(irreducible(acc) * (T / n))
    sub = 0.5 * (sig[:, :, 0] + sig[:, :, 0].transpose(0, 1).conj())
    out = 0.5 * (sig - sub[:, :, None])
    return out.cpu().numpy(), None
