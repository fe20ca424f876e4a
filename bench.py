#!/usr/bin/env python
"""Time to a converged FLEX self-energy plus the linearized-Eliashberg
eigenvalue on one GB300, for the 5-orbital 64x64x2048 model (config c2).

One step = one full solve of the reference's calc_lin_eliashberg_eq path
(mkself to the residual eps -> G -> tail-corrected chi0 -> lin_eliash), run
through the engine's C ABI (pyrpa_gb_flex_eliash, host buffers in and out),
in the fast form: coarse-mesh warm start, FP32 then double-float bulk, a
double-float judging iteration.  lin_eliash runs 20-step Arnoldi cycles,
restarted until the Ritz residual is below 1e-8 of lambda: the reference's
single 10-step pass stops 20% short of the leading eigenvalue on this model.
  value        device seconds of the solve with the inputs already in HBM
               (CUDA events on the library stream, between upload and download)
  e2e          wall seconds of the whole ABI call from host buffers, copies included
  plain_fp64   after the timed steps, the same model solved once in plain FP64
               from G0 (no warm start): the metric's denominator, with the
               lambda, Sigma and mu differences of the fast form from it
  strict_judging  then the fast form once more with a fresh DIIS history in
               its judging phase, which also removes the middle phase's Sigma
               bias: its time and its differences from plain FP64
  roofline     the FFT passes (fft2_kernel<R, A, B>; every pass of the 64x64x4096
               transforms), the kernel that moves the most bytes, timed live per
               launch with CUDA events during the timed steps
  cpu_baseline the oracle's restatement of the reference's CPU path, every
               stage of a FLEX iteration and of an Eliashberg application timed
               on a bounded full-size sample on all host cores and scaled to
               one solve with the plain FP64 solve's iteration and application
               counts (cpu_reference_estimate)
Inputs are larger than L2 (every FFT array is >= 134 MB), so no L2 flush is
needed between steps.  `--impl reference` prints the CPU line only.
Under torchrun every rank solves its own copy of the model (replicas, no
collective on the data path); the reported time is the maximum over ranks.
"""
from __future__ import annotations

import argparse
import json
import multiprocessing as mp
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
METRIC = "time-to-converged FLEX Σ+λ, 5-orb 64²×2048: FP32+warm-start vs plain FP64"


# ------------------------------------------------------ profiling cases
# Small launches of single engine kernels for ncu captures: each runs one ABI
# call on a synthetic input larger than L2 (129 MB) but a few hundred MB at
# most, so that a capture of one launch replays quickly.
#   vertex  get_vsigma_flex_nosoc_ on a 5-orbital chi0 (Nchi = 25), 130
#           irreducible q x 512 frequencies = 66,560 matrices
#   chi0    get_chi0_tail on a 5-orbital mesh (default 16x16, 512 frequencies)
#   flex    mkself, one FLEX iteration of the same model (--profile-mesh, --profile-nw)
#   eliash  bare chi0 and a 4-step lin_eliash of the same model (V_Delta, mkfk,
#           the mkdelta contraction)
#   fft     get_chi0 of a 1-orbital 64x64 mesh with 2048 frequencies: FFT
#           passes over 64x64x4096 arrays (134 MB in FP32)
def _profile_model(F, models, Norb=5, N=16, Nw=512, temp=0.02):
    rvec, ham_r = models.seeded_hoppings(Norb, 4, [(1, 0, 0), (1, 1, 0), (2, 0, 0)], dim=2, bandwidth=4.0)
    klist, kmap, invk = F.gen_irr_k_TRS(N, N, 1)
    hamk = F.gen_ham(klist, ham_r, rvec)
    eig, uni = F.get_eig(hamk)
    olist, site = F.get_chi_orb_list(Norb)
    S, C = F.gen_SCmatrix(olist, site, 1.2, 0.2)
    w = F.gen_kpoint_weight(invk, len(klist))
    mu = models.bare_mu(eig, w, 0.6 * Norb, temp)
    return dict(Norb=Norb, N=N, Nw=Nw, temp=temp, klist=klist, kmap=kmap, invk=invk, hamk=hamk, eig=eig, uni=uni,
                olist=olist, S=S, C=C, mu=mu)


def profile_case(case: str, precision: int, repeat: int, mesh: int = 16, nw: int = 512) -> int:
    sys.path.insert(0, str(ROOT))
    from pyrpa_gb300 import flibs as F, models
    F.load_library()
    F.set_verbose(0)
    F.set_precision(precision)
    t0 = time.perf_counter()
    for _ in range(repeat):
        if case == "vertex":
            Nchi, Nk, Nw = 25, 130, 512
            rng = np.random.default_rng(0)
            chi = 0.05 * (rng.standard_normal((Nchi, Nchi, Nw, Nk)) + 1j * rng.standard_normal((Nchi, Nchi, Nw, Nk)))
            olist, site = F.get_chi_orb_list(5)
            S, C = F.gen_SCmatrix(olist, site, 1.2, 0.2)
            # the raw entry with explicit Nk, Nw (the Python wrapper reads
            # them off the array the way the reference wrapper does)
            F._call("get_vsigma_flex_nosoc_", chi, S, C, F.i64(Nk), F.i64(Nw), F.i64(Nchi))
        elif case == "chi0":
            m = _profile_model(F, models, N=mesh, Nw=nw)
            Gk = F.gen_Green0(m["eig"], m["uni"], m["mu"], m["temp"], m["Nw"])
            F.get_chi0_tail(m["S"], m["C"], Gk, m["eig"], m["uni"], m["olist"], m["kmap"], m["invk"], m["mu"],
                            m["temp"], m["N"], m["N"], 1)
        elif case == "eliash":
            m = _profile_model(F, models, N=mesh, Nw=nw)
            Gk = F.gen_Green0(m["eig"], m["uni"], m["mu"], m["temp"], m["Nw"])
            chi, _ = F.get_chi0(m["S"], m["C"], Gk, m["olist"], m["kmap"], m["invk"], m["temp"], m["N"], m["N"], 1)
            init = F.get_initial_gap(m["klist"], m["Norb"], 0)
            F.linearized_eliashberg(chi, Gk, m["uni"], init, m["S"], m["C"], m["olist"], np.ones(m["Norb"]),
                                    m["kmap"], m["invk"], m["N"], m["N"], 1, m["temp"], 0, arnoldi_m=4)
        elif case == "fft":
            m = _profile_model(F, models, Norb=1, N=64, Nw=2048, temp=0.01)
            Gk = F.gen_Green0(m["eig"], m["uni"], m["mu"], m["temp"], m["Nw"])
            F.get_chi0(m["S"], m["C"], Gk, m["olist"], m["kmap"], m["invk"], m["temp"], m["N"], m["N"], 1)
        else:
            m = _profile_model(F, models, N=mesh, Nw=nw)
            F.mkself(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"], m["uni"], m["mu"],
                     0.6 * m["Norb"], m["temp"], m["Nw"], m["N"], m["N"], 1, False, False, scf_loop=1, eps=1e-4,
                     pp=0.5, sw_tail=True, sw_rescale=True)
    print(f"{case}: {repeat} call(s) in {time.perf_counter() - t0:.3f} s", flush=True)
    return 0


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--profile-case", choices=["vertex", "chi0", "flex", "fft", "eliash"],
                   help="run one small profiling case instead of the benchmark")
    p.add_argument("--repeat", type=int, default=1, help="calls of the profiling case")
    p.add_argument("--profile-mesh", type=int, default=16, help="k mesh side of the chi0 and flex cases")
    p.add_argument("--profile-nw", type=int, default=512, help="Matsubara frequencies of the chi0 and flex cases")
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=2)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    p.add_argument("--config", default="c2", choices=["c1", "c2", "c5"])
    p.add_argument("--precision", default="mixed", choices=["mixed", "32", "64", "48"],
                   help="mixed: FP32 bulk to the FP32 rounding floor, then double-float bulk to eps")
    p.add_argument("--eps", type=float, default=1.0e-4)
    p.add_argument("--scf-loop", type=int, default=300)
    p.add_argument("--no-tail", action="store_true")
    p.add_argument("--coarse", default="2,2",
                   help="warm start: k-mesh and frequency divisors of the coarse solve ('1,1' = cold start)")
    p.add_argument("--arnoldi-m", type=int, default=20, help="Krylov steps per Arnoldi cycle of lin_eliash")
    p.add_argument("--arnoldi-tol", type=float, default=1.0e-8,
                   help="restart the Arnoldi pass until the Ritz residual over |lambda| is below this "
                        "(0: the reference's single fixed-size pass)")
    p.add_argument("--no-fp64", action="store_true",
                   help="skip the plain FP64 cold-start solve after the timed steps (the metric's denominator)")
    p.add_argument("--no-strict", action="store_true",
                   help="skip the fast form with a fresh DIIS history in the judging phase after the timed steps")
    p.add_argument("--flex-iters", type=int, default=0, help="reference arm: FLEX iterations to scale with")
    p.add_argument("--applies", type=int, default=0, help="reference arm: Eliashberg applications to scale with")
    return p.parse_args()


# ---------------------------------------------------------------- clocks
class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.idx = gpu_index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.idx}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in self.lines:
            f = [x.strip() for x in l.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


# ----------------------------------------------------------- CPU baseline
# The reference's CPU path, restated by the oracle, timed stage by stage on a
# bounded sample of the full-size workload and scaled to one solve.  Each unit
# below is one piece of the reference's own loop structure at the full mesh:
#   chi0    one bubble of one irreducible orbital pair of chi0_conv_acc
#           (fchi.f90:508-613): pads, 2 forward 4-D FFTs, product, backward;
#           with sw_tail a pair takes two (G and G0) and
#   tailref the analytic tau reference of one pair (fchi.f90:637-850)
#   sigma   one (l, m) pair of calc_sigma (fself.f90:159-285): 3 FFTs
#   delta   one pair of mkdelta_nsoc (feliash.f90:486-635): 3 FFTs
#   vertex  get_vsigma_flex_nosoc (fUJ.f90:318-365) on a slice of the (q, i nu)
#           matrices
#   mu      the zgeev of H + Sigma per (k, i w) of renew_mu (fself.f90:689-711)
#           plus MU_EVALS fillings get_rn (fself.f90:662-687), on a slice
#   dyson   gen_green_inv + getinv (fself.f90:43-157) on a slice
#   diis    compare_sigma (fself.f90:449-542): the Gram matrix of a full
#           history and the extrapolation, on a slice
#   stoner  ckchi (fchi.f90:352-399): zgeev of chi0(q, 0) S at every q
#   mkfk    mkfk_trs_nsoc (feliash.f90:445-484) on a slice
# Every unit runs in its own spawned worker, all at once on the host cores,
# and the solve's time is sum(units x seconds per unit) / workers, which
# assumes the reference spreads each stage perfectly over the cores (its
# FFTs are serial): a lower bound on the reference's time.
MU_EVALS = 16          # fillings per renew_mu: bracket plus the inverse-quadratic search
SLICE = 128            # the vertex, mu, Dyson, DIIS and mkfk samples are 1/SLICE of the full size
# FLEX iterations and Eliashberg applications of the plain FP64 cold-start
# GPU solve of each configuration (eps 1e-4, DIIS 5, pp 0.5, 20-step Arnoldi
# cycles restarted to a Ritz residual of 1e-10), from that solve's own
# statistics; the reference arm, which has no GPU run of its own, scales
# with them
PLAIN_FP64_COUNTS = {"c2": (24, 60), "c1": (11, 40), "c5": (29, 40)}


def _cpu_unit(job):
    kind, cfg, tail, seed = job
    sys.path.insert(0, str(ROOT))
    from oracle import flex_oracle as FO
    rng = np.random.default_rng(seed)
    Nx, Ny, Nz, Nw, No, temp = cfg["Nx"], cfg["Ny"], cfg["Nz"], cfg["Nw"], cfg["Norb"], cfg["temp"]
    nchi = No * No
    K = FO.irr_k_count(Nx, Ny, Nz) * Nw

    def crand(*shape):
        return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)

    if kind in ("chi0", "tailref", "sigma", "delta"):
        klist, kmap, invk = FO.generate_irr_kpoint_inv(Nx, Ny, Nz)
        grid = FO.KGrid(kmap, invk, Nx, Ny, Nz)
        Nk = len(klist)
        ol = np.array([[1, 1]])
        one = np.ones((1, 1))
        G = 0.1 * crand(Nk, Nw, 1, 1)
        t0 = time.perf_counter()
        if kind == "tailref":
            chi_map, irr = FO.get_chi_map(ol)
            U = np.ones((Nk, 1, 1), dtype=complex)
            e = rng.uniform(-1, 1, (Nk, 1))
            FO.gen_green0_F(e, U, 0.0, temp, Nw)
            FO.chi0_ref_tau(np.zeros((Nk, Nw, 1, 1), dtype=complex), e, U, 0.0, grid, ol, temp, Nw, chi_map, irr)
        elif kind == "chi0":
            FO.get_chi0_conv(G, grid, ol, temp)
        elif kind == "sigma":
            FO.calc_sigma(G, 0.1 * crand(Nk, Nw, 1, 1), one, one, grid, ol, temp)
        else:
            FO.mkdelta_nsoc(G, 0.1 * crand(Nk, Nw, 1, 1), one, one, grid, np.ones(1), ol, True)
        return kind, time.perf_counter() - t0, 1
    n = max(1, K // SLICE)
    if kind == "vertex":
        S = rng.standard_normal((nchi, nchi))
        S = 0.05 * (S + S.T)
        chi = 0.05 * crand(n, 1, nchi, nchi)
        t0 = time.perf_counter()
        FO.vsigma_flex_nosoc(chi, S, 0.5 * S)
        return kind, time.perf_counter() - t0, n
    if kind == "stoner":
        nq = FO.irr_k_count(Nx, Ny, Nz)
        S = rng.standard_normal((nchi, nchi))
        chi = 0.05 * crand(nq, 1, nchi, nchi)
        t0 = time.perf_counter()
        FO.ckchi(chi, S, 0.5 * S)
        return kind, time.perf_counter() - t0, 1
    A = crand(n, No, No)
    if kind == "mu":
        z = (0.1 + 1j * np.linspace(0.01, 10.0, n))[:, None]
        e = rng.uniform(-1, 1, (n, No))
        t0 = time.perf_counter()
        lam = np.linalg.eigvals(A)
        for _ in range(MU_EVALS):
            np.sum((1.0 / (z - lam) - 1.0 / (z - e)).real)
        return kind, time.perf_counter() - t0, n
    if kind == "dyson":
        t0 = time.perf_counter()
        np.linalg.inv(A + 2j * np.eye(No))
        return kind, time.perf_counter() - t0, n
    if kind == "mkfk":
        t0 = time.perf_counter()
        FO.hermitize_lower(-(A @ A @ np.conj(np.swapaxes(A, -1, -2))))
        return kind, time.perf_counter() - t0, n
    # diis: Gram matrix of 5 residuals, extrapolation and the relative change
    hist = [crand(n, No, No) for _ in range(5)]
    t0 = time.perf_counter()
    B = np.array([[np.sum(np.conj(a) * b).real for b in hist] for a in hist])
    sd = sum(c * h for c, h in zip(np.linalg.solve(B + np.eye(5), np.ones(5)), hist))
    np.abs((hist[0] - sd) / np.where(np.abs(sd) > 1e-10, sd, 1.0)).max()
    return kind, time.perf_counter() - t0, n


def _irr_count(cfg):
    sys.path.insert(0, str(ROOT))
    from oracle import flex_oracle as FO
    return FO.irr_k_count(cfg["Nx"], cfg["Ny"], cfg["Nz"])


def cpu_reference_estimate(cfg, tail: bool, iters: int, applies: int):
    """Seconds of one solve on the host cores (see the table above), the
    workers used and a description of what was timed."""
    cores = os.cpu_count() or 1
    No = cfg["Norb"]
    nchi = No * No
    nirr = nchi * (nchi + 1) // 2
    K = _irr_count(cfg) * cfg["Nw"]
    kinds = ["chi0", "sigma", "delta", "vertex", "mu", "dyson", "diis", "stoner", "mkfk"] + (["tailref"] if tail else [])
    jobs = [(k, cfg, tail, i) for i, k in enumerate(kinds)]
    jobs += [(k, cfg, tail, 100 + i) for i, k in enumerate((["chi0", "sigma"] * cores)[: max(0, cores - len(jobs))])]
    ctx = mp.get_context("spawn")
    # one BLAS / OpenMP thread per worker: the children read these when they
    # import numpy, before any unit runs
    saved = {k: os.environ.get(k) for k in ("OMP_NUM_THREADS", "OPENBLAS_NUM_THREADS", "MKL_NUM_THREADS")}
    os.environ.update({k: "1" for k in saved})
    try:
        t0 = time.perf_counter()
        with ctx.Pool(processes=min(cores, len(jobs))) as pool:
            res = pool.map(_cpu_unit, jobs)
        wall = time.perf_counter() - t0
    finally:
        for k, v in saved.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v
    per = {}
    for kind, sec, n in res:
        per.setdefault(kind, []).append(sec / n)
    u = {k: statistics.mean(v) for k, v in per.items()}
    per_apply = sum(1 for a in range(No) for c in range(No) for b in range(No) for d in range(No) if a >= b)
    # with sw_tail an irreducible pair is two bubbles (of G and of G0) and the tau reference
    pair = 2 * u["chi0"] + u["tailref"] if tail else u["chi0"]
    it = (nirr * pair + u["stoner"] + K * u["vertex"] + nchi * nchi * u["sigma"] + K * u["diis"]
          + K * u["mu"] + K * u["dyson"])
    final = K * u["dyson"] + nirr * pair + K * u["vertex"]
    app = per_apply * u["delta"] + K * u["mkfk"]
    total = (iters * it + final + applies * app) / cores
    sample = (f"oracle (numpy FP64) on {cores} spawned workers, {wall:.1f} s: at the full {cfg['Nx']}x{cfg['Ny']}x"
              f"{cfg['Nz']}x{cfg['Nw']} mesh one irreducible-pair chi0 bubble {u['chi0']:.2f} s"
              f"{(', tau reference %.2f s' % u['tailref']) if tail else ''}, one Sigma pair {u['sigma']:.2f} s, "
              f"one mkdelta pair {u['delta']:.2f} s, Stoner {u['stoner']:.2f} s; per (k,w) matrix (1/{SLICE} "
              f"slices): vertex {u['vertex'] * 1e6:.1f} us, mu {u['mu'] * 1e6:.2f} us, Dyson "
              f"{u['dyson'] * 1e6:.2f} us, DIIS {u['diis'] * 1e6:.2f} us, mkfk {u['mkfk'] * 1e6:.2f} us; per FLEX "
              f"iteration {nirr} chi0 pairs + {nchi * nchi} Sigma pairs, per application {per_apply} mkdelta "
              f"pairs; x {iters} FLEX iterations + {applies} Eliashberg applications, divided by {cores} workers")
    return total, cores, sample


# ------------------------------------------------------------------ main
def pair_classes(Norb: int) -> int:
    """Classes of pair elements (l, m) ~ (m, l) ~ (Pl, Pm), P(a, b) = (b, a): the
    transforms of an even model (175 at five orbitals)."""
    pairs = [(a, b) for a in range(Norb) for b in range(Norb)]
    return len({frozenset([(x, y), (y, x), (x[::-1], y[::-1]), (y[::-1], x[::-1])]) for x in pairs for y in pairs})


def solve_traffic(Norb: int, Nk: int, Nkall: int, Nw: int, stats: dict, precision: str,
                  half_mesh: int | None = None) -> float:
    """Algorithmic HBM bytes of one fine solve (the coarse warm start left
    out), with P = Nkall 2Nw, K = Nk Nw, Nchi = Norb^2 and an ideal 4-D FFT of
    two read-write sweeps:
      per FLEX iteration        B [4P (2 Norb^2 + Nchi(Nchi+1)/2 + Nchi^2) + P Nchi^2 + 16 K Norb^2]
                                + Bv 2 K Nchi^2
      per Eliashberg application  Be [8P Norb^2 + 2P Nchi^2 + 4K Norb^2]
    B, Bv and Be are the bytes of a complex chi0/Sigma, vertex and Eliashberg
    element in each phase: 8 for FP32, 16 for FP64 and double-float.  half_mesh:
    the points of half the mesh, for an even model, whose arrays have half_mesh Nw
    elements, Norb (Norb + 1) / 2 orbital elements and pair_classes pair elements."""
    nchi = Norb * Norb
    P, K = Nkall * 2 * Nw, Nk * Nw
    n_el, n_fwd, n_pair = Norb ** 2, nchi * (nchi + 1) // 2, nchi ** 2
    if half_mesh:
        P, n_el, n_fwd, n_pair = half_mesh * Nw, Norb * (Norb + 1) // 2, pair_classes(Norb), pair_classes(Norb)

    def it_bytes(B, Bv):
        return (B * (4 * P * (2 * n_el + n_fwd + n_pair) + P * n_pair + 16 * K * Norb ** 2)
                + Bv * 2 * K * n_pair)

    n = int(stats["iterations"])
    if precision == "mixed":
        n32, nmid = int(stats["iterations_fp32"]), int(stats["iterations_fp64_fp32vertex"])
        flex = n32 * it_bytes(8, 8) + nmid * it_bytes(16, 8) + (n - n32 - nmid) * it_bytes(16, 16)
        be = 16
    elif precision == "32":
        flex, be = n * it_bytes(8, 8), 8
    else:
        flex, be = n * it_bytes(16, 16), 16
    return float(flex + int(stats["applies"]) * be * (8 * P * n_el + 2 * P * n_pair + 4 * K * Norb ** 2))


def max_over_ranks(values, dist):
    """Replicas: every rank solved its own instance; the job's time is the
    slowest rank's (all-reduce MAX, then a barrier)."""
    import torch
    t = torch.tensor(values, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    dist.barrier()
    return [float(x) for x in t]


def main():
    a = parse()
    if a.precision == "48" and not a.profile_case:
        raise SystemExit("--precision 48 (double-float chi0 and Sigma) is for the profiling cases only")
    if a.profile_case:
        return profile_case(a.profile_case, {"mixed": 32, "32": 32, "64": 64, "48": 48}[a.precision], a.repeat,
                            a.profile_mesh, a.profile_nw)
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        os.environ["CUDA_VISIBLE_DEVICES"] = str(local)
    sys.path.insert(0, str(ROOT))
    from pyrpa_gb300 import models

    cfg = dict(models.CONFIGS[a.config])
    tail = not a.no_tail
    config = {"workload": f"{a.config}: {cfg['Norb']}-orbital {cfg['Nx']}x{cfg['Ny']}x{cfg['Nz']} k-mesh, "
                          f"{cfg['Nw']} Matsubara, FLEX+linearized Eliashberg",
              "Norb": cfg["Norb"], "k_mesh": [cfg["Nx"], cfg["Ny"], cfg["Nz"]], "Nw": cfg["Nw"],
              "U": cfg["U"], "J": cfg["J"], "T": cfg["temp"], "fill_per_spin": cfg["fill"], "eps": a.eps,
              "chi0": "tail-corrected" if tail else "sharp cutoff",
              "parallelism": f"replicas x{a.gpus}" if a.gpus > 1 else "single GPU",
              "l2": "inputs larger than L2 (FFT arrays >= 134 MB); no flush"}

    if a.impl == "reference":
        if rank != 0:
            return 0
        iters = a.flex_iters or PLAIN_FP64_COUNTS[a.config][0]
        applies = a.applies or PLAIN_FP64_COUNTS[a.config][1]
        vals = []
        for i in range(a.warmup + a.steps):
            v, cores, sample = cpu_reference_estimate(cfg, tail, iters, applies)
            if i >= a.warmup:
                vals.append(v)
        v = statistics.mean(vals)
        line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "s", "n_gpus": 0, "steps": a.steps,
                "warmup": a.warmup, "ms_per_step": v * 1e3, "higher_is_better": False, "scaling": "weak",
                "vs_baseline": None, "dtype": "c128", "data": "synthetic seeded tight-binding model",
                "config": config,
                "cpu_baseline": {"value": v, "unit": "s", "cores": cores, "kind": "port",
                                 "sample": sample + " (mean over the timed steps; the counts are those of the plain "
                                                    "FP64 cold-start GPU solve of this configuration)"},
                "e2e": {"value": v, "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line), flush=True)
        return 0

    from pyrpa_gb300 import flibs as F

    F.load_library()
    F.set_verbose(0)
    F.set_precision({"mixed": F.MIXED, "32": 32, "64": 64}[a.precision])
    F.set_arnoldi_tol(a.arnoldi_tol)
    m = models.prepare(a.config)
    c = m["cfg"]
    coarse = tuple(int(x) for x in a.coarse.split(","))
    call = dict(mu=m["mu"], fill=c["fill"], temp=c["temp"], Nw=c["Nw"], Nx=c["Nx"], Ny=c["Ny"], Nz=c["Nz"],
                gap_sym=c["gap_sym"], eps=a.eps, scf_loop=a.scf_loop, sw_tail=tail, sw_rescale=True, coarse=coarse,
                arnoldi_m=a.arnoldi_m)
    config["arnoldi"] = (f"{a.arnoldi_m} steps a cycle, restarted until the Ritz residual is below "
                         f"{a.arnoldi_tol:g} of lambda" if a.arnoldi_tol > 0 else
                         f"the reference's two passes of {a.arnoldi_m} steps")
    config["warm_start"] = ("none (cold G0 start)" if coarse == (1, 1) else
                            f"coarse-mesh seed: {c['Nx'] // coarse[0]}x{c['Ny'] // coarse[0]} k mesh, "
                            f"{c['Nw'] // coarse[1]} frequencies, FP32 bulk (itself seeded one level further "
                            f"down), interpolated to the full mesh")

    def solve():
        return F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"], m["uni"],
                             m["init"], m["plist"], **call)

    for _ in range(a.warmup):
        solve()
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("gloo")
        dist.barrier()
    F.fft_profile(True)
    F.fft_stats()
    k0 = F.kernel_launches()
    dev, wall, res = [], [], None
    with ClockSampler(local if world == 1 else 0) as clk:
        for _ in range(a.steps):
            t0 = time.perf_counter()
            res = solve()
            wall.append(time.perf_counter() - t0)
            dev.append(res["compute_ms"] / 1e3)
    F.fft_profile(False)
    fft = F.fft_stats()
    launches = F.kernel_launches() - k0
    stats = F.last_stats()
    value, e2e = max(dev), max(wall)
    if dist is not None:
        value, e2e = max_over_ranks([value, e2e], dist)
    if rank != 0:
        return 0
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    peak = peaks.get("hbm_gbs", 6800.0)
    achieved = (fft["bytes"] / (fft["ms"] / 1e3) / 1e9) if fft["ms"] > 0 else None
    per_launch_bytes = fft["bytes"] / max(1, fft["launches"])
    # DRAM bytes per algorithmic byte of a time-axis pass over the half mesh, from
    # ncu captures of fft2_kernel<dfl,8,8> and <dfl,4,8> on one 2112x2048 array
    # (dram__bytes_read.sum + dram__bytes_write.sum = 75.8 MB over 138.4 MB
    # algorithmic, mean of 6 launches from a flushed cache; most of the result is
    # still in L2 at kernel end.  The FP32 passes: 34.6 over 69.2 MB)
    traffic_per_byte = 75.8 / 138.4
    in_bytes = sum(x.nbytes for x in (m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"],
                                        m["uni"], m["init"], m["plist"]))
    out_bytes = res["sigmak"].nbytes + res["gap"].nbytes
    iters, applies = int(stats["iterations"]), int(stats["applies"])
    # the library takes the even form for a symmetric H(k)
    even = (abs(m["hamk"] - m["hamk"].transpose(0, 2, 1)).max() <= 1e-13 * abs(m["hamk"]).max()
            and os.environ.get("PYRPA_GB_EVEN") != "0")
    axis = c["Nz"] if c["Nz"] > 1 else c["Ny"]
    half = len(m["kmap"]) // axis * (axis // 2 + 1) if even else None
    solve_bytes = solve_traffic(c["Norb"], len(m["klist"]), len(m["kmap"]), c["Nw"], stats, a.precision, half)
    solve_s = value - stats["t_warm_ms"] / 1e3
    ritz = [float(x) for x in F.last_ritz(4)]
    fp64 = None if a.no_fp64 else plain_fp64_comparison(F, solve_args=(m, call), res=res)
    strict = None if (a.no_strict or not fp64 or a.precision != "mixed") else strict_form(F, (m, call), fp64)
    cpu_counts = ((fp64["flex_iterations"], fp64["eliashberg_applications"]) if fp64
                  else PLAIN_FP64_COUNTS[a.config])
    cpu_v, cores, cpu_sample = cpu_reference_estimate(c, tail, *cpu_counts)
    config.update({"flex_iterations": iters, "eliashberg_applications": applies, "lambda": res["lam"],
                   "lambda_top4": ritz, "ritz_residual": stats["ritz_residual"],
                   "arnoldi_cycles": int(stats["arnoldi_cycles"]),
                   "warm_start_iterations": int(stats["iterations_coarse"]),
                   "warm_start_ms": stats["t_warm_ms"],
                   "stoner": res["stoner"], "mu": res["mu"], "esterr": stats["esterr"],
                   "precision": {"mixed": f"FP32 bulk for {int(stats['iterations_fp32'])} iterations, double-float chi0 "
                                          f"and Sigma with FP32 vertex for {int(stats['iterations_fp64_fp32vertex'])}, "
                                          f"then double-float chi0, vertex and Sigma to eps; Eliashberg stage "
                                          f"double-float (chi0, V_Delta, contractions)",
                                 "32": "FP32 bulk", "64": "FP64"}[a.precision]})
    line = {
        "metric": METRIC, "value": value, "unit": "s", "n_gpus": a.gpus, "steps": a.steps, "warmup": a.warmup,
        "ms_per_step": value * 1e3, "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
        "dtype": {"mixed": "c64+c128", "32": "c64", "64": "c128"}[a.precision], "data": "synthetic seeded tight-binding model",
        "config": config,
        "e2e": {"value": e2e, "unit": "s", "h2d_bytes_per_step": int(in_bytes), "d2h_bytes_per_step": int(out_bytes)},
        "gpu_launches": int(launches),
        "roofline": {"bound": "hbm", "kernel": "fft2_kernel, fft2_tma_kernel (FFT passes)", "achieved": achieved, "peak": peak,
                     "unit": "GB/s", "frac": (achieved / peak) if achieved else None,
                     "peak_source": "measured (MEASURED_PEAKS.json hbm_gbs)" if peaks else "fallback",
                     "bytes_per_launch": per_launch_bytes, "launches": fft["launches"],
                     "avg_launch_ms": fft["ms"] / max(1, fft["launches"]),
                     "traffic": per_launch_bytes * traffic_per_byte,
                     "traffic_source": "ncu captures of double-float time-axis passes over 2112x2048 points, scaled by "
                                       "bytes per launch"},
        "solve_roofline": {"bound": "hbm", "bytes": solve_bytes, "seconds": solve_s,
                           "achieved": solve_bytes / solve_s / 1e9 if solve_s > 0 else None, "peak": peak,
                           "unit": "GB/s", "frac": solve_bytes / solve_s / 1e9 / peak if solve_s > 0 else None,
                           "scope": "fine FLEX iterations and Eliashberg applications, algorithmic bytes with an "
                                    "ideal two-sweep 4-D FFT; the coarse warm start is left out of bytes and time"},
        "cpu_baseline": {"value": cpu_v, "unit": "s", "cores": cores, "kind": "port",
                         "sample": cpu_sample + (" (counts of this run's plain FP64 cold-start solve)" if fp64 else
                                                 " (counts of an earlier plain FP64 cold-start solve)")},
        "clocks": clk.summary(),
        "stages_ms": {k: v for k, v in stats.items() if k.startswith("t_")},
    }
    if fp64:
        fp64.pop("_lambda", None)
        fp64.pop("_sigma", None)
        line["plain_fp64"] = fp64
        line["speedup_vs_plain_fp64"] = fp64["seconds"] / value
    if strict:
        line["strict_judging"] = strict
    print(json.dumps(line), flush=True)
    return 0


def strict_form(F, solve_args, fp64) -> dict:
    """The fast form with a fresh DIIS history in the judging phase
    (PYRPA_GB_JUDGE_DIIS=fresh), solved once: it removes the middle phase's
    FP32-vertex bias from Sigma at the cost of more judging iterations.  Its
    device seconds, iterations and lambda / Sigma differences from the plain
    FP64 solve."""
    m, call = solve_args
    os.environ["PYRPA_GB_JUDGE_DIIS"] = "fresh"
    try:
        r = F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"], m["uni"],
                          m["init"], m["plist"], **call)
    finally:
        os.environ.pop("PYRPA_GB_JUDGE_DIIS", None)
    st = F.last_stats()
    ref_lam, ref_sig = fp64.pop("_lambda"), fp64.pop("_sigma")
    return {"seconds": r["compute_ms"] / 1e3, "flex_iterations": int(st["iterations"]),
            "speedup_vs_plain_fp64": fp64["seconds"] / (r["compute_ms"] / 1e3), "lambda": r["lam"],
            "lambda_rel_diff": abs(r["lam"] - ref_lam) / abs(ref_lam),
            "sigma_max_rel_diff": float(np.abs(r["sigmak"] - ref_sig).max() / np.abs(ref_sig).max())}


def plain_fp64_comparison(F, solve_args, res) -> dict:
    """The same model solved in plain FP64 from G0 (no warm start), to the same
    eps: its device seconds and how far the fast form's lambda, Sigma and mu
    sit from it."""
    m, call = solve_args
    prec = F.get_precision()
    F.set_precision(64)
    try:
        ref = F.flex_eliash(m["S"], m["C"], m["kmap"], m["invk"], m["olist"], m["hamk"], m["eig"], m["uni"],
                            m["init"], m["plist"], **dict(call, coarse=(1, 1)))
    finally:
        F.set_precision(prec)
    st = F.last_stats()
    return {"seconds": ref["compute_ms"] / 1e3, "flex_iterations": int(st["iterations"]),
            "eliashberg_applications": int(st["applies"]), "lambda": ref["lam"],
            "ritz_residual": st["ritz_residual"],
            "lambda_rel_diff": abs(res["lam"] - ref["lam"]) / abs(ref["lam"]),
            "sigma_max_rel_diff": float(np.abs(res["sigmak"] - ref["sigmak"]).max() / np.abs(ref["sigmak"]).max()),
            "mu_diff": abs(res["mu"] - ref["mu"]), "_lambda": ref["lam"], "_sigma": ref["sigmak"]}


if __name__ == "__main__":
    sys.exit(main())
