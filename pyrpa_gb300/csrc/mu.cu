// Chemical-potential search of the FLEX loop on the device.
//
// The filling of get_rn needs, per (k, iw_j), sum_n 1/(z - lambda_n) with
// lambda_n the eigenvalues of H(k) + Sigma(k, iw_j) and z = mu + i w_j
// (fself.f90:662-711).  That sum is p'(z)/p(z) for p(z) = det(z - H - Sigma),
// so the search stores the coefficients of p instead of the eigenvalues:
// a pivoted elimination to Hessenberg form and the Hessenberg determinant
// recursion p_{m+1} = (z - h_mm) p_m - sum_{i<m} h_im (h_{i+1,i} ... h_{m,m-1}) p_i,
// with no iteration.  The coefficients are those in mu - center, with the
// shift by i w_j done once, so that p and p' of a trial mu are two Horner sums
// with real multipliers.
//
// The reference subtracts the bare bands' finite sum from each term and adds
// their exact filling.  The finite sum is known in closed form,
//   sum_{j<Nw} x/(x^2 + w_j^2) = tanh(x/2T)/4T - Im psi(Nw + 1/2 + i x/2 pi T) / 2 pi T,
// the tanh cancels the Fermi functions, and the filling is
//   n = Norb/2 + (1/Nk) [ sum_{k,n} Im psi(Nw + 1/2 + i x/2 pi T) / pi + 2 T sum_{k,j} Re p'/p ].
// psi is summed from its asymptotic series (Abramowitz and Stegun 6.3.18).
//
// One launch runs the whole search (bracketing, then inverse quadratic
// interpolation / bisection): every block evaluates its share of the
// points, the partial sums meet at a grid barrier, and every block takes the
// same scalar decisions from the same total.  A host-driven search paid two
// launches, a copy and a wait for each of its 30 to 40 evaluations.
// Measured, search with its coefficients (two searches of one FLEX iteration):
// one orbital 32x32x1024 2.6 -> 0.8 ms; five orbitals 64x64x1024 26 -> 5.5 ms (9.8
// with a Householder reduction).
#include <algorithm>
#include <cstdlib>

#include "flex.cuh"
#include "flex_dev.cuh"

namespace pgb {
namespace {

template <int N>
__global__ void k_charpoly_gk(double2* cp, const double2* hamk, const double2* sig, double center,
                              double temp, int Nk, int Nw) {
  const long long K = (long long)Nk * Nw;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < K;
       idx += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(idx % Nk), j = (int)(idx / Nk);
    double2 A[N][N];
#pragma unroll
    for (int l = 0; l < N; ++l)
#pragma unroll
      for (int m = 0; m < N; ++m)
        A[m][l] = hamk[m + N * (l + (long long)N * k)] + sig[fidx(k, j, m, l, Nk, Nw, N)];
#pragma unroll
    for (int l = 0; l < N; ++l) A[l][l].x -= center;
    // Hessenberg form by eliminations with pivoting (a similarity transform): a
    // third of the multiplications of the Householder reduction and no square
    // roots, and |Re p'/p| of 6000 random five-orbital cases came out with an
    // rms error of 1.2e-16 against 1.8e-16
#pragma unroll
    for (int c = 0; c + 2 < N; ++c) {
      int p = c + 1;
      double best = fabs(A[c + 1][c].x) + fabs(A[c + 1][c].y);
#pragma unroll
      for (int i = c + 2; i < N; ++i) {
        const double v = fabs(A[i][c].x) + fabs(A[i][c].y);
        if (v > best) {
          best = v;
          p = i;
        }
      }
      if (best == 0) continue;
#pragma unroll
      for (int i = c + 2; i < N; ++i) {
        const bool sw = p == i;
#pragma unroll
        for (int j = c; j < N; ++j) {
          const double2 x = A[c + 1][j], y = A[i][j];
          A[c + 1][j] = sw ? y : x;
          A[i][j] = sw ? x : y;
        }
#pragma unroll
        for (int r = 0; r < N; ++r) {
          const double2 x = A[r][c + 1], y = A[r][i];
          A[r][c + 1] = sw ? y : x;
          A[r][i] = sw ? x : y;
        }
      }
      const double2 ip = crecip(A[c + 1][c]);
      auto fms = [](double2 acc, double2 u, double2 v, double s) {  // acc + s u v, s = +-1
        const double2 w = mkc(s * u.x, s * u.y);
        return mkc(fma(w.x, v.x, fma(-w.y, v.y, acc.x)), fma(w.x, v.y, fma(w.y, v.x, acc.y)));
      };
#pragma unroll
      for (int i = c + 2; i < N; ++i) {
        const double2 m = A[i][c] * ip;
        A[i][c] = mkc(0.0, 0.0);
#pragma unroll
        for (int j = c + 1; j < N; ++j) A[i][j] = fms(A[i][j], m, A[c + 1][j], -1.0);
#pragma unroll
        for (int r = 0; r < N; ++r) A[r][c + 1] = fms(A[r][c + 1], m, A[r][i], 1.0);
      }
    }
    // P[m][d]: coefficient d of p_m (degree m, monic)
    double2 P[N + 1][N + 1];
#pragma unroll
    for (int m = 0; m <= N; ++m)
#pragma unroll
      for (int d = 0; d <= N; ++d) P[m][d] = mkc(0.0, 0.0);
    P[0][0] = mkc(1.0, 0.0);
#pragma unroll
    for (int m = 0; m < N; ++m) {
#pragma unroll
      for (int d = 0; d <= m; ++d) {
        P[m + 1][d + 1] += P[m][d];
        P[m + 1][d] -= A[m][m] * P[m][d];
      }
      double2 prod = mkc(1.0, 0.0);
#pragma unroll
      for (int i = m - 1; i >= 0; --i) {
        prod = prod * A[i + 1][i];
        const double2 f = A[i][m] * prod;
#pragma unroll
        for (int d = 0; d <= i; ++d) P[m + 1][d] -= f * P[i][d];
      }
    }
    // z = (mu - center) + i w: the polynomial in mu - center alone, by synthetic
    // division with i w, so that a trial mu needs real multipliers only
    const double w = (2.0 * j + 1.0) * kPi * temp;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int d = N - 1; d >= i; --d) {
        const double2 u = P[N][d + 1];
        P[N][d] = mkc(fma(-w, u.y, P[N][d].x), fma(w, u.x, P[N][d].y));
      }
#pragma unroll
    for (int d = 0; d < N; ++d) cp[d * K + idx] = P[N][d];
  }
}

// Im psi(a + i y)
__device__ double im_digamma(double a, double y) {
  double s = 0.0;
  for (; a < 14.0; a += 1.0) s += y / fma(a, a, y * y);
  const double d = 1.0 / fma(a, a, y * y);
  const double2 r = mkc(a * d, -y * d), r2 = r * r;
  const double c[7] = {1.0 / 12, -1.0 / 120, 1.0 / 252, -1.0 / 240, 1.0 / 132, -691.0 / 32760, 1.0 / 12};
  double2 t = mkc(0.0, 0.0);
#pragma unroll
  for (int k = 6; k >= 0; --k) t = (t + mkc(c[k], 0.0)) * r2;
  return s + atan2(y, a) - 0.5 * r.y - t.y;
}

constexpr int kMuThreads = 256;
constexpr long long kMuWaitCycles = 4000000000LL;  // about 2 s
constexpr int kMuAttempts = 40;

// Cycles of a wait between the blocks in the first attempt (PYRPA_GB_MU_WAIT; a
// search whose blocks gave up starts again with eight times as many)
long long mu_wait_cycles() {
  const char* s = std::getenv("PYRPA_GB_MU_WAIT");
  return s ? std::min(kMuWaitCycles, std::max(1LL, std::atoll(s))) : kMuWaitCycles;
}

// Sum over the grid of v, the same in every thread.  Blocks meet at a counter
// that only grows; every wait is bounded, and a block that gives up tells the
// caller through `dead`.  The launch is cooperative, so all blocks are resident
// at once, but another thread's kernel may hold some SMs for longer than a wait
// (the vertex of a large FP64 model runs for seconds): mu_search then starts again.
__device__ double grid_sum(double v, double* part, unsigned* bar, unsigned round, long long wait, bool& dead) {
  __shared__ double red[kMuThreads / 32];
  __shared__ double total;
  __shared__ int gave_up;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto warp_sum = [](double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
  v = warp_sum(v);
  if (lane == 0) red[w] = v;
  __syncthreads();
  double* p = part + (round & 1) * gridDim.x;
  if (threadIdx.x == 0) {
    gave_up = 0;
    double mine = red[0];
    for (int i = 1; i < nw; ++i) mine += red[i];
    __stcg(p + blockIdx.x, mine);
    __threadfence();
    atomicAdd(bar, 1u);
    const unsigned want = (round + 1) * gridDim.x;
    const long long t0 = clock64();
    while (*(volatile unsigned*)bar < want)
      if (clock64() - t0 > wait) {
        gave_up = 1;
        break;
      }
    __threadfence();
  }
  __syncthreads();
  dead = dead || gave_up;
  // the blocks' sums by one warp: an FP64 add of every warp would cost as much as
  // a trial point of every thread
  if (w == 0) {
    double s = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(p + b);
    s = warp_sum(s);
    if (lane == 0) total = s;
  }
  __syncthreads();
  return total;
}

template <int N>
__global__ void __launch_bounds__(kMuThreads) k_mu_search(MuState* io, const double2* cp, double center,
                                                          const double* eig, double fill, double esterr, double temp,
                                                          int Nk, int Nw, double* part, unsigned* bar, long long wait) {
  const long long K = (long long)Nk * Nw, S = (long long)gridDim.x * blockDim.x;
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  MuState st = *io;
  unsigned round = 0;
  bool dead = false;
  // points whose terms share one division (their |p|^2 multiply: fewer for
  // high degrees, to stay far from overflow)
  constexpr int G = N <= 4 ? 4 : 2;
  auto get_rn = [&](double rmu) {
    const double x = rmu - center;
    double acc = 0.0, tail = 0.0;
    // dealt out block by block: one digamma costs as much FP64 as a few points, and
    // the first blocks would hold all others up
    for (long long t = threadIdx.x * (long long)gridDim.x + blockIdx.x; t < (long long)Nk * N; t += S)
      tail += im_digamma(Nw + 0.5, (rmu - eig[t]) / (2.0 * kPi * temp));
    for (long long i = first; i < K; i += G * S) {
      double num[G], den[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        num[g] = 0.0;
        den[g] = 1.0;
        const long long at = i + g * S;
        if (at < K) {
          double2 p = cp[(N - 1) * K + at], dp;
          p.x += x;
#pragma unroll
          for (int d = N - 2; d >= 0; --d) {
            const double2 c = cp[d * K + at];
            dp = d == N - 2 ? mkc(x + p.x, p.y) : mkc(fma(dp.x, x, p.x), fma(dp.y, x, p.y));
            p = mkc(fma(p.x, x, c.x), fma(p.y, x, c.y));
          }
          num[g] = N == 1 ? p.x : fma(dp.x, p.x, dp.y * p.y);
          den[g] = fma(p.x, p.x, p.y * p.y);
        }
      }
#pragma unroll
      for (int h = 1; h < G; h <<= 1)
#pragma unroll
        for (int g = 0; g + h < G; g += 2 * h) {
          num[g] = fma(num[g], den[g + h], num[g + h] * den[g]);
          den[g] *= den[g + h];
        }
      acc += num[0] / den[0];
    }
    const double s = grid_sum(fma(2.0 * temp, acc, tail / kPi), part, bar, round, wait, dead);
    ++round;
    return 0.5 * N + s / Nk;
  };
  double mu = st.mu;
  const double eps = esterr > 1.0e-2 ? 1.0e-8 : esterr * 1.0e-1;
  double dmu = fabs(mu - st.mu_old) * 2.0;
  if (dmu < eps * 4.0) dmu = eps * 4.0;
  double muS = 0, muL = 0, rnS = 0, rnL = 0;
  bool found = false;
  int err = 0;
  st.cached = 0;
  if (st.bracket_valid) {
    rnS = get_rn(st.muS);
    rnL = get_rn(st.muL);
    if (rnS < fill && rnL > fill) {
      muS = st.muS;
      muL = st.muL;
      found = true;
      st.cached = 1;
    } else {
      st.cached = 2;
    }
  }
  if (!found) {
    muL = mu + dmu;
    muS = mu - dmu;
    for (int it = 1; it <= 100 && !dead; ++it) {
      rnL = get_rn(muL);
      if (!(rnL < fill)) break;
      if (fabs(fill - rnL) > 0.5) muL += 1.0;
      else if (fabs(fill - rnL) > dmu) muL += 0.5;
      else muL += dmu;
      if (it == 100) err = 1;
    }
    for (int it = 1; it <= 100 && !dead && !err; ++it) {
      rnS = get_rn(muS);
      if (!(rnS > fill)) break;
      if (fabs(rnS - fill) > 0.5) muS -= 1.0;
      else if (fabs(rnS - fill) > dmu) muS -= 0.5;
      else muS -= dmu;
      if (it == 100) err = 1;
    }
  }
  st.muS = muS;
  st.muL = muL;
  st.bracket_valid = 1;
  rnL -= fill;
  rnS -= fill;
  double rnc = rnS, muc = muS, mud = 0.0, muM = 0.0, rnM = 0.0;
  bool flag = false;
  // inverse quadratic interpolation / bisection hybrid (fself.f90:623-654)
  for (int it = 1; it <= 100 && !dead && !err; ++it) {
    if (rnc != rnS && rnc != rnL)
      muM = (muL * rnS * rnc * (rnS - rnc) + muS * rnL * rnc * (rnc - rnL) + muc * rnL * rnS * (rnL - rnS)) /
            ((rnL - rnS) * (rnc - rnL) * (rnc - rnS));
    else
      muM = muL - rnL * (muL - muS) / (rnL - rnS);
    if ((0.25 * (3.0 * muS + muL) > muM || muM > muL) || (flag && fabs(muM - muL) >= fabs(muL - muc) * 0.5) ||
        (!flag && fabs(muM - muL) >= fabs(muc - mud) * 0.5) || (flag && fabs(muL - muc) < 1.0e-8) ||
        (!flag && fabs(muc - mud) < 1.0e-8)) {
      muM = (muL + muS) * 0.5;
      flag = true;
    } else {
      flag = false;
    }
    if (fabs(muL - muM) < eps) break;
    rnM = get_rn(muM);
    mud = muc;
    muc = muL;
    rnc = rnL;
    if (rnS * (rnM - fill) < 0) {
      muL = muM;
      rnL = rnM - fill;
    } else {
      muS = muM;
      rnS = rnM - fill;
    }
    if (fabs(rnS) < fabs(rnL)) {
      double t = muL;
      muL = muS;
      muS = t;
      t = rnL;
      rnL = rnS;
      rnS = t;
    }
    if (it == 100) err = 2;
  }
  if (!err && !dead) {
    mu = (rnL == rnS) ? (muS + muL) * 0.5 : (muS * rnL - muL * rnS) / (rnL - rnS);
    rnM = get_rn(mu);
  }
  // any block that gave up: the host starts again from the same state
  if (threadIdx.x == 0 && dead) atomicMax(&io->err, 3);
  if (threadIdx.x == 0 && blockIdx.x == 0 && !dead) {
    io->mu = io->mu_old = mu;
    io->muS = st.muS;
    io->muL = st.muL;
    io->bracket_valid = st.bracket_valid;
    io->cached = st.cached;
    io->filling = rnM;
    atomicMax(&io->err, err);
  }
}

template <int N>
void mu_launch(MuState* io, const double2* cp, double center, const double* eig, double fill, double esterr, double temp,
               int Nk, int Nw, double* part, unsigned* bar, long long wait, unsigned blocks, unsigned threads) {
  void* args[] = {&io, &cp, &center, &eig, &fill, &esterr, &temp, &Nk, &Nw, &part, &bar, &wait};
  PGB_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&k_mu_search<N>), dim3(blocks), dim3(threads),
                                       args, 0, ctx().stream));
}

}  // namespace

void charpoly_gk(double2* cp, const double2* hamk, const double2* sig, double center, double temp, int Nk, int Nw,
                 int Norb) {
  const long long K = (long long)Nk * Nw;
  const unsigned gb = grid_1d(K, 64, 1 << 20);
  switch (Norb) {
#define PGB_CP(n_) case n_: k_charpoly_gk<n_><<<gb, 64, 0, ctx().stream>>>(cp, hamk, sig, center, temp, Nk, Nw); break;
    PGB_CP(1) PGB_CP(2) PGB_CP(3) PGB_CP(4) PGB_CP(5) PGB_CP(6) PGB_CP(7) PGB_CP(8)
#undef PGB_CP
    default: throw Error("Norb above the engine limit of 8 orbitals");
  }
  count_launch("charpoly_gk");
}

void mu_search(MuState& s, const double2* cp, double center, const double* eig, double fill, double esterr, double temp,
               int Nk, int Nw, int Norb) {
  cudaStream_t st = ctx().stream;
  const long long K = (long long)Nk * Nw;
  // One block per SM at most (co-residency with other contexts' kernels).  A
  // trial is bound by the FP64 pipe, which a few warps per SM keep busy, so a small
  // problem spreads over the SMs (two warps at least) before a block gets more:
  // 16640 points at five orbitals on 9 blocks of 16 warps took 31 us a trial,
  // 12 us on 130 of two; 526336 at one orbital on 152 of 16 27 us, 21 us on 152 of 8.
  const long long per = 64 * 2;
  const unsigned blocks = (unsigned)std::max(1LL, std::min<long long>(ctx().num_sms, (K + per - 1) / per));
  const long long want = (K + 2LL * blocks - 1) / (2LL * blocks);
  const unsigned threads = (unsigned)std::max(64LL, std::min<long long>(kMuThreads, (want + 31) / 32 * 32));
  DBuf<MuState> io(1);
  DBuf<double> part(2 * blocks);
  DBuf<unsigned> bar(1);
  const MuState start = s;
  long long wait = mu_wait_cycles();
  for (int attempt = 1;; ++attempt) {
    s = start;
    bar.zero();
    io.upload(&s, 1);
    switch (Norb) {
#define PGB_MU(n_) case n_: mu_launch<n_>(io.p, cp, center, eig, fill, esterr, temp, Nk, Nw, part.p, bar.p, wait, blocks, threads); break;
      PGB_MU(1) PGB_MU(2) PGB_MU(3) PGB_MU(4) PGB_MU(5) PGB_MU(6) PGB_MU(7) PGB_MU(8)
#undef PGB_MU
      default: throw Error("Norb above the engine limit of 8 orbitals");
    }
    count_launch("mu_search");
    io.download(&s, 1);
    sync();
    if (s.err != 3 || attempt == kMuAttempts) break;
    wait = std::min(kMuWaitCycles, 8 * wait);
  }
  PGB_CHECK(s.err != 1, "Too many");
  PGB_CHECK(s.err != 2, "Too many loop!");
  PGB_CHECK(s.err == 0, "the chemical-potential search gave up a wait between its blocks");
}

}  // namespace pgb
