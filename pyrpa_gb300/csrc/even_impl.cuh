// Kernels and stages of even.cuh, instantiated per bulk type in even_*.cu.
#pragma once

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "even.cuh"
#include "fft_dev.cuh"
#include "flex_dev.cuh"

namespace pgb {
namespace {

// ------------------------------------------------------------ space transform
enum SpaceIn { kInPlain, kInBoson, kInFermi64, kInFermi, kInPostBoson, kInPostFermi, kInAny };
enum SpaceOut { kOutPlain, kOutChi, kOutSigma, kOutAny };  // kInAny, kOutAny: SpaceArgs says which
__host__ __device__ constexpr bool fermi_mode(int in) { return in == kInFermi || in == kInFermi64 || in == kInPostFermi; }

template <typename R> struct SpaceArgs {
  const void* src;
  void* dst;
  int nx, ny, nplanes;         // nplanes: planes per slot (1, or Nz/2 + 1)
  int H, Nk, Nw, sign;
  int in, out;                 // SpaceIn, SpaceOut
  int nst[2], radix[2][8];
  const cx<R>* tab[2];         // roots of nx and ny
  const cx<R>* root;           // roots of M (bosons) or 2M (fermions)
  const int *h_irr, *irr_h;
  const int *korder, *koff;    // irreducible k by plane of the half grid
  const int* el;               // boson in: element per array; fermion in / Sigma out: orbital element
  const R* stat;               // boson in: static part per array
  // chi out
  const int *mem, *memcj, *nmem;
  const cx<R>* J;              // per array; null without the tail
  const cx<R>* sawc;
  int full;
  // Sigma out
  const int* elt;              // transposed element
  const double* c0;            // constant per array
  double scale;
  int thresh;
};

// slot of block b: a slot and its partner of the pre/post-processing are
// neighbours in the launch, so that their common inputs meet in L2
__device__ __forceinline__ int boson_slot(int b, int Nw) { return (b & 1) ? (b + 1) >> 1 : (b ? Nw - (b >> 1) : 0); }
__device__ __forceinline__ int fermi_slot(int b, int Nw) { return (b & 1) ? Nw - 1 - (b >> 1) : (b >> 1); }

template <typename R>
__device__ __forceinline__ cx<R> pre_mix(cx<R> p, cx<R> q, cx<R> w) {
  return (p + q) + muli((p - q) * w, (R)1);
}
// F(j) from C(j) and C(partner): E + conj(w) O
template <typename R>
__device__ __forceinline__ cx<R> post_mix(cx<R> c, cx<R> cp, cx<R> w) {
  const R half = (R)0.5f;
  const cx<R> e = half * (c + conj(cp)), o = muli(half * (c - conj(cp)), (R)-1);
  return e + conj(w) * o;
}
template <typename R> __device__ __forceinline__ cx<R> from64(double2 v) { return cmk<R>((R)v.x, (R)v.y); }

// value of the space transform's input at half-grid point h of slot j
template <typename R, int IN>
__device__ __forceinline__ cx<R> space_load(const SpaceArgs<R>& a, int h, int j, int arr, cx<R> w, R stat) {
  if constexpr (IN == kInAny) {
    switch (a.in) {
      case kInBoson: return space_load<R, kInBoson>(a, h, j, arr, w, stat);
      case kInFermi64: return space_load<R, kInFermi64>(a, h, j, arr, w, stat);
      case kInFermi: return space_load<R, kInFermi>(a, h, j, arr, w, stat);
      case kInPostBoson: return space_load<R, kInPostBoson>(a, h, j, arr, w, stat);
      case kInPostFermi: return space_load<R, kInPostFermi>(a, h, j, arr, w, stat);
      default: return space_load<R, kInPlain>(a, h, j, arr, w, stat);
    }
  } else if constexpr (IN == kInBoson) {
    const cx<R>* v = static_cast<const cx<R>*>(a.src) + (long long)a.el[arr] * a.Nk * a.Nw + a.h_irr[h];
    // without the static part, which is a constant in the result (k_even_const)
    cx<R> p = v[(long long)a.Nk * j], q = cmk<R>((R)0, (R)0);
    p.x = p.x - stat;
    if (j) {
      q = conj(v[(long long)a.Nk * (a.Nw - j)]);
      q.x = q.x - stat;
    }
    return pre_mix<R>(p, q, w);
  } else if constexpr (IN == kInFermi64) {
    const double2* v = static_cast<const double2*>(a.src) + (long long)a.el[arr] * a.Nk * a.Nw + a.h_irr[h];
    return pre_mix<R>(from64<R>(v[(long long)a.Nk * j]), conj(from64<R>(v[(long long)a.Nk * (a.Nw - 1 - j)])), w);
  } else if constexpr (IN == kInFermi) {
    const cx<R>* v = static_cast<const cx<R>*>(a.src) + (long long)a.el[arr] * a.Nk * a.Nw + a.h_irr[h];
    return pre_mix<R>(v[(long long)a.Nk * j], conj(v[(long long)a.Nk * (a.Nw - 1 - j)]), w);
  } else {
    const cx<R>* v = static_cast<const cx<R>*>(a.src) + (long long)arr * a.H * a.Nw + h;
    const cx<R> c = v[(long long)a.H * j];
    if constexpr (IN == kInPostBoson) return post_mix<R>(c, v[(long long)a.H * (j ? a.Nw - j : 0)], w);
    if constexpr (IN == kInPostFermi) return post_mix<R>(c, v[(long long)a.H * (a.Nw - 1 - j)], w);
    return c;
  }
}

template <typename R> __device__ __forceinline__ cx<R> space_root(const SpaceArgs<R>& a, int in, int j) {
  if (in == kInPlain) return cmk<R>((R)0, (R)0);
  return twid<R>(a.root, fermi_mode(in) ? 2 * j + 1 : j, -1);
}

template <typename R>
__device__ __forceinline__ void space_store(const SpaceArgs<R>& a, int out, cx<R> v, int k, int j, int arr, cx<R> J, cx<R> saw) {
  const long long K = (long long)a.Nk * a.Nw, at = k + (long long)a.Nk * j;
  if (out == kOutChi) {
    cx<R>* chi = static_cast<cx<R>*>(a.dst);
    if (a.J) v += J * saw;
    if (abs_below(v.x, kThresh)) v.x = 0;
    if (abs_below(v.y, kThresh)) v.y = 0;
    const int n = (a.full || j == 0) ? a.nmem[arr] : 1;
    for (int i = 0; i < n; ++i) chi[a.mem[4 * arr + i] * K + at] = a.memcj[4 * arr + i] ? conj(v) : v;
  } else {
    double2* s = static_cast<double2*>(a.dst);
    double2 d = mkc((double)v.x, (double)v.y);
    d = a.scale * d;
    d.x += a.c0[arr];
    if (a.thresh) d = thresh(d);
    s[a.el[arr] * K + at] = d;
    if (a.elt[arr] != a.el[arr]) s[a.elt[arr] * K + at] = d;
  }
}

template <typename R, int N>
__device__ __forceinline__ void axis_stages(cx<R>*& in, cx<R>*& out, int L, int nl, int es, int ls, int nst,
                                            const int* radix, int sign, const cx<R>* tab) {
  if constexpr (N > 0) {
    stage_strided<R, 8>(in, out, N, 1, nl, es, ls, sign, tab);
    __syncthreads();
    stage_strided<R, N / 8>(out, in, N, 8, nl, es, ls, sign, tab);
    __syncthreads();
  } else {
    plane_axis<R, N < 0>(in, out, L, nl, es, ls, nst, radix, sign, tab);
  }
}

// One (x, y) plane of one slot and array per CTA.  HALF (2-D meshes): the half
// plane y <= Ny/2 of a function even in (x, y); rows are transformed in x,
// column x <= Nx/2 in y with its upper half read from the mirrored column, and
// the result is again even.  Otherwise the whole plane.  N: the compile-time
// side of square planes (0: sides of radices up to 8, -1: any sides).  The pre- and post-processing of the
// half-length time transform, the gather from the irreducible points and the
// scatter to them ride on the load and the store, so that no padded copy of
// the array exists.
template <typename R, int IN, int OUT, bool HALF, int N>
__global__ void __launch_bounds__(256) k_space(SpaceArgs<R> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = N > 0 ? N : a.nx, ny = N > 0 ? N : a.ny;
  const int mi = IN == kInAny ? a.in : IN, mo = OUT == kOutAny ? a.out : OUT;
  const int sx = nx + 1, rows = HALF ? ny / 2 + 1 : ny, nxc = nx / 2 + 1;
  const int buf = HALF ? (rows * sx > ny * nxc ? rows * sx : ny * nxc) : ny * sx;
  cx<R>* in = reinterpret_cast<cx<R>*>(smem_raw);
  cx<R>* out = in + buf;
  const int arr = blockIdx.y;
  const int b = HALF ? blockIdx.x : blockIdx.x / a.nplanes, z = HALF ? 0 : blockIdx.x % a.nplanes;
  const int j = fermi_mode(mi) ? fermi_slot(b, a.Nw) : boson_slot(b, a.Nw);
  const cx<R> w = space_root<R>(a, mi, j);
  const R stat = mi == kInBoson ? a.stat[arr] : (R)0;
  const int npl = rows * nx, h0 = z * npl;
  for (int e = threadIdx.x; e < npl; e += blockDim.x) {
    const int y = e / nx, x = e - y * nx;
    in[y * sx + x] = space_load<R, IN>(a, h0 + e, j, arr, w, stat);
  }
  __syncthreads();
  axis_stages<R, N>(in, out, nx, rows, 1, sx, a.nst[0], a.radix[0], a.sign, a.tab[0]);
  int cs = sx;
  if constexpr (HALF) {
    // columns x <= Nx/2, all rows: row y above Ny/2 is row Ny - y at -x
    for (int e = threadIdx.x; e < ny * nxc; e += blockDim.x) {
      const int y = e / nxc, x = e - y * nxc;
      out[e] = y < rows ? in[y * sx + x] : in[(ny - y) * sx + (x ? nx - x : 0)];
    }
    __syncthreads();
    cx<R>* t = in;
    in = out;
    out = t;
    cs = nxc;
    axis_stages<R, N>(in, out, ny, nxc, cs, 1, a.nst[1], a.radix[1], a.sign, a.tab[1]);
  } else {
    axis_stages<R, N>(in, out, ny, nx, cs, 1, a.nst[1], a.radix[1], a.sign, a.tab[1]);
  }
  auto at = [&](int x, int y) {
    if (HALF && x >= nxc) {
      x = nx - x;
      y = y ? ny - y : 0;
    }
    return in[y * cs + x];
  };
  if (mo == kOutPlain) {
    cx<R>* d = static_cast<cx<R>*>(a.dst) + (long long)arr * a.H * a.Nw + (long long)a.H * j + h0;
    for (int e = threadIdx.x; e < npl; e += blockDim.x) {
      const int y = e / nx, x = e - y * nx;
      d[e] = at(x, y);
    }
  } else {
    cx<R> J = cmk<R>((R)0, (R)0), saw = J;
    if (mo == kOutChi && a.J) {
      J = a.J[arr];
      saw = a.sawc[j];
    }
    const int k0 = a.koff[z], k1 = a.koff[z + 1];
    for (int i = k0 + threadIdx.x; i < k1; i += blockDim.x) {
      const int k = a.korder[i], h = a.irr_h[k] - h0;
      const int y = h / nx, x = h - y * nx;
      space_store<R>(a, mo, at(x, y), k, j, arr, J, saw);
    }
  }
}

template <typename R, int IN, int OUT>
void space_launch(const Even& ev, SpaceArgs<R>& a, int narr, int sign, cudaStream_t st) {
  a.nx = ev.nx;
  a.ny = ev.ny;
  a.H = ev.H;
  a.Nw = ev.Nw;
  a.sign = sign;
  a.h_irr = ev.h_irr.p;
  a.irr_h = ev.irr_h.p;
  a.korder = ev.korder.p;
  a.koff = ev.koff.p;
  a.nplanes = ev.three_d ? ev.nz / 2 + 1 : 1;
  PGB_CHECK(fft_factor(ev.nx, a.radix[0], &a.nst[0]) && fft_factor(ev.ny, a.radix[1], &a.nst[1]),
            "mesh side with a prime factor above 13");
  a.tab[0] = fft_roots<R>(ev.nx);
  a.tab[1] = fft_roots<R>(ev.ny);
  a.root = fft_roots<R>(fermi_mode(IN) ? 4 * ev.Nw : 2 * ev.Nw);
  a.in = IN;
  a.out = OUT;
  bool small = true;  // no radix above 8
  for (int x = 0; x < 2; ++x)
    for (int s = 0; s < a.nst[x]; ++s) small = small && a.radix[x][s] <= 8 && a.radix[x][s] != 7;
  const int rows = ev.three_d ? ev.ny : ev.ny / 2 + 1;
  const size_t buf = ev.three_d ? (size_t)ev.ny * (ev.nx + 1)
                                : std::max((size_t)rows * (ev.nx + 1), (size_t)ev.ny * (ev.nx / 2 + 1));
  const size_t smem = 2 * buf * sizeof(cx<R>);
  constexpr size_t lim = 200 * 1024;
  const dim3 grid((unsigned)(ev.Nw * a.nplanes), (unsigned)narr);
#define PGB_SPACE(IN_, OUT_, HALF_, N_)                                \
  do {                                                                 \
    PGB_SMEM_LIMIT_ONCE((k_space<R, IN_, OUT_, HALF_, N_>), lim);      \
    k_space<R, IN_, OUT_, HALF_, N_><<<grid, 256, smem, st>>>(a);      \
  } while (0)
  // the sides of most meshes with their stages and index arithmetic at compile
  // time; other sides choose stages and modes at run time, in a build that
  // leaves out the large radices (128 instead of 250 registers) where it can
  if (!ev.three_d && ev.nx == 64 && ev.ny == 64) PGB_SPACE(IN, OUT, true, 64);
  else if (!ev.three_d && ev.nx == 32 && ev.ny == 32) PGB_SPACE(IN, OUT, true, 32);
  else if (!ev.three_d && ev.nx == 16 && ev.ny == 16) PGB_SPACE(IN, OUT, true, 16);
  else if (ev.three_d && small) PGB_SPACE(kInAny, kOutAny, false, 0);
  else if (ev.three_d) PGB_SPACE(kInAny, kOutAny, false, -1);
  else if (small) PGB_SPACE(kInAny, kOutAny, true, 0);
  else PGB_SPACE(kInAny, kOutAny, true, -1);
#undef PGB_SPACE
  count_launch("even_space");
}

// The z axis of a 3-D mesh: each line pair (p, -p) of plane cells takes one
// transform of the whole axis, whose upper half is the mirrored line; with
// IN = post the halves of the time transform are taken apart on the load
// (both cells are still real there), into another array.
template <typename R, bool BIG>
__global__ void __launch_bounds__(256) k_zaxis(SpaceArgs<R> a, const int2* pairs, int npairs, int nz, int nst,
                                               SpaceArgs<R> rad, int lines) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nch = (npairs + lines - 1) / lines;
  const int b = blockIdx.x / nch, p0 = (blockIdx.x % nch) * lines, arr = blockIdx.y;
  const int nl = min(lines, npairs - p0), half = nz / 2 + 1, nxy = a.nx * a.ny;
  const int j = fermi_mode(a.in) ? fermi_slot(b, a.Nw) : boson_slot(b, a.Nw);
  const cx<R> w = space_root<R>(a, a.in, j);
  cx<R>* in = reinterpret_cast<cx<R>*>(smem_raw);
  cx<R>* out = in + lines * nz;
  for (int e = threadIdx.x; e < nl * nz; e += blockDim.x) {
    const int z = e / nl, l = e - z * nl;
    const int2 pp = pairs[p0 + l];
    const int h = z < half ? pp.x + nxy * z : pp.y + nxy * (nz - z);
    in[z * nl + l] = space_load<R, kInAny>(a, h, j, arr, w, (R)0);
  }
  __syncthreads();
  plane_axis<R, BIG>(in, out, nz, nl, nl, 1, nst, rad.radix[0], a.sign, rad.tab[0]);
  cx<R>* d = static_cast<cx<R>*>(a.dst) + (long long)arr * a.H * a.Nw + (long long)a.H * j;
  for (int e = threadIdx.x; e < nl * half; e += blockDim.x) {
    const int z = e / nl, l = e - z * nl;
    const int2 pp = pairs[p0 + l];
    d[pp.x + nxy * z] = in[z * nl + l];
    if (pp.y != pp.x) d[pp.y + nxy * z] = in[(z ? nz - z : 0) * nl + l];
  }
}

template <typename R, int IN>
void zaxis_launch(const Even& ev, const cx<R>* src, cx<R>* dst, int narr, int sign, cudaStream_t st) {
  SpaceArgs<R> a{}, rad{};
  a.src = src;
  a.dst = dst;
  a.nx = ev.nx;
  a.ny = ev.ny;
  a.H = ev.H;
  a.Nw = ev.Nw;
  a.sign = sign;
  a.root = fft_roots<R>(IN == kInPostFermi ? 4 * ev.Nw : 2 * ev.Nw);
  a.in = IN;
  PGB_CHECK(fft_factor(ev.nz, rad.radix[0], &rad.nst[0]), "mesh side with a prime factor above 13");
  rad.tab[0] = fft_roots<R>(ev.nz);
  const int lines = std::max(1, std::min(64, (int)(1536 / ev.nz)));
  const int nch = (ev.nzp + lines - 1) / lines;
  const size_t smem = 2 * (size_t)lines * ev.nz * sizeof(cx<R>);
  bool small = true;
  for (int s = 0; s < rad.nst[0]; ++s) small = small && rad.radix[0][s] <= 8 && rad.radix[0][s] != 7;
  const dim3 grid((unsigned)(ev.Nw * nch), (unsigned)narr);
  PGB_SMEM_LIMIT_ONCE((k_zaxis<R, false>), 64 * 1024);
  PGB_SMEM_LIMIT_ONCE((k_zaxis<R, true>), 64 * 1024);
  if (small) k_zaxis<R, false><<<grid, 256, smem, st>>>(a, ev.zpairs.p, ev.nzp, ev.nz, rad.nst[0], rad, lines);
  else k_zaxis<R, true><<<grid, 256, smem, st>>>(a, ev.zpairs.p, ev.nzp, ev.nz, rad.nst[0], rad, lines);
  count_launch("even_zaxis");
}

// forward transform of arrays that the load of IN makes from `src`
template <typename R, int IN>
void even_forward(const Even& ev, SpaceArgs<R> a, cx<R>* dst, int narr, bool time, cudaStream_t st) {
  a.dst = dst;
  space_launch<R, IN, kOutPlain>(ev, a, narr, -1, st);
  if (ev.three_d) zaxis_launch<R, kInPlain>(ev, dst, dst, narr, -1, st);
  if (time) fft_plan_t(ev.H, ev.Nw, (int)sizeof(cx<R>)).forward<R>(dst, narr, st);
}
// backward transform of T (overwritten); POST and OUT as in k_space
template <typename R, int POST, int OUT>
void even_backward(const Even& ev, SpaceArgs<R> a, cx<R>* T, cx<R>* T2, int narr, cudaStream_t st) {
  fft_plan_t(ev.H, ev.Nw, (int)sizeof(cx<R>)).backward<R>(T, narr, st);
  if (ev.three_d) {
    zaxis_launch<R, POST>(ev, T, T2, narr, 1, st);
    a.src = T2;
    space_launch<R, kInPlain, OUT>(ev, a, narr, 1, st);
  } else {
    a.src = T;
    space_launch<R, POST, OUT>(ev, a, narr, 1, st);
  }
}

// ---------------------------------------------------------- pointwise stages
// the half-integer phase of a transformed fermionic array: c *= e^{-i pi s/Nw}
template <typename R>
__global__ void k_even_phase(cx<R>* F, const cx<R>* root, const int* lt, int H, int Nw) {
  MeshTau q;
  if (!mesh_tau(H, Nw, q)) return;
  cx<R>* f = F + (long long)blockIdx.y * H * Nw + q.r;
  for (int p = q.t0; p < q.t1; ++p) f[(long long)H * p] = f[(long long)H * p] * twid<R>(root, lt[p], -1);
}

template <typename R>
void fermi_transform(const Even& ev, SpaceArgs<R> a, cx<R>* F, int narr, bool bulk, cudaStream_t st) {
  if (bulk) even_forward<R, kInFermi>(ev, a, F, narr, true, st);
  else even_forward<R, kInFermi64>(ev, a, F, narr, true, st);
  const FFT4D& ft = fft_plan_t(ev.H, ev.Nw, (int)sizeof(cx<R>));
  k_even_phase<R><<<mesh_tau_grid(ev.H, ev.Nw, narr), 256, 0, st>>>(F, fft_roots<R>(2 * ev.Nw), ft.d_logical(3), ev.H,
                                                                    ev.Nw);
  count_launch("even_phase");
}

// The reference bubble's tau kernel on the half grid (k_ref_tau's A): element
// (a <= b) at slots 2s and 2s+1 as the two parts of one number.  Its B is
// B(tau) = -A(beta - tau), read off A by k_even_product.
template <typename R, typename T>
__global__ void k_even_ref_tau(cx<R>* A, const T* gp, const cx<T>* cf, const int* h_irr, const int* sym_el, int H, int Nk,
                               int No, int Nw) {
  MeshTau q;
  if (!mesh_tau(H, Nw, q)) return;
  const int k = h_irr[q.r];
  const cx<T>* c = cf + ((long long)k * No * No + sym_el[blockIdx.y]) * No;
  const long long o = (long long)blockIdx.y * H * Nw + q.r;
  for (int s = q.t0; s < q.t1; ++s) {
    T a[2] = {(T)0, (T)0};
#pragma unroll
    for (int h = 0; h < 2; ++h)
      for (int n = 0; n < No; ++n) a[h] += gp[((long long)(2 * s + h) * No + n) * Nk + k] * c[n].x;
    A[o + (long long)H * s] = cmk<R>((R)a[0], (R)a[1]);
  }
}

// tau = 0 jump of the classes (tail_jump) from the band sums rb, in the bulk type
template <typename R>
__global__ void k_even_jump(cx<R>* J, const EvenPair* pairs, const double2* rb, int No, int nc) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const EvenPair p = pairs[c];
  double2 v = make_double2(0, 0);
  if (p.a13 == p.b13) v = v + rb[p.a42 + No * p.b42];
  if (p.a42 == p.b42) v = v - rb[p.a13 + No * p.b13];
  J[c] = cmk<R>((R)v.x, (R)v.y);
}

// static parts a S + b C of the classes' vertex
template <typename R>
__global__ void k_even_static(R* out, const double* S, const double* C, const int* cls_el, double a, double b, int nc) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < nc) out[c] = (R)(__dmul_rn(a, S[cls_el[c]]) + __dmul_rn(b, C[cls_el[c]]));
}

// chi0(r, tau) of the classes: G13(tau) G42(-tau) (both fermionic phases gone:
// their product is -1, except at tau = 0), minus G0's, minus the analytic bubble
template <typename R>
__global__ void k_even_product(cx<R>* out, const cx<R>* F, const cx<R>* F0, const cx<R>* A,
                               const EvenPair* pairs, int H, int Nw, const int* pos, const int* lt, R sc, R sr, R n0) {
  const EvenPair pr = pairs[blockIdx.y];
  const long long P = (long long)H * Nw;
  const cx<R>*a13 = F + pr.f13 * P, *b42 = F + pr.f42 * P;
  cx<R>* o = out + (long long)blockIdx.y * P;
  MeshTau q;
  if (!mesh_tau(H, Nw, q)) return;
  for (int p = q.t0; p < q.t1; ++p) {
    const int s = lt[p];
    const long long i = q.r + (long long)H * p, ie = q.r + (long long)H * pos[s ? Nw - s : 0],
                    io = q.r + (long long)H * pos[Nw - 1 - s];
    const cx<R> a = a13[i];
    R vx = a.x * b42[ie].x, vy = a.y * b42[io].y;
    if (F0) {
      const cx<R> a0 = F0[pr.f13 * P + i];
      vx = vx - a0.x * F0[pr.f42 * P + ie].x;
      vy = vy - a0.y * F0[pr.f42 * P + io].y;
    }
    if (s == 0) vx = -vx;
    vx = sc * vx;
    vy = sc * vy;
    if (A) {
      // B at slots 2s, 2s+1: minus A at slots 2(Nw-s), 2(Nw-1-s)+1; at tau = 0
      // the projectors' completeness, A(beta) = -delta_ab N delta_r0 - A(0)
      const cx<R> ta = A[pr.f13 * P + q.r + (long long)H * s], *u = A + pr.f42 * P + q.r;
      R bx = -u[(long long)H * (s ? Nw - s : 0)].x;
      if (s == 0) bx = (pr.a42 == pr.b42 && q.r == 0 ? n0 : (R)0) - bx;
      vx = vx - sr * (ta.x * bx);
      vy = vy + sr * (ta.y * u[(long long)H * (Nw - 1 - s)].y);
    }
    o[i] = cmk<R>(vx, vy);
  }
}

// Fermionic outputs sum_t w_t(r, tau) g_t(r, tau) of real factors, with the
// half-integer phase of the backward transform; the output runs fastest over the blocks, so
// that the outputs of one tile of points share its w and g in L2
template <typename R>
__global__ void k_even_contract(cx<R>* out, const cx<R>* W, const cx<R>* F, const EvenTerm* terms, const int* tb,
                                const cx<R>* root, int H, int Nw, const int* pos, const int* lt, int no) {
  const int o = (int)(blockIdx.x % (unsigned)no);
  const long long P = (long long)H * Nw;
  const unsigned tile = blockIdx.x / (unsigned)no, nrb = (unsigned)((H + 255) / 256), rb = tile % nrb;
  const int h = (int)(rb * 256u + threadIdx.x), p = (int)(tile / nrb);
  if (h >= H) return;
  const int s = lt[p];
  const long long i = h + (long long)H * p, ie = h + (long long)H * pos[s ? Nw - s : 0],
                  io = h + (long long)H * pos[Nw - 1 - s];
  R x = (R)0, y = (R)0;
  for (int t = tb[o]; t < tb[o + 1]; ++t) {
    const EvenTerm m = terms[t];
    const cx<R>* w = W + m.c * P;
    cx<R> g;
    if (m.rev & 2) {
      g = cmk<R>(F[m.f * P + ie].x, -F[m.f * P + io].y);
      if (s) g.x = -g.x;
    } else {
      g = F[m.f * P + i];
    }
    if (m.rev & 1) {
      x = mad(w[ie].x, g.x, x);
      y = mad(w[io].y, g.y, y);
    } else {
      const cx<R> v = w[i];
      x = mad(v.x, g.x, x);
      y = mad(v.y, g.y, y);
    }
  }
  out[o * P + i] = cmk<R>(x, y) * twid<R>(root, s, 1);
}

// What the static part of W gives an output: its transform is one spike at r = tau = 0,
// so a constant in (k, i omega).  The spike is as large as all frequencies together, and
// its rounding in the transforms was what FP32 Sigma's error came from: one orbital
// 16x16x256 1.06e-6 of its norm in this stage (general form 6.5e-7).
template <typename R>
__global__ void k_even_const(double* c0, const R* stat, const cx<R>* F, const EvenTerm* terms, const int* tb, long long P,
                             const int* pos, int H, double scale, int no) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= no) return;
  const long long at = (long long)H * pos[0];
  double s = 0.0;
  for (int t = tb[o]; t < tb[o + 1]; ++t) s += (double)stat[terms[t].c] * (double)F[terms[t].f * P + at].x;
  c0[o] = scale * s;
}

// ------------------------------------------------------------------- vertex
// Real-basis index tables.  vin, entry (row p, column q) at q N + p:
// value = ca t[a] + cb t[b] with t[2 c + part] the parts of class c's matrix
// element; word: see even.cuh.  vout, per class two
// words (real, imaginary part): value = cf (sa v[a] + sb v[b]) over the result
// v[q N + p]; word = a | b << 10 | (sa + 1) << 20 | (sb + 1) << 22 | (cf = 1/2) << 24.
__device__ __forceinline__ float real_mag(float a) { return fabsf(a); }
__device__ __forceinline__ float real_mag(double a) { return (float)fabs(a); }
__device__ __forceinline__ float real_mag(dfl a) { return fabsf(a.hi); }

template <typename R> __host__ __device__ constexpr int rrow_pad() { return sizeof(R) == 4 ? 4 : 2; }
template <typename R> __host__ __device__ constexpr int rrow_len(int n) { return (n + rrow_pad<R>() + 2) & ~3; }

// entries 1 .. N-1 of a row in 16-byte words (d aligned), and two of them back
template <typename R, int N> __device__ __forceinline__ void row_put(R* d, const R (&a)[N]) {
  if constexpr (sizeof(R) == 4) {
    float4* d4 = reinterpret_cast<float4*>(d);
#pragma unroll
    for (int s = 1; s < N; s += 4)
      d4[(s - 1) >> 2] = make_float4(a[s], s + 1 < N ? a[s + 1 < N ? s + 1 : 0] : 0.f,
                                     s + 2 < N ? a[s + 2 < N ? s + 2 : 0] : 0.f,
                                     s + 3 < N ? a[s + 3 < N ? s + 3 : 0] : 0.f);
  } else if constexpr (std::is_same<R, dfl>::value) {
    float4* d4 = reinterpret_cast<float4*>(d);
#pragma unroll
    for (int s = 1; s < N; s += 2) {
      const dfl b = s + 1 < N ? a[s + 1 < N ? s + 1 : 0] : dfl(0.f);
      d4[(s - 1) >> 1] = make_float4(a[s].hi, a[s].lo, b.hi, b.lo);
    }
  } else {
    double2* d2 = reinterpret_cast<double2*>(d);
#pragma unroll
    for (int s = 1; s < N; s += 2) d2[(s - 1) >> 1] = make_double2(a[s], s + 1 < N ? a[s + 1 < N ? s + 1 : 0] : 0.0);
  }
}
__device__ __forceinline__ void row_get(const double* d, double& a, double& b) {
  const double2 v = *reinterpret_cast<const double2*>(d);
  a = v.x;
  b = v.y;
}
__device__ __forceinline__ void row_get(const dfl* d, dfl& a, dfl& b) {
  const float4 v = *reinterpret_cast<const float4*>(d);
  a = dfl(v.x, v.y);
  b = dfl(v.z, v.w);
}
__device__ __forceinline__ void row_get(const float*, float&, float&) {}  // float rows go in fours

// Real warp_inverse_rot (flex.cu) of the group's matrix: lane i of a group of N
// lanes holds row i.  The pivot row goes through shared memory with entry s at
// s + pad - 1, so that entries 1.. start a 16-byte word.
template <typename R, int N>
__device__ __forceinline__ bool real_inverse_rot(R (&a)[N], R* prow, int* piv, int* pos, int& label, R& scale,
                                                 int base, int i, bool act) {
  constexpr int PAD = rrow_pad<R>(), PL = rrow_len<R>(N);
  label = i;
  scale = (R)0;
  bool ok = true;
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    const R ak = a[0];
    unsigned best = 0u;
    if (act && label >= k) {
      best = (__float_as_uint(real_mag(ak)) & ~31u) | (unsigned)(31 - label);
    }
    // the largest key of the group: one redux for a whole warp, else windows
    // of doubling width around the group (they may overlap: a maximum)
    if constexpr (N > 16) {
      best = __reduce_max_sync(0xffffffffu, best);
    } else {
#pragma unroll
      for (int off = 1; off < N; off <<= 1) {
        const int j = i + off;
        best = max(best, __shfl_sync(0xffffffffu, best, base + (j < N ? j : j - N)));
      }
    }
    const int plabel = 31 - (int)(best & 31u);
    if (act && !(__uint_as_float(best & ~31u) > 0.f)) ok = false;
    const bool is_piv = act && label == plabel;
    if (label == k) label = plabel;
    else if (is_piv) label = k;
    if (act && i == 0) piv[k] = plabel;
    R* buf = prow + (k & 1) * PL;
    if (is_piv) {
      buf[PAD - 1] = a[0];
      row_put<R, N>(buf + PAD, a);
    }
    __syncwarp();
    const R p = buf[PAD - 1];
    const R ip = ok ? (R)1 / p : (R)0;
    if (is_piv) scale = ip;
    const R f = is_piv ? (R)0 : -(ak * ip);
    if constexpr (sizeof(R) == 4) {
      const float4* b4 = reinterpret_cast<const float4*>(buf + PAD);
#pragma unroll
      for (int s = 1; s < N; s += 4) {
        const float4 v = b4[(s - 1) >> 2];
        a[s - 1] = mad(f, v.x, a[s]);
        if (s + 1 < N) a[s] = mad(f, v.y, a[s + 1]);
        if (s + 2 < N) a[s + 1] = mad(f, v.z, a[s + 2]);
        if (s + 3 < N) a[s + 2] = mad(f, v.w, a[s + 3]);
      }
    } else {
#pragma unroll
      for (int s = 1; s < N; s += 2) {
        R q0, q1;
        row_get(buf + PAD + s - 1, q0, q1);
        a[s - 1] = mad(f, q0, a[s]);
        if (s + 1 < N) a[s] = mad(f, q1, a[s + 1]);
      }
    }
    a[N - 1] = is_piv ? (R)1 : f;
  }
  __syncwarp();
  if (act) {
    int c = i;
#pragma unroll 1
    for (int k = N - 1; k >= 0; --k) {
      const int p = piv[k];
      if (c == k) c = p;
      else if (c == p) c = k;
    }
    pos[i] = c;
  }
  __syncwarp();
  return ok;
}

struct EvenVertexTabs {
  const int *vin, *vout, *rep, *mem, *memcj, *nmem;
  int ncls, nself, nplus, full;
  // the matrices to take, and their number; null: all of them
  const unsigned *list, *count;
};

// The FLEX vertex in the real basis.  A warp holds 32 / N matrices (one row per
// lane), a CTA stages a tile of them through shared memory; the accumulator of
// V is real.  consts: Si, Ci (inverses of S and C), D = S + C, S, C in the
// basis, row-major; D is dense on the nself same-orbital pairs and diagonal
// elsewhere.  FP64: bound by its pipe (91 % at N = 25, 33 ms for 263,168
// matrices; general form 122 ms, k_vertex_sym 22).  FP32: issue bound; predecoded source offsets,
// the pivot row in 16-byte stores and D's row in registers took 2.1 M matrices from
// 24.0 to 20.4 ms (general form 45 ms), D's product from the left through the transposed
// entries instead of five shuffles a column to 19.0.
template <typename R, int N, int W, int mode>
__global__ void __launch_bounds__(32 * W, sizeof(R) == 4 ? 4 : 2)
    k_vertex_even(cx<R>* chi, long long nmat, long long estride, const R* consts, EvenVertexTabs tb, int* err) {
  constexpr int G = 32 / N, T = W * G, TP = T + 1, PL = rrow_len<R>(N);
  if (tb.list) {
    nmat = *tb.count;
    if (nmat == 0) return;
  }
  extern __shared__ __align__(16) unsigned char smraw[];
  R* prow = reinterpret_cast<R*>(smraw);                    // [T][2][PL]
  cx<R>* tile = reinterpret_cast<cx<R>*>(prow + (size_t)T * 2 * PL);  // [ncls][TP]
  R* vb = reinterpret_cast<R*>(tile + (size_t)tb.ncls * TP);  // [T][N*N], entry (p, q) at q N + p
  R* cs = vb + (size_t)T * N * N;                            // Si, Ci (column-major), then D row-major
  int2* vin = reinterpret_cast<int2*>(cs + 3 * N * N + (N & 1));  // [N*N]
  int* pv = reinterpret_cast<int*>(vin + N * N);             // [T][N]
  int* ps = pv + T * N;                                      // [T][N]
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int p = e % N, q = e / N;  // stored column-major for the row-per-lane reads
    cs[e] = consts[p * N + q];
    cs[N * N + e] = consts[N * N + p * N + q];
    cs[2 * N * N + e] = consts[2 * N * N + e];
    // the two sources as offsets into the tile, with the signs in bit 31 and
    // "twice" in bit 30 of the first, "absent" in bit 30 of the second
    const int word = tb.vin[e];
    const int ia = src_a(word), ib = src_b(word), ca = src_ca(word), cb = src_cb(word);
    const unsigned oa = (unsigned)((ia >> 1) * TP * 2 + (ia & 1)), ob = (unsigned)((ib >> 1) * TP * 2 + (ib & 1));
    vin[e] = make_int2((int)(oa | (ca < 0 ? 1u << 31 : 0u) | (ca == 2 || ca == -2 ? 1u << 30 : 0u)),
                       (int)(ob | (cb < 0 ? 1u << 31 : 0u) | (cb == 0 ? 1u << 30 : 0u)));
  }
  const R* Sm = consts + 3 * N * N;
  const R* Cm = consts + 4 * N * N;
  const R* D = cs + 2 * N * N;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / N < G ? lane / N : 0;
  const bool act = lane < G * N;
  const int i = act ? lane - g * N : 0;
  const int t = w * G + g;
  R* pw = prow + (size_t)t * 2 * PL;
  R* vw = vb + (size_t)t * N * N;
  int *pvw = pv + t * N, *psw = ps + t * N;
  const R c1 = mode == 2 ? (R)-0.5f : (R)1.5f;
  const R c2 = mode == 0 ? (R)-0.5f : (R)0.5f;
  const R* tr = reinterpret_cast<const R*>(tile);
  for (long long m0 = (long long)blockIdx.x * T; m0 < nmat; m0 += (long long)gridDim.x * T) {
    const int nt = (int)min((long long)T, nmat - m0);
    __syncthreads();
    for (int idx = threadIdx.x; idx < tb.ncls * T; idx += blockDim.x) {
      const int tt = idx % T, e = idx / T;
      // matrices past the end repeat the last one: every group has a regular matrix
      const long long m = m0 + min(tt, nt - 1);
      tile[e * TP + tt] = chi[(tb.list ? tb.list[m] : m) + estride * tb.rep[e]];
    }
    __syncthreads();
    R a[N];
    const R* mine = tr + 2 * t;
    auto entry = [&](int q) {
      const int2 word = vin[q * N + i];
      R v = mine[word.x & 0x3fffffff];
      if (word.x < 0) v = -v;
      if (word.x & (1 << 30)) v = v + v;
      if (!(word.y & (1 << 30))) {
        const R u = mine[word.y & 0x3fffffff];
        v = v + (word.y < 0 ? -u : u);
      }
      return v;
    };
    int lab;
    R sc;
#pragma unroll
    for (int q = 0; q < N; ++q) a[q] = cs[q * N + i] - entry(q);
    bool ok = real_inverse_rot<R, N>(a, pw, pvw, psw, lab, sc, g * N, i, act);
    if (act) {
      const R s1 = c1 * sc;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const int c = psw[q];
        R v = s1 * a[q];
        if (mode == 1) v = v - Sm[lab * N + c];
        else if (mode == 2) v = v + (Sm[lab * N + c] - Cm[lab * N + c]);
        vw[c * N + lab] = v;
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < N; ++q) a[q] = cs[N * N + q * N + i] + entry(q);
    ok &= real_inverse_rot<R, N>(a, pw, pvw, psw, lab, sc, g * N, i, act);
    if (act) {
      const R s2 = c2 * sc;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const int c = psw[q];
        vw[c * N + lab] = vw[c * N + lab] + s2 * a[q];
      }
    }
    __syncwarp();
    if (mode == 0) {
      // -1/4 D X D: row i of X D, then D from the left
      const int ns = tb.nself;
#pragma unroll
      for (int q = 0; q < N; ++q) a[q] = entry(q);
      {
        R head[N < 8 ? N : 8];
        constexpr int NH = N < 8 ? N : 8;
#pragma unroll
        for (int q = 0; q < NH; ++q) head[q] = (R)0;
#pragma unroll
        for (int r = 0; r < NH; ++r)
          if (r < ns) {
#pragma unroll
            for (int q = 0; q < NH; ++q)
              if (q < ns) head[q] = mad(a[r], D[r * N + q], head[q]);
          }
#pragma unroll
        for (int q = 0; q < N; ++q) {
          if (q < NH && q < ns) a[q] = head[q < NH ? q : 0];
          else a[q] = a[q] * D[q * N + q];
        }
      }
      const R m4 = (R)-0.25f;
      const R dl = m4 * D[i * N + i];
      constexpr int NH = N < 8 ? N : 8;
      const bool head = i < ns;
      // D from the left mixes the ns same-orbital rows only.  Outside of their block
      // they are the columns of the others, row i entry q / row q entry i = h_i / h_q
      // with h = 1, 2, -2 for the three kinds of rows
      const R hi = (R)(i < tb.nplus ? 0.5f : -0.5f);
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const R v = dl * a[q];
        if (act && !head) {
          vw[q * N + i] = vw[q * N + i] + v;
          if (q < NH && q < ns) vw[i * N + q] = vw[i * N + q] + hi * v;
        }
      }
      R dh[NH];
#pragma unroll
      for (int r = 0; r < NH; ++r) dh[r] = r < ns ? m4 * D[i * N + r] : (R)0;
#pragma unroll
      for (int q = 0; q < NH; ++q) {
        if (q >= ns) continue;
        R sum = (R)0;
#pragma unroll
        for (int r = 0; r < NH; ++r)
          if (r < ns) sum = mad(dh[r], shfl_idx(a[q], g * N + r), sum);
        if (act && head) vw[q * N + i] = vw[q * N + i] + sum;
      }
    }
    if (!ok && act && t < nt) atomicExch(err, 3);
    __syncthreads();
    for (int idx = threadIdx.x; idx < tb.ncls * T; idx += blockDim.x) {
      const int tt = idx % T, e = idx / T;
      if (tt >= nt) continue;
      const R* v = vb + (size_t)tt * N * N;
      R part[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int word = tb.vout[2 * e + h];
        const R x = v[word & 1023], y = v[(word >> 10) & 1023];
        const int sa = ((word >> 20) & 3) - 1, sb = ((word >> 22) & 3) - 1;
        R r = sa == 0 ? (R)0 : (sa > 0 ? x : -x);
        if (sb) r = r + (sb > 0 ? y : -y);
        if (word >> 24) r = (R)0.5f * r;
        part[h] = r;
      }
      const cx<R> z = cmk<R>(part[0], part[1]);
      const int n = tb.full ? tb.nmem[e] : 1;
      const long long mat = tb.list ? tb.list[m0 + tt] : m0 + tt;
      for (int m = 0; m < n; ++m)
        chi[mat + estride * tb.mem[4 * e + m]] = tb.memcj[4 * e + m] ? conj(z) : z;
    }
  }
}

// The vertex of FP64 with the spin inverse (S^-1 - X)^-1 from the symmetric form of the
// real basis (even.cu, build_sym).  Row-per-lane elimination (k_vertex_even) spends N
// FMAs a row and step, and 7 of 32 lanes idle at N = 25; here
//  * a row keeps its N / 2 + 1 cyclic diagonals, in registers: half of the FMAs.
//    Row i needs entries i + d of the pivot column, which lies in shared memory twice
//    over, so that the offsets are constants;
//  * a warp works on G matrices, their rows dealt out over four register rows per lane:
//    125 of 128 at N = 25;
//  * the inverse is swept in place, M -> -M^-1 after every diagonal entry has been
//    the pivot once, the largest that is left each time: no interchanges.  A pivot
//    below an eighth of its column (an indefinite M, which no chi0 below its
//    instability gives) or not finite sends the matrix to k_vertex_even through `list`.
// The charge inverse keeps the row pivots: C's same-orbital block is indefinite (an
// eigenvalue -J among 2 U' - J + ...), and a sweep of C^-1 + X doubled the error of
// Sigma (four orbitals, 16x16x128: 1.5e-15 with row pivots, 3.5e-15 swept, of its norm).
// Bound by the FP64 pipe (75 % busy with both inverses swept).  Eight warps, two to a
// scheduler, are what shared memory holds at N = 25 if X is staged twice, in halves of the
// tile: 15.9 ms against 17.4 with six and X kept (263,168 matrices, both inverses swept).
constexpr int kSymRows = 4;
template <int N> __host__ __device__ constexpr int sym_group() { return 32 * kSymRows / N; }
template <int N> __host__ __device__ constexpr int sym_half() { return (N / 2 + 1) * N; }
template <int N> __host__ __device__ constexpr int sym_keys() { return (N + 3) & ~3; }
// place of entry (p, q); at even N the diagonal d = N / 2 holds its pairs twice, the
// first half is read
template <int N> __device__ __forceinline__ int sym_at(int p, int q) {
  const int d = q >= p ? q - p : q - p + N;
  return 2 * d < N || (2 * d == N && p < q) ? d * N + p : (N - d) * N + q;
}

// magnitude as an ordered integer; kSymExpo is a factor of two
__device__ __forceinline__ unsigned sym_mag(double a) { return (unsigned)__double2hiint(a) & 0x7fffffffu; }
constexpr unsigned kSymExpo = 1u << 20;

struct SymTabs {
  const int *sin, *sout, *rep, *mem, *memcj, *nmem;
  int ncls, nself, full;
  unsigned *list, *count;  // out: the matrices left to k_vertex_even
};

template <typename R, int N, int W> struct SymSmem {
  static constexpr int G = sym_group<N>(), T = W * G, TH = T / 2, HL = sym_half<N>(), KP = sym_keys<N>();
  static_assert(T % 2 == 0, "the tile is staged in two halves");
  static __host__ __device__ size_t tile(int ncls) { return sizeof(cx<R>) * (size_t)ncls * (TH + 1); }
  static constexpr int CS = (2 * HL + N * N + N + 65) & ~1;  // constants, an even number
  static __host__ __device__ size_t bytes(int ncls) {
    return tile(ncls) + sizeof(R) * ((size_t)T * HL + CS + T * (3 * N + 1)) +
           sizeof(int) * ((size_t)T * KP + HL + 3 * T + 64 * W);
  }
};

// consts: Si (as M) and the coefficients of the sandwich, HL entries each; Ci
// column-major, N^2; 1 / h, N; the nself x nself block of S + C, 64; then the W forms
// of S and C, HL each
template <typename R, int N, int W>
__global__ void __launch_bounds__(32 * W, N == 9 ? 2 : 1)
    k_vertex_sym(cx<R>* chi, long long nmat, long long estride, const R* consts, SymTabs tb, int mode, int* err) {
  using L = SymSmem<R, N, W>;
  constexpr int G = L::G, T = L::T, TH = L::TH, TP = TH + 1, HL = L::HL, KP = L::KP, DG = N / 2 + 1, SL = kSymRows;
  constexpr int DK = (N & 1) ? DG : DG - 1;  // diagonals that the pivot row publishes
  extern __shared__ __align__(16) unsigned char smraw[];
  cx<R>* tile = reinterpret_cast<cx<R>*>(smraw);  // [ncls][TP]: half of the matrices at a time
  unsigned* keys = reinterpret_cast<unsigned*>(smraw + L::tile(tb.ncls));  // [T][KP]
  R* xb = reinterpret_cast<R*>(keys + T * KP);                             // [T][HL]: X, then the result
  R* cst = xb + T * HL;
  const R *K = cst + HL, *Ci = cst + 2 * HL, *hinv = Ci + N * N, *qh = hinv + N;
  R* cbuf = cst + L::CS;       // [T][2N]
  R* diag = cbuf + T * 2 * N;  // [T][N]
  R* ipb = diag + T * N;       // [T]
  int* sin = reinterpret_cast<int*>(ipb + T);  // [HL]
  int* pvb = sin + HL;                         // [T]
  unsigned* pkb = reinterpret_cast<unsigned*>(pvb + T);  // [T]
  int* badb = reinterpret_cast<int*>(pkb + T);           // [T]
  int* perm = badb + T;                                  // [W][64]
  const int ns = tb.nself;
  for (int e = threadIdx.x; e < L::CS; e += blockDim.x) cst[e] = consts[e];
  for (int e = threadIdx.x; e < HL; e += blockDim.x) sin[e] = tb.sin[e];
  for (int e = threadIdx.x; e < T * KP; e += blockDim.x) keys[e] = 0u;
  const R *WS = consts + L::CS, *WC = WS + HL;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const R c1 = mode == 2 ? (R)0.5f : (R)-1.5f;  // of the swept -M^-1
  const R c2 = mode == 0 ? (R)-0.5f : (R)0.5f;
  // the lane's rows: matrix t (of the CTA's tile) and row i; rows past the last one
  // mirror it without writing
  int rt[SL], ri[SL];
  bool act[SL];
#pragma unroll
  for (int s = 0; s < SL; ++s) {
    const int r = s * 32 + lane, rr = min(r, G * N - 1);
    act[s] = r < G * N;
    rt[s] = w * G + rr / N;
    ri[s] = rr % N;
  }
  R a[SL][DG];
  // half h of the tile; matrices past the end repeat the last one, so that every row
  // belongs to a regular matrix
  auto stage = [&](long long m0, int nt, int h) {
    for (int idx = threadIdx.x; idx < tb.ncls * TH; idx += blockDim.x) {
      const int tt = idx % TH, e = idx / TH;
      tile[e * TP + tt] = chi[m0 + min(h * TH + tt, nt - 1) + estride * tb.rep[e]];
    }
    __syncthreads();
  };
  // entry e of the symmetric form of X, of matrix tt of the staged half
  auto entry = [&](int e, int tt) {
    const R* tr = reinterpret_cast<const R*>(tile) + 2 * tt;
    const int word = sin[e], ia = src_a(word), ib = src_b(word);
    R v = tr[2 * (ia >> 1) * TP + (ia & 1)];
    if (src_flag(word, 0)) v = -v;
    if (src_flag(word, 2)) {
      const R u = tr[2 * (ib >> 1) * TP + (ib & 1)];
      v = v + (src_flag(word, 1) ? -u : u);
    }
    if (src_flag(word, 3)) v = v + v;
    return v;
  };
  for (long long m0 = (long long)blockIdx.x * T; m0 < nmat; m0 += (long long)gridDim.x * T) {
    const int nt = (int)min((long long)T, nmat - m0);
    __syncthreads();
    if (threadIdx.x < T) badb[threadIdx.x] = 0;
    for (int h = 0; h < 2; ++h) {
      stage(m0, nt, h);
      for (int idx = threadIdx.x; idx < HL * TH; idx += blockDim.x) {
        const int tt = idx % TH, e = idx / TH;
        xb[(h * TH + tt) * HL + e] = entry(e, tt);
      }
      __syncthreads();
    }
    // (Si - X)^-1 by sweeps, into registers
#pragma unroll
    for (int s = 0; s < SL; ++s)
#pragma unroll
      for (int d = 0; d < DG; ++d) a[s][d] = cst[d * N + ri[s]] - xb[rt[s] * HL + d * N + ri[s]];
    unsigned done = 0u;
#pragma unroll
    for (int s = 0; s < SL; ++s)
      if (act[s]) {
        diag[rt[s] * N + ri[s]] = a[s][0];
        keys[rt[s] * KP + ri[s]] = (sym_mag(a[s][0]) & ~31u) | (unsigned)(31 - ri[s]);
      }
    __syncwarp();
#pragma unroll 1
    for (int step = 0; step < N; ++step) {
      if (lane < G) {
        const int t = w * G + lane;
        const uint4* k4 = reinterpret_cast<const uint4*>(keys + t * KP);
        unsigned best = 0u;
#pragma unroll
        for (int x = 0; x < KP / 4; ++x) {
          const uint4 v = k4[x];
          best = max(best, max(max(v.x, v.y), max(v.z, v.w)));
        }
        const int k = 31 - (int)(best & 31u);
        const unsigned ex = best / kSymExpo;
        if (ex == 0u || ex == 0x7fffffffu / kSymExpo) badb[t] = 1;  // zero, tiny or not finite
        pvb[t] = k;
        pkb[t] = best;
        ipb[t] = (R)1 / diag[t * N + k];
      }
      __syncwarp();
      int dd[SL];
#pragma unroll
      for (int s = 0; s < SL; ++s) {
        const int i = ri[s], x = pvb[rt[s]] - i;
        dd[s] = x < 0 ? x + N : x;
        if (!act[s]) continue;
        R* cb = cbuf + rt[s] * 2 * N;
        R c = a[s][0];
#pragma unroll
        for (int d = 1; d < DG; ++d) {
          const R x = a[s][d];
          c = d == dd[s] ? x : c;
        }
        if (dd[s] < DG) cb[i] = cb[i + N] = c;
        if (dd[s] == 0) {
#pragma unroll
          for (int d = 1; d < DK; ++d) {
            const int j = i + d < N ? i + d : i + d - N;
            cb[j] = cb[j + N] = a[s][d];
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int s = 0; s < SL; ++s) {
        const R* cb = cbuf + rt[s] * 2 * N + ri[s];
        const bool piv = dd[s] == 0;
        const R c = cb[0], ip = ipb[rt[s]];
        if (act[s] && !piv && !(done >> s & 1u) && sym_mag(c) > pkb[rt[s]] + 3u * kSymExpo) badb[rt[s]] = 1;
        const R f = piv ? ip : -(c * ip);
#pragma unroll
        for (int d = 0; d < DG; ++d) {
          const R v = mad(f, cb[d], piv ? (R)0 : a[s][d]);
          a[s][d] = d == dd[s] ? -f : v;
        }
        if (piv) done |= 1u << s;
        if (act[s]) {
          diag[rt[s] * N + ri[s]] = a[s][0];
          keys[rt[s] * KP + ri[s]] =
              (done >> s & 1u) ? 0u : ((sym_mag(a[s][0]) & ~31u) | (unsigned)(31 - ri[s]));
        }
      }
      __syncwarp();
    }
    // (Ci + X)^-1 with row pivots, 32 / N matrices of the warp at a time, over X
    constexpr int GP = 32 / N, PL = rrow_len<R>(N);
    const int gp = lane / N < GP ? lane / N : 0;
    const bool actp = lane < GP * N;
    const int ip = actp ? lane - gp * N : 0;
#pragma unroll 1
    for (int m = 0; m < G; m += GP) {
      const int t = w * G + min(m + gp, G - 1);
      const bool keep = actp && m + gp < G;
      R b[N];
#pragma unroll
      for (int q = 0; q < N; ++q) b[q] = mad(xb[t * HL + sym_at<N>(ip, q)], hinv[q], Ci[q * N + ip]);
      int lab;
      R sc;
      int* pp = perm + w * 64 + gp * 2 * N;
      const bool ok = real_inverse_rot<R, N>(b, cbuf + w * G * 2 * N + gp * 2 * PL, pp, pp + N, lab, sc, gp * N, ip, actp);
      if (!ok && keep && t < nt) atomicExch(err, 3);
      const R f = c2 * (sc * hinv[lab]);
      if (keep) {
#pragma unroll
        for (int q = 0; q < N; ++q) {
          const int c = pp[N + q], d = c >= lab ? c - lab : c - lab + N;
          if (2 * d < N || (2 * d == N && lab < c)) xb[t * HL + d * N + lab] = f * b[q];
        }
      }
      __syncwarp();
    }
#pragma unroll
    for (int s = 0; s < SL; ++s)
#pragma unroll
      for (int d = 0; d < DG; ++d) {
        const int e = d * N + ri[s];
        R* v = xb + rt[s] * HL + e;
        if (!act[s] || (2 * d == N && 2 * ri[s] >= N)) continue;
        R c = mad(c1, a[s][d], *v);
        if (mode == 1) c = c - WS[e];
        else if (mode == 2) c = c + (WS[e] - WC[e]);
        *v = c;
      }
    for (int h = 0; mode == 0 && h < 2; ++h) {
      // -1/4 (S + C) X (S + C), X staged once more (keeping it would take the shared
      // memory of two warps): S + C is dense on the ns same-orbital pairs, diagonal
      // elsewhere.  K: -1/4 and the products with the diagonal ones
      __syncthreads();
      stage(m0, nt, h);
      for (int idx = threadIdx.x; idx < HL * TH; idx += blockDim.x) {
        const int tt = idx % TH, e = idx / TH, p = e % N, q = p + e / N < N ? p + e / N : p + e / N - N;
        if (p < ns || q < ns) continue;
        R* v = xb + (h * TH + tt) * HL + e;
        *v = mad(K[e], entry(e, tt), *v);
      }
      auto add = [&](int t, int p, int q, R v) {
        const int e = sym_at<N>(p, q);
        xb[t * HL + e] = mad(K[e], v, xb[t * HL + e]);
      };
      // the dense block's rows, column j; its own columns go to z for the other side
      constexpr int NH = N < 8 ? N : 8;
      for (int idx = threadIdx.x; idx < TH * N; idx += blockDim.x) {
        const int tt = idx % TH, j = idx / TH, t = h * TH + tt;
        R* z = cbuf + t * 2 * N;
        R in[NH];
#pragma unroll
        for (int r = 0; r < NH; ++r) in[r] = r < ns ? entry(sym_at<N>(r, j), tt) : (R)0;
        for (int r = 0; r < ns; ++r) {
          R sum = (R)0;
#pragma unroll
          for (int q = 0; q < NH; ++q)
            if (q < ns) sum = mad(qh[r * ns + q], in[q], sum);
          if (j >= ns) add(t, r, j, sum);
          else z[j * ns + r] = sum;
        }
      }
      __syncthreads();
      for (int idx = threadIdx.x; idx < TH * ns * ns; idx += blockDim.x) {
        const int t = h * TH + idx % TH, p = idx / TH / ns, q = idx / TH % ns;
        if (p > q) continue;
        const R* z = cbuf + t * 2 * N;
        R sum = (R)0;
        for (int s = 0; s < ns; ++s) sum = mad(z[s * ns + p], qh[s * ns + q], sum);
        add(t, p, q, sum);
      }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < tb.ncls * T; idx += blockDim.x) {
      const int tt = idx % T, e = idx / T;
      if (tt >= nt || badb[tt]) continue;
      const R* v = xb + (size_t)tt * HL;
      R part[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int word = tb.sout[2 * e + h], sa = word >> 20 & 3, sb = word >> 22 & 3;
        R r = sa == 1 ? (R)0 : v[word & 1023];
        if (sa == 0) r = -r;
        if (sb != 1) {
          const R y = v[(word >> 10) & 1023];
          r = r + (sb == 0 ? -y : y);
        }
        part[h] = r;
      }
      const cx<R> z = cmk<R>(part[0], part[1]);
      const int n = tb.full ? tb.nmem[e] : 1;
      for (int m = 0; m < n; ++m)
        chi[m0 + tt + estride * tb.mem[4 * e + m]] = tb.memcj[4 * e + m] ? conj(z) : z;
    }
    if (threadIdx.x < nt && badb[threadIdx.x]) tb.list[atomicAdd(tb.count, 1u)] = (unsigned)(m0 + threadIdx.x);
  }
}

// A^-1 of a real matrix that host_inverse accepts, in the arithmetic of the kernels:
// their elimination of S^-1 -+ X then undoes these roundings.  The rounding of an exact
// C^-1 does not cancel like that; C^-1's same-orbital block has entries of 30 times its
// smallest eigenvalue, and the error is the same in every matrix, so that it adds up in
// Sigma.  A matrix that is singular in this arithmetic though not in FP64 (C of J within
// 1e-8 of U / 5, in FP32) takes `fp64`, its FP64 inverse, rounded.
template <typename R> std::vector<R> inverse_as(const std::vector<double>& X, const std::vector<double>& fp64, int n) {
  std::vector<R> A((size_t)n * n);
  for (size_t e = 0; e < A.size(); ++e) A[e] = (R)X[e];
  std::vector<int> piv(n);
  for (int k = 0; k < n; ++k) {
    int p = k;
    for (int r = k + 1; r < n; ++r)
      if (std::fabs((double)A[r * n + k]) > std::fabs((double)A[p * n + k])) p = r;
    piv[k] = p;
    if (p != k)
      for (int j = 0; j < n; ++j) std::swap(A[k * n + j], A[p * n + j]);
    const R d = (R)1 / A[k * n + k];
    A[k * n + k] = (R)1;
    for (int j = 0; j < n; ++j) A[k * n + j] = A[k * n + j] * d;
    for (int r = 0; r < n; ++r) {
      if (r == k) continue;
      const R f = A[r * n + k];
      A[r * n + k] = (R)0;
      for (int j = 0; j < n; ++j) A[r * n + j] = A[r * n + j] - f * A[k * n + j];
    }
  }
  for (int k = n - 1; k >= 0; --k)
    if (piv[k] != k)
      for (int r = 0; r < n; ++r) std::swap(A[r * n + k], A[r * n + piv[k]]);
  bool finite = true;
  for (const R& v : A) finite = finite && std::isfinite((double)v);
  if (!finite)
    for (size_t e = 0; e < A.size(); ++e) A[e] = (R)fp64[e];
  return A;
}

template <typename R, int N>
void vertex_even_launch(const Even& ev, cx<R>* chi, long long nmat, long long estride, const R* dc, int mode, bool full,
                        const unsigned* list = nullptr, const unsigned* count = nullptr) {
  constexpr int W = 8, T = W * (32 / N);
  const int nc = (int)ev.cls.size();
  const size_t smem = sizeof(R) * ((size_t)T * 2 * rrow_len<R>(N) + (size_t)T * N * N + 3 * N * N) +
                      sizeof(cx<R>) * (size_t)nc * (T + 1) + sizeof(R) + sizeof(int) * (2 * N * N + 2 * T * N);
  EvenVertexTabs tb{ev.d_vin.p, ev.d_vout.p, ev.cls_el.p, ev.mem.p, ev.memcj.p, ev.nmem.p, nc, ev.nself, ev.nplus, full ? 1 : 0,
                    list, count};
  const long long tiles = (nmat + T - 1) / T;
  const long long blocks = std::min<long long>(tiles, (long long)ctx().num_sms * 16);
#define PGB_VE(m_)                                                                                                      \
  do {                                                                                                                 \
    PGB_SMEM_LIMIT_ONCE((k_vertex_even<R, N, W, m_>), 220 * 1024);                                                     \
    k_vertex_even<R, N, W, m_><<<(unsigned)std::max(1LL, blocks), 32 * W, smem, ctx().stream>>>(chi, nmat, estride, dc, \
                                                                                               tb, ctx().err);         \
  } while (0)
  if (mode == 0) PGB_VE(0);
  else if (mode == 1) PGB_VE(1);
  else PGB_VE(2);
#undef PGB_VE
  count_launch("vertex_even");
}

// k_vertex_sym, then k_vertex_even on the matrices that it has left; false where a
// pair list's same-orbital block or classes do not fit its buffers
template <typename R, int N, int W>
bool vertex_sym_launch(const Even& ev, cx<R>* chi, long long nmat, long long estride, const R* dc, int mode, bool full) {
  using L = SymSmem<R, N, W>;
  constexpr int HL = L::HL;
  const int nc = (int)ev.cls.size(), ns = ev.nself;
  if (ns * ns > 2 * N || ns * ns > 64 || L::bytes(nc) > 220 * 1024 || nmat >= (1LL << 32)) return false;
  std::vector<R> c(L::CS + 2 * HL);
  std::vector<double> Si(ev.Sb), Ci(ev.Cb), Q((size_t)N * N);
  PGB_CHECK(host_inverse(Si, N) && host_inverse(Ci, N), "singular interaction matrix in the real-basis vertex");
  for (int e = 0; e < N * N; ++e) Q[e] = ev.Sb[e] + ev.Cb[e];
  for (int p = 0; p < N; ++p) {
    for (int d = 0; d <= N / 2; ++d) {
      const int q = (p + d) % N, e = d * N + p, pq = p * N + q;
      const double hp = ev.hsc[p], hq = ev.hsc[q];
      c[e] = (R)(Si[pq] * hq);
      // the rows of the dense block are multiplied through before
      c[HL + e] = (R)(-0.25 * (p < ns ? 1.0 : Q[p * N + p] / hp) * (q < ns ? 1.0 : Q[q * N + q] / hq));
      c[L::CS + e] = (R)(ev.Sb[pq] / hp);
      c[L::CS + HL + e] = (R)(ev.Cb[pq] / hp);
    }
    for (int q = 0; q < N; ++q) c[2 * HL + q * N + p] = (R)Ci[p * N + q];
    c[2 * HL + N * N + p] = (R)(1.0 / ev.hsc[p]);
  }
  for (int p = 0; p < ns; ++p)
    for (int q = 0; q < ns; ++q) c[2 * HL + N * N + N + p * ns + q] = (R)Q[p * N + q];
  DBuf<R> ds(c.size());
  ds.upload(c.data(), c.size());
  DBuf<unsigned> list(nmat);
  unsigned* count = reinterpret_cast<unsigned*>(ctx().err + 1);  // zeroed with the error flag
  PGB_SMEM_LIMIT_ONCE((k_vertex_sym<R, N, W>), 220 * 1024);
  SymTabs tb{ev.d_sin.p, ev.d_sout.p, ev.cls_el.p, ev.mem.p, ev.memcj.p, ev.nmem.p, nc, ns, full ? 1 : 0, list.p, count};
  const long long tiles = (nmat + L::T - 1) / L::T;
  const long long blocks = std::max(1LL, std::min<long long>(tiles, (long long)ctx().num_sms * 8));
  k_vertex_sym<R, N, W><<<(unsigned)blocks, 32 * W, L::bytes(nc), ctx().stream>>>(chi, nmat, estride, ds.p, tb, mode,
                                                                                        ctx().err);
  count_launch("vertex_sym");
  vertex_even_launch<R, N>(ev, chi, nmat, estride, dc, mode, full, list.p, count);
  return true;
}

// ------------------------------------------------------------------- stoner
// Largest eigenvalue of chi0(q, 0) S.  At nu = 0 the real-basis matrix X is
// symmetric and splits into two blocks (the sums with the same-orbital pairs,
// and the differences); with S = L L^T the eigenvalues of X S are those of
// K = L^T X L.  One warp per (q, block) reduces K to tridiagonal form
// (Householder) and finds its largest eigenvalue by 32-fold section with Sturm
// counts, all in FP64 and without a QR iteration.  514 q points of five
// orbitals take 0.25 ms against 7.4 ms for k_stoner's complex FP64 QR of X S and -X C.
constexpr int kEvenStonerWarps = 4;
__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename R>
__global__ void __launch_bounds__(32 * kEvenStonerWarps) k_stoner_even(double* out, const cx<R>* chi, const int* vin,
                                                                       const int* rep, const double* L, int Nk,
                                                                       long long K, int n, int nself, int nplus,
                                                                       int mx, int* err) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, ld = mx + 1;
  double* A = reinterpret_cast<double*>(smraw) + (size_t)w * (mx * ld + 3 * 32);
  double *d = A + mx * ld, *e2 = d + 32, *v = e2 + 32;
  const int t = blockIdx.x * kEvenStonerWarps + w;
  if (t >= 2 * Nk) return;
  const int k = t % Nk, blk = t / Nk, i0 = blk ? nplus : 0, m = blk ? n - nplus : nplus;
  if (m == 0) {
    if (lane == 0) out[t] = -1.0e300;
    return;
  }
  auto part = [&](int s) {
    const cx<R> c = chi[rep[s >> 1] * K + k];
    return (double)((s & 1) ? c.y : c.x);
  };
  // row `lane` of X L, then of L^T (X L)
  if (lane < m) {
    for (int q = 0; q < m; ++q) {
      const int word = vin[(i0 + q) * n + i0 + lane];
      const int ca = src_ca(word), cb = src_cb(word);
      double x = ca * part(src_a(word));
      if (cb) x += cb * part(src_b(word));
      const bool a = i0 + lane < nself, b = i0 + q < nself;
      if (a != b) x *= a ? 1.4142135623730951 : 0.70710678118654752;
      A[lane * ld + q] = x;
    }
  }
  __syncwarp();
  double row[32];
  if (lane < m)
    for (int q = 0; q < m; ++q) {
      double s = 0.0;
      for (int r = q; r < m; ++r) s = fma(A[lane * ld + r], L[(i0 + r) * n + i0 + q], s);
      row[q] = s;
    }
  __syncwarp();
  if (lane < m)
    for (int q = 0; q < m; ++q) A[lane * ld + q] = row[q];
  __syncwarp();
  if (lane < m)
    for (int q = 0; q < m; ++q) {
      double s = 0.0;
      for (int r = lane; r < m; ++r) s = fma(L[(i0 + r) * n + i0 + lane], A[r * ld + q], s);
      row[q] = s;
    }
  __syncwarp();
  if (lane < m)
    for (int q = 0; q < m; ++q) A[lane * ld + q] = row[q];
  __syncwarp();
  // tridiagonal form: A <- H A H, H = I - sc v v^T
  for (int c = 0; c + 2 < m; ++c) {
    const double x = (lane > c && lane < m) ? A[lane * ld + c] : 0.0;
    const double tail = wsum(lane > c + 1 ? x * x : 0.0);
    if (tail == 0.0) continue;
    const double x0 = __shfl_sync(0xffffffffu, x, c + 1);
    const double nrm = sqrt(fma(x0, x0, tail)), al = x0 > 0 ? -nrm : nrm;
    const double vl = lane == c + 1 ? x0 - al : x;
    v[lane] = vl;
    __syncwarp();
    const double sc = 2.0 / wsum(vl * vl);
    double p = 0.0;
    if (lane < m)
      for (int q = c + 1; q < m; ++q) p = fma(A[lane * ld + q], v[q], p);
    p *= sc;
    const double h = 0.5 * sc * wsum(p * vl);
    const double u = p - h * vl;
    d[lane] = u;  // scratch
    __syncwarp();
    if (lane < m)
      for (int q = c; q < m; ++q) {
        const double vq = q > c ? v[q] : 0.0;
        A[lane * ld + q] = A[lane * ld + q] - (vl * d[q] + u * vq);
      }
    __syncwarp();
    if (lane > c && lane < m) A[c * ld + lane] = A[lane * ld + c];
    __syncwarp();
  }
  double dl = 0.0, el = 0.0;
  if (lane < m) dl = A[lane * ld + lane];
  if (lane + 1 < m) el = A[lane * ld + lane + 1];
  __syncwarp();
  d[lane] = dl;
  e2[lane] = el * el;
  __syncwarp();
  // Gershgorin interval
  const double below = __shfl_up_sync(0xffffffffu, fabs(el), 1);
  const double rad = fabs(el) + (lane > 0 ? below : 0.0);
  double hi = lane < m ? dl + rad : -1e300, lo = lane < m ? dl : -1e300, ref = lane < m ? fabs(dl) + rad : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    lo = fmax(lo, __shfl_xor_sync(0xffffffffu, lo, o));  // the largest diagonal entry bounds it from below
    ref = fmax(ref, __shfl_xor_sync(0xffffffffu, ref, o));
  }
  const double tol = 4.4e-16 * ref;
  const bool bad = wsum(lane < m ? dl + el : 0.0) * 0.0 != 0.0;  // a NaN or an infinity in K
  for (int it = 0; it < 64 && !bad && hi - lo > tol; ++it) {
    // lane's point, and whether an eigenvalue lies above it: some pivot of T - x is not negative
    const double x = lo + (hi - lo) * ((lane + 1) * (1.0 / 33.0));
    double q = d[0] - x;
    bool above = q > 0.0;
    for (int i = 1; i < m; ++i) {
      if (q == 0.0) q = -1e-300;
      q = d[i] - x - e2[i - 1] / q;
      above |= q > 0.0;
    }
    const unsigned ab = __ballot_sync(0xffffffffu, above);
    const int na = ab ? 32 - __clz(ab) : 0;  // points 0 .. na-1 have one above
    const double nlo = na ? __shfl_sync(0xffffffffu, x, na - 1) : lo;
    const double nhi = na < 32 ? __shfl_sync(0xffffffffu, x, na) : hi;
    if (!(nhi < hi || nlo > lo)) break;
    lo = nlo;
    hi = nhi;
  }
  if (lane == 0) {
    if (bad) atomicExch(err, 2);
    out[t] = 0.5 * (lo + hi);
  }
}

template <typename To, typename From>
__global__ void k_convert_el(cx<To>* out, const cx<From>* in, const int* el, long long K) {
  const long long o = (long long)el[blockIdx.y] * K;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < K; i += (long long)gridDim.x * blockDim.x)
    cvt(out[o + i], in[o + i]);
}

}  // namespace

template <typename To, typename From>
void convert_even(const Even& ev, cx<To>* out, const cx<From>* in, long long K) {
  const unsigned nb = (unsigned)std::min<long long>((K + 255) / 256, 1024);
  k_convert_el<To, From><<<dim3(nb, (unsigned)ev.cls.size()), 256, 0, ctx().stream>>>(out, in, ev.cls_el.p, K);
  count_launch("convert_even");
}

// arrays per batch: about 64 MB, so that a batch stays in L2 from the pointwise
// kernel through the passes
template <typename R> int even_batch(const Even& ev) {
  const double bytes = (double)sizeof(cx<R>) * ev.H * ev.Nw;
  return (int)std::max(1.0, std::min(65535.0, 64e6 / bytes));
}

template <typename R>
void chi0_even(const Geom& g, const double2* G, double temp, const TailRef* tail, cx<R>* chi, bool full) {
  const Even& ev = *g.even;
  cudaStream_t st = ctx().stream;
  const int ns = ev.nsym, No = g.Norb, H = ev.H, Nw = ev.Nw;
  const size_t P = (size_t)H * Nw;
  DBuf<cx<R>> F(ns * P), F0, A, sawc, dJ;
  SpaceArgs<R> a{};
  a.Nk = g.Nk;
  a.src = G;
  a.el = ev.d_sym_el.p;
  fermi_transform<R>(ev, a, F.p, ns, false, st);
  const int nc = (int)ev.cls.size();
  if (tail) {
    DBuf<double2> G0((size_t)g.K * No * No);
    green0(G0.p, tail->eig, tail->uni, tail->mu, temp, g.Nk, g.Nw, No, true);
    F0.alloc(ns * P);
    a.src = G0.p;
    fermi_transform<R>(ev, a, F0.p, ns, false, st);
    G0.release();
    using T = typename std::conditional<std::is_same<R, float>::value, float, double>::type;
    TailTables<T> tt;
    tail_tables<T>(g, *tail, temp, tt, false);
    A.alloc(ns * P);
    k_even_ref_tau<R, T><<<mesh_tau_grid(H, Nw, ns), 256, 0, st>>>(A.p, tt.gp.p, tt.projectors(), ev.h_irr.p,
                                                                  ev.d_sym_el.p, H, g.Nk, No, Nw);
    count_launch("even_ref_tau");
    SpaceArgs<R> r{};
    r.Nk = g.Nk;
    r.src = A.p;
    even_forward<R, kInPlain>(ev, r, A.p, ns, false, st);
    DBuf<double2> rb(No * No);
    tail_rhobar(g, *tail, tt.ff.p, rb.p);
    dJ.alloc(nc);
    k_even_jump<R><<<(nc + 127) / 128, 128, 0, st>>>(dJ.p, ev.pairs.p, rb.p, No, nc);
    count_launch("even_jump");
    sawc.alloc(g.Nw);
    narrow<R>(sawc.p, tail_sawtooth(g, temp), g.Nw);
  }
  const int ch = std::min(nc, even_batch<R>(ev));
  DBuf<cx<R>> T(ch * P), T2;
  if (ev.three_d) T2.alloc(ch * P);
  const FFT4D& ft = fft_plan_t(H, Nw, (int)sizeof(cx<R>));
  const double P4 = (double)g.P;
  const R sc = (R)(temp / (double)g.Nkall / P4), sr = (R)(1.0 / (temp * (double)g.Nkall) / P4);
  SpaceArgs<R> o{};
  o.Nk = g.Nk;
  o.dst = chi;
  o.sawc = sawc.p;
  o.full = full ? 1 : 0;
  for (int c0 = 0; c0 < nc; c0 += ch) {
    const int n = std::min(ch, nc - c0);
    k_even_product<R><<<mesh_tau_grid(H, Nw, n), 256, 0, st>>>(T.p, F.p, F0.p, A.p, ev.pairs.p + c0, H, Nw, ft.d_pos(3),
                                                               ft.d_logical(3), sc, sr, (R)(double)g.Nkall);
    count_launch("even_product");
    o.mem = ev.mem.p + 4 * c0;
    o.memcj = ev.memcj.p + 4 * c0;
    o.nmem = ev.nmem.p + c0;
    o.J = tail ? dJ.p + c0 : nullptr;
    even_backward<R, kInPostBoson, kOutChi>(ev, o, T.p, T2.p, n, st);
  }
}

// transforms of the classes' vertex elements V without their static parts stat = a S + b C
template <typename R>
void vertex_transforms(const Geom& g, const cx<R>* V, const double* S, const double* C, double wS, double wC, cx<R>* W,
                       DBuf<R>& stat, cudaStream_t st) {
  const Even& ev = *g.even;
  const int nc = (int)ev.cls.size(), ch = even_batch<R>(ev);
  const size_t P = (size_t)ev.H * ev.Nw;
  stat.alloc(nc);
  k_even_static<R><<<(nc + 127) / 128, 128, 0, st>>>(stat.p, S, C, ev.cls_el.p, wS, wC, nc);
  count_launch("even_static");
  SpaceArgs<R> b{};
  b.Nk = g.Nk;
  b.src = V;
  for (int c0 = 0; c0 < nc; c0 += ch) {
    b.el = ev.cls_el.p + c0;
    b.stat = stat.p + c0;
    even_forward<R, kInBoson>(ev, b, W + c0 * P, std::min(ch, nc - c0), true, st);
  }
}

template <typename R>
void sigma_even(const Geom& g, const double2* G, const cx<R>* V, const double* S, const double* C,
                double temp, double2* sig) {
  const Even& ev = *g.even;
  cudaStream_t st = ctx().stream;
  const int ns = ev.nsym, H = ev.H, Nw = ev.Nw, nc = (int)ev.cls.size();
  const size_t P = (size_t)H * Nw;
  PGB_CHECK(ev.sig_tb.n == (size_t)ns + 1, "the even form's pair list has no Sigma terms");
  DBuf<cx<R>> F(ns * P), W((size_t)nc * P), T(ns * P), T2;
  if (ev.three_d) T2.alloc(ns * P);
  SpaceArgs<R> a{};
  a.Nk = g.Nk;
  a.src = G;
  a.el = ev.d_sym_el.p;
  fermi_transform<R>(ev, a, F.p, ns, false, st);
  DBuf<R> stat;
  DBuf<double> c0(ns);
  vertex_transforms<R>(g, V, S, C, 1.5, -0.5, W.p, stat, st);
  const FFT4D& ft = fft_plan_t(H, Nw, (int)sizeof(cx<R>));
  const unsigned tiles = (unsigned)(((H + 255) / 256) * Nw);
  k_even_contract<R><<<tiles * ns, 256, 0, st>>>(T.p, W.p, F.p, ev.sig_terms.p, ev.sig_tb.p, fft_roots<R>(2 * Nw), H, Nw, ft.d_pos(3),
                                                ft.d_logical(3), ns);
  count_launch("even_contract");
  SpaceArgs<R> o{};
  o.Nk = g.Nk;
  o.dst = sig;
  o.el = ev.d_sym_el.p;
  o.elt = ev.d_sym_elt.p;
  o.scale = temp / (double)g.Nkall / (double)g.P;
  o.thresh = 1;
  o.c0 = c0.p;
  k_even_const<R><<<(ns + 31) / 32, 32, 0, st>>>(c0.p, stat.p, F.p, ev.sig_terms.p, ev.sig_tb.p, (long long)P, ft.d_pos(3), H,
                                                o.scale * (double)g.P, ns);
  count_launch("even_const");
  even_backward<R, kInPostFermi, kOutSigma>(ev, o, T.p, T2.p, ns, st);
}

template <typename R>
void mkdelta_even(const Geom& g, const Pairs& p, const double2* F64, const cx<R>* Fbulk, const cx<R>* Vd,
                  const double* S, const double* C, double scale, double2* out, DeltaKernelCache<R>& cache) {
  const Even& ev = *g.even;
  cudaStream_t st = ctx().stream;
  const int ns = ev.nsym, No = g.Norb, Nchi = g.Nchi, H = ev.H, Nw = ev.Nw, nc = (int)ev.cls.size();
  const size_t P = (size_t)H * Nw;
  if (!cache.built) {
    cache.built = true;
    cache.W.alloc((size_t)nc * P);
    vertex_transforms<R>(g, Vd, S, C, 0.5, 0.5, cache.W.p, cache.stat, st);
    std::vector<EvenTerm> terms;
    std::vector<int> tb(1, 0), el;
    for (int e = 0; e < No * No; ++e) {
      if (p.delta[e].empty()) continue;
      for (const Term& t : p.delta[e]) {
        const int x = t.m + Nchi * t.l, a = t.ef % No, b = t.ef / No;
        // F_ba = conj F_ab: the copy of a <= b at the reversed tau
        terms.push_back(EvenTerm{ev.cls_of[x], ev.sym_of[t.ef], ev.cj_of[x] | (a > b ? 2 : 0)});
      }
      tb.push_back((int)terms.size());
      el.push_back(e);
    }
    cache.out_elems = el;
    cache.ef.alloc(3 * std::max<size_t>(1, terms.size()));
    cache.ef.upload(terms.data(), 3 * terms.size());
    cache.tb.alloc(tb.size());
    cache.tb.upload(tb.data(), tb.size());
    el.insert(el.end(), ev.sym_el.begin(), ev.sym_el.end());
    cache.els.alloc(el.size());
    cache.els.upload(el.data(), el.size());
    sync();
  }
  const int no = (int)cache.out_elems.size();
  DBuf<cx<R>> F(ns * P), T((size_t)std::max(1, no) * P), T2;
  if (ev.three_d) T2.alloc((size_t)std::max(1, no) * P);
  SpaceArgs<R> a{};
  a.Nk = g.Nk;
  a.src = Fbulk ? static_cast<const void*>(Fbulk) : F64;
  a.el = cache.els.p + no;
  fermi_transform<R>(ev, a, F.p, ns, Fbulk != nullptr, st);
  PGB_CUDA(cudaMemsetAsync(out, 0, sizeof(double2) * (size_t)g.K * No * No, st));
  if (no > 0) {
    const FFT4D& ft = fft_plan_t(H, Nw, (int)sizeof(cx<R>));
    const unsigned tiles = (unsigned)(((H + 255) / 256) * Nw);
    k_even_contract<R><<<tiles * no, 256, 0, st>>>(T.p, cache.W.p, F.p, reinterpret_cast<const EvenTerm*>(cache.ef.p),
                                                  cache.tb.p, fft_roots<R>(2 * Nw), H, Nw, ft.d_pos(3),
                                                  ft.d_logical(3), no);
    count_launch("even_contract");
    SpaceArgs<R> o{};
    o.Nk = g.Nk;
    o.dst = out;
    o.el = o.elt = cache.els.p;
    o.scale = scale;
    DBuf<double> c0(no);
    o.c0 = c0.p;
    k_even_const<R><<<(no + 31) / 32, 32, 0, st>>>(c0.p, cache.stat.p, F.p, reinterpret_cast<const EvenTerm*>(cache.ef.p),
                                                  cache.tb.p, (long long)P, ft.d_pos(3), H, scale * (double)g.P, no);
    count_launch("even_const");
    even_backward<R, kInPostFermi, kOutSigma>(ev, o, T.p, T2.p, no, st);
  }
  hermitize(out, g.K, No);
}

template <typename R>
bool vertex_even(const Even& ev, cx<R>* chi, long long nmat, long long estride, int mode, bool full) {
  const int n = (int)ev.perm.size();
  std::vector<double> Si(ev.Sb), Ci(ev.Cb);
  PGB_CHECK(host_inverse(Si, n) && host_inverse(Ci, n), "singular interaction matrix in the real-basis vertex");
  std::vector<R> Sr(Si.size(), (R)0), Cr(Sr);
  if (n > 1) {
    Sr = inverse_as<R>(ev.Sb, Si, n);
    Cr = inverse_as<R>(ev.Cb, Ci, n);
  } else {
    Sr[0] = (R)Si[0];
    Cr[0] = (R)Ci[0];
  }
  std::vector<R> consts(5 * n * n);
  for (int e = 0; e < n * n; ++e) {
    consts[e] = Sr[e];
    consts[n * n + e] = Cr[e];
    consts[2 * n * n + e] = (R)(ev.Sb[e] + ev.Cb[e]);
    consts[3 * n * n + e] = (R)ev.Sb[e];
    consts[4 * n * n + e] = (R)ev.Cb[e];
  }
  DBuf<R> dc(consts.size());
  dc.upload(consts.data(), consts.size());
  reset_err();
  // FP64, where the pipe bounds an elimination, takes k_vertex_sym: three orbitals
  // 32x32x512 (263,168 matrices) 2.74 -> 1.73 ms, four 32x32x256 (131,584) 4.43 -> 3.32,
  // five 16.6 -> 11.0.  In double-float its bookkeeping takes as long as it saves
  // (N = 9 even, 16 slower), FP32 and N <= 4 are bound by instructions of other kinds.
  if constexpr (std::is_same<R, double>::value) {
    bool done = false;
    if (n == 9) done = vertex_sym_launch<R, 9, 8>(ev, chi, nmat, estride, dc.p, mode, full);
    if (n == 16) done = vertex_sym_launch<R, 16, 8>(ev, chi, nmat, estride, dc.p, mode, full);
    if (n == 25) done = vertex_sym_launch<R, 25, 8>(ev, chi, nmat, estride, dc.p, mode, full);
    if (done) return fetch_err() == 0;
  }
  switch (n) {
    case 1: vertex_even_launch<R, 1>(ev, chi, nmat, estride, dc.p, mode, full); break;
    case 4: vertex_even_launch<R, 4>(ev, chi, nmat, estride, dc.p, mode, full); break;
    case 9: vertex_even_launch<R, 9>(ev, chi, nmat, estride, dc.p, mode, full); break;
    case 16: vertex_even_launch<R, 16>(ev, chi, nmat, estride, dc.p, mode, full); break;
    case 25: vertex_even_launch<R, 25>(ev, chi, nmat, estride, dc.p, mode, full); break;
    default: throw Error("no real-basis vertex for this number of orbital pairs");
  }
  return fetch_err() == 0;
}

template <typename R>
bool stoner_even(const Geom& g, const cx<R>* chi, std::vector<double>& out) {
  const Even& ev = *g.even;
  const int n = g.Nchi, mx = std::max(ev.nplus, n - ev.nplus);
  DBuf<double> d(2 * (size_t)g.Nk);
  reset_err();
  const size_t smem = (size_t)kEvenStonerWarps * (mx * (mx + 1) + 3 * 32) * sizeof(double);
  PGB_SMEM_LIMIT_ONCE(k_stoner_even<R>, 64 * 1024);
  const unsigned blocks = (unsigned)((2LL * g.Nk + kEvenStonerWarps - 1) / kEvenStonerWarps);
  k_stoner_even<R><<<blocks, 32 * kEvenStonerWarps, smem, ctx().stream>>>(
      d.p, chi, ev.d_vin.p, ev.cls_el.p, ev.d_schol.p, g.Nk, g.K, n, ev.nself, ev.nplus, mx, ctx().err);
  count_launch("stoner_even");
  std::vector<double> h(2 * (size_t)g.Nk);
  d.download(h.data(), h.size());
  const bool ok = fetch_err() == 0;
  out.resize(g.Nk);
  for (int k = 0; k < g.Nk; ++k) out[k] = std::max(h[k], h[g.Nk + k]);
  return ok;
}

#define PGB_EVEN_INST(R)                                                                                              \
  template void chi0_even<R>(const Geom&, const double2*, double, const TailRef*, cx<R>*, bool);         \
  template void sigma_even<R>(const Geom&, const double2*, const cx<R>*, const double*, const double*,   \
                              double, double2*);                                                                      \
  template void mkdelta_even<R>(const Geom&, const Pairs&, const double2*, const cx<R>*, const cx<R>*, const double*,  \
                                const double*, double, double2*, DeltaKernelCache<R>&);                               \
  template bool vertex_even<R>(const Even&, cx<R>*, long long, long long, int, bool);                                 \
  template bool stoner_even<R>(const Geom&, const cx<R>*, std::vector<double>&);

}  // namespace pgb
