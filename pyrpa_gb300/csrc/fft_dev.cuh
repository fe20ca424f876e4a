// Device building blocks of the FFT kernels: roots, radix butterflies and the
// Stockham stages over lines in shared memory.
#pragma once

#include "fft.cuh"

namespace pgb {
namespace {

// tab[t] = exp(-2 pi i t / L); sign < 0 uses it as is, sign > 0 its conjugate
template <typename R>
__device__ __forceinline__ cx<R> twid(const cx<R>* tab, int t, int sign) {
  cx<R> w = __ldg(tab + t);
  return cmk<R>(w.x, sign < 0 ? w.y : -w.y);
}
template <typename R> __device__ __forceinline__ const cx<R>* line_tab(const PassDesc& d);
template <> __device__ __forceinline__ const double2* line_tab<double>(const PassDesc& d) { return d.tw_line; }
template <> __device__ __forceinline__ const float2* line_tab<float>(const PassDesc& d) { return d.tw_line_f; }
template <typename R> __device__ __forceinline__ const cx<R>* full_tab(const PassDesc& d);
template <> __device__ __forceinline__ const double2* full_tab<double>(const PassDesc& d) { return d.tw_full; }
template <> __device__ __forceinline__ const float2* full_tab<float>(const PassDesc& d) { return d.tw_full_f; }
template <> __device__ __forceinline__ const cdf* line_tab<dfl>(const PassDesc& d) { return d.tw_line_d; }
template <typename R> __device__ __forceinline__ const cx<R>* line_tab_y(const PassDesc& d);
template <> __device__ __forceinline__ const double2* line_tab_y<double>(const PassDesc& d) { return d.tw_line_y; }
template <> __device__ __forceinline__ const float2* line_tab_y<float>(const PassDesc& d) { return d.tw_line_y_f; }
template <> __device__ __forceinline__ const cdf* line_tab_y<dfl>(const PassDesc& d) { return d.tw_line_y_d; }
template <> __device__ __forceinline__ const cdf* full_tab<dfl>(const PassDesc& d) { return d.tw_full_d; }
// double-float roots: one 16-byte read-only load {re.hi, re.lo, im.hi, im.lo}
template <> __device__ __forceinline__ cdf twid<dfl>(const cdf* tab, int t, int sign) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(tab + t));
  return mkc(dfl(v.x, v.y), sign < 0 ? dfl(v.z, v.w) : dfl(-v.z, -v.w));
}

// Butterfly sums.  For float and double the plain sum.  For double-float the
// sum of the high words by two-sum plus the low words, without the final
// renormalization (8 flops instead of Dekker's 11): the radix-4 and radix-8
// butterflies chain two or three of these and renormalize their outputs
// once (bnorm).  Within a butterfly the low word stays a few units in the
// last place of the high word, so the normwise error stays a few 2^-47
// (|a| + |b|), as for the renormalized sum.
__device__ __forceinline__ float2 badd(float2 a, float2 b) { return a + b; }
__device__ __forceinline__ float2 bsub(float2 a, float2 b) { return a - b; }
__device__ __forceinline__ float2 bnorm(float2 a) { return a; }
__device__ __forceinline__ double2 badd(double2 a, double2 b) { return a + b; }
__device__ __forceinline__ double2 bsub(double2 a, double2 b) { return a - b; }
__device__ __forceinline__ double2 bnorm(double2 a) { return a; }
__device__ __forceinline__ dfl lazy_add(dfl a, dfl b) {
  const dfl s = two_sum(a.hi, b.hi);
  return dfl(s.hi, s.lo + (a.lo + b.lo));
}
__device__ __forceinline__ cdf badd(cdf a, cdf b) { return mkc(lazy_add(a.x, b.x), lazy_add(a.y, b.y)); }
__device__ __forceinline__ cdf bsub(cdf a, cdf b) { return mkc(lazy_add(a.x, -b.x), lazy_add(a.y, -b.y)); }
__device__ __forceinline__ cdf bnorm(cdf a) {
  return mkc(fast_two_sum(a.x.hi, a.x.lo), fast_two_sum(a.y.hi, a.y.lo));
}

template <typename R, int RAD> struct Dft {
  // generic radix: direct O(RAD^2) evaluation with roots from the line table
  __device__ static void run(cx<R>* v, int sign, const cx<R>* tab, int L) {
    cx<R> o[RAD];
    const int step = L / RAD;
#pragma unroll
    for (int k = 0; k < RAD; ++k) {
      cx<R> acc = v[0];
#pragma unroll
      for (int r = 1; r < RAD; ++r) acc += v[r] * twid<R>(tab, ((r * k) % RAD) * step, sign);
      o[k] = acc;
    }
#pragma unroll
    for (int k = 0; k < RAD; ++k) v[k] = o[k];
  }
};

template <typename R> struct Dft<R, 2> {
  __device__ static void run(cx<R>* v, int, const cx<R>*, int) {
    cx<R> a = v[0] + v[1], b = v[0] - v[1];
    v[0] = a;
    v[1] = b;
  }
};

template <typename R> struct Dft<R, 4> {
  // outputs left unrenormalized (the radix-8 butterfly goes on with them)
  __device__ static void run_lazy(cx<R>* v, int sign) {
    cx<R> a0 = badd(v[0], v[2]), a1 = bsub(v[0], v[2]), a2 = badd(v[1], v[3]);
    cx<R> a3 = muli(bsub(v[1], v[3]), (R)sign);
    v[0] = badd(a0, a2);
    v[1] = badd(a1, a3);
    v[2] = bsub(a0, a2);
    v[3] = bsub(a1, a3);
  }
  __device__ static void run(cx<R>* v, int sign, const cx<R>*, int) {
    run_lazy(v, sign);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = bnorm(v[k]);
  }
};

template <typename R> struct Dft<R, 3> {
  __device__ static void run(cx<R>* v, int sign, const cx<R>*, int) {
    const R h = (R)0.86602540378443864676372317075294;  // sqrt(3)/2
    cx<R> t1 = v[1] + v[2], t2 = v[1] - v[2];
    cx<R> m = v[0] - (R)0.5 * t1;
    cx<R> u = h * muli(t2, (R)sign);
    v[0] = v[0] + t1;
    v[1] = m + u;
    v[2] = m - u;
  }
};

template <typename R> struct Dft<R, 5> {
  __device__ static void run(cx<R>* v, int sign, const cx<R>*, int) {
    const R c1 = (R)0.30901699437494742410229341718282;   // cos(2 pi/5)
    const R c2 = (R)-0.80901699437494742410229341718282;  // cos(4 pi/5)
    const R s1 = (R)0.95105651629515357211643933337938;   // sin(2 pi/5)
    const R s2 = (R)0.58778525229247312916870595463907;   // sin(4 pi/5)
    cx<R> a1 = v[1] + v[4], b1 = v[1] - v[4], a2 = v[2] + v[3], b2 = v[2] - v[3];
    cx<R> p1 = v[0] + c1 * a1 + c2 * a2, p2 = v[0] + c2 * a1 + c1 * a2;
    cx<R> q1 = muli(s1 * b1 + s2 * b2, (R)sign), q2 = muli(s2 * b1 - s1 * b2, (R)sign);
    v[0] = v[0] + a1 + a2;
    v[1] = p1 + q1;
    v[4] = p1 - q1;
    v[2] = p2 + q2;
    v[3] = p2 - q2;
  }
};

template <typename R> struct Dft<R, 8> {
  __device__ static void run(cx<R>* v, int sign, const cx<R>* t, int L) {
    const R h = (R)0.70710678118654752440084436210485;
    cx<R> e[4] = {v[0], v[2], v[4], v[6]};
    cx<R> o[4] = {v[1], v[3], v[5], v[7]};
    Dft<R, 4>::run_lazy(e, sign);
    Dft<R, 4>::run_lazy(o, sign);
    const R s = (R)sign;
    // o1 = o[1] (h + i s h), o3 = o[3] (-h + i s h): a sum and a difference
    // times h instead of a full complex product (fewer double-word operations)
    const cx<R> a1 = o[1], a3 = o[3];
    cx<R> o1, o3;
    if (sign > 0) {
      o1 = h * cmk<R>(a1.x - a1.y, a1.x + a1.y);
      o3 = h * cmk<R>(-(a3.x + a3.y), a3.x - a3.y);
    } else {
      o1 = h * cmk<R>(a1.x + a1.y, a1.y - a1.x);
      o3 = h * cmk<R>(a3.y - a3.x, -(a3.x + a3.y));
    }
    const cx<R> o2 = muli(o[2], s);
    v[0] = bnorm(badd(e[0], o[0]));
    v[4] = bnorm(bsub(e[0], o[0]));
    v[1] = bnorm(badd(e[1], o1));
    v[5] = bnorm(bsub(e[1], o1));
    v[2] = bnorm(badd(e[2], o2));
    v[6] = bnorm(bsub(e[2], o2));
    v[3] = bnorm(badd(e[3], o3));
    v[7] = bnorm(bsub(e[3], o3));
  }
};

// One Stockham stage (Govindaraju et al., "High performance discrete Fourier
// transforms on graphics processors", SC08, Fig. 2) over nl lines in smem.
template <typename R, int RAD>
__device__ void stage(const cx<R>* in, cx<R>* out, int L, int Ns, int nl, int sign,
                      const cx<R>* tab) {
  const int nbf = L / RAD;
  const int total = nl * nbf;
  const int tstride = L / (Ns * RAD);
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int b = idx / nbf;
    const int j = idx - b * nbf;
    const cx<R>* li = in + (size_t)b * L;
    cx<R>* lo = out + (size_t)b * L;
    const int jj = j % Ns;
    cx<R> v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) {
      v[r] = li[j + r * nbf];
      if (r > 0 && jj > 0) v[r] = v[r] * twid<R>(tab, r * jj * tstride, sign);
    }
    Dft<R, RAD>::run(v, sign, tab, L);
    const int idxD = (j / Ns) * Ns * RAD + jj;
#pragma unroll
    for (int r = 0; r < RAD; ++r) lo[idxD + r * Ns] = v[r];
  }
}

// The same stage over nl lines whose line b starts at b * ls and whose
// element j sits at j * es (the plane pass's rows and columns).
template <typename R, int RAD>
__device__ void stage_strided(const cx<R>* in, cx<R>* out, int L, int Ns, int nl, int es, int ls, int sign,
                              const cx<R>* tab) {
  const int nbf = L / RAD;
  const int total = nl * nbf;
  const int tstride = L / (Ns * RAD);
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int b = idx / nbf;
    const int j = idx - b * nbf;
    const cx<R>* li = in + (size_t)b * ls;
    cx<R>* lo = out + (size_t)b * ls;
    const int jj = j % Ns;
    cx<R> v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) {
      v[r] = li[(size_t)(j + r * nbf) * es];
      if (r > 0 && jj > 0) v[r] = v[r] * twid<R>(tab, r * jj * tstride, sign);
    }
    Dft<R, RAD>::run(v, sign, tab, L);
    const int idxD = (j / Ns) * Ns * RAD + jj;
#pragma unroll
    for (int r = 0; r < RAD; ++r) lo[(size_t)(idxD + r * Ns) * es] = v[r];
  }
}

// All stages of one axis of the plane, ping-ponging in/out (swapped on return
// so that `in` holds the result).  BIG: with the radices 7, 11 and 13.
template <typename R, bool BIG = true>
__device__ void plane_axis(cx<R>*& in, cx<R>*& out, int L, int nl, int es, int ls, int nst, const int* radix,
                           int sign, const cx<R>* tab) {
  int Ns = 1;
  for (int st = 0; st < nst; ++st) {
    const int rad = radix[st];
    switch (rad) {
      case 2: stage_strided<R, 2>(in, out, L, Ns, nl, es, ls, sign, tab); break;
      case 3: stage_strided<R, 3>(in, out, L, Ns, nl, es, ls, sign, tab); break;
      case 4: stage_strided<R, 4>(in, out, L, Ns, nl, es, ls, sign, tab); break;
      case 5: stage_strided<R, 5>(in, out, L, Ns, nl, es, ls, sign, tab); break;
      case 7:
        if constexpr (BIG) stage_strided<R, 7>(in, out, L, Ns, nl, es, ls, sign, tab);
        break;
      case 8: stage_strided<R, 8>(in, out, L, Ns, nl, es, ls, sign, tab); break;
      case 11:
        if constexpr (BIG) stage_strided<R, 11>(in, out, L, Ns, nl, es, ls, sign, tab);
        break;
      case 13:
        if constexpr (BIG) stage_strided<R, 13>(in, out, L, Ns, nl, es, ls, sign, tab);
        break;
      default: break;
    }
    __syncthreads();
    cx<R>* t = in;
    in = out;
    out = t;
    Ns *= rad;
  }
}

}  // namespace
}  // namespace pgb
