// Helpers shared by the kernel files: array indices, the small-part zeroing,
// the device error flag, launch grids.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "flex.cuh"

namespace pgb {
namespace {

constexpr double kPi = 3.141592653589793238462643383279;
constexpr double kThresh = 1.0e-9;  // small-part zeroing of chi0 and Sigma (fchi.f90:483-506)

__host__ __device__ __forceinline__ long long fidx(long long k, long long j, long long a, long long b,
                                                   long long Nk, long long Nw, long long n) {
  return k + Nk * (j + Nw * (a + n * b));
}

template <typename T> __device__ __forceinline__ T thresh(T v) {
  if (fabs((double)v.x) < kThresh) v.x = 0;
  if (fabs((double)v.y) < kThresh) v.y = 0;
  return v;
}

// every launch of a flag-raising kernel follows a reset_err on its context
inline void reset_err() {
  PGB_CHECK(ctx().err != nullptr, "the engine context is not set up (no device error flag)");
  PGB_CUDA(cudaMemsetAsync(ctx().err, 0, 2 * sizeof(int), ctx().stream));
}
inline int fetch_err() {
  int e[2] = {0, 0};
  PGB_CUDA(cudaMemcpyAsync(e, ctx().err, sizeof(e), cudaMemcpyDeviceToHost, ctx().stream));
  sync();
  ctx().pivoted_vertices += e[1];
  return e[0];
}

inline void count_launch(const char* what) {
  launch_check(what);
  ctx().kernel_launches++;
}

inline unsigned grid_1d(long long n, int threads, long long cap = 1LL << 30) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (unsigned)b;
}

// ====================================================== mesh x time grids ==
// Kernels over a padded array of P = Nkall x M points (mesh point r fastest)
// give each thread one mesh point r and up to kTauChunk consecutive slices t
// (blocks of 256 threads: the mesh in blocks, then the slices in chunks).
// The mesh index is split once per thread in 32-bit arithmetic, and the
// per-point tables (grid_irr, grid_flag, reversed indices) are read once;
// a grid-stride loop over P would split every element's index with 64-bit
// divisions, which on GB300 cost far more than the element's own loads.
constexpr int kTauChunk = 8;

inline dim3 mesh_tau_grid(long long Nkall, long long M, unsigned ny, int chunk = kTauChunk) {
  const long long nrb = (Nkall + 255) / 256, nch = (M + chunk - 1) / chunk;
  return dim3((unsigned)(nrb * nch), ny);
}

struct MeshTau {
  int r, t0, t1;
};
__device__ __forceinline__ bool mesh_tau(long long Nkall, long long M, MeshTau& q, int chunk = kTauChunk) {
  const unsigned nrb = (unsigned)((Nkall + 255) / 256);
  const unsigned rb = blockIdx.x % nrb, tc = blockIdx.x / nrb;
  q.r = (int)(rb * 256u + threadIdx.x);
  q.t0 = (int)tc * chunk;
  q.t1 = min((int)M, q.t0 + chunk);
  return q.r < Nkall;
}

// conversions between bulk types (double-float <-> float without the FP64 pipe)
__device__ __forceinline__ void cvt(float2& o, float2 v) { o = v; }
__device__ __forceinline__ void cvt(double2& o, double2 v) { o = v; }
__device__ __forceinline__ void cvt(cdf& o, cdf v) { o = v; }
__device__ __forceinline__ void cvt(float2& o, double2 v) { o = make_float2((float)v.x, (float)v.y); }
__device__ __forceinline__ void cvt(double2& o, float2 v) { o = make_double2(v.x, v.y); }
__device__ __forceinline__ void cvt(cdf& o, float2 v) { o = mkc(dfl(v.x), dfl(v.y)); }
__device__ __forceinline__ void cvt(float2& o, cdf v) { o = make_float2(v.x.hi + v.x.lo, v.y.hi + v.y.lo); }
__device__ __forceinline__ void cvt(cdf& o, double2 v) { o = mkc(dfl(v.x), dfl(v.y)); }
__device__ __forceinline__ void cvt(double2& o, cdf v) { o = make_double2((double)v.x, (double)v.y); }

// host inverse of a small real matrix (row-major), false if (nearly) singular
inline bool host_inverse(std::vector<double>& A, int n) {
  std::vector<int> piv(n);
  double amax = 0;
  for (double v : A) amax = std::max(amax, std::fabs(v));
  for (int k = 0; k < n; ++k) {
    int p = k;
    for (int r = k + 1; r < n; ++r)
      if (std::fabs(A[r * n + k]) > std::fabs(A[p * n + k])) p = r;
    piv[k] = p;
    if (std::fabs(A[p * n + k]) <= 1e-12 * std::max(amax, 1e-300)) return false;
    if (p != k)
      for (int j = 0; j < n; ++j) std::swap(A[k * n + j], A[p * n + j]);
    const double d = 1.0 / A[k * n + k];
    A[k * n + k] = 1.0;
    for (int j = 0; j < n; ++j) A[k * n + j] *= d;
    for (int r = 0; r < n; ++r) {
      if (r == k) continue;
      const double f = A[r * n + k];
      A[r * n + k] = 0.0;
      for (int j = 0; j < n; ++j) A[r * n + j] -= f * A[k * n + j];
    }
  }
  for (int k = n - 1; k >= 0; --k)
    if (piv[k] != k)
      for (int r = 0; r < n; ++r) std::swap(A[r * n + k], A[r * n + piv[k]]);
  return true;
}

}  // namespace
}  // namespace pgb
