// C ABI of the GB300 engine: the symbols of the reference libfmod.so that the
// pyrpa ctypes wrappers (libs/flibs/*.py) bind, with the same argument order
// and meaning (every argument by reference, Fortran column-major arrays).
// Declarations and the reference interface each one replaces: include/fmod.h.
//
// Differences from the reference on purpose: a failure prints a message,
// records it for pyrpa_gb_last_error() and fills the outputs with NaN instead
// of terminating the process (the Fortran code calls `stop`).
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <limits>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "drivers.cuh"
#include "even.cuh"
#include "flex.cuh"
#include "linalg.cuh"
#include "lws.cuh"

namespace pgb {

static Context& process_context() {
  static Context c;
  return c;
}
// the calling thread's own context, if it asked for one
static thread_local Context* t_context = nullptr;
// thread contexts no thread holds, for reuse (streams and flag slots are kept)
static std::mutex g_thread_ctx_mu;
static std::vector<Context*> g_thread_ctx_free;
static int g_thread_ctx_made = 0;

Context& ctx() { return t_context ? *t_context : process_context(); }

void ensure_context() {
  if (t_context) return;  // thread contexts are made ready
  Context& c = process_context();
  if (c.ready) return;
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0)
    throw Error("no CUDA device is visible: this library runs the FLEX/RPA path only on the GPU");
  PGB_CUDA(cudaGetDevice(&c.device));
  cudaDeviceProp prop;
  PGB_CUDA(cudaGetDeviceProperties(&prop, c.device));
  c.num_sms = prop.multiProcessorCount;
  PGB_CUDA(cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking));
  cudaMemPool_t pool;
  PGB_CUDA(cudaDeviceGetDefaultMemPool(&pool, c.device));
  uint64_t thr = std::numeric_limits<uint64_t>::max();
  PGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr));
  if (const char* s = std::getenv("PYRPA_GB_PRECISION")) {
    std::string v(s);
    if (v == "32" || v == "fp32" || v == "FP32") c.precision = 32;
    if (v == "3264" || v == "mixed" || v == "MIXED") c.precision = kPrecMixed;
    if (v == "48" || v == "df" || v == "DF") c.precision = kPrecDF;
  }
  if (const char* s = std::getenv("PYRPA_GB_VERBOSE")) c.verbose = std::atoi(s);
  if (const char* s = std::getenv("PYRPA_GB_ARNOLDI_TOL")) c.arnoldi_tol = std::atof(s);
  c.err = err_slot_address(0);
  c.ready = true;
}

// Gives the calling thread a context of its own (on != 0) or hands it back
// (on == 0).  The thread context copies the process context's settings, and
// later settings calls from this thread change only it.
void set_thread_context(bool on) {
  if (on) {
    if (t_context) return;
    ensure_context();
    const Context& pc = process_context();
    Context* c = nullptr;
    {
      std::lock_guard<std::mutex> lk(g_thread_ctx_mu);
      if (!g_thread_ctx_free.empty()) {
        c = g_thread_ctx_free.back();
        g_thread_ctx_free.pop_back();
      } else {
        if (g_thread_ctx_made + 1 >= kErrSlots)
          throw Error("more than " + std::to_string(kErrSlots - 1) + " thread contexts at once");
        c = new Context();
        c->err = err_slot_address(++g_thread_ctx_made);
        PGB_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
      }
    }
    c->device = pc.device;
    c->num_sms = pc.num_sms;
    c->precision = pc.precision;
    c->verbose = pc.verbose;
    c->arnoldi_tol = pc.arnoldi_tol;
    c->kernel_launches = 0;
    c->pivoted_vertices = 0;
    c->ready = true;
    t_context = c;
  } else {
    if (!t_context) return;
    PGB_CUDA(cudaStreamSynchronize(t_context->stream));
    std::lock_guard<std::mutex> lk(g_thread_ctx_mu);
    g_thread_ctx_free.push_back(t_context);
    t_context = nullptr;
  }
}

}  // namespace pgb

using namespace pgb;

namespace {

// the last failure of an entry point called from this thread
thread_local std::string g_last_error;
thread_local int64_t g_last_code = 0;

void report(const char* fn, const char* what, int64_t code = 1) {
  g_last_error = std::string(fn) + ": " + what;
  g_last_code = code;
  fprintf(stderr, "pyrpa_gb300 error in %s: %s\n", fn, what);
  fflush(stderr);
}

template <typename T> void nan_fill(T* p, size_t n) {
  if (!p) return;
  const double q = std::numeric_limits<double>::quiet_NaN();
  double* d = reinterpret_cast<double*>(p);
  for (size_t i = 0; i < n * sizeof(T) / sizeof(double); ++i) d[i] = q;
}

void nan_fill_f(float* p, size_t n) {
  if (!p) return;
  for (size_t i = 0; i < n; ++i) p[i] = std::numeric_limits<float>::quiet_NaN();
}

// FP32 bulk for every entry point except FP64 mode (the mixed schedule only
// changes the FLEX loop)
bool fp32() { return ctx().precision == 32 || ctx().precision == kPrecMixed; }

// --------------------------------------------------------- setup kernels
__global__ void k_gen_ham(double2* hk, const double* klist, const double2* hr, const double* rvec, int64_t Nk,
                          int64_t Nr, int No) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < Nk; i += (long long)gridDim.x * blockDim.x) {
    double2 acc[kMaxOrb * kMaxOrb];
    for (int e = 0; e < No * No; ++e) acc[e] = make_double2(0, 0);
    for (long long j = 0; j < Nr; ++j) {
      const double d = klist[3 * i] * rvec[3 * j] + klist[3 * i + 1] * rvec[3 * j + 1] + klist[3 * i + 2] * rvec[3 * j + 2];
      double s, c;
      sincospi(2.0 * d, &s, &c);
      const double2 ph = make_double2(c, -s);
      for (int l = 0; l < No; ++l)
        for (int m = l; m < No; ++m) acc[m + No * l] += hr[m + No * (l + (long long)No * j)] * ph;
    }
    double2* out = hk + (long long)No * No * i;
    for (int l = 0; l < No; ++l) {
      out[l + No * l] = make_double2(acc[l + No * l].x, 0.0);
      for (int m = l + 1; m < No; ++m) {
        out[m + No * l] = acc[m + No * l];
        out[l + No * m] = conj(acc[m + No * l]);
      }
    }
  }
}

__global__ void k_get_eig(double* eig, double2* uni, const double2* hk, int64_t Nk, int No) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < Nk; i += (long long)gridDim.x * blockDim.x) {
    double2 A[kMaxOrb * kMaxOrb], V[kMaxOrb * kMaxOrb];
    double w[kMaxOrb];
    const double2* h = hk + (long long)No * No * i;
    for (int m = 0; m < No; ++m)
      for (int l = 0; l < No; ++l) A[m * No + l] = h[m + No * l];
    jacobi_herm(A, No, w, V);
    for (int n = 0; n < No; ++n) {
      eig[n + (long long)No * i] = w[n];
      for (int m = 0; m < No; ++m) uni[m + No * (n + (long long)No * i)] = V[m * No + n];
    }
  }
}

// G^-1(k, iw_j)_ml = sum_n U_mn conj(U_ln) (mu + i w_j - e_n) - Sigma_ml with
// whatever U is given (fself.f90:85-129): U U^dagger multiplies i w + mu, so a
// U that is not exactly unitary gives the reference's values too.  One thread
// per (k, j), k fastest, so each (m, l) plane is written in coalesced runs.
__global__ void k_green_inv_eig(double2* G, const double2* sig, const double2* uni, const double* eig, double mu,
                                double temp, int64_t Nk, int64_t Nw, int No) {
  const long long KW = Nk * Nw;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < KW; t += (long long)gridDim.x * blockDim.x) {
    const long long i = t % Nk, j = t / Nk;
    const double2 iw = make_double2(mu, (double)(2 * j + 1) * 3.141592653589793238462643383279 * temp);
    const double2* U = uni + (long long)No * No * i;
    const double* e = eig + (long long)No * i;
    for (int l = 0; l < No; ++l)
      for (int m = 0; m < No; ++m) {
        double2 acc = make_double2(0.0, 0.0);
        for (int n = 0; n < No; ++n) acc += (U[m + No * n] * conj(U[l + No * n])) * (iw - make_double2(e[n], 0.0));
        const long long idx = t + KW * (m + (long long)No * l);
        G[idx] = acc - sig[idx];
      }
  }
}

// get_eig_mlo (fmod.f90:250-310): canonical orthogonalization of a
// non-orthogonal basis.  Per k: S = V_s diag(s) V_s^H from S's upper triangle
// (zheev 'U'), X = V_s diag(1/sqrt(s)) with the columns of s <= 1e-8 set to
// zero (near-linear dependence), H_orth = X^H H X (its upper triangle), then
// H_orth = V diag(e) V^H and uni = X V.  A discarded direction leaves an
// eigenvalue 0 in eig, as in the reference.
__global__ void k_get_eig_mlo(double* eig, double2* uni, const double2* hk, const double2* sk, int64_t Nk, int No) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < Nk; i += (long long)gridDim.x * blockDim.x) {
    double2 A[kMaxOrb * kMaxOrb], V[kMaxOrb * kMaxOrb], X[kMaxOrb * kMaxOrb], T[kMaxOrb * kMaxOrb];
    double w[kMaxOrb];
    const double2* h = hk + (long long)No * No * i;
    const double2* s = sk + (long long)No * No * i;
    for (int r = 0; r < No; ++r)
      for (int c = 0; c < No; ++c) A[r * No + c] = r <= c ? s[r + No * c] : conj(s[c + No * r]);
    jacobi_herm(A, No, w, V);
    for (int j = 0; j < No; ++j) {
      const double sc = w[j] > 1.0e-8 ? 1.0 / sqrt(w[j]) : 0.0;
      for (int r = 0; r < No; ++r) X[r * No + j] = sc * V[r * No + j];
    }
    for (int r = 0; r < No; ++r)  // T = H X (the full H, as the reference's zgemm reads it)
      for (int c = 0; c < No; ++c) {
        double2 acc = make_double2(0.0, 0.0);
        for (int k = 0; k < No; ++k) acc += h[r + No * k] * X[k * No + c];
        T[r * No + c] = acc;
      }
    for (int r = 0; r < No; ++r)  // upper triangle of X^H T, Hermitian
      for (int c = r; c < No; ++c) {
        double2 acc = make_double2(0.0, 0.0);
        for (int k = 0; k < No; ++k) acc += conj(X[k * No + r]) * T[k * No + c];
        A[r * No + c] = r == c ? make_double2(acc.x, 0.0) : acc;
        if (r != c) A[c * No + r] = conj(acc);
      }
    jacobi_herm(A, No, w, V);
    for (int n = 0; n < No; ++n) {
      eig[n + (long long)No * i] = w[n];
      for (int m = 0; m < No; ++m) {
        double2 acc = make_double2(0.0, 0.0);
        for (int k = 0; k < No; ++k) acc += X[m * No + k] * V[k * No + n];
        uni[m + No * (n + (long long)No * i)] = acc;
      }
    }
  }
}

__global__ void k_ffermi(double* f, const double* eig, double mu, double itemp, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    f[i] = 0.5 - 0.5 * tanh((eig[i] - mu) * itemp);
}

__global__ void k_extract_nu0(double2* out, const double2* chi, long long Nk, long long K, int nel) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < Nk * nel; i += (long long)gridDim.x * blockDim.x) {
    const long long k = i % Nk, e = i / Nk;
    out[i] = chi[k + K * e];
  }
}

__global__ void k_eig_or_tr(double2* vals, const double2* chi, int64_t Nk, int n, int sw_eig) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < Nk; k += (long long)gridDim.x * blockDim.x) {
    if (!sw_eig) {
      double2 t = make_double2(0, 0);
      for (int l = 0; l < n; ++l) t += chi[k + Nk * (l + (long long)n * l)];
      vals[k] = t;
      continue;
    }
    double2 A[kMaxChi * kMaxChi], w[kMaxChi];
    for (int a = 0; a < n; ++a)
      for (int b = 0; b < n; ++b) A[a * n + b] = chi[k + Nk * (a + (long long)n * b)];
    double best = -1e300;
    if (eigvals_general(A, n, w) < 0) best = nan("");
    else
      for (int i = 0; i < n; ++i) best = fmax(best, w[i].x);
    vals[k] = make_double2(best, 0.0);
  }
}

__global__ void k_map_full(double2* out, const double2* vals, const int64_t* invk, int64_t Nkall) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < Nkall; i += (long long)gridDim.x * blockDim.x)
    out[i] = vals[invk[3 * i] - 1];
}

__global__ void k_remap_delta(double2* out, const double2* d0, const double* prt, const int64_t* invk, int64_t Nkall,
                              int64_t Nk, int64_t Nw, int No, double dprt) {
  const long long N = Nkall * Nw * No * No;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < N; idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx % Nkall;
    const long long j = (idx / Nkall) % Nw;
    const int m = (int)((idx / (Nkall * Nw)) % No), l = (int)(idx / (Nkall * Nw * No));
    const long long k = invk[3 * i] - 1;
    double2 v = d0[k + Nk * (j + Nw * (m + (long long)No * l))];
    if (invk[3 * i + 1] == 1) v = (dprt * prt[m] * prt[l]) * v;
    else if (invk[3 * i + 1] != 0) v = make_double2(0, 0);
    out[idx] = v;
  }
}

__global__ void k_orb_to_band(double2* out, const double2* delta, const double2* uni, const double* prt,
                              const int64_t* invk, int64_t Nkall, int64_t Nk, int No, double dprt) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < Nkall; i += (long long)gridDim.x * blockDim.x) {
    const long long k = invk[3 * i] - 1;
    const int fl = (int)invk[3 * i + 1];
    const double2* U = uni + (long long)No * No * k;
    double2 D[kMaxOrb * kMaxOrb], T[kMaxOrb * kMaxOrb];
    // compact first-Matsubara slice: element (a,b) of k at k + Nk*(a + No*b)
    for (int a = 0; a < No; ++a)
      for (int b = 0; b < No; ++b) D[a * No + b] = delta[k + Nk * (long long)(a + No * b)];
    for (int a = 0; a < No; ++a)
      for (int b = 0; b < No; ++b) {
        double2 acc = make_double2(0, 0);
        for (int c = 0; c < No; ++c) {
          // L = U^H (direct) or U^T diag(prt) (via -k); L[a][c]
          double2 L = fl == 0 ? conj(U[c + No * a]) : U[c + No * a] * prt[c];
          acc += L * D[c * No + b];
        }
        T[a * No + b] = fl == 0 ? acc : acc * (dprt * prt[b]);
      }
    for (int a = 0; a < No; ++a)
      for (int b = 0; b < No; ++b) {
        double2 acc = make_double2(0, 0);
        for (int c = 0; c < No; ++c) {
          double2 Rm = fl == 0 ? U[c + No * b] : conj(U[c + No * b]);
          acc += T[a * No + c] * Rm;
        }
        if (fl != 0 && fl != 1) acc = make_double2(0, 0);
        out[i + Nkall * (a + (long long)No * b)] = acc;
      }
  }
}

unsigned g1(long long n, int t) { return (unsigned)std::max(1LL, std::min<long long>((n + t - 1) / t, 65536)); }

// ------------------------------------------------------- irreducible k mesh
int64_t irr_count(int64_t Nx, int64_t Ny, int64_t Nz) {
  const int64_t N = Nx * Ny * Nz;
  if (N % 2 == 0) {
    if (Nz % 2 == 0) {
      if (Nx % 2 == 0 && Ny % 2 == 0) return N / 2 + 4;
      if (Nx % 2 == 0 || Ny % 2 == 0) return N / 2 + 2;
      return N / 2 + 1;
    }
    if (Nx % 2 == 0 && Ny % 2 == 0) return N / 2 + 2;
    return N / 2 + 1;
  }
  return (N + 1) / 2;
}

// irreducible list in the reference's order (finv.f90:117-288)
std::vector<std::array<int64_t, 3>> irr_grid(int64_t Nx, int64_t Ny, int64_t Nz, int64_t Nk) {
  std::vector<std::array<int64_t, 3>> kl(Nk, {0, 0, 0});
  auto put = [&](int64_t it, int64_t i, int64_t j, int64_t k) {
    PGB_CHECK(it >= 1 && it <= Nk, "irreducible k index outside the list");
    kl[it - 1] = {i, j, k};
  };
  auto half_plane = [&](int64_t ini, int64_t k) -> int64_t {
    if (Nx % 2 == 0 && Ny % 2 == 0) {
      for (int64_t j = 0; j <= Ny / 2; ++j)
        for (int64_t i = 0; i <= Nx / 2; ++i) put(ini + i + (Nx / 2 + 1) * j, i, j, k);
      const int64_t ini2 = ini + (Nx / 2 + 1) * (Ny / 2 + 1) - 1;
      for (int64_t j = Ny / 2 + 1; j < Ny; ++j)
        for (int64_t i = 1; i < Nx / 2; ++i) put(ini2 + i + (Nx / 2 - 1) * (j - Ny / 2 - 1), i, j, k);
      return ini + Nx * Ny / 2 + 2;
    }
    int64_t it = ini;
    if ((Nx * Ny) % 2 == 0) {
      PGB_CHECK(Nx % 2 == 0, "odd Nx with even Ny: the irreducible k list is undefined for this mesh");
      for (int64_t j = 0; j <= (Ny - 1) / 2; ++j)
        for (int64_t i = 0; i <= Nx / 2; ++i) put(it++, i, j, k);
      for (int64_t j = (Ny + 1) / 2; j < Ny; ++j)
        for (int64_t i = 1; i < Nx / 2; ++i) put(it++, i, j, k);
      return it;
    }
    for (int64_t j = 0; j <= (Ny - 1) / 2; ++j)
      for (int64_t i = 0; i <= (Nx - 1) / 2; ++i) put(it++, i, j, k);
    for (int64_t j = (Ny + 1) / 2; j < Ny; ++j)
      for (int64_t i = 1; i <= (Nx - 1) / 2; ++i) put(it++, i, j, k);
    return it;
  };
  int64_t ini = half_plane(1, 0);
  if (Nz > 1) {
    const int64_t nfull = (Nz % 2 == 0) ? Nz / 2 - 1 : (Nz - 1) / 2;
    for (int64_t k = 1; k <= nfull; ++k)
      for (int64_t j = 0; j < Ny; ++j)
        for (int64_t i = 0; i < Nx; ++i) put(ini + i + Nx * j + Nx * Ny * (k - 1), i, j, k);
    ini += Nx * Ny * nfull;
    if (Nz % 2 == 0) half_plane(ini, Nz / 2);
  }
  return kl;
}

}  // namespace

namespace {
// klist (3,Nk), kmap (3,Nkall) and invk (3,Nkall) of generate_irr_kpoint_inv (finv.f90:1-290)
void irr_mesh_fill(int64_t nx, int64_t ny, int64_t nz, int64_t nk, double* klist, int64_t* kmap, int64_t* invk) {
  PGB_CHECK(nx > 0 && ny > 0 && nz > 0, "non-positive mesh");
  PGB_CHECK(nk == irr_count(nx, ny, nz), "Nk differs from the irreducible count of this mesh");
  auto irr = irr_grid(nx, ny, nz, nk);
  std::unordered_map<int64_t, int64_t> direct, inverse;
  auto key = [&](int64_t x, int64_t y, int64_t z) { return x + nx * (y + ny * z); };
  for (int64_t j = 0; j < nk; ++j) {
    const auto& c = irr[j];
    if (klist) {
      klist[3 * j] = (double)c[0] / (double)nx;
      klist[3 * j + 1] = (double)c[1] / (double)ny;
      klist[3 * j + 2] = (double)c[2] / (double)nz;
    }
    direct.emplace(key(c[0], c[1], c[2]), j);
    inverse.emplace(key((nx - c[0]) % nx, (ny - c[1]) % ny, (nz - c[2]) % nz), j);
  }
  for (int64_t z = 0; z < nz; ++z)
    for (int64_t y = 0; y < ny; ++y)
      for (int64_t x = 0; x < nx; ++x) {
        const int64_t i = key(x, y, z);
        kmap[3 * i] = x;
        kmap[3 * i + 1] = y;
        kmap[3 * i + 2] = z;
        auto d = direct.find(i), v = inverse.find(i);
        PGB_CHECK(d != direct.end() || v != inverse.end(), "k point without irreducible partner");
        if (d != direct.end() && (v == inverse.end() || d->second <= v->second)) {
          invk[3 * i] = d->second + 1;
          invk[3 * i + 1] = 0;
        } else {
          invk[3 * i] = v->second + 1;
          invk[3 * i + 1] = 1;
        }
        invk[3 * i + 2] = key((nx - x) % nx, (ny - y) % ny, (nz - z) % nz) + 1;
      }
}
}  // namespace

namespace pgb {
int64_t make_irr_mesh(int64_t nx, int64_t ny, int64_t nz, std::vector<int64_t>& kmap, std::vector<int64_t>& invk) {
  const int64_t nk = irr_count(nx, ny, nz);
  kmap.assign(3 * nx * ny * nz, 0);
  invk.assign(3 * nx * ny * nz, 0);
  irr_mesh_fill(nx, ny, nz, nk, nullptr, kmap.data(), invk.data());
  return nk;
}
}  // namespace pgb

// chi0 entry shared by get_chi0 / get_chi0_tail / get_chi0_conv_
namespace {
// Whether the even form is the faster one for a get_chi0 of `work` padded mesh points times
// pair elements.  Its tables and checks take 60 us and 0.008 us for each of the `points`
// mesh points.  Against them stand, per 2^20 of work, the us below, least for the cheapest
// arithmetic; FP32 transforms of several pairs are bound by memory in both forms.  From
// four pairs on (FP32: 16) the complex QR of the Stoner factor that it spares decides alone.
// General and even form in us, calls on both sides of the line:
//   FP64                 one orbital 32x32x200 351 and 352, 32x32x400 522 and 446; 64x64x64 408 and 446,
//                        64x64x100 582 and 501; two 16x16x64 390 and 340
//   double-float         one 32x32x512 400 and 423, 32x32x1024 635 and 571; 64x64x128 430 and 478,
//                        64x64x256 661 and 624; two 16x16x64 367 and 330
//   double-float, tail   one 32x32x200 497 and 487, 32x32x400 694 and 601; 64x64x64 581 and 593
//   FP32                 one 32x32x1024 493 and 531, 32x32x2048 822 and 809; two 64x64x32 710 and 813,
//                        32x32x200 967 and 963; three 32x32x32 818 and 848, 32x32x40 989 and 973;
//                        four 8x8x16 457 and 440
//   FP32, tail           one 32x32x512 515 and 539, 32x32x1024 749 and 715; two 64x64x32 896 and 987,
//                        32x32x200 1177 and 1104
template <typename R> bool even_chi0_pays(double work, double points, int64_t n, bool tail) {
  constexpr bool fp32 = std::is_same<R, float>::value;
  if (work < (1 << 19)) return false;
  if (n >= (fp32 ? 16 : 4)) return true;
  double saved = 165.0;
  if (fp32) saved = n >= 4 ? 11.0 : (tail ? 48.0 : 25.0);
  else if (std::is_same<R, dfl>::value && !tail) saved = 60.0;
  return saved * work / (1 << 20) >= 60.0 + 0.008 * points;
}
template <typename R>
double chi0_entry(double2* chi_out, const double* Smat, const double* Cmat, const double2* Gk, const int64_t* kmap,
                  const int64_t* invk, const int64_t* olist, double temp, int64_t Nx, int64_t Ny, int64_t Nz, int64_t Nw,
                  int64_t Nk, int64_t Nkall, int64_t Norb, int64_t Nchi, const double* eig, const double2* uni,
                  double mu, bool tail, bool with_stoner, const int32_t* irr_chi, const int32_t* chi_map) {
  PGB_CHECK(Nkall == Nx * Ny * Nz, "Nkall differs from Nx*Ny*Nz");
  Geom g;
  build_geom(g, kmap, invk, Nx, Ny, Nz, Nk, Nw, Norb, Nchi);
  Pairs p;
  build_pairs(p, olist, (int)Norb, (int)Nchi, irr_chi, chi_map);
  const long long KE = g.K * Norb * Norb, KC = g.K * Nchi * Nchi;
  HostPrefault pages(chi_out, sizeof(double2) * KC);
  DBuf<double2> G(KE);
  G.upload(Gk, KE);
  DBuf<double> e, S, C;
  DBuf<double2> u;
  TailRef tr;
  if (tail) {
    e.alloc(Norb * Nk);
    e.upload(eig, Norb * Nk);
    u.alloc(Norb * Norb * Nk);
    u.upload(uni, Norb * Norb * Nk);
    tr.eig = e.p;
    tr.uni = u.p;
    tr.mu = mu;
  }
  DBuf<cx<R>> chi(KC);
  // The even form for a symmetric G; a caller's own pair maps keep the general
  // one, and so do
  //  * the tail-corrected FP64 bubble: it is what lin_eliash is given, whose
  //    fixed-size two-pass Krylov space amplifies a change of 1e-16 in chi0 to
  //    1e-9 .. 2e-8 of the gap (twelve two-orbital models), so its bits stay;
  //  * small calls (even_chi0_pays).
  // A G without the symmetry shows it in a few host elements, which spares it the
  // check on the device and its wait (50 us of 1.2 ms: three orbitals 16x16x64).
  const bool even_call = !irr_chi && !chi_map && !(tail && std::is_same<R, double>::value) &&
                         even_chi0_pays<R>((double)g.P * Nchi * Nchi, (double)Nkall, Nchi, tail);
  if (even_call && symmetric_sample(Gk, g.K, (int)Norb) && (!tail || symmetric_bands(eig, uni, Nk, (int)Norb)) &&
      symmetric_blocks(G.p, g.K, (int)Norb, 1.0e-12)) {
    if (with_stoner) g.even = make_even(g, p, Smat, Cmat, (int)sizeof(cx<R>));
    if (!g.even) g.even = make_even(g, p, nullptr, nullptr, (int)sizeof(cx<R>));
  }
  chi0<R>(g, p, G.p, temp, tail ? &tr : nullptr, chi.p);
  G.release();
  double sdw = 0;
  if (with_stoner) {
    S.alloc(Nchi * Nchi);
    C.alloc(Nchi * Nchi);
    S.upload(Smat, Nchi * Nchi);
    C.upload(Cmat, Nchi * Nchi);
    double cdw = 0;
    int qs = 0, qc = 0;
    stoner<R>(g, chi.p, S.p, C.p, &sdw, &cdw, &qs, &qc);
    ckchi_print(g, sdw, cdw, qs, qc);
  }
  if (std::is_same<R, double>::value) {
    pages.join();
    chi.download(chi_out, KC);
  } else {
    DBuf<double2> w(KC);
    widen<R>(w.p, chi.p, KC);
    pages.join();
    w.download(chi_out, KC);
  }
  sync();
  return sdw;
}
// chi0 entry of the current precision: double-float convolutions in mode 48
auto chi0_fn() {
  return ctx().precision == kPrecDF ? chi0_entry<dfl> : (fp32() ? chi0_entry<float> : chi0_entry<double>);
}
}  // namespace

// ============================================== allocation-free variant ==
// pyrpa_gb_eig_or_tr_chi_noalloc computes what get_eig_or_tr_chi computes, on
// buffers that are already in device memory, and takes no device memory of
// its own while it runs.  It serves callers that cannot let a library
// allocate: a host framework whose own caching allocator has reserved nearly
// all of HBM (an allocation by this library could then fail for want of
// memory), and loops that enqueue work on their own stream and must not wait
// for an allocation or a host copy on every call.  Its only scratch, one value
// per irreducible q point, is the fixed array below.
//
// What the first call on a device takes: with CUDA's lazy module loading
// (the default), the module that holds this array and these kernels, and the
// local memory of the eigenvalue kernel (a 32x32 complex-double working matrix
// per thread), are mapped on that device only when the module is first used.
// The first call on each device therefore does a set-up (the array's address,
// and one empty launch of each kernel) that takes that memory.  Make that
// first call before the host's allocator reserves most of HBM, and before any
// stream capture; later calls take nothing.
namespace {
// 65,536 irreducible q points at most: 1 MiB on every device that loads the
// library, held until the process exits
constexpr int64_t kNoAllocMaxNk = 65536;
__device__ __align__(256) double2 g_noalloc_vals[kNoAllocMaxNk];
constexpr int kNoAllocMaxDevices = 64;
double2* g_noalloc_ptr[kNoAllocMaxDevices] = {};  // address of the array on each device
std::mutex g_noalloc_mu;

// k_map_full with the irreducible index checked: an invk(1,i) outside [1,Nk]
// gives NaN instead of a read outside the scratch
__global__ void k_map_full_checked(double2* out, const double2* vals, const int64_t* invk, int64_t Nkall,
                                   int64_t Nk) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < Nkall;
       i += (long long)gridDim.x * blockDim.x) {
    const int64_t k = invk[3 * i];
    out[i] = (k >= 1 && k <= Nk) ? vals[k - 1] : make_double2(nan(""), nan(""));
  }
}
}  // namespace

#define ABI_TRY try {
#define ABI_CATCH(name, onerr)            \
  }                                       \
  catch (const BadInput& e) {             \
    report(name, e.what(), 2);            \
    onerr;                                \
  }                                       \
  catch (const std::exception& e) {       \
    report(name, e.what());               \
    onerr;                                \
  }

extern "C" {

// ============================================================== extras ==
void pyrpa_gb_set_precision(const int64_t* bits) {
  ctx().precision = (*bits == 32 || *bits == kPrecMixed || *bits == kPrecDF) ? (int)*bits : 64;
}
void pyrpa_gb_get_precision(int64_t* bits) {
  ABI_TRY ensure_context(); ABI_CATCH("pyrpa_gb_get_precision", (void)0)
  *bits = ctx().precision;
}
void pyrpa_gb_set_verbose(const int64_t* v) { ctx().verbose = (int)*v; }
void pyrpa_gb_set_arnoldi_tol(const double* tol) {
  ABI_TRY
  PGB_CHECK(*tol >= 0.0, "the Arnoldi residual tolerance must be >= 0");
  ensure_context();
  ctx().arnoldi_tol = *tol;
  ABI_CATCH("pyrpa_gb_set_arnoldi_tol", (void)0)
}
void pyrpa_gb_last_error(char* buf, const int64_t* len, int64_t* code) {
  if (buf && len && *len > 0) {
    const size_t n = std::min<size_t>((size_t)*len - 1, g_last_error.size());
    memcpy(buf, g_last_error.data(), n);
    buf[n] = 0;
  }
  if (code) *code = g_last_code;
}
void pyrpa_gb_clear_error() {
  g_last_error.clear();
  g_last_code = 0;
}
void pyrpa_gb_set_thread_stream(const int64_t* on) {
  ABI_TRY set_thread_context(*on != 0); ABI_CATCH("pyrpa_gb_set_thread_stream", (void)0)
}
void pyrpa_gb_kernel_launches(int64_t* n) { *n = ctx().kernel_launches; }
void pyrpa_gb_pivoted_vertices(int64_t* n) { *n = ctx().pivoted_vertices; }
void pyrpa_gb_last_stats(double* out) {
  const LastStats& s = last_stats();
  const double v[20] = {(double)s.iterations, s.esterr, s.stoner, s.mu, s.lambda, (double)s.applies, s.t_chi0,
                        s.t_vertex, s.t_sigma, s.t_diis, s.t_mu, s.t_dyson, s.t_apply, (double)s.iterations32,
                        (double)s.iterations_coarse, s.t_warm, s.t_stoner, (double)s.iterations_finish32,
                        s.ritz_residual, (double)s.arnoldi_cycles};
  memcpy(out, v, sizeof(v));
}
void pyrpa_gb_last_ritz(double* out, const int64_t* n, int64_t* count) {
  const LastStats& s = last_stats();
  *count = s.nritz;
  for (int64_t i = 0; i < std::min<int64_t>(*n, s.nritz); ++i) out[i] = s.ritz[i];
}
void pyrpa_gb_fft_profile(const int64_t* on) { fft_profile_enable(*on != 0); }
void pyrpa_gb_fft_stats(double* out) {
  ABI_TRY fft_profile_collect(&out[0], &out[1], &out[2]);
  ABI_CATCH("pyrpa_gb_fft_stats", (out[0] = out[1] = out[2] = 0))
}
void pyrpa_gb_device_info(int64_t* num_sms, int64_t* device) {
  ABI_TRY ensure_context(); *num_sms = ctx().num_sms; *device = ctx().device;
  ABI_CATCH("pyrpa_gb_device_info", (*num_sms = 0, *device = -1))
}

// ================================================================ setup ==
void openmp_params(int64_t* omp_num, bool* omp_check) {
  // no OpenMP in this library: the work runs on the GPU
  *omp_num = 0;
  *omp_check = false;
}

void generate_irr_kpoint_inv(double* klist, int64_t* kmap, int64_t* invk, const int64_t* Nk, const int64_t* Nx,
                             const int64_t* Ny, const int64_t* Nz) {
  ABI_TRY
  irr_mesh_fill(*Nx, *Ny, *Nz, *Nk, klist, kmap, invk);
  ABI_CATCH("generate_irr_kpoint_inv", (void)0)
}

void get_kweight(double* weight, const int64_t* invk, const int64_t* Nk, const int64_t* Nkall) {
  ABI_TRY
  for (int64_t k = 0; k < *Nk; ++k) weight[k] = 0.0;
  for (int64_t i = 0; i < *Nkall; ++i) {
    const int64_t k = invk[3 * i] - 1;
    PGB_CHECK(k >= 0 && k < *Nk, "invk(1,:) outside [1,Nk]");
    weight[k] += 1.0;
  }
  ABI_CATCH("get_kweight", (void)0)
}

void get_scmat(double* Smat, double* Cmat, const int64_t* ol, const int64_t* site, const double* Uval,
               const double* Jval, const int64_t* Nchi) {
  const int64_t n = *Nchi;
  const double U = *Uval, J = *Jval, Up = U - 2 * J;
  for (int64_t i = 0; i < n; ++i)
    for (int64_t j = 0; j < n; ++j) {
      double s = 0, c = 0;
      const int64_t i1 = ol[i], i2 = ol[n + i], j1 = ol[j], j2 = ol[n + j];
      if (site[i] == site[j]) {
        if (i1 == i2 && j1 == j2) {
          if (i1 == j1) { s = U; c = U; }
          else { s = J; c = 2 * Up - J; }
        } else if (i1 == j1 && i2 == j2) {
          s = Up; c = -Up + 2 * J;
        } else if (i1 == j2 && i2 == j1) {
          s = J; c = J;
        }
      }
      Smat[j + n * i] = s;
      Cmat[j + n * i] = c;
    }
}

void get_scmat_orb(double* Smat, double* Cmat, const int64_t* ol, const int64_t* site, const double* Umat,
                   const double* Jmat, const int64_t* Nchi, const int64_t* Norb) {
  const int64_t n = *Nchi, no = *Norb;
  auto Uf = [&](int64_t a, int64_t b) { return Umat[(a - 1) + no * (b - 1)]; };
  auto Jf = [&](int64_t a, int64_t b) { return Jmat[(a - 1) + no * (b - 1)]; };
  for (int64_t i = 0; i < n; ++i)
    for (int64_t j = 0; j < n; ++j) {
      double s = 0, c = 0;
      const int64_t i1 = ol[i], i2 = ol[n + i], j1 = ol[j], j2 = ol[n + j];
      if (site[i] == site[j]) {
        if (i1 == i2 && j1 == j2) {
          if (i1 == j1) { s = Uf(i1, i1); c = s; }
          else { s = Jf(i1, j1); c = 2 * Uf(i1, j1) - Jf(i1, j1); }
        } else if (i1 == j1 && i2 == j2) {
          s = Uf(i1, i2); c = -Uf(i1, i2) + 2 * Jf(i1, i2);
        } else if (i1 == j2 && i2 == j1) {
          s = Jf(i1, i2); c = s;
        }
      }
      Smat[j + n * i] = s;
      Cmat[j + n * i] = c;
    }
}

void get_parity_prop(double* Pmn, const double* rvec, const double2* ham_r, const int64_t* Norb, const int64_t* Nr) {
  const int64_t no = *Norb, nr = *Nr;
  std::vector<double> num(no * no, 0.0), den(no * no, 0.0);
  for (int64_t i = 0; i < nr; ++i)
    for (int64_t j = i + 1; j < nr; ++j) {
      const double d = std::fabs(rvec[3 * i] + rvec[3 * j]) + std::fabs(rvec[3 * i + 1] + rvec[3 * j + 1]) +
                       std::fabs(rvec[3 * i + 2] + rvec[3 * j + 2]);
      if (d < 1e-6) {
        for (int64_t e = 0; e < no * no; ++e) {
          const double2 a = ham_r[e + no * no * j], b = ham_r[e + no * no * i];
          num[e] += a.x * b.x + a.y * b.y;
          den[e] += b.x * b.x + b.y * b.y;
        }
        break;
      }
    }
  for (int64_t e = 0; e < no * no; ++e) {
    const double p = den[e] > 1e-10 ? num[e] / den[e] : 0.0;
    Pmn[e] = p >= 0.0 ? 1.0 : -1.0;
  }
}

void gen_ham(double2* ham_k, const double* klist, const double2* ham_r, const double* rvec, const int64_t* Nk,
             const int64_t* Nr, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, nr = *Nr, no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  DBuf<double2> hk(no * no * nk), hr(no * no * nr);
  DBuf<double> kl(3 * nk), rv(3 * nr);
  hr.upload(ham_r, no * no * nr);
  kl.upload(klist, 3 * nk);
  rv.upload(rvec, 3 * nr);
  k_gen_ham<<<g1(nk, 64), 64, 0, ctx().stream>>>(hk.p, kl.p, hr.p, rv.p, nk, nr, (int)no);
  launch_check("gen_ham");
  hk.download(ham_k, no * no * nk);
  sync();
  ABI_CATCH("gen_ham", nan_fill(ham_k, (size_t)(*Norb) * (*Norb) * (*Nk)))
}

void get_eig(double* eig, double2* uni, const double2* ham_k, const int64_t* Nk, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  DBuf<double2> hk(no * no * nk), u(no * no * nk);
  DBuf<double> e(no * nk);
  hk.upload(ham_k, no * no * nk);
  k_get_eig<<<g1(nk, 64), 64, 0, ctx().stream>>>(e.p, u.p, hk.p, nk, (int)no);
  launch_check("get_eig");
  e.download(eig, no * nk);
  u.download(uni, no * no * nk);
  sync();
  ABI_CATCH("get_eig", (nan_fill(eig, (size_t)(*Norb) * (*Nk)), nan_fill(uni, (size_t)(*Norb) * (*Norb) * (*Nk))))
}

void get_eig_mlo(double* eig, double2* uni, const double2* ham_k, const double2* Ovlk, const int64_t* Nk,
                 const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  DBuf<double2> hk(no * no * nk), sk(no * no * nk), u(no * no * nk);
  DBuf<double> e(no * nk);
  hk.upload(ham_k, no * no * nk);
  sk.upload(Ovlk, no * no * nk);
  k_get_eig_mlo<<<g1(nk, 64), 64, 0, ctx().stream>>>(e.p, u.p, hk.p, sk.p, nk, (int)no);
  launch_check("get_eig_mlo");
  e.download(eig, no * nk);
  u.download(uni, no * no * nk);
  sync();
  ABI_CATCH("get_eig_mlo", (nan_fill(eig, (size_t)(*Norb) * (*Nk)), nan_fill(uni, (size_t)(*Norb) * (*Norb) * (*Nk))))
}

void get_ffermi(double* ffermi, const double* eig, const double* mu, const double* temp, const int64_t* Nk,
                const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const long long n = (*Nk) * (*Norb);
  DBuf<double> e(n), f(n);
  e.upload(eig, n);
  const double t = std::max(*temp, 1.0e-12);
  k_ffermi<<<g1(n, 256), 256, 0, ctx().stream>>>(f.p, e.p, *mu, 0.5 / t, n);
  launch_check("ffermi");
  f.download(ffermi, n);
  sync();
  ABI_CATCH("get_ffermi", nan_fill(ffermi, (size_t)(*Nk) * (*Norb)))
}

// ================================================================ green ==
void gen_green0_(double2* Gk, const double* eig, const double2* uni, const double* mu, const double* temp,
                 const int64_t* Nk, const int64_t* Nw, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, nw = *Nw, no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  DBuf<double> e(no * nk);
  DBuf<double2> u(no * no * nk), G(nk * nw * no * no);
  e.upload(eig, no * nk);
  u.upload(uni, no * no * nk);
  HostPrefault pages(Gk, G.bytes());
  green0(G.p, e.p, u.p, *mu, *temp, (int)nk, (int)nw, (int)no);
  pages.join();
  G.download(Gk, nk * nw * no * no);
  sync();
  ABI_CATCH("gen_green0_", nan_fill(Gk, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)))
}

void gen_green_inv_(double2* Gk, const double2* self, const double2* hamk, const double* mu, const double* temp,
                    const int64_t* Nk, const int64_t* Nw, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, nw = *Nw, no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  const long long KE = nk * nw * no * no;
  DBuf<double2> s(KE), h(no * no * nk), G(KE);
  HostPrefault pages(Gk, G.bytes());
  s.upload(self, KE);
  h.upload(hamk, no * no * nk);
  green_inv_only(G.p, s.p, h.p, *mu, *temp, (int)nk, (int)nw, (int)no);
  pages.join();
  G.download(Gk, KE);
  sync();
  ABI_CATCH("gen_green_inv_", nan_fill(Gk, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)))
}

// fself.f90:85-129: G^-1(k, iw)_ml = sum_n U_mn conj(U_ln) (iw + mu - e_n) - Sigma_ml.  With U unitary
// that is (iw + mu) delta_ml - H_ml - Sigma_ml for H = U diag(e) U^dagger, so H is rebuilt on the host
// (Nk Norb^3 operations) and the G^-1 kernel of gen_green_inv_ does the rest.
void gen_green_inv_from_eig(double2* Gk, const double2* self, const double2* uni, const double* eig,
                            const double* mu, const double* temp, const int64_t* Nk, const int64_t* Nw,
                            const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, nw = *Nw, no = *Norb;
  PGB_CHECK(no >= 1 && no <= kMaxOrb, "Norb must be in [1, 8]");
  const long long KE = nk * nw * no * no;
  DBuf<double2> s(KE), u(no * no * nk), G(KE);
  DBuf<double> e(no * nk);
  s.upload(self, KE);
  u.upload(uni, no * no * nk);
  e.upload(eig, no * nk);
  k_green_inv_eig<<<g1(nk * nw, 128), 128, 0, ctx().stream>>>(G.p, s.p, u.p, e.p, *mu, *temp, nk, nw, (int)no);
  launch_check("green_inv_eig");
  G.download(Gk, KE);
  sync();
  ABI_CATCH("gen_green_inv_from_eig", nan_fill(Gk, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)))
}

void getinv_(double2* Gk, const int64_t* Nk, const int64_t* Nw, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, nw = *Nw, no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  const long long K = nk * nw, KE = K * no * no;
  DBuf<double2> G(KE);
  G.upload(Gk, KE);
  PGB_CHECK(invert_blocks(G.p, K, (int)no, 1, K), "zgetrf failed in getinv: singular matrix");
  G.download(Gk, KE);
  sync();
  ABI_CATCH("getinv_", nan_fill(Gk, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)))
}

// ================================================================== chi ==

void get_chi0(double2* chi, const double* Smat, const double* Cmat, const double2* Gk, const int64_t* kmap,
              const int64_t* invk, const int64_t* olist, const double* temp, const int64_t* Nx, const int64_t* Ny,
              const int64_t* Nz, const int64_t* Nw, const int64_t* Nk, const int64_t* Nkall, const int64_t* Norb,
              const int64_t* Nchi, double* maxchi0s_out) {
  ABI_TRY
  ensure_context();
  auto f = chi0_fn();
  *maxchi0s_out = f(chi, Smat, Cmat, Gk, kmap, invk, olist, *temp, *Nx, *Ny, *Nz, *Nw, *Nk, *Nkall, *Norb, *Nchi,
                    nullptr, nullptr, 0.0, false, true, nullptr, nullptr);
  ABI_CATCH("get_chi0", (nan_fill(chi, (size_t)(*Nk) * (*Nw) * (*Nchi) * (*Nchi)), *maxchi0s_out = NAN))
}

void get_chi0_tail(double2* chi, const double* Smat, const double* Cmat, const double2* Gk, const double* eig,
                   const double2* uni, const int64_t* kmap, const int64_t* invk, const int64_t* olist, const double* mu,
                   const double* temp, const int64_t* Nx, const int64_t* Ny, const int64_t* Nz, const int64_t* Nw,
                   const int64_t* Nk, const int64_t* Nkall, const int64_t* Norb, const int64_t* Nchi,
                   double* maxchi0s_out) {
  ABI_TRY
  ensure_context();
  auto f = chi0_fn();
  *maxchi0s_out = f(chi, Smat, Cmat, Gk, kmap, invk, olist, *temp, *Nx, *Ny, *Nz, *Nw, *Nk, *Nkall, *Norb, *Nchi,
                    eig, uni, *mu, true, true, nullptr, nullptr);
  ABI_CATCH("get_chi0_tail", (nan_fill(chi, (size_t)(*Nk) * (*Nw) * (*Nchi) * (*Nchi)), *maxchi0s_out = NAN))
}

void get_chi0_conv_(double2* chi, const double2* Gk, const int64_t* kmap, const int64_t* invk, const int32_t* irr_chi,
                    const int32_t* chi_map, const int64_t* olist, const double* temp, const int64_t* Nx,
                    const int64_t* Ny, const int64_t* Nz, const int64_t* Nw, const int64_t* Nk, const int64_t* Nkall,
                    const int64_t* Norb, const int64_t* Nchi) {
  ABI_TRY
  ensure_context();
  auto f = chi0_fn();
  f(chi, nullptr, nullptr, Gk, kmap, invk, olist, *temp, *Nx, *Ny, *Nz, *Nw, *Nk, *Nkall, *Norb, *Nchi, nullptr,
    nullptr, 0.0, false, false, irr_chi, chi_map);
  ABI_CATCH("get_chi0_conv_", nan_fill(chi, (size_t)(*Nk) * (*Nw) * (*Nchi) * (*Nchi)))
}

void get_chis(double2* chis, const double2* chi0, const double* Smat, const int64_t* Nchi, const int64_t* Nw) {
  ABI_TRY
  ensure_context();
  const int64_t n = *Nchi, nw = *Nw;
  PGB_CHECK(n <= kMaxChi, "Nchi above the engine limit of 32 orbital pairs");
  DBuf<double2> X(n * n * nw);
  DBuf<double> S(n * n);
  X.upload(chi0, n * n * nw);
  S.upload(Smat, n * n);
  PGB_CHECK(vertex<double>(X.p, nw, -1, (int)n, S.p, S.p, 3), "zgesv failed: singular (I - chi0 S)");
  X.download(chis, n * n * nw);
  sync();
  ABI_CATCH("get_chis", nan_fill(chis, (size_t)(*Nchi) * (*Nchi) * (*Nw)))
}

void get_chis_chic(double2* chis, double2* chic, const double2* chi, const double* Smat, const double* Cmat,
                   const int64_t* Nk, const int64_t* Nw, const int64_t* Nchi) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, nw = *Nw, n = *Nchi;
  PGB_CHECK(n <= kMaxChi, "Nchi above the engine limit of 32 orbital pairs");
  const long long K = nk * nw;
  DBuf<double2> X(K * n * n), A(nk * n * n), B(nk * n * n);
  DBuf<double> S(n * n), C(n * n);
  X.upload(chi, K * n * n);
  S.upload(Smat, n * n);
  C.upload(Cmat, n * n);
  k_extract_nu0<<<g1(nk * n * n, 256), 256, 0, ctx().stream>>>(A.p, X.p, nk, K, (int)(n * n));
  launch_check("extract_nu0");
  X.release();
  PGB_CUDA(cudaMemcpyAsync(B.p, A.p, A.bytes(), cudaMemcpyDeviceToDevice, ctx().stream));
  PGB_CHECK(vertex<double>(A.p, nk, nk, (int)n, S.p, C.p, 3), "zgesv failed: singular (I - chi0 S)");
  PGB_CHECK(vertex<double>(B.p, nk, nk, (int)n, S.p, C.p, 4), "zgesv failed: singular (I + chi0 C)");
  A.download(chis, nk * n * n);
  B.download(chic, nk * n * n);
  sync();
  ABI_CATCH("get_chis_chic", (nan_fill(chis, (size_t)(*Nk) * (*Nchi) * (*Nchi)),
                              nan_fill(chic, (size_t)(*Nk) * (*Nchi) * (*Nchi))))
}

void get_eig_or_tr_chi(double2* chiqout, const double2* chi, const int64_t* invk, const int64_t* Nkall,
                       const int64_t* Nk, const int64_t* Nchi, const bool* sw_eig) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, n = *Nchi, nkall = *Nkall;
  PGB_CHECK(n <= kMaxChi, "Nchi above the engine limit of 32 orbital pairs");
  for (int64_t i = 0; i < nkall; ++i) PGB_CHECK(invk[3 * i] >= 1 && invk[3 * i] <= nk, "invk(1,:) outside [1,Nk]");
  DBuf<double2> X(nk * n * n), v(nk), out(nkall);
  DBuf<int64_t> iv(3 * nkall);
  X.upload(chi, nk * n * n);
  iv.upload(invk, 3 * nkall);
  k_eig_or_tr<<<g1(nk, 32), 32, 0, ctx().stream>>>(v.p, X.p, nk, (int)n, (*sw_eig) ? 1 : 0);
  launch_check("eig_or_tr");
  k_map_full<<<g1(nkall, 256), 256, 0, ctx().stream>>>(out.p, v.p, iv.p, nkall);
  launch_check("map_full");
  out.download(chiqout, nkall);
  sync();
  ABI_CATCH("get_eig_or_tr_chi", nan_fill(chiqout, (size_t)(*Nkall)))
}

void get_vsigma_flex_nosoc_(double2* chi, const double* Smat, const double* Cmat, const int64_t* Nk,
                            const int64_t* Nw, const int64_t* Nchi) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, nw = *Nw, n = *Nchi;
  PGB_CHECK(n <= kMaxChi, "Nchi above the engine limit of 32 orbital pairs");
  const long long K = nk * nw;
  DBuf<double2> X(K * n * n);
  DBuf<double> S(n * n), C(n * n);
  X.upload(chi, K * n * n);
  S.upload(Smat, n * n);
  C.upload(Cmat, n * n);
  if (ctx().precision == kPrecDF) {  // the double-float solve of the mixed schedule's judging phase
    DBuf<cdf> Xd(K * n * n);
    narrow<dfl>(Xd.p, X.p, K * n * n);
    PGB_CHECK(vertex<dfl>(Xd.p, K, K, (int)n, S.p, C.p, 0), "zgesv failed in V_sigma");
    widen<dfl>(X.p, Xd.p, K * n * n);
  } else {
    PGB_CHECK(vertex<double>(X.p, K, K, (int)n, S.p, C.p, 0), "zgesv failed in V_sigma");
  }
  X.download(chi, K * n * n);
  sync();
  ABI_CATCH("get_vsigma_flex_nosoc_", nan_fill(chi, (size_t)(*Nk) * (*Nw) * (*Nchi) * (*Nchi)))
}

// ================================================================= flex ==
void mkself(double2* sigmak, double* mu, const double* Smat, const double* Cmat, const int64_t* kmap,
            const int64_t* invk, const int64_t* olist, const double2* hamk, const double* eig, const double2* uni,
            const double* mu_init, const double* rfill, const double* temp, const int64_t* scf_loop, const double* pp,
            const double* eps, const int64_t* Nkall, const int64_t* Nk, const int64_t* Nw, const int64_t* Norb,
            const int64_t* Nchi, const int64_t* Nx, const int64_t* Ny, const int64_t* Nz, const int64_t* sub_sigma,
            const bool* sw_out, const bool* sw_in, const int64_t* m_diis, const bool* sw_rescale, const bool* sw_tail,
            const double* sigma_scale) {
  ABI_TRY
  ensure_context();
  MkselfArgs a{sigmak, mu, Smat, Cmat, kmap, invk, olist, hamk, eig, uni, *mu_init, *rfill, *temp, *scf_loop, *pp,
               *eps, *Nkall, *Nk, *Nw, *Norb, *Nchi, *Nx, *Ny, *Nz, *sub_sigma, *sw_out, *sw_in, *m_diis,
               *sw_rescale, *sw_tail, *sigma_scale};
  run_mkself(a, ctx().precision);
  ABI_CATCH("mkself", (nan_fill(sigmak, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)), *mu = NAN))
}

void lin_eliash(double2* delta, double2* chi, const double2* Gk, const double2* uni, const double* init_delta,
                const double* Smat, const double* Cmat, const int64_t* olist, const double* prt, const int64_t* kmap,
                const int64_t* invk, const double* temp, const double* eps, const int64_t* Nkall, const int64_t* Nk,
                const int64_t* Nw, const int64_t* Nchi, const int64_t* Norb, const int64_t* Nx, const int64_t* Ny,
                const int64_t* Nz, const int64_t* itemax, const int64_t* gap_sym, const int64_t* arnoldi_m,
                double* lambda_out) {
  ABI_TRY
  ensure_context();
  LinEliashArgs a{delta, chi, Gk, uni, init_delta, Smat, Cmat, olist, prt, kmap, invk, *temp, *eps, *Nkall, *Nk, *Nw,
                  *Nchi, *Norb, *Nx, *Ny, *Nz, *itemax, *gap_sym, *arnoldi_m, lambda_out};
  if (fp32()) run_lin_eliash<float>(a);
  else run_lin_eliash<double>(a);
  ABI_CATCH("lin_eliash", (nan_fill(delta, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)), *lambda_out = NAN))
}

void pyrpa_gb_flex_eliash(double2* sigmak, double* mu, double2* delta, double* lambda_out, double* stoner,
                          double* times_ms, const double* Smat, const double* Cmat, const int64_t* kmap,
                          const int64_t* invk, const int64_t* olist, const double2* hamk, const double* eig,
                          const double2* uni, const double* init_delta, const double* prt, const double2* sigma_seed,
                          const double* seed_mu, const double* seed_mu_old, const double* mu_init,
                          const double* rfill, const double* temp, const int64_t* scf_loop, const double* pp,
                          const double* eps, const int64_t* Nkall, const int64_t* Nk, const int64_t* Nw,
                          const int64_t* Norb, const int64_t* Nchi, const int64_t* Nx, const int64_t* Ny,
                          const int64_t* Nz, const int64_t* sub_sigma, const int64_t* m_diis, const bool* sw_rescale,
                          const bool* sw_tail, const int64_t* gap_sym, const int64_t* arnoldi_m,
                          const int64_t* itemax, const double* eps_eliash, const int64_t* coarse) {
  ABI_TRY
  ensure_context();
  PipelineArgs a{sigmak, mu, delta, lambda_out, stoner, times_ms, Smat, Cmat, kmap, invk, olist, hamk, eig, uni,
                 init_delta, prt, sigma_seed, seed_mu ? *seed_mu : 0.0, seed_mu_old ? *seed_mu_old : 0.0, *mu_init,
                 *rfill, *temp, *scf_loop, *pp, *eps, *Nkall, *Nk, *Nw, *Norb, *Nchi, *Nx, *Ny, *Nz, *sub_sigma,
                 *m_diis, *sw_rescale, *sw_tail, *gap_sym, *arnoldi_m, *itemax, *eps_eliash};
  if (coarse) {
    PGB_CHECK(coarse[0] >= 1 && coarse[1] >= 1, "coarse divisors must be >= 1");
    a.coarse_kdiv = coarse[0];
    a.coarse_wdiv = coarse[1];
  }
  run_pipeline(a, ctx().precision);
  ABI_CATCH("pyrpa_gb_flex_eliash", (nan_fill(sigmak, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)),
                                     nan_fill(delta, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)), *mu = NAN,
                                     *lambda_out = NAN))
}

void pyrpa_gb_regrid_sigma(double2* out, const double2* sig, const int64_t* Nk, const int64_t* Nw_old,
                           const int64_t* Nw_new, const int64_t* Norb, const double* temp_old, const double* temp_new,
                           const double* w_scale) {
  ABI_TRY
  ensure_context();
  const long long n_old = (*Nk) * (*Nw_old) * (*Norb) * (*Norb), n_new = (*Nk) * (*Nw_new) * (*Norb) * (*Norb);
  DBuf<double2> s(n_old), o(n_new);
  s.upload(sig, n_old);
  regrid_sigma(o.p, s.p, (int)*Nk, (int)*Nw_old, (int)*Nw_new, (int)*Norb, *temp_old, *temp_new, *w_scale);
  o.download(out, n_new);
  sync();
  ABI_CATCH("pyrpa_gb_regrid_sigma", nan_fill(out, (size_t)(*Nk) * (*Nw_new) * (*Norb) * (*Norb)))
}

}  // extern "C"

namespace {

// Every record of a gfortran sequential file (4-byte length, payload, the
// same length again).  The scan stops at the first record whose markers
// do not close, so a damaged tail reads as an absent footer.
std::vector<std::string> sequential_records(const char* path) {
  std::ifstream f(path, std::ios::binary);
  if (!f.good()) throw BadInput(std::string("cannot open ") + path);
  std::vector<std::string> out;
  for (;;) {
    int32_t head = 0, tail = -1;
    if (!f.read(reinterpret_cast<char*>(&head), 4) || head < 0) break;
    std::string body((size_t)head, '\0');
    if (head && !f.read(&body[0], head)) break;
    if (!f.read(reinterpret_cast<char*>(&tail), 4) || tail != head) break;
    out.push_back(std::move(body));
  }
  return out;
}

void put_record(std::ofstream& f, const void* p, size_t n) {
  if (n >= 2147483639ULL) throw Error("a sigma.bin record above 2 GiB is not supported");
  const int32_t len = (int32_t)n;
  f.write(reinterpret_cast<const char*>(&len), 4);
  f.write(reinterpret_cast<const char*>(p), (std::streamsize)n);
  f.write(reinterpret_cast<const char*>(&len), 4);
}

// |given - stored| <= 1e-8 |stored|: the footer agreement test of the seed regrid
void footer_agrees(const char* what, double given, double stored) {
  if (!(std::fabs(given - stored) <= 1e-8 * std::fabs(stored)))
    throw BadInput(std::string(what) + " = " + std::to_string(given) + " disagrees with the value " +
                   std::to_string(stored) + " stored in the file's (temp, Nw, Norb, Nk) record");
}

}  // namespace

extern "C" {

void pyrpa_gb_regrid_sigma_file(const char* in_path, const char* out_path, const double* temp_old,
                                const double* temp_new, const int64_t* Norb, const int64_t* Nw_old,
                                const int64_t* Nw_new, const double* w_scale, int64_t* Nk_out,
                                int64_t* Nw_new_out) {
  ABI_TRY
  *Nk_out = *Nw_new_out = -1;
  if (!std::isfinite(*temp_new)) throw BadInput("the target temperature temp_new must be given");
  const std::vector<std::string> rec = sequential_records(in_path);
  if (rec.size() < 3 || rec[0].size() != 8 || rec[1].size() != 8 || rec[2].size() % sizeof(double2))
    throw BadInput(std::string(in_path) + " does not start with the mu, mu_OLD and Sigma records of io_sigma");
  const bool footer = rec.size() >= 4 && rec[3].size() == 4 * sizeof(double);
  double t_old = *temp_old;
  int64_t nw_old = *Nw_old, norb = *Norb;
  double meta[4] = {0, 0, 0, 0};
  if (footer) {
    memcpy(meta, rec[3].data(), sizeof(meta));
    if (std::isfinite(t_old)) footer_agrees("temp_old", t_old, meta[0]);
    if (nw_old > 0) footer_agrees("Nw_old", (double)nw_old, (double)std::llround(meta[1]));
    if (norb > 0) footer_agrees("Norb", (double)norb, (double)std::llround(meta[2]));
    t_old = meta[0];
    nw_old = std::llround(meta[1]);
    norb = std::llround(meta[2]);
  } else if (!std::isfinite(t_old) || nw_old <= 0 || norb <= 0) {
    throw BadInput(std::string(in_path) + " has no (temp, Nw, Norb, Nk) record, so temp_old, Norb and Nw_old "
                   "have to be passed");
  }
  if (nw_old <= 0 || norb <= 0) throw BadInput("the stored Nw and Norb must be positive");
  const int64_t nw_new = *Nw_new > 0 ? *Nw_new : nw_old;
  const int64_t nvals = (int64_t)(rec[2].size() / sizeof(double2)), per_k = nw_old * norb * norb;
  if (nvals % per_k)
    throw BadInput("the Sigma record holds " + std::to_string(nvals) + " values, not a multiple of Nw_old*Norb^2 = " +
                   std::to_string(per_k));
  const int64_t nk = nvals / per_k;
  if (footer && nk != std::llround(meta[3]))
    throw BadInput("the Sigma record gives Nk = " + std::to_string(nk) + " but the file's last record says " +
                   std::to_string(std::llround(meta[3])));
  ensure_context();
  DBuf<double2> s(nvals), o(nk * nw_new * norb * norb);
  s.upload(reinterpret_cast<const double2*>(rec[2].data()), nvals);
  regrid_sigma(o.p, s.p, (int)nk, (int)nw_old, (int)nw_new, (int)norb, t_old, *temp_new, *w_scale);
  std::vector<double2> host((size_t)(nk * nw_new * norb * norb));
  o.download(host.data(), (long long)host.size());
  sync();
  std::ofstream f(out_path, std::ios::binary | std::ios::trunc);
  if (!f.good()) throw BadInput(std::string("cannot write ") + out_path);
  put_record(f, rec[0].data(), 8);
  put_record(f, rec[1].data(), 8);
  put_record(f, host.data(), host.size() * sizeof(double2));
  const double footer_new[4] = {*temp_new, (double)nw_new, (double)norb, (double)nk};
  put_record(f, footer_new, sizeof(footer_new));
  f.close();
  if (!f) throw Error(std::string("writing ") + out_path + " failed");
  *Nk_out = nk;
  *Nw_new_out = nw_new;
  ABI_CATCH("pyrpa_gb_regrid_sigma_file", (*Nk_out = -1, *Nw_new_out = -1))
}

void pyrpa_gb_wannier_r(double2* out, const double2* data, const int64_t* kmap, const int64_t* invk,
                        const int64_t* Nx, const int64_t* Ny, const int64_t* Nz, const int64_t* Nk_data,
                        const int64_t* Nw, const int64_t* Norb, const int64_t* Ncut) {
  ABI_TRY
  ensure_context();
  const int64_t nkall = (*Nx) * (*Ny) * (*Nz), no = *Norb, nw = *Nw, ncut = std::min(*Ncut, *Nw);
  PGB_CHECK(*Ncut >= 1, "N_cut must be positive");
  const bool full_bz = (*Nk_data == nkall) && (irr_count(*Nx, *Ny, *Nz) != nkall);
  int64_t nk = *Nk_data;
  if (full_bz) nk = irr_count(*Nx, *Ny, *Nz);
  Geom g;
  build_geom(g, kmap, invk, *Nx, *Ny, *Nz, nk, 1, no, no * no <= kMaxChi ? no * no : 1);
  const long long n_in = (*Nk_data) * nw * no * no, n_out = nkall * ncut * no * no;
  DBuf<double2> d(n_in), o(n_out);
  d.upload(data, n_in);
  wannier_r(o.p, d.p, g, (int)nw, (int)no, (int)ncut, full_bz);
  o.download(out, n_out);
  sync();
  ABI_CATCH("pyrpa_gb_wannier_r", nan_fill(out, (size_t)((*Nx) * (*Ny) * (*Nz) * std::min(*Ncut, *Nw) * (*Norb) * (*Norb))))
}

// -------------------------------------------------------- FFT tuning --
void pyrpa_gb_fft_candidates(const int64_t* n, const int64_t* elem_bytes, int64_t* out, const int64_t* cap,
                             int64_t* count) {
  ABI_TRY
  const std::vector<AxisTune> c = fft_axis_candidates((int)*n, (int)*elem_bytes);
  *count = (int64_t)c.size();
  for (size_t i = 0; i < c.size() && (int64_t)i < *cap; ++i) {
    out[2 * i] = c[i].L1;
    out[2 * i + 1] = c[i].lines;
  }
  ABI_CATCH("pyrpa_gb_fft_candidates", *count = -1)
}

// ------------------------------------------------- coarse-mesh seed --
void pyrpa_gb_sigma_interp(double2* sig_f, const double2* sig_c, const int64_t* kmap_c, const int64_t* invk_c,
                           const int64_t* Nx_c, const int64_t* Ny_c, const int64_t* Nz_c, const int64_t* Nk_c,
                           const int64_t* Nw_c, const int64_t* kmap_f, const int64_t* invk_f, const int64_t* Nx_f,
                           const int64_t* Ny_f, const int64_t* Nz_f, const int64_t* Nk_f, const int64_t* Nw_f,
                           const int64_t* Norb, const double* temp) {
  ABI_TRY
  ensure_context();
  const int64_t no = *Norb;
  PGB_CHECK(no >= 1 && no <= 8, "Norb must be in [1, 8]");
  PGB_CHECK(*Nw_c >= 1 && *Nw_f >= *Nw_c, "the fine Matsubara set must hold the coarse one");
  const int64_t nchi = no * no <= kMaxChi ? no * no : 1;
  Geom gc, gf;
  build_geom(gc, kmap_c, invk_c, *Nx_c, *Ny_c, *Nz_c, *Nk_c, *Nw_c, no, nchi);
  build_geom(gf, kmap_f, invk_f, *Nx_f, *Ny_f, *Nz_f, *Nk_f, *Nw_f, no, nchi);
  const size_t nc = (size_t)(*Nk_c) * (*Nw_c) * no * no, nf = (size_t)(*Nk_f) * (*Nw_f) * no * no;
  DBuf<double2> c(nc), f(nf);
  c.upload(sig_c, nc);
  sigma_interp(gc, gf, c.p, f.p, (int)no, *temp);
  f.download(sig_f, nf);
  sync();
  ABI_CATCH("pyrpa_gb_sigma_interp", nan_fill(sig_f, (size_t)(*Nk_f) * (*Nw_f) * (*Norb) * (*Norb)))
}

// --------------------------------------------------- learned warm start --
static LwsDesc lws_desc(const double* d) { return LwsDesc{d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], d[8]}; }

void pyrpa_gb_lws_create(int64_t* handle) {
  ABI_TRY *handle = lws_create();
  ABI_CATCH("pyrpa_gb_lws_create", *handle = 0)
}
void pyrpa_gb_lws_destroy(const int64_t* handle) {
  ABI_TRY lws_destroy(*handle);
  ABI_CATCH("pyrpa_gb_lws_destroy", (void)0)
}
void pyrpa_gb_lws_set_params(const int64_t* handle, const float* theta, const int64_t* n) {
  ABI_TRY ensure_context(); lws_set_params(lws_get(*handle), theta, *n);
  ABI_CATCH("pyrpa_gb_lws_set_params", (void)0)
}
void pyrpa_gb_lws_get_params(const int64_t* handle, float* theta, const int64_t* n) {
  ABI_TRY ensure_context(); lws_get_params(lws_get(*handle), theta, *n);
  ABI_CATCH("pyrpa_gb_lws_get_params", nan_fill_f(theta, (size_t)*n))
}
void pyrpa_gb_lws_add_samples(const int64_t* handle, const double2* sig_seed, const double2* sig_fine,
                              const double2* uni, const double* eig, const int64_t* kn, const int64_t* npairs,
                              const int64_t* Nk, const int64_t* Nw, const int64_t* Nw_c, const int64_t* Norb,
                              const double* desc) {
  ABI_TRY
  ensure_context();
  lws_add_samples(lws_get(*handle), sig_seed, sig_fine, uni, eig, kn, *npairs, (int)*Nk, (int)*Nw, (int)*Nw_c,
                  (int)*Norb, lws_desc(desc));
  ABI_CATCH("pyrpa_gb_lws_add_samples", (void)0)
}
void pyrpa_gb_lws_clear_samples(const int64_t* handle) {
  ABI_TRY ensure_context(); lws_clear_samples(lws_get(*handle));
  ABI_CATCH("pyrpa_gb_lws_clear_samples", (void)0)
}
void pyrpa_gb_lws_num_samples(const int64_t* handle, int64_t* rows) {
  ABI_TRY *rows = lws_get(*handle).M;
  ABI_CATCH("pyrpa_gb_lws_num_samples", *rows = -1)
}
void pyrpa_gb_lws_features(float* x, float* t, const double2* sig_seed, const double2* sig_fine, const double2* uni,
                           const double* eig, const int64_t* kn, const int64_t* npairs, const int64_t* Nk,
                           const int64_t* Nw, const int64_t* Nw_c, const int64_t* Norb, const double* desc) {
  ABI_TRY
  lws_features_host(x, t, sig_seed, sig_fine, uni, eig, kn, *npairs, (int)*Nk, (int)*Nw, (int)*Nw_c, (int)*Norb,
                    lws_desc(desc));
  ABI_CATCH("pyrpa_gb_lws_features", nan_fill_f(x, (size_t)(*npairs) * (*Norb) * (*Norb) * kLwsNF))
}
void pyrpa_gb_lws_forward(const int64_t* handle, const float* x, const int64_t* rows, float* y) {
  ABI_TRY ensure_context(); lws_forward_host(lws_get(*handle), x, *rows, y);
  ABI_CATCH("pyrpa_gb_lws_forward", nan_fill_f(y, (size_t)(*rows) * 2))
}
void pyrpa_gb_lws_loss_grad(const int64_t* handle, double* loss, float* grad) {
  ABI_TRY ensure_context(); *loss = lws_loss_grad(lws_get(*handle), grad);
  ABI_CATCH("pyrpa_gb_lws_loss_grad", (*loss = std::numeric_limits<double>::quiet_NaN(),
                                       nan_fill_f(grad, (size_t)kLwsNParam)))
}
void pyrpa_gb_lws_step(const int64_t* handle, const double* lr, const double* beta1, const double* beta2,
                       const double* eps, double* loss) {
  ABI_TRY ensure_context(); lws_step_full(lws_get(*handle), *lr, *beta1, *beta2, *eps, loss);
  ABI_CATCH("pyrpa_gb_lws_step", *loss = std::numeric_limits<double>::quiet_NaN())
}
void pyrpa_gb_lws_train(const int64_t* handle, const int64_t* steps, const int64_t* batch, const double* lr,
                        const double* beta1, const double* beta2, const double* eps, const int64_t* seed,
                        double* loss) {
  ABI_TRY
  ensure_context();
  lws_train(lws_get(*handle), *steps, *batch, *lr, *beta1, *beta2, *eps, (uint64_t)*seed, loss);
  ABI_CATCH("pyrpa_gb_lws_train", nan_fill(loss, (size_t)std::max<int64_t>(0, *steps)))
}
void pyrpa_gb_lws_apply(const int64_t* handle, double2* sigma, const double2* uni, const double* eig,
                        const int64_t* Nk, const int64_t* Nw, const int64_t* Nw_c, const int64_t* Norb,
                        const double* desc) {
  ABI_TRY
  ensure_context();
  lws_apply(lws_get(*handle), sigma, uni, eig, (int)*Nk, (int)*Nw, (int)*Nw_c, (int)*Norb, lws_desc(desc));
  ABI_CATCH("pyrpa_gb_lws_apply", nan_fill(sigma, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)))
}

void eliashberg(double2* delta, double2* sigmak, double2* Gk, const double2* hamk, const double* Smat,
                const double* Cmat, const int64_t* olist, const double* prt, const int64_t* kmap, const int64_t* invk,
                const double* mu, const double* temp, const double* eps, const int64_t* Nkall, const int64_t* Nk,
                const int64_t* Nw, const int64_t* Nchi, const int64_t* Norb, const int64_t* Nx, const int64_t* Ny,
                const int64_t* Nz, const int64_t* itemax, const int64_t* gap_sym, const bool* sw_sigma,
                const bool* sw_Vconst, const int64_t* m_diis, const double* gap_min, const bool* sw_amp_newton) {
  ABI_TRY
  ensure_context();
  NonlinArgs a{delta, sigmak, Gk, hamk, Smat, Cmat, olist, prt, kmap, invk, *mu, *temp, *eps, *Nkall, *Nk, *Nw,
               *Nchi, *Norb, *Nx, *Ny, *Nz, *itemax, *gap_sym, *sw_sigma, *sw_Vconst, *m_diis, *gap_min,
               *sw_amp_newton};
  run_nonlin_eliash(a);
  ABI_CATCH("eliashberg", (nan_fill(delta, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)),
                           nan_fill(sigmak, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb))))
}

void pyrpa_gb_chi0sc(double2* xs, double2* xc, const double2* Gk, const double2* Fk, const double* Smat,
                     const double* Cmat, const int64_t* olist, const double* prt, const int64_t* kmap,
                     const int64_t* invk, const double* temp, const int64_t* Nkall, const int64_t* Nk,
                     const int64_t* Nw, const int64_t* Nchi, const int64_t* Norb, const int64_t* Nx, const int64_t* Ny,
                     const int64_t* Nz, const int64_t* gap_sym, const int64_t* vertex) {
  ABI_TRY
  ensure_context();
  nonlin_bubbles(xs, xc, Gk, Fk, Smat, Cmat, olist, prt, kmap, invk, *temp, *Nkall, *Nk, *Nw, *Nchi, *Norb, *Nx, *Ny,
                 *Nz, *gap_sym >= 0, *vertex != 0);
  ABI_CATCH("pyrpa_gb_chi0sc", (nan_fill(xs, (size_t)(*Nk) * (*Nw) * (*Nchi) * (*Nchi)),
                                nan_fill(xc, (size_t)(*Nk) * (*Nw) * (*Nchi) * (*Nchi))))
}

void pyrpa_gb_sc_dyson(double2* Gk, double2* fk, const double2* G0, const double2* delta, const int64_t* Nk,
                       const int64_t* Nw, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  const long long K = (*Nk) * (*Nw), KE = K * no * no;
  DBuf<double2> G(KE), F(KE), G0d(KE), D(KE);
  G0d.upload(G0, KE);
  F.upload(fk, KE);
  D.upload(delta, KE);
  mkgreliah(G.p, G0d.p, F.p, D.p, K, (int)no);
  mkfkeliash(F.p, G0d.p, G.p, D.p, K, (int)no);
  G.download(Gk, KE);
  F.download(fk, KE);
  sync();
  ABI_CATCH("pyrpa_gb_sc_dyson", (nan_fill(Gk, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)),
                                  nan_fill(fk, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb))))
}

// -------------------------------------------------------- real frequency --
// k+q lookups (fchi.f90:1-93, fphi.f90:1-87): coordinates keyed at 2^-20 as
// int(x*2^20 + 0.5) mod 2^20 (Fortran truncation and sign of the dividend); a
// repeated key keeps the last index; a miss falls back to index 1.
namespace {
constexpr int64_t kKeyScale = 1048576;
int64_t kkey(const double* x) {
  int64_t k[3];
  for (int c = 0; c < 3; ++c) {
    const int64_t i = (int64_t)(x[c] * (double)kKeyScale + 0.5);  // truncation toward zero
    k[c] = i % kKeyScale;                                            // C++ %: sign of the dividend
  }
  return k[0] + k[1] * kKeyScale + k[2] * kKeyScale * kKeyScale;
}
void kq_lookup(int64_t* out, const double* qpoint, const double* klist, int64_t Nk, bool minus_k) {
  std::unordered_map<int64_t, int64_t> table;
  table.reserve((size_t)Nk * 2);
  for (int64_t j = 0; j < Nk; ++j) table[kkey(klist + 3 * j)] = j + 1;
  int64_t nmiss = 0;
  for (int64_t i = 0; i < Nk; ++i) {
    double t[3];
    for (int c = 0; c < 3; ++c) {
      t[c] = (minus_k ? 1.0 - klist[3 * i + c] : klist[3 * i + c]) + qpoint[c];
      if (t[c] >= 1.0) t[c] -= 1.0;
      else if (t[c] < 0.0) t[c] += 1.0;
    }
    auto it = table.find(kkey(t));
    if (it == table.end()) {
      out[i] = 1;
      ++nmiss;
    } else {
      out[i] = it->second;
    }
  }
  if (nmiss > 0)
    log("WARNING(get_%sqshift): %lld of %lld k+q points not found on the k-mesh.\n", minus_k ? "i" : "",
        (long long)nmiss, (long long)Nk);
}

struct RfInputs {
  DBuf<double2> uni;
  DBuf<double> eig, ff;
  std::vector<int> o1, o2;
};
void rf_upload(RfInputs& r, const double2* uni, const double* eig, const double* ffermi, const int64_t* ol,
               int64_t Nchi, int64_t Norb, int64_t Nk) {
  PGB_CHECK(Norb <= kMaxOrb && Nchi <= kMaxChi, "Norb or Nchi above the engine limits");
  r.uni.alloc((size_t)Norb * Norb * Nk);
  r.uni.upload(uni, (size_t)Norb * Norb * Nk);
  r.eig.alloc((size_t)Norb * Nk);
  r.eig.upload(eig, (size_t)Norb * Nk);
  r.ff.alloc((size_t)Norb * Nk);
  r.ff.upload(ffermi, (size_t)Norb * Nk);
  r.o1.resize(Nchi);
  r.o2.resize(Nchi);
  for (int64_t l = 0; l < Nchi; ++l) {
    r.o1[l] = (int)ol[l] - 1;
    r.o2[l] = (int)ol[Nchi + l] - 1;
    PGB_CHECK(r.o1[l] >= 0 && r.o1[l] < Norb && r.o2[l] >= 0 && r.o2[l] < Norb, "olist entry outside [1,Norb]");
  }
}
std::vector<int> qshift_0based(const int64_t* qs, int64_t Nk) {
  std::vector<int> out(Nk);
  for (int64_t i = 0; i < Nk; ++i) {
    PGB_CHECK(qs[i] >= 1 && qs[i] <= Nk, "qshift entry outside [1,Nk]");
    out[i] = (int)qs[i] - 1;
  }
  return out;
}
void rf_irr(double2* out, const double2* uni, const double* eig, const double* ffermi, const int64_t* qshift,
            const int64_t* ol, const double* wl, int64_t Nchi, int64_t Norb, int64_t Nk, int64_t Nw, double idelta,
            double eps, double mu, double temp, bool phi) {
  RfInputs r;
  rf_upload(r, uni, eig, ffermi, ol, Nchi, Norb, Nk);
  std::vector<int> qs = qshift_0based(qshift, Nk);
  DBuf<int> dq(Nk);
  dq.upload(qs.data(), Nk);
  std::vector<RfJob> jobs(Nw);
  for (int64_t w = 0; w < Nw; ++w) jobs[w] = RfJob{wl[w], idelta, 0};
  DBuf<double2> d((size_t)Nchi * Nchi * Nw);
  bubble_rf(d.p, r.uni.p, r.eig.p, r.ff.p, dq.p, jobs, r.o1, r.o2, (int)Nk, (int)Norb, (int)Nchi, mu, temp, eps, phi);
  d.download(out, (size_t)Nchi * Nchi * Nw);
  sync();
}
// q = ((i-1)/Nx, (j-1)/Ny, 0) in the reference's (i, j) order, job index i*Ny + j
std::vector<int> map_qshifts(const double* klist, int64_t Nx, int64_t Ny, int64_t Nk, bool minus_k) {
  std::vector<int> all((size_t)Nx * Ny * Nk);
  std::vector<int64_t> one(Nk);
  for (int64_t i = 0; i < Nx; ++i)
    for (int64_t j = 0; j < Ny; ++j) {
      const double q[3] = {(double)i / (double)Nx, (double)j / (double)Ny, 0.0};
      kq_lookup(one.data(), q, klist, Nk, minus_k);
      for (int64_t k = 0; k < Nk; ++k) all[(size_t)(i * Ny + j) * Nk + k] = (int)one[k] - 1;
    }
  return all;
}
}  // namespace

void get_qshift_(const double* qpoint, const double* klist, int64_t* qshift, const int64_t* Nk) {
  ABI_TRY
  kq_lookup(qshift, qpoint, klist, *Nk, false);
  ABI_CATCH("get_qshift_", (void)0)
}

void get_iqshift_(const double* qpoint, const double* klist, int64_t* qshift, const int64_t* Nk) {
  ABI_TRY
  kq_lookup(qshift, qpoint, klist, *Nk, true);
  ABI_CATCH("get_iqshift_", (void)0)
}

void get_chi_irr(double2* chi, const double2* uni, const double* eig, const double* ffermi, const int64_t* qshift,
                 const int64_t* ol, const double* wl, const int64_t* Nchi, const int64_t* Norb, const int64_t* Nk,
                 const int64_t* Nw, const double* idelta, const double* eps, const double* temp) {
  ABI_TRY
  ensure_context();
  rf_irr(chi, uni, eig, ffermi, qshift, ol, wl, *Nchi, *Norb, *Nk, *Nw, *idelta, *eps, 0.0, *temp, false);
  ABI_CATCH("get_chi_irr", nan_fill(chi, (size_t)(*Nchi) * (*Nchi) * (*Nw)))
}

void get_phi_irr(double2* phi, const double2* uni, const double* eig, const double* ffermi, const int64_t* qshift,
                 const int64_t* ol, const double* wl, const int64_t* Nchi, const int64_t* Norb, const int64_t* Nk,
                 const int64_t* Nw, const double* idelta, const double* eps, const double* mu, const double* temp) {
  ABI_TRY
  ensure_context();
  rf_irr(phi, uni, eig, ffermi, qshift, ol, wl, *Nchi, *Norb, *Nk, *Nw, *idelta, *eps, *mu, *temp, true);
  ABI_CATCH("get_phi_irr", nan_fill(phi, (size_t)(*Nchi) * (*Nchi) * (*Nw)))
}

void chiq_map(double2* trchis, double2* trchi, const double2* uni, const double* eig, const double* ffermi,
              const double* klist, const double* Smat, const int64_t* ol, const double* temp, const double* ecut,
              const double* idelta, const double* eps, const int64_t* Nx, const int64_t* Ny, const int64_t* Nk,
              const int64_t* Norb, const int64_t* Nchi) {
  ABI_TRY
  ensure_context();
  const int64_t nq = (*Nx) * (*Ny), n = *Nchi;
  RfInputs r;
  rf_upload(r, uni, eig, ffermi, ol, n, *Norb, *Nk);
  std::vector<int> qs = map_qshifts(klist, *Nx, *Ny, *Nk, false);
  DBuf<int> dq(qs.size());
  dq.upload(qs.data(), qs.size());
  std::vector<RfJob> jobs(nq);
  for (int64_t q = 0; q < nq; ++q) jobs[q] = RfJob{*ecut, *idelta, q * (*Nk)};
  DBuf<double2> chi((size_t)n * n * nq), ts(nq), t0(nq);
  bubble_rf(chi.p, r.uni.p, r.eig.p, r.ff.p, dq.p, jobs, r.o1, r.o2, (int)*Nk, (int)*Norb, (int)n, 0.0, *temp, *eps,
            false);
  std::vector<int> dmask(n);
  for (int64_t l = 0; l < n; ++l) dmask[l] = r.o1[l] == r.o2[l] ? 1 : 0;
  DBuf<int> dm(n);
  dm.upload(dmask.data(), n);
  DBuf<double> S((size_t)n * n);
  S.upload(Smat, (size_t)n * n);
  rpa_trace(ts.p, t0.p, chi.p, S.p, dm.p, (int)n, (int)nq);
  ts.download(trchis, nq);  // trchis(Ny, Nx): element (j, i) at j + Ny i = job i*Ny + j
  t0.download(trchi, nq);
  sync();
  ABI_CATCH("chiq_map", (nan_fill(trchis, (size_t)(*Nx) * (*Ny)), nan_fill(trchi, (size_t)(*Nx) * (*Ny))))
}

void phiq_map(double2* trphi, const double2* uni, const double* eig, const double* ffermi, const double* klist,
              const int64_t* ol, const double* mu, const double* temp, const double* ecut, const double* idelta,
              const double* eps, const int64_t* Nx, const int64_t* Ny, const int64_t* Nk, const int64_t* Norb,
              const int64_t* Nchi, const bool* sw_omega) {
  ABI_TRY
  ensure_context();
  const int64_t nq = (*Nx) * (*Ny), n = *Nchi;
  RfInputs r;
  rf_upload(r, uni, eig, ffermi, ol, n, *Norb, *Nk);
  std::vector<int> qs = map_qshifts(klist, *Nx, *Ny, *Nk, true);
  DBuf<int> dq(qs.size());
  dq.upload(qs.data(), qs.size());
  const double wre = *sw_omega ? *ecut : 0.0, wim = *sw_omega ? *idelta : 0.0;
  std::vector<RfJob> jobs(nq);
  for (int64_t q = 0; q < nq; ++q) jobs[q] = RfJob{wre, wim, q * (*Nk)};
  DBuf<double2> phi((size_t)n * n * nq), tr(nq);
  bubble_rf(phi.p, r.uni.p, r.eig.p, r.ff.p, dq.p, jobs, r.o1, r.o2, (int)*Nk, (int)*Norb, (int)n, *mu, *temp, *eps,
            true);
  trace_jobs(tr.p, phi.p, (int)n, (int)nq);
  tr.download(trphi, nq);
  sync();
  ABI_CATCH("phiq_map", nan_fill(trphi, (size_t)(*Nx) * (*Ny)))
}

// orbital traces of chi_s / chi_0 / phi per frequency (fchi.f90:160-196, fphi.f90:164-193)
void get_tr_chi(double2* trchis, double2* trchi0, double2* chis_orb, const double2* chis, const double2* chi0,
                const int64_t* olist, const int64_t* Nw, const int64_t* Nchi, const int64_t* Norb) {
  ABI_TRY
  const int64_t nw = *Nw, n = *Nchi, no = *Norb;
  for (int64_t i = 0; i < nw; ++i) {
    trchis[i] = mkc(0.0, 0.0);
    trchi0[i] = mkc(0.0, 0.0);
    for (int64_t o = 0; o < no + 2; ++o) chis_orb[o + (no + 2) * i] = mkc(0.0, 0.0);
  }
  for (int64_t i = 0; i < nw; ++i)
    for (int64_t j = 0; j < n; ++j) {
      if (olist[j] != olist[n + j]) continue;
      for (int64_t k = 0; k < n; ++k) {
        if (olist[k] != olist[n + k]) continue;
        const double2 cs = chis[k + n * (j + n * i)];
        trchis[i] += cs;
        trchi0[i] += chi0[k + n * (j + n * i)];
        if (olist[j] == olist[k]) {
          PGB_CHECK(olist[j] >= 1 && olist[j] <= no, "olist entry outside [1,Norb]");
          chis_orb[(olist[j] - 1) + (no + 2) * i] = cs;
        }
        if (olist[k] == 2 && olist[j] == 3) chis_orb[no + (no + 2) * i] = cs;
        if (olist[k] == 2 && olist[j] == 4) chis_orb[no + 1 + (no + 2) * i] = cs;
      }
    }
  ABI_CATCH("get_tr_chi", (void)0)
}

void get_tr_phi(double2* trphi, double2* phi_orb, const double2* phi, const int64_t* olist, const int64_t* Nw,
                const int64_t* Nchi, const int64_t* Norb) {
  ABI_TRY
  const int64_t nw = *Nw, n = *Nchi, no = *Norb;
  for (int64_t i = 0; i < nw; ++i) {
    trphi[i] = mkc(0.0, 0.0);
    for (int64_t o = 0; o < no + 2; ++o) phi_orb[o + (no + 2) * i] = mkc(0.0, 0.0);
  }
  for (int64_t i = 0; i < nw; ++i)
    for (int64_t j = 0; j < n; ++j) {
      trphi[i] += phi[j + n * (j + n * i)];
      if (olist[j] != olist[n + j]) continue;
      for (int64_t k = 0; k < n; ++k) {
        if (olist[k] != olist[n + k]) continue;
        const double2 v = phi[k + n * (j + n * i)];
        if (olist[j] == olist[k]) {
          PGB_CHECK(olist[j] >= 1 && olist[j] <= no, "olist entry outside [1,Norb]");
          phi_orb[(olist[j] - 1) + (no + 2) * i] = v;
        }
        if (olist[k] == 2 && olist[j] == 3) phi_orb[no + (no + 2) * i] = v;
        if (olist[k] == 2 && olist[j] == 4) phi_orb[no + 1 + (no + 2) * i] = v;
      }
    }
  ABI_CATCH("get_tr_phi", (void)0)
}

// Pade continued fraction of one series (fpade.f90:1-55), host code: the
// coefficients need Np^2/2 operations.  Only the entries j >= i of g_i are
// formed, the ones the later steps read.
void get_a_(double2* a, const double2* xn, const double2* inp, const int64_t* Np) {
  ABI_TRY
  const int64_t n = *Np;
  std::vector<double2> g(inp, inp + n);
  if (n > 0) a[0] = g[0];
  for (int64_t i = 1; i < n; ++i) {
    const double2 gp = g[i - 1], xp = xn[i - 1];
    for (int64_t j = i; j < n; ++j) {
      const double2 gj = g[j];
      g[j] = (gj.x == 0.0 && gj.y == 0.0) ? mkc(0.0, 0.0) : cdiv(gp - gj, (xn[j] - xp) * gj);
    }
    a[i] = g[i];
  }
  ABI_CATCH("get_a_", (void)0)
}

void get_qp_(double2* P, double2* Q, const double2* a, const double2* xn, const double2* wlist, const int64_t* Nw,
             const int64_t* Np) {
  ABI_TRY
  for (int64_t w = 0; w < *Nw; ++w) {
    double2 P0 = mkc(0.0, 0.0), P1 = a[0], Q0 = mkc(1.0, 0.0), Q1 = mkc(1.0, 0.0);
    for (int64_t i = 1; i < *Np; ++i) {
      const double2 t = a[i] * (wlist[w] - xn[i - 1]);
      const double2 p = P1 + t * P0, q = Q1 + t * Q0;
      P0 = P1;
      P1 = p;
      Q0 = Q1;
      Q1 = q;
    }
    P[w] = P1;
    Q[w] = Q1;
  }
  ABI_CATCH("get_qp_", (void)0)
}

void pade_with_trace(const double2* arrayin, double2* arrayout, const double2* iwlist, const double2* wlist,
                     const int64_t* Nk, const int64_t* Niw, const int64_t* Nw, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t nk = *Nk, np = *Niw, nw = *Nw, no = *Norb;
  PGB_CHECK(np >= 1, "pade_with_trace needs at least one Matsubara point");
  DBuf<double2> A((size_t)nk * np * no * no), xn(np), wl(nw), out((size_t)nw * nk);
  A.upload(arrayin, (size_t)nk * np * no * no);
  xn.upload(iwlist, np);
  wl.upload(wlist, nw);
  pade_trace(out.p, A.p, xn.p, wl.p, (int)nk, (int)np, (int)nw, (int)no);
  out.download(arrayout, (size_t)nw * nk);
  sync();
  ABI_CATCH("pade_with_trace", nan_fill(arrayout, (size_t)(*Nw) * (*Nk)))
}

// ------------------------------------------------------------ spin-orbit --
// Onsite vertex with spin-orbit coupling (fUJ.f90:109-180 and, with
// orbital-dependent U/J, :182-251); host code, written as V(j,i).
namespace {
void vmat_soc(double* Vmat, const int64_t* ol, const int64_t* sl, const int64_t* site, const int64_t* invs,
              double U, double J, const double* Umat, const double* Jmat, int64_t n, int64_t no) {
  const double Up = U - 2 * J;
  const bool orb = Umat != nullptr;
  auto Uf = [&](int64_t a, int64_t b) { return Umat[a + no * b]; };  // 0-based
  auto Jf = [&](int64_t a, int64_t b) { return Jmat[a + no * b]; };
  auto inv = [&](int64_t a) { return invs[a] - 1; };
  auto s = [&](int64_t a) { return sl[a]; };
  for (int64_t i = 0; i < n; ++i)
    for (int64_t j = 0; j < n; ++j) {
      double v = 0.0;
      const int64_t i1 = ol[i] - 1, i2 = ol[n + i] - 1, j1 = ol[j] - 1, j2 = ol[n + j] - 1;
      PGB_CHECK(i1 >= 0 && i1 < no && i2 >= 0 && i2 < no && j1 >= 0 && j1 < no && j2 >= 0 && j2 < no,
                "olist entry outside [1,Norb]");
      if (site[i] == site[j]) {
        if (s(i1) == s(i2) && s(j1) == s(j2)) {
          if (s(i1) == s(j1)) {  // equal spins: (C-S)/2
            if (i1 == j2 && j1 == i2) {
              v = 0.0;
            } else if (i1 == i2 && j1 == j2) {
              v = orb ? Uf(i1, j1) - Jf(i1, j1) : Up - J;
            } else if (i1 == j1 && i2 == j2) {
              v = orb ? Jf(i1, i2) - Uf(i1, i2) : J - Up;
            }
          } else {  // opposite spins: (C+S)/2
            if (i1 == i2 && j1 == j2) {
              v = i1 == inv(j1) ? (orb ? Uf(i1, i1) : U) : (orb ? Uf(i1, j1) : Up);
            } else if (i1 == inv(j1) && i2 == inv(j2)) {
              v = orb ? Jf(i1, i2) : J;
            } else if (i1 == inv(j2) && j1 == inv(i2)) {
              v = orb ? Jf(i1, i2) : J;
            }
          }
        } else if (s(i1) == s(j1) && s(i2) == s(j2)) {  // spin flip: -S
          if (i1 == inv(i2) && j1 == inv(j2)) {
            v = i1 == j1 ? -(orb ? Uf(i1, i1) : U) : -(orb ? Jf(i1, j1) : J);
          } else if (i1 == j1 && i2 == j2) {
            v = -(orb ? Uf(i1, i2) : Up);
          } else if (i1 == inv(j2) && j1 == inv(i2)) {
            v = -(orb ? Jf(i1, i2) : J);
          }
        }
      }
      Vmat[j + n * i] = v;
    }
}
}  // namespace

void get_vmat_soc(double* Vmat, const int64_t* ol, const int64_t* sl, const int64_t* site, const int64_t* invs,
                  const double* Uval, const double* Jval, const int64_t* Nchi, const int64_t* Norb) {
  ABI_TRY
  vmat_soc(Vmat, ol, sl, site, invs, *Uval, *Jval, nullptr, nullptr, *Nchi, *Norb);
  ABI_CATCH("get_vmat_soc", nan_fill(Vmat, (size_t)(*Nchi) * (*Nchi)))
}

void get_vmat_soc_orb(double* Vmat, const int64_t* ol, const int64_t* sl, const int64_t* site, const int64_t* invs,
                      const double* Umat, const double* Jmat, const int64_t* Nchi, const int64_t* Norb) {
  ABI_TRY
  vmat_soc(Vmat, ol, sl, site, invs, 0.0, 0.0, Umat, Jmat, *Nchi, *Norb);
  ABI_CATCH("get_vmat_soc_orb", nan_fill(Vmat, (size_t)(*Nchi) * (*Nchi)))
}

void mkself_soc(double2* sigmak, double* mu, const double* Vmat, const int64_t* kmap, const int64_t* invk,
                const int64_t* invs, const int64_t* olist, const int64_t* slist, const double2* hamk, const double* eig,
                const double2* uni, const double* mu_init, const double* rfill, const double* temp,
                const int64_t* scf_loop, const double* pp, const double* eps, const int64_t* Nkall, const int64_t* Nk,
                const int64_t* Nw, const int64_t* Norb, const int64_t* Nchi, const int64_t* Nx, const int64_t* Ny,
                const int64_t* Nz, const int64_t* sub_sigma, const bool* sw_out, const bool* sw_in,
                const int64_t* m_diis, const bool* sw_rescale, const double* sigma_scale) {
  ABI_TRY
  ensure_context();
  MkselfArgs a{sigmak, mu, Vmat, Vmat, kmap, invk, olist, hamk, eig, uni, *mu_init, *rfill, *temp, *scf_loop, *pp,
               *eps, *Nkall, *Nk, *Nw, *Norb, *Nchi, *Nx, *Ny, *Nz, *sub_sigma, *sw_out, *sw_in, *m_diis,
               *sw_rescale, false, *sigma_scale};
  run_mkself_soc(a, SocSpin{invs, slist});
  ABI_CATCH("mkself_soc", (nan_fill(sigmak, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)), *mu = NAN))
}

void get_chi0_soc(double2* chi, double* sgnsig, double* sgnsig2, int64_t* invschi, const double* Vmat,
                  const double2* Gk, const int64_t* kmap, const int64_t* invk, const int64_t* invs,
                  const int64_t* olist, const int64_t* slist, const double* temp, const int64_t* Nx, const int64_t* Ny,
                  const int64_t* Nz, const int64_t* Nw, const int64_t* Nk, const int64_t* Nkall, const int64_t* Nchi,
                  const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t n = *Nchi, no = *Norb;
  // sign tables and the spin-flipped chi index (fchi0withsoc.f90:136-154, 200-214)
  for (int64_t j = 0; j < no; ++j)
    for (int64_t i = 0; i < no; ++i) sgnsig[i + no * j] = (double)(slist[i] * slist[j]);
  auto ps = [&](int64_t l) { return slist[olist[l] - 1] * slist[olist[n + l] - 1]; };
  for (int64_t j = 0; j < n; ++j)
    for (int64_t i = 0; i < n; ++i) sgnsig2[i + n * j] = (double)(ps(i) * ps(j));
  for (int64_t l = 0; l < n; ++l) {
    invschi[l] = 0;
    const int64_t i = invs[olist[l] - 1], j = invs[olist[n + l] - 1];
    for (int64_t m = 0; m < n; ++m)
      if (olist[m] == i && olist[n + m] == j) {
        invschi[l] = m + 1;
        break;
      }
  }
  run_chi0_soc(chi, Vmat, Gk, kmap, invk, olist, SocSpin{invs, slist}, *temp, *Nx, *Ny, *Nz, *Nw, *Nk, *Nkall, n, no);
  ABI_CATCH("get_chi0_soc", nan_fill(chi, (size_t)(*Nk) * (*Nw) * (*Nchi) * (*Nchi)))
}

void get_chis_chic_soc(double2* chic, double2* chiszz, double2* chispm, const double2* chi, const double* Vmat,
                       const int64_t* orb_list, const int64_t* olist, const int64_t* slist, const int64_t* invs,
                       const int64_t* Nk, const int64_t* Nw, const int64_t* Nchi, const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  (void)invs;
  run_chis_chic_soc(chic, chiszz, chispm, chi, Vmat, orb_list, olist, slist, *Nk, *Nw, *Nchi, *Norb);
  ABI_CATCH("get_chis_chic_soc", (nan_fill(chic, (size_t)(*Nk) * (*Nchi / 4) * (*Nchi / 4)),
                                  nan_fill(chiszz, (size_t)(*Nk) * (*Nchi / 4) * (*Nchi / 4)),
                                  nan_fill(chispm, (size_t)(*Nk) * (*Nchi / 4) * (*Nchi / 4))))
}

void lin_eliash_soc(double2* delta, double2* chi, const double2* Gk, const double2* uni, const double* init_delta,
                    const double* Vmat, const double* sgnsig, const double* sgnsig2, const double* prt,
                    const int64_t* olist, const int64_t* slist, const int64_t* kmap, const int64_t* invk,
                    const int64_t* invs, const int64_t* invschi, const double* temp, const double* eps,
                    const int64_t* Nkall, const int64_t* Nk, const int64_t* Nw, const int64_t* Nchi,
                    const int64_t* Norb, const int64_t* Nx, const int64_t* Ny, const int64_t* Nz,
                    const int64_t* itemax, const int64_t* gap_sym, const int64_t* arnoldi_m) {
  ABI_TRY
  ensure_context();
  (void)sgnsig;  // recomputed from slist
  (void)sgnsig2;
  (void)prt;
  LinEliashSocArgs a{delta, chi, Gk, uni, init_delta, Vmat, olist, kmap, invk, invschi, SocSpin{invs, slist},
                     *temp, *eps, *Nkall, *Nk, *Nw, *Nchi, *Norb, *Nx, *Ny, *Nz, *itemax, *gap_sym, *arnoldi_m};
  run_lin_eliash_soc(a);
  ABI_CATCH("lin_eliash_soc", nan_fill(delta, (size_t)(*Nkall) * (*Nw) * (*Norb) * (*Norb)))
}

void mkfk_trs_soc_(double2* fk, const double2* Gk, const double2* delta, const double* sgnsig, const int64_t* slist,
                   const int64_t* invk, const int64_t* invs, const int64_t* Nkall, const int64_t* Nk,
                   const int64_t* Nw, const int64_t* Norb, const int64_t* gap_sym) {
  ABI_TRY
  ensure_context();
  (void)sgnsig;
  run_mkfk_soc(fk, Gk, delta, invk, SocSpin{invs, slist}, *Nkall, *Nk, *Nw, *Norb, *gap_sym);
  ABI_CATCH("mkfk_trs_soc_", nan_fill(fk, (size_t)(*Nkall) * (*Nw) * (*Norb) * (*Norb)))
}

void conv_delta_orb_to_band_soc(double2* deltab, const double2* delta, const double2* uni, const int64_t* invk,
                                const int64_t* invs, const int64_t* slist, const int64_t* Norb, const int64_t* Nkall,
                                const int64_t* Nk, const int64_t* Nw) {
  ABI_TRY
  ensure_context();
  run_orb_to_band_soc(deltab, delta, uni, invk, SocSpin{invs, slist}, *Norb, *Nkall, *Nk, *Nw);
  ABI_CATCH("conv_delta_orb_to_band_soc", nan_fill(deltab, (size_t)(*Nkall) * (*Norb) * (*Norb)))
}

void mkfk_trs_nsoc_(double2* fk, const double2* Gk, const double2* delta, const int64_t* Nk, const int64_t* Nw,
                    const int64_t* Norb) {
  ABI_TRY
  ensure_context();
  const int64_t no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  const long long K = (*Nk) * (*Nw), KE = K * no * no;
  DBuf<double2> G(KE), D(KE), F(KE);
  G.upload(Gk, KE);
  D.upload(delta, KE);
  mkfk(F.p, G.p, D.p, K, (int)no);
  F.download(fk, KE);
  sync();
  ABI_CATCH("mkfk_trs_nsoc_", nan_fill(fk, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)))
}

void get_initial_delta_(double2* delta, const double* init_delta, const double2* uni, const int64_t* kmap,
                        const int64_t* invk, const int64_t* Nkall, const int64_t* Nk, const int64_t* Nw,
                        const int64_t* Norb, const int64_t* gap_sym) {
  ABI_TRY
  ensure_context();
  (void)kmap;
  const int64_t nk = *Nk, nw = *Nw, no = *Norb;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  const long long KE = nk * nw * no * no;
  std::vector<double> w(nk, 0.0);
  for (int64_t i = 0; i < *Nkall; ++i) {
    const int64_t k = invk[3 * i] - 1;
    PGB_CHECK(k >= 0 && k < nk, "invk(1,:) outside [1,Nk]");
    w[k] += 1.0;
  }
  DBuf<double> kw(nk), init(nk * no);
  DBuf<double2> u(no * no * nk), D(KE);
  kw.upload(w.data(), nk);
  init.upload(init_delta, nk * no);
  u.upload(uni, no * no * nk);
  initial_delta(D.p, init.p, u.p, (int)nk, (int)nw, (int)no, (int)*gap_sym);
  const double nrm = inner_w(D.p, D.p, kw.p, (int)nk, KE).x;
  PGB_CHECK(nrm > 0, "Error: get_initial_delta norm <= 0");
  scal(D.p, 1.0 / std::sqrt(2.0 * nrm), KE);
  D.download(delta, KE);
  sync();
  ABI_CATCH("get_initial_delta_", nan_fill(delta, (size_t)(*Nk) * (*Nw) * (*Norb) * (*Norb)))
}

void remap_delta_(double2* delta, const double2* delta0, const double* prt, const int64_t* invk, const int64_t* Nkall,
                  const int64_t* Nk, const int64_t* Nw, const int64_t* Norb, const int64_t* gap_sym) {
  ABI_TRY
  ensure_context();
  const int64_t nkall = *Nkall, nk = *Nk, nw = *Nw, no = *Norb;
  for (int64_t i = 0; i < nkall; ++i) PGB_CHECK(invk[3 * i] >= 1 && invk[3 * i] <= nk, "invk(1,:) outside [1,Nk]");
  DBuf<double2> d0(nk * nw * no * no), out(nkall * nw * no * no);
  DBuf<double> pr(no);
  DBuf<int64_t> iv(3 * nkall);
  d0.upload(delta0, nk * nw * no * no);
  pr.upload(prt, no);
  iv.upload(invk, 3 * nkall);
  k_remap_delta<<<g1(nkall * nw * no * no, 256), 256, 0, ctx().stream>>>(out.p, d0.p, pr.p, iv.p, nkall, nk, nw,
                                                                         (int)no, (*gap_sym < 0) ? -1.0 : 1.0);
  launch_check("remap_delta");
  out.download(delta, nkall * nw * no * no);
  sync();
  ABI_CATCH("remap_delta_", nan_fill(delta, (size_t)(*Nkall) * (*Nw) * (*Norb) * (*Norb)))
}

void conv_delta_orb_to_band(double2* deltab, const double2* delta, const double2* uni, const double* prt,
                            const int64_t* invk, const int64_t* Norb, const int64_t* Nkall, const int64_t* Nk,
                            const int64_t* Nw, const int64_t* gap_sym) {
  ABI_TRY
  ensure_context();
  const int64_t no = *Norb, nkall = *Nkall, nk = *Nk;
  PGB_CHECK(no <= kMaxOrb, "Norb above the engine limit of 8 orbitals");
  for (int64_t i = 0; i < nkall; ++i) PGB_CHECK(invk[3 * i] >= 1 && invk[3 * i] <= nk, "invk(1,:) outside [1,Nk]");
  // only the first Matsubara slice is used: copy delta(:,1,:,:) compactly
  std::vector<double2> d0((size_t)nk * no * no);
  for (int64_t e = 0; e < no * no; ++e)
    memcpy(&d0[(size_t)nk * e], delta + (size_t)nk * (*Nw) * e, sizeof(double2) * nk);
  DBuf<double2> d(nk * no * no), u(no * no * nk), out(nkall * no * no);
  DBuf<double> pr(no);
  DBuf<int64_t> iv(3 * nkall);
  d.upload(d0.data(), nk * no * no);
  u.upload(uni, no * no * nk);
  pr.upload(prt, no);
  iv.upload(invk, 3 * nkall);
  k_orb_to_band<<<g1(nkall, 64), 64, 0, ctx().stream>>>(out.p, d.p, u.p, pr.p, iv.p, nkall, nk, (int)no,
                                                        (*gap_sym < 0) ? -1.0 : 1.0);
  launch_check("orb_to_band");
  out.download(deltab, nkall * no * no);
  sync();
  ABI_CATCH("conv_delta_orb_to_band", nan_fill(deltab, (size_t)(*Nkall) * (*Norb) * (*Norb)))
}

// ============================================== outside the FLEX/RPA path ==
// Present so that `import libs.flibs` binds every symbol; each reports that
// it is not part of this engine.
#define PGB_STUB(name)                                                                                    \
  void name() {                                                                                            \
    report(#name, "not part of the GB300 FLEX/RPA/Eliashberg engine (outside the accelerated path)");      \
  }
PGB_STUB(calc_kn)
PGB_STUB(calc_lij)
PGB_STUB(calc_lij_wl)
PGB_STUB(calc_sigma_hall)
PGB_STUB(calc_tau_epa)
PGB_STUB(calc_tdf)
PGB_STUB(gen_dos)
PGB_STUB(gen_imp_ham)
PGB_STUB(gen_tr_greenw_0)
PGB_STUB(get_band_to_orb_delta)
PGB_STUB(get_chi_irr_sc)
PGB_STUB(get_dft_imp_ham)
PGB_STUB(get_imass0)
PGB_STUB(get_imassk)
PGB_STUB(get_spectrum_spaghetti)
PGB_STUB(get_tau)
PGB_STUB(get_veloc)
PGB_STUB(get_vlm0)
PGB_STUB(get_vnm)
PGB_STUB(matrix_riccati_batch)
PGB_STUB(matrix_riccati_chords)
PGB_STUB(mkbdghamk)
PGB_STUB(riccati_chords)
PGB_STUB(solve_cpa_array)

// ============================================== allocation-free variant ==
int pyrpa_gb_eig_or_tr_chi_noalloc(void* chiqout_v, const void* chi_v, const int64_t* invk, int64_t Nkall,
                                   int64_t Nk, int64_t Nchi, int32_t sw_eig, void* stream) {
  double2* chiqout = static_cast<double2*>(chiqout_v);
  const double2* chi = static_cast<const double2*>(chi_v);
  try {
    if (Nk < 1 || Nk > kNoAllocMaxNk)
      throw Error("Nk = " + std::to_string(Nk) + " is outside [1, 65536], the size of the fixed scratch");
    if (Nchi < 1 || Nchi > kMaxChi) throw Error("Nchi above the engine limit of 32 orbital pairs");
    if (Nkall < 1) throw Error("Nkall must be positive");
    if (!chiqout || !chi || !invk) throw Error("null device pointer");
    int dev = -1;
    PGB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) throw Error("device ordinal above 63");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // each launch is checked by its own return status, which leaves an error
    // that the caller's earlier work left pending where it is
    auto eig_launch = [&](double2* v, int64_t nk, int sw, unsigned grid) {
      int n = (int)Nchi;
      void* args[] = {(void*)&v, (void*)&chi, (void*)&nk, (void*)&n, (void*)&sw};
      PGB_CUDA(cudaLaunchKernel((const void*)k_eig_or_tr, dim3(grid), dim3(32), args, 0, st));
    };
    auto map_launch = [&](const double2* v, int64_t nkall, unsigned grid, unsigned block) {
      int64_t nk = Nk;
      void* args[] = {(void*)&chiqout, (void*)&v, (void*)&invk, (void*)&nkall, (void*)&nk};
      PGB_CUDA(cudaLaunchKernel((const void*)k_map_full_checked, dim3(grid), dim3(block), args, 0, st));
    };
    double2* vals = nullptr;
    {
      std::lock_guard<std::mutex> lk(g_noalloc_mu);
      if (!g_noalloc_ptr[dev]) {
        // set-up, once per device with that device current: the address of
        // the scratch, and one empty launch of each kernel, so that what the
        // module and its kernels need on this device is taken now
        void* p = nullptr;
        PGB_CUDA(cudaGetSymbolAddress(&p, g_noalloc_vals));
        eig_launch(static_cast<double2*>(p), 0, 1, 1);
        map_launch(static_cast<double2*>(p), 0, 1, 32);
        g_noalloc_ptr[dev] = static_cast<double2*>(p);
      }
      vals = g_noalloc_ptr[dev];
    }
    eig_launch(vals, Nk, sw_eig ? 1 : 0, (unsigned)g1(Nk, 32));
    map_launch(vals, Nkall, (unsigned)g1(Nkall, 256), 256);
    ctx().kernel_launches += 2;
    return 0;
  } catch (const std::exception& e) {
    report("pyrpa_gb_eig_or_tr_chi_noalloc", e.what());
    return 1;
  }
}

}  // extern "C"
