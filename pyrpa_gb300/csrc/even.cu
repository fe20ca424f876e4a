// Tables and checks of the even-model stages (see even.cuh).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <string>

#include "even.cuh"
#include "fft.cuh"
#include "flex_dev.cuh"

namespace pgb {

namespace {

// PYRPA_GB_EVEN=0 keeps every model on the general form
bool even_enabled() {
  const char* s = std::getenv("PYRPA_GB_EVEN");
  return !(s && std::string(s) == "0");
}

constexpr size_t kEvenSmem = 200 * 1024;  // two plane buffers of one CTA (space_launch)

// P of each pair, or false where the list is not closed under it
bool pair_perm(const Pairs& p, std::vector<int>& perm) {
  const int n = p.Nchi;
  perm.assign(n, -1);
  std::vector<int> at((size_t)p.Norb * p.Norb, -1);
  for (int l = 0; l < n; ++l) {
    int& s = at[p.o1[l] + (size_t)p.Norb * p.o2[l]];
    if (s >= 0) return false;  // a pair listed twice
    s = l;
  }
  for (int l = 0; l < n; ++l) {
    perm[l] = at[p.o2[l] + (size_t)p.Norb * p.o1[l]];
    if (perm[l] < 0) return false;
  }
  return true;
}

void build_classes(Even& ev, int n) {
  ev.cls_of.assign((size_t)n * n, -1);
  ev.cj_of.assign((size_t)n * n, 0);
  for (int l = 0; l < n; ++l)
    for (int m = 0; m < n; ++m) {
      if (ev.cls_of[m + n * l] >= 0) continue;
      EvenClass c{};
      c.l = l;
      c.m = m;
      c.el = m + n * l;
      const int pl = ev.perm[l], pm = ev.perm[m];
      const int el[4] = {m + n * l, l + n * m, pm + n * pl, pl + n * pm}, cj[4] = {0, 0, 1, 1};
      for (int i = 0; i < 4; ++i) {
        if (ev.cls_of[el[i]] >= 0) continue;
        ev.cls_of[el[i]] = (int)ev.cls.size();
        ev.cj_of[el[i]] = cj[i];
        c.mem[c.nmem] = el[i];
        c.cj[c.nmem++] = cj[i];
      }
      ev.cls.push_back(c);
    }
}

struct RealBasis {
  int kind, l;  // 0 same orbital, 1 sum, 2 i times the difference; the pair of smaller index
};

// index tables of the real basis: its matrix from the class representatives (vin) and back (vout)
void build_index(Even& ev, int n, const std::vector<RealBasis>& basis, const std::vector<int>* idx) {
  PGB_CHECK(2 * ev.cls.size() <= (size_t)kSrcMask + 1, "more pair classes than the real-basis tables can address");
  auto src = [&](int row, int col, int part, int* sign) {  // part of element (row, col) of the vertex matrix
    const int x = row + n * col;
    *sign = (part && ev.cj_of[x]) ? -1 : 1;
    return 2 * ev.cls_of[x] + part;
  };
  ev.vin.assign((size_t)n * n, 0);
  for (int p = 0; p < n; ++p)
    for (int q = 0; q < n; ++q) {
      const RealBasis r = basis[p], c = basis[q];
      const int l = r.l, m = c.l, pm = ev.perm[m];
      const bool im = (r.kind == 2) != (c.kind == 2);
      int ca = 1, cb = 0, s = 1;
      if (r.kind == 1 && c.kind == 0) ca = 2;
      else if (r.kind == 2 && c.kind == 0) ca = -2;
      else if (r.kind == 1 && c.kind == 1) cb = 1;
      else if (r.kind == 2 && c.kind == 2) cb = -1;
      else if (r.kind == 1 && c.kind == 2) cb = -1;
      else if (r.kind == 2 && c.kind == 1) ca = cb = -1;
      const int a = src(l, m, im, &s);
      ca *= s;
      int b = 0;
      if (cb) {
        b = src(l, pm, im, &s);
        cb *= s;
      }
      ev.vin[(size_t)q * n + p] = a | b << kSrcBits | (ca + 2) << 2 * kSrcBits | (cb + 2) << (2 * kSrcBits + 3);
    }
  ev.vout.clear();
  for (const EvenClass& c : ev.cls) {
    const int x = c.m, y = c.l;  // row and column of element el = m + n l
    const int sx = x <= ev.perm[x] ? 1 : -1, sy = y <= ev.perm[y] ? 1 : -1;
    const bool xs = ev.perm[x] == x, ys = ev.perm[y] == y;
    auto at = [&](int kx, int ky) { return idx[ky][y] * n + idx[kx][x]; };
    int a[2], b[2] = {0, 0}, sa[2], sb[2] = {0, 0}, half = 0;
    if (xs && ys) {
      a[0] = at(0, 0); sa[0] = 1;
      a[1] = 0; sa[1] = 0;
    } else if (xs) {
      a[0] = at(0, 1); sa[0] = 1;
      a[1] = at(0, 2); sa[1] = sy;
    } else if (ys) {
      half = 1;
      a[0] = at(1, 0); sa[0] = 1;
      a[1] = at(2, 0); sa[1] = -sx;
    } else {
      half = 1;
      a[0] = at(1, 1); sa[0] = 1;
      b[0] = at(2, 2); sb[0] = sx * sy;
      a[1] = at(1, 2); sa[1] = sy;
      b[1] = at(2, 1); sb[1] = -sx;
    }
    for (int h = 0; h < 2; ++h)
      ev.vout.push_back(a[h] | b[h] << 10 | (sa[h] + 1) << 20 | (sb[h] + 1) << 22 | half << 24);
  }
}

// The symmetric form of the real basis.  An element (l,m) and (m,l) are the same
// function, so with h = 1 (same orbital), 2 (sums), -2 (differences) the matrix
// M_pq = A_pq h_q is symmetric and A^-1 = diag(h) M^-1.  A symmetric matrix is kept
// as its cyclic diagonals: entry (p, (p + d) mod n), d <= n/2, at d n + p.
// sin: entry of M from the class representatives; sout: part of a class's result
// A = diag(h) W from W, every coefficient +-1.
int sym_at(int n, int p, int q) {
  const int d = (q - p + n) % n;
  return 2 * d < n || (2 * d == n && p < q) ? d * n + p : (n - d) * n + q;
}
void build_sym(Even& ev, int n, const std::vector<RealBasis>& basis) {
  ev.hsc.clear();
  for (const RealBasis& b : basis) ev.hsc.push_back(b.kind == 0 ? 1.0 : (b.kind == 1 ? 2.0 : -2.0));
  ev.sin.clear();
  for (int d = 0; d <= n / 2; ++d)
    for (int p = 0; p < n; ++p) {
      const int q = (p + d) % n, w = ev.vin[(size_t)q * n + p];
      const int ca = src_ca(w) * (int)ev.hsc[q], cb = src_cb(w) * (int)ev.hsc[q];
      ev.sin.push_back(src_a(w) | src_b(w) << kSrcBits |
                       ((ca < 0) | (cb < 0) << 1 | (cb != 0) << 2 | (std::abs(ca) == 2) << 3) << 2 * kSrcBits);
    }
  ev.sout.clear();
  for (int w : ev.vout) {
    const int at[2] = {w & 1023, (w >> 10) & 1023}, sg[2] = {((w >> 20) & 3) - 1, ((w >> 22) & 3) - 1};
    int word = 0;
    for (int x = 0; x < 2; ++x) {
      const int p = at[x] % n, q = at[x] / n, neg = sg[x] * (ev.hsc[p] < 0 ? -1 : 1);
      word |= sym_at(n, p, q) << (10 * x) | (neg + 1) << (20 + 2 * x);
    }
    ev.sout.push_back(word);
  }
}

// The real basis: same-orbital pairs, then the sums, then i times the
// differences, of the pairs (a,b), (b,a) with the smaller index first.  With
// rows e_l, e_l + e_Pl, i (e_l - e_Pl) and the inverse's columns e_l,
// (e_l + e_Pl)/2, -i (e_l - e_Pl)/2 all coefficients are 1, 2 or 1/2.
void build_vertex(Even& ev, int n, const double* S, const double* C) {
  std::vector<RealBasis> basis;
  std::vector<int> idx[3];
  for (int k = 0; k < 3; ++k) {
    idx[k].assign(n, -1);
    for (int l = 0; l < n; ++l) {
      const bool self = ev.perm[l] == l;
      if ((k == 0) != self || (k > 0 && l > ev.perm[l])) continue;
      idx[k][l] = (int)basis.size();
      if (k > 0) idx[k][ev.perm[l]] = (int)basis.size();
      basis.push_back({k, l});
    }
    if (k == 0) ev.nself = (int)basis.size();
    if (k == 1) ev.nplus = (int)basis.size();
  }
  // S and C
  auto to_basis = [&](const double* X, std::vector<double>& out) {
    out.assign((size_t)n * n, 0.0);
    auto x = [&](int a, int b) { return X[a + n * b]; };
    for (int p = 0; p < n; ++p)
      for (int q = 0; q < n; ++q) {
        const RealBasis r = basis[p], c = basis[q];
        const int l = r.l, pl = ev.perm[l], m = c.l, pm = ev.perm[m];
        double v = 0;
        if (r.kind == 0 && c.kind == 0) v = x(l, m);
        else if (r.kind == 0 && c.kind == 1) v = 0.5 * (x(l, m) + x(l, pm));
        else if (r.kind == 1 && c.kind == 0) v = x(l, m) + x(pl, m);
        else if (r.kind == 1 && c.kind == 1) v = 0.5 * (x(l, m) + x(l, pm) + x(pl, m) + x(pl, pm));
        else if (r.kind == 2 && c.kind == 2) v = 0.5 * (x(l, m) - x(l, pm) - x(pl, m) + x(pl, pm));
        out[(size_t)p * n + q] = v;
      }
  };
  to_basis(S, ev.Sb);
  to_basis(C, ev.Cb);
  build_index(ev, n, basis, idx);
  build_sym(ev, n, basis);
  // Cholesky factors (lower) of S's blocks in the orthonormal basis
  std::vector<double> R((size_t)n * n, 0.0);
  ev.stoner_ok = n <= 32;
  for (int blk = 0; blk < 2 && ev.stoner_ok; ++blk) {
    const int i0 = blk ? ev.nplus : 0, i1 = blk ? n : ev.nplus;
    for (int p = i0; p < i1 && ev.stoner_ok; ++p)
      for (int q = i0; q <= p; ++q) {
        // e_l against (e_l + e_Pl) / sqrt 2
        const double sc = (p < ev.nself) == (q < ev.nself) ? 1.0 : (p < ev.nself ? std::sqrt(2.0) : std::sqrt(0.5));
        double v = sc * ev.Sb[(size_t)p * n + q];
        for (int k = i0; k < q; ++k) v -= R[(size_t)p * n + k] * R[(size_t)q * n + k];
        if (p == q) {
          if (!(v > 1e-10 * std::fabs(ev.Sb[(size_t)p * n + p]))) {
            ev.stoner_ok = false;
            break;
          }
          R[(size_t)p * n + p] = std::sqrt(v);
        } else {
          R[(size_t)p * n + q] = v / R[(size_t)q * n + q];
        }
      }
  }
  if (ev.stoner_ok) {
    ev.d_schol.alloc(R.size());
    ev.d_schol.upload(R.data(), R.size());
    sync();
  }
  std::vector<double> si(ev.Sb), ci(ev.Cb);
  const bool size_ok = n == 1 || n == 4 || n == 9 || n == 16 || n == 25;
  bool sparse = ev.nself <= 8;
  for (int p = 0; p < n; ++p)
    for (int q = 0; q < n; ++q)
      if (p != q && (p >= ev.nself || q >= ev.nself) && ev.Sb[(size_t)p * n + q] + ev.Cb[(size_t)p * n + q] != 0.0)
        sparse = false;
  ev.vertex_ok = size_ok && sparse && host_inverse(si, n) && host_inverse(ci, n);
}

// out[0], out[1]: the largest d and m of the launch, one atomic per warp (one per
// thread took 0.35 ms on two orbitals 32x32x512); non-negative doubles order
// as their bits, and a NaN above them all
__device__ __forceinline__ void max_bits(unsigned long long* out, double d, double m) {
  unsigned long long a = (unsigned long long)__double_as_longlong(d), b = (unsigned long long)__double_as_longlong(m);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, a);
    atomicMax(out + 1, b);
  }
}
// out[0]: max |X_ab - X_ba| (|Re| + |Im|), out[1]: max |X|
__global__ void k_sym_check(unsigned long long* out, const double2* X, long long n, int No) {
  double d = 0, m = 0;
  bool bad = false;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    for (int b = 0; b < No; ++b)
      for (int a = 0; a <= b; ++a) {
        const double2 u = X[i + n * (a + No * b)], v = X[i + n * (b + No * a)];
        const double e = fabs(u.x - v.x) + fabs(u.y - v.y), s = fabs(u.x) + fabs(u.y);
        bad |= !(e <= 1e300) || !(s <= 1e300);
        d = fmax(d, e);
        m = fmax(m, s);
      }
  if (bad) d = __longlong_as_double(0x7ff8000000000000LL);
  max_bits(out, d, m);
}
__global__ void k_symmetrize(double2* X, long long n, int No) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    for (int b = 0; b < No; ++b)
      for (int a = 0; a < b; ++a) {
        const double2 u = X[i + n * (a + No * b)], v = X[i + n * (b + No * a)];
        const double2 s = 0.5 * (u + v);
        X[i + n * (a + No * b)] = s;
        X[i + n * (b + No * a)] = s;
      }
}
// the largest deviation of an element from its class representative, and at
// nu = 0 from a real value; block y = class member
__global__ void k_even_check(unsigned long long* out, const double2* chi, const int* el, const int* mem, const int* cj,
                             const int* nmem, long long K, long long Nk) {
  const int c = blockIdx.y >> 2, i = blockIdx.y & 3;
  if (i >= nmem[c]) return;
  const double2 *r = chi + el[c] * K, *x = chi + mem[4 * c + i] * K;
  const double s = cj[4 * c + i] ? -1.0 : 1.0;
  double d = 0, m = 0;
  bool bad = false;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K; k += (long long)gridDim.x * blockDim.x) {
    const double2 u = x[k], v = r[k];
    double e = fabs(u.x - v.x) + fabs(u.y - s * v.y);
    if (k < Nk) e = fmax(e, fabs(u.y));
    const double a = fabs(u.x) + fabs(u.y);
    bad |= !(e <= 1e300) || !(a <= 1e300);
    d = fmax(d, e);
    m = fmax(m, a);
  }
  if (bad) d = __longlong_as_double(0x7ff8000000000000LL);
  max_bits(out, d, m);
}

bool within(DBuf<unsigned long long>& out, double tol) {
  unsigned long long h[2];
  out.download(h, 2);
  sync();
  double v[2];
  static_assert(sizeof(v) == sizeof(h), "");
  memcpy(v, h, sizeof(h));
  return v[0] <= tol * v[1];
}

}  // namespace

std::shared_ptr<Even> make_even(const Geom& g, const Pairs& p, const double* S, const double* C, int elem_bytes) {
  if (!even_enabled() || g.spin.on || g.Ny < 2 || g.Nw < 2) return nullptr;
  const int n = p.Nchi;
  auto ev = std::make_shared<Even>();
  ev->nx = g.Nx;
  ev->ny = g.Ny;
  ev->nz = g.Nz;
  ev->Nw = g.Nw;
  ev->three_d = g.Nz > 1;
  // the planes have to fit in shared memory, and the lengths to factor
  const size_t row = (size_t)(g.Nx + 1) * (ev->three_d ? g.Ny : g.Ny / 2 + 1);
  const size_t buf = ev->three_d ? row : std::max(row, (size_t)g.Ny * (g.Nx / 2 + 1));
  int rad[kMaxStages], nst = 0;
  if (2 * buf * elem_bytes > kEvenSmem || g.Nz > 512) return nullptr;
  for (int len : {g.Nx, g.Ny, g.Nz, g.Nw})
    if (!fft_factor(len, rad, &nst) || nst > 8 + (len == g.Nw ? 8 : 0)) return nullptr;
  if (!pair_perm(p, ev->perm)) return nullptr;
  if (S && C) {
    double mx = 0;
    for (int i = 0; i < n * n; ++i) mx = std::max({mx, std::fabs(S[i]), std::fabs(C[i])});
    for (const double* X : {S, C})
      for (int a = 0; a < n; ++a)
        for (int b = 0; b < n; ++b) {
          const double v = X[a + n * b];
          if (!(std::fabs(v - X[b + n * a]) <= 1e-14 * mx) ||
              !(std::fabs(v - X[ev->perm[a] + n * ev->perm[b]]) <= 1e-14 * mx))
            return nullptr;
        }
  }
  // half grid; -k of a mesh cell has to be the same irreducible point.  By rows of x, with a
  // 32-bit division for some cells: several 64-bit ones a cell made these tables take
  // 0.035 us a mesh point, now 0.008
  const int hy = ev->three_d ? g.Ny : g.Ny / 2 + 1, hz = ev->three_d ? g.Nz / 2 + 1 : 1;
  const int nx = g.Nx, nrows = g.Ny * g.Nz;
  ev->H = nx * hy * hz;
  std::vector<int> mrow(nrows);  // row of -k
  for (int z = 0, r = 0; z < g.Nz; ++z)
    for (int y = 0; y < g.Ny; ++y, ++r) mrow[r] = (y ? g.Ny - y : 0) + g.Ny * (z ? g.Nz - z : 0);
  for (int r = 0; r < nrows; ++r) {
    const int *row = &g.h_grid_irr[(size_t)r * nx], *m = &g.h_grid_irr[(size_t)mrow[r] * nx];
    bool same = row[0] == m[0];
    for (int x = 1; x < nx; ++x) same = same && row[x] == m[nx - x];
    if (!same) return nullptr;
  }
  // the half grid is the leading part of the mesh in its own order
  std::vector<int> h_irr(g.h_grid_irr.begin(), g.h_grid_irr.begin() + ev->H), irr_h(g.Nk, -1);
  for (int k = 0; k < g.Nk; ++k) {
    int h = (int)g.h_irr_grid[k];
    if (h >= ev->H) {
      const int r = h / nx, x = h - r * nx;
      h = mrow[r] * nx + (x ? nx - x : 0);
    }
    if (h >= ev->H) return nullptr;
    irr_h[k] = h;
  }
  const int npl = ev->H / hz;
  std::vector<int> order(g.Nk), koff(hz + 1, 0);
  std::iota(order.begin(), order.end(), 0);
  if (hz == 1) {
    koff[1] = g.Nk;
  } else {
    std::vector<int> plane(g.Nk);
    for (int k = 0; k < g.Nk; ++k) ++koff[(plane[k] = irr_h[k] / npl) + 1];
    for (int z = 0; z < hz; ++z) koff[z + 1] += koff[z];
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return plane[a] < plane[b]; });
  }
  auto put = [](DBuf<int>& d, const std::vector<int>& h) {
    d.alloc(h.size());
    d.upload(h.data(), h.size());
  };
  put(ev->h_irr, h_irr);
  put(ev->irr_h, irr_h);
  put(ev->korder, order);
  put(ev->koff, koff);
  std::vector<int2> zp;
  if (ev->three_d) {
    for (int c = 0; c < npl; ++c) {
      const int x = c % g.Nx, y = c / g.Nx, m = (g.Nx - x) % g.Nx + g.Nx * ((g.Ny - y) % g.Ny);
      if (c <= m) zp.push_back(make_int2(c, m));
    }
    ev->nzp = (int)zp.size();
    ev->zpairs.alloc(zp.size());
    ev->zpairs.upload(zp.data(), zp.size());
  }
  const int No = p.Norb;
  ev->sym_of.assign((size_t)No * No, 0);
  for (int b = 0; b < No; ++b)
    for (int a = 0; a <= b; ++a) {
      ev->sym_of[a + No * b] = ev->sym_of[b + No * a] = (int)ev->sym_el.size();
      ev->sym_el.push_back(a + No * b);
    }
  ev->nsym = (int)ev->sym_el.size();
  build_classes(*ev, n);
  if (S && C) build_vertex(*ev, n, S, C);
  std::vector<int> el, mem, cj, nm;
  for (const EvenClass& c : ev->cls) {
    el.push_back(c.el);
    nm.push_back(c.nmem);
    mem.insert(mem.end(), c.mem, c.mem + 4);
    cj.insert(cj.end(), c.cj, c.cj + 4);
  }
  put(ev->cls_el, el);
  put(ev->mem, mem);
  put(ev->memcj, cj);
  put(ev->nmem, nm);
  std::vector<int> elt;
  for (int x : ev->sym_el) elt.push_back(x / No + No * (x % No));
  put(ev->d_sym_el, ev->sym_el);
  put(ev->d_sym_elt, elt);
  std::vector<EvenPair> hp;
  for (const EvenClass& c : ev->cls) {
    const int a13 = p.o1[c.l], b13 = p.o1[c.m], a42 = p.o2[c.m], b42 = p.o2[c.l];
    hp.push_back(EvenPair{ev->sym_of[a13 + No * b13], ev->sym_of[a42 + No * b42], a13, b13, a42, b42});
  }
  ev->pairs.alloc(hp.size());
  ev->pairs.upload(hp.data(), hp.size());
  std::vector<EvenTerm> terms;
  std::vector<int> tb(1, 0);
  if (p.sigma.size() == (size_t)No * No) {
    for (int e : ev->sym_el) {
      for (const Term& t : p.sigma[e]) {
        const int x = t.m + n * t.l;
        terms.push_back(EvenTerm{ev->cls_of[x], ev->sym_of[t.ef], ev->cj_of[x]});
      }
      tb.push_back((int)terms.size());
    }
    ev->sig_terms.alloc(std::max<size_t>(1, terms.size()));
    ev->sig_terms.upload(terms.data(), terms.size());
    put(ev->sig_tb, tb);
  }
  if (S && C) {
    put(ev->d_vin, ev->vin);
    put(ev->d_vout, ev->vout);
    put(ev->d_sin, ev->sin);
    put(ev->d_sout, ev->sout);
  }
  sync();
  return ev;
}

bool symmetric_sample(const double2* X, long long n, int No) {
  double d = 0, m = 0;
  const long long pts = std::min<long long>(n, 8);  // every element read is a cache miss
  for (long long s = 0; s < pts; ++s) {
    const double2* x = X + s * (n / pts);
    for (int b = 0; b < No; ++b)
      for (int a = 0; a <= b; ++a) {
        const double2 u = x[n * (a + No * b)], v = x[n * (b + No * a)];
        d = std::max(d, std::fabs(u.x - v.x) + std::fabs(u.y - v.y));
        m = std::max(m, std::fabs(u.x) + std::fabs(u.y));
      }
  }
  return !(d > 1e-9 * m);
}

bool symmetric_blocks(const double2* X, long long n, int No, double tol) {
  DBuf<unsigned long long> out(2);
  out.zero();
  k_sym_check<<<grid_1d(n, 256, 608), 256, 0, ctx().stream>>>(out.p, X, n, No);
  count_launch("sym_check");
  return within(out, tol);
}

bool symmetric_h(const double2* H, long long Nk, int No) {
  double d = 0, m = 0;
  for (long long k = 0; k < Nk; ++k)
    for (int b = 0; b < No; ++b)
      for (int a = 0; a <= b; ++a) {
        const double2 u = H[a + No * (b + No * k)], v = H[b + No * (a + No * k)];
        const double e = std::fabs(u.x - v.x) + std::fabs(u.y - v.y);
        if (!(e <= 1e300)) return false;
        d = std::max(d, e);
        m = std::max(m, std::fabs(u.x) + std::fabs(u.y));
      }
  return d <= 1e-13 * m || d == 0;
}

bool symmetric_bands(const double* eig, const double2* uni, long long Nk, int No) {
  double d = 0, m = 0;
  for (long long k = 0; k < Nk; ++k)
    for (int b = 0; b < No; ++b)
      for (int a = 0; a <= b; ++a) {
        double re = 0, im = 0, one = 0;
        for (int n = 0; n < No; ++n) {
          const double2 u = uni[a + No * (n + No * k)], v = uni[b + No * (n + No * k)];
          const double c = u.x * v.x + u.y * v.y, s = u.y * v.x - u.x * v.y, e = eig[n + No * k];
          re += e * c;
          im += e * s;
          one += s;
        }
        if (!(std::fabs(im) <= 1e300) || !(std::fabs(re) <= 1e300)) return false;
        // one: the completeness sum, whose imaginary part vanishes for any
        // unitary; a set of vectors that is not unitary stays general
        d = std::max({d, std::fabs(im), std::fabs(one)});
        m = std::max(m, std::fabs(re));
      }
  return d <= 1e-12 * std::max(m, 1e-300) || d == 0;
}

void symmetrize_blocks(double2* X, long long n, int No) {
  if (No < 2) return;
  k_symmetrize<<<grid_1d(n, 256, 65536), 256, 0, ctx().stream>>>(X, n, No);
  count_launch("symmetrize");
}

bool even_chi(const Geom& g, const Even& ev, const double2* chi, double tol) {
  DBuf<unsigned long long> out(2);
  out.zero();
  const unsigned nb = (unsigned)std::min<long long>((g.K + 255) / 256, 256);
  k_even_check<<<dim3(nb, 4 * (unsigned)ev.cls.size()), 256, 0, ctx().stream>>>(out.p, chi, ev.cls_el.p, ev.mem.p,
                                                                               ev.memcj.p, ev.nmem.p, g.K, g.Nk);
  count_launch("even_check");
  return within(out, tol);
}

}  // namespace pgb
