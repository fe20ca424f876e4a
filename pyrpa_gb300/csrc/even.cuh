// Convolutions and vertices of models whose H(k) is symmetric.
//
// If H(k) = H(k)^T on every k point (orbitals of one parity under inversion,
// real hoppings), time reversal makes H, G and Sigma even in k, and with the
// Hermiticity in frequency every function of (r, tau) is real (a fermionic
// one up to the phase e^{i pi s / M} of its half-integer frequencies) and even
// in r.  The three stages then need a quarter of the data of the general form:
//
//  * only the mesh points of one half of the Brillouin zone, in k and in r:
//    H = Nx (Ny/2 + 1) points (3-D: Nx Ny (Nz/2 + 1));
//  * an Nw-point complex transform instead of the M = 2 Nw point one: the real
//    values at slots 2s and 2s+1 are the two parts of one complex number c(s).
//    With w = e^{-2 pi i j / M} and F(j + Nw) the value at the padded slot
//    j + Nw, DFT_Nw of (F(j) + F(j+Nw)) + i w (F(j) - F(j+Nw)) is c; back,
//    F(j) = E + O / w with E, iO the halves of C(j) +- conj C(Nw - j).
//    A fermionic array has j + 1/2 in place of j and Nw - 1 - j for Nw - j;
//  * one transform per class of orbital-pair elements {(l,m), (m,l)} and their
//    conjugates {(Pl,Pm), (Pm,Pl)}, P(a,b) = (b,a): 175 of 625 at five orbitals;
//    the conjugate element is the same array at the reversed tau.
//
// A vertex matrix A = A(q, i nu) obeys P A P = conj A, so it is real in the basis
// of the sums and i times the differences of the pairs (a,b) and (b,a), and its
// two inverses are real ones.
//
// Measured on one FLEX iteration of five orbitals, general form -> this one:
// 32x32 points and 512 frequencies in FP64, where both are bound by the FP64
// pipe, chi0 44 -> 9.4 ms, Sigma 62 -> 10.1 ms, vertex 122 -> 22 ms; 64x64 and
// 1024 in FP32 chi0 40 -> 9.3 ms, Sigma 51 -> 10.2 ms, vertex 45 -> 19 ms.
// Without the symmetry (complex or s-p like hoppings), for planes that do not
// fit in shared memory and for spin-orbit models the general form remains.
//
// The space transform of a half plane transforms Ny/2 + 1 rows in x and the
// first Nx/2 + 1 columns in y, the missing rows and columns being mirror images.
#pragma once

#include <memory>

#include "flex.cuh"

namespace pgb {

struct EvenClass {
  int el;                 // stored element m + Nchi l of the representative
  int l, m;
  int nmem;               // members (the representative first) and their conjugation
  int mem[4], cj[4];
};

// A word of vin names its two sources 2 class + part in kSrcBits each, then their
// coefficients ca + 2 and cb + 2 in three bits each; a word of sin has four flags after
// the sources (k_vertex_sym).  Two four-orbital sites, the most pairs (32) of the
// engine, have 288 classes: sources up to 575.
constexpr int kSrcBits = 10, kSrcMask = (1 << kSrcBits) - 1;
__host__ __device__ constexpr int src_a(int w) { return w & kSrcMask; }
__host__ __device__ constexpr int src_b(int w) { return w >> kSrcBits & kSrcMask; }
__host__ __device__ constexpr int src_ca(int w) { return (w >> 2 * kSrcBits & 7) - 2; }
__host__ __device__ constexpr int src_cb(int w) { return (w >> (2 * kSrcBits + 3) & 7) - 2; }
__host__ __device__ constexpr bool src_flag(int w, int i) { return w >> (2 * kSrcBits + i) & 1; }

struct EvenPair {
  int f13, f42;  // a <= b copies of G13 and G42
  int a13, b13, a42, b42;  // their orbitals
};
struct EvenTerm {
  int c, f;  // class of the vertex element, fermionic copy
  int rev;   // bit 0: the vertex at the reversed tau, bit 1: the fermionic copy (antiperiodic)
};

struct Even {
  int nx = 1, ny = 1, nz = 1, Nw = 1, H = 1, nsym = 1;
  bool three_d = false;
  std::vector<EvenClass> cls;
  std::vector<int> cls_of, cj_of;   // per element m + Nchi l
  std::vector<int> sym_of;          // orbital element a + Norb b -> index of its a <= b copy
  std::vector<int> sym_el;          // and back
  std::vector<int> perm;            // P of each pair
  DBuf<int> h_irr, irr_h;           // irreducible k of a half-grid point, and back
  DBuf<int> korder, koff;           // irreducible k by plane of the half grid, first entry of each plane
  DBuf<int2> zpairs;                // 3-D: (p, -p) of the plane cells, p <= -p
  int nzp = 0;
  DBuf<int> cls_el;                 // device: el of each class
  DBuf<int> mem, memcj, nmem;       // device: members (4 per class)
  DBuf<int> d_sym_el, d_sym_elt;    // device: sym_el, and the transposed elements
  DBuf<EvenPair> pairs;             // device: per class
  DBuf<EvenTerm> sig_terms;         // device: the terms of Sigma, by a <= b output
  DBuf<int> sig_tb;                 // and the first of each output
  bool vertex_ok = false;           // the real-basis vertex applies (constants in vs/vc)
  std::vector<double> Sb, Cb;       // S and C in the real basis, row-major
  std::vector<int> vin, vout;       // index tables of the real basis (see even_impl.cuh)
  std::vector<int> sin, sout;       // the same for its symmetric form (k_vertex_sym)
  std::vector<double> hsc;          // and the scaling h of its rows (even.cu, build_sym)
  int nself = 0, nplus = 0;         // same-orbital pairs; pairs in the first (even) block at nu = 0
  bool stoner_ok = false;           // S positive definite: Cholesky factors of its two blocks in d_schol
  DBuf<double> d_schol;
  DBuf<int> d_vin, d_vout, d_sin, d_sout;
};

// The even-model tables of a mesh and pair list, or null where they do not
// apply (mesh too large for a plane in shared memory, pair list not closed
// under P, S or C not symmetric).  The caller vouches for G.  S, C: host
// (Nchi, Nchi), null for stages that do not use them.
std::shared_ptr<Even> make_even(const Geom& g, const Pairs& p, const double* S, const double* C, int elem_bytes);

// max |X_ab - X_ba| <= tol max |X| over n matrices of No x No elements at
// X[i + n (a + No b)]
bool symmetric_blocks(const double2* X, long long n, int No, double tol);
// the same of eight of the n matrices in host memory, to 1e-9: false where the whole
// cannot pass, without the wait for the device that symmetric_blocks ends with
bool symmetric_sample(const double2* X, long long n, int No);
// the same with H(k) in the (No, No, Nk) layout of the boundary, on the host
bool symmetric_h(const double2* H, long long Nk, int No);
// bands and eigenvectors of a symmetric H: U e U^+ symmetric on every k (host)
bool symmetric_bands(const double* eig, const double2* uni, long long Nk, int No);
// X_ab = X_ba = (X_ab + X_ba) / 2
void symmetrize_blocks(double2* X, long long n, int No);
// chi (K, Nchi, Nchi) has the relations of an even model: symmetric in its pair
// indices, P chi P = conj chi, real at nu = 0
bool even_chi(const Geom& g, const Even& ev, const double2* chi, double tol);

// chi0, Sigma, V and Delta of an even model.  full: every element is written;
// otherwise the class representatives, and every element at nu = 0.
template <typename R>
void chi0_even(const Geom& g, const double2* G, double temp, const TailRef* tail, cx<R>* chi, bool full);
template <typename R>
void sigma_even(const Geom& g, const double2* G, const cx<R>* V, const double* S, const double* C,
                double temp, double2* sig);
// Delta = scale sum_kq V_Delta F (singlet, orbitals of one parity) from F in
// FP64 or, when given, in the bulk type
template <typename R>
void mkdelta_even(const Geom& g, const Pairs& p, const double2* F64, const cx<R>* Fbulk, const cx<R>* Vd,
                  const double* S, const double* C, double scale, double2* out, DeltaKernelCache<R>& cache);
template <typename R>
bool vertex_even(const Even& ev, cx<R>* chi, long long nmat, long long estride, int mode, bool full);
// largest eigenvalue of chi0(q,0) S per irreducible q, into out (host, Nk)
template <typename R>
bool stoner_even(const Geom& g, const cx<R>* chi, std::vector<double>& out);
// out = in between bulk types on the class representatives
template <typename To, typename From>
void convert_even(const Even& ev, cx<To>* out, const cx<From>* in, long long K);

}  // namespace pgb
