// gh_kernels.cuh -- sm_100a kernels of the gauge + Higgs molecular-dynamics path.
//
// Device layout (component-major, so that a warp's load of one component for 32
// consecutive sites is one 512 B (FP64) or 256 B (FP32) coalesced transaction;
// complex = {re,im} vector load):
//   U   [lat][mu][site/32][i*N+j][site%32]  complex R  (reference: [site*D+mu] N x N, src/core/fields.hpp:12-20)
//        blocks of 32 sites, the N*N components of a block side by side: the
//        components of one link lie at a fixed stride of 32 elements, so one
//        address serves all N*N loads (immediate offsets); the volume is padded
//        to a multiple of 32 (LatDev::Vp)
//   P   [lat][mu][site/32][a][site%32]  real R     (reference: [site*D+mu][a], src/core/fields.hpp:46-57)
//   phi [lat][site/32][k][site%32]      complex R  (reference: [site*d+k], src/core/scalar_field.hpp:15)
// R = double (FP64 mode) or float (FP32-MD mode).  Several lattices of unequal
// extents live back to back; every kernel walks a table of Work items (lattice,
// direction, first site, count), one per block, so a single launch covers all
// lattices of a batch.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>
#include "gh_math.cuh"
#include "gh_rng.cuh"

namespace ghk {
using namespace ghm;

enum { REP_NONE = 0, REP_FUND = 1, REP_ADJ = 2, REP_GEN = 3 };
enum { F_GAUGE = 1, F_MATTER = 2 };
enum { M_UPDATE = 0, M_WRITE = 1 };
constexpr int KBLOCK = 128;    // threads per block of site/link kernels
#ifndef GH_KICK_LOG2
#define GH_KICK_LOG2 7
#endif
constexpr int KICK_LOG2 = GH_KICK_LOG2;      // sites per kick tile (= threads per kick block), log2
constexpr int KICK_BLOCK = 1 << KICK_LOG2;
constexpr int GEN_WARPS = 4;   // warps per block of the general-irrep kernel
constexpr int NRED = 6;        // per-site partial sums of the measure kernel
constexpr int ULANE = 32;      // sites per block of the link-field layout
enum { POT_QUARTIC = 0, POT_MULTI = 1 };
// Multi-invariant potential superoperator A[(r*d+q)][(i*d+j)], nonzeros only: CSR over
// the row pairs rq = r*d + q, column pair ij packed as i | j << 8, values in the
// precision of the arithmetic that reads them (double2 or float2).
struct PotA { const int* ptr; const unsigned short* ij; const void* v; };
constexpr int POT_DMAX = 32;   // largest representation the multi-invariant potential accepts

// Programmatic dependent launch: kernels of the MD path are launched so that the
// next one in the stream may be scheduled while this one finishes.  Each waits for
// its predecessor's results (griddepcontrol.wait: the predecessor grid has completed
// and its writes are visible) before reading anything, then lets its own successor
// launch.  Without the launch attribute both instructions are no-ops.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct LatDev {
  int L[4];
  int stride[4];
  int V;
  int Vp;                        // V rounded up to a multiple of ULANE (link-field plane size)
  int cidx;                      // coupling index (tempering bookkeeping)
  long long u_off, p_off, f_off, g_off;  // complex / real / complex / complex element offsets
  double beta, kappa, lambda;
  unsigned long long seed;
  unsigned long long traj, accepted, nonfinite;
  int last_acc;
  int lt[4];                     // kick tile shape: log2 of the tile extent per direction
  unsigned mag[4];               // floor(2^32 / L) (L = 1: 2^32 - 1): site_divmod's multiplier
  // Domain decomposition (src/mpi/gauge_mpi.hpp:26-80): a subdomain is stored with a
  // width-1 halo in every split direction.  Kernels act on the active box [lo, hi) only
  // (the whole lattice when not decomposed), and the counter RNG is keyed on the global
  // site index sum_mu (x_mu - lo_mu + goff_mu) * gstr_mu, so a decomposed lattice draws
  // the same numbers as the whole one.
  int lo[4], hi[4];
  int goff[4];
  long long gstr[4];
  int Vi;                        // active sites (normalises the lattice's sums)
  int dec;                       // 1: a subdomain with halo sites
};
// Site s inside the active box (always true for a lattice that is not decomposed).
__device__ __forceinline__ bool active_site(const LatDev& L, int s) {
  if (!L.dec) return true;
  int r = s;
#pragma unroll
  for (int mu = 0; mu < 4; ++mu) {
    const int x = r % L.L[mu];
    r /= L.L[mu];
    if (x < L.lo[mu] || x >= L.hi[mu]) return false;
  }
  return true;
}
// Below the active box's upper end in every direction: the interior and the lower halo
// layer, where the general-irrep link kernels also write psi_b = D(U)^dag phi, which the
// scalar force of the first interior layer reads at x - mu.
template <int D> __device__ __forceinline__ bool below_hi(const LatDev& L, const int* x) {
  bool in = true;
#pragma unroll
  for (int mu = 0; mu < D; ++mu) in = in && (x[mu] < L.hi[mu]);
  return in;
}
template <int D> __device__ __forceinline__ bool in_box(const LatDev& L, const int* x) {
  bool in = true;
#pragma unroll
  for (int mu = 0; mu < D; ++mu) in = in && (x[mu] >= L.lo[mu]) && (x[mu] < L.hi[mu]);
  return in;
}
// Global site index of local site s (the RNG key's site).
__device__ __forceinline__ long long global_site(const LatDev& L, int s) {
  if (!L.dec) return s;
  long long g = 0;
  int r = s;
#pragma unroll
  for (int mu = 0; mu < 4; ++mu) {
    const int x = r % L.L[mu];
    r /= L.L[mu];
    g += (long long)(x - L.lo[mu] + L.goff[mu]) * L.gstr[mu];
  }
  return g;
}
// Block work item.  Linear items: sites s0 .. s0+n-1.  Kick items (tiles): s0 is
// the tile's origin site and n packs the origin coordinates, 8 bits each.
// mu = -1 marks a site item, mu >= 0 a link item of direction mu.  Linear kick items
// carry mu + KICK_LINEAR, except kick_site_gen's (mu = -1), which hold up to 32 sites.
struct Work { int lat, mu, s0, n; };
constexpr int KICK_SITE_SPLIT_D = 9;   // components from which on kick_site_gen is used
constexpr int KICK_LINEAR = 16;

struct GenTables {                 // general irrep (src/rep/rep_general.hpp), sparse
  int d, n, dimT, ng;
  int powN[18];
  // division by powN[k] as a multiply-high: q = umulhi(f, pmag[k]) for k >= 1 (exact for
  // f * powN[k] < 2^32, which N^n <= 200000 guarantees); powN[0] = 1 needs none
  unsigned pmag[18];
  const int* wt_ptr; const int* wt_l; const double2* wt_v;   // lift: CSR over tensor index
  const int* w_ptr;  const int* w_i;  const double2* w_v;    // project: CSR over basis vector
  const int* t_ptr;  const int* t_j;  const double2* t_v;    // T^a_R: CSR over (a, row)
  // single-row irreps: D(U) in closed form (host term lists, gh_sympow.h); null: tensor path
  const int* sp_ptr; const double2* sp_c; const unsigned char* sp_e;
  // SU(2): the same D(U) as real sums over |a|^2, |b|^2 (k_gen_spin); null: not used
  const int4* spin_ent; const double* spin_c;
  int warp_bytes;                                            // shared memory of one warp
  int px_off;                                                // byte offset of px in a warp's region
  // irreps inside the K-fold adjoint product (host: gh_adjprod.h): the isometric
  // intertwiner Q [A][d] in both precisions; null: not available
  // rows of Q the kernel lifts into (all A, or for a symmetric / antisymmetric coefficient
  // matrix the pairs a <= b / a < b): prow[r] = a ng + b, the first pndiag diagonal
  const double2* pq64; const float2* pq32;
  const int* prow;
  int pnrows, pndiag, psym;
  int s2;                          // 1: the two-fold product as symmetric tensors (k_gen_sym2; Bufs::s2tab)
  // irreps that are N x N matrices (two slots, or the one-fold adjoint product): the map
  // W [d][N*N] dense in both precisions, and whether it is real; null: not used
  const double2* w2_64; const float2* w2_32;
  int w2_real;
};

template <typename R> struct V2;
template <> struct V2<double> { typedef double2 t; };
template <> struct V2<float> { typedef float2 t; };
template <typename R> struct Cmp { typedef R t; };

template <typename C, typename R> __device__ __forceinline__ cx<C> ldc(const R* __restrict__ p, long long i) {
  const typename V2<R>::t v = __ldg(reinterpret_cast<const typename V2<R>::t*>(p) + i);
  return mk<C>((C)v.x, (C)v.y);
}
template <typename C, typename R> __device__ __forceinline__ cx<C> ldc_rw(const R* p, long long i) {
  const typename V2<R>::t v = reinterpret_cast<const typename V2<R>::t*>(p)[i];
  return mk<C>((C)v.x, (C)v.y);
}
template <typename C, typename R> __device__ __forceinline__ void stc(R* p, long long i, cx<C> z) {
  typename V2<R>::t v;
  v.x = (R)z.re;
  v.y = (R)z.im;
  reinterpret_cast<typename V2<R>::t*>(p)[i] = v;
}
// Sites are never negative: the 32-site block and lane come from a shift and a mask
// (a signed division by 32 costs the rounding fix-up on every address).
__device__ __forceinline__ long long site_blk(int s) { return (long long)((unsigned)s >> 5); }
__device__ __forceinline__ int site_lane(int s) { return (int)((unsigned)s & (ULANE - 1)); }
// Element index of component c of link (mu, s); component c + k sits k * ULANE further on.
__device__ __forceinline__ long long u_index(const LatDev& L, int nn, int mu, int c, int s) {
  return L.u_off + (long long)mu * nn * L.Vp + (site_blk(s) * nn + c) * ULANE + site_lane(s);
}
// Momenta P: [mu][site/32][a][site%32] (ng components, direction planes of ng * Vp)
__device__ __forceinline__ long long p_index(const LatDev& L, int ng, int mu, int g, int s) {
  return L.p_off + (long long)mu * ng * L.Vp + (site_blk(s) * ng + g) * ULANE + site_lane(s);
}
// Scalar fields phi, pi: [site/32][k][site%32] (d components)
__device__ __forceinline__ long long f_index(const LatDev& L, int d, int k, int s) {
  return L.f_off + (site_blk(s) * d + k) * ULANE + site_lane(s);
}
// General-irrep scratch psi_f, psi_b: [mu][site/32][k][site%32]
__device__ __forceinline__ long long g_index(const LatDev& L, int d, int mu, int k, int s) {
  return L.g_off + (long long)mu * d * L.Vp + (site_blk(s) * d + k) * ULANE + site_lane(s);
}
template <int N, typename C, typename R>
__device__ __forceinline__ Mat<N, C> ld_link(const R* __restrict__ U, const LatDev& L, int mu, int s) {
  Mat<N, C> M;
  const long long base = u_index(L, N * N, mu, 0, s);
#pragma unroll
  for (int c = 0; c < N * N; ++c) M.e[c] = ldc<C>(U, base + c * ULANE);
  return M;
}
// An SU(N) link for the force: SU(2) from its first row (a, b), the second is (-conj b,
// conj a) -- half the loads, and the products below use one row (kick of a ladder of 16
// SU(2) lattices of 6, 8, 10, 12: FP32 34.3 -> 18.8 us, FP64 60.3 -> 28.6 us).  Other
// N: every entry.
template <int N, typename C, typename R>
__device__ __forceinline__ Mat<N, C> ld_su(const R* __restrict__ U, const LatDev& L, int mu, int s) {
  if constexpr (N == 2) {
    Mat<N, C> M;
    const long long base = u_index(L, N * N, mu, 0, s);
    M.e[0] = ldc<C>(U, base);
    M.e[1] = ldc<C>(U, base + ULANE);
    su2_second_row(M);
    return M;
  } else {
    return ld_link<N, C>(U, L, mu, s);
  }
}
template <int N, typename C, typename R>
__device__ __forceinline__ Mat<N, C> ld_link_rw(const R* U, const LatDev& L, int mu, int s) {
  Mat<N, C> M;
  const long long base = u_index(L, N * N, mu, 0, s);
#pragma unroll
  for (int c = 0; c < N * N; ++c) M.e[c] = ldc_rw<C>(U, base + c * ULANE);
  return M;
}
template <int N, typename C, typename R>
__device__ __forceinline__ void st_link(R* U, const LatDev& L, int mu, int s, const Mat<N, C>& M) {
  const long long base = u_index(L, N * N, mu, 0, s);
#pragma unroll
  for (int c = 0; c < N * N; ++c) stc<C>(U, base + c * ULANE, M.e[c]);
}

// (q, r) = (s / L, s % L) as a multiply-high and one correction: with mag = floor(2^32 / L)
// the estimate s mag / 2^32 lies below s / L by s (2^32 / L - mag) / 2^32 < 1 for every
// 32-bit s (L = 1: mag = 2^32 - 1, below by s / 2^32), so it is q or q - 1.
__host__ __device__ __forceinline__ void site_divmod(unsigned s, unsigned L, unsigned mag, unsigned& q, unsigned& r) {
#if defined(__CUDA_ARCH__)
  q = __umulhi(s, mag);
#else
  q = (unsigned)(((unsigned long long)s * mag) >> 32);
#endif
  r = s - q * L;
  if (r >= L) { r -= L; ++q; }
}
__host__ inline unsigned site_mag(int L) { return L == 1 ? 0xFFFFFFFFu : (unsigned)((1ULL << 32) / (unsigned)L); }
template <int D> __device__ __forceinline__ void coords(const LatDev& L, int s, int* x) {
  unsigned rest = (unsigned)s;
#pragma unroll
  for (int mu = 0; mu < D; ++mu) {
    if (mu == D - 1) { x[mu] = (int)rest; break; }
    unsigned q, r;
    site_divmod(rest, (unsigned)L.L[mu], L.mag[mu], q, r);
    x[mu] = (int)r;
    rest = q;
  }
}
// neighbour of site s (whose coordinate in direction mu is xm) in +mu / -mu
__device__ __forceinline__ int nfwd(const LatDev& L, int s, int xm, int mu) {
  return (xm + 1 < L.L[mu]) ? s + L.stride[mu] : s - xm * L.stride[mu];
}
__device__ __forceinline__ int nbwd(const LatDev& L, int s, int xm, int mu) {
  return (xm > 0) ? s - L.stride[mu] : s + (L.L[mu] - 1) * L.stride[mu];
}
// Site of thread `tid` inside a kick tile: the tile's origin comes from the work
// item, the offset from tid split by the power-of-two tile extents.  Threads that
// fall outside the lattice's active box (partial tiles, halo sites) return false.
template <int D>
__device__ __forceinline__ bool tile_site(const LatDev& L, const Work& w, int tid, int& s, int* x) {
  s = w.s0;
  bool in = true;
  int r = tid;
#pragma unroll
  for (int mu = 0; mu < D; ++mu) {
    const int l = r & ((1 << L.lt[mu]) - 1);
    r >>= L.lt[mu];
    x[mu] = ((w.n >> (8 * mu)) & 0xFF) + l;
    in = in && (x[mu] >= L.lo[mu]) && (x[mu] < L.hi[mu]);
    s += l * L.stride[mu];
  }
  return in && (r == 0);
}

// ---------------------------------------------------------------------------
// Representation apply for the register-resident reps.
// Fundamental: D(U) = U (src/rep/rep_fundamental.hpp:15-25).
// Adjoint: D_ab = 2 Re Tr(T^a U T^b U^dag) (src/rep/rep_adjoint.hpp:27-40) applied
// without forming D: (D phi)_a = 2 Tr(T^a U Phi U^dag), Phi = sum_b phi_b T^b.
// ---------------------------------------------------------------------------
template <int N, typename C>
__device__ __forceinline__ void fund_apply(const Mat<N, C>& U, const cx<C>* v, cx<C>* o, bool dag) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    cx<C> s = zero<C>();
#pragma unroll
    for (int j = 0; j < N; ++j) s = dag ? cfma_cj(s, U.e[j * N + i], v[j]) : cfma(s, U.e[i * N + j], v[j]);
    o[i] = s;
  }
}
template <int N, typename C>
__device__ __forceinline__ void adj_apply(const Mat<N, C>& U, const cx<C>* v, cx<C>* o, bool dag) {
  const Mat<N, C> Phi = alg_to_mat_c<N, C>(v);
  Mat<N, C> Psi = dag ? mm(mm_dn(U, Phi), U) : mm_nd(mm(U, Phi), U);
  tr2_proj<N, C>(Psi, o);
}

template <int N, int REP> struct RepDim { static constexpr int d = (REP == REP_FUND) ? N : (REP == REP_ADJ) ? N * N - 1 : 1; };

// ---------------------------------------------------------------------------
// Kick: link items (gauge force + matter back-reaction, P -= eps F) and site
// items (scalar force, pi += eps F_phi) of one launch.
//   gauge force  F^a = (beta/N) Im Tr(T^a U Sigma)      src/action/gauge_wilson.hpp:11-27,70-83
//   matter force F^a = -kappa g^a                        src/action/scalar_higgs.hpp:113-128
//   scalar force F_phi = -2 dV/dphi* + 2 kappa sum_mu [D phi_{x+mu} + D^dag phi_{x-mu}]
//                                                        src/action/scalar_higgs.hpp:71-108
// Fundamental rep: -kappa g^a = 2 kappa Im Tr(T^a psi phi_x^dag), psi = U phi_{x+mu},
// so one projection of (beta/N) U Sigma + 2 kappa psi phi_x^dag gives the total link force.
// Adjoint rep: -kappa g^a = -4 kappa Im Tr(T^a [conj(Phi_x), U Phi_y U^dag]).
// ---------------------------------------------------------------------------
struct KickArgs {
  const Work* work;
  const LatDev* lats;
  const void* U;
  void* P;
  const void* phi;
  void* pi;
  const void* psif;   // general irrep scratch: D(U_mu(x)) phi_{x+mu}
  const void* psib;   // general irrep scratch: D(U_mu(x))^dag phi_x
  double eps;
  int mode;           // M_UPDATE or M_WRITE
  int flags;          // F_GAUGE | F_MATTER
  int d;              // rep dimension (general irreps)
  double* out;        // M_WRITE destination (SoA like P / like phi, FP64)
  int pot;            // POT_QUARTIC or POT_MULTI
  double mu2;         // multi-invariant potential: -mu2 phi^dag phi
  PotA sa;            // multi-invariant potential: A = sum_c 2 f_c P_c, values in the field precision
  const double2* wpot;  // general irreps: w = A(M) phi per site, written by k_gen_links
};

// The direction is a template parameter so that every index into the lattice
// descriptor is static (no local-memory copy of the descriptor).
template <int D, int N, typename R, int REP, int MU>
__device__ __forceinline__ void kick_link(const KickArgs& a, const LatDev& L, int s, const int* x) {
  typedef typename Cmp<R>::t C;
  constexpr int mu = MU;
  const R* U = (const R*)a.U;
  const int spm = nfwd(L, s, x[mu], mu);
  // U_mu(x) is loaded after the staple loop: its 2 N^2 registers stay free while the
  // neighbour links are in flight (measured: FP64 kick -7%, FP32 -1%)
  Mat<N, C> Om;
  set_zero(Om);
  Mat<N, C> Umu;
  // rows of the staple sum: a real combination of SU(2) matrices has the form of one, so its
  // first row is all of it
  constexpr int ROWS = N == 2 ? 1 : N;
  if (!(a.flags & F_GAUGE)) Umu = ld_su<N, C>(U, L, mu, s);
  if (a.flags & F_GAUGE) {
    Mat<N, C> sig;
    set_zero(sig);
#pragma unroll
    for (int nu = 0; nu < D; ++nu) {
      if (nu == mu) continue;
      const int spn = nfwd(L, s, x[nu], nu);
      const int smn = nbwd(L, s, x[nu], nu);
      const int spm_mn = nbwd(L, spm, x[nu], nu);
      // upper staple U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag, lower U_nu(x+mu-nu)^dag U_mu(x-nu)^dag U_nu(x-nu)
      // (the inner products of two links through mm_su: their last row from unitarity)
      mm_core<N, C, false, true, true, ROWS>(mm_su<N, C, false, true>(ld_su<N, C>(U, L, nu, spm), ld_su<N, C>(U, L, mu, spn)),
                                             ld_su<N, C>(U, L, nu, s), sig);
      mm_core<N, C, false, false, true, ROWS>(mm_su<N, C, true, true>(ld_su<N, C>(U, L, nu, spm_mn), ld_su<N, C>(U, L, mu, smn)),
                                              ld_su<N, C>(U, L, nu, smn), sig);
    }
    if constexpr (N == 2) su2_second_row(sig);
    Umu = ld_su<N, C>(U, L, mu, s);
    mm_core<N, C, false, false, false, ROWS>(Umu, sig, Om);
    const C c = (C)(L.beta / N);
#pragma unroll
    for (int i = 0; i < ROWS * N; ++i) Om.e[i] = scale(Om.e[i], c);
    if constexpr (N == 2) su2_second_row(Om);
  }
  if ((a.flags & F_MATTER) && (REP == REP_FUND || REP == REP_ADJ)) {
    constexpr int d = RepDim<N, REP>::d;
    const R* phi = (const R*)a.phi;
    cx<C> px[d], py[d];
#pragma unroll
    for (int k = 0; k < d; ++k) {
      px[k] = ldc<C>(phi, f_index(L, d, k, s));
      py[k] = ldc<C>(phi, f_index(L, d, k, spm));
    }
    const C kap = (C)L.kappa;
    if (REP == REP_FUND) {
      cx<C> psi[N];
      fund_apply<N, C>(Umu, py, psi, false);
      const C k2 = C(2) * kap;
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) Om.e[i * N + j] = add(Om.e[i * N + j], scale(mulc(psi[i], px[j]), k2));
    } else {
      cx<C> pxc[d];
#pragma unroll
      for (int k = 0; k < d; ++k) pxc[k] = conj(px[k]);
      const Mat<N, C> Phx = alg_to_mat_c<N, C>(pxc);
      const Mat<N, C> Psi = mm_nd(mm(Umu, alg_to_mat_c<N, C>(py)), Umu);
      const Mat<N, C> c1 = mm(Phx, Psi), c2 = mm(Psi, Phx);
      const C k4 = C(-4) * kap;
#pragma unroll
      for (int i = 0; i < N * N; ++i) Om.e[i] = add(Om.e[i], scale(sub(c1.e[i], c2.e[i]), k4));
    }
  }
  C F[N * N - 1];
  im_tr_proj<N, C>(Om, F);
  constexpr int ng = N * N - 1;
  const long long pb = p_index(L, ng, mu, 0, s);
  if (a.mode == M_UPDATE) {
    R* P = (R*)a.P;
    const C eps = (C)a.eps;
#pragma unroll
    for (int g = 0; g < ng; ++g) P[pb + g * ULANE] = (R)((C)P[pb + g * ULANE] - eps * F[g]);
  } else {
#pragma unroll
    for (int g = 0; g < ng; ++g) a.out[pb + g * ULANE] = (double)F[g];
  }
}

// ---------------------------------------------------------------------------
// Multi-invariant onsite potential at site s (src/action/scalar_invariants.hpp):
// with M = phi phi^dag and A = sum_c 2 f_c P_c the combined channel superoperator
// ((d^2) x (d^2), vec index i*d + j),
//   w = A(M) phi,  dV/dphi^* = -mu2 phi + w,  V = -mu2 phi^dag phi + Re(phi^dag w) / 2.
// Writes w (when given) and returns V.  One thread per site; A is held sparse (the
// weight of the Cartan generators is conserved, so 75-95% of its d^4 entries
// vanish: 1469 of 28561 for SU(2){12}), read through L1 (every thread of a warp
// reads the same entry).
// ---------------------------------------------------------------------------
template <typename C, typename R>
__device__ __noinline__ C pot_multi(const R* phi, const LatDev& L, int d, int s, const PotA A, C mu2, cx<C>* w) {
  typedef typename V2<C>::t VT;
  const VT* __restrict__ av = reinterpret_cast<const VT*>(A.v);
  cx<C> p[POT_DMAX];
  C n2 = C(0);
  for (int k = 0; k < d; ++k) {
    p[k] = ldc<C>(phi, f_index(L, d, k, s));
    n2 += norm2(p[k]);
  }
  C re = C(0);
  for (int r = 0; r < d; ++r) {
    cx<C> acc = zero<C>();
    for (int q = 0; q < d; ++q) {
      const int b = __ldg(A.ptr + r * d + q), e = __ldg(A.ptr + r * d + q + 1);
      if (b == e) continue;
      cx<C> y = zero<C>();                 // A(M)_rq = sum_ij A_{rq,ij} phi_i conj(phi_j)
      for (int z = b; z < e; ++z) {
        const int ij = __ldg(A.ij + z);
        const VT a = __ldg(av + z);
        y = cfma(y, mk<C>(a.x, a.y), mulc(p[ij & 0xFF], p[ij >> 8]));
      }
      acc = cfma(acc, y, p[q]);
    }
    if (w) w[r] = acc;
    re = fmad(p[r].re, acc.re, fmad(p[r].im, acc.im, re));
  }
  return -mu2 * n2 + C(0.5) * re;
}

template <int D, int N, typename R, int REP>
__device__ __forceinline__ void kick_site(const KickArgs& a, const LatDev& L, int s, const int* x) {
  typedef typename Cmp<R>::t C;
  const R* U = (const R*)a.U;
  const R* phi = (const R*)a.phi;
  const C kap2 = C(2) * (C)L.kappa;
  if (REP == REP_FUND || REP == REP_ADJ) {
    constexpr int d = RepDim<N, REP>::d;
    cx<C> F[d], v[d], o[d];
    C n2 = C(0);
#pragma unroll
    for (int k = 0; k < d; ++k) { v[k] = ldc<C>(phi, f_index(L, d, k, s)); n2 += norm2(v[k]); }
    if (a.pot == POT_MULTI) {          // -2 dV/dphi^* = 2 mu2 phi - 2 A(M) phi
      cx<C> w[d];
      pot_multi<C, R>(phi, L, d, s, a.sa, (C)a.mu2, w);
#pragma unroll
      for (int k = 0; k < d; ++k) F[k] = sub(scale(v[k], C(2) * (C)a.mu2), scale(w[k], C(2)));
    } else {                           // -2 dV/dphi^* = -2 [1 + 2 lambda (n2 - 1)] phi
      const C cc = C(1) + C(2) * (C)L.lambda * (n2 - C(1));
#pragma unroll
      for (int k = 0; k < d; ++k) F[k] = scale(v[k], C(-2) * cc);
    }
#pragma unroll
    for (int mu = 0; mu < D; ++mu) {
      const int yf = nfwd(L, s, x[mu], mu), yb = nbwd(L, s, x[mu], mu);
      cx<C> o2[d];
#pragma unroll
      for (int k = 0; k < d; ++k) v[k] = ldc<C>(phi, f_index(L, d, k, yf));
      {
        const Mat<N, C> Uf = ld_su<N, C>(U, L, mu, s);
        if (REP == REP_FUND) fund_apply<N, C>(Uf, v, o, false); else adj_apply<N, C>(Uf, v, o, false);
      }
#pragma unroll
      for (int k = 0; k < d; ++k) v[k] = ldc<C>(phi, f_index(L, d, k, yb));
      {
        const Mat<N, C> Ub = ld_su<N, C>(U, L, mu, yb);
        if (REP == REP_FUND) fund_apply<N, C>(Ub, v, o2, true); else adj_apply<N, C>(Ub, v, o2, true);
      }
#pragma unroll
      for (int k = 0; k < d; ++k) F[k] = add(F[k], scale(add(o[k], o2[k]), kap2));
    }
    const long long fb = f_index(L, d, 0, s);
    if (a.mode == M_UPDATE) {
      R* pi = (R*)a.pi;
      const C eps = (C)a.eps;
#pragma unroll
      for (int k = 0; k < d; ++k) stc<C>(pi, fb + k * ULANE, add(ldc_rw<C>(pi, fb + k * ULANE), scale(F[k], eps)));
    } else {
      double2* out = reinterpret_cast<double2*>(a.out);
#pragma unroll
      for (int k = 0; k < d; ++k) out[fb + k * ULANE] = make_double2((double)F[k].re, (double)F[k].im);
    }
  } else if (REP == REP_GEN) {
    const int d = a.d;
    const R* psif = (const R*)a.psif;
    const R* psib = (const R*)a.psib;
    C n2 = C(0);
    for (int k = 0; k < d; ++k) n2 += norm2(ldc<C>(phi, f_index(L, d, k, s)));
    const C cc = C(1) + C(2) * (C)L.lambda * (n2 - C(1));
    int yb[D];
#pragma unroll
    for (int mu = 0; mu < D; ++mu) yb[mu] = nbwd(L, s, x[mu], mu);
    for (int k = 0; k < d; ++k) {
      const cx<C> pk = ldc<C>(phi, f_index(L, d, k, s));
      cx<C> F;
      if (a.pot == POT_MULTI) {
        const double2 wk = a.wpot[f_index(L, d, k, s)];
        F = sub(scale(pk, C(2) * (C)a.mu2), scale(mk<C>((C)wk.x, (C)wk.y), C(2)));
      } else {
        F = scale(pk, C(-2) * cc);
      }
#pragma unroll
      for (int mu = 0; mu < D; ++mu) {
        F = add(F, scale(add(ldc<C>(psif, g_index(L, d, mu, k, s)), ldc<C>(psib, g_index(L, d, mu, k, yb[mu]))), kap2));
      }
      const long long fi = f_index(L, d, k, s);
      if (a.mode == M_UPDATE) {
        R* pi = (R*)a.pi;
        stc<C>(pi, fi, add(ldc_rw<C>(pi, fi), scale(F, (C)a.eps)));
      } else {
        reinterpret_cast<double2*>(a.out)[fi] = make_double2((double)F.re, (double)F.im);
      }
    }
  }
}

// Scalar force of a general irrep of many components (KICK_SITE_SPLIT_D): a block takes
// one 32-site block, a lane per site, and its warps split the d components (psi_f, psi_b
// and w come from memory, so a thread that walks all d alone waits for 9 d loads in turn
// with few threads beside it).  Measured, whole kicks at SU(3) 12^4, one thread per site
// and split: 27-plet FP64 154.8 and 148.1 us, FP32 89.3 and 80.0; octet (d = 8) FP64 35.8
// and 36.5, sextet (d = 6) 31.8 and 32.8: the sum of |phi|^2 over the warps costs more than
// two components per thread give back, so d <= 8 keeps one thread per site.
template <int D, typename R>
__device__ __forceinline__ void kick_site_gen(const KickArgs& a, const LatDev& L, const Work& w) {
  typedef typename Cmp<R>::t C;
  constexpr int NW = KICK_BLOCK / 32;
  __shared__ C part[NW][32];
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5, d = a.d;
  const int s = w.s0 + (lane < w.n ? lane : 0);
  int x[D], yb[D];
  coords<D>(L, s, x);
  const bool live = lane < w.n && in_box<D>(L, x);
  const R* phi = (const R*)a.phi;
  const R* psif = (const R*)a.psif;
  const R* psib = (const R*)a.psib;
  C n2 = C(0);
  for (int k = q; k < d; k += NW) n2 += norm2(ldc<C>(phi, f_index(L, d, k, s)));
  part[q][lane] = n2;
  __syncthreads();
  if (!live) return;
  n2 = C(0);
#pragma unroll
  for (int i = 0; i < NW; ++i) n2 += part[i][lane];
  const C kap2 = C(2) * (C)L.kappa;
  const C cc = C(1) + C(2) * (C)L.lambda * (n2 - C(1));
#pragma unroll
  for (int mu = 0; mu < D; ++mu) yb[mu] = nbwd(L, s, x[mu], mu);
  for (int k = q; k < d; k += NW) {
    const long long fi = f_index(L, d, k, s);
    const cx<C> pk = ldc<C>(phi, fi);
    cx<C> F;
    if (a.pot == POT_MULTI) {
      const double2 wk = a.wpot[fi];
      F = sub(scale(pk, C(2) * (C)a.mu2), scale(mk<C>((C)wk.x, (C)wk.y), C(2)));
    } else {
      F = scale(pk, C(-2) * cc);
    }
#pragma unroll
    for (int mu = 0; mu < D; ++mu)
      F = add(F, scale(add(ldc<C>(psif, g_index(L, d, mu, k, s)), ldc<C>(psib, g_index(L, d, mu, k, yb[mu]))), kap2));
    if (a.mode == M_UPDATE) {
      R* pi = (R*)a.pi;
      stc<C>(pi, fi, add(ldc_rw<C>(pi, fi), scale(F, (C)a.eps)));
    } else {
      reinterpret_cast<double2*>(a.out)[fi] = make_double2((double)F.re, (double)F.im);
    }
  }
}

template <int D, int N, typename R, int REP>
__device__ __forceinline__ void kick_link_dispatch(const KickArgs& a, const LatDev& L, int mu, int s, const int* x) {
  if (mu == 0) kick_link<D, N, R, REP, 0>(a, L, s, x);
  else if (mu == 1) kick_link<D, N, R, REP, 1>(a, L, s, x);
  else if constexpr (D > 2) {
    if (mu == 2) kick_link<D, N, R, REP, 2>(a, L, s, x);
    else if constexpr (D > 3) kick_link<D, N, R, REP, 3>(a, L, s, x);
  }
}

// Occupancy: resident kick blocks per SM.  FP32: 7 (72 registers; the fundamental spills 40
// bytes with tiles, 84 with consecutive sites), the adjoint 5 (its commutator terms spill 432
// bytes at 72 registers against 28 at 96); FP64: 4 (128 registers, 88 and 8 bytes spilled), the
// adjoint 3 (it spills 1.3 KB at 128 registers).  General irreps, whose link part is the gauge
// force alone, gain from the same: trajectories at SU(3) 12^4, FP32 5 and 7 blocks, octet 1366
// and 1275 us, sextet 1225 and 1185; FP64 3 and 4, 27-plet 6650 and 6425.  Pure gauge does not
// (nothing else runs between its kicks but the drift) and keeps 5 and 3: kick at 6^4, 12^4, 16^4
// with 5 / 7 blocks FP32 4.6 / 5.4, 10.3 / 12.1, 20.9 / 20.8 us, with 3 / 4 blocks FP64 5.2 / 6.1,
// 14.3 / 15.1, 33.2 / 35.0.  Measured at
// SU(3) 16^4 (fundamental): the kick alone runs the same at FP32 5 and 7 blocks (24.5
// us) and at FP64 3 and 4 (40.7 / 40.9 us), while the trajectory with the higher
// occupancy is 1.4% (FP32) and 1.7% (FP64) faster -- the next launch's blocks find room
// sooner; FP32 6 blocks (80 registers) was 2.5% slower; FP32 4 / FP64 2 lose ~4%.
// SU(2) (links from their first row, ld_su): FP32 8 and FP64 5.  A ladder of 16 lattices of
// 6, 8, 10, 12 / one 6^4, trajectories in us: FP32 7 blocks 1184 / 126, 8 1134 / 124, 9 1128 /
// 126; FP64 4 1851 / 141, 5 1702 / 138, 6 (spills) 1674 / 144.
#ifndef GH_KICK_MINB_F32
#define GH_KICK_MINB_F32 5
#endif
#ifndef GH_KICK_MINB_F32_FUND
#define GH_KICK_MINB_F32_FUND 7
#endif
#ifndef GH_KICK_MINB_F32_SU2
#define GH_KICK_MINB_F32_SU2 8
#endif
#ifndef GH_KICK_MINB_F64_SU2
#define GH_KICK_MINB_F64_SU2 5
#endif
#ifndef GH_KICK_MINB_F64
#define GH_KICK_MINB_F64 3
#endif
#ifndef GH_KICK_MINB_F64_FUND
#define GH_KICK_MINB_F64_FUND 4
#endif
template <int N, typename R, int REP> struct KickMinBlocks {
  static constexpr int b = N == 2 ? GH_KICK_MINB_F32_SU2 : REP == REP_FUND || REP == REP_GEN ? GH_KICK_MINB_F32_FUND : GH_KICK_MINB_F32;
  static constexpr int v = b * 128 / KICK_BLOCK;
};
template <int N, int REP> struct KickMinBlocks<N, double, REP> {
  static constexpr int b = N == 2 ? GH_KICK_MINB_F64_SU2 : REP == REP_FUND || REP == REP_GEN ? GH_KICK_MINB_F64_FUND : GH_KICK_MINB_F64;
  static constexpr int v = b * 128 / KICK_BLOCK > 0 ? b * 128 / KICK_BLOCK : 1;
};

// LIN: the table holds linear items (and perhaps tiles); without, tiles only.  SPLIT: its
// site items are kick_site_gen's.  Instances of their own: the FP32 kernel at 72 registers
// lost 1.7% at 16^4 with both link forms inside, the FP64 sextet 2% with both site forms.
template <int D, int N, typename R, int REP, bool LIN, bool SPLIT>
__global__ void __launch_bounds__(KICK_BLOCK, KickMinBlocks<N, R, REP>::v) k_kick(const KickArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  const LatDev& L = a.lats[w.lat];
  if constexpr (SPLIT) {
    if (w.mu < 0) {
      kick_site_gen<D, R>(a, L, w);
      return;
    }
  }
  int s, x[D], mu = w.mu;
  if (LIN && mu >= KICK_LINEAR - 1) {
    // consecutive sites: extents that power-of-two tiles do not divide (rule and figures
    // at kick_linear, gh_ctx.cu)
    mu -= KICK_LINEAR;
    if ((int)threadIdx.x >= w.n) return;
    s = w.s0 + (int)threadIdx.x;
    coords<D>(L, s, x);
    if (L.dec && !in_box<D>(L, x)) return;
  } else if (!tile_site<D>(L, w, threadIdx.x, s, x)) {
    return;
  }
  if (mu >= 0) kick_link_dispatch<D, N, R, REP>(a, L, mu, s, x);
  else if (REP != REP_NONE && !SPLIT) kick_site<D, N, R, REP>(a, L, s, x);
}

// ---------------------------------------------------------------------------
// General irrep: one warp per link.  D^(R)(U) phi is applied matrix-free on the
// tensor space V^{xn} exactly as src/rep/rep_general.hpp:184-220 does (lift with
// the basis W, apply U on each of the n slots, project with W^dag), but W and
// T^a_R are held sparse (97% / 94% zeros for the SU(3) 27-plet) and the lanes of
// the warp split the tensor index / slot fibres / basis vectors between them.
// Single-row irreps whose term list the host built (GenTables::sp_ptr) take D(U)
// in closed form instead (sympow_matrix: the lanes split the d*d entries), then
// two d x d matrix-vector products.
//   mode 0: psi_f = D phi_{x+mu}, psi_b = D^dag phi_x -> scratch; P -= eps F_matter
//   mode 1: psi_f only (for the scalar action and the link energy)
//   mode 2: F_matter -> out (no P update), psi_f, psi_b -> scratch
// hop_link_g: src/rep/representation.hpp:36-46 / rep_general.hpp:151-159.
// ---------------------------------------------------------------------------
struct GenArgs {
  const Work* work;
  const LatDev* lats;
  const void* U;
  void* P;
  const void* phi;
  void* psif;
  void* psib;
  GenTables t;
  double eps;
  int mode;
  double* out;
  int pot;            // POT_MULTI: the warps of mu = 0 also write w = A(M) phi_x
  PotA sa;            // superoperator rows, FP64 values
  double2* wpot;      // w per site, FP64, laid out like phi
};

template <int N, typename C>
__device__ void gen_apply(const GenTables& t, const Mat<N, C>& M, bool dag, const cx<C>* vin, cx<C>* buf,
                          cx<C>* vout, int lane) {
  // lift: buf[i] = sum_l vin[l] W_l[i]
  for (int i = lane; i < t.dimT; i += 32) {
    cx<C> s = zero<C>();
    for (int p = t.wt_ptr[i]; p < t.wt_ptr[i + 1]; ++p) {
      const double2 w = t.wt_v[p];
      s = cfma(s, vin[t.wt_l[p]], mk<C>((C)w.x, (C)w.y));
    }
    buf[i] = s;
  }
  __syncwarp();
  // slot applies: fibre f of slot sl holds the N entries base + j*blk
  const int nf = t.dimT / N;
  for (int sl = 0; sl < t.n; ++sl) {
    const int k = t.n - 1 - sl;
    const int blk = t.powN[k];
    const unsigned mag = t.pmag[k];
    // fibre f = hi * blk + lo starts at hi * blk * N + lo.  Odd N in FP64 with more than
    // 64 fibres per slot (over two per lane) walks them as f = lo * N^(n-1-k) + hi instead (consecutive
    // lanes step hi): the same fibres, each computed alike, so the results do not change;
    // SU(3) 27-plet FP64 trajectories +8%, while the sextet, the octet and FP32 ran 1-4%
    // slower with it, so they keep the plain order
    const int kq = t.n - 1 - k;
    const unsigned magq = t.pmag[kq];
    const bool swap = (sizeof(C) == 8) && (N & 1) && nf > 64;
    for (int f = lane; f < nf; f += 32) {
      int base;
      if (swap) {
        const int lo = (kq == 0) ? f : (int)__umulhi((unsigned)f, magq);
        base = (f - lo * t.powN[kq]) * blk * N + lo;
      } else {
        const int q = (k == 0) ? f : (int)__umulhi((unsigned)f, mag);
        base = q * blk * (N - 1) + f;              // (f / blk) * blk * N + f % blk
      }
      cx<C> v[N];
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = buf[base + j * blk];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        cx<C> s = zero<C>();
#pragma unroll
        for (int g = 0; g < N; ++g) s = dag ? cfma_cj(s, M.e[g * N + j], v[g]) : cfma(s, M.e[j * N + g], v[g]);
        buf[base + j * blk] = s;
      }
    }
    __syncwarp();
  }
  // project: vout[k] = sum_i conj(W_k[i]) buf[i]
  for (int k = lane; k < t.d; k += 32) {
    cx<C> s = zero<C>();
    for (int p = t.w_ptr[k]; p < t.w_ptr[k + 1]; ++p) {
      const double2 w = t.w_v[p];
      s = cfma_cj(s, mk<C>((C)w.x, (C)w.y), buf[t.w_i[p]]);
    }
    vout[k] = s;
  }
  __syncwarp();
}

// D(U) of a single-row irrep from its term list, FP64, one warp:
//   D[k][l] = sum_terms c prod_ij U_ij^K_ij
// with the powers U_ij^p (p = 0..n) tabulated first (entry ij*(n+1) + p) and each term
// given by its offsets into that table.  Dm: d*d, Pw: N*N*(n+1) entries of this warp's
// shared memory.
template <int N, typename C>
__device__ void sympow_matrix(const GenTables& t, const Mat<N, C>& M, cx<double>* Dm, cx<double>* Pw, int lane) {
  const int n = t.n, d = t.d;
  if (lane < N * N) {
    const cx<double> u = mk<double>((double)M.e[lane].re, (double)M.e[lane].im);
    cx<double> p = mk<double>(1.0, 0.0);
    for (int q = 0; q <= n; ++q) {
      Pw[lane * (n + 1) + q] = p;
      p = mul(p, u);
    }
  }
  __syncwarp();
  for (int e = lane; e < d * d; e += 32) {
    cx<double> acc = zero<double>();
    for (int q = t.sp_ptr[e]; q < t.sp_ptr[e + 1]; ++q) {
      const double2 c = t.sp_c[q];
      cx<double> pr = mk<double>(c.x, c.y);
      // offsets into the power table, N*N bytes per term in whole 32-bit words: SU(2)
      // multiplies all four factors (an exponent 0 points at a 1), larger N the nonzero
      // factors up to the first 0xFF
      constexpr int EW = (N * N + 3) / 4;
      const unsigned* ex = reinterpret_cast<const unsigned*>(t.sp_e) + (size_t)q * EW;
      unsigned w[EW];
#pragma unroll
      for (int i = 0; i < EW; ++i) w[i] = __ldg(ex + i);
      if constexpr (N == 2) {
#pragma unroll
        for (int f = 0; f < 4; ++f) pr = mul(pr, Pw[(w[0] >> (8 * f)) & 0xFF]);
      } else {
#pragma unroll
        for (int f = 0; f < N * N; ++f) {
          const unsigned o = (w[f >> 2] >> (8 * (f & 3))) & 0xFF;
          if (o == 0xFF) break;
          pr = mul(pr, Pw[o]);
        }
      }
      acc = add(acc, pr);
    }
    Dm[e] = acc;
  }
  __syncwarp();
}

template <int D, int N, typename R>
__global__ void __launch_bounds__(GEN_WARPS * 32) k_gen_links(const GenArgs a) {
  pdl_enter();
  typedef typename Cmp<R>::t C;
  extern __shared__ unsigned char smem_raw[];
  const Work w = a.work[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp >= w.n) return;
  const LatDev L = a.lats[w.lat];
  const int mu = w.mu, s = w.s0 + warp;
  const int d = a.t.d, dimT = a.t.dimT;
  // this warp's shared memory: tensor path [buf: dimT][px py pf pb: d each];
  // closed-form path [Dm: d*d][Pw: N*N*(n+1)] (FP64) then [px py pf pb]
  unsigned char* wbase = smem_raw + (size_t)warp * a.t.warp_bytes;
  const bool sp = a.t.sp_ptr != nullptr;
  cx<double>* Dm = reinterpret_cast<cx<double>*>(wbase);
  cx<double>* Pw = Dm + d * d;
  cx<C>* buf = reinterpret_cast<cx<C>*>(wbase);
  // the region before px (the tensor buffer or D and the powers) also holds, before it
  // is filled, A(M) of the potential (d*d FP64 complex) where that fits, and, after,
  // the matter force's partial sums (ng*d doubles, which the host makes room for)
  cx<C>* px = reinterpret_cast<cx<C>*>(wbase + a.t.px_off);
  cx<C>* py = px + d;
  cx<C>* pf = py + d;
  cx<C>* pb = pf + d;
  const R* U = (const R*)a.U;
  const R* phi = (const R*)a.phi;
  int x[D];
  coords<D>(L, s, x);
  if (!below_hi<D>(L, x)) return;                // upper halo link of a subdomain (whole warp)
  const bool own = in_box<D>(L, x);              // the link's momentum belongs to this subdomain
  const int spm = nfwd(L, s, x[mu], mu);
  const Mat<N, C> M = ld_link<N, C>(U, L, mu, s);
  for (int k = lane; k < d; k += 32) {
    px[k] = ldc<C>(phi, f_index(L, d, k, s));
    py[k] = ldc<C>(phi, f_index(L, d, k, spm));
  }
  __syncwarp();
  if (a.pot == POT_MULTI && mu == 0) {
    // multi-invariant potential of site s (FP64):
    //   A(M)_rq = sum_ij A_{rq,ij} phi_i conj(phi_j),  w_r = sum_q A(M)_rq phi_q.
    // Where A(M) fits in the region before px (always on the closed-form path) the
    // lanes split the row pairs rq, then one lane per r sums over q; otherwise one
    // lane per r does both.  Fixed summation order either way.
    const double2* __restrict__ av = reinterpret_cast<const double2*>(a.sa.v);
    const bool split = (size_t)d * d * sizeof(cx<double>) <= (size_t)a.t.px_off;
    cx<double>* AM = reinterpret_cast<cx<double>*>(wbase);
    auto am = [&](int rq) {
      const int b = __ldg(a.sa.ptr + rq), e = __ldg(a.sa.ptr + rq + 1);
      cx<double> y = zero<double>();
      for (int z = b; z < e; ++z) {
        const int ij = __ldg(a.sa.ij + z);
        const double2 v = __ldg(av + z);
        const cx<C> pi = px[ij & 0xFF], pj = px[ij >> 8];
        y = cfma(y, mk<double>(v.x, v.y), mulc(mk<double>(pi.re, pi.im), mk<double>(pj.re, pj.im)));
      }
      return y;
    };
    if (split) {
      for (int rq = lane; rq < d * d; rq += 32) AM[rq] = am(rq);
      __syncwarp();
    }
    for (int r = lane; r < d; r += 32) {
      cx<double> acc = zero<double>();
      for (int q = 0; q < d; ++q) acc = cfma(acc, split ? AM[r * d + q] : am(r * d + q), mk<double>(px[q].re, px[q].im));
      a.wpot[f_index(L, d, r, s)] = make_double2(acc.re, acc.im);
    }
    __syncwarp();
  }
  if (sp) {
    sympow_matrix<N, C>(a.t, M, Dm, Pw, lane);
    // psi_f = D phi_y on lanes 0..d-1, psi_b = D^dag phi_x on the next d lanes
    const int nv = a.mode == 1 ? d : 2 * d;
    for (int t = lane; t < nv; t += 32) {
      cx<double> acc = zero<double>();
      if (t < d) {
        for (int l = 0; l < d; ++l) acc = cfma(acc, Dm[t * d + l], mk<double>((double)py[l].re, (double)py[l].im));
        pf[t] = mk<C>((C)acc.re, (C)acc.im);
      } else {
        const int k = t - d;
        for (int l = 0; l < d; ++l) acc = cfma_cj(acc, Dm[l * d + k], mk<double>((double)px[l].re, (double)px[l].im));
        pb[k] = mk<C>((C)acc.re, (C)acc.im);
      }
    }
    __syncwarp();
  } else {
    gen_apply<N, C>(a.t, M, false, py, buf, pf, lane);
    if (a.mode != 1) gen_apply<N, C>(a.t, M, true, px, buf, pb, lane);
  }
  R* psif = (R*)a.psif;
  R* psib = (R*)a.psib;
  for (int k = lane; k < d; k += 32) {
    const long long gi = g_index(L, d, mu, k, s);
    stc<C>(psif, gi, pf[k]);
    if (a.mode != 1) stc<C>(psib, gi, pb[k]);
  }
  if (a.mode == 1 || !own) return;
  // matter force: g^a = -2 Im(phi_x^dag T^a_R psi_f), F^a = -kappa g^a.  The lanes
  // split the (a, row) pairs; the rows of each a are then summed in order.
  constexpr int ng = N * N - 1;
  double* zc = reinterpret_cast<double*>(wbase);
  for (int r = lane; r < ng * d; r += 32) {
    const int i = r % d;
    cx<C> ti = zero<C>();
    for (int p = a.t.t_ptr[r]; p < a.t.t_ptr[r + 1]; ++p) {
      const double2 tv = a.t.t_v[p];
      ti = cfma(ti, mk<C>((C)tv.x, (C)tv.y), pf[a.t.t_j[p]]);
    }
    zc[r] = (double)px[i].re * (double)ti.im - (double)px[i].im * (double)ti.re;   // Im(conj(phi_i) t_i)
  }
  __syncwarp();
  for (int g = lane; g < ng; g += 32) {
    double zim = 0.0;
    for (int i = 0; i < d; ++i) zim += zc[g * d + i];
    const C F = -(C)L.kappa * (C(-2) * (C)zim);
    const long long pi_ = p_index(L, ng, mu, g, s);
    if (a.mode == 0) {
      R* P = (R*)a.P;
      P[pi_] = (R)((C)P[pi_] - (C)a.eps * F);
    } else {
      a.out[pi_] = (double)F;
    }
  }
}

// ---------------------------------------------------------------------------
// SU(2) irreps {n} in closed form, 32 links per block.  With U's first row (a, b), x = |a|^2
// and y = |b|^2 the entries of D(U) with k + l <= n are
//   D_kl = a^(n-k-l) b^(l-k) sum_i s_i x^(m-i) y^i,  m = min(k, l)
// (conj(b)^(k-l) for l < k; s_i the coefficients of the term list with the signs of U's
// second row (-conj b, conj a)), and D_(n-k)(n-l) = (-1)^(k+l) conj(D_kl) gives the others:
// for n = 12 91 entries of 3.3 real terms on average, where the term list has 455 products
// of four complex powers (k_gen_links).  A lane is a link; the warps split the powers, then
// the entries, then the rows of psi_f = D phi_y and psi_b = D^dag phi_x; all in FP64
// whatever the fields.  Work items with mu < 0 are 32 sites for the multi-invariant
// potential (they come first, being the longest): the upper triangle of M = phi phi^dag, then
// w = A(M) phi row by row from the nonzeros of A.  Modes and outputs as k_gen_links.
// Bound: latency of the four phases and shared memory.  SU(2) {12} 8^4 FP64 with the
// 13-channel potential, cold caches: 43 us against k_gen_links' 111.
// ---------------------------------------------------------------------------
constexpr int SPIN_WARPS = 8, SPIN_ROWS = 3;      // rows per warp: d <= 18
__host__ __device__ constexpr int spin_entries(int n) { return (n + 1) * (n + 2) / 2; }
__host__ __device__ constexpr int spin_at(int n, int k, int l) { return k * (n + 1) - k * (k - 1) / 2 + l; }
__host__ __device__ constexpr size_t spin_smem(int n) {
  return (size_t)32 * (16 * (spin_entries(n) + 2 * (n + 1)) + 8 * 2 * (n / 2 + 1));
}
// what the kernel can take: its rows, a block's shared memory, and room over D's entries for the
// force's partial sums (3 per warp), which must not reach the vectors behind them: n >= 4
__host__ __device__ constexpr bool spin_fits(int n) {
  return n + 1 <= SPIN_WARPS * SPIN_ROWS && spin_smem(n) <= 227 * 1024 && 16 * spin_entries(n) >= 8 * 3 * SPIN_WARPS;
}
template <int D, typename R>
__global__ void __launch_bounds__(SPIN_WARPS * 32, 3) k_gen_spin(const GenArgs a) {
  pdl_enter();
  typedef typename Cmp<R>::t C;
  extern __shared__ unsigned char smem_raw[];
  const Work w = a.work[blockIdx.x];
  const LatDev& L = a.lats[w.lat];
  const int n = a.t.n, d = n + 1;
  const int c = threadIdx.x & 31, q = threadIdx.x >> 5;
  cx<double>* Dm = reinterpret_cast<cx<double>*>(smem_raw) + c;      // [entries][32]
  cx<double>* Pa = Dm + 32 * spin_entries(n);                        // [d][32] powers of a, later phi_{x+mu}
  cx<double>* Pb = Pa + 32 * d;                                      // [d][32] powers of b, later phi_x
  double* X = reinterpret_cast<double*>(Pb - c + 32 * d) + c;        // [n/2+1][32] powers of x, then of y
  double* Y = X + 32 * (n / 2 + 1);
  const int s = w.s0 + (c < w.n ? c : 0);                            // lanes past the lattice's end repeat site s0
  int x[D];
  coords<D>(L, s, x);
  const bool live = c < w.n && below_hi<D>(L, x);
  const R* phi = (const R*)a.phi;
  if (w.mu < 0) {                                                    // potential of 32 sites
    for (int k = q; k < d; k += SPIN_WARPS) Pb[k * 32] = ldc<double>(phi, f_index(L, d, k, s));
    __syncthreads();
    for (int e = q; e < d * d; e += SPIN_WARPS) {                    // M_ij, i <= j, at [i][j - i] of a triangle
      const int i = e / d, j = e - i * d;
      if (i <= j) Dm[spin_at(n, i, j - i) * 32] = mulc(Pb[i * 32], Pb[j * 32]);
    }
    __syncthreads();
    const double2* __restrict__ av = reinterpret_cast<const double2*>(a.sa.v);
    const auto m = [&](int ij) {
      const int i = ij & 0xFF, j = ij >> 8;
      cx<double> z = Dm[spin_at(n, i < j ? i : j, i < j ? j - i : i - j) * 32];
      if (i > j) z.im = -z.im;
      return z;
    };
    const auto am = [&](int rq) {
      cx<double> y = zero<double>();
      const int e1 = __ldg(a.sa.ptr + rq + 1);
      int z = __ldg(a.sa.ptr + rq);
      for (; z + 4 <= e1; z += 4) {                                  // four in flight
        int ij[4];
        double2 v[4];
        cx<double> t[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) { ij[k] = __ldg(a.sa.ij + z + k); v[k] = __ldg(av + z + k); }
#pragma unroll
        for (int k = 0; k < 4; ++k) t[k] = m(ij[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) y = cfma(y, mk<double>(v[k].x, v[k].y), t[k]);
      }
      for (; z < e1; ++z) {
        const double2 v = __ldg(av + z);
        y = cfma(y, mk<double>(v.x, v.y), m(__ldg(a.sa.ij + z)));
      }
      return y;
    };
    for (int r = q; r < d; r += SPIN_WARPS) {
      cx<double> acc = zero<double>();
      for (int k = 0; k < d; ++k) acc = cfma(acc, am(r * d + k), Pb[k * 32]);
      if (c < w.n) a.wpot[f_index(L, d, r, s)] = make_double2(acc.re, acc.im);
    }
    return;
  }
  const int mu = w.mu;
  const bool own = live && in_box<D>(L, x);
  const int spm = nfwd(L, s, x[mu], mu);
  cx<double> px[SPIN_ROWS], py[SPIN_ROWS];
#pragma unroll
  for (int t = 0; t < SPIN_ROWS; ++t) {
    const int k = q + SPIN_WARPS * t;
    if (k < d) { px[t] = ldc<double>(phi, f_index(L, d, k, s)); py[t] = ldc<double>(phi, f_index(L, d, k, spm)); }
  }
  if (q < 4) {
    const cx<double> u = ldc<double>((const R*)a.U, u_index(L, 4, mu, q & 1, s));
    if (q < 2) {
      cx<double>* P = q ? Pb : Pa;
      cx<double> p = mk<double>(1.0, 0.0);
      for (int k = 0; k < d; ++k) { P[k * 32] = p; p = mul(p, u); }
    } else {
      double* P = q == 3 ? Y : X;
      const double r = norm2(u);
      double p = 1.0;
      for (int k = 0; k <= n / 2; ++k) { P[k * 32] = p; p *= r; }
    }
  }
  __syncthreads();
  for (int e = q; e < spin_entries(n); e += SPIN_WARPS) {
    const int4 t = __ldg(a.t.spin_ent + e);                          // k, l, first coefficient
    const int m = t.x < t.y ? t.x : t.y;
    double r = 0.0;
#pragma unroll 4
    for (int i = 0; i <= m; ++i) r = fmad(__ldg(a.t.spin_c + t.z + i) * X[(m - i) * 32], Y[i * 32], r);
    const cx<double> pb = Pb[(t.y >= t.x ? t.y - t.x : t.x - t.y) * 32];
    const cx<double> pa = scale(Pa[(n - t.x - t.y) * 32], r);
    Dm[e * 32] = t.y >= t.x ? mul(pa, pb) : mulc(pa, pb);
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < SPIN_ROWS; ++t) {
    const int k = q + SPIN_WARPS * t;
    if (k < d) { Pa[k * 32] = py[t]; Pb[k * 32] = px[t]; }
  }
  __syncthreads();
  const auto entry = [&](int k, int l) {
    if (k + l <= n) return Dm[spin_at(n, k, l) * 32];
    const cx<double> z = Dm[spin_at(n, n - k, n - l) * 32];
    return (k + l) & 1 ? mk<double>(-z.re, z.im) : mk<double>(z.re, -z.im);
  };
  cx<double> f[SPIN_ROWS];
#pragma unroll
  for (int t = 0; t < SPIN_ROWS; ++t) {
    const int k = q + SPIN_WARPS * t;
    f[t] = zero<double>();
    if (k >= d) continue;
#pragma unroll 4
    for (int l = 0; l < d; ++l) f[t] = cfma(f[t], entry(k, l), Pa[l * 32]);
    if (live) stc<double>((R*)a.psif, g_index(L, d, mu, k, s), f[t]);
  }
  if (a.mode == 1) return;
#pragma unroll
  for (int t = 0; t < SPIN_ROWS; ++t) {
    const int k = q + SPIN_WARPS * t;
    if (k >= d) continue;
    cx<double> z = zero<double>();
#pragma unroll 4
    for (int l = 0; l < d; ++l) z = cfma_cj(z, entry(l, k), Pb[l * 32]);
    if (live) stc<double>((R*)a.psib, g_index(L, d, mu, k, s), z);
  }
  __syncthreads();                                                   // phi_{x+mu} and D are read
#pragma unroll
  for (int t = 0; t < SPIN_ROWS; ++t)
    if (q + SPIN_WARPS * t < d) Pa[(q + SPIN_WARPS * t) * 32] = f[t];
  __syncthreads();
  // matter force g^a = -2 Im(phi_x^dag T^a_R psi_f): the warps split the rows
  double F[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int t = 0; t < SPIN_ROWS; ++t) {
    const int i = q + SPIN_WARPS * t;
    if (i >= d) continue;
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      cx<double> ti = zero<double>();
      const int e1 = __ldg(a.t.t_ptr + g * d + i + 1);
      for (int e = __ldg(a.t.t_ptr + g * d + i); e < e1; ++e) {
        const double2 tv = __ldg(a.t.t_v + e);
        ti = cfma(ti, mk<double>(tv.x, tv.y), Pa[__ldg(a.t.t_j + e) * 32]);
      }
      F[g] += px[t].re * ti.im - px[t].im * ti.re;
    }
  }
  double* Fs = reinterpret_cast<double*>(smem_raw) + c;
#pragma unroll
  for (int g = 0; g < 3; ++g) Fs[(q * 3 + g) * 32] = F[g];
  __syncthreads();
  if (q < 3 && own) {
    double z = 0.0;
#pragma unroll
    for (int k = 0; k < SPIN_WARPS; ++k) z += Fs[(k * 3 + q) * 32];
    const C Fa = -(C)L.kappa * (C(-2) * (C)z);
    const long long pi_ = p_index(L, 3, mu, q, s);
    if (a.mode == 0) {
      R* P = (R*)a.P;
      P[pi_] = (R)((C)P[pi_] - (C)a.eps * Fa);
    } else {
      a.out[pi_] = (double)Fa;
    }
  }
}

// ---------------------------------------------------------------------------
// General irreps inside the two-fold adjoint product that are no symmetric tensors (10bar
// {3,3}; host set-up and the algebra in gh_adjprod.h): with the fixed isometric
// intertwiner Q (A x d, A = (N^2 - 1)^2) from the reference's basis into the product,
//   D_R(U) phi = Q^dag (G (x) G) Q phi,   G_ab = 2 Re Tr(T^a U T^b U^dag),
// and D_R(U)^dag phi with G^T.  One block takes the 32 links of one 32-site block and
// one direction, 8 threads per link: the lift Q phi and the projection Q^dag y are
// 64 x 27 and 27 x 64 products shared by the 32 links (every warp reads the same Q
// entry, every lane its own link); G (x) G acts as X -> G X G^T on each link's 8 x 8
// coefficient matrix, one row per thread.  Same modes and outputs as k_gen_links
// (psi_f, psi_b, matter force); the multi-invariant potential's w stays there.
// The matter force is g^a = -2 Im(phi_x^dag T^a_R psi_f) (src/rep/rep_general.hpp:151-159),
// one generator per thread, rows summed in order.
// ---------------------------------------------------------------------------
constexpr int GP_LINKS = 32;      // links per block (one 32-site block, one direction)
constexpr int GP_THREADS = 256;   // 8 per link
template <int N> struct AdjProd {
  static constexpr int NG = N * N - 1;
  static constexpr int A = NG * NG;
  static constexpr int RA = (A + 7) / 8;      // rows of A (and of d <= A) per thread
};
template <int N, typename C> __host__ __device__ constexpr size_t gen_prod_smem(int d, int nrows) {
  return (size_t)nrows * d * sizeof(cx<C>) + (size_t)(2 * d + AdjProd<N>::A) * GP_LINKS * sizeof(cx<C>) +
         (size_t)AdjProd<N>::NG * AdjProd<N>::NG * GP_LINKS * sizeof(C);
}

// out[i] = (D phi)_k, k = q + 8 i, for the link in lane c; Pin: [d][32] input vectors;
// Qs: [nrows][d] the rows of Q in shared memory; X: [A][32] work space; G: [NG][NG][32]
// adjoint matrices.  Every thread of the block calls it.
template <int N, typename C>
__device__ __forceinline__ void gp_apply(const GenTables& t, const cx<C>* Qs, int d, const cx<C>* Pin, cx<C>* X,
                                         const C* G, bool dag, int c, int q, cx<C>* out) {
  constexpr int NG = AdjProd<N>::NG, RA = AdjProd<N>::RA, LB = GP_LINKS;
  const int nr = t.pnrows;
  cx<C> acc[RA];
#pragma unroll
  for (int i = 0; i < RA; ++i) acc[i] = zero<C>();
  for (int l = 0; l < d; ++l) {                         // lift: the needed rows of X = Q phi
    const cx<C> p = Pin[l * LB + c];
#pragma unroll
    for (int i = 0; i < RA; ++i) {
      const int r = q + 8 * i;
      if (r < nr) acc[i] = cfma(acc[i], Qs[r * d + l], p);
    }
  }
  __syncthreads();                                      // earlier readers of X are done
  if (t.psym < 0 && q < NG) X[(q * NG + q) * LB + c] = zero<C>();   // antisymmetric: zero diagonal
#pragma unroll
  for (int i = 0; i < RA; ++i) {
    const int r = q + 8 * i;
    if (r < nr) {
      const int e = __ldg(t.prow + r);
      X[e * LB + c] = acc[i];
      if (t.psym != 0) {
        const int a = e / NG, b = e - a * NG;
        if (a != b) X[(b * NG + a) * LB + c] = t.psym > 0 ? acc[i] : mk<C>(-acc[i].re, -acc[i].im);
      }
    }
  }
  __syncthreads();
  auto g = [&](int a, int b) { return dag ? G[(b * NG + a) * LB + c] : G[(a * NG + b) * LB + c]; };
  {                                                     // Y = G X G^T, row a of this thread
    const int a = q;
    cx<C> y[NG];
    if (a < NG) {
      cx<C> z[NG];
#pragma unroll
      for (int b = 0; b < NG; ++b) {
        cx<C> sacc = zero<C>();
#pragma unroll
        for (int k = 0; k < NG; ++k) sacc = add(sacc, scale(X[(k * NG + b) * LB + c], g(a, k)));
        z[b] = sacc;
      }
#pragma unroll
      for (int b = 0; b < NG; ++b) {
        cx<C> sacc = zero<C>();
#pragma unroll
        for (int k = 0; k < NG; ++k) sacc = add(sacc, scale(z[k], g(b, k)));
        y[b] = sacc;
      }
    }
    __syncthreads();
    if (a < NG)
#pragma unroll
      for (int b = 0; b < NG; ++b) X[(a * NG + b) * LB + c] = y[b];
  }
  __syncthreads();
  // project: out = Q^dag y over the needed rows; off-diagonal pairs of a symmetric or
  // antisymmetric coefficient matrix count twice (their mirror entries are equal terms)
#pragma unroll
  for (int i = 0; i < RA; ++i) {
    const int k = q + 8 * i;
    cx<C> s1 = zero<C>(), s2 = zero<C>();
    if (k < d) {
      for (int r = 0; r < t.pndiag; ++r) s1 = cfma_cj(s1, Qs[r * d + k], X[__ldg(t.prow + r) * LB + c]);
      for (int r = t.pndiag; r < nr; ++r) s2 = cfma_cj(s2, Qs[r * d + k], X[__ldg(t.prow + r) * LB + c]);
    }
    out[i] = add(s1, scale(s2, C(2)));
  }
}

template <int D, int N, typename R>
__global__ void __launch_bounds__(GP_THREADS) k_gen_prod(const GenArgs a) {
  pdl_enter();
  typedef typename Cmp<R>::t C;
  constexpr int NG = AdjProd<N>::NG, A = AdjProd<N>::A, RA = AdjProd<N>::RA, LB = GP_LINKS;
  extern __shared__ unsigned char smem_raw[];
  const Work w = a.work[blockIdx.x];
  const LatDev& L = a.lats[w.lat];
  const int d = a.t.d;
  const int c = threadIdx.x & (LB - 1), q = threadIdx.x >> 5;
  cx<C>* Qs = reinterpret_cast<cx<C>*>(smem_raw);       // [nrows][d] the rows of Q the lift uses
  cx<C>* Px = Qs + a.t.pnrows * d;                      // [d][32] phi_x
  cx<C>* Py = Px + d * LB;                              // [d][32] phi_{x+mu}, then psi_f
  cx<C>* X = Py + d * LB;                               // [A][32]
  C* G = reinterpret_cast<C*>(X + A * LB);              // [NG][NG][32]
  {
    const typename V2<C>::t* Qv = reinterpret_cast<const typename V2<C>::t*>(
        sizeof(C) == sizeof(double) ? (const void*)a.t.pq64 : (const void*)a.t.pq32);
    for (int i = threadIdx.x; i < a.t.pnrows * d; i += GP_THREADS) {
      const typename V2<C>::t v = __ldg(Qv + i);
      Qs[i] = mk<C>(v.x, v.y);
    }
  }
  const int mu = w.mu;
  const int s = w.s0 + (c < w.n ? c : 0);              // lanes past the lattice's end compute on site s0
  int x[D];
  coords<D>(L, s, x);
  const bool live = c < w.n && below_hi<D>(L, x);      // and store nothing, as upper halo sites of a subdomain
  const bool own = live && in_box<D>(L, x);            // momentum updates: interior links only
  const int spm = nfwd(L, s, x[mu], mu);
  const R* phi = (const R*)a.phi;
  for (int k = q; k < d; k += 8) {
    Px[k * LB + c] = ldc<C>(phi, f_index(L, d, k, s));
    Py[k * LB + c] = ldc<C>(phi, f_index(L, d, k, spm));
  }
  {
    const Mat<N, C> U = ld_link<N, C>((const R*)a.U, L, mu, s);
    for (int b = q; b < NG; b += 8) {                   // column b of G: 2 Tr(T^a U T^b U^dag)
      C e[NG];
#pragma unroll
      for (int k = 0; k < NG; ++k) e[k] = (k == b) ? C(1) : C(0);
      const Mat<N, C> M = mm_nd(mm(U, alg_to_mat<N, C>(e)), U);
      cx<C> o[NG];
      tr2_proj<N, C>(M, o);
#pragma unroll
      for (int k = 0; k < NG; ++k) G[(k * NG + b) * LB + c] = o[k].re;
    }
  }
  __syncthreads();
  R* psif = (R*)a.psif;
  R* psib = (R*)a.psib;
  cx<C> o[RA];
  gp_apply<N, C>(a.t, Qs, d, Py, X, G, false, c, q, o);  // psi_f = D phi_{x+mu}
#pragma unroll
  for (int i = 0; i < RA; ++i) {
    const int k = q + 8 * i;
    if (k < d) {
      Py[k * LB + c] = o[i];
      if (live) stc<C>(psif, g_index(L, d, mu, k, s), o[i]);
    }
  }
  if (a.mode == 1) return;
  gp_apply<N, C>(a.t, Qs, d, Px, X, G, true, c, q, o);   // psi_b = D^dag phi_x
#pragma unroll
  for (int i = 0; i < RA; ++i) {
    const int k = q + 8 * i;
    if (k < d && live) stc<C>(psib, g_index(L, d, mu, k, s), o[i]);
  }
  __syncthreads();
  for (int gi = q; gi < NG; gi += 8) {                  // matter force, generator gi
    double zim = 0.0;
    for (int i = 0; i < d; ++i) {
      const int r = gi * d + i;
      cx<C> ti = zero<C>();
      for (int p = a.t.t_ptr[r]; p < a.t.t_ptr[r + 1]; ++p) {
        const double2 tv = a.t.t_v[p];
        ti = cfma(ti, mk<C>((C)tv.x, (C)tv.y), Py[a.t.t_j[p] * LB + c]);
      }
      const cx<C> pxi = Px[i * LB + c];
      zim += (double)pxi.re * (double)ti.im - (double)pxi.im * (double)ti.re;   // Im(conj(phi_i) t_i)
    }
    if (!own) continue;
    const C F = -(C)L.kappa * (C(-2) * (C)zim);
    const long long pi_ = p_index(L, NG, mu, gi, s);
    if (a.mode == 0) {
      R* P = (R*)a.P;
      P[pi_] = (R)((C)P[pi_] - (C)a.eps * F);
    } else {
      a.out[pi_] = (double)F;
    }
  }
}

// ---------------------------------------------------------------------------
// Irreps of the two-fold adjoint product that are symmetric tensors: D_R(U) acts on
//   Phi^{ij}_{kl} = 2 sum_ab (Q phi)_ab T^a_ik T^b_jl   as   U U Phi U^dag U^dag,
// and when Phi is symmetric in (i, j) and in (k, l) (SU(3) 27-plet {4,2}, SU(2) {4}; the
// host checks it, ghadj::sym2_map) its NS x NS entries, NS = N (N + 1) / 2, carry the irrep.
// A column (fixed k <= l) is a symmetric N x N matrix M that becomes V M V^T with V = U,
// a row (fixed i <= j) the same with V = conj(U), each by one thread with U in registers
// (SU(3): 45 complex multiply-adds).  Lift and projection are real and sparse in this
// basis (27-plet: 55 nonzeros of 36 x 27, where the intertwiner into the generators'
// basis is dense: 2 x 972 complex multiply-adds per apply).  The matter force
// g^a = -2 Im phi_x^dag T^a_R psi, with T^a_R acting on every index, is
//   F = 4 kappa Im Tr T^a (A - B^T),  A = sum_J w_J M_psi M_x^dag, B = sum_I w_I N_psi N_x^dag
// over columns J and rows I (w = 1 on the diagonal pairs, 2 off it).
// Split: one block per 32 links of a direction, a warp per column (then per row), a lane
// per link: shared memory is read without conflicts and every table entry is uniform.
// Bound: latency, on 18 warps per SM (FP64 pipe 29% busy, shared memory 45%; about 7,000
// multiply-adds per link).  3 blocks per SM (284 bytes spilled) beat 2 without spills by 4%.
// FP32 fields, whose force is summed in double too: kick and drift at 12^4 with 3 / 4 / 5 blocks
// 98.9 / 93.6 / 103.1 us (83.1 with the force in FP32, 350 with k_gen_prod).
// ---------------------------------------------------------------------------
constexpr int S2_NNZ = 64, S2_DMAX = 36, S2_PAIRS = 36;   // largest tables the kernel takes
struct Sym2Tab {
  unsigned char lptr[S2_PAIRS + 4], lm[S2_NNZ];    // lift: rows IJ, components m
  unsigned char pptr[S2_DMAX + 4], pe[S2_NNZ];     // projection: rows m, entries IJ
  double lc64[S2_NNZ], pc64[S2_NNZ];               // pc: conj of the lift times w_I w_J
  float lc32[S2_NNZ], pc32[S2_NNZ];
};
struct Sym2Args { GenArgs g; Sym2Tab t; };
template <int N> struct Sym2 {
  static constexpr int NS = N * (N + 1) / 2, THREADS = 32 * NS;
  __host__ __device__ static constexpr int pair(int i, int j) { return i <= j ? i * N - i * (i - 1) / 2 + j - i : j * N - j * (j - 1) / 2 + i - j; }
};
// 32-lane complex rows of the phi_{x+mu} buffer, which the force's NS x ng partial sums (double)
// take over once it is lifted
template <int N, typename C> __host__ __device__ constexpr int sym2_rows(int d) {
  constexpr int need = Sym2<N>::NS * (N * N - 1) * (int)sizeof(double) / (int)sizeof(cx<C>) + 1;
  return d > need ? d : need;
}
// phi_x, phi_{x+mu} (then the partial sums), the tensor
template <int N, typename C> __host__ __device__ constexpr size_t sym2_smem(int d) {
  return (size_t)(d + sym2_rows<N, C>(d) + Sym2<N>::NS * Sym2<N>::NS) * 32 * sizeof(cx<C>);
}
// O = V M V^T for a symmetric M (pairs i <= j); V_ij = U_ij, transposed (TR) and / or conjugated (CJ)
template <int N, bool TR, bool CJ, typename C>
__device__ __forceinline__ void sym2_rotate(const Mat<N, C>& U, const cx<C>* M, cx<C>* O) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    cx<C> t[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      t[j] = zero<C>();
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const cx<C> v = U.e[TR ? k * N + i : i * N + k];
        t[j] = CJ ? cfma_cj(t[j], v, M[Sym2<N>::pair(k, j)]) : cfma(t[j], v, M[Sym2<N>::pair(k, j)]);
      }
    }
#pragma unroll
    for (int j = i; j < N; ++j) {
      cx<C> s = zero<C>();
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const cx<C> v = U.e[TR ? k * N + j : j * N + k];
        s = CJ ? cfma_cj(s, v, t[k]) : cfma(s, v, t[k]);
      }
      O[Sym2<N>::pair(i, j)] = s;
    }
  }
}
// F += or -= w Im Tr T^a (P X^dag)  (or its transpose), P and X symmetric; in double whatever
// the fields, since the rows' and the columns' terms cancel in part
template <int N, bool MINUS_T, typename C>
__device__ __forceinline__ void sym2_force(const cx<C>* P, const cx<C>* X, double w, double* F) {
  Mat<N, double> R;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      cx<double> s = zero<double>();
#pragma unroll
      for (int k = 0; k < N; ++k) s = cfma_cj(s, cvt<double>(X[Sym2<N>::pair(k, j)]), cvt<double>(P[Sym2<N>::pair(i, k)]));
      R.e[MINUS_T ? j * N + i : i * N + j] = s;
    }
  double f[N * N - 1];
  im_tr_proj<N, double>(R, f);
#pragma unroll
  for (int g = 0; g < N * N - 1; ++g) F[g] = fmad(MINUS_T ? -w : w, f[g], F[g]);
}

template <typename C> __device__ __forceinline__ C s2_lift(const Sym2Tab& t, int p) {
  if constexpr (sizeof(C) == sizeof(double)) return t.lc64[p];
  else return t.lc32[p];
}
template <typename C> __device__ __forceinline__ C s2_proj(const Sym2Tab& t, int p) {
  if constexpr (sizeof(C) == sizeof(double)) return t.pc64[p];
  else return t.pc32[p];
}

template <int D, int N, typename R>
__global__ void __launch_bounds__(Sym2<N>::THREADS, sizeof(R) == 8 ? 3 : 4) k_gen_sym2(const __grid_constant__ Sym2Args a) {
  pdl_enter();
  typedef typename Cmp<R>::t C;
  constexpr int NS = Sym2<N>::NS, ng = N * N - 1;
  extern __shared__ unsigned char smem_raw[];
  const Work w = a.g.work[blockIdx.x];
  const LatDev& L = a.g.lats[w.lat];
  const int d = a.g.t.d;
  const int c = threadIdx.x & 31, q = threadIdx.x >> 5;   // lane: link; warp: column J, then row I
  cx<C>* Px = reinterpret_cast<cx<C>*>(smem_raw) + c;     // [d][32] phi_x
  cx<C>* Py = Px + 32 * d;                                // [d][32] phi_{x+mu}
  cx<C>* X = Py + 32 * sym2_rows<N, C>(d);                // [NS][NS][32]
  double* Fs = reinterpret_cast<double*>(Py - c) + c;     // [NS][ng][32], once phi_{x+mu} is lifted
  const int mu = w.mu;
  const int s = w.s0 + (c < w.n ? c : 0);                 // lanes past the lattice's end compute on site s0
  int x[D];
  coords<D>(L, s, x);
  const bool live = c < w.n && below_hi<D>(L, x);         // and store nothing, as upper halo sites of a subdomain
  const bool own = live && in_box<D>(L, x);               // momentum updates: interior links only
  const int spm = nfwd(L, s, x[mu], mu);
  const R* phi = (const R*)a.g.phi;
  for (int k = q; k < d; k += NS) {
    Px[k * 32] = ldc<C>(phi, f_index(L, d, k, s));
    Py[k * 32] = ldc<C>(phi, f_index(L, d, k, spm));
  }
  const Mat<N, C> U = ld_link<N, C>((const R*)a.g.U, L, mu, s);
  auto lift = [&](const cx<C>* v, int e0, int step, cx<C>* M) {   // entries e0 + step i of the tensor of v
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      M[i] = zero<C>();
      const int e = e0 + step * i, p1 = a.t.lptr[e + 1];
      for (int p = a.t.lptr[e]; p < p1; ++p) {
        const cx<C> z = v[a.t.lm[p] * 32];
        const C l = s2_lift<C>(a.t, p);
        M[i].re = fmad(l, z.re, M[i].re);
        M[i].im = fmad(l, z.im, M[i].im);
      }
    }
  };
  auto project = [&](R* out) {
    for (int m = q; m < d; m += NS) {
      cx<C> z = zero<C>();
      const int p1 = a.t.pptr[m + 1];
      for (int p = a.t.pptr[m]; p < p1; ++p) {
        const cx<C> v = X[a.t.pe[p] * 32];
        const C l = s2_proj<C>(a.t, p);
        z.re = fmad(l, v.re, z.re);
        z.im = fmad(l, v.im, z.im);
      }
      if (live) stc<C>(out, g_index(L, d, mu, m, s), z);
    }
  };
  // w_q: 1 on the diagonal pairs, 2 off it
  bool diag = false;
#pragma unroll
  for (int i = 0; i < N; ++i) diag = diag || q == Sym2<N>::pair(i, i);
  const double k4 = 4.0 * L.kappa * (diag ? 1.0 : 2.0);
  __syncthreads();
  cx<C> M[NS], O[NS];
  lift(Py, q, NS, M);                                     // psi_f = D phi_{x+mu}: columns, U
  sym2_rotate<N, false, false, C>(U, M, O);
#pragma unroll
  for (int i = 0; i < NS; ++i) X[(i * NS + q) * 32] = O[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NS; ++i) M[i] = X[(q * NS + i) * 32];   // rows, conj(U)
  sym2_rotate<N, false, true, C>(U, M, O);
#pragma unroll
  for (int i = 0; i < NS; ++i) X[(q * NS + i) * 32] = O[i];
  double F[ng];
  if (a.g.mode != 1) {
#pragma unroll
    for (int g = 0; g < ng; ++g) F[g] = 0.0;
    lift(Px, q * NS, 1, M);
    sym2_force<N, true, C>(O, M, k4, F);
  }
  __syncthreads();
  project((R*)a.g.psif);
  if (a.g.mode == 1) return;
#pragma unroll
  for (int i = 0; i < NS; ++i) O[i] = X[(i * NS + q) * 32];
  lift(Px, q, NS, M);
  sym2_force<N, false, C>(O, M, k4, F);
#pragma unroll
  for (int g = 0; g < ng; ++g) Fs[(q * ng + g) * 32] = F[g];
  __syncthreads();
  if (own)
    for (int g = q; g < ng; g += NS) {
      double f = 0.0;
#pragma unroll
      for (int j = 0; j < NS; ++j) f += Fs[(j * ng + g) * 32];
      const long long pi_ = p_index(L, ng, mu, g, s);
      if (a.g.mode == 0) {
        R* P = (R*)a.g.P;
        P[pi_] = (R)((C)P[pi_] - (C)a.g.eps * (C)f);
      } else {
        a.g.out[pi_] = f;
      }
    }
  sym2_rotate<N, true, true, C>(U, M, O);                 // psi_b = D^dag phi_x: columns, U^dag
#pragma unroll
  for (int i = 0; i < NS; ++i) X[(i * NS + q) * 32] = O[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NS; ++i) M[i] = X[(q * NS + i) * 32];   // rows, U^T
  sym2_rotate<N, true, false, C>(U, M, O);
#pragma unroll
  for (int i = 0; i < NS; ++i) X[(q * NS + i) * 32] = O[i];
  __syncthreads();
  project((R*)a.g.psib);
}

// ---------------------------------------------------------------------------
// Irreps that are N x N matrices, in registers, one thread per link.  With the map
// Phi = sum_b phi_b W_b of d components to N x N matrices (an isometry, d x N^2 entries):
//  ADJ false, two-slot irreps (n = 2: the symmetric and antisymmetric squares of V, e.g.
//   the SU(3) sextet {2} and antitriplet {1,1}), W the irrep basis with tensor index
//   i*N + j for the slots (i, j); the reference's tensor apply
//   (src/rep/rep_general.hpp:184-220: lift with W, U on each slot, project with W^H) is
//   Psi = U Phi U^T, and D^dag phi the same with U^dag Phi conj(U).  Every W_b is symmetric
//   or antisymmetric, so phi_x^dag T^a_R psi_f = Tr(Phi_x^dag (T^a Psi + Psi T^aT))
//   = 2 Tr(T^a Psi Phi_x^dag), and the matter force -kappa g^a, g^a = -2 Im(phi_x^dag
//   T^a_R D phi_{x+mu}) (src/rep/representation.hpp:36-46), is 4 kappa Im Tr(T^a Psi
//   Phi_x^dag): one N x N product and the projection the fundamental uses.
//  ADJ true, the one-fold adjoint product (SU(3) octet {2,1}, SU(2) {2}), W_b = sqrt 2
//   sum_a Q_ab T^a of the intertwiner Q: Psi = U Phi U^dag, D^dag the same with U^dag, and
//   T^a_R psi the commutator [T^a, Psi], so the force is 2 kappa Im Tr T^a (Psi Phi_x^dag
//   - Phi_x^dag Psi).
// RW: W is real (every basis that gh_rep_general_build makes), a multiply-add per part.
// psi_b then psi_f components leave by coalesced stores; modes and outputs as k_gen_links.
// Bound: FP pipe and the latency of one link's chain of products.  ADJ against the 8 x 8
// adjoint matrices in shared memory that it replaced (k_gen_prod), SU(3) octet 12^4 FP32:
// kick with it 62.4 -> 25.4 us (FP64 98.0 -> 35.8); RW on the sextet: FP64 kick 42.1 -> 31.9 us
// together with consecutive-site kick blocks.  5 FP32 blocks per SM (72 bytes spilled by the
// octet): 12^4 has 4.4 blocks per SM, and 4 resident took 29.1 us.
// ---------------------------------------------------------------------------
template <int N, bool RW, typename C, typename R>
__device__ __forceinline__ Mat<N, C> pair_lift(const typename V2<C>::t* Wt, int d, const R* phi, const LatDev& L, int s) {
  Mat<N, C> M;
  set_zero(M);
  for (int b = 0; b < d; ++b) {
    const cx<C> f = ldc<C>(phi, f_index(L, d, b, s));
#pragma unroll
    for (int t = 0; t < N * N; ++t) {
      const typename V2<C>::t v = __ldg(Wt + b * N * N + t);
      if (RW) {
        M.e[t].re = fmad(f.re, v.x, M.e[t].re);
        M.e[t].im = fmad(f.im, v.x, M.e[t].im);
      } else {
        M.e[t] = cfma(M.e[t], f, mk<C>(v.x, v.y));
      }
    }
  }
  return M;
}
template <int N, bool RW, typename C, typename R>
__device__ __forceinline__ void pair_project(const typename V2<C>::t* Wt, int d, const Mat<N, C>& M, R* out,
                                             const LatDev& L, int mu, int s) {
  for (int b = 0; b < d; ++b) {
    cx<C> z = zero<C>();
#pragma unroll
    for (int t = 0; t < N * N; ++t) {
      const typename V2<C>::t v = __ldg(Wt + b * N * N + t);
      if (RW) {
        z.re = fmad(M.e[t].re, v.x, z.re);
        z.im = fmad(M.e[t].im, v.x, z.im);
      } else {
        z = cfma(z, mk<C>(v.x, -v.y), M.e[t]);
      }
    }
    stc<C>(out, g_index(L, d, mu, b, s), z);
  }
}
template <int N, typename C> __device__ __forceinline__ Mat<N, C> conj_mat(const Mat<N, C>& A) {
  Mat<N, C> B;
#pragma unroll
  for (int i = 0; i < N * N; ++i) B.e[i] = conj(A.e[i]);
  return B;
}
template <int D, int N, typename R, bool ADJ, bool RW>
__global__ void __launch_bounds__(KBLOCK, sizeof(R) == 8 ? 3 : 5) k_gen_pair(const GenArgs a) {
  pdl_enter();
  typedef typename Cmp<R>::t C;
  const Work w = a.work[blockIdx.x];
  if ((int)threadIdx.x >= w.n) return;
  const LatDev& L = a.lats[w.lat];
  const int mu = w.mu, s = w.s0 + threadIdx.x;
  int x[D];
  coords<D>(L, s, x);
  if (!below_hi<D>(L, x)) return;                      // upper halo sites of a subdomain store nothing
  const int d = a.t.d;
  const typename V2<C>::t* Wt = reinterpret_cast<const typename V2<C>::t*>(
      sizeof(C) == sizeof(double) ? (const void*)a.t.w2_64 : (const void*)a.t.w2_32);
  const R* phi = (const R*)a.phi;
  const Mat<N, C> U = ld_link<N, C>((const R*)a.U, L, mu, s);
  const int spm = nfwd(L, s, x[mu], mu);
  // psi_f = D phi_{x+mu}: U Phi U^T = (U Phi) conj(U)^dag, or U Phi U^dag
  const Mat<N, C> Psi = mm_nd(mm(U, pair_lift<N, RW, C>(Wt, d, phi, L, spm)), ADJ ? U : conj_mat(U));
  pair_project<N, RW, C>(Wt, d, Psi, (R*)a.psif, L, mu, s);
  if (a.mode == 1) return;
  const Mat<N, C> Phx = pair_lift<N, RW, C>(Wt, d, phi, L, s);
  // psi_b = D^dag phi_x: U^dag Phi conj(U), or U^dag Phi U
  pair_project<N, RW, C>(Wt, d, mm(mm_dn(U, Phx), ADJ ? U : conj_mat(U)), (R*)a.psib, L, mu, s);
  if (!in_box<D>(L, x)) return;                        // momentum updates: interior links only
  // the commutator's terms cancel in part: in double, whatever the fields (FP32 octet force
  // against FP64: 6.99e-8 rms with it, 9.34e-8 in FP32, 9.06e-8 in k_gen_prod's double sums)
  typedef typename std::conditional<ADJ, double, C>::type S;
  constexpr int ng = N * N - 1;
  S F[ng];
  {
    Mat<N, S> Ps, Px;
#pragma unroll
    for (int i = 0; i < N * N; ++i) { Ps.e[i] = cvt<S>(Psi.e[i]); Px.e[i] = cvt<S>(Phx.e[i]); }
    Mat<N, S> M = mm_nd(Ps, Px);
    if (ADJ) {
      const Mat<N, S> M2 = mm_dn(Px, Ps);
#pragma unroll
      for (int i = 0; i < N * N; ++i) M.e[i] = sub(M.e[i], M2.e[i]);
    }
    const S kf = S(ADJ ? 2 : 4) * (S)L.kappa;
#pragma unroll
    for (int i = 0; i < N * N; ++i) M.e[i] = scale(M.e[i], kf);
    im_tr_proj<N, S>(M, F);
  }
  const long long pb = p_index(L, ng, mu, 0, s);
  if (a.mode == 0) {
    R* P = (R*)a.P;
    const C eps = (C)a.eps;
#pragma unroll
    for (int g = 0; g < ng; ++g) P[pb + g * ULANE] = (R)((C)P[pb + g * ULANE] - eps * (C)F[g]);
  } else {
#pragma unroll
    for (int g = 0; g < ng; ++g) a.out[pb + g * ULANE] = (double)F[g];
  }
}

// ---------------------------------------------------------------------------
// Drift: U <- exp(i eps P) U (src/hmc/gauge_higgs_hmc.hpp:136-143); site items:
// phi += eps pi (:145-146).  The link update (exponential, product with U,
// projection) runs in the arithmetic type A, whatever the storage type R:
//   FP64 mode       R = double, A = double, no projection (the reference's
//                   reunitarisation once per trajectory, k_reunit);
//   FP32-MD         R = float,  A = double: FP32 links and momenta are widened,
//                   exp(i eps P) (scaling, Cayley-Hamilton series), its product
//                   with U and the Gram-Schmidt projection back to SU(N) are
//                   FP64, the result is rounded to FP32 once;
//   FP32-MD, all    R = float,  A = float: the same steps in FP32 (non-default
//   FP32            variant, GH_PREC_FP32_ALL).
// ---------------------------------------------------------------------------
// Projection back to SU(N) after each FP32-MD drift: Gram-Schmidt on the first
// N-1 rows, the last row fixed by det = 1 (SU(2): (-conj u01, conj u00); SU(3):
// conj(row0 x row1)).  The trajectory-end reunitarisation of the FP64 mode keeps
// the reference's algorithm (k_reunit).
template <int N, typename T>
__device__ __forceinline__ void project_su(Mat<N, T>& U) {
  // rows stay within ~1e-6 of unit norm between projections: one Newton step of
  // 1/sqrt from 1 (x^-1/2 ~ (3 - x)/2) is exact to ~1e-12, a second to FP64 resolution
  T n0 = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) n0 += norm2(U.e[j]);
  T i0 = T(1.5) - T(0.5) * n0;
  i0 = i0 * (T(1.5) - T(0.5) * n0 * i0 * i0);
  if (fabs(n0 - T(1)) > T(1e-3)) i0 = rsqrt(n0);    // far from unitary (links set by the caller)
#pragma unroll
  for (int j = 0; j < N; ++j) U.e[j] = scale(U.e[j], i0);
  if (N == 2) {
    U.e[2] = mk<T>(-U.e[1].re, U.e[1].im);
    U.e[3] = mk<T>(U.e[0].re, -U.e[0].im);
    return;
  }
  cx<T> p = zero<T>();
#pragma unroll
  for (int j = 0; j < N; ++j) p = add(p, cmul(U.e[j], U.e[N + j]));
  T n1 = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) { U.e[N + j] = sub(U.e[N + j], mul(p, U.e[j])); n1 += norm2(U.e[N + j]); }
  T i1 = T(1.5) - T(0.5) * n1;
  i1 = i1 * (T(1.5) - T(0.5) * n1 * i1 * i1);
  if (fabs(n1 - T(1)) > T(1e-3)) i1 = rsqrt(n1);
#pragma unroll
  for (int j = 0; j < N; ++j) U.e[N + j] = scale(U.e[N + j], i1);
  if (N == 3) {
    U.e[6] = conj(sub(mul(U.e[1], U.e[5]), mul(U.e[2], U.e[4])));
    U.e[7] = conj(sub(mul(U.e[2], U.e[3]), mul(U.e[0], U.e[5])));
    U.e[8] = conj(sub(mul(U.e[0], U.e[4]), mul(U.e[1], U.e[3])));
  }
}

struct DriftArgs {
  const Work* work;
  const LatDev* lats;
  void* U;
  const void* P;
  void* phi;
  void* pi;
  double eps;
  int d;
  int frozen;          // |phi_x| = 1: geodesic (great-circle) drift of (phi, pi)
};
// PROJ: the link update is projected back to SU(N) (the FP32 modes' drift)
template <int N, typename R, typename A, bool PROJ>
__global__ void __launch_bounds__(KBLOCK) k_drift(const DriftArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  if ((int)threadIdx.x >= w.n) return;
  const LatDev L = a.lats[w.lat];
  const int s = w.s0 + threadIdx.x;
  if (!active_site(L, s)) return;
  if (w.mu >= 0) {
    const int mu = w.mu;
    constexpr int ng = N * N - 1;
    const R* P = (const R*)a.P;
    A v[ng];
    const long long pb = p_index(L, ng, mu, 0, s);
    const A eps = (A)a.eps;
#pragma unroll
    for (int g = 0; g < ng; ++g) v[g] = (A)P[pb + g * ULANE] * eps;   // eps P in algebra coefficients
    const Mat<N, A> E = expi<N>(alg_to_mat<N, A>(v));
    const Mat<N, A> Uo = ld_link_rw<N, A>((const R*)a.U, L, mu, s);
    Mat<N, A> Un;
    if constexpr (PROJ) {
      // the projection reads the first N-1 rows of E U and rebuilds the last, so the
      // last row of the product (and of E) is never formed
      mm_core<N, A, false, false, false, N - 1>(E, Uo, Un);
      project_su<N, A>(Un);
    } else {
      Un = mm(E, Uo);
    }
    st_link<N, A>((R*)a.U, L, mu, s, Un);
  } else if (a.frozen) {
    // Frozen length (src/hmc/gauge_higgs_hmc.hpp:84-102): the exact constrained free
    // flow on the unit sphere, r = |pi|:
    //   phi' = cos(r eps) phi + sin(r eps) pi / r,  pi' = -r sin(r eps) phi + cos(r eps) pi.
    // FP64 arithmetic in both precisions; FP32 fields are put back on the sphere
    // (phi' / |phi'|) before they are stored, so that FP32 rounding does not let
    // |phi| wander over many steps.
    R* phi = (R*)a.phi;
    R* pi = (R*)a.pi;
    double r2 = 0.0;
    for (int k = 0; k < a.d; ++k) r2 += norm2(ldc_rw<double>(pi, f_index(L, a.d, k, s)));
    const double r = sqrt(r2);
    if (r < 1e-300) return;
    double sn, c;
    sincos(r * a.eps, &sn, &c);
    const double sr = sn / r, rs = -r * sn;
    double inv = 1.0;
    if (sizeof(R) != sizeof(double)) {
      double n2 = 0.0;
      for (int k = 0; k < a.d; ++k) {
        const long long i = f_index(L, a.d, k, s);
        n2 += norm2(add(scale(ldc_rw<double>(phi, i), c), scale(ldc_rw<double>(pi, i), sr)));
      }
      inv = 1.0 / sqrt(n2);
    }
    for (int k = 0; k < a.d; ++k) {
      const long long i = f_index(L, a.d, k, s);
      const cx<double> f = ldc_rw<double>(phi, i), p = ldc_rw<double>(pi, i);
      stc<double>(phi, i, scale(add(scale(f, c), scale(p, sr)), inv));
      stc<double>(pi, i, add(scale(f, rs), scale(p, c)));
    }
  } else {
    typedef typename Cmp<R>::t C;
    R* phi = (R*)a.phi;
    const R* pi = (const R*)a.pi;
    for (int k = 0; k < a.d; ++k) {
      const long long i = f_index(L, a.d, k, s);
      stc<C>(phi, i, add(ldc_rw<C>(phi, i), scale(ldc<C>(pi, i), (C)a.eps)));
    }
  }
}

// ---------------------------------------------------------------------------
// Frozen-length scalar helpers, one thread per site (src/hmc/gauge_higgs_hmc.hpp:61-82):
//   what 0: pi <- pi - Re(phi^dag pi) phi   (momentum onto the sphere's tangent space)
//   what 1: phi <- phi / |phi|              (put the field on the unit sphere)
// FP64 arithmetic in both precisions.
// ---------------------------------------------------------------------------
struct SphereArgs { const Work* work; const LatDev* lats; void* phi; void* pi; int d; int what; };
template <typename R>
__global__ void __launch_bounds__(KBLOCK) k_sphere(const SphereArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  if ((int)threadIdx.x >= w.n) return;
  const LatDev& L = a.lats[w.lat];
  const int s = w.s0 + threadIdx.x;
  if (!active_site(L, s)) return;
  R* phi = (R*)a.phi;
  R* pi = (R*)a.pi;
  if (a.what == 0) {
    double rp = 0.0;
    for (int k = 0; k < a.d; ++k) {
      const long long i = f_index(L, a.d, k, s);
      const cx<double> f = ldc_rw<double>(phi, i), p = ldc_rw<double>(pi, i);
      rp += f.re * p.re + f.im * p.im;
    }
    for (int k = 0; k < a.d; ++k) {
      const long long i = f_index(L, a.d, k, s);
      stc<double>(pi, i, sub(ldc_rw<double>(pi, i), scale(ldc_rw<double>(phi, i), rp)));
    }
  } else {
    double n2 = 0.0;
    for (int k = 0; k < a.d; ++k) n2 += norm2(ldc_rw<double>(phi, f_index(L, a.d, k, s)));
    if (!(n2 > 0.0)) return;
    const double inv = 1.0 / sqrt(n2);
    for (int k = 0; k < a.d; ++k) {
      const long long i = f_index(L, a.d, k, s);
      stc<double>(phi, i, scale(ldc_rw<double>(phi, i), inv));
    }
  }
}

// Reunitarise all links (src/core/fields.hpp:36, src/group/sun.hpp:48-71), FP64.
struct LinkArgs { const Work* work; const LatDev* lats; void* U; const void* Us; };
template <int N, typename R>
__global__ void __launch_bounds__(KBLOCK) k_reunit(const LinkArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  if ((int)threadIdx.x >= w.n || w.mu < 0) return;
  const LatDev L = a.lats[w.lat];
  const int s = w.s0 + threadIdx.x;
  if (!active_site(L, s)) return;
  Mat<N, double> M = ld_link_rw<N, double>((const R*)a.U, L, w.mu, s);
  reunitarize<N, double>(M);
  st_link<N, double>((R*)a.U, L, w.mu, s, M);
}

// ---------------------------------------------------------------------------
// Measure: one pass over sites producing the six per-site sums behind
// H = 1/2 sum P^2 + 1/2 sum |pi|^2 + S_g + S_H (src/hmc/gauge_higgs_hmc.hpp:105-110)
// and the observables plaquette, L_link, L_phi (src/action/gauge_wilson.hpp:31-65,
// src/action/scalar_higgs.hpp:43-65,132-154), all accumulated in FP64:
//   r0 sum_{mu<nu} Re Tr U_pl   r1 sum V(phi)   r2 sum_mu Re phi_x^dag D phi_{x+mu}
//   r3 sum P^2                  r4 sum |pi|^2   r5 sum |phi|^2
// Warp-shuffle tree reduction, then one partial per block (deterministic order).
// ---------------------------------------------------------------------------
struct MeasArgs {
  const Work* work;
  const LatDev* lats;
  const void* U;
  const void* P;
  const void* phi;
  const void* pi;
  const void* psif;
  int pot;
  double mu2;
  PotA sa;               // multi-invariant potential superoperator (FP64 values)
  const double2* wpot;   // general irreps: w = A(M) phi per site, written by k_gen_links
  int d;
  int scalar;
  double* partials;   // [block][NRED]
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

template <int D, int N, typename R, int REP>
__global__ void __launch_bounds__(KBLOCK) k_measure(const MeasArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  double r[NRED] = {0, 0, 0, 0, 0, 0};
  if ((int)threadIdx.x < w.n && active_site(a.lats[w.lat], w.s0 + (int)threadIdx.x)) {
    const LatDev L = a.lats[w.lat];
    const int s = w.s0 + threadIdx.x;
    const R* U = (const R*)a.U;
    int x[D];
    coords<D>(L, s, x);
    // plaquettes: Re Tr(U_mu(x) U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag) = Re Tr(A B^dag)
#pragma unroll
    for (int mu = 0; mu < D; ++mu) {
      const int spm = nfwd(L, s, x[mu], mu);
      const Mat<N, double> Umu = ld_link<N, double>(U, L, mu, s);
#pragma unroll
      for (int nu = mu + 1; nu < D; ++nu) {
        const int spn = nfwd(L, s, x[nu], nu);
        const Mat<N, double> A = mm(Umu, ld_link<N, double>(U, L, nu, spm));
        const Mat<N, double> B = mm(ld_link<N, double>(U, L, nu, s), ld_link<N, double>(U, L, mu, spn));
        r[0] += retr_nd(A, B);
      }
    }
    constexpr int ng = N * N - 1;
    const R* P = (const R*)a.P;
#pragma unroll
    for (int mu = 0; mu < D; ++mu)
#pragma unroll
      for (int g = 0; g < ng; ++g) {
        const double p = (double)P[p_index(L, ng, mu, g, s)];
        r[3] += p * p;
      }
    if (a.scalar) {
      const R* phi = (const R*)a.phi;
      const R* pi = (const R*)a.pi;
      double n2 = 0.0;
      for (int k = 0; k < a.d; ++k) {
        n2 += norm2(ldc<double>(phi, f_index(L, a.d, k, s)));
        r[4] += norm2(ldc<double>(pi, f_index(L, a.d, k, s)));
      }
      r[5] = n2;
      if (a.pot != POT_MULTI) {
        r[1] = n2 + L.lambda * (n2 - 1.0) * (n2 - 1.0);
      } else if (REP == REP_GEN) {         // V = -mu2 phi^dag phi + Re(phi^dag w) / 2, w from k_gen_links
        double re = 0.0;
        for (int k = 0; k < a.d; ++k) {
          const cx<double> pk = ldc<double>(phi, f_index(L, a.d, k, s));
          const double2 wk = a.wpot[f_index(L, a.d, k, s)];
          re = fmad(pk.re, wk.x, fmad(pk.im, wk.y, re));
        }
        r[1] = -a.mu2 * n2 + 0.5 * re;
      } else {
        r[1] = pot_multi<double, R>(phi, L, a.d, s, a.sa, a.mu2, nullptr);
      }
      if (REP == REP_FUND || REP == REP_ADJ) {
        constexpr int d = RepDim<N, REP>::d;
        cx<double> px[d], py[d], o[d];
#pragma unroll
        for (int k = 0; k < d; ++k) px[k] = ldc<double>(phi, f_index(L, d, k, s));
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
          const int y = nfwd(L, s, x[mu], mu);
#pragma unroll
          for (int k = 0; k < d; ++k) py[k] = ldc<double>(phi, f_index(L, d, k, y));
          const Mat<N, double> Umu = ld_link<N, double>(U, L, mu, s);
          if (REP == REP_FUND) fund_apply<N, double>(Umu, py, o, false); else adj_apply<N, double>(Umu, py, o, false);
          double h = 0.0;
#pragma unroll
          for (int k = 0; k < d; ++k) h += px[k].re * o[k].re + px[k].im * o[k].im;
          r[2] += h;
        }
      } else if (REP == REP_GEN) {
        const R* psif = (const R*)a.psif;
#pragma unroll
        for (int mu = 0; mu < D; ++mu) {
          double h = 0.0;
          for (int k = 0; k < a.d; ++k) {
            const cx<double> p = ldc<double>(phi, f_index(L, a.d, k, s));
            const cx<double> o = ldc<double>(psif, g_index(L, a.d, mu, k, s));
            h += p.re * o.re + p.im * o.im;
          }
          r[2] += h;
        }
      }
    }
  }
  __shared__ double red[KBLOCK / 32][NRED];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NRED; ++k) {
    const double v = warp_sum(r[k]);
    if (lane == 0) red[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < NRED) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < KBLOCK / 32; ++q) v += red[q][threadIdx.x];
    a.partials[(size_t)blockIdx.x * NRED + threadIdx.x] = v;
  }
}

// Per-lattice totals of the measure partials and the derived quantities.
// res[l][slot][k]: 0 H, 1 S_g, 2 S_H, 3 kin_P, 4 kin_pi, 5 plaquette, 6 L_link, 7 L_phi
constexpr int NRES = 8;
struct FinArgs {
  const LatDev* lats;
  const int* blk_first;   // [nlat+1] block range of each lattice in the measure launch
  const double* partials;
  double* res;
  int slot;               // 0 or 1 (initial / final configuration)
  int D, N;
  int scalar;
};
static __global__ void k_finalize(const FinArgs a) {
  pdl_enter();
  const int l = blockIdx.x;
  const int b0 = a.blk_first[l], b1 = a.blk_first[l + 1];
  __shared__ double sh[NRED][32];
  double v[NRED] = {0, 0, 0, 0, 0, 0};
  for (int b = b0 + (int)threadIdx.x; b < b1; b += 32)
#pragma unroll
    for (int k = 0; k < NRED; ++k) v[k] += a.partials[(size_t)b * NRED + k];
#pragma unroll
  for (int k = 0; k < NRED; ++k) sh[k][threadIdx.x] = v[k];
  __syncwarp();
  if (threadIdx.x == 0) {
    double t[NRED];
#pragma unroll
    for (int k = 0; k < NRED; ++k) { t[k] = 0.0; for (int q = 0; q < 32; ++q) t[k] += sh[k][q]; }
    const LatDev L = a.lats[l];
    const double Vd = (double)L.Vi;              // active sites (all of a lattice that is not decomposed)
    const double nplaq = Vd * (a.D * (a.D - 1) / 2);
    const double Sg = (L.beta / a.N) * ((double)a.N * nplaq - t[0]);
    const double SH = a.scalar ? (t[1] - 2.0 * L.kappa * t[2]) : 0.0;
    const double kP = 0.5 * t[3], kpi = 0.5 * t[4];
    double* o = a.res + ((size_t)l * 2 + a.slot) * NRES;
    o[0] = kP + kpi + Sg + SH;
    o[1] = Sg;
    o[2] = SH;
    o[3] = kP;
    o[4] = kpi;
    o[5] = t[0] / ((double)a.N * nplaq);
    o[6] = a.scalar ? t[2] / (Vd * a.D) : 0.0;
    o[7] = a.scalar ? t[5] / Vd : 0.0;
  }
}

// ---------------------------------------------------------------------------
// Metropolis (src/hmc/gauge_higgs_hmc.hpp:183-191, src/hmc/hmc.hpp:280-287): one
// thread per lattice; dH from the two measure slots, ++traj, coin
// uniform(key(0xE5 | 0xB2, traj)); NaN/Inf dH rejects (as in the reference,
// where every comparison with NaN is false) and is counted.  Appends a record.
// ---------------------------------------------------------------------------
struct TrajRec { double dH; int accepted; int traj; double plaq, L_phi, L_link, kappa, beta; };
struct MetroArgs { LatDev* lats; const double* res; TrajRec* hist; TrajRec* last; int hist_cap; int nlat; int pure; };
static __global__ void k_metropolis(const MetroArgs a) {
  pdl_enter();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= a.nlat) return;
  LatDev& L = a.lats[l];
  const double* r0 = a.res + (size_t)l * 2 * NRES;
  const double* r1 = r0 + NRES;
  const double dH = r1[0] - r0[0];
  L.traj += 1;
  const double u = ghrng::uniform(L.seed, ghrng::key(a.pure ? 0xB2 : 0xE5, L.traj));
  const bool finite = isfinite(dH);
  const int acc = (dH <= 0.0) || (u < exp(-dH));
  if (!finite) L.nonfinite += 1;
  L.last_acc = acc;
  L.accepted += acc;
  if (a.hist && a.hist_cap > 0) {
    TrajRec& h = a.hist[(size_t)l * a.hist_cap + (int)((L.traj - 1) % (unsigned long long)a.hist_cap)];
    const double* ro = acc ? r1 : r0;
    h.dH = dH;
    h.accepted = acc;
    h.traj = (int)L.traj;
    h.plaq = ro[5];
    h.L_phi = ro[7];
    h.L_link = ro[6];
    h.kappa = L.kappa;
    h.beta = L.beta;
    a.last[l] = h;
  }
}

// Restore the saved configuration of lattices whose trajectory was rejected.
struct RestoreArgs { const Work* work; const LatDev* lats; void* U; const void* Us; void* phi; const void* phis; int N; int d; };
template <typename R>
__global__ void __launch_bounds__(KBLOCK) k_restore(const RestoreArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  if ((int)threadIdx.x >= w.n) return;
  const LatDev& L = a.lats[w.lat];
  if (L.last_acc) return;
  const int s = w.s0 + threadIdx.x;
  typedef typename V2<R>::t V;
  if (w.mu >= 0) {
    const int NN = a.N * a.N;
    const long long b = u_index(L, NN, w.mu, 0, s);
    for (int c = 0; c < NN; ++c) reinterpret_cast<V*>(a.U)[b + c * ULANE] = reinterpret_cast<const V*>(a.Us)[b + c * ULANE];
  } else {
    for (int k = 0; k < a.d; ++k) {
      const long long i = f_index(L, a.d, k, s);
      reinterpret_cast<V*>(a.phi)[i] = reinterpret_cast<const V*>(a.phis)[i];
    }
  }
}

// ---------------------------------------------------------------------------
// Halo planes of a subdomain (src/mpi/gauge_mpi.hpp:101-139): gather (pack) or scatter
// (unpack) every site of the local lattice with x_nu = layer, all components of the
// links (kind 0: D N^2 complex per site) or of phi (kind 1: d complex per site), to or
// from a contiguous buffer [component][plane site], the plane's sites in mixed radix
// over the other directions, direction 0 fastest.  Whole planes, halo sites of the other
// directions included, so that exchanging the split directions one after the other
// also fills the edges and corners, as the reference's sequential exchange does.
// ---------------------------------------------------------------------------
struct HaloArgs {
  const LatDev* lats;
  int lat;
  void* f;              // the field (U or phi)
  void* buf;            // device buffer, ncomp * nplane complex R
  int kind, nu, layer, unpack, D, nn, d;
  long long nplane;
  int ncomp;
};
template <typename R>
__global__ void __launch_bounds__(256) k_halo(const HaloArgs a) {
  typedef typename V2<R>::t V;
  const LatDev& L = a.lats[a.lat];
  const long long total = a.nplane * a.ncomp;
  V* f = reinterpret_cast<V*>(a.f);
  V* b = reinterpret_cast<V*>(a.buf);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int comp = (int)(i / a.nplane);
    long long r = i - (long long)comp * a.nplane;
    int s = a.layer * L.stride[a.nu];
    for (int mu = 0; mu < a.D; ++mu) {
      if (mu == a.nu) continue;
      s += (int)(r % L.L[mu]) * L.stride[mu];
      r /= L.L[mu];
    }
    const long long e = a.kind == 0 ? u_index(L, a.nn, comp / a.nn, comp % a.nn, s) : f_index(L, a.d, comp, s);
    if (a.unpack) f[e] = b[i];
    else b[i] = f[e];
  }
}

// ---------------------------------------------------------------------------
// Counter-RNG field initialisation (bit-exact keys of the reference):
//   hot start  U = expi(alg_to_mat(sigma * gauss(key(1, s, mu, a))))  src/core/fields.hpp:25-34
//   momenta    P^a = gauss(key(stream, s, mu, a))                       src/core/fields.hpp:59-66
//   vectors    re = sigma gauss(key(stream, s, 2k)), im = sigma gauss(key(stream, s, 2k+1)) or 0
//                                                                       src/core/scalar_field.hpp:40-50
//   refresh streams key(0xC3|0xA1, traj) and key(0xD4, traj)           src/hmc/gauge_higgs_hmc.hpp:167-173
// ---------------------------------------------------------------------------
struct InitArgs {
  const Work* work;
  const LatDev* lats;
  void* U;
  void* P;
  void* vec;          // phi or pi
  int what;           // 0 hot start, 1 momentum refresh (trajectory keys), 2 vector gaussian
                      // 3 momentum with explicit stream, 4 cold links, 5 cold vector
  int pure;           // pure gauge keys (0xA1) for what == 1
  int real;
  int d;
  double sigma;
  unsigned long long stream;
  void* Us;           // what == 1: also save U and phi here (the trajectory's reject copy); null: no
  const void* phi;
  void* phis;
};
// components c0, c0 + cs, ... of the `nc` of a site or link, saved at the same place
template <typename V>
__device__ __forceinline__ void save_components(const void* from, void* to, long long first, int nc, int c0, int cs) {
  for (int c = c0; c < nc; c += cs) reinterpret_cast<V*>(to)[first + c * ULANE] = reinterpret_cast<const V*>(from)[first + c * ULANE];
}
// Gaussian draw for a field stored as R: the correctly rounded draw for FP64
// fields, the CUDA-libm draw for FP32 fields (identical after rounding to FP32
// but for ~1e-8 of draws).
template <typename R> __device__ __forceinline__ double gauss_r(uint64_t seed, uint64_t k) {
  return sizeof(R) == sizeof(double) ? ghrng::gauss(seed, k) : ghrng::gauss_md(seed, k);
}

// SPLIT (Gaussian draws): four blocks per item, a lane per site and the components of a
// link or vector split over the warps.  A thread that draws all of them in turn is a chain
// of 8 (links) to 2 d draws, which a launch of few blocks waits for; beyond
// INIT_SPLIT_BLOCKS items the chains of other threads hide it, and the key's common part
// would be hashed by four threads.  Refresh in us, whole and split: 6^4 SU(2) FP64 9.0 and 7.2,
// SU(3) 9^3 x 12 adjoint 22.3 and 14.9, 12^4 sextet 40.9 and 33.0, 27-plet 75.8 and 44.9, SU(2)
// {12} 8^4 37.1 and 15.5.
constexpr int INIT_SPLIT_BLOCKS = 148 * 6;   // one wave of whole items at 80 registers
constexpr int INIT_SPLIT_D = 9;              // from this many vector components on in any launch
template <int N, typename R, bool SPLIT>
__global__ void __launch_bounds__(KBLOCK) k_init(const InitArgs a) {
  pdl_enter();
  typedef typename Cmp<R>::t C;
  static_assert(KBLOCK == 4 * ULANE, "a split item is four blocks of 32 sites");
  const Work w = a.work[SPLIT ? blockIdx.x >> 2 : blockIdx.x];
  const int i = SPLIT ? (int)(blockIdx.x & 3) * ULANE + (int)(threadIdx.x & (ULANE - 1)) : (int)threadIdx.x;
  if (i >= w.n) return;
  const LatDev L = a.lats[w.lat];
  const int s = w.s0 + i;
  // this thread's components: c0, c0 + cs, ...
  const int c0 = SPLIT ? (int)threadIdx.x / ULANE : 0;
  constexpr int cs = SPLIT ? 4 : 1;
  if (a.what == 1 && a.Us) {
    if (w.mu >= 0) save_components<typename V2<R>::t>(a.U, a.Us, u_index(L, N * N, w.mu, 0, s), N * N, c0, cs);
    else save_components<typename V2<R>::t>(a.phi, a.phis, f_index(L, a.d, 0, s), a.d, c0, cs);
  }
  if (!active_site(L, s)) return;                 // halo sites come from the neighbours
  const long long gs = global_site(L, s);         // the RNG key's site
  constexpr int ng = N * N - 1;
  if (w.mu >= 0) {
    const int mu = w.mu;
    if (a.what == 0 || a.what == 4) {
      Mat<N, double> M;
      if (a.what == 0) {
        double v[ng];
#pragma unroll
        for (int g = 0; g < ng; ++g) v[g] = a.sigma * ghrng::gauss(L.seed, ghrng::key(1, gs, mu, g));
        M = expi<N>(alg_to_mat<N, double>(v));
      } else {
        set_ident(M);
      }
      st_link<N, double>((R*)a.U, L, mu, s, M);
    } else if (a.what == 1 || a.what == 3) {
      const unsigned long long st = (a.what == 1) ? ghrng::key(a.pure ? 0xA1 : 0xC3, L.traj) : a.stream;
      R* P = (R*)a.P;
      const long long pb = p_index(L, ng, mu, 0, s);
#pragma unroll
      for (int q = 0; q < (ng + cs - 1) / cs; ++q) {
        const int g = c0 + q * cs;
        if (g < ng) P[pb + g * ULANE] = (R)gauss_r<R>(L.seed, ghrng::key(st, gs, mu, g));
      }
    }
    return;
  }
  // site items: vectors (pi on refresh, phi on gaussian / cold start)
  if (a.what == 1 && a.pure) return;
  if (a.what == 1 || a.what == 2) {
    const unsigned long long st = (a.what == 1) ? ghrng::key(0xD4, L.traj) : a.stream;
    const double sg = (a.what == 1) ? 1.0 : a.sigma;
    R* vec = (R*)a.vec;
    for (int k = c0; k < a.d; k += cs) {
      const double re = sg * gauss_r<R>(L.seed, ghrng::key(st, gs, 2 * k));
      const double im = a.real ? 0.0 : sg * gauss_r<R>(L.seed, ghrng::key(st, gs, 2 * k + 1));
      stc<double>(vec, f_index(L, a.d, k, s), mk<double>(re, im));
    }
  } else if (a.what == 5) {
    R* vec = (R*)a.vec;
    for (int k = 0; k < a.d; ++k) stc<double>(vec, f_index(L, a.d, k, s), mk<double>(k == 0 ? a.sigma : 0.0, 0.0));
  }
}

// ---------------------------------------------------------------------------
// Polyakov loop (src/measure/observables.hpp:17-34): one thread per site with
// x_t = 0, product of the L_t links in direction t, FP64.
// ---------------------------------------------------------------------------
struct PolyArgs { const Work* work; const LatDev* lats; const void* U; int tdir; double* partials; };
template <int D, int N, typename R>
__global__ void __launch_bounds__(KBLOCK) k_polyakov(const PolyArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  double v = 0.0;
  if ((int)threadIdx.x < w.n) {
    const LatDev L = a.lats[w.lat];
    const int s = w.s0 + threadIdx.x;
    int x[D];
    coords<D>(L, s, x);
    if (x[a.tdir] == 0) {
      const int t = a.tdir;
      Mat<N, double> P = ld_link<N, double>((const R*)a.U, L, t, s);
      int cur = s, xt = 0;
      for (int k = 1; k < L.L[t]; ++k) {
        cur = nfwd(L, cur, xt, t);
        ++xt;
        P = mm(P, ld_link<N, double>((const R*)a.U, L, t, cur));
      }
      for (int i = 0; i < N; ++i) v += P.e[i * N + i].re;
    }
  }
  __shared__ double red[KBLOCK / 32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < KBLOCK / 32; ++q) t += red[q];
    a.partials[blockIdx.x] = t;
  }
}

// ---------------------------------------------------------------------------
// Loops traced in a probe irrep (src/measure/observables.hpp:36-101).
// Re chi_lambda(W) for an SU(N) matrix W and Young rows lambda (m rows): the Schur
// polynomial of W's eigenvalues by Jacobi-Trudi, s_lambda = det[h_{lambda_i - i + j}],
// with the complete symmetric polynomials h_k from the power sums p_k = Tr W^k by
// Newton's identities, k h_k = sum_{i=1}^{k} p_i h_{k-i}.  This is Tr D^(lambda)(W),
// the trace of the representation matrix, without forming it.
// ---------------------------------------------------------------------------
constexpr int CHAR_KMAX = 24;     // largest h index lambda_1 + m - 1
constexpr int CHAR_MMAX = 4;      // most Young rows

template <int N>
__device__ double re_character(const Mat<N, double>& W, const int* lam, int m) {
  const int K = lam[0] + m - 1;
  cx<double> p[CHAR_KMAX + 1], h[CHAR_KMAX + 1];
  Mat<N, double> Wk = W;
  for (int k = 1; k <= K; ++k) {
    if (k > 1) Wk = mm(Wk, W);
    cx<double> t = zero<double>();
    for (int i = 0; i < N; ++i) t = add(t, Wk.e[i * N + i]);
    p[k] = t;
  }
  h[0] = mk<double>(1.0, 0.0);
  for (int k = 1; k <= K; ++k) {
    cx<double> t = zero<double>();
    for (int i = 1; i <= k; ++i) t = cfma(t, p[i], h[k - i]);
    h[k] = scale(t, 1.0 / k);
  }
  cx<double> M[CHAR_MMAX * CHAR_MMAX];
  for (int i = 0; i < m; ++i)
    for (int j = 0; j < m; ++j) {
      const int k = lam[i] - i + j;
      M[i * m + j] = (k < 0) ? zero<double>() : h[k];
    }
  // determinant by elimination with partial pivoting (m <= 4)
  cx<double> det = mk<double>(1.0, 0.0);
  for (int c = 0; c < m; ++c) {
    int piv = c;
    for (int r = c + 1; r < m; ++r)
      if (norm2(M[r * m + c]) > norm2(M[piv * m + c])) piv = r;
    if (norm2(M[piv * m + c]) == 0.0) return 0.0;
    if (piv != c) {
      for (int j = 0; j < m; ++j) { const cx<double> t = M[c * m + j]; M[c * m + j] = M[piv * m + j]; M[piv * m + j] = t; }
      det = scale(det, -1.0);
    }
    det = mul(det, M[c * m + c]);
    const cx<double> inv = scale(conj(M[c * m + c]), 1.0 / norm2(M[c * m + c]));
    for (int r = c + 1; r < m; ++r) {
      const cx<double> f = mul(M[r * m + c], inv);
      for (int j = c; j < m; ++j) M[r * m + j] = sub(M[r * m + j], mul(f, M[c * m + j]));
    }
  }
  return det.re;
}

// mode 0: Polyakov line in direction tdir from every site with x_tdir = 0;
// mode 1: the Ra x Rb rectangle of every plane mu < nu based at every site
//         (path order of wilson_rect, src/measure/observables.hpp:36-46).
// Per block: sum over its sites of Re chi(loop), into partials (FP64).
struct LoopArgs {
  const Work* work; const LatDev* lats; const void* U; double* partials;
  int mode, tdir, Ra, Rb, m; int lam[CHAR_MMAX];
};
template <int D, int N, typename R>
__global__ void __launch_bounds__(KBLOCK) k_loops(const LoopArgs a) {
  pdl_enter();
  const Work w = a.work[blockIdx.x];
  double v = 0.0;
  if ((int)threadIdx.x < w.n) {
    const LatDev L = a.lats[w.lat];
    const int s = w.s0 + threadIdx.x;
    const R* U = (const R*)a.U;
    int x0[D];
    coords<D>(L, s, x0);
    if (a.mode == 0) {
      if (x0[a.tdir] == 0) {
        const int t = a.tdir;
        Mat<N, double> P = ld_link<N, double>(U, L, t, s);
        int cur = s, xt = 0;
        for (int k = 1; k < L.L[t]; ++k) {
          cur = nfwd(L, cur, xt, t);
          ++xt;
          P = mm(P, ld_link<N, double>(U, L, t, cur));
        }
        v = re_character<N>(P, a.lam, a.m);
      }
    } else {
      for (int mu = 0; mu < D; ++mu)
        for (int nu = mu + 1; nu < D; ++nu) {
          int x[D];
          for (int q = 0; q < D; ++q) x[q] = x0[q];
          int c = s;
          Mat<N, double> W = ld_link<N, double>(U, L, mu, c);
          c = nfwd(L, c, x[mu], mu); x[mu] = (x[mu] + 1 == L.L[mu]) ? 0 : x[mu] + 1;
          for (int i = 1; i < a.Ra; ++i) {
            W = mm(W, ld_link<N, double>(U, L, mu, c));
            c = nfwd(L, c, x[mu], mu); x[mu] = (x[mu] + 1 == L.L[mu]) ? 0 : x[mu] + 1;
          }
          for (int j = 0; j < a.Rb; ++j) {
            W = mm(W, ld_link<N, double>(U, L, nu, c));
            c = nfwd(L, c, x[nu], nu); x[nu] = (x[nu] + 1 == L.L[nu]) ? 0 : x[nu] + 1;
          }
          for (int i = 0; i < a.Ra; ++i) {
            c = nbwd(L, c, x[mu], mu); x[mu] = (x[mu] == 0) ? L.L[mu] - 1 : x[mu] - 1;
            W = mm_nd(W, ld_link<N, double>(U, L, mu, c));
          }
          for (int j = 0; j < a.Rb; ++j) {
            c = nbwd(L, c, x[nu], nu); x[nu] = (x[nu] == 0) ? L.L[nu] - 1 : x[nu] - 1;
            W = mm_nd(W, ld_link<N, double>(U, L, nu, c));
          }
          v += re_character<N>(W, a.lam, a.m);
        }
    }
  }
  __shared__ double red[KBLOCK / 32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < KBLOCK / 32; ++q) t += red[q];
    a.partials[blockIdx.x] = t;
  }
}

// ---------------------------------------------------------------------------
// Layout conversion between the reference's AoS host arrays (FP64) and the
// device SoA planes (R).  kind: 0 links (N*N complex per (site,mu)),
// 1 momenta (ng reals per (site,mu)), 2 vectors (d complex per site).
// ---------------------------------------------------------------------------
struct XferArgs { const LatDev* lats; int lat; int kind; int D; int ncomp; double* host_aos; void* dev; int to_dev; };
template <typename R>
__global__ void k_xfer(const XferArgs a) {
  pdl_enter();
  const LatDev L = a.lats[a.lat];
  const long long per_site = (a.kind == 2) ? a.ncomp : (long long)a.D * a.ncomp;
  const long long total = (long long)L.V * per_site;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int s = (int)(e / per_site);
    const int r = (int)(e % per_site);
    if (a.kind == 1) {
      const long long di = p_index(L, a.ncomp, r / a.ncomp, r % a.ncomp, s);   // r = mu*ng + g
      R* P = (R*)a.dev;
      if (a.to_dev) P[di] = (R)a.host_aos[e]; else a.host_aos[e] = (double)P[di];
    } else {
      // r = mu*NN + c (links) or k (vectors)
      const long long di = (a.kind == 0) ? u_index(L, a.ncomp, r / a.ncomp, r % a.ncomp, s) : f_index(L, a.ncomp, r, s);
      if (a.to_dev) stc<double>((R*)a.dev, di, mk<double>(a.host_aos[2 * e], a.host_aos[2 * e + 1]));
      else { const cx<double> z = ldc_rw<double>((const R*)a.dev, di); a.host_aos[2 * e] = z.re; a.host_aos[2 * e + 1] = z.im; }
    }
  }
}

}  // namespace ghk
