// lbm_adjoint.cu -- reverse-mode (adjoint) kernels of one time step (sm_100a).
//
// The forward level n (the step kernel) maps, node by node,
//   f*(n) --pull + BC--> F(n) --> rho, u_pred, G (SPM, last disk wins),
//   u = u_pred + G/2, FORCE(n) = sum rho*phi*(u_pred - u_p)     C1:546-570
//   f*(n+1) = M^-1 [m - S(m - m_eq) + (1 - S/2) m_F]             C1:875-1048
//   omega(n+1) = 1/(3 nu_A/rho + 1/2), nu_A Papanastasiou        C6:903-958
// and the particle kernel of step n+1 maps (records n, FORCE(n)) to records
// n+1 (C1:247-259, C6:300-312).  The kernels below run the transposed
// Jacobians of those maps, level by level from the last step back to the
// first:
//   k_adj_lattice   one node per thread: gathers dJ/df*(n+1) from the adjoint
//                   field of level n+1 (a plain pull along +c_k), re-derives
//                   the forward intermediates from f*(n) and the records of
//                   step n, and writes its own entries of the adjoint field
//                   and dJ/domega(n); per-disk sums of dJ/d(x, y, u, v, w) go
//                   to FP64 accumulators, dJ/dnu and dJ/dtau_y to one FP64
//                   slot per block.
//   k_adj_particles one thread per disk: the transposed Newton-Euler update
//                   and repulsion (walls and pairs), the objective's own
//                   term, dJ/drho_p.
//   k_adj_levels    both, for many levels of a small lattice in one launch.
// The collision is differentiated in moment space: with the orthogonal D2Q9
// transform, M^-T = D^-1 M, D = diag(9, 36, 36, 6, 12, 6, 12, 4, 4), and the
// strain rate of C6:903-916 reduces to sums of S*m_neq moments,
//   D11 = kappa(-y1/4 - 3y7/4) + 3/4((s7-s1)G.u - 2 s7 Gx ux), y = S*m_neq,
// kappa = 36*d_mrt the scale of the reference's inverse transform.
// T = float: populations and node arithmetic in FP32 (the forward's shifted
// populations); reductions in FP64.  T = double: FP64 throughout.
#include <cuda_runtime.h>

#include <algorithm>

#include "lbm_lattice.cuh"

namespace lbm {

namespace {

__device__ __forceinline__ int cxk(int k) { return k == 1 || k == 5 || k == 8 ? 1 : (k == 3 || k == 6 || k == 7 ? -1 : 0); }
__device__ __forceinline__ int cyk(int k) { return k == 2 || k == 5 || k == 6 ? 1 : (k == 4 || k == 7 || k == 8 ? -1 : 0); }
__device__ __forceinline__ int oppk(int k) { return k == 0 ? 0 : (k < 5 ? ((k + 1) & 3) + 1 : ((k - 3) & 3) + 5); }

// Unknown k of node (i, j) that the boundary sets by half-way bounce-back
// from the node's own post-collision population opp(k): the corners (both
// boundary kinds, C1:1390-1414) and, for LBM_BC_HALFWAY_BB, the edges
// (C6:1206-1219, C6:1285-1294).
__device__ __forceinline__ bool bb_set(const Geometry& g, int bc, int k, int i, int j) {
  const bool L = i == 0, R = i == g.nx, B = j == 0, U = j == g.ny;
  if ((L || R) && (B || U)) {
    if (L && B) return k == 1 || k == 5 || k == 2;
    if (L && U) return k == 1 || k == 8 || k == 4;
    if (R && U) return k == 3 || k == 7 || k == 4;
    return k == 2 || k == 6 || k == 3;
  }
  if (bc != 1) return false;
  if (U) return k == 8 || k == 4 || k == 7;
  if (B) return k == 5 || k == 2 || k == 6;
  if (R) return k == 6 || k == 3 || k == 7;
  if (L) return k == 5 || k == 1 || k == 8;
  return false;
}

// The adjoint field holds, of each node, dJ/dr(k) of the raw pulled values --
// before the boundary routine: r(k) = F*(k, x - c_k) -- so the boundary
// routine is transposed in registers by the node that writes them, and what
// reads them is a plain pull along +c_k.  (The boundary's transpose in the
// gather instead, with its dependent loads at every node within two of a wall:
// k_adj_lattice at 401 x 1201 spilled at 64 registers, 62 against 55 us per
// step of the whole FP32 gradient, 129 against 93 FP64; in k_adj_levels the
// gather took 5400 to 11000 cycles of a level where this one takes 1700.)
// Where the source x - c_k lies
// outside, no neighbour reads entry k: it holds what the node's own F*(opp(k))
// gets from its own boundary values (the condition for that entry is the same,
// x + c_opp(k) outside).

// Entries of node (i, j) from its dJ/dF, in place.
//   Half-way bounce-back side: F(k) = F*(opp(k)) of the node, nothing changes.
//   Zou-He side with zero wall velocity (C1:1250-1258, C1:1341-1363): the
//   unknown opposite a k into the wall holds r(k); the inward diagonals take
//   half of the difference of the k along the wall; an unknown's own r(k) is
//   overwritten.
//   Corner (C1:1390-1414): bounce-back for the three in bb_set; the other two
//   whose source lies outside keep the node's own F*(k).
template <class T>
__device__ __forceinline__ void adj_boundary(const Geometry& g, int bc, int i, int j, T* a) {
  const bool L = i == 0, R = i == g.nx, B = j == 0, U = j == g.ny;
  if (!(L || R || B || U)) return;
  const bool corner = (L || R) && (B || U);
  if (bc == 1 && !corner) return;
  T s[9];
  s[0] = a[0];
#pragma unroll
  for (int k = 1; k < 9; ++k) {
    const int ko = oppk(k);
    if (corner) {
      const bool src = i - cxk(k) >= 0 && i - cxk(k) <= g.nx && j - cyk(k) >= 0 && j - cyk(k) <= g.ny;
      s[k] = src || bb_set(g, bc, k, i, j) ? a[k] : a[ko];
      continue;
    }
    // c_k along the side's outward normal
    const int out = L ? -cxk(k) : R ? cxk(k) : B ? -cyk(k) : cyk(k);
    s[k] = out < 0 ? (T)0 : out > 0 ? a[k] + a[ko] : a[k];
    if (k <= 4 && out == 0) {  // the inward diagonals with and against k
      const T with = k == 1 ? (U ? a[8] : a[5]) : k == 3 ? (U ? a[7] : a[6])
                   : k == 2 ? (L ? a[5] : a[6]) : (L ? a[8] : a[7]);
      const T against = k == 1 ? (U ? a[7] : a[6]) : k == 3 ? (U ? a[8] : a[5])
                      : k == 2 ? (L ? a[8] : a[7]) : (L ? a[5] : a[6]);
      s[k] += (T)0.5 * (against - with);
    }
  }
#pragma unroll
  for (int k = 1; k < 9; ++k) a[k] = s[k];
}

// dJ/df*(k) of node (i, j): the transpose of pull streaming + boundary.
template <class T, bool CG>
__device__ __forceinline__ void adj_gather(const T* __restrict__ A, const Geometry& g, int i,
                                           int j, T* a) {
  const long long n = (long long)j * g.pitch + i;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int xi = i + cxk(k), xj = j + cyk(k);
    const bool in = (cxk(k) == 0 || (cxk(k) < 0 ? xi >= 0 : xi <= g.nx)) &&
                    (cyk(k) == 0 || (cyk(k) < 0 ? xj >= 0 : xj <= g.ny));
    const long long here = plane_of(oppk(k)) * g.plane + n;
    const long long there = plane_of(k) * g.plane + n + cxk(k) + (long long)cyk(k) * g.pitch;
    a[k] = ld<CG>(A + (in ? there : here));
  }
}

// The D2Q9 moments of C6:878-886.
template <class T>
__device__ __forceinline__ void moments9(const T* f, T* m) {
  const T s14 = f[1] + f[2] + f[3] + f[4], s58 = f[5] + f[6] + f[7] + f[8];
  m[0] = f[0] + s14 + s58;
  m[1] = (T)-4 * f[0] - s14 + (T)2 * s58;
  m[2] = (T)4 * f[0] - (T)2 * s14 + s58;
  m[3] = f[1] - f[3] + f[5] - f[6] - f[7] + f[8];
  m[4] = (T)-2 * (f[1] - f[3]) + f[5] - f[6] - f[7] + f[8];
  m[5] = f[2] - f[4] + f[5] + f[6] - f[7] - f[8];
  m[6] = (T)-2 * (f[2] - f[4]) + f[5] + f[6] - f[7] - f[8];
  m[7] = f[1] - f[2] + f[3] - f[4];
  m[8] = f[5] - f[6] + f[7] - f[8];
}

// M^T a (the adjoint of m = M f).
template <class T>
__device__ __forceinline__ void moments9_t(const T* a, T* f) {
  const T c0 = a[0] - a[1] - (T)2 * a[2];
  const T d0 = a[0] + (T)2 * a[1] + a[2];
  f[0] = a[0] - (T)4 * a[1] + (T)4 * a[2];
  f[1] = c0 + a[3] - (T)2 * a[4] + a[7];
  f[2] = c0 + a[5] - (T)2 * a[6] - a[7];
  f[3] = c0 - a[3] + (T)2 * a[4] + a[7];
  f[4] = c0 - a[5] + (T)2 * a[6] - a[7];
  f[5] = d0 + a[3] + a[4] + a[5] + a[6] + a[8];
  f[6] = d0 - a[3] - a[4] + a[5] + a[6] - a[8];
  f[7] = d0 - a[3] - a[4] - a[5] - a[6] + a[8];
  f[8] = d0 + a[3] + a[4] - a[5] - a[6] - a[8];
}

__device__ __forceinline__ float tsqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double tsqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float texp(float x) { return expf(x); }
__device__ __forceinline__ double texp(double x) { return exp(x); }
__device__ __forceinline__ float tcos(float x) { return cosf(x); }
__device__ __forceinline__ double tcos(double x) { return cos(x); }
__device__ __forceinline__ float texpm1(float x) { return expm1f(x); }
__device__ __forceinline__ double texpm1(double x) { return expm1(x); }

// Taylor coefficients: g1 = (1 - e^-x)/x = sum_k (-1)^(k+1) x^(k-1)/k! and
// r = (1 - e^-x - x e^-x)/x^2 = sum_k (-1)^k (k-1) x^(k-2)/k!; 1/k! below.
#define LBM_IF(k) (1.0 / (k))
__device__ __forceinline__ double inv_fact(int k) {
  constexpr double F[15] = {1.0, 1.0, LBM_IF(2.0), LBM_IF(6.0), LBM_IF(24.0), LBM_IF(120.0),
                            LBM_IF(720.0), LBM_IF(5040.0), LBM_IF(40320.0), LBM_IF(362880.0),
                            LBM_IF(3628800.0), LBM_IF(39916800.0), LBM_IF(479001600.0),
                            LBM_IF(6227020800.0), LBM_IF(87178291200.0)};
  return F[k];
}
#undef LBM_IF
__device__ __forceinline__ double g1_coef(int k) { return (k % 2 ? 1.0 : -1.0) * inv_fact(k); }
__device__ __forceinline__ double r_coef(int k) { return (k % 2 ? -1.0 : 1.0) * (k - 1) * inv_fact(k); }

// g1 and r for x >= 0 without cancellation: the series below x = 0.1 (terms
// to x^7 in FP32, x^13 in FP64; the first omitted term is below the type's
// rounding), expm1 above.  The Papanastasiou viscosity is
// nu + tau_y m g1(m gamma) and its derivative in gamma -tau_y m^2 r(m gamma).
template <class T>
__device__ __forceinline__ void papanastasiou_terms(T x, T* g1, T* r) {
  constexpr int K = sizeof(T) == 8 ? 14 : 8;
  if (x < (T)0.1) {
    T sg = (T)g1_coef(K), sr = (T)r_coef(K);
#pragma unroll
    for (int k = K - 1; k >= 1; --k) sg = sg * x + (T)g1_coef(k);
#pragma unroll
    for (int k = K - 1; k >= 2; --k) sr = sr * x + (T)r_coef(k);
    *g1 = sg;
    *r = sr;
    return;
  }
  const T ix = (T)1 / x;
  const T em = -texpm1(-x);
  *g1 = em * ix;
  *r = (em - x * texp(-x)) * ix * ix;
}

template <class T>
__device__ __forceinline__ T phi_of(T di, T dj, T R, const Model& m) {
  if (sizeof(T) == 8) return (T)phi_double((double)di, (double)dj, (double)R, m.zeta, m.pi);
  return (T)phi_float((float)di, (float)dj, (float)R, m.zeta_f, m.pi_f);
}

// dphi/dD / r of the smoothed profile, D = R - r (0 outside the shell).
template <class T>
__device__ __forceinline__ T dphi_of(T di, T dj, T R, const Model& m) {
  const T r = tsqrt(di * di + dj * dj), D = R - r, zh = (T)(0.5 * m.zeta);
  if (!(D > -zh && D < zh && r > (T)0)) return (T)0;
  const T k = (T)(m.pi / m.zeta);
  return (T)0.5 * k * tcos(k * D) / r;
}

constexpr int ADJ_TPB = TPB;
// Blocks per SM that k_adj_lattice's registers allow, at 401 x 1201 (us per step
// of the whole gradient): FP32 1 / 3 / 4 / 5: 61.9 / 57.4 / 55.7 / 58; FP64
// 1 / 2 / 3: 116 / 92.3 / 93.4.
#ifndef LBM_ADJ_MINB_F32
#define LBM_ADJ_MINB_F32 4
#endif
#ifndef LBM_ADJ_MINB_F64
#define LBM_ADJ_MINB_F64 2
#endif
template <class T>
constexpr int ADJ_MINB = sizeof(T) == 4 ? LBM_ADJ_MINB_F32 : LBM_ADJ_MINB_F64;

// The fields one reverse level reads and writes.
template <class T>
struct AdjIO {
  const T* fs;     // f*(n)
  const T* oms;    // omega(n), Bingham
  const T* a_in;   // adjoint field of level n+1, null: zero
  const T* aw_in;  // dJ/domega(n+1)
  T* a_out;        // adjoint field of level n
  T* aw_out;       // dJ/domega(n), Bingham
  bool level0;     // the collision of step 1 from INITIALIZE's state
};

// A disk's record of step n.
struct AdjDisk {
  double x, y, r, u, v, w;
};

// One node through a reverse level.
template <class T>
struct AdjNode {
  T rho, ir, upx, upy;        // density, 1/density, velocity before the correction
  int win;                    // disk that sets G (-1: none), its phi and velocity
  T phw, dphw, usxw, usyw;    // (dphw: -dphi/dr / r)
  T aM[9], arho, aupx, aupy;  // dJ/d(moments), dJ/drho, dJ/du_pred
  T aGx, aGy;
};

// F(n) of the node as shifted populations, and omega(n).
template <class T>
__device__ __forceinline__ void adj_load_fwd(const Geometry& g, const Model& m, const AdjIO<T>& io,
                                             int i, int j, bool act, T* h, T& om) {
  if (io.level0 || !act) {
    double fe[9];
    feq_double(m, 0.0, 0.0, m.rho0, fe);
#pragma unroll
    for (int k = 0; k < 9; ++k) h[k] = (T)(fe[k] - wexact(k) * m.rho0);
  } else {
    pull_bc<T>(io.fs, g, m.bc, i, j, h);
    if (sizeof(T) == 8) {
#pragma unroll
      for (int k = 0; k < 9; ++k) h[k] = h[k] - (T)(wexact(k) * m.rho0);
    }
  }
  om = m.bingham && !io.level0 && act ? io.oms[(long long)j * g.pitch + i] : (T)m.omega;
}

// dJ/df*(n+1) of the node from the adjoint field of level n+1, and
// dJ/domega(n+1) (CG: past the L1 cache).
template <class T, bool CG>
__device__ __forceinline__ void adj_load_adj(const Geometry& g, const Model& m, const AdjIO<T>& io,
                                             int i, int j, bool act, T* ahs, T& awo) {
  if (io.a_in && act) {
    adj_gather<T, CG>(io.a_in, g, i, j, ahs);
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) ahs[k] = (T)0;
  }
  awo = (m.bingham && io.aw_in && act) ? ld<CG>(io.aw_in + (long long)j * g.pitch + i) : (T)0;
}

// Density and velocity from the moments mh of the shifted populations.
template <class T>
__device__ __forceinline__ void adj_macro(const Model& m, bool fluid, const T* mh, AdjNode<T>& v) {
  v.rho = (T)m.rho0;
  if (fluid) v.rho = (T)m.rho0 + mh[0];
  v.ir = (T)1 / v.rho;
  // divided, not times 1/rho: the sums over a disk that cancel (dJ/dy0 of one
  // between two nodes) show its last bit, 1e-5 of the entry in FP32
  v.upx = fluid ? mh[3] / v.rho : (T)0;
  v.upy = fluid ? mh[5] / v.rho : (T)0;
  v.win = -1;
  v.phw = v.dphw = v.usxw = v.usyw = (T)0;
}

// Disk c (called in index order): the last one with phi > 0 sets G.
template <class T>
__device__ __forceinline__ void adj_winner(const Model& m, int c, const AdjDisk& D, int i, int j,
                                           AdjNode<T>& v) {
  const T di = (T)((double)i - D.x), dj = (T)((double)j - D.y);
  const T phi = phi_of<T>(di, dj, (T)D.r, m);
  if (phi > (T)0) {
    v.win = c;
    v.phw = phi;
    v.dphw = dphi_of<T>(di, dj, (T)D.r, m);
    v.usxw = (T)D.u - (T)D.w * dj;
    v.usyw = (T)D.v + (T)D.w * di;
  }
}

// The transposed collision of a node: from dJ/df*(n+1) (ahs) and
// dJ/domega(n+1) (awo) to the fields of v, dJ/domega(n) (returned; for a
// model with one omega 0, its share is in gnu) and the node's dJ/dnu and
// dJ/dtau_y.
template <class T>
__device__ __forceinline__ T adj_collide(const Model& m, double kappa, bool node_omega, bool act,
                                         bool fluid, const T* mh, const T* ahs, T om, T awo,
                                         AdjNode<T>& v, double& gnu, double& gty) {
  const T drho = fluid ? mh[0] : (T)0;
  T Gx = (T)0, Gy = (T)0;
  if (v.win >= 0) {
    Gx = v.phw * (v.usxw - v.upx);
    Gy = v.phw * (v.usyw - v.upy);
  }
  const T ux = v.upx + (T)0.5 * Gx, uy = v.upy + (T)0.5 * Gy;
  const T sw = om;
  const T i8w = (T)1 / ((T)8 - om);
  const T sq = m.q_of_omega ? (T)8 * ((T)2 - om) * i8w : (T)m.s_q;
  const T s1 = (T)m.s_e, s2 = (T)m.s_eps;
  const T kap = (T)kappa;
  const T U2 = ux * ux + uy * uy;
  const T mne1 = mh[1] + (T)2 * drho - (T)3 * v.rho * U2;
  const T mne4 = mh[4] + v.rho * ux, mne6 = mh[6] + v.rho * uy;
  const T mne7 = mh[7] - v.rho * (ux * ux - uy * uy), mne8 = mh[8] - v.rho * ux * uy;
  const T Fx = v.rho * Gx, Fy = v.rho * Gy;
  const T mf4 = -Fx, mf6 = -Fy, mf7 = (T)2 * (Fx * ux - Fy * uy), mf8 = Fy * ux + Fx * uy;

  // f*(n+1) = kappa M^-1 m' + const  ->  dJ/dm' = kappa D^-1 M dJ/df*
  T am[9];
  moments9<T>(ahs, am);
  {
    const T k36 = kap * (T)(1.0 / 36.0);
    am[0] *= (T)4 * k36;
    am[1] *= k36;
    am[2] *= k36;
    am[3] *= (T)6 * k36;
    am[4] *= (T)3 * k36;
    am[5] *= (T)6 * k36;
    am[6] *= (T)3 * k36;
    am[7] *= (T)9 * k36;
    am[8] *= (T)9 * k36;
  }
  // m' = M - S m_neq + (1 - S/2) m_F
#pragma unroll
  for (int k = 0; k < 9; ++k) v.aM[k] = am[k];
  T an1 = -s1 * am[1], an2 = -s2 * am[2], an4 = -sq * am[4], an6 = -sq * am[6];
  T an7 = -sw * am[7], an8 = -sw * am[8];
  T asq = -(mne4 + (T)0.5 * mf4) * am[4] - (mne6 + (T)0.5 * mf6) * am[6];
  T asw = -(mne7 + (T)0.5 * mf7) * am[7] - (mne8 + (T)0.5 * mf8) * am[8];
  T aux = (T)0, auy = (T)0;
  v.arho = v.aGx = v.aGy = (T)0;

  // Papanastasiou viscosity and omega(n+1) (C6:903-958)
  if (m.bingham) {
    const T y1 = s1 * mne1, y7 = sw * mne7, y8 = sw * mne8;
    const T Pg = Gx * ux + Gy * uy;
    const T D11 = kap * ((T)-0.25 * y1 - (T)0.75 * y7) +
                  (T)0.75 * ((sw - s1) * Pg - (T)2 * sw * Gx * ux);
    const T D22 = kap * ((T)-0.25 * y1 + (T)0.75 * y7) +
                  (T)0.75 * ((sw - s1) * Pg - (T)2 * sw * Gy * uy);
    const T D12 = kap * ((T)-1.5 * y8) + (T)0.75 * (-sw * (Gx * uy + Gy * ux));
    const T ir = v.ir;
    const T d11 = D11 * ir, d22 = D22 * ir, d12 = D12 * ir;
    const T gam = tsqrt((T)2 * fabs(d11 * d11 + d22 * d22 + (T)2 * (d12 * d12)));
    const T nu = (T)m.nu, ty = (T)m.tau_y, mp = (T)m.m_pap;
    const bool low = gam < (T)m.gamma_min;
    T g1 = (T)1, rq = (T)0.5;
    if (!low) papanastasiou_terms<T>(mp * gam, &g1, &rq);
    const T nuA = nu + ty * mp * g1;
    const T wout = (T)1 / ((T)3 * nuA * ir + (T)0.5);
    const T az = -wout * wout * awo;
    const T anuA = (T)3 * az * ir;
    v.arho += (T)-3 * nuA * ir * ir * az;
    gnu += (double)anuA;
    gty += (double)(anuA * mp * g1);
    const T agam = low ? (T)0 : -anuA * ty * mp * mp * rq;
    T ad11 = (T)0, ad22 = (T)0, ad12 = (T)0;
    if (gam > (T)0) {
      const T q = (T)2 * agam / gam;
      ad11 = q * d11;
      ad22 = q * d22;
      ad12 = (T)2 * q * d12;
    }
    v.arho -= (ad11 * d11 + ad22 * d22 + ad12 * d12) * ir;
    const T aD11 = ad11 * ir, aD22 = ad22 * ir, aD12 = ad12 * ir;
    const T ay1 = (T)-0.25 * kap * (aD11 + aD22);
    const T ay7 = (T)0.75 * kap * (aD22 - aD11);
    const T ay8 = (T)-1.5 * kap * aD12;
    const T aP = (T)0.75 * (sw - s1) * (aD11 + aD22);
    asw += (T)0.75 * Pg * (aD11 + aD22) - (T)1.5 * (Gx * ux * aD11 + Gy * uy * aD22) -
           (T)0.75 * (Gx * uy + Gy * ux) * aD12 + mne7 * ay7 + mne8 * ay8;
    an1 += s1 * ay1;
    an7 += sw * ay7;
    an8 += sw * ay8;
    v.aGx += aP * ux - (T)1.5 * sw * ux * aD11 - (T)0.75 * sw * uy * aD12;
    v.aGy += aP * uy - (T)1.5 * sw * uy * aD22 - (T)0.75 * sw * ux * aD12;
    aux += aP * Gx - (T)1.5 * sw * Gx * aD11 - (T)0.75 * sw * Gy * aD12;
    auy += aP * Gy - (T)1.5 * sw * Gy * aD22 - (T)0.75 * sw * Gx * aD12;
  }

  // m_neq = M - m_eq(v.rho, u)
  v.aM[1] += an1; v.aM[2] += an2; v.aM[4] += an4; v.aM[6] += an6; v.aM[7] += an7; v.aM[8] += an8;
  {
    const T q1 = -an1, q2 = -an2, q4 = -an4, q6 = -an6, q7 = -an7, q8 = -an8;
    v.arho += q1 * ((T)-2 + (T)3 * U2) + q2 * ((T)1 - (T)3 * U2) - q4 * ux - q6 * uy +
            q7 * (ux * ux - uy * uy) + q8 * ux * uy;
    aux += (T)6 * v.rho * ux * (q1 - q2) - v.rho * q4 + (T)2 * v.rho * ux * q7 + v.rho * uy * q8;
    auy += (T)6 * v.rho * uy * (q1 - q2) - v.rho * q6 - (T)2 * v.rho * uy * q7 + v.rho * ux * q8;
  }
  // forcing moments m_F(v.rho G, u) (C1:995-1016)
  {
    const T b1 = ((T)1 - (T)0.5 * s1) * am[1], b2 = ((T)1 - (T)0.5 * s2) * am[2];
    const T b3 = am[3], b4 = ((T)1 - (T)0.5 * sq) * am[4];
    const T b5 = am[5], b6 = ((T)1 - (T)0.5 * sq) * am[6];
    const T b7 = ((T)1 - (T)0.5 * sw) * am[7], b8 = ((T)1 - (T)0.5 * sw) * am[8];
    const T aFx = (T)6 * ux * (b1 - b2) + b3 - b4 + (T)2 * ux * b7 + uy * b8;
    const T aFy = (T)6 * uy * (b1 - b2) + b5 - b6 - (T)2 * uy * b7 + ux * b8;
    aux += (T)6 * Fx * (b1 - b2) + (T)2 * Fx * b7 + Fy * b8;
    auy += (T)6 * Fy * (b1 - b2) - (T)2 * Fy * b7 + Fx * b8;
    v.arho += aFx * Gx + aFy * Gy;
    v.aGx += v.rho * aFx;
    v.aGy += v.rho * aFy;
  }
  // rates of omega (C6:1002-1021)
  T aom = asw;
  if (m.q_of_omega) aom += asq * (T)-48 * i8w * i8w;
  if (!node_omega && act) gnu += (double)(aom * (T)(-3.0 * m.omega * m.omega));  // omega = 1/(3 nu + 1/2)
  // u = u_pred + G/2 (C1:1138-1152); G = phi (u_p - u_pred) of the winner
  v.aupx = aux;
  v.aupy = auy;
  v.aGx += (T)0.5 * aux;
  v.aGy += (T)0.5 * auy;
  if (v.win >= 0) {
    v.aupx -= v.phw * v.aGx;
    v.aupy -= v.phw * v.aGy;
  }
  return aom;
}

// Disk c at the node: G of the winner, FORCE(n) (aH = dJ/dFORCE(n) of the
// disk), phi and the rigid velocity; the node's share of dJ/d(x, y, u, v, w)
// of the disk in s[5].
template <class T>
__device__ __forceinline__ void adj_disk(const Model& m, int c, const AdjDisk& D,
                                         const double* aH, int i, int j, AdjNode<T>& v, double* s) {
  const T di = (T)((double)i - D.x), dj = (T)((double)j - D.y);
  // a disk after the winner has phi = 0 here, without a winner every disk has
  T phi = (T)0;
  if (c == v.win) phi = v.phw;
  else if (c < v.win) phi = phi_of<T>(di, dj, (T)D.r, m);
  if (!(phi > (T)0)) return;
  const T W = (T)D.w;
  const T usx = (T)D.u - W * dj, usy = (T)D.v + W * di;
  T aphi = (T)0, ausx = (T)0, ausy = (T)0, adi = (T)0, adj = (T)0;
  if (c == v.win) {
    aphi += v.aGx * (usx - v.upx) + v.aGy * (usy - v.upy);
    ausx += v.phw * v.aGx;
    ausy += v.phw * v.aGy;
  }
  const T aHx = (T)aH[0], aHy = (T)aH[1], aT = (T)aH[2];
  const T ex = v.upx - usx, ey = v.upy - usy;
  const T tq = di * ey - dj * ex;
  const T sdot = aHx * ex + aHy * ey + aT * tq;
  v.arho += phi * sdot;
  aphi += v.rho * sdot;
  const T rp = v.rho * phi;
  const T aex = rp * (aHx - aT * dj), aey = rp * (aHy + aT * di);
  v.aupx += aex;
  v.aupy += aey;
  ausx -= aex;
  ausy -= aey;
  adi += rp * aT * ey;
  adj -= rp * aT * ex;
  s[2] = (double)ausx;
  s[3] = (double)ausy;
  s[4] = (double)(-dj * ausx + di * ausy);
  adj -= W * ausx;
  adi += W * ausy;
  const T aD = aphi * (c == v.win ? v.dphw : dphi_of<T>(di, dj, (T)D.r, m));
  adi -= aD * di;
  adj -= aD * dj;
  s[0] = -(double)adi;
  s[1] = -(double)adj;
}

// Warp sums of a disk's s[5] into its accumulators (every lane calls it).
__device__ __forceinline__ void adj_add(double* a_p, long long st, int p, double* s, int lane) {
  const bool any = __any_sync(0xffffffffu, s[0] != 0.0 || s[1] != 0.0 || s[2] != 0.0 ||
                                               s[3] != 0.0 || s[4] != 0.0);
  if (!any) return;
#pragma unroll
  for (int k = 0; k < 5; ++k) s[k] = warp_sum(s[k]);
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 5; ++k) atomicAdd(a_p + k * st + p, s[k]);
  }
}

// u_pred = j / rho, rho = rho0 + sum h, j = sum c h: dJ/dF(n) of the node, and
// from it the node's entries of the adjoint field.
template <class T>
__device__ __forceinline__ void adj_store(const Geometry& g, int bc, const AdjIO<T>& io, int i,
                                          int j, AdjNode<T>& v) {
  const T ir = v.ir;
  v.arho -= (v.aupx * v.upx + v.aupy * v.upy) * ir;
  v.aM[0] += v.arho;
  v.aM[3] += v.aupx * ir;
  v.aM[5] += v.aupy * ir;
  T ah[9];
  moments9_t<T>(v.aM, ah);
  adj_boundary<T>(g, bc, i, j, ah);
  const long long n = (long long)j * g.pitch + i;
#pragma unroll
  for (int k = 0; k < 9; ++k) io.a_out[plane_of(k) * g.plane + n] = ah[k];
}

}  // namespace

template <class T>
__global__ void __launch_bounds__(ADJ_TPB, ADJ_MINB<T>) k_adj_lattice(const AdjLatticeArgs a) {
  const Geometry& g = a.g;
  const Model& m = a.m;
  __shared__ AdjDisk s_d[ADJ_MAX_PARTICLES];
  __shared__ double s_a[ADJ_MAX_PARTICLES][3];
  __shared__ int s_idx[ADJ_MAX_PARTICLES];
  __shared__ int s_nc;
  __shared__ double s_g[ADJ_TPB / 32][2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i = blockIdx.x * TX + (tid % TX), j = blockIdx.y * TY + (tid / TX);
  // the next particle adjoint kernel may launch; it waits for this grid
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // disks whose support reaches this block, in index order (records of step
  // n, written by the forward pass)
  if (tid == 0) {
    int c = 0;
    if (!a.level0) {
      const double i0 = blockIdx.x * TX, i1 = i0 + TX - 1, j0 = blockIdx.y * TY, j1 = j0 + TY - 1;
      for (int p = 0; p < a.np; ++p) {
        const PRef P{const_cast<double*>(a.ps) + p, a.npad};
        const double x = P[P_X], y = P[P_Y], r = 0.5 * P[P_D];
        const double rs = r + 0.5 * m.zeta + 1.0;
        if (x + rs < i0 || x - rs > i1 || y + rs < j0 || y - rs > j1) continue;
        s_idx[c] = p;
        s_d[c] = AdjDisk{x, y, r, P[P_U], P[P_V], P[P_W]};
        ++c;
      }
    }
    s_nc = c;
  }
  __syncthreads();
  const int nc = s_nc;
  const bool act = i <= g.nx && j <= g.ny;
  const long long n = (long long)j * g.pitch + i;
  const AdjIO<T> io{static_cast<const T*>(a.fs), static_cast<const T*>(a.oms),
                    static_cast<const T*>(a.a_in), static_cast<const T*>(a.aw_in),
                    static_cast<T*>(a.a_out), static_cast<T*>(a.aw_out), a.level0 != 0};
  double gnu = 0.0, gty = 0.0;
  T h[9], ahs[9], mh[9], om, awo;
  adj_load_fwd<T>(g, m, io, i, j, act, h, om);
  adj_load_adj<T, false>(g, m, io, i, j, act, ahs, awo);
  moments9<T>(h, mh);
  AdjNode<T> v;
  adj_macro<T>(m, act && !io.level0, mh, v);
  if (act)
    for (int c = 0; c < nc; ++c) adj_winner<T>(m, c, s_d[c], i, j, v);
  const bool node_omega = m.bingham && !io.level0;
  const T aom = adj_collide<T>(m, a.kappa, node_omega, act, act && !io.level0, mh, ahs, om, awo,
                               v, gnu, gty);
  if (node_omega && act) io.aw_out[n] = aom;

  // ---- disks ---------------------------------------------------------------
  // dJ/dFORCE(n) comes from the particle adjoint kernel launched before this
  // one, which also clears a_p after reading it: wait for it here.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid < nc) {
    const int p = s_idx[tid];
#pragma unroll
    for (int k = 0; k < 3; ++k) s_a[tid][k] = a.a_h[k * a.npad + p];
  }
  __syncthreads();
  for (int c = 0; c < nc; ++c) {
    double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (act) adj_disk<T>(m, c, s_d[c], s_a[c], i, j, v, sum);
    adj_add(a.a_p, a.npad, s_idx[c], sum, lane);
  }
  if (act && !io.level0) adj_store<T>(g, m.bc, io, i, j, v);

  // ---- dJ/dnu, dJ/dtau_y: one slot per block, fixed order ------------------
  gnu = warp_sum(gnu);
  gty = warp_sum(gty);
  if (lane == 0) {
    s_g[warp][0] = gnu;
    s_g[warp][1] = gty;
  }
  __syncthreads();
  if (tid == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int w = 0; w < ADJ_TPB / 32; ++w) {
      t0 += s_g[w][0];
      t1 += s_g[w][1];
    }
    double* slot = a.gacc + 2 * ((long long)blockIdx.y * gridDim.x + blockIdx.x);
    slot[0] += t0;
    slot[1] += t1;
  }
}

// ---------------------------------------------------------------------------
// Glowinski repulsion magnitude g(r) along the centre line and g'(r)
// (C1:701-768, C3:739-804): range rc = contact + zeta; g = eps C q^2,
// q = (r - rc)/zeta, plus E C (contact - r)/zeta when overlapping.
__device__ __forceinline__ void glowinski(double r, double contact, double zeta, double eps,
                                          double E, double C, double* gv, double* gd) {
  *gv = 0.0;
  *gd = 0.0;
  if (r > contact + zeta) return;
  const double q = (r - contact - zeta) / zeta;
  *gv = eps * C * q * q;
  *gd = 2.0 * eps * C * q / zeta;
  if (r <= contact) {
    *gv += E * C * (contact - r) / zeta;
    *gd -= E * C / zeta;
  }
}

// What the transposed update of step n needs of the records alone: rho0/rho_p,
// 1/M, 1/I, the factors of dJ/drho_p and the walls' share of dJ/d(x, y) per
// unit of dJ/dFORCE.
struct AdjCoef {
  double rr, im, ii, kx, ky, kt, wx, wy;
};

// Of disk p: prev, cur are the records of steps n-1 and n.
//   X(n) = X(n-1) + (V(n) + V(n-1))/2; V(n) = V + (FORCE + F_H_IN + F_COL)/M
//   (+ buoyancy); F_H_IN/M = (rho0/rho_p)(V - V_OLD) (C1:247-259)
// and the walls (C1:737-745 mirror images, C3:775-783 wall disks): the image
// lies along one axis, e = s*(coordinate) + const with s = 2 or 1.
__device__ __forceinline__ AdjCoef adj_coef(const AdjParticleArgs& a, int p, const double* prev,
                                            const double* cur) {
  const PRef Q{const_cast<double*>(prev) + p, a.npad};
  const PRef C{const_cast<double*>(cur) + p, a.npad};
  const double irho = 1.0 / Q[P_RHO];
  AdjCoef c;
  c.rr = a.rho0 * irho;
  c.im = 1.0 / Q[P_M];
  c.ii = 1.0 / Q[P_I];
  c.kx = irho * ((C[P_FX] + C[P_FCX]) * c.im + c.rr * (Q[P_U] - Q[P_UO]));
  c.ky = irho * ((C[P_FY] + C[P_FCY]) * c.im + c.rr * (Q[P_V] - Q[P_VO]) - c.rr * a.gravity);
  c.kt = irho * (C[P_TZ] * c.ii + c.rr * (Q[P_W] - Q[P_WO]));
  c.wx = c.wy = 0.0;
  if (a.wall_model != 2) {
    const double x = Q[P_X], y = Q[P_Y], D = Q[P_D];
#pragma unroll
    for (int iw = 1; iw <= 4; ++iw) {
      double e, sc;
      const bool ydir = (iw == 1 || iw == 3);
      if (a.wall_model == 0) {
        sc = 2.0;
        e = iw == 1 ? 2.0 * y : iw == 2 ? 2.0 * x - 2.0 * (double)a.nx
          : iw == 3 ? 2.0 * y - a.mirror_top : 2.0 * x - a.mirror_left;
      } else {
        sc = 1.0;
        e = iw == 1 ? y + 0.5 * D : iw == 2 ? x - (double)a.nx - 0.5 * D
          : iw == 3 ? y - (double)a.ny - 0.5 * D : x + 0.5 * D;
      }
      double gv, gd;
      glowinski(fabs(e), D, a.rep_zeta, a.eps_w, a.e_w, a.c_ij, &gv, &gd);
      if (ydir) c.wy += sc * gd;
      else c.wx += sc * gd;
    }
  }
  return c;
}

// dJ/d(state) of a disk before the update of step n (but for the pairs' part
// of X and Y), dJ/dFORCE(n-1) and the disk's share of dJ/drho_p.
struct AdjUpdate {
  double s[8];        // x y u v w uo vo wo
  double fx, fy, tz;  // dJ/dFORCE(n-1)
  double rho;
};

// From dJ/d(state) after the update (s[8], with the lattice's part).
__device__ __forceinline__ AdjUpdate adj_newton(const AdjParticleArgs& a, long long n, int p,
                                                const AdjCoef& c, double* s) {
  if (p == a.obj_p && n >= a.n0 && n <= a.n1) {
    const int o = a.obj_c == P_X ? 0 : a.obj_c == P_Y ? 1 : a.obj_c == P_U ? 2
                : a.obj_c == P_V ? 3 : 4;
#pragma unroll
    for (int k = 0; k < 5; ++k)
      if (k == o) s[k] += a.obj_w;
  }
  const double bx = s[2] + 0.5 * s[0], by = s[3] + 0.5 * s[1], bw = s[4];
  AdjUpdate r;
  r.fx = bx * c.im;
  r.fy = by * c.im;
  r.tz = bw * c.ii;
  r.s[0] = s[0] + c.wx * r.fx;
  r.s[1] = s[1] + c.wy * r.fy;
  r.s[2] = 0.5 * s[0] + bx + s[5] + c.rr * bx;
  r.s[3] = 0.5 * s[1] + by + s[6] + c.rr * by;
  r.s[4] = bw + s[7] + c.rr * bw;
  r.s[5] = -c.rr * bx;
  r.s[6] = -c.rr * by;
  r.s[7] = -c.rr * bw;
  r.rho = -(bx * c.kx + by * c.ky + bw * c.kt);
  return r;
}

// The pair repulsion's part of dJ/d(x, y) of disk p at step n-1, from
// dJ/dFORCE of all disks (s_fx, s_fy): F_p = g(r) e/r, e = X_p - X_q;
// dF/de = g' e e^T/r^2 + g/r (I - e e^T/r^2).
__device__ __forceinline__ void adj_pairs(const AdjParticleArgs& a, int p, const double* prev,
                                          const double* s_fx, const double* s_fy, double& aX,
                                          double& aY) {
  if (a.np < 2) return;
  const PRef Q{const_cast<double*>(prev) + p, a.npad};
  const double x = Q[P_X], y = Q[P_Y], D = Q[P_D];
  const double fx = s_fx[p], fy = s_fy[p];
  for (int q = 0; q < a.np; ++q) {
    if (q == p) continue;
    const PRef Qq{const_cast<double*>(prev) + q, a.npad};
    const double ex = x - Qq[P_X], ey = y - Qq[P_Y];
    const double r = sqrt(ex * ex + ey * ey);
    if (!(r > 0.0)) continue;
    double gv, gd;
    glowinski(r, 0.5 * D + 0.5 * Qq[P_D], a.rep_zeta, a.eps_p, a.e_p, a.c_ij, &gv, &gd);
    if (gv == 0.0 && gd == 0.0) continue;
    const double nx_ = ex / r, ny_ = ey / r;
    const double dfx = fx - s_fx[q], dfy = fy - s_fy[q];
    const double en = nx_ * dfx + ny_ * dfy;
    const double t = gv / r;
    aX += gd * en * nx_ + t * (dfx - en * nx_);
    aY += gd * en * ny_ + t * (dfy - en * ny_);
  }
}

__global__ void __launch_bounds__(ADJ_MAX_PARTICLES) k_adj_particles(const AdjParticleArgs a) {
  __shared__ double s_fx[ADJ_MAX_PARTICLES], s_fy[ADJ_MAX_PARTICLES];
  const int p = threadIdx.x;
  // launched as a programmatic dependent of the lattice adjoint kernel of
  // the same step: its per-disk sums and dJ/dF must be complete
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long st = a.npad;
  AdjUpdate r;
  if (p < a.np) {
    double s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] = a.a_state[k * st + p];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      s[k] += a.a_p[k * st + p];
      a.a_p[k * st + p] = 0.0;
    }
    r = adj_newton(a, a.n, p, adj_coef(a, p, a.prev, a.cur), s);
    a.a_h[p] = r.fx;
    a.a_h[st + p] = r.fy;
    a.a_h[2 * st + p] = r.tz;
    s_fx[p] = r.fx;
    s_fy[p] = r.fy;
    a.a_rho[p] += r.rho;
  }
  __syncthreads();
  if (p < a.np) {
    adj_pairs(a, p, a.prev, s_fx, s_fy, r.s[0], r.s[1]);
#pragma unroll
    for (int k = 0; k < 8; ++k) a.a_state[k * st + p] = r.s[k];
  }
}

// ---------------------------------------------------------------------------
// Levels n_hi .. n_lo of a small lattice in one launch (a cooperative launch,
// one block per SM), with the particle adjoints between them.  At 101 x 301
// nodes (FP64) a level in kernels of its own is a chain of two dependent
// launches, about 15 us; here it takes 7.1 us, in cycles of a warp with a disk
// (the longest): gather 1500, collision 1600, disk 2500, store 900, and about
// 6600 from its arrival at the grid barrier to the next level, 4800 of them
// spent on that level's forward half.  A block owns a contiguous
// range of 32-node row segments, one warp takes every 16th of them; one
// grid-wide barrier per level.  Every block keeps dJ/d(state) of all disks in
// shared memory and updates all of them, from the same sums and so to the
// same bits; the sums of the levels rotate through three sets (level l adds
// to one, reads the previous level's and clears the next level's).  What
// needs no adjoint field -- f*(n) pulled, its moments, the disk that sets G,
// the coefficients of the disks' update -- is done for a warp's first segment
// while the barrier is waited for; the disks' update overlaps the segments'
// gather and collision.
constexpr int LEVELS_TPB = 512;
constexpr int LEVELS_WARPS = LEVELS_TPB / 32;
// Segments a block has at least (the gradient of 400 steps at 101 x 301 with 16
// / 12 / 8 / 4, here and in k_steps: 9.8 / 9.35 / 9.2 / 9.3 ms FP64).
constexpr int LEVELS_MIN_SEGS = 8;
constexpr uint32_t LEVELS_WAIT = 1u << 22;  // polls of dJ/dFORCE before giving up

template <class T>
__global__ void __launch_bounds__(LEVELS_TPB, 1) k_adj_levels(const AdjLevelsArgs a) {
  __shared__ AdjDisk s_d[2][ADJ_MAX_PARTICLES];     // records of level n at [n & 1]
  __shared__ double s_st[8][ADJ_MAX_PARTICLES];     // dJ/d(state)
  __shared__ double s_rho[ADJ_MAX_PARTICLES];       // dJ/drho_p
  __shared__ AdjCoef s_c[ADJ_MAX_PARTICLES];        // of the next update
  __shared__ double s_h[3][ADJ_MAX_PARTICLES];      // dJ/dFORCE(n)
  __shared__ double s_g[LEVELS_WARPS][2];
  __shared__ uint64_t s_force;                      // mbarrier: dJ/dFORCE(n) is in s_h
  __shared__ int s_stop;
  const Geometry& g = a.g;
  const Model& m = a.m;
  const AdjParticleArgs& q = a.p;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int spr = (g.nx + 32) / 32;  // 32-node segments per row
  const int nseg = spr * (g.ny + 1);
  const int seg0 = (int)((long long)nseg * blockIdx.x / gridDim.x);
  const int seg1 = (int)((long long)nseg * (blockIdx.x + 1) / gridDim.x);
  const long long st = q.npad, rec = PS * st;
  // the last two warps update the disks: they have the fewest segments
  const int p = tid - (LEVELS_TPB - ADJ_MAX_PARTICLES);
  const bool disk_warp = p >= 0, disk = disk_warp && p < q.np;
  auto load_disk = [&](long long n) {
    const PRef P{const_cast<double*>(a.hist + rec * n) + p, q.npad};
    s_d[n & 1][p] = AdjDisk{P[P_X], P[P_Y], 0.5 * P[P_D], P[P_U], P[P_V], P[P_W]};
  };
  const uint32_t force_bar = (uint32_t)__cvta_generic_to_shared(&s_force);
  if (tid == 0) {
    s_stop = timed_out(a.status) ? 1 : 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(force_bar) : "memory");
  }
  if (disk) {
#pragma unroll
    for (int k = 0; k < 8; ++k) s_st[k][p] = q.a_state[k * st + p];
#pragma unroll
    for (int k = 0; k < 3; ++k) s_h[k][p] = q.a_h[k * st + p];
    s_rho[p] = q.a_rho[p];
    load_disk(a.n_hi);
  }
  __syncthreads();
  if (s_stop) return;
  double gnu = 0.0, gty = 0.0;
  // the forward half of one segment at level n
  int i = 0, j = 0;
  bool act = false;
  unsigned near[2] = {0u, 0u};  // disks that may reach the segment
  T mh[9], om = (T)0;
  AdjNode<T> v;
  AdjIO<T> io;
  auto level_io = [&](long long n) {
    const unsigned char* slot = a.slots + (size_t)(n - a.n_lo) * a.slot_bytes;
    const int b = (int)((a.in0 + (a.n_hi - n)) & 1);
    const bool zero = n == a.n_hi && !a.have;
    io = AdjIO<T>{reinterpret_cast<const T*>(slot), reinterpret_cast<const T*>(slot) + 9 * g.plane,
                  zero ? nullptr : static_cast<const T*>(a.a[b]),
                  zero ? nullptr : static_cast<const T*>(a.aw[b]), static_cast<T*>(a.a[b ^ 1]),
                  static_cast<T*>(a.aw[b ^ 1]), false};
  };
  auto forward = [&](int seg, long long n) {
    j = seg / spr;
    const int i0 = (seg - j * spr) * 32;
    i = i0 + lane;
    act = i <= g.nx && LBM_IN(i0, g.nx + 1, a.status) && LBM_IN(j, g.ny + 1, a.status) &&
          LBM_IN(n - a.n_lo, a.n_hi - a.n_lo + 1, a.status);
    T h[9];
    adj_load_fwd<T>(g, m, io, i, j, act, h, om);
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int c = 32 * w + lane;
      bool nr = false;
      if (c < q.np) {
        const AdjDisk& D = s_d[n & 1][c];
        const double dl = (double)i0 - D.x, dr = dl + 31.0;
        const double dx = dl > 0.0 ? dl : (dr < 0.0 ? -dr : 0.0), dy = (double)j - D.y;
        const double reach = D.r + 0.5 * m.zeta + 1.0;
        nr = dx * dx + dy * dy < reach * reach;
      }
      near[w] = __ballot_sync(0xffffffffu, nr);
    }
    moments9<T>(h, mh);
    adj_macro<T>(m, act, mh, v);
#pragma unroll
    for (int w = 0; w < 2; ++w)
      for (unsigned b = near[w]; b; b &= b - 1) {
        const int c = 32 * w + __ffs(b) - 1;
        if (act) adj_winner<T>(m, c, s_d[n & 1][c], i, j, v);
      }
  };
  level_io(a.n_hi);
  if (seg0 + warp < seg1) forward(seg0 + warp, a.n_hi);
  for (long long n = a.n_hi;; --n) {
    const int l = (int)(a.n_hi - n);
    double* const sums = q.a_p + (long long)((a.ap0 + l) % 3) * 5 * st;
    if (disk_warp) {
      if (l > 0) {  // the update of step n + 1
        const double* const prev = a.hist + rec * n;
        AdjUpdate r;
        if (disk) {
          const double* const sp = q.a_p + (long long)((a.ap0 + l - 1) % 3) * 5 * st + p;
          double s[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) s[k] = s_st[k][p];
#pragma unroll
          for (int k = 0; k < 5; ++k) s[k] += __ldcg(sp + k * st);
          r = adj_newton(q, n + 1, p, s_c[p], s);
          s_h[0][p] = r.fx;
          s_h[1][p] = r.fy;
          s_h[2][p] = r.tz;
          s_rho[p] += r.rho;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(force_bar);
        if (q.np > 1) asm volatile("bar.sync 1, 64;" ::: "memory");
        if (disk) {
          adj_pairs(q, p, prev, s_h[0], s_h[1], r.s[0], r.s[1]);
#pragma unroll
          for (int k = 0; k < 8; ++k) s_st[k][p] = r.s[k];
        }
      } else if (lane == 0) {
        mbar_arrive(force_bar);
      }
      if (disk && n > a.n_lo) load_disk(n - 1);
      // the next level's sums (read last before the previous barrier)
      if (disk && p % (int)gridDim.x == (int)blockIdx.x) {
        double* const nxt = q.a_p + (long long)((a.ap0 + l + 1) % 3) * 5 * st + p;
#pragma unroll
        for (int k = 0; k < 5; ++k) nxt[k * st] = 0.0;
      }
    }
    bool waited = false;  // for dJ/dFORCE(n)
    for (int seg = seg0 + warp; seg < seg1; seg += LEVELS_WARPS) {
      if (seg != seg0 + warp) forward(seg, n);
      T ahs[9], awo;
      adj_load_adj<T, true>(g, m, io, i, j, act, ahs, awo);
      const T aom = adj_collide<T>(m, a.kappa, m.bingham != 0, act, act, mh, ahs, om, awo, v,
                                   gnu, gty);
      const long long nd = (long long)j * g.pitch + i;
      if (m.bingham && act) io.aw_out[nd] = aom;
      if (near[0] | near[1]) {
        if (!waited && !mbar_wait(force_bar, l & 1, LEVELS_WAIT)) {
          atomicOr(a.status, ST_TIMEOUT);
          s_stop = 1;
        }
        waited = true;
#pragma unroll
        for (int w = 0; w < 2; ++w)
          for (unsigned b = near[w]; b; b &= b - 1) {
            const int c = 32 * w + __ffs(b) - 1;
            const double aH[3] = {s_h[0][c], s_h[1][c], s_h[2][c]};
            double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
            if (act) adj_disk<T>(m, c, s_d[n & 1][c], aH, i, j, v, sum);
            adj_add(sums, st, c, sum, lane);
          }
      }
      if (act) adj_store<T>(g, m.bc, io, i, j, v);
    }
    if (n == a.n_lo) break;
    __syncthreads();
    if (tid == 0) grid_arrive(a.bar);
    if (disk) {
      const double* const prev = a.hist + rec * (n - 1);
      s_c[p] = adj_coef(q, p, prev, prev + rec);
    }
    level_io(n - 1);
    if (seg0 + warp < seg1) forward(seg0 + warp, n - 1);
    if (tid == 0 && !grid_wait(a.bar, a.bar0 + (unsigned)(l + 1) * gridDim.x, a.status))
      s_stop = 1;
    __syncthreads();
    if (s_stop) return;
  }
  // ---- dJ/dnu, dJ/dtau_y: one slot per block, fixed order; the disks -------
  gnu = warp_sum(gnu);
  gty = warp_sum(gty);
  if (lane == 0) {
    s_g[warp][0] = gnu;
    s_g[warp][1] = gty;
  }
  __syncthreads();
  if (tid == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int w = 0; w < LEVELS_WARPS; ++w) {
      t0 += s_g[w][0];
      t1 += s_g[w][1];
    }
    a.gacc[2 * blockIdx.x] += t0;
    a.gacc[2 * blockIdx.x + 1] += t1;
  }
  // (every block has read these: it has passed a barrier of this launch)
  if (disk && blockIdx.x == 0 && a.n_hi > a.n_lo) {
#pragma unroll
    for (int k = 0; k < 8; ++k) q.a_state[k * st + p] = s_st[k][p];
    q.a_rho[p] = s_rho[p];
  }
}

template <class T>
cudaError_t launch_levels(const AdjLevelsArgs& a, cudaStream_t s, int* grid_out) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return e;
  // one slot of gacc per block: never more blocks than nbx * nby
  const long long nseg = (long long)((a.g.nx + 32) / 32) * (a.g.ny + 1);
  const long long want = std::min<long long>((nseg + LEVELS_MIN_SEGS - 1) / LEVELS_MIN_SEGS,
                                             (long long)a.g.nbx * a.g.nby);
  const int grid = (int)std::min<long long>(want, sms);
  *grid_out = grid;
  AdjLevelsArgs la = a;
  void* args[] = {&la};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&k_adj_levels<T>), dim3(grid),
                                     dim3(LEVELS_TPB), args, 0, s);
}

template <class K, class A>
cudaError_t launch_pdl(K kernel, dim3 grid, int block, const A& a, cudaStream_t s, int pdl) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

cudaError_t launch_adj_lattice_fp32(const AdjLatticeArgs& a, cudaStream_t s, int pdl) {
  return launch_pdl(k_adj_lattice<float>, dim3(a.g.nbx, a.g.nby), ADJ_TPB, a, s, pdl);
}
cudaError_t launch_adj_lattice_fp64(const AdjLatticeArgs& a, cudaStream_t s, int pdl) {
  return launch_pdl(k_adj_lattice<double>, dim3(a.g.nbx, a.g.nby), ADJ_TPB, a, s, pdl);
}
cudaError_t launch_adj_levels_fp32(const AdjLevelsArgs& a, cudaStream_t s, int* grid) {
  return launch_levels<float>(a, s, grid);
}
cudaError_t launch_adj_levels_fp64(const AdjLevelsArgs& a, cudaStream_t s, int* grid) {
  return launch_levels<double>(a, s, grid);
}
cudaError_t launch_adj_particles(const AdjParticleArgs& a, cudaStream_t s) {
  return launch_pdl(k_adj_particles, dim3(1), ADJ_MAX_PARTICLES, a, s, 1);
}

__global__ void k_set_ll(long long* p, long long v) { *p = v; }

cudaError_t launch_set_ll(long long* p, long long v, cudaStream_t s) {
  k_set_ll<<<1, 1, 0, s>>>(p, v);
  return cudaGetLastError();
}

}  // namespace lbm
