// lbm_disk.cuh -- arithmetic of one disk's time step (repulsion, C1:701-768,
// C3:739-804; Newton-Euler, C1:247-259, C6:300-312), shared by the particle
// kernel and the multi-step kernel.
//
// Rn is an FP64 value whose operations are rounded one by one (never
// contracted to fused multiply-adds, whatever the translation unit's flags),
// so a disk's update gives the reference's bits in every kernel.
#pragma once

#include <cuda_runtime.h>

#include "lbm_internal.h"

namespace lbm {

struct Rn {
  double v;
  __device__ __forceinline__ Rn() {}
  __device__ __forceinline__ Rn(double x) : v(x) {}
};
__device__ __forceinline__ Rn operator+(Rn a, Rn b) { return __dadd_rn(a.v, b.v); }
__device__ __forceinline__ Rn operator-(Rn a, Rn b) { return __dsub_rn(a.v, b.v); }
__device__ __forceinline__ Rn operator-(Rn a) { return -a.v; }
__device__ __forceinline__ Rn operator*(Rn a, Rn b) { return __dmul_rn(a.v, b.v); }
__device__ __forceinline__ Rn operator/(Rn a, Rn b) { return __ddiv_rn(a.v, b.v); }

// Whether two disks may be within the repulsion range: no false negatives
// (the margin is far above the rounding of the squares), so a pair it rejects
// has D_PP > r_a + r_b + ZITA and a force of exactly 0.
__device__ __forceinline__ bool pair_near(double ax, double ay, double ad, double bx, double by,
                                          double bd, double zita) {
  const double dx = ax - bx, dy = ay - by;
  const double lim = 0.5 * ad + 0.5 * bd + zita;
  return !(dx * dx + dy * dy > lim * lim * (1.0 + 1e-9));
}

// Pair force of (lo, hi), lo < hi, as the reference evaluates F_PP for
// IP = lo, JP = hi (C3:758-766); the contact branch tests D_PP or the stale
// wall distance D_PW.
__device__ __forceinline__ void pair_force(const ParticleArgs& a, Rn ax, Rn ay, Rn ad, Rn bx,
                                           Rn by, Rn bd, double test_stale, double* F) {
  const Rn ZITA = a.rep_zeta, CIJ = a.c_ij, EPS_P = a.eps_p, E_P = a.e_p;
  const Rn dx = ax - bx, dy = ay - by;
  const Rn D_PP = __dsqrt_rn((dx * dx + dy * dy).v);
  const Rn rsum = Rn(0.5) * ad + Rn(0.5) * bd;
  const double test = a.contact == 1 ? test_stale : D_PP.v;
  F[0] = 0.0;
  F[1] = 0.0;
  if (D_PP.v > (rsum + ZITA).v) return;
  const Rn q = (D_PP - Rn(0.5) * ad - Rn(0.5) * bd - ZITA) / ZITA;
  if (D_PP.v <= (rsum + ZITA).v && test > rsum.v) {
    F[0] = (EPS_P * CIJ * (q * q) * dx / D_PP).v;
    F[1] = (EPS_P * CIJ * (q * q) * dy / D_PP).v;
  } else if (test <= rsum.v) {
    const Rn e = E_P * CIJ * (rsum - D_PP) / ZITA;
    F[0] = ((EPS_P * CIJ * (q * q) + e) * dx / D_PP).v;
    F[1] = ((EPS_P * CIJ * (q * q) + e) * dy / D_PP).v;
  }
}

// Force of wall iw (1 bottom, 2 right, 3 top, 4 left) on a disk at (x, y)
// (C1:735-768 mirror images; C3:775-804 wall disks); returns D_PW.  The image
// lies on one axis with the disk, so the reference's sqrt(ex*ex + ey*ey) is
// |e| exactly (the square root of a rounded square is the number itself).
__device__ __forceinline__ double wall_force(const ParticleArgs& a, int iw, double xd, double yd,
                                             double D, double* F) {
  const Rn x = xd, y = yd;
  const bool vert = iw == 1 || iw == 3;  // along y
  Rn e;
  if (a.wall_model == 0) {
    const Rn img = iw == 1   ? -y
                   : iw == 2 ? Rn(2.0) * Rn((double)a.nx) - x
                   : iw == 3 ? Rn(a.mirror_top) - y
                             : Rn(a.mirror_left) - x;
    e = (vert ? y : x) - img;
  } else {
    const Rn img = iw == 1   ? Rn(-0.5) * Rn(D)
                   : iw == 2 ? Rn((double)a.nx) + Rn(0.5) * Rn(D)
                   : iw == 3 ? Rn((double)a.ny) + Rn(0.5) * Rn(D)
                             : Rn(-0.5) * Rn(D);
    e = (vert ? y : x) - img;
  }
  const double D_PW = fabs(e.v);
  F[0] = 0.0;
  F[1] = 0.0;
  const Rn ZITA = a.rep_zeta;
  if (!(D_PW > (Rn(D) + ZITA).v)) {
    const Rn CIJ = a.c_ij, EPS_W = a.eps_w, E_W = a.e_w, W = D_PW;
    const Rn q = (W - Rn(D) - ZITA) / ZITA;
    Rn f = 0.0;
    if (D_PW <= (Rn(D) + ZITA).v && D_PW > D) {
      f = EPS_W * CIJ * (q * q) * e / W;
    } else if (D_PW <= D) {
      const Rn c = E_W * CIJ * (Rn(D) - W) / ZITA;
      f = (EPS_W * CIJ * (q * q) + c) * e / W;
    }
    if (vert) F[1] = f.v;
    else F[0] = f.v;
  }
  return D_PW;
}

// State of one disk through its update.
struct DiskStep {
  double x, y, ang;           // in: old; out: new
  double u, v, w;             // in: V; out: new V
  double uo, vo, wo;          // in: VP_OLD
  double fx, fy, tz;          // FORCE of the last lattice step
  double rho_p, M, I;
  double fcx, fcy;            // F_COL
  double fhx, fhy, fht;       // out: F_H_IN
};

// Newton-Euler with the internal-mass correction (C1:250-258, C6:312), or the
// prescribed oscillation (C4:222-228) with F_H_IN of this step's velocity
// change (C4:270-272), in two parts: what needs no FORCE (s.fcx, s.fcy and
// the old velocities set), then the update.  Afterwards u..w hold the new
// velocity, uo..wo the old.
struct DiskTerms {
  double hx, hy, ht, cx, cy, b;  // F_H_IN / M, F_COL / M, buoyancy
};

__device__ __forceinline__ DiskTerms newton_terms(const ParticleArgs& a, long long kk,
                                                  DiskStep& s) {
  const Rn u0 = s.u, u1 = s.v, u2 = s.w, M = s.M, I = s.I;
  const Rn RHO0 = a.rho0;
  const Rn rr = RHO0 / Rn(s.rho_p);
  Rn fh0, fh1, fh2;
  DiskTerms t = {};
  if (a.motion == MOTION_OSCILLATE) {
    t.b = -(a.osc_u * cos(((Rn(2.0) * Rn(a.pi)) * Rn((double)kk) / Rn(a.osc_period)).v));
    fh0 = rr * M * (Rn(t.b) - u0);
    fh1 = rr * M * (Rn(0.0) - u1);
    fh2 = rr * I * (Rn(0.0) - u2);
  } else {
    fh0 = rr * M * (u0 - Rn(s.uo));
    fh1 = rr * M * (u1 - Rn(s.vo));
    fh2 = rr * I * (u2 - Rn(s.wo));
    t.hx = (fh0 / M).v;
    t.hy = (fh1 / M).v;
    t.ht = (fh2 / I).v;
    t.cx = (Rn(s.fcx) / M).v;
    t.cy = (Rn(s.fcy) / M).v;
    t.b = ((Rn(1.0) - RHO0 / Rn(s.rho_p)) * Rn(a.gravity)).v;
  }
  s.fhx = fh0.v;
  s.fhy = fh1.v;
  s.fht = fh2.v;
  return t;
}

__device__ __forceinline__ void newton_update(const ParticleArgs& a, const DiskTerms& t,
                                              DiskStep& s) {
  const Rn u0 = s.u, u1 = s.v, u2 = s.w, M = s.M, I = s.I;
  Rn v0, v1, v2;
  if (a.motion == MOTION_OSCILLATE) {
    v0 = t.b;
    v1 = 0.0;
    v2 = 0.0;
  } else {
    v0 = u0 + Rn(s.fx) / M + Rn(t.hx) + Rn(t.cx);
    v1 = u1 + Rn(s.fy) / M + Rn(t.hy) + Rn(t.b) + Rn(t.cy);
    v2 = u2 + Rn(s.tz) / I + Rn(t.ht);
  }
  s.x = (Rn(s.x) + Rn(0.5) * (v0 + u0)).v;
  s.y = (Rn(s.y) + Rn(0.5) * (v1 + u1)).v;
  if (a.integrate_angle) s.ang = (Rn(s.ang) + Rn(0.5) * (v2 + u2)).v;
  s.uo = u0.v;
  s.vo = u1.v;
  s.wo = u2.v;
  s.u = v0.v;
  s.v = v1.v;
  s.w = v2.v;
}

}  // namespace lbm
