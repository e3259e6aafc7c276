// lbm_steps.cuh -- several time steps of a small simulation in one launch.
//
// A small lattice does not fill the GPU for long: 201 x 601 nodes are two
// passes of one 512-thread block per SM, and what a step takes in kernels of
// its own (9.7 us FP64, 8.6 us FP32) is the chain of two dependent kernels,
// their start-up and the particle kernel's own latency.  k_steps stays resident over many steps
// (a cooperative launch, one block per SM): each block owns a contiguous range
// of 32-node row segments, the populations stay in L2 (17 MB of the 126 MB at
// that size), and the only synchronisation between blocks is one grid-wide
// barrier per step.  It takes 7.2 us (FP64) and 6.3 us (FP32): about 2 us the
// barrier, 1 us the disk's update, the rest the node arithmetic; a history
// record every step costs 0.6 us more.
//
// There is no particle kernel: every block holds the state of all disks in
// shared memory and updates all of them, from the same inputs and so to the
// same bits (lbm_disk.cuh); the blocks exchange nothing but the force sums
// and the populations.  The block that owns a disk (disk mod blocks) writes
// its history record and clears its accumulators (three sets: step k adds to
// one, reads the previous step's and clears the next step's).  The warps that
// update the disks do that first; the others meanwhile take the segments that
// no disk reaches by the previous step's positions, and after one block-wide
// barrier the rest is done with the new positions.  Pair lists and the list
// of disks that reach the block's rows are kept with a skin of 2 lu and
// rebuilt, in every block at the same step, when some disk has moved 1 lu.
//
// Everything that another block writes during the launch is read past the L1
// cache (ld.global.cg).
#pragma once

#include "lbm_disk.cuh"
#include "lbm_lattice.cuh"

namespace lbm {

constexpr int STEPS_TPB = 512;
constexpr int STEPS_WARPS = STEPS_TPB / 32;

struct StepsShared {
  double rec[PS][STEPS_MAX_DISKS];     // disk records (P_X, P_Y: pos instead)
  double pos[2][2][STEPS_MAX_DISKS];   // centres of step k at [k & 1]
  double ref[2][STEPS_MAX_DISKS];      // centres at the last list build
  double term[6][STEPS_MAX_DISKS];     // DiskTerms of the next update
  unsigned char nbr[MAX_NEIGH][STEPS_MAX_DISKS];
  int nn[STEPS_MAX_DISKS];
  int idx[STEPS_MAX_DISKS];            // disks that may reach the block's rows
  int wcount[STEPS_WARPS];
  int late[STEPS_MAX_SEGS];            // segments that wait for the disks
  int next, next_late, n_late;         // the block's segment queues
  unsigned long long mass;
  double stale;                        // D_PW left by the previous step
  int n, moved, stop;
  long long kk_stop;                   // the step at which stop was set
};
static_assert(STEPS_MAX_DISKS <= 256, "pair lists hold byte indices");

// The block's listed disks at centres pos, as node_force reads them.
struct BlockCand {
  const StepsShared& S;
  const double* px;
  const double* py;
  int n;
  unsigned long long* acc;  // the step's force accumulators
  static constexpr int CAP = STEPS_MAX_DISKS;
  __device__ __forceinline__ unsigned long long* facc(const LatticeArgs&) const { return acc; }
  __device__ __forceinline__ double x(int c) const { return px[S.idx[c]]; }
  __device__ __forceinline__ double y(int c) const { return py[S.idx[c]]; }
  __device__ __forceinline__ double diam(int c) const { return S.rec[P_D][S.idx[c]]; }
  __device__ __forceinline__ double u(int c) const { return S.rec[P_U][S.idx[c]]; }
  __device__ __forceinline__ double v(int c) const { return S.rec[P_V][S.idx[c]]; }
  __device__ __forceinline__ double w(int c) const { return S.rec[P_W][S.idx[c]]; }
  __device__ __forceinline__ int id(int c) const { return S.idx[c]; }
};

// Pair lists and the block's disk list from the centres at parity b (the
// whole block calls it).
static __device__ __noinline__ void steps_lists(const ParticleArgs& p, StepsShared& S, int b, int row0, int row1) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double *X = S.pos[b][0], *Y = S.pos[b][1], *D = S.rec[P_D];
  bool need = false;
  if (tid < p.np) {
    const double x = X[tid], y = Y[tid], d = D[tid];
    S.ref[0][tid] = x;
    S.ref[1][tid] = y;
    int nn = 0;
    for (int o = 0; o < p.np; ++o) {
      if (o == tid || !pair_near(x, y, d, X[o], Y[o], D[o], p.rep_zeta + SKIN)) continue;
      if (nn < MAX_NEIGH) S.nbr[nn++][tid] = (unsigned char)o;
      else atomicOr(p.status, ST_OVERFLOW);
    }
    S.nn[tid] = nn;
    const double r = 0.5 * d + 0.5 * p.zeta + 1.0 + SKIN;
    need = !(y + r < (double)row0 || y - r > (double)row1);
  }
  const unsigned m = __ballot_sync(0xffffffffu, need);
  if (lane == 0) S.wcount[warp] = __popc(m);
  __syncthreads();
  int before = 0, total = 0;
  for (int w = 0; w * 32 < p.np; ++w) {
    if (w < warp) before += S.wcount[w];
    total += S.wcount[w];
  }
  const int pos = before + __popc(m & ((1u << lane) - 1));
  if (need && LBM_IN(pos, STEPS_MAX_DISKS, p.status)) S.idx[pos] = tid;
  if (tid == 0) S.n = total;
  __syncthreads();
}

// Disk tid between two steps (the warps with a disk call it): what the update
// of step kk needs beside the force -- repulsion and the internal-mass terms.
// Done while the grid barrier is waited for.
__device__ __forceinline__ void steps_disk_terms(const ParticleArgs& p, StepsShared& S,
                                                 long long kk) {
  const int id = threadIdx.x;
  double D_PW = S.stale;
  if (id < p.np) {
    const double *X = S.pos[(kk - 1) & 1][0], *Y = S.pos[(kk - 1) & 1][1];
    const double px = X[id], py = Y[id], pd = S.rec[P_D][id];
    double wf[4][2], fcx = 0.0, fcy = 0.0;
    if (p.wall_model != 2) {
#pragma unroll
      for (int iw = 1; iw <= 4; ++iw) D_PW = wall_force(p, iw, px, py, pd, wf[iw - 1]);
    }
    int nn = S.nn[id];
    if (!LBM_IN(nn, MAX_NEIGH + 1, p.status)) nn = 0;
    for (int k = 0; k < nn; ++k) {  // pairs, then walls 1 to 4: the reference's order
      const int o = S.nbr[k][id];
      if (!LBM_IN(o, p.np, p.status)) continue;
      const double ox = X[o], oy = Y[o], od = S.rec[P_D][o];
      if (!pair_near(px, py, pd, ox, oy, od, p.rep_zeta)) continue;
      double F[2];
      if (o < id) {
        pair_force(p, ox, oy, od, px, py, pd, S.stale, F);
        fcx = fcx - F[0];
        fcy = fcy - F[1];
      } else {
        pair_force(p, px, py, pd, ox, oy, od, S.stale, F);
        fcx = fcx + F[0];
        fcy = fcy + F[1];
      }
    }
    if (p.wall_model != 2) {
#pragma unroll
      for (int iw = 0; iw < 4; ++iw) {
        fcx = fcx + wf[iw][0];
        fcy = fcy + wf[iw][1];
      }
    }
    DiskStep d;
    d.u = S.rec[P_U][id];
    d.v = S.rec[P_V][id];
    d.w = S.rec[P_W][id];
    d.uo = S.rec[P_UO][id];
    d.vo = S.rec[P_VO][id];
    d.wo = S.rec[P_WO][id];
    d.rho_p = S.rec[P_RHO][id];
    d.M = S.rec[P_M][id];
    d.I = S.rec[P_I][id];
    d.fcx = fcx;
    d.fcy = fcy;
    const DiskTerms t = newton_terms(p, kk, d);
    S.term[0][id] = t.hx;
    S.term[1][id] = t.hy;
    S.term[2][id] = t.ht;
    S.term[3][id] = t.cx;
    S.term[4][id] = t.cy;
    S.term[5][id] = t.b;
    S.rec[P_FCX][id] = fcx;
    S.rec[P_FCY][id] = fcy;
    S.rec[P_FHX][id] = d.fhx;
    S.rec[P_FHY][id] = d.fhy;
    S.rec[P_FHT][id] = d.fht;
  }
  // D_PW of the last disk, for the next step (the pairs above read the old)
  const int nw = (p.np + 31) / 32;
  if (nw == 1) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"r"(nw * 32) : "memory");
  if (id == p.np - 1) S.stale = D_PW;
}

// Update of disk tid in step kk (launch step s) from the force sums; then, in
// the block that owns the disk, the cleared accumulators, the history and the
// status bits.
__device__ __forceinline__ void steps_disk_update(const ParticleArgs& p, const StepsArgs& q,
                                                  StepsShared& S, long long kk, int s) {
  const int id = threadIdx.x;
  if (id >= p.np) return;
  const int st = p.npad;
  DiskStep d;
  if (s > 1 || q.decode0) {
    const unsigned long long* acc = q.facc + (long long)((q.facc0 + s - 1) % 3) * 6 * st + id;
    unsigned long long w[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = __ldcg(acc + (long long)k * st);
    d.fx = decode_force(w[0], w[1]);
    d.fy = decode_force(w[2], w[3]);
    d.tz = decode_force(w[4], w[5]);
  } else {
    d.fx = S.rec[P_FX][id];
    d.fy = S.rec[P_FY][id];
    d.tz = S.rec[P_TZ][id];
  }
  const DiskTerms t = {S.term[0][id], S.term[1][id], S.term[2][id],
                       S.term[3][id], S.term[4][id], S.term[5][id]};
  d.x = S.pos[(kk - 1) & 1][0][id];
  d.y = S.pos[(kk - 1) & 1][1][id];
  d.ang = S.rec[P_ANG][id];
  d.u = S.rec[P_U][id];
  d.v = S.rec[P_V][id];
  d.w = S.rec[P_W][id];
  d.M = S.rec[P_M][id];
  d.I = S.rec[P_I][id];
  newton_update(p, t, d);
  S.pos[kk & 1][0][id] = d.x;
  S.pos[kk & 1][1][id] = d.y;
  S.rec[P_ANG][id] = d.ang;
  S.rec[P_U][id] = d.u;
  S.rec[P_V][id] = d.v;
  S.rec[P_W][id] = d.w;
  S.rec[P_UO][id] = d.uo;
  S.rec[P_VO][id] = d.vo;
  S.rec[P_WO][id] = d.wo;
  S.rec[P_FX][id] = d.fx;
  S.rec[P_FY][id] = d.fy;
  S.rec[P_TZ][id] = d.tz;
  const double tx = d.x - S.ref[0][id], ty = d.y - S.ref[1][id];
  if (!(tx * tx + ty * ty <= 0.25 * SKIN * SKIN)) S.moved = 1;
  if (id % (int)gridDim.x != (int)blockIdx.x) return;
  unsigned long long* nxt = q.facc + (long long)((q.facc0 + s + 1) % 3) * 6 * st + id;
#pragma unroll
  for (int k = 0; k < 6; ++k) nxt[(long long)k * st] = 0ull;
  if (!isfinite(d.x) || !isfinite(d.y) || !isfinite(d.u) || !isfinite(d.v) || !isfinite(d.fx) ||
      !isfinite(d.fy) || !isfinite(d.tz))
    atomicOr(p.status, ST_NAN);
  else if (d.x < 0.0 || d.x > (double)p.nx || d.y < 0.0 || d.y > (double)p.ny)
    atomicOr(p.status, ST_PARTICLE);
  if (p.series != nullptr && p.series_every > 0 && kk % p.series_every == 0 && id < p.series_np) {
    const long long slot = (kk / p.series_every - 1) % p.series_cap;
    const long long off = slot * p.series_len + 2 + 12LL * id;
    if (LBM_IN(off + 11, (long long)p.series_cap * p.series_len, p.status)) {
      double* r = p.series + off;
      r[0] = d.x; r[1] = d.y; r[2] = d.ang;
      r[3] = d.u; r[4] = d.v; r[5] = d.w;
      r[6] = d.fx; r[7] = d.fy; r[8] = d.tz;
      r[9] = S.rec[P_FHX][id]; r[10] = S.rec[P_FHY][id]; r[11] = S.rec[P_FHT][id];
    }
  }
  if (p.hist && kk < p.hist_n && LBM_IN(kk, p.hist_n, p.status)) {
    double* h = p.hist + kk * (long long)PS * st + id;
    for (int f = 2; f < PS; ++f) h[(long long)f * st] = S.rec[f][id];
    h[P_X * (long long)st] = d.x;
    h[P_Y * (long long)st] = d.y;
  }
}

template <class T, bool STRESS>
__global__ void __launch_bounds__(STEPS_TPB, 1)
    k_steps(const LatticeArgs a, const ParticleArgs p, const StepsArgs q) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  StepsShared& S = *reinterpret_cast<StepsShared*>(s_raw);
  constexpr bool F64 = sizeof(T) == 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Geometry& g = a.g;
  const Model& m = a.m;
  const int spr = (g.nx + 32) / 32;  // 32-node segments per row
  const int nseg = spr * (g.ny + 1);
  const int seg0 = (int)((long long)nseg * blockIdx.x / gridDim.x);
  const int seg1 = (int)((long long)nseg * (blockIdx.x + 1) / gridDim.x);
  const int row0 = seg0 / spr, row1 = (seg1 - 1) / spr;
  // row of a segment: exact for fewer than 2^21 of them
  const float inv_spr = 1.0f / (float)spr;
  auto row_of = [&](int seg) { return (int)(((float)seg + 0.5f) * inv_spr); };
  // ---- the state of step kk0 ----------------------------------------------
  for (int e = tid; e < PS * p.np; e += STEPS_TPB) {
    const int f = e / p.np, id = e - f * p.np;
    const double v = __ldcg(q.ps[0] + (long long)f * p.npad + id);
    S.rec[f][id] = v;
    if (f == P_X || f == P_Y) S.pos[q.kk0 & 1][f == P_X ? 0 : 1][id] = v;
  }
  if (tid == 0) {
    S.stop = timed_out(a.status) ? 1 : 0;
    S.moved = S.n = 0;
    S.kk_stop = q.kk0;
    S.next = S.next_late = S.n_late = 0;
    S.mass = 0ull;
    S.stale = __ldcg(q.stale + q.stale0);
  }
  __syncthreads();
  if (p.np > 0) steps_lists(p, S, (int)(q.kk0 & 1), row0, row1);
  const bool disk_warp = warp * 32 < p.np;
  if (disk_warp) steps_disk_terms(p, S, q.kk0 + 1);
  for (int s = 1; s <= q.nsteps && !S.stop; ++s) {
    const long long kk = q.kk0 + s;
    const bool rec = p.series != nullptr && p.series_every > 0 && kk % p.series_every == 0;
    const long long from = (s - 1) & q.mask, to = s & q.mask;
    const StepIO<T> io{reinterpret_cast<const T*>(q.f + from * q.f_stride),
                       reinterpret_cast<T*>(q.f + to * q.f_stride),
                       reinterpret_cast<const T*>(q.om + from * q.om_stride),
                       reinterpret_cast<T*>(q.om + to * q.om_stride), kk};
    unsigned long long* const facc = q.facc + (long long)((q.facc0 + s) % 3) * 6 * p.npad;
    long long mass_q = 0;
    // one segment of 32 nodes; nc listed disks at the centres of step kk
    auto segment = [&](int seg, int nc) {
      const int j = row_of(seg), i0 = (seg - j * spr) * 32, i = i0 + lane;
      if (!LBM_IN(seg - seg0, seg1 - seg0, a.status) || !LBM_IN(j, g.ny + 1, a.status) ||
          !LBM_IN(i0, g.nx + 1, a.status))
        return;
      const bool act = i <= g.nx;
      const long long nd = (long long)j * g.pitch + i;
      NodeVals<T> v;
      T omn = (T)0;
      if (act) {
        if (STRESS && m.bingham) omn = __ldcg(io.om_src + nd);
        // a segment with an edge node takes the general gather in every lane
        // (it costs the interior lanes a few selects, not a second pass)
        if (i0 > 0 && i0 + 32 <= g.nx && j > 0 && j < g.ny)
          pull_interior<T, true>(io.src, g, nd, v.f);
        else if (m.bc == BC_EQUILIBRIUM && (i == 0 || i == g.nx || j == 0 || j == g.ny))
          edge_equilibrium<T, true>(a, i, j, (int)((kk - 1) & 1), v.f);
        else
          pull_bc<T, true>(io.src, g, m.bc, i, j, v.f);
      } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) v.f[k] = (T)0;
      }
      bool waited = true;
      const BlockCand C{S, S.pos[kk & 1][0], S.pos[kk & 1][1], nc, facc};
      node_force<T, false, void>(a, C, (T*)nullptr, i, j, act, lane, waited, v);
      if (rec && act)
        mass_q += F64 ? __double2ll_rn((double)v.drho * MASS_FIX) : mass_share32((float)v.drho);
      if (act) node_collide<T, STRESS>(a, io, v, i, j, nd, omn);
    };
    // Whether a listed disk may reach the segment in this step, by its centre
    // before the update (a disk moves less than the skin in a step, as the
    // particle kernel's tile lists assume too).
    auto may_reach = [&](int seg) {
      const double *X = S.pos[(kk - 1) & 1][0], *Y = S.pos[(kk - 1) & 1][1];
      const int j = row_of(seg), i0 = (seg - j * spr) * 32;
      for (int c0 = 0; c0 < S.n; c0 += 32) {
        bool nr = false;
        const int id = c0 + lane < S.n ? S.idx[c0 + lane] : -1;
        if (id >= 0 && LBM_IN(id, p.np, a.status)) {
          const double dl = (double)i0 - X[id], dr = dl + 31.0;
          const double dx = dl > 0.0 ? dl : (dr < 0.0 ? -dr : 0.0), dy = (double)j - Y[id];
          const double reach = 0.5 * S.rec[P_D][id] + 0.5 * m.zeta + 1.0 + SKIN;
          nr = dx * dx + dy * dy < reach * reach;
        }
        if (__any_sync(0xffffffffu, nr)) return true;
      }
      return false;
    };
    // next entry of a queue of the block, -1 when it is empty
    auto take = [&](int* ctr, int n) {
      int e = 0;
      if (lane == 0) e = atomicAdd(ctr, 1);
      e = __shfl_sync(0xffffffffu, e, 0);
      return e < n ? e : -1;
    };
    if (disk_warp) {
      steps_disk_update(p, q, S, kk, s);
      __syncwarp();
    }
    for (int e; (e = take(&S.next, seg1 - seg0)) >= 0;) {
      if (S.n > 0 && may_reach(seg0 + e)) {
        if (lane == 0) {
          const int w = atomicAdd(&S.n_late, 1);
          if (LBM_IN(w, STEPS_MAX_SEGS, a.status)) S.late[w] = seg0 + e;
        }
      } else {
        segment(seg0 + e, 0);
      }
    }
    if (p.np > 0) {
      __syncthreads();
      if (S.moved) {  // the same in every block
        steps_lists(p, S, (int)(kk & 1), row0, row1);
        if (tid == 0) S.moved = 0;  // read again only after the grid barrier
      }
      for (int e; (e = take(&S.next_late, S.n_late)) >= 0;) segment(S.late[e], S.n);
    }
    if (rec) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mass_q += __shfl_down_sync(0xffffffffu, mass_q, o);
      if (lane == 0 && mass_q != 0) atomicAdd(&S.mass, (unsigned long long)mass_q);
      __syncthreads();
      if (tid == 0) {
        const long long slot = (kk / p.series_every - 1) % p.series_cap;
        const bool in = LBM_IN(slot, p.series_cap, a.status);
        if (S.mass && in) atomicAdd(p.mass_acc + slot, S.mass);
        S.mass = 0ull;
        if (blockIdx.x == 0 && in) {
          p.series[slot * p.series_len + 0] = (double)kk;
          p.series[slot * p.series_len + 1] = __longlong_as_double(0x7ff8000000000000LL);
        }
      }
    }
    // ---- to the next step: the last warp keeps the barrier, the first ones
    //      prepare the disks meanwhile
    __syncthreads();
    if (s == q.nsteps) break;
    if (tid == STEPS_TPB - 32) {
      S.next = S.next_late = S.n_late = 0;
      grid_arrive(q.bar);
      if (!grid_wait(q.bar, q.bar0 + (unsigned)s * gridDim.x, a.status)) {
        S.stop = 1;
        S.kk_stop = kk;
      }
    }
    if (disk_warp) steps_disk_terms(p, S, kk + 1);
    __syncthreads();
  }
  // ---- the state of the last step, into the other copy (a block that starts
  //      late may still be reading the first); after an expired wait too, as
  //      the host goes on with that copy ---------------------------------------
  if (blockIdx.x == 0) {
    const long long kk = S.stop ? S.kk_stop : q.kk0 + q.nsteps;
    for (int e = tid; e < PS * p.np; e += STEPS_TPB) {
      const int f = e / p.np, id = e - f * p.np;
      const double v = f == P_X || f == P_Y ? S.pos[kk & 1][f == P_X ? 0 : 1][id] : S.rec[f][id];
      q.ps[1][(long long)f * p.npad + id] = v;
    }
    if (tid == 0) {
      q.stale[q.stale0 ^ 1] = S.stale;
      *p.kk = kk;
    }
  }
}

template <class T>
cudaError_t launch_steps(const LatticeArgs& a, const ParticleArgs& p, const StepsArgs& q,
                         cudaStream_t s, int grid) {
  const int sx = (a.m.bingham || a.m.record_stress) ? 1 : 0;
  void (*const kern)(const LatticeArgs, const ParticleArgs, const StepsArgs) =
      sx ? k_steps<T, true> : k_steps<T, false>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(StepsShared));
  if (e != cudaSuccess) return e;
  LatticeArgs la = a;
  ParticleArgs pa = p;
  StepsArgs qa = q;
  void* args[] = {&la, &pa, &qa};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(grid),
                                     dim3(STEPS_TPB), args, sizeof(StepsShared), s);
}

}  // namespace lbm
