// Direct-forcing IBM on the device (crates/lbm-core/src/solver.rs:3016-3282).
//
// The reference runs this on the host over full-grid f64 arrays. Here only
// the stencil cells ("slots") are touched, and one call is one kernel of one
// thread-block cluster per body (ibm_chain), whose phases are separated by
// hardware cluster barriers:
//   prep     per slot:   rho, u_now from the populations (and the cleared field)
//   impulse  per marker: um, mobility, impulse, represented force
//   spread   per slot:   spread / du gathered in marker order
//   slip     per marker: slip statistics of the sweep, and the impulse of the
//                        next one (it interpolates the same velocity)
//   commit   per slot:   force field += spread (storage precision)
// A sweep is spread + slip; every block reduces the largest slip by itself
// and takes the reference's early exit, so no host round trip and no launch
// of a sweep that is not run.
//
// What bounds it: latency. The data (a few MB) sits in L2 and each phase is
// two or three dependent gathers, so the time is the number of phases times
// (gathers + barrier). Per runner step on B200, as 2 + 3 x sweeps dependent
// kernels -> in this form: 46.2 -> 22.0 us (48 x 48 x 60 tank, 1,139 slots; 20
// us of it the call), 74.7 -> 36.9 us (96 x 96 x 120), 133 -> 88 us (128 x 128
// x 160, D3Q19); 121 -> 117 us (128 x 128 x 160, D3Q27, pair sweep) and 415 ->
// 399 us (256 x 256 x 320, fp16), where the sweep hides it. Bodies of many more
// markers take the wide form at the end of this file.
//
// Summation order: per slot the contributions are gathered in ascending
// marker order (the reference's loop order), so spread, du and the cell
// kernel sum are bit-identical to the reference; the global diagnostics
// are fixed-order tree sums over 32-entry chunks (independent of the block
// size, deterministic run to run).
#pragma once
#include "common.cuh"
#include "lattice.cuh"
#include "quotient.hpp"

namespace lbmb {

// Blocks of a body's cluster. A block takes all registers of its SM where one
// body is forced beside a full-grid sweep: next to the sweep's own blocks the
// phases' gathers wait behind its accesses (128 x 128 x 160 tank: 80-100 us
// for the call with 16 blocks of 256 threads among the sweep's).
constexpr int IBM_CLUSTER = 8;
// Entries per partial sum of the global diagnostics.
constexpr int IBM_CHUNK = 32;

// All threads of the cluster; writes before it are visible after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

struct IbmDiagDev {
  double slip_max, slip_rms, slip_max_rel, slip_rms_rel;
  double torque[3], fluid_force[3], marker_force[3];
  double momentum_error_rel;
  int iterations;
  int pad;
};

struct IbmWide;

struct IbmArgs {
  // markers
  int64_t nm;
  const double* pos;     // nm x 3
  const double* weight;  // nm
  const int32_t* st_off;   // nm + 1
  const int32_t* st_slot;  // active (non-solid) stencil points -> global slot
  const double* st_w;
  const double* st_cks;    // cell kernel sum of the point's cell (this body)
  const double* wsum;      // nm: sum of the marker's weights
  // slots touched by this body
  int64_t ns;
  const int32_t* bslot;    // body slot -> global slot
  const int4* brec;        // body slot -> {global slot, cell, solid-neighbour mask, 0}
  const int32_t* cs_off;   // ns + 1, contributions in marker order
  const int32_t* cs_marker;
  const double* cs_w;
  // per global slot state
  double* rho;       // cached density (f64 view)
  double* u_now;     // x3
  double* du;        // x3
  double4* urec;     // {u_now + du, 1 / rho}: what a marker gathers from a slot
  double* spread;    // x3
  // per marker state
  double* imp;       // x3
  double* mob;
  double* inv_mob;   // reciprocal(mob)
  double* rmf;       // x3 represented marker force of this sweep
  // partials
  double* part_spread;  // 2 x ceil(ns / IBM_CHUNK) x 3 (two sweeps in flight)
  double* part_diag;    // 2 x ceil(nm / IBM_CHUNK) x 9 (8 sums, then the maxima)
  IbmDiagDev* diag;
  IbmWide* wide;        // state of the wide form
  double center[3], omega[3];
  double scale, relax, tol;
};

__device__ __forceinline__ void ibm_target(const IbmArgs& a, int64_t m, double t[3], double r[3]) {
  r[0] = a.pos[3 * m + 0] - a.center[0];
  r[1] = a.pos[3 * m + 1] - a.center[1];
  r[2] = a.pos[3 * m + 2] - a.center[2];
  t[0] = a.omega[1] * r[2] - a.omega[2] * r[1];
  t[1] = a.omega[2] * r[0] - a.omega[0] * r[2];
  t[2] = a.omega[0] * r[1] - a.omega[1] * r[0];
}

// Where post-stream population q of a cell sits in the swapped AA layout
// (parity 1), as an element offset. A select of addresses and no branch: with
// a load behind a branch per direction the Q loads of a cell follow each
// other (19 x ~700 cycles in the direct forcing's first phase, measured with
// the clock register; ~3,000 in all as one batch).
// 32-bit offsets (Q x plane < 2^31): in 64 bits their registers halve the
// blocks of a kernel of 27 directions (total mass of a 240^3 D3Q27 grid, the
// whole call, 0.80 ms against 0.39).
template <int Q>
__device__ __forceinline__ uint32_t post_stream_offset(uint32_t pl, uint32_t cell, const Nbr& nb, uint32_t mask,
                                                       int q) {
  using L = Lat<Q>;
  const int o = opp(q);
  const bool wall = (mask >> o) & 1u;
  uint32_t e = wall ? q * pl + cell : o * pl + uint32_t(nb.at(-L::cx(q), -L::cy(q), -L::cz(q)));
  if (slips_in<Q>(q)) {
    const bool slip = wall && (mask & NBR_SLIP) && !((mask >> planar<Q>(o)) & 1u);
    e = slip ? opp(mirror_z<Q>(q)) * pl + uint32_t(nb.at(-L::cx(q), -L::cy(q), 0)) : e;
  }
  return e;
}

// Post-stream populations of one cell in the AA layout of the given parity
// (0: normal, 1: swapped after an even step), as the arithmetic type.
template <int Q, class S>
__device__ __forceinline__ void load_post_stream(const S* fb, int64_t pl, int64_t cell, int x, int y,
                                                 int z, int nx, int ny, int nz, uint32_t mask,
                                                 int parity, typename Codec<S>::A (&f)[Q]) {
  using L = Lat<Q>;
  if (parity == 0) {
#pragma unroll
    for (int q = 0; q < Q; ++q) f[q] = Codec<S>::ld(fb + q * pl + cell);
  } else {
    const Nbr nb(x, y, z, nx, ny, nz);
#pragma unroll
    for (int q = 0; q < Q; ++q)
      f[q] = Codec<S>::ld(fb + post_stream_offset<Q>(uint32_t(pl), uint32_t(cell), nb, mask, q));
  }
}

template <int N>
__device__ __forceinline__ void block_sum(double (&v)[N], double* sh) {
  // sh: N * (blockDim/32) doubles. Fixed-order warp + block tree.
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  if (lane == 0)
    for (int k = 0; k < N; ++k) sh[k * nw + wid] = v[k];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 0; k < N; ++k) {
      double s = 0.0;
      for (int w = 0; w < nw; ++w) s += sh[k * nw + w];
      v[k] = s;
    }
}

// What one apply_rotating_ibm call works on besides the body.
template <class S>
struct IbmRun {
  using A = typename Codec<S>::A;
  const S* fb;
  int64_t pl;
  int nx, ny, nz, parity;
  Vec4<A>* fcur;       // force field by global slot
  int64_t nslots;
  int field_at_call;   // fcur counts in u_now
  int clear;           // fcur is zeroed first (only without field_at_call)
  int sweeps;
  double gx, gy, gz;   // uniform force
  // per-step series (null: not recorded)
  double* series_torque;
  double* series_ff;
  int32_t* series_iters;
  int64_t* step_counter;
  // where the adjoint keeps the intermediates of the step (null: not kept):
  // rho, u_now (per slot), mobility (per marker), du at the start of each
  // sweep (per slot, sv_slots rows) and each sweep's impulse (per marker)
  double *sv_rho, *sv_u, *sv_mob, *sv_du, *sv_imp;
  int64_t sv_slots;
};

// u_now over the body's slots (solver.rs:3036-3087): cached rho (storage
// arithmetic: 1 + sum f) and (sum c f + F/2) / rho in f64 with the force
// field current at call time.
template <int Q, class S>
__device__ __forceinline__ void ibm_prep_slot(const IbmArgs& a, const IbmRun<S>& r, int64_t i) {
  using A = typename Codec<S>::A;
  using L = Lat<Q>;
  const int4 rec = a.brec[i];
  const int32_t g = rec.x;
  const int64_t cell = rec.y;
  const uint32_t mask = uint32_t(rec.z);  // zero away from solids
  const int nxy = r.nx * r.ny;
  const int z = rec.y / nxy, yx = rec.y - z * nxy, y = yx / r.nx, x = yx - y * r.nx;
  A f[Q];
  load_post_stream<Q, S>(r.fb, r.pl, cell, x, y, z, r.nx, r.ny, r.nz, mask, r.parity, f);
  A dr = A(0);
  double mom[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    dr = dr + f[q];
    const double fq = double(f[q]);
    mom[0] += double(L::cx(q)) * fq;
    mom[1] += double(L::cy(q)) * fq;
    mom[2] += double(L::cz(q)) * fq;
  }
  const double rho = double(A(1) + dr);
  double force[3] = {r.gx, r.gy, r.gz};
  if (r.field_at_call) {
    const Vec4<A> fc = r.fcur[g];
    force[0] += double(fc.x);
    force[1] += double(fc.y);
    force[2] += double(fc.z);
  }
  const double inv_rho = 1.0 / fmax(rho, 1.0e-30);
  a.rho[g] = rho;
  if (r.sv_rho) r.sv_rho[g] = rho;
  double u3[3];
  for (int k = 0; k < 3; ++k) {
    const double u = (mom[k] + 0.5 * force[k]) * inv_rho;
    u3[k] = u;
    a.u_now[3 * g + k] = u;
    if (r.sv_u) r.sv_u[3 * g + k] = u;
  }
  a.urec[g] = make_double4(u3[0], u3[1], u3[2], inv_rho);
}

// Row of a marker's stencil points, or of a slot's contributions: its range
// and the first NB indices. These never change between calls, and a thread
// loads its first row of each kind at the start of the kernel, so that every
// phase begins with its gather instead of two dependent index loads.
template <int NB>
struct IbmIndex {
  int32_t k0, k1, at[NB];
  __device__ __forceinline__ void load(const int32_t* off, const int32_t* index, int64_t row) {
    k0 = off[row];
    k1 = off[row + 1];
#pragma unroll
    for (int j = 0; j < NB; ++j) at[j] = k1 > k0 ? index[k0 + j < k1 ? k0 + j : k1 - 1] : 0;
  }
};

// Interpolated velocity of a marker from its stencil points [k0, k1) in
// order, NB gathers in flight (points past the end repeat the last one with
// weight 0), and, with MOB, its mobility (solver.rs:3131-3140).
template <int NB, bool MOB>
__device__ __forceinline__ void ibm_marker_velocity(const IbmArgs& a, const IbmIndex<NB>& ix, double (&um)[3],
                                                    double& mobility) {
  const int32_t k0 = ix.k0, k1 = ix.k1;
  um[0] = um[1] = um[2] = 0.0;
  mobility = 0.0;
  for (int32_t k = k0; k < k1; k += NB) {
    double w[NB], n[NB], rho[NB];
    double4 v[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const bool in = k + j < k1;
      const int32_t kk = in ? k + j : k1 - 1;
      const int32_t s = k == k0 ? ix.at[j] : a.st_slot[kk];
      v[j] = a.urec[s];
      w[j] = in ? a.st_w[kk] : 0.0;
      if (MOB) {
        n[j] = a.st_cks[kk];
        rho[j] = a.rho[s];
      }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      um[0] += w[j] * v[j].x;
      um[1] += w[j] * v[j].y;
      um[2] += w[j] * v[j].z;
      if (MOB) mobility += quotient(w[j] * n[j], fmax(rho[j], 1.0e-30), v[j].w);
    }
  }
}

// Impulse of a marker from the interpolated velocity (solver.rs:3118-3173),
// none without mobility. The quotients here and in the mobility round as the
// reference's divisions: plain products with the reciprocals differ in the
// last place, and now and then a force in 32 bits with them, which a long
// 16-bit run amplifies. Divisions proper call a subroutine, whose register
// limits make the phases spill: 48 x 48 x 60 and 96 x 96 x 120 tank 22.8 and
// 39.4 us per step, 21.5 and 37.2 us in this form.
template <class S>
__device__ __forceinline__ void ibm_impulse(const IbmArgs& a, const IbmRun<S>& r, int64_t m, const double (&t)[3],
                                            const double (&um)[3], double mob, double inv_mob, int sweep) {
  const double ws = a.wsum[m];
  for (int c = 0; c < 3; ++c) {
    const double imp = mob != 0.0 ? quotient(a.relax * (t[c] - um[c]), mob, inv_mob) : 0.0;
    a.imp[3 * m + c] = imp;
    a.rmf[3 * m + c] = imp * ws;
    if (r.sv_imp) r.sv_imp[(int64_t(sweep) * a.nm + m) * 3 + c] = imp;
  }
}

// Spread the impulses into slot i, in marker order (solver.rs:3174-3209);
// ff: the slot's share of the fluid force.
template <int NB, class S>
__device__ __forceinline__ void ibm_spread_slot(const IbmArgs& a, const IbmRun<S>& r, int sweep,
                                                const IbmIndex<NB>& ix, int32_t g, double (&ff)[3]) {
  const int32_t k0 = ix.k0, k1 = ix.k1;
  double sp[3] = {0.0, 0.0, 0.0}, d[3] = {0.0, 0.0, 0.0};
  const double inv_rho = a.urec[g].w;
  if (sweep > 0)
    for (int c = 0; c < 3; ++c) {
      sp[c] = a.spread[3 * g + c];
      d[c] = a.du[3 * g + c];
    }
  if (r.sv_du)
    for (int c = 0; c < 3; ++c) r.sv_du[(int64_t(sweep) * r.sv_slots + g) * 3 + c] = d[c];
  const double un[3] = {a.u_now[3 * g], a.u_now[3 * g + 1], a.u_now[3 * g + 2]};
  for (int32_t k = k0; k < k1; k += NB) {
    double w[NB], v[NB][3];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const bool in = k + j < k1;
      const int32_t kk = in ? k + j : k1 - 1;
      const double* im = a.imp + 3 * int64_t(k == k0 ? ix.at[j] : a.cs_marker[kk]);
      w[j] = in ? a.cs_w[kk] : 0.0;
      v[j][0] = im[0];
      v[j][1] = im[1];
      v[j][2] = im[2];
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double cf = v[j][c] * w[j];
        sp[c] += cf;
        d[c] += cf * inv_rho;
        ff[c] += cf;
      }
  }
  for (int c = 0; c < 3; ++c) {
    a.spread[3 * g + c] = sp[c];
    a.du[3 * g + c] = d[c];
  }
  a.urec[g] = make_double4(un[0] + d[0], un[1] + d[1], un[2] + d[2], inv_rho);
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// First impulse of marker m, its mobility with it.
template <int NB, class S>
__device__ __forceinline__ void ibm_first_impulse(const IbmArgs& a, const IbmRun<S>& r, int64_t m,
                                                  const IbmIndex<NB>& ix) {
  double t[3], x[3], um[3], mob;
  ibm_target(a, m, t, x);
  ibm_marker_velocity<NB, true>(a, ix, um, mob);
  const double inv = reciprocal(mob);
  a.mob[m] = mob;
  a.inv_mob[m] = inv;
  if (r.sv_mob) r.sv_mob[m] = mob;
  ibm_impulse(a, r, m, t, um, mob, inv, 0);
}

// Slip statistics of marker m after sweep s (solver.rs:3211-3253): v = ssq,
// wsum, force, torque; and the next sweep's impulse.
template <int NB, class S>
__device__ __forceinline__ void ibm_slip_marker(const IbmArgs& a, const IbmRun<S>& r, int s, int64_t m,
                                                const IbmIndex<NB>& ix, double (&v)[8], double& smax) {
  double t[3], x[3], um[3], none;
  const double* f = a.rmf + 3 * m;
  const double f0 = f[0], f1 = f[1], f2 = f[2], wt = a.weight[m];
  const double mob = a.mob[m], inv = a.inv_mob[m];
  ibm_target(a, m, t, x);
  ibm_marker_velocity<NB, false>(a, ix, um, none);
  if (ix.k1 > ix.k0) {
    const double sl[3] = {t[0] - um[0], t[1] - um[1], t[2] - um[2]};
    const double s2 = sl[0] * sl[0] + sl[1] * sl[1] + sl[2] * sl[2];
    const double mag = sqrt(s2);
    smax = fmax(mag, 0.0);  // a diverged state (NaN) has no slip
    v[0] = wt * mag * mag;
    v[1] = wt;
  }
  v[2] = f0;
  v[3] = f1;
  v[4] = f2;
  v[5] = x[1] * f2 - x[2] * f1;
  v[6] = x[2] * f0 - x[0] * f2;
  v[7] = x[0] * f1 - x[1] * f0;
  if (s + 1 < r.sweeps) ibm_impulse(a, r, m, t, um, mob, inv, s + 1);
}

// Force field += spread of slot i in the storage arithmetic
// (solver.rs:3256-3279).
template <class S>
__device__ __forceinline__ void ibm_commit_slot(const IbmArgs& a, const IbmRun<S>& r, int64_t i) {
  using A = typename Codec<S>::A;
  const int32_t g = a.brec[i].x;
  Vec4<A> v = r.fcur[g];
  v.x = v.x + A(a.spread[3 * g + 0]);
  v.y = v.y + A(a.spread[3 * g + 1]);
  v.z = v.z + A(a.spread[3 * g + 2]);
  r.fcur[g] = v;
}

// Diagnostics and series of a call by one warp, lane k holding the call's sum
// k (0..1 slip, 2..4 marker force, 5..7 marker torque, 8..10 fluid force); the
// torque on the body is minus the marker torque. slip_max, ssq, wsum: of the
// last sweep, done: its number.
template <class S>
__device__ __forceinline__ void ibm_write_diag(const IbmArgs& a, const IbmRun<S>& r, int lane, double run,
                                               double slip_max, double ssq, double wsum, int done) {
  IbmDiagDev* d = a.diag;
  const double sgn = lane >= 5 && lane < 8 ? -run : run;
  const double e = __shfl_sync(0xffffffffu, run, lane < 3 ? lane + 8 : 0) -
                   __shfl_sync(0xffffffffu, run, lane < 3 ? lane + 2 : 0);
  const double f = __shfl_sync(0xffffffffu, run, lane < 3 ? lane + 2 : 0);
  const double e0 = __shfl_sync(0xffffffffu, e, 0), e1 = __shfl_sync(0xffffffffu, e, 1),
               e2 = __shfl_sync(0xffffffffu, e, 2);
  const double f0 = __shfl_sync(0xffffffffu, f, 0), f1 = __shfl_sync(0xffffffffu, f, 1),
               f2 = __shfl_sync(0xffffffffu, f, 2);
  const int64_t st = r.step_counter ? *r.step_counter : 0;
  __syncwarp();
  if (lane >= 2 && lane < 5) d->marker_force[lane - 2] = run;
  if (lane >= 5 && lane < 8) d->torque[lane - 5] = sgn;
  if (lane >= 8 && lane < 11) d->fluid_force[lane - 8] = run;
  if (r.step_counter) {
    if (lane == 7 && r.series_torque) r.series_torque[st] = -sgn;
    if (lane >= 8 && lane < 11 && r.series_ff) r.series_ff[3 * st + lane - 8] = run;
  }
  if (lane == 0) {
    d->slip_max = slip_max;
    d->slip_max_rel = slip_max / a.scale;
    d->iterations = done;
    if (r.step_counter) {
      if (r.series_iters) r.series_iters[st] = done;
      *r.step_counter = st + 1;
    }
  }
  if (lane == 1) {
    const double rms = wsum > 0.0 ? sqrt(ssq / wsum) : 0.0;
    d->slip_rms = rms;
    d->slip_rms_rel = rms / a.scale;
  }
  if (lane == 11)
    d->momentum_error_rel =
        sqrt(e0 * e0 + e1 * e1 + e2 * e2) / fmax(sqrt(f0 * f0 + f1 * f1 + f2 * f2), 1.0e-12);
}

// One apply_rotating_ibm call of one body by one cluster; rank: block in the
// cluster, ncta: its blocks; NB: gathers in flight per thread. Every barrier
// is reached by every thread: the sweep loop's exit is decided from the same
// value in every block.
template <int Q, class S, int NB>
__device__ __forceinline__ void ibm_chain(const IbmArgs& a, const IbmRun<S>& r, int rank, int ncta) {
  using A = typename Codec<S>::A;
  __shared__ double tot[11];
  const int lane = int(threadIdx.x) & 31, warp = int(threadIdx.x) >> 5;
  const int64_t nthr = int64_t(ncta) * blockDim.x;
  const int64_t tid = (int64_t(warp) * ncta + rank) * 32 + lane;  // few entries spread over the blocks
  IbmIndex<NB> mine, slots;  // of this thread's first marker and first slot
  if (tid < a.nm) mine.load(a.st_off, a.st_slot, tid);
  if (tid < a.ns) slots.load(a.cs_off, a.cs_marker, tid);
  const int32_t my_slot = tid < a.ns ? a.brec[tid].x : 0;
  auto marker_row = [&](int64_t m) {
    if (m == tid) return mine;
    IbmIndex<NB> x;
    x.load(a.st_off, a.st_slot, m);
    return x;
  };
  const int64_t nc_m = (a.nm + IBM_CHUNK - 1) / IBM_CHUNK, nc_s = (a.ns + IBM_CHUNK - 1) / IBM_CHUNK;
  for (int64_t i = tid; i < a.ns; i += nthr) ibm_prep_slot<Q, S>(a, r, i);
  if (r.clear)
    for (int64_t s = tid; s < r.nslots; s += nthr) r.fcur[s] = Vec4<A>{A(0), A(0), A(0), A(0)};
  cluster_sync();
  for (int64_t m = tid; m < a.nm; m += nthr) ibm_first_impulse<NB>(a, r, m, marker_row(m));
  cluster_sync();
  // block 0: running sums of the call, thread k of the first warp holding sum
  // k of ibm_write_diag
  double run = 0.0, slip_max = 0.0, ssq = 0.0, wsum = 0.0;
  int done = 0;
  for (int s = 0; s < r.sweeps; ++s) {
    double* const ps = a.part_spread + (s & 1) * 3 * nc_s;
    double* const pd = a.part_diag + (s & 1) * 9 * nc_m;
    double* const px = pd + 8 * nc_m;
    for (int64_t i0 = tid - lane; i0 < a.ns; i0 += nthr) {
      double ff[3] = {0.0, 0.0, 0.0};
      const int64_t i = i0 + lane;
      if (i == tid && i < a.ns) {
        ibm_spread_slot<NB>(a, r, s, slots, my_slot, ff);
      } else if (i < a.ns) {
        IbmIndex<NB> ix;
        ix.load(a.cs_off, a.cs_marker, i);
        ibm_spread_slot<NB>(a, r, s, ix, a.brec[i].x, ff);
      }
      for (int c = 0; c < 3; ++c) {
        const double v = warp_sum(ff[c]);
        if (lane == 0) ps[3 * (i0 / IBM_CHUNK) + c] = v;
      }
    }
    cluster_sync();
    for (int64_t m0 = tid - lane; m0 < a.nm; m0 += nthr) {
      const int64_t m = m0 + lane;
      double v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, smax = 0.0;
      if (m < a.nm) ibm_slip_marker<NB>(a, r, s, m, marker_row(m), v, smax);
      smax = warp_max(smax);
      if (lane == 0) px[m0 / IBM_CHUNK] = smax;
      double* const p = pd + 8 * (m0 / IBM_CHUNK);
      for (int k = 0; k < 8; ++k) {
        const double y = warp_sum(v[k]);
        if (lane == 0) p[k] = y;
      }
    }
    cluster_sync();
    // the largest slip, by every warp
    double amax = 0.0;
    for (int64_t c = lane; c < nc_m; c += 32) amax = fmax(amax, px[c]);
    amax = __shfl_sync(0xffffffffu, warp_max(amax), 0);
    if (rank == 0) {
      // the first block sums the partials, one warp per sum (8 slip sums, then
      // the 3 spread sums): four sums over every 128th chunk per lane, a tree
      // for each, and the four in order, as the wide form's block of 128 does
      for (int k = warp; k < 11; k += int(blockDim.x) >> 5) {
        const double* const p = k < 8 ? pd + k : ps + k - 8;
        const int64_t n = k < 8 ? nc_m : nc_s, w = k < 8 ? 8 : 3;
        double y[4] = {0.0, 0.0, 0.0, 0.0};
        for (int64_t c = lane; c < n; c += 128)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (c + 32 * j < n) y[j] += p[w * (c + 32 * j)];
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) v += warp_sum(y[j]);
        if (lane == 0) tot[k] = v;
      }
      __syncthreads();
      if (threadIdx.x < 11) run += tot[threadIdx.x];
      slip_max = amax;
      ssq = tot[0];
      wsum = tot[1];
      __syncthreads();  // tot is written again by the next sweep
    }
    done = s + 1;
    if (!r.sv_imp && amax / a.scale <= a.tol) break;  // the adjoint records a fixed number of sweeps
  }
  // the commit by the blocks that have no diagnostics to write
  if (rank > 0 || ncta == 1) {
    const int first = ncta > 1 ? 1 : 0;
    const int64_t t0 = (int64_t(warp) * (ncta - first) + rank - first) * 32 + lane;
    const int64_t step = int64_t(ncta - first) * blockDim.x;
    for (int64_t i = t0; i < a.ns; i += step) ibm_commit_slot(a, r, i);
  }
  if (rank == 0 && warp == 0) ibm_write_diag(a, r, lane, run, slip_max, ssq, wsum, done);
}

// The sweep of the unforced cells is launched as this kernel's programmatic
// dependent: it starts once every block of the cluster runs, so that the
// cluster is resident before the sweep fills the chip.
__device__ __forceinline__ void release_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// NT threads per block and NB gathers in flight: 512 and 8 (128 registers a
// thread) or 1024 and 4 (64).
template <int Q, class S, int NT, int NB>
__global__ void __launch_bounds__(NT, 1) ibm_chain_kernel(IbmArgs a, IbmRun<S> r) {
  release_dependents();
  ibm_chain<Q, S, NB>(a, r, int(blockIdx.x), int(gridDim.x));
}

// ---- wide form ------------------------------------------------------------
// The same phases as one full-chip kernel each, for bodies of so many entries
// (slots or markers) that eight SMs take longer than the launches do. One entry
// per thread; the last block of a slip kernel sums the sweep's partials (in the
// cluster's order: both forms give the same bits) and decides the early exit,
// and every kernel of a later sweep then returns at once. Each kernel is the
// programmatic dependent of the one before and waits for its writes.
constexpr int IBM_WIDE_BLOCK = 128;
// Entries above which a call runs in this form: on its own, one round of the
// cluster's smaller blocks (call with its readback on B200, cluster / wide, one
// sweep: 3,836 slots 47 / 51 us, 4,553 48 / 53, 6,292 74 / 58, 13,694 106 / 61,
// 133,915 552 / 90; three sweeps: 3,836 74 / 74, 6,292 108 / 82).
constexpr int64_t IBM_WIDE_ALONE = IBM_CLUSTER * 512;
// Beside a sweep of n cells, which hides the cluster on its own SMs but shares
// the chip with the wide form, more of them: D3Q19 fp32 boxes, us per step with
// the cluster / wide form, one sweep and three: 64^3 4,553 slots 32 / 36 and 52
// / 53, 7,752 42 / 38 and 70 / 60, 20,421 93 / 44 and 163 / 69; 128^3 11,825 77
// / 103 and 99 / 123, 18,285 85 / 105 and 130 / 127, 30,382 121 / 109 and 200 /
// 135; 200^3 39,789 247 / 276 and 285 / 296, 63,598 283 / 281 and 423 / 316.
inline int64_t ibm_wide_beside(int64_t n) { return 6000 + n / 200; }

struct IbmWide {
  double run[11];  // sums of the call (see ibm_write_diag)
  double slip_max, ssq, wsum;
  int done, converged;
  unsigned int ticket;
  int pad;
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The phases for block `blk` of a body's blocks (all of a block's threads).
template <int Q, class S>
__device__ __forceinline__ void wide_prep(const IbmArgs& a, const IbmRun<S>& r, int64_t blk) {
  using A = typename Codec<S>::A;
  const int64_t i = blk * IBM_WIDE_BLOCK + threadIdx.x;
  if (i == 0) *a.wide = IbmWide{};
  if (i < a.ns) ibm_prep_slot<Q, S>(a, r, i);
  if (r.clear && i < r.nslots) r.fcur[i] = Vec4<A>{A(0), A(0), A(0), A(0)};
}

template <class S>
__device__ __forceinline__ void wide_impulse(const IbmArgs& a, const IbmRun<S>& r, int64_t blk) {
  const int64_t m = blk * IBM_WIDE_BLOCK + threadIdx.x;
  IbmIndex<8> ix;
  if (m < a.nm) ix.load(a.st_off, a.st_slot, m);
  pdl_wait();
  if (m < a.nm) ibm_first_impulse<8>(a, r, m, ix);
}

template <class S>
__device__ __forceinline__ void wide_spread(const IbmArgs& a, const IbmRun<S>& r, int s, int64_t blk) {
  const int64_t i = blk * IBM_WIDE_BLOCK + threadIdx.x, i0 = i - (i & 31);
  IbmIndex<8> ix;
  if (i < a.ns) ix.load(a.cs_off, a.cs_marker, i);
  pdl_wait();
  if (a.wide->converged || i0 >= a.ns) return;
  double ff[3] = {0.0, 0.0, 0.0};
  if (i < a.ns) ibm_spread_slot<8>(a, r, s, ix, a.brec[i].x, ff);
  for (int c = 0; c < 3; ++c) {
    const double v = warp_sum(ff[c]);
    if ((i & 31) == 0) a.part_spread[3 * (i0 / IBM_CHUNK) + c] = v;
  }
}

// nblk: the body's blocks.
template <class S>
__device__ __forceinline__ void wide_slip(const IbmArgs& a, const IbmRun<S>& r, int s, int64_t blk, unsigned nblk) {
  __shared__ double sh[12 * (IBM_WIDE_BLOCK / 32)];
  __shared__ bool last;
  const int64_t m = blk * IBM_WIDE_BLOCK + threadIdx.x, m0 = m - (m & 31);
  const int64_t nc_m = (a.nm + IBM_CHUNK - 1) / IBM_CHUNK, nc_s = (a.ns + IBM_CHUNK - 1) / IBM_CHUNK;
  double* const px = a.part_diag + 8 * nc_m;
  IbmIndex<8> ix;
  if (m < a.nm) ix.load(a.st_off, a.st_slot, m);
  pdl_wait();
  IbmWide* const w = a.wide;
  if (w->converged) return;  // the same in every thread: only the last block sets it, at the end
  if (m0 < a.nm) {
    double v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, smax = 0.0;
    if (m < a.nm) ibm_slip_marker<8>(a, r, s, m, ix, v, smax);
    smax = warp_max(smax);
    if ((m & 31) == 0) px[m0 / IBM_CHUNK] = smax;
    for (int k = 0; k < 8; ++k) {
      const double y = warp_sum(v[k]);
      if ((m & 31) == 0) a.part_diag[8 * (m0 / IBM_CHUNK) + k] = y;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&w->ticket, 1u) == nblk - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // thread t takes chunks t, t + 128, ... in order, then a tree
  double acc[11] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}, amax = 0.0;
  for (int64_t c = threadIdx.x; c < nc_m; c += IBM_WIDE_BLOCK) {
    amax = fmax(amax, __ldcg(px + c));
    for (int k = 0; k < 8; ++k) acc[k] += __ldcg(a.part_diag + 8 * c + k);
  }
  for (int64_t c = threadIdx.x; c < nc_s; c += IBM_WIDE_BLOCK)
    for (int k = 0; k < 3; ++k) acc[8 + k] += __ldcg(a.part_spread + 3 * c + k);
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) sh[11 * (IBM_WIDE_BLOCK / 32) + (threadIdx.x >> 5)] = amax;
  block_sum<11>(acc, sh);
  if (threadIdx.x != 0) return;
  for (int k = 0; k < IBM_WIDE_BLOCK / 32; ++k) amax = fmax(amax, sh[11 * (IBM_WIDE_BLOCK / 32) + k]);
  for (int k = 0; k < 11; ++k) w->run[k] += acc[k];
  w->slip_max = amax;
  w->ssq = acc[0];
  w->wsum = acc[1];
  w->done = s + 1;
  w->converged = !r.sv_imp && amax / a.scale <= a.tol;  // the adjoint records a fixed number of sweeps
  w->ticket = 0;
}

template <class S>
__device__ __forceinline__ void wide_commit(const IbmArgs& a, const IbmRun<S>& r, int64_t blk) {
  pdl_wait();
  const int64_t i = blk * IBM_WIDE_BLOCK + threadIdx.x;
  if (i < a.ns) ibm_commit_slot(a, r, i);
  if (i < 32) {
    const IbmWide* w = a.wide;
    ibm_write_diag(a, r, int(i), i < 11 ? w->run[i] : 0.0, w->slip_max, w->ssq, w->wsum, w->done);
  }
}

template <int Q, class S>
__global__ void __launch_bounds__(IBM_WIDE_BLOCK) ibm_wide_prep_kernel(IbmArgs a, IbmRun<S> r) {
  wide_prep<Q, S>(a, r, blockIdx.x);
}
template <class S>
__global__ void __launch_bounds__(IBM_WIDE_BLOCK) ibm_wide_impulse_kernel(IbmArgs a, IbmRun<S> r) {
  wide_impulse(a, r, blockIdx.x);
}
template <class S>
__global__ void __launch_bounds__(IBM_WIDE_BLOCK) ibm_wide_spread_kernel(IbmArgs a, IbmRun<S> r, int s) {
  wide_spread(a, r, s, blockIdx.x);
}
template <class S>
__global__ void __launch_bounds__(IBM_WIDE_BLOCK) ibm_wide_slip_kernel(IbmArgs a, IbmRun<S> r, int s) {
  wide_slip(a, r, s, blockIdx.x, gridDim.x);
}
template <class S>
__global__ void __launch_bounds__(IBM_WIDE_BLOCK) ibm_wide_commit_kernel(IbmArgs a, IbmRun<S> r) {
  wide_commit(a, r, blockIdx.x);
}

}  // namespace lbmb
