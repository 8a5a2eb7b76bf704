// Batched stirred-tank runner: many tanks of different sizes advanced in
// lockstep, one launch per kernel family per step for all of them.
//
// Reference: the sweep runs its cases one after another, each through the
// full runner loop (crates/lbm-cli/src/sweep.rs:47-106, runner.rs:1079-1129).
// Here every case keeps its own device state (an Engine); a batch holds a
// device table of per-case descriptors (the case's HydroParams, its IBM
// arguments, force slots and per-step series) and launches
//
//   direct forcing: one cluster per case (ibm_chain), or for large bodies its
//                   phases over all their cases on the side stream
//   side stream:    forced cells, then the cached-field refresh (fprev = fcur)
//   main stream:    full-grid sweep of every case (lean TRT kernel), started
//                   as soon as every cluster runs
//
// per step, the last three over the concatenation of all cases' cells or
// slots. A block never straddles two cases: each family has a table of
// per-case block offsets, and a block finds its case by binary search. The
// per-case IBM early exit, the diagnostics reduction and the step counters
// are per case, so every case follows exactly the sequence it would follow
// alone.
#pragma once
#include "hydro_lean.cuh"
#include "ibm.cuh"

namespace lbmb {

constexpr int BATCH_BLOCK = 128;
static_assert(BATCH_BLOCK == LEAN_BLOCK, "one block size for the cell families");

struct BatchCase {
  HydroParams<float> hp;
  uint32_t n;  // cells
  int nx, ny, nz;
  const int64_t* slot_cell;  // forced cells (= force slots)
  int64_t nslots;
  Vec4<float>* fcur;
  Vec4<float>* fprev;
  IbmArgs ibm;
  double* series_torque;  // per step
  int64_t* counter;
};

// Case of block b: the last c with off[c] <= b (off has ncase + 1 entries).
__device__ __forceinline__ int batch_case(const int32_t* off, int ncase, int b) {
  int lo = 0, hi = ncase;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(off + mid) <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <int Q, class S, bool ODD, int MINB>
__global__ void __launch_bounds__(BATCH_BLOCK, MINB)
    batch_hydro_kernel(const BatchCase* cs, const int32_t* off, int ncase) {
  const int k = batch_case(off, ncase, blockIdx.x);
  const BatchCase& b = cs[k];
  const uint32_t c = uint32_t(int(blockIdx.x) - __ldg(off + k)) * BATCH_BLOCK + threadIdx.x;
  if (c >= b.n) return;
  lean_cell<Q, S, ODD>(b.hp, c);
}

template <int Q, class S, bool ODD>
static __global__ void __launch_bounds__(BATCH_BLOCK) batch_cells_kernel(const BatchCase* cs, const int32_t* off, int ncase) {
  const int k = batch_case(off, ncase, blockIdx.x);
  const BatchCase& b = cs[k];
  const int64_t i = int64_t(int(blockIdx.x) - __ldg(off + k)) * BATCH_BLOCK + threadIdx.x;
  if (i >= b.nslots) return;
  forced_cell<Q, S, COLL_TRT, ODD>(b.hp, uint32_t(b.slot_cell[i]));
}

template <class S>
__device__ __forceinline__ IbmRun<S> batch_run(const BatchCase& b, int parity, int sweeps) {
  IbmRun<S> r = {};
  r.fb = static_cast<const S*>(b.hp.f);
  r.pl = int64_t(b.hp.plane);
  r.nx = b.nx;
  r.ny = b.ny;
  r.nz = b.nz;
  r.parity = parity;
  r.fcur = b.fcur;
  r.nslots = b.nslots;
  r.clear = 1;
  r.sweeps = sweeps;
  r.series_torque = b.series_torque;
  r.step_counter = b.counter;
  return r;
}

// The direct forcing of the cases list[0..], one cluster each; the runner
// clears the force field before it, so the field at call time is zero.
// Small blocks (64 registers a thread, which spill 296 bytes and load 436), so
// that the clusters of many cases run at once: the sweep starts when the last
// of them has.
constexpr int BATCH_IBM_THREADS = 256;
template <int Q, class S>
static __global__ void __launch_bounds__(BATCH_IBM_THREADS, 4)
    batch_ibm_kernel(const BatchCase* cs, const int32_t* list, int parity, int sweeps) {
  release_dependents();
  int rank, ncta;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
  const BatchCase& b = cs[list[int(blockIdx.x) / ncta]];
  const IbmRun<S> r = batch_run<S>(b, parity, sweeps);
  const IbmArgs a = b.ibm;
  ibm_chain<Q, S, 4>(a, r, rank, ncta);
}

// The cases list[0..k) with larger bodies, in the wide form: block offsets per
// phase family (prep: slots of the body and of the grid, slots, markers).
static_assert(BATCH_BLOCK == IBM_WIDE_BLOCK, "block offsets count blocks of one size");
enum { WIDE_PREP, WIDE_IMPULSE, WIDE_SPREAD, WIDE_SLIP, WIDE_COMMIT };
template <int PHASE, int Q, class S>
static __global__ void __launch_bounds__(IBM_WIDE_BLOCK)
    batch_wide_kernel(const BatchCase* cs, const int32_t* list, const int32_t* off, int ncase, int parity, int sweeps,
                      int s) {
  const int k = batch_case(off, ncase, blockIdx.x);
  const BatchCase& b = cs[list[k]];
  const int b0 = __ldg(off + k);
  const int64_t blk = int(blockIdx.x) - b0;
  const IbmRun<S> r = batch_run<S>(b, parity, sweeps);
  if (PHASE == WIDE_PREP) wide_prep<Q, S>(b.ibm, r, blk);
  if (PHASE == WIDE_IMPULSE) wide_impulse(b.ibm, r, blk);
  if (PHASE == WIDE_SPREAD) wide_spread(b.ibm, r, s, blk);
  if (PHASE == WIDE_SLIP) wide_slip(b.ibm, r, s, blk, unsigned(__ldg(off + k + 1) - b0));
  if (PHASE == WIDE_COMMIT) wide_commit(b.ibm, r, blk);
}
// Entries (slots or markers) of a body above which its case is one of them, of
// a batch of n cells in all, which hide the clusters. us per step, clusters
// alone / with this rule, one sweep: one box of 64 cells with 11,976 slots 84 /
// 65, eight with 20,421 214 / 205, two with 36,122 231 / 97, four of 128 cells
// with 47,359 506 / 431.
inline int64_t batch_wide_from(int64_t n) { return 4096 + n / 400; }

static __global__ void __launch_bounds__(BATCH_BLOCK) batch_fprev_kernel(const BatchCase* cs, const int32_t* off, int ncase) {
  const int k = batch_case(off, ncase, blockIdx.x);
  const BatchCase& b = cs[k];
  const int64_t i = int64_t(int(blockIdx.x) - __ldg(off + k)) * BATCH_BLOCK + threadIdx.x;
  if (i < b.nslots) b.fprev[i] = b.fcur[i];
}

}  // namespace lbmb
