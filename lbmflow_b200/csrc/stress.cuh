// Shear-rate and stress QOIs on the device.
//
// * Native strain rate (Solver::strain_rate_at / gather_shear_rate,
//   solver.rs:5393-5599): Pi_neq = sum c c (f - feq(rho, u)) over the
//   post-stream populations and the cached moments, + 0.5 (uF + Fu) with the
//   current force, times -1 / (2 cs^2 rho tau_eff), tau_eff = 1 / omega_p;
//   in the storage's arithmetic type, like the reference's T.
// * Velocity-gradient stress (stress.rs:32-82 compute_stress_field as the
//   bioprocess runner calls it, runner.rs:1648-1690): f64 central
//   differences of the SI velocity (lattice velocity x dx/dt), one-sided
//   next to a solid or the domain edge, gamma_dot = sqrt(2 S:S), viscous
//   stress mu gamma_dot. The percentile summary (stress.rs:84-100) selects
//   the values of its few ranks on the device: a histogram of the values'
//   leading 16 bits, the bins the ranks fall in, and a sort of those bins'
//   values only; the host interpolates between ranks.
// * Wall-shear proxy (stress.rs:102-294): fluid cells with a solid among
//   their 26 in-domain neighbours, compacted in cell order on the device.
#pragma once
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>

#include "aux.cuh"

namespace lbmb {

// Arguments of the native strain rate of a cell.
template <class S>
struct StrainArgs {
  using A = typename Codec<S>::A;
  const S* fb;
  int64_t pl;
  const uint8_t* flags;
  const uint32_t* nbr;
  int nx, ny, nz, parity;
  const int32_t* fslot;
  const Vec4<A>* fprev;
  const Vec4<A>* fcur;
  int field_present;
  A gx, gy, gz, tau_eff;
};

// Native strain rate of fluid cell `cell` into pi (A precision) and its
// cached velocity into u.
template <int Q, class S>
__device__ __forceinline__ void strain_cell(const StrainArgs<S>& a, int64_t cell, typename Codec<S>::A (&pi)[6],
                                            typename Codec<S>::A (&u)[3]) {
  using A = typename Codec<S>::A;
  using L = Lat<Q>;
  const uint8_t fl = a.flags[cell];
  int x, y, z;
  cell_xyz(cell, a.nx, a.ny, x, y, z);
  const uint32_t mask = (fl & F_BOUNDARY) ? a.nbr[cell] : 0u;
  A f[Q];
  load_post_stream<Q, S>(a.fb, a.pl, cell, x, y, z, a.nx, a.ny, a.nz, mask, a.parity, f);
  // cached moments, as moments_kernel (the field inside them is fprev)
  A dr = A(0), m0 = A(0), m1 = A(0), m2 = A(0);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    dr = dr + f[q];
    if (L::cx(q) == 1) m0 = m0 + f[q];
    if (L::cx(q) == -1) m0 = m0 - f[q];
    if (L::cy(q) == 1) m1 = m1 + f[q];
    if (L::cy(q) == -1) m1 = m1 - f[q];
    if (L::cz(q) == 1) m2 = m2 + f[q];
    if (L::cz(q) == -1) m2 = m2 - f[q];
  }
  A Fx = a.gx, Fy = a.gy, Fz = a.gz;  // force in the cached moments
  A Gx = a.gx, Gy = a.gy, Gz = a.gz;  // current force (KParams::force_at)
  if (fl & F_FORCED) {
    const int32_t sl = a.fslot[cell];
    const Vec4<A> v = a.fprev[sl];
    Fx = Fx + v.x;
    Fy = Fy + v.y;
    Fz = Fz + v.z;
    if (a.field_present) {
      const Vec4<A> b = a.fcur[sl];
      Gx = Gx + b.x;
      Gy = Gy + b.y;
      Gz = Gz + b.z;
    }
  }
  const A r = A(1) + dr;
  const A inv = A(1) / r;
  u[0] = (m0 + A(0.5) * Fx) * inv;
  u[1] = (m1 + A(0.5) * Fy) * inv;
  u[2] = (m2 + A(0.5) * Fz) * inv;
  // equilibrium in deviation form (kernels.rs:103-121)
  const A usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
  const A drho = r - A(1);
#pragma unroll
  for (int k = 0; k < 6; ++k) pi[k] = A(0);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const A cx = A(L::cx(q)), cy = A(L::cy(q)), cz = A(L::cz(q));
    const A cu = cx * u[0] + cy * u[1] + cz * u[2];
    const A feq = A(L::w(q)) * (drho + r * (A(3) * cu + A(4.5) * cu * cu - A(1.5) * usq));
    const A fneq = f[q] - feq;
    pi[0] = pi[0] + cx * cx * fneq;
    pi[1] = pi[1] + cy * cy * fneq;
    pi[2] = pi[2] + cz * cz * fneq;
    pi[3] = pi[3] + cx * cy * fneq;
    pi[4] = pi[4] + cx * cz * fneq;
    pi[5] = pi[5] + cy * cz * fneq;
  }
  const A half = A(0.5);
  pi[0] = pi[0] + u[0] * Gx;
  pi[1] = pi[1] + u[1] * Gy;
  pi[2] = pi[2] + u[2] * Gz;
  pi[3] = pi[3] + half * (u[0] * Gy + u[1] * Gx);
  pi[4] = pi[4] + half * (u[0] * Gz + u[2] * Gx);
  pi[5] = pi[5] + half * (u[1] * Gz + u[2] * Gy);
  const A scale = -(A(1) / (A(2.0 / 3.0) * r * a.tau_eff));
#pragma unroll
  for (int k = 0; k < 6; ++k) pi[k] = pi[k] * scale;
}

// Cached velocity of a fluid cell (the arithmetic of moments_kernel).
template <int Q, class S>
__device__ __forceinline__ void cell_velocity(const StrainArgs<S>& a, int64_t cell, double (&u)[3]) {
  using A = typename Codec<S>::A;
  using L = Lat<Q>;
  const uint8_t fl = a.flags[cell];
  int x, y, z;
  cell_xyz(cell, a.nx, a.ny, x, y, z);
  const uint32_t mask = (fl & F_BOUNDARY) ? a.nbr[cell] : 0u;
  A f[Q];
  load_post_stream<Q, S>(a.fb, a.pl, cell, x, y, z, a.nx, a.ny, a.nz, mask, a.parity, f);
  A dr = A(0), m0 = A(0), m1 = A(0), m2 = A(0);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    dr = dr + f[q];
    if (L::cx(q) == 1) m0 = m0 + f[q];
    if (L::cx(q) == -1) m0 = m0 - f[q];
    if (L::cy(q) == 1) m1 = m1 + f[q];
    if (L::cy(q) == -1) m1 = m1 - f[q];
    if (L::cz(q) == 1) m2 = m2 + f[q];
    if (L::cz(q) == -1) m2 = m2 - f[q];
  }
  A Fx = a.gx, Fy = a.gy, Fz = a.gz;
  if (fl & F_FORCED) {
    const Vec4<A> v = a.fprev[a.fslot[cell]];
    Fx = Fx + v.x;
    Fy = Fy + v.y;
    Fz = Fz + v.z;
  }
  const A inv = A(1) / (A(1) + dr);
  u[0] = double((m0 + A(0.5) * Fx) * inv);
  u[1] = double((m1 + A(0.5) * Fy) * inv);
  u[2] = double((m2 + A(0.5) * Fz) * inv);
}

template <int Q, class S>
__global__ void strain_rate_kernel(StrainArgs<S> a, double* s6, double* gamma, int64_t c0, int64_t c1) {
  using A = typename Codec<S>::A;
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t cell = c0 + i;
  if (cell >= c1) return;
  if (a.flags[cell] & F_SOLID) {  // solid cells report zero strain
    if (s6)
      for (int k = 0; k < 6; ++k) s6[6 * i + k] = 0.0;
    if (gamma) gamma[i] = 0.0;
    return;
  }
  A pi[6], u[3];
  strain_cell<Q, S>(a, cell, pi, u);
  if (s6)
    for (int k = 0; k < 6; ++k) s6[6 * i + k] = double(pi[k]);
  if (gamma) {
    const A ss = pi[0] * pi[0] + pi[1] * pi[1] + pi[2] * pi[2] + A(2) * (pi[3] * pi[3] + pi[4] * pi[4] + pi[5] * pi[5]);
    gamma[i] = double(sqrt(A(2) * ss));
  }
}

// Velocity gradient of a fluid cell (Solver::gather_velocity_gradient,
// solver.rs:5482-5582): symmetric off-diagonal part from the native strain
// rate, diagonal and rotation from differences of the cached velocity
// (u3 = [ux | uy | uz] in f64, exact copies of the A values): central
// between fluid cells, -4/3 w + u + 1/3 u(+1) (mirrored) next to a solid
// whose wall velocity w counts, one-sided at a non-periodic domain edge,
// periodic faces wrapped.
template <int Q, class S>
__device__ __forceinline__ void vel_grad_cell(const StrainArgs<S>& a, const double* u3, const Vec4<typename Codec<S>::A>* wall_u,
                                              int per_x, int per_y, int per_z, int64_t cell,
                                              typename Codec<S>::A (&g)[3][3]) {
  using A = typename Codec<S>::A;
  A st[6], uc[3];
  strain_cell<Q, S>(a, cell, st, uc);
  const int64_t n = int64_t(a.nx) * a.ny * a.nz;
  int x, y, z;
  cell_xyz(cell, a.nx, a.ny, x, y, z);
  const int pos[3] = {x, y, z}, d[3] = {a.nx, a.ny, a.nz}, per[3] = {per_x, per_y, per_z};
  const A own[3] = {A(u3[cell]), A(u3[n + cell]), A(u3[2 * n + cell])};
  A fd[3][3];
  for (int ax = 0; ax < 3; ++ax) {
    // neighbours along ax: 0 none, 1 fluid, 2 solid (wall velocity)
    int kind[2];
    A v[2][3];
    for (int side = 0; side < 2; ++side) {
      int pp[3] = {pos[0], pos[1], pos[2]};
      pp[ax] += side == 0 ? 1 : -1;
      kind[side] = 0;
      if (pp[ax] < 0 || pp[ax] >= d[ax]) {
        if (!per[ax]) continue;
        pp[ax] = (pp[ax] + d[ax]) % d[ax];
      }
      const int64_t j = (int64_t(pp[2]) * a.ny + pp[1]) * a.nx + pp[0];
      if (a.flags[j] & F_SOLID) {
        const Vec4<A> w = wall_u[j];
        v[side][0] = w.x;
        v[side][1] = w.y;
        v[side][2] = w.z;
        kind[side] = 2;
      } else {
        v[side][0] = A(u3[j]);
        v[side][1] = A(u3[n + j]);
        v[side][2] = A(u3[2 * n + j]);
        kind[side] = 1;
      }
    }
    for (int comp = 0; comp < 3; ++comp) {
      const A pv = v[0][comp], mv = v[1][comp];
      A val = A(0);
      if (kind[0] == 1 && kind[1] == 1) val = (pv - mv) * A(0.5);
      else if (kind[0] == 1 && kind[1] == 2) val = -A(4.0 / 3.0) * mv + own[comp] + A(1.0 / 3.0) * pv;
      else if (kind[0] == 2 && kind[1] == 1) val = A(4.0 / 3.0) * pv - own[comp] - A(1.0 / 3.0) * mv;
      else if (kind[0] == 1 && kind[1] == 0) val = pv - own[comp];
      else if (kind[0] == 0 && kind[1] == 1) val = own[comp] - mv;
      fd[comp][ax] = val;
    }
  }
  const A sm[3][3] = {{st[0], st[3], st[4]}, {st[3], st[1], st[5]}, {st[4], st[5], st[2]}};
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int q = 0; q < 3; ++q) g[r][q] = r == q ? fd[r][q] : sm[r][q] + A(0.5) * (fd[r][q] - fd[q][r]);
}

// Velocity gradient of every cell (g9, n x 9 row-major) and / or WALE
// (les.rs:120-211, Cw 0.325, Delta 1): nu_t and the omega+ field for the
// next collision, cells [c0, c1) (g9 and nu_t start at cell c0); clip bound
// nu_t_max when clip != 0; counts[0] = clipped cells, maxbits = bits of the
// largest nu_t before clipping (non-negative, so integer order is value
// order).
constexpr int WALE_BLOCK = 128;
template <int Q, class S>
__global__ void __launch_bounds__(WALE_BLOCK)
    wale_kernel(StrainArgs<S> a, const double* u3, const Vec4<typename Codec<S>::A>* wall_u, int per_x, int per_y,
                int per_z, typename Codec<S>::A nu0, int clip, typename Codec<S>::A nu_t_max, double* g9,
                double* nu_t, typename Codec<S>::A* omega, unsigned long long* counts, unsigned long long* maxbits,
                int64_t c0, int64_t c1) {
  using A = typename Codec<S>::A;
  const int64_t first = c0 + int64_t(blockIdx.x) * WALE_BLOCK, cell = first + threadIdx.x;
  A g[3][3];
  if (cell >= c1 || (a.flags[cell] & F_SOLID)) {
    for (int i = 0; i < 9; ++i) g[i / 3][i % 3] = A(0);
  } else {
    vel_grad_cell<Q, S>(a, u3, wall_u, per_x, per_y, per_z, cell, g);
  }
  if (g9) {  // through shared memory: consecutive threads write consecutive values over PCIe
    __shared__ double sh[9 * WALE_BLOCK];
    for (int i = 0; i < 9; ++i) sh[9 * threadIdx.x + i] = double(g[i / 3][i % 3]);
    __syncthreads();
    const int count = 9 * int(c1 - first < WALE_BLOCK ? c1 - first : WALE_BLOCK);
    for (int i = threadIdx.x; i < count; i += WALE_BLOCK) g9[9 * (first - c0) + i] = sh[i];
  }
  if (!omega || cell >= c1) return;
  A sr[3][3], g2[3][3], sd[3][3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) sr[i][j] = A(0.5) * (g[i][j] + g[j][i]);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      g2[i][j] = A(0);
      for (int k = 0; k < 3; ++k) g2[i][j] = g2[i][j] + g[i][k] * g[k][j];
    }
  const A tr = g2[0][0] + g2[1][1] + g2[2][2];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      sd[i][j] = A(0.5) * (g2[i][j] + g2[j][i]);
      if (i == j) sd[i][j] = sd[i][j] - tr / A(3);
    }
  A ss = A(0), sdsd = A(0);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      ss = ss + sr[i][j] * sr[i][j];
      sdsd = sdsd + sd[i][j] * sd[i][j];
    }
  const A cwd = A(0.325) * A(1);
  const A denom = pow(ss, A(2.5)) + pow(sdsd, A(1.25));
  A nut = denom > A(0) ? (cwd * cwd) * pow(sdsd, A(1.5)) / denom : A(0);
  if (nut == nut) {  // the reference's max ignores NaN
    const double nd = double(nut);
    atomicMax(maxbits, (unsigned long long)__double_as_longlong(nd));
  }
  if (clip && nut > nu_t_max) {
    atomicAdd(counts, 1ull);
    nut = nu_t_max;
  }
  if (nu_t) nu_t[cell - c0] = double(nut);
  omega[cell] = A(1) / (A(3) * (nu0 + nut) + A(0.5));
}

// Bin of a finite non-negative value: its exponent and four leading mantissa
// bits (such values order like their bits; -0 counts as 0).
constexpr int VALUE_BINS = 1 << 15;
__device__ __forceinline__ int value_bin(double v) {
  return int((unsigned long long)__double_as_longlong(v + 0.0) >> 48) & (VALUE_BINS - 1);
}

// compute_stress_field on the cached velocity moments (lattice units, f64;
// solid entries are never read), cells [c0, c1), outputs from cell c0.
// key[i]: gamma_dot of a fluid cell when finite, else NaN (solid or
// non-finite); hist counts the finite ones by bin.
static __global__ void stress_field_kernel(const double* ux, const double* uy, const double* uz, const uint8_t* flags,
                                    int nx, int ny, int nz, double dx, double vscale, double mu, double* s6,
                                    double* gamma, double* viscous, double* key, unsigned int* hist,
                                    int64_t c0, int64_t c1) {
  const int64_t o = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t i = c0 + o;
  if (i < c1) {
    double gd = __longlong_as_double(0x7ff8000000000000ll);
    if (!(flags[i] & F_SOLID)) {
      int x, y, z;
      cell_xyz(i, nx, ny, x, y, z);
      const int d[3] = {nx, ny, nz};
      const int pos[3] = {x, y, z};
      const double* fld[3] = {ux, uy, uz};
      double g[3][3];
      for (int comp = 0; comp < 3; ++comp)
        for (int axis = 0; axis < 3; ++axis) {
          g[comp][axis] = 0.0;
          if (d[axis] <= 1) continue;
          const int64_t stride = axis == 0 ? 1 : (axis == 1 ? int64_t(nx) : int64_t(nx) * ny);
          const bool hp = pos[axis] + 1 < d[axis] && !(flags[i + stride] & F_SOLID);
          const bool hm = pos[axis] - 1 >= 0 && !(flags[i - stride] & F_SOLID);
          const double own = fld[comp][i] * vscale;
          if (hp && hm) {
            const double pv = fld[comp][i + stride] * vscale, mv = fld[comp][i - stride] * vscale;
            g[comp][axis] = (pv - mv) / (2.0 * dx);
          } else if (hp) {
            g[comp][axis] = (fld[comp][i + stride] * vscale - own) / dx;
          } else if (hm) {
            g[comp][axis] = (own - fld[comp][i - stride] * vscale) / dx;
          }
        }
      const double s[6] = {g[0][0], g[1][1], g[2][2], 0.5 * (g[0][1] + g[1][0]), 0.5 * (g[0][2] + g[2][0]),
                           0.5 * (g[1][2] + g[2][1])};
      const double ss = s[0] * s[0] + s[1] * s[1] + s[2] * s[2] + 2.0 * (s[3] * s[3] + s[4] * s[4] + s[5] * s[5]);
      const double v = sqrt(2.0 * ss);
      if (s6)
        for (int k = 0; k < 6; ++k) s6[6 * o + k] = s[k];
      if (gamma) gamma[o] = v;
      if (viscous) viscous[o] = mu * v;
      if (isfinite(v)) {
        gd = v;
        if (hist) {  // one add per bin and warp (a fluid at rest has one bin)
          const int bin = value_bin(v);
          const unsigned same = __match_any_sync(__activemask(), bin);
          if ((threadIdx.x & 31) == unsigned(__ffs(int(same)) - 1)) atomicAdd(hist + bin, unsigned(__popc(same)));
        }
      }
    } else {
      if (s6)
        for (int k = 0; k < 6; ++k) s6[6 * o + k] = 0.0;
      if (gamma) gamma[o] = 0.0;
      if (viscous) viscous[o] = 0.0;
    }
    if (key) key[o] = gd;
  }
}

// The ranks of a percentile summary (stress.rs:296-309): floor and ceiling
// ranks of the quantiles 0.5, 0.9, 0.95, 0.99, and the maximum.
constexpr int N_RANKS = 9;
struct RankSelect {
  unsigned long long count;          // finite values
  unsigned long long rank[N_RANKS];  // wanted ranks, then their positions among the selected values
  unsigned long long n_selected;     // values in the bins of the ranks
  unsigned long long above[2];       // values above the thresholds
  unsigned int mark[VALUE_BINS / 32];  // bins of the ranks
};

// One block: turns the histogram into ranks, marked bins and each rank's
// position among the marked bins' values in ascending order.
constexpr int SELECT_BLOCK = 1024;
static __global__ void __launch_bounds__(SELECT_BLOCK) select_ranks_kernel(const unsigned int* hist, RankSelect* r) {
  constexpr int PER = VALUE_BINS / SELECT_BLOCK;  // consecutive bins of a thread: one mark word
  static_assert(PER == 32, "a thread's bins are one mark word");
  __shared__ unsigned long long part[SELECT_BLOCK];
  __shared__ unsigned int words[SELECT_BLOCK];
  __shared__ unsigned long long rank[N_RANKS], pos[N_RANKS];
  const int t = int(threadIdx.x);
  unsigned long long own = 0;
  for (int k = 0; k < PER; ++k) own += hist[t * PER + k];
  part[t] = own;
  words[t] = 0u;
  __syncthreads();
  for (int d = 1; d < SELECT_BLOCK; d <<= 1) {  // inclusive scan
    const unsigned long long v = t >= d ? part[t - d] : 0ull;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  const unsigned long long n = part[SELECT_BLOCK - 1];
  if (t < N_RANKS && n > 0) {
    const double q[4] = {0.50, 0.90, 0.95, 0.99};
    const double x = t < 8 ? q[t >> 1] * double(n - 1) : double(n - 1);
    rank[t] = (unsigned long long)(t < 8 ? ((t & 1) ? ceil(x) : floor(x)) : x);
  }
  __syncthreads();
  if (n > 0) {
    for (int j = 0; j < N_RANKS; ++j) {
      unsigned long long lo = part[t] - own;
      if (rank[j] < lo || rank[j] >= part[t]) continue;
      for (int k = 0; k < PER; ++k) {
        const unsigned long long h = hist[t * PER + k];
        if (rank[j] < lo + h) {
          words[t] |= 1u << k;
          pos[j] = rank[j] - lo;
          break;
        }
        lo += h;
      }
    }
  }
  __syncthreads();
  // values of the marked bins before each thread's
  unsigned long long sel = 0;
  for (int k = 0; k < PER; ++k)
    if ((words[t] >> k) & 1u) sel += hist[t * PER + k];
  const unsigned long long end = part[t];
  __syncthreads();
  part[t] = sel;
  __syncthreads();
  for (int d = 1; d < SELECT_BLOCK; d <<= 1) {
    const unsigned long long v = t >= d ? part[t - d] : 0ull;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  if (n > 0) {
    for (int j = 0; j < N_RANKS; ++j) {
      unsigned long long lo = end - own, before = part[t] - sel;
      if (rank[j] < lo || rank[j] >= end) continue;
      for (int k = 0; k < PER; ++k) {
        const unsigned long long h = hist[t * PER + k];
        if (rank[j] < lo + h) {
          r->rank[j] = before + pos[j];
          break;
        }
        lo += h;
        if ((words[t] >> k) & 1u) before += h;
      }
    }
  }
  r->mark[t] = words[t];
  if (t == 0) {
    r->count = n;
    r->n_selected = part[SELECT_BLOCK - 1];
  }
}

// Values of the marked bins, in any order, and the counts above the
// thresholds (values scaled first, as the reference forms mu gamma_dot before
// it counts; thresholds +inf: none counted).
static __global__ void select_values_kernel(const double* key, int64_t n, RankSelect* r, unsigned long long* cursor,
                                            double* out, double t_gamma, double mu, double t_tau) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const double v = i < n ? key[i] : __longlong_as_double(0x7ff8000000000000ll);
  const bool ok = isfinite(v);
  const int lane = int(threadIdx.x) & 31;
  const int bin = ok ? value_bin(v) : 0;
  const bool take = ok && ((r->mark[bin >> 5] >> (bin & 31)) & 1u);
  const unsigned b = __ballot_sync(0xffffffffu, take);
  unsigned long long at = 0;
  if (lane == 0 && b) at = atomicAdd(cursor, (unsigned long long)__popc(b));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (take) out[at + __popc(b & ((1u << lane) - 1u))] = v + 0.0;
  const unsigned g = __ballot_sync(0xffffffffu, ok && v > t_gamma), w = __ballot_sync(0xffffffffu, ok && mu * v > t_tau);
  if (lane == 0) {
    if (g) atomicAdd(&r->above[0], (unsigned long long)__popc(g));
    if (w) atomicAdd(&r->above[1], (unsigned long long)__popc(w));
  }
}

// The selected ranks' values from the sorted selection.
static __global__ void rank_values_kernel(const double* sorted, const RankSelect* r, double* out) {
  if (threadIdx.x < N_RANKS) out[threadIdx.x] = sorted[r->rank[threadIdx.x]];
}

// A cell of the wall-shear proxy: a fluid cell with a solid among its 26
// in-domain neighbours and a nonzero wall normal (unit), and the number of
// those solids.
struct WallCell {
  int64_t cell;
  double normal[3];
  double count;
};

// wall_shear_proxy's geometry per cell, which no step changes: flag[i] = 1
// where the proxy has an entry (cells == null), or the entries of the listed
// cells.
static __global__ void wall_cells_kernel(const uint8_t* flags, int nx, int ny, int nz, uint8_t* flag,
                                         const int64_t* cells, WallCell* out, int64_t n) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t i = cells ? cells[t] : t;
  if (!cells) flag[i] = 0;
  if (flags[i] & F_SOLID) return;
  int x, y, z;
  cell_xyz(i, nx, ny, x, y, z);
  WallCell w = {i, {0.0, 0.0, 0.0}, 0.0};
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dxo = -1; dxo <= 1; ++dxo) {
        if (!dxo && !dy && !dz) continue;
        const int a = x + dxo, b = y + dy, c = z + dz;
        if (a < 0 || b < 0 || c < 0 || a >= nx || b >= ny || c >= nz) continue;
        const int64_t j = (int64_t(c) * ny + b) * nx + a;
        if (!(flags[j] & F_SOLID)) continue;
        w.normal[0] += double(dxo);
        w.normal[1] += double(dy);
        w.normal[2] += double(dz);
        w.count += 1.0;
      }
  if (w.count == 0.0) return;
  const double mag = sqrt(w.normal[0] * w.normal[0] + w.normal[1] * w.normal[1] + w.normal[2] * w.normal[2]);
  if (mag == 0.0) return;
  if (!cells) {
    flag[i] = 1;
    return;
  }
  for (int k = 0; k < 3; ++k) w.normal[k] /= mag;
  out[t] = w;
}

// wall_shear_proxy (stress.rs:102-294) of entries [c0, c1) of the wall-cell
// list, 8 values each in lbmb_wall_shear's layout; the velocity is computed
// for the listed cells only.
template <int Q, class S>
__global__ void wall_shear_kernel(StrainArgs<S> g, const Vec4<typename Codec<S>::A>* wall_u, const WallCell* list,
                                  double dx, double vscale, double rho, double mu, double* out, int64_t c0,
                                  int64_t c1) {
  const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c0 + r >= c1) return;
  const WallCell w = list[c0 + r];
  const int64_t i = w.cell;
  int x, y, z;
  cell_xyz(i, g.nx, g.ny, x, y, z);
  double wu[3] = {0.0, 0.0, 0.0};
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dxo = -1; dxo <= 1; ++dxo) {
        if (!dxo && !dy && !dz) continue;
        const int a = x + dxo, b = y + dy, c = z + dz;
        if (a < 0 || b < 0 || c < 0 || a >= g.nx || b >= g.ny || c >= g.nz) continue;
        const int64_t j = (int64_t(c) * g.ny + b) * g.nx + a;
        if (!(g.flags[j] & F_SOLID)) continue;
        const Vec4<typename Codec<S>::A> v = wall_u[j];
        wu[0] += double(v.x) * vscale;
        wu[1] += double(v.y) * vscale;
        wu[2] += double(v.z) * vscale;
      }
  double u[3];
  cell_velocity<Q, S>(g, i, u);
  for (int k = 0; k < 3; ++k) u[k] = u[k] * vscale - wu[k] / w.count;
  const double un = u[0] * w.normal[0] + u[1] * w.normal[1] + u[2] * w.normal[2];
  const double t[3] = {u[0] - un * w.normal[0], u[1] - un * w.normal[1], u[2] - un * w.normal[2]};
  const double up = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
  const double y_m = 0.5 * dx;
  const double tw = mu * up / y_m;
  double* const o = out + 8 * r;
  o[0] = __longlong_as_double(i);
  o[1] = tw;
  o[2] = y_m * sqrt(tw / rho) / (mu / rho);
  o[3] = up;
  o[4] = y_m;
  o[5] = w.normal[0];
  o[6] = w.normal[1];
  o[7] = w.normal[2];
}

static __global__ void iota_kernel(int64_t* out, int64_t n) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) out[i] = i;
}

}  // namespace lbmb
