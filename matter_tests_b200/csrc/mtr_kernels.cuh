// mtr_kernels.cuh — the sm_100a kernels of one explicit MPM step
// (Simulation::advanceStep, simulation.cpp:219-273).
//
// Step pipeline (all on one stream, no host round trip, CUDA-graph capturable):
//   k_bbox        per-block min/max x, max |v|^2 and sum v    update_dt.cpp, remesh.cpp
//   k_header      dt, gravity ramp, remesh + arange axes      update_dt.cpp:5-66, remesh.cpp:38-311
//   k_sort_*      stable counting sort by blocked cell key    (new: locality for P2G); the cell
//                 starts it leaves are the particle ranges of every cell and 4^3 (2D: 8^2) tile
//   k_p2g_w       tile block(s) -> shared grid patch -> one global atomic per node and channel
//                 (mass, momentum with APIC, force tau.grad w, MIBF friction)
//                                                              p2g.cpp:6-100, explicit_euler_update.cpp:15-77
//   k_grid        normalise, v += -dt V0 f/m + dt g, boundary collision, flip, FP64 balances
//                                                              p2g.cpp:84-98, explicit_euler_update.cpp:83-132
//   USL:  k_g2p_t gather pic/B/flip/grad v, F update, return mapping, tau, x/v update, coalesced stores
//                                                              g2p.cpp, deformation_update.cpp, plasticity.cpp,
//                                                              position_update.cpp
//   MUSL: k_g2p_musl_w (gather + v blend + re-scatter), k_defgrad_t
//                                                              musl.cpp:6-96
//   k_tail        plate motion, clock, frame and end test     object_plate.hpp:136-162, simulation.cpp:176-200
//
// Particle state is SoA, one array per component (x + a*Np), double buffered:
// the step reads the `in` set through the sort permutation and writes the
// `out` set in sorted order, so the particle order follows the cell order and
// every later read of the same data is nearly coalesced.
//
// Precision.  Every kernel that touches particle or grid state is templated
// on the storage type R.  R = double is FP64 throughout, the reference's
// formulas with sums over a stencil factorised and the SVD of a deformation near
// the identity replaced by a series.  R = float is the mixed-precision form: particle
// v, F, B, stress and plastic scalars, the grid mass, momentum, force,
// friction and flip channels, the spline weights, the P2G and MUSL sums and
// the G2P gathers are FP32.  FP64 stays on the positions, the clock, the grid
// axes and node velocities, the deformation update, the SVD, the Hencky
// log/exp, the return mapping with its projections, and the mass and
// momentum balances.  F is stored as F - I in FP32, so its rounding is
// relative to the strain (about 1e-3) rather than to 1; the gathers work on
// FP32 deviations from a per-tile reference velocity, so the FP32 sums that
// form grad v do not cancel a common velocity.
#pragma once
#include <type_traits>

#include "mtr_boundary.cuh"
#include "mtr_device.cuh"
#include "mtr_plasticity.cuh"

namespace mtr {

template <typename R>
struct PBufT {
  double* x;     // [D][Np] positions, FP64 on both paths
  R* v;          // [D][Np]
  R* F;          // [D*D][Np], entry (r,c) at (r*D + c); FP32 path: F - I
  R* B;          // [D*D][Np]
  R* sc;         // [6][Np] MTR_SCALAR_* order
  R* tau;        // [Sym<D>::n][Np] Kirchhoff stress carried to the next P2G
  uint32_t* id;  // original particle index
};
using PBuf = PBufT<double>;

// What every kernel of a step shares, whatever the storage type.
struct StepCommon {
  const DevParams* P;
  StepHeader* H;
  BBoxPartial* partials;
  int npartials;
  uint32_t Np;
  double *gx, *gy, *gz;
  uint32_t cap_axis[3];
  uint32_t cap_nodes;
  uint32_t cap_tiles;
  const double* xin;  // positions of the step's input buffer (sort keys)
  uint32_t* keys0;      // cell key of each particle in input order
  uint32_t* perm_rank;  // rank of each particle among its cell's arrivals, then the sorted permutation
  uint32_t* perm_tmp;   // permutation with the cells in order and each cell's particles in arrival order
  uint32_t* cell_count; // [cap_tiles * 64 + 1], zero between steps
  uint32_t* cell_start; // [cap_tiles * 64 + 2]: first sorted particle of each cell of the last sort
  uint32_t* super;      // particles of each kSuperCells cells, zero between steps
  uint32_t* big_cells;  // cells with more than kBigCell particles (H->nbig of them)
  const uint32_t* perm; // = perm_rank, the sorted permutation
  int out_parity;         // particle buffer this step writes
};

template <typename R>
struct StepArgsT : StepCommon {
  R* acc;         // [NCH][cap_nodes] P2G accumulators: mass, mom[D], force[D], friction
  double* nv;     // [D][cap_nodes] node velocity after the update (FP64 on both paths)
  R* nflip;       // [D][cap_nodes]
  R* nmass;       // [cap_nodes]
  R* nfric;       // [cap_nodes]
  double* v2;     // [D][cap_nodes] MUSL re-projection accumulator (FP64 on both paths), not divided by m_i / m_p
  PBufT<R> in, out;
  R* pic;   // optional [D][Np] in output order
  R* flip;  // optional [D][Np]
};
using StepArgs = StepArgsT<double>;

template <typename R>
constexpr bool kFP64 = std::is_same<R, double>::value;

constexpr uint32_t kMaxAxisNodes = 1u << 22;
constexpr int kSortThreads = 256;
constexpr int kSuperCells = 4096;  // cells scanned by one block of k_sort_scan
constexpr uint32_t kBigCell = 1024;  // cells with more particles are ordered by a whole block

template <int D>
struct Tiling {
  static constexpr int TB = D == 3 ? 4 : 8;     // cells per tile edge
  static constexpr int SH = D == 3 ? 2 : 3;     // log2(TB)
  static constexpr int PN = TB + 3;             // patch nodes per edge (stencil -1..+2)
  static constexpr int NODES = D == 3 ? PN * PN * PN : PN * PN;
  static constexpr int NCH = 2 + 2 * D;         // mass, mom[D], force[D], friction
};

constexpr size_t align16(size_t b) { return (b + 15) & ~size_t(15); }

__device__ __forceinline__ bool step_inactive(const StepHeader* H) {
  return H->done || H->abort || H->frame >= H->stop_frame || H->step >= H->stop_step;
}

__device__ __forceinline__ uint32_t node_index(const StepHeader* H, int i, int j, int k) {
  return ((uint32_t)i * H->N[1] + (uint32_t)j) * H->N[2] + (uint32_t)k;
}

// sums over the block of N per-thread values, each added once to dst[i] (all
// threads call): one barrier for all of them
template <int N>
__device__ __forceinline__ void block_add(double (&v)[N], double* const (&dst)[N]) {
  __shared__ double red[N][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], off);
    if (lane == 0) red[i][warp] = v[i];
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[threadIdx.x][w];
    if (s != 0.0) atomicAdd(dst[threadIdx.x], s);
  }
}

// plastic particles of the block, one global atomic per block
__device__ __forceinline__ void block_count(unsigned n, unsigned long long* dst) {
  __shared__ unsigned cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(&cnt, n);
  __syncthreads();
  if (threadIdx.x == 0 && cnt) atomicAdd(dst, (unsigned long long)cnt);
}

// ---------------------------------------------------------------------------
// 1. bbox / vmax / sum v partials
// ---------------------------------------------------------------------------
// Bound: the latency of its loads.  A thread takes kBBoxItems particles and
// issues all their loads before it uses one.
constexpr int kBBoxItems = 4;
template <int D, typename R>
__device__ __forceinline__ void bbox_body(const StepArgsT<R>& A, const uint32_t bid, const uint32_t nblk) {
  if (step_inactive(A.H)) return;
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300}, v2 = 0.0, vs[3] = {0.0, 0.0, 0.0};
  for (uint32_t i0 = bid * (256 * kBBoxItems) + threadIdx.x; i0 < A.Np; i0 += nblk * (256 * kBBoxItems)) {
    double x[kBBoxItems][D];
    R v[kBBoxItems][D];
#pragma unroll
    for (int k = 0; k < kBBoxItems; ++k) {
      // past the end: the first particle again, counted once below
      const uint32_t i = i0 + k * 256 < A.Np ? i0 + k * 256 : i0;
#pragma unroll
      for (int a = 0; a < D; ++a) {
        x[k][a] = A.in.x[(size_t)a * A.Np + i];
        v[k][a] = A.in.v[(size_t)a * A.Np + i];
      }
    }
#pragma unroll
    for (int k = 0; k < kBBoxItems; ++k) {
      const bool in = i0 + k * 256 < A.Np;
      double vv[3];
#pragma unroll
      for (int a = 0; a < D; ++a) {
        mn[a] = fmin(mn[a], x[k][a]);
        mx[a] = fmax(mx[a], x[k][a]);
        vv[a] = v[k][a];
        vs[a] += in ? vv[a] : 0.0;
      }
      double s = __dadd_rn(__dmul_rn(vv[0], vv[0]), __dmul_rn(vv[1], vv[1]));
      if constexpr (D == 3) s = __dadd_rn(s, __dmul_rn(vv[2], vv[2]));
      v2 = fmax(v2, s);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int a = 0; a < D; ++a) {
      mn[a] = fmin(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], off));
      mx[a] = fmax(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], off));
      vs[a] += __shfl_xor_sync(0xffffffffu, vs[a], off);
    }
    v2 = fmax(v2, __shfl_xor_sync(0xffffffffu, v2, off));
  }
  __shared__ BBoxPartial wp[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      wp[warp].mn[a] = mn[a];
      wp[warp].mx[a] = mx[a];
      wp[warp].vsum[a] = vs[a];
    }
    wp[warp].v2 = v2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    BBoxPartial r = wp[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        r.mn[a] = fmin(r.mn[a], wp[w].mn[a]);
        r.mx[a] = fmax(r.mx[a], wp[w].mx[a]);
        r.vsum[a] += wp[w].vsum[a];
      }
      r.v2 = fmax(r.v2, wp[w].v2);
    }
    A.partials[bid] = r;
  }
}

template <int D, typename R>
__global__ void __launch_bounds__(256) k_bbox(StepArgsT<R> A) {
  bbox_body<D, R>(A, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// 2. step header: dt (update_dt.cpp:5-66) and grid (remesh.cpp:38-311)
// ---------------------------------------------------------------------------
// value, value + dx, (value + dx) + dx, ... up to stop, each sum rounded as in
// the serial loop it restates, by one warp: within a binade the increment is a
// constant, so the lanes guess 32 values at once and keep the leading ones that
// each follow from the one before by the rounded addition.  Returns the count,
// exact up to kMaxAxisNodes so that the host can size a regrowth in one go; the
// bound also ends the loop for non-finite extents.
// The serial loop's addition, test and store took 25 cycles a node; with the
// commit of the step before in the same kernel, us per step: 211,777 particles
// on a 2D grid of 450 x 230 nodes 100 -> 86, 51,200 in 2D 69 -> 65.
__device__ __forceinline__ uint32_t arange_axis(double value, double stop, double dx, uint32_t cap, double* ax) {
  const int lane = threadIdx.x & 31;
  if (!isfinite(value)) return value < stop ? kMaxAxisNodes : 0u;
  uint32_t n = 0;
  for (;;) {
    const double d = __dsub_rn(__dadd_rn(value, dx), value);
    const double guess = lane == 0 ? value : __fma_rn((double)lane, d, value);
    const double before = __shfl_up_sync(0xffffffffu, guess, 1);
    const unsigned good = __ballot_sync(0xffffffffu, lane == 0 || __dadd_rn(before, dx) == guess);
    const int len = good == 0xffffffffu ? 32 : __ffs(~good) - 1;
    const unsigned in = __ballot_sync(0xffffffffu, lane < len && guess < stop && n + lane < kMaxAxisNodes);
    const int cnt = in == 0xffffffffu ? 32 : __ffs(~in) - 1;
    if (lane < cnt && n + lane < cap) ax[n + lane] = guess;
    n += (uint32_t)cnt;
    if (cnt < len) return n;
    value = __dadd_rn(__shfl_sync(0xffffffffu, guess, len - 1), dx);
  }
}

template <int D>
__device__ __forceinline__ void header_body(const StepCommon& A) {
  StepHeader* H = A.H;
  const DevParams& P = *A.P;
  if (step_inactive(H)) return;
  // the block (256 threads) reduces the bbox partials; thread 0 then does the
  // step's scalars and one warp per axis the grid coordinates
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300}, v2 = 0.0, vs[3] = {0.0, 0.0, 0.0};
  for (int b = threadIdx.x; b < A.npartials; b += blockDim.x) {
    const BBoxPartial& q = A.partials[b];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = fmin(mn[a], q.mn[a]);
      mx[a] = fmax(mx[a], q.mx[a]);
      vs[a] += q.vsum[a];
    }
    v2 = fmax(v2, q.v2);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = fmin(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], off));
      mx[a] = fmax(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], off));
      vs[a] += __shfl_xor_sync(0xffffffffu, vs[a], off);
    }
    v2 = fmax(v2, __shfl_xor_sync(0xffffffffu, v2, off));
  }
  if (nw > 1) {
    __shared__ BBoxPartial wred[8];
    if (lane == 0) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        wred[wid].mn[a] = mn[a];
        wred[wid].mx[a] = mx[a];
        wred[wid].vsum[a] = vs[a];
      }
      wred[wid].v2 = v2;
    }
    __syncthreads();
    for (int w = 1; w < nw && wid == 0; ++w) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        mn[a] = fmin(mn[a], wred[w].mn[a]);
        mx[a] = fmax(mx[a], wred[w].mx[a]);
        vs[a] += wred[w].vsum[a];
      }
      v2 = fmax(v2, wred[w].v2);
    }
  }
  __shared__ double s_low[3], s_high[3], s_stop[3];
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    H->nbig = 0;
    // balances of this step (read back by mtr_balance)
    H->grid_mass = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      H->grid_mom[a] = 0.0;
      H->part_mom[a] = P.particle_mass * vs[a];
    }
    // updateDt
    const double max_speed = sqrt(v2);
    double dt;
    if (fabs(max_speed) > 1e-10) {
      double dt_cfl = P.cfl * P.dx / max_speed;
      dt = dmin(dt_cfl, P.dt_max);
    } else {
      dt = P.dt_max;
    }
    dt = dmin(dt, __dsub_rn(__dmul_rn(P.frame_dt, (double)(H->frame + 1)), H->time));
    dt = dmin(dt, __dsub_rn(P.final_time, H->time));
    H->dt = dt;
    if (P.gravity_special) {
#pragma unroll
      for (int a = 0; a < D; ++a)
        H->gravity[a] = (H->time < P.gravity_time) ? P.gravity_final[a] * H->time / P.gravity_time : P.gravity_final[a];
    }
    // remesh
    const double dx = P.dx;
    if (P.pbc) {  // remeshFixed(4), remesh.cpp:14-36: the same fixed grid every step
      const double e1 = 5.0, e2 = 6.0;  // 1 + extra_nodes, 2 + extra_nodes
#pragma unroll
      for (int a = 0; a < D; ++a) {
        s_low[a] = a == 1 ? -dx : __dmul_rn(-dx, e1);
        s_stop[a] = __dadd_rn(P.L[a], __dmul_rn(e2, dx));
      }
    } else if (H->step == 0) {  // remeshFixedInit(2,2,2)
      if (P.grid_ref[0] < 1e10) {
#pragma unroll
        for (int a = 0; a < D; ++a) {
          if (P.grid_ref[a] < mn[a])
            mn[a] = P.grid_ref[a];
          else if (P.grid_ref[a] > mx[a])
            mx[a] = P.grid_ref[a];
        }
      }
#pragma unroll
      for (int a = 0; a < D; ++a) {
        H->max_init[a] = mx[a];
        H->min_init[a] = mn[a];
        H->low_init[a] = __dsub_rn(mn[a], __dmul_rn(dx, 2.0));
        H->high_init[a] = __dadd_rn(mx[a], __dmul_rn(dx, 2.0));
        s_low[a] = H->low_init[a];
        s_high[a] = H->high_init[a];
      }
    } else {  // remeshFixedCont
      // explicit roundings: each product and difference is rounded on its own,
      // as in the host code this restates (no fused multiply-add)
      const double tiny = __dmul_rn(1e-8, dx);
      for (int a = 0; a < D; ++a) {
        double hi, lo;
        if (mx[a] < H->max_init[a]) {
          unsigned int f = (unsigned int)floor(dmax(0.0, __dsub_rn(__ddiv_rn(__dsub_rn(H->max_init[a], mx[a]), dx), tiny)));
          hi = __dsub_rn(H->high_init[a], __dmul_rn((double)f, dx));
        } else {
          unsigned int f = (unsigned int)floor(dmax(0.0, __dsub_rn(__ddiv_rn(__dsub_rn(mx[a], H->max_init[a]), dx), tiny)));
          hi = __dadd_rn(H->high_init[a], __dmul_rn((double)f, dx));
        }
        if (mn[a] > H->min_init[a]) {
          unsigned int f = (unsigned int)floor(dmax(0.0, __dsub_rn(__ddiv_rn(__dsub_rn(mn[a], H->min_init[a]), dx), tiny)));
          lo = __dadd_rn(H->low_init[a], __dmul_rn((double)f, dx));
        } else {
          unsigned int f = (unsigned int)floor(dmax(0.0, __dsub_rn(__ddiv_rn(__dsub_rn(H->min_init[a], mn[a]), dx), tiny)));
          lo = __dsub_rn(H->low_init[a], __dmul_rn((double)f, dx));
        }
        s_low[a] = lo;
        s_high[a] = hi;
      }
    }
    if (!P.pbc) {
#pragma unroll
      for (int a = 0; a < D; ++a) s_stop[a] = __dadd_rn(s_high[a], dx);
    }
    s_ok = 1;
  }
  __syncthreads();
  // arange (tools.hpp:291-296): one warp per axis
  if (wid < D) {
    double* ax = wid == 0 ? A.gx : (wid == 1 ? A.gy : A.gz);
    const uint32_t cap = A.cap_axis[wid];
    const uint32_t n = arange_axis(s_low[wid], s_stop[wid], P.dx, cap, ax);
    if (lane == 0) {
      H->N[wid] = n;
      H->org[wid] = s_low[wid];
      if (n > cap || n < 4 || n >= kMaxAxisNodes) atomicExch(&s_ok, 0);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (D == 2) {
      H->N[2] = 1;
      H->org[2] = 0.0;
    }
    constexpr int TB = Tiling<D>::TB;
    uint64_t G = (uint64_t)H->N[0] * H->N[1] * H->N[2];
    H->T[0] = (H->N[0] + TB - 1) / TB;
    H->T[1] = (H->N[1] + TB - 1) / TB;
    H->T[2] = D == 3 ? (H->N[2] + TB - 1) / TB : 1;
    uint64_t nt = (uint64_t)H->T[0] * H->T[1] * H->T[2];
    if (!s_ok || G > A.cap_nodes || nt > A.cap_tiles) {
      H->abort = 1;
      atomicOr(&H->status, MTR_STATUS_GRID_OVERFLOW);
    }
    H->G = (uint32_t)G;
    H->ntiles = (uint32_t)nt;
  }
}

template <int D>
__device__ __forceinline__ void tail_body(const StepCommon& A, int out_parity);

// AFTER_TAIL: commits the step before first (its k_tail), for steps enqueued
// one behind the other: one launch less per step
template <int D, bool AFTER_TAIL = false>
__global__ void __launch_bounds__(256) k_header(StepCommon A) {
  if constexpr (AFTER_TAIL) {
    tail_body<D>(A, 1 - A.out_parity);  // the step before wrote what this one reads
    __syncthreads();
  }
  header_body<D>(A);
}

// ---------------------------------------------------------------------------
// 3. stable counting sort of (blocked cell key, input position), four launches:
//   k_sort_keys   key of every particle; its arrival rank in the cell from one
//                 atomic per warp and cell; counts per cell and per kSuperCells cells
//   k_sort_scan   exclusive scan of the cell counts (one block per kSuperCells
//                 cells, whose base is the sum of the super counts before it);
//                 leaves cell_start and clears the counts for the next step
//   k_sort_place  particle index to cell_start + arrival rank
//   k_sort_rank   stable order inside each cell: a particle's place is the
//                 number of smaller indices in its cell
// The last state is nearly in cell order, so all accesses are nearly
// coalesced.  Bound: launches and memory latency.  An LSD radix sort of the
// same keys needs three launches per 8-bit digit (9 for the 18-bit keys of the
// 1M-particle collapse) and a pass over the sorted keys for the tile ranges,
// which here are cell_start itself.
// Measured on a B200, per step: the radix sort with its memsets and tile ranges
// 11-16 launches and about 80 us at 1,024,000 particles; this one 4 launches,
// 49 us (CUDA events around every launch, 4 us each of which is the event).
// Whole steps: 5k particles in 2D 122 -> 100 us, 51,200 in 2D 138 -> 111 us,
// 150k in 3D 250 -> 210 us, 1,024,000 in 3D FP64 1123 -> 1089 us.
// A cell's ranking is quadratic in its particles (about 8 in 3D), which up to
// kBigCell of them costs less than another launch; larger cells are ordered by
// a whole block each (order_cell).
// Keys past the grid's cells (particles outside every tile) share one cell
// after the last, which no tile reads.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ uint32_t cell_key(const StepHeader* H, double ioh, const double (&x)[3]) {
  constexpr int SH = Tiling<D>::SH, TB = Tiling<D>::TB;
  int c[3] = {0, 0, 0};
#pragma unroll
  for (int a = 0; a < D; ++a) c[a] = (int)floor((x[a] - H->org[a]) * ioh);
  uint32_t t, in;
  if constexpr (D == 3) {
    t = ((uint32_t)(c[0] >> SH) * H->T[1] + (uint32_t)(c[1] >> SH)) * H->T[2] + (uint32_t)(c[2] >> SH);
    in = ((uint32_t)(c[0] & (TB - 1)) * TB + (uint32_t)(c[1] & (TB - 1))) * TB + (uint32_t)(c[2] & (TB - 1));
  } else {
    t = (uint32_t)(c[0] >> SH) * H->T[1] + (uint32_t)(c[1] >> SH);
    in = (uint32_t)(c[0] & (TB - 1)) * TB + (uint32_t)(c[1] & (TB - 1));
  }
  return t * 64u + in;
}

__device__ __forceinline__ uint32_t sort_cell(const StepHeader* H, uint32_t key) {
  const uint32_t last = H->ntiles * 64u;
  return key < last ? key : last;
}

// counts the key of particle i (all threads of the block call) and keeps its
// arrival rank.  The super counts are few, so their atomics are merged over the
// block: one per run of warps that lie within the same kSuperCells cells.
__device__ __forceinline__ void sort_count(const StepCommon& A, uint32_t i, bool valid, uint32_t key) {
  __shared__ uint32_t wsup[kSortThreads / 32], wnum[kSortThreads / 32];
  const uint32_t cell = valid ? sort_cell(A.H, key) : 0xffffffffu;
  const unsigned peers = __match_any_sync(0xffffffffu, cell);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, leader = __ffs(peers) - 1;
  uint32_t first = 0;
  if (valid && lane == leader) first = atomicAdd(&A.cell_count[cell], (uint32_t)__popc(peers));
  const uint32_t sup = valid ? cell / kSuperCells : 0xffffffffu;
  const unsigned speers = __match_any_sync(0xffffffffu, sup);
  if (lane == 0) {
    wsup[warp] = sup;
    wnum[warp] = valid ? (uint32_t)__popc(speers) : 0u;
  } else if (valid && lane == __ffs(speers) - 1) {
    atomicAdd(&A.super[sup], (uint32_t)__popc(speers));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = wsup[0], n = wnum[0];
#pragma unroll
    for (int w = 1; w < kSortThreads / 32; ++w) {
      if (wsup[w] != s) {
        if (n) atomicAdd(&A.super[s], n);
        s = wsup[w];
        n = 0;
      }
      n += wnum[w];
    }
    if (n) atomicAdd(&A.super[s], n);
  }
  first = __shfl_sync(0xffffffffu, first, leader);
  if (valid) A.perm_rank[i] = first + __popc(peers & ((1u << lane) - 1u));
}

template <int D>
__device__ __forceinline__ void sort_keys_body(const StepCommon& A, const uint32_t bid) {
  if (step_inactive(A.H)) return;
  const uint32_t i = bid * kSortThreads + threadIdx.x;
  const bool valid = i < A.Np;
  uint32_t k = 0;
  if (valid) {
    double x[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < D; ++a) x[a] = A.xin[(size_t)a * A.Np + i];
    k = cell_key<D>(A.H, A.P->one_over_dx, x);
    A.keys0[i] = k;
  }
  sort_count(A, i, valid, k);
}

template <int D>
__global__ void __launch_bounds__(kSortThreads) k_sort_keys(StepCommon A) {
  sort_keys_body<D>(A, blockIdx.x);
}

// sum over the block's 256 threads, to every thread; `ws` holds 8 values
__device__ __forceinline__ uint32_t block_sum256(uint32_t v, uint32_t* ws) {
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t s = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) s += ws[w];
  __syncthreads();
  return s;
}

// exclusive prefix over the block's 256 threads; total to every thread
__device__ __forceinline__ uint32_t block_prefix256(uint32_t v, uint32_t* ws, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += u;
  }
  if (lane == 31) ws[warp] = incl;
  __syncthreads();
  uint32_t pre = 0, sum = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    pre += w < warp ? ws[w] : 0u;
    sum += ws[w];
  }
  __syncthreads();
  total = sum;
  return pre + incl - v;
}

static __device__ __forceinline__ void sort_scan_body(const StepCommon& A, const uint32_t bid) {
  StepHeader* H = A.H;
  if (step_inactive(H)) return;
  const uint32_t ncell = H->ntiles * 64u + 1u, first = bid * kSuperCells;  // the last one: past the grid
  if (first >= ncell) return;
  __shared__ uint32_t ws[8];
  uint32_t before = 0;
  for (uint32_t s = threadIdx.x; s < bid; s += kSortThreads) before += A.super[s];
  const uint32_t base = block_sum256(before, ws);
  constexpr int PER = kSuperCells / kSortThreads;
  uint4* cnt = reinterpret_cast<uint4*>(A.cell_count + first) + threadIdx.x * (PER / 4);
  uint4* out = reinterpret_cast<uint4*>(A.cell_start + first) + threadIdx.x * (PER / 4);
  uint32_t c[PER], sum = 0;
#pragma unroll
  for (int q = 0; q < PER / 4; ++q) {
    const uint4 u = cnt[q];
    c[4 * q] = u.x;
    c[4 * q + 1] = u.y;
    c[4 * q + 2] = u.z;
    c[4 * q + 3] = u.w;
  }
#pragma unroll
  for (int q = 0; q < PER; ++q) sum += c[q];
  uint32_t total;
  uint32_t at = base + block_prefix256(sum, ws, total);
  if (sum) {
#pragma unroll
    for (int q = 0; q < PER / 4; ++q) cnt[q] = make_uint4(0u, 0u, 0u, 0u);
  }
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const uint32_t n = c[q], cell = first + threadIdx.x * PER + q;
    if (n > kBigCell && cell + 1 < ncell) A.big_cells[atomicAdd(&H->nbig, 1u)] = cell;
    c[q] = at;
    at += n;
  }
#pragma unroll
  for (int q = 0; q < PER / 4; ++q) out[q] = make_uint4(c[4 * q], c[4 * q + 1], c[4 * q + 2], c[4 * q + 3]);
}

static __global__ void __launch_bounds__(kSortThreads) k_sort_scan(StepCommon A) { sort_scan_body(A, blockIdx.x); }

static __device__ __forceinline__ void sort_place_body(const StepCommon& A, const uint32_t bid) {
  if (step_inactive(A.H)) return;
  if (bid == 0)  // the scan has read the super counts
    for (uint32_t s = threadIdx.x; s * kSuperCells <= A.H->ntiles * 64u; s += kSortThreads) A.super[s] = 0u;
  const uint32_t i = bid * kSortThreads + threadIdx.x;
  if (i < A.Np) A.perm_tmp[A.cell_start[sort_cell(A.H, A.keys0[i])] + A.perm_rank[i]] = i;
}

static __global__ void __launch_bounds__(kSortThreads) k_sort_place(StepCommon A) { sort_place_body(A, blockIdx.x); }

// Orders the members of one large cell, perm_tmp[b, e), by a whole block: they
// are marked in a bitmap of the indices from the least one not yet placed, and a
// member's place is the count of marks before its own.  After a step a cell's
// members lie close together, so one or two windows of the bitmap hold them all;
// in shuffled input a cell of m members takes at most N / 65536 + 1 windows of two
// passes over the m.  Every window places its first member at least.
// Bound: the latency of a few passes over the cell's members.  A walk over the keys
// of all particles instead takes 4000 rounds a cell at 1M particles: the kernel
// lasted 1516 us with one cell of 3000 among 1M, 11 us without it; us per step
// 3477 -> 1968 (FP64), 3156 -> 1667 (mixed).
constexpr uint32_t kMarkWords = 2048;
static __device__ void order_cell(const StepCommon& A, uint32_t b, uint32_t e) {
  constexpr uint32_t WIN = kMarkWords * 32, PER = kMarkWords / kSortThreads;
  __shared__ uint32_t marks[kMarkWords], pre[kMarkWords], ws[kSortThreads / 32];
  auto block_min = [&](uint32_t v) {
    v = __reduce_min_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    for (int w = 0; w < kSortThreads / 32; ++w) v = min(v, ws[w]);
    __syncthreads();
    return v;
  };
  uint32_t lo = 0xffffffffu;
  for (uint32_t q = b + threadIdx.x; q < e; q += kSortThreads) lo = min(lo, A.perm_tmp[q]);
  lo = block_min(lo);
  for (uint32_t at = b; at < e && lo != 0xffffffffu;) {  // (lo is an index while members are left)
    for (uint32_t w = threadIdx.x; w < kMarkWords; w += kSortThreads) marks[w] = 0u;
    __syncthreads();
    uint32_t next = 0xffffffffu;
    for (uint32_t q = b + threadIdx.x; q < e; q += kSortThreads) {
      const uint32_t i = A.perm_tmp[q], d = i - lo;
      if (i < lo) continue;  // placed by an earlier window
      if (d < WIN)
        atomicOr(&marks[d >> 5], 1u << (d & 31u));
      else
        next = min(next, i);
    }
    __syncthreads();
    uint32_t n = 0, total;
    for (uint32_t w = 0; w < PER; ++w) n += __popc(marks[threadIdx.x * PER + w]);
    n = block_prefix256(n, ws, total);
    for (uint32_t w = 0; w < PER; ++w) {
      pre[threadIdx.x * PER + w] = n;
      n += __popc(marks[threadIdx.x * PER + w]);
    }
    __syncthreads();
    for (uint32_t q = b + threadIdx.x; q < e; q += kSortThreads) {
      const uint32_t i = A.perm_tmp[q], d = i - lo;
      if (i >= lo && d < WIN) A.perm_rank[at + pre[d >> 5] + __popc(marks[d >> 5] & ((1u << (d & 31u)) - 1u))] = i;
    }
    at += total;
    lo = block_min(next);
  }
}

static __device__ __forceinline__ void sort_rank_body(const StepCommon& A, const uint32_t bid, const uint32_t nblk) {
  const StepHeader* H = A.H;
  if (step_inactive(H)) return;
  const uint32_t p = bid * kSortThreads + threadIdx.x;
  if (p < A.Np) {
    const uint32_t i = A.perm_tmp[p], cell = A.keys0[i];
    if (cell >= H->ntiles * 64u) {
      A.perm_rank[p] = i;
    } else {
      const uint32_t b = A.cell_start[cell], e = A.cell_start[cell + 1];
      if (e - b <= kBigCell) {
        uint32_t r = b;
        for (uint32_t q = b; q < e; ++q) r += A.perm_tmp[q] < i ? 1u : 0u;
        A.perm_rank[r] = i;
      }
    }
  }
  const uint32_t nbig = H->nbig;
  if (bid >= nbig) return;  // the whole block together below
  for (uint32_t g = bid; g < nbig; g += nblk) {
    const uint32_t cell = A.big_cells[g];
    order_cell(A, A.cell_start[cell], A.cell_start[cell + 1]);
  }
}

static __global__ void __launch_bounds__(kSortThreads) k_sort_rank(StepCommon A) {
  sort_rank_body(A, blockIdx.x, gridDim.x);
}

// particles [pb, pe) of tile t
__device__ __forceinline__ void tile_range(const StepCommon& A, uint32_t t, uint32_t& pb, uint32_t& pe) {
  pb = A.cell_start[t * 64u];
  pe = A.cell_start[t * 64u + 64u];
}

// Blocks that a tile of n particles takes of the `launched` ones: each loads,
// clears and adds a patch of its own, so a block gets an eighth of a full tile
// (at 8 particles a cell in 3D, 4 in 2D), a chunk a warp, before the next one takes
// part.  us per step with all launched blocks and with this rule, FP64 and mixed:
// 20k particles at one a cell 144 -> 118 and 120 -> 100, 150k 456 -> 361 and 330 ->
// 265, 60k in a layer one cell thick in x 151 -> 134 and 133 -> 114; full tiles (60k,
// 125k) 130, 131 and 167, 167.  A quarter of a tile a block: 106 and 95 for the first,
// but 8553 particles, whose tiles are half full, 82 -> 87 (mixed), here 83.
template <int D>
__device__ __forceinline__ uint32_t tile_blocks(uint32_t n, uint32_t launched) {
  constexpr uint32_t unit = D == 3 ? 64 : 32;
  return min(launched, (n + unit - 1) / unit);
}

// Share `part` of `parts` of a tile's particles [pb, pe): even, cut at whole warps.
__device__ __forceinline__ void part_range(uint32_t part, uint32_t parts, uint32_t& pb, uint32_t& pe) {
  const uint32_t n = pe - pb, b = pb;
  pb = b + (n * part / parts & ~31u);
  if (part + 1 < parts) pe = b + (n * (part + 1) / parts & ~31u);
}

// This warp's run [b, e) of a tile's sorted particles, one of at most 32 (4 blocks
// of 8 warps), each a lane's below.  The tile's 64 cells are shared out evenly, so
// that a run starts with a row of cells, unless a run then holds far more than its
// share of the particles and takes more chunks of CH: such tiles (crowded cells,
// layers) are cut by particles, at whole chunks where every run has one.  us per
// step, equal cells and this rule: 960k particles in a layer one cell thick in x
// 1762, 981 (mixed 1128, 748); 1M and one cell of 3000 more 1968, 846 (mixed 1667,
// 718).  FAR: 2.5 times the share.  In FP64 with one block a tile a quarter over it
// is enough (EVEN), which the faces of a body gain from: 96 steps of the 1M column
// 89.6 -> 86.6 ms, 500k two cells thick in x 598 -> 440 us a step.  More blocks have
// runs of one or two chunks, and a run that starts inside a row of cells adds a
// window: 42k particles 102 -> 104 us a step with the lower line.  In FP32 four warps
// instead of two on the same nodes of a face order their sums in more ways: 1M column
// 63.5 -> 62.4 ms, but 15-18 in 100 runs then leave the FP64 run's side of a stick-slip
// threshold at the floor within 80 steps, 1 in 100 with FAR.
// TRIM: the tile takes fewer blocks than launched where it is sparse.  False if
// the block has none.  All lanes call together; `cs` = the tile's 65 cell starts,
// lo and hi = even_run of all launched warps, which a kernel loads before it looks
// at the header (one memory latency less: us per step of 51,200 particles in 2D
// 70.4 -> 69.5, per no-allocation transfer of 4k 38.8 -> 37.4).
__device__ __forceinline__ void even_run(const uint32_t* __restrict__ cs, int runs, uint32_t& lo, uint32_t& hi) {
  const int lane = threadIdx.x & 31;
  lo = cs[64 * min(lane, runs) / runs];
  hi = cs[64 * min(lane + 1, runs) / runs];
}
template <int D, uint32_t CH, bool EVEN, bool TRIM = true>
__device__ __forceinline__ bool warp_run(const uint32_t* __restrict__ cs, int part, int launched, uint32_t lo, uint32_t hi,
                                         uint32_t& b, uint32_t& e) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  int runs = launched * nwarps;
  const uint32_t p0 = __shfl_sync(0xffffffffu, lo, 0), n = __shfl_sync(0xffffffffu, hi, runs - 1) - p0;
  const int parts = TRIM ? (int)tile_blocks<D>(n, launched) : launched;
  if (part >= parts) return false;
  if (TRIM && parts < launched) {
    runs = parts * nwarps;
    even_run(cs, runs, lo, hi);
  }
  const uint32_t worst = __reduce_max_sync(0xffffffffu, hi - lo);
  const uint32_t share = (n + runs - 1) / runs;
  const bool far = EVEN && launched == 1 ? worst - worst / 5 > share : worst / 5 * 2 > share;
  if (far && (worst + CH - 1) / CH > (share + CH - 1) / CH) {
    const uint32_t r = min(lane, runs), unit = n >= CH * runs ? CH : 1, m = (n + unit - 1) / unit;
    lo = p0 + min(n, m * r / runs * unit);
    hi = p0 + min(n, m * min(r + 1, (uint32_t)runs) / runs * unit);
  }
  const int first = part * nwarps;
  b = __shfl_sync(0xffffffffu, lo, first + warp);
  e = __shfl_sync(0xffffffffu, hi, first + warp);
  return __shfl_sync(0xffffffffu, lo, first) != __shfl_sync(0xffffffffu, hi, first + nwarps - 1);
}

// the cell of a tile that holds its sorted particle k (all lanes call together)
__device__ __forceinline__ int cell_of(const uint32_t (&cstart)[65], uint32_t k) {
  const int lane = threadIdx.x & 31;
  return __popc(__ballot_sync(0xffffffffu, cstart[lane + 1] <= k)) + __popc(__ballot_sync(0xffffffffu, cstart[lane + 33] <= k));
}

template <int D>
__device__ __forceinline__ void tile_coords(const StepHeader* H, uint32_t t, int (&tc)[3]) {
  if constexpr (D == 3) {
    tc[2] = (int)(t % H->T[2]);
    uint32_t r = t / H->T[2];
    tc[1] = (int)(r % H->T[1]);
    tc[0] = (int)(r / H->T[1]);
  } else {
    tc[2] = 0;
    tc[1] = (int)(t % H->T[1]);
    tc[0] = (int)(t / H->T[1]);
  }
}

// Sets the patch origin n0 of tile t and copies the grid coordinates its
// stencils can reach into crd.
template <int D>
__device__ __forceinline__ void load_tile_setup(const StepCommon& A, const StepHeader* H, uint32_t t, int (&n0)[3],
                                                double (*crd)[Tiling<D>::PN]) {
  constexpr int PN = Tiling<D>::PN, TB = Tiling<D>::TB;
  int tc[3];
  tile_coords<D>(H, t, tc);
  n0[0] = tc[0] * TB - 1;
  n0[1] = tc[1] * TB - 1;
  n0[2] = D == 3 ? tc[2] * TB - 1 : 0;
  for (int i = threadIdx.x; i < D * PN; i += blockDim.x) {
    const int a = i / PN, o = i % PN;
    const int g = n0[a] + o;
    const double* ax = a == 0 ? A.gx : (a == 1 ? A.gy : A.gz);
    crd[a][o] = (g >= 0 && g < (int)H->N[a]) ? ax[g] : 0.0;
  }
}

// local stencil base of a particle in its tile patch; false if outside
template <int D>
__device__ __forceinline__ bool local_base(const StepHeader* H, const double (&xp)[3], double ioh, const int (&n0)[3],
                                           bool clamp, int (&lb)[3]) {
  constexpr int PN = Tiling<D>::PN;
  bool ok = true;
  lb[0] = lb[1] = lb[2] = 0;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    int b = (int)floor((xp[a] - H->org[a]) * ioh) - 1;
    if (clamp) b = b < 0 ? 0 : b;
    lb[a] = b - n0[a];
    if (b < 0 || lb[a] < 0 || lb[a] > PN - 4 || b + 3 >= (int)H->N[a]) ok = false;
  }
  return ok;
}

// global node of patch entry n, or false outside the grid
template <int D>
__device__ __forceinline__ bool patch_node(const StepHeader* H, const int (&n0)[3], int n, uint32_t& l) {
  constexpr int PN = Tiling<D>::PN;
  int li, lj, lk;
  if constexpr (D == 3) {
    lk = n % PN;
    lj = (n / PN) % PN;
    li = n / (PN * PN);
  } else {
    lk = 0;
    lj = n % PN;
    li = n / PN;
  }
  const int gi = n0[0] + li, gj = n0[1] + lj, gk = n0[2] + lk;
  if (gi < 0 || gj < 0 || gk < 0 || gi >= (int)H->N[0] || gj >= (int)H->N[1] || gk >= (int)H->N[2]) return false;
  l = node_index(H, gi, gj, gk);
  return true;
}

// ---------------------------------------------------------------------------
// 5. P2G + stress force, one block per tile (or per part of one), each warp on
// its own.
//
// A warp takes a run of the tile's cells, whose sorted particles lie together.
// It stages 16 particles at a time in its own part of shared memory (weights,
// offsets and the factors of momentum and force), then every lane accumulates
// its stencil column over them, cell by cell.  A column is the 4 nodes along
// the innermost axis; its sums stay in registers as a window that slides with
// the cells, so a node is added to the shared patch once per row of cells (7
// nodes for 4 cells) instead of once per cell or per few particles.  All
// control flow is the same for the whole warp: the cells' ranges come from the
// sort.  Where a particle's columns leave lanes over (2D, or without the
// force), the warp's groups of lanes take the cell's particles in turn and their
// sums are exchanged when a node leaves the window.  There is no block barrier
// between the start and the flush of the patch (one global atomic per node and
// channel).
//
// The lanes of a group come in two roles with the same code: role 0 sums mass
// and momentum, role 1 the force (and friction).  With per-axis factors w and
// a (role 0: weight times offset x_i - x_p; role 1: weight derivative) a
// column's contribution to channel c is
//   f1_h A_c + f2_h B_c,   f1 = w, f2 = a along the innermost axis,
//   A_c = w w V_c + a w X_c + w a Y_c,  B_c = w w Z_c,
// with V, X, Y, Z the velocity and the columns of B D^-1 (role 0), or zero and
// the rows of the stress (role 1): 2 multiply-adds per node and channel.
// A particle's 16 columns (2D: 4) take 32 lanes (2D: 8); half of that, two
// columns a lane, needed 28% more registers and measured slower (FP64 0.41 ms
// against 0.33 on the 1M collapse).
//
// Bound: FP64 issue and shared-memory loads of the factors.
// In the sum phase the shared-memory pipe is 73% busy in FP64 (32 wavefronts a
// particle, most of them 16-byte loads of the factors; ncu).  ms per launch:
// 1,024,000 particles, cubic, FP64 0.403 -> 0.280, mixed 0.242 -> 0.183; 2M
// quadratic mixed 0.465 -> 0.320; 51,200 in 2D FP64 0.062 -> 0.020.  A group of
// lanes on its own run of 4 cells, with its particles' bases checked one by one,
// took 0.291, 0.191, 0.351 and 0.024.
// Tried: holding the next chunk's particles in registers while one is summed
// (spills, 0.35 -> 0.52), a third register bound (80 registers, 0.45).
// ---------------------------------------------------------------------------
constexpr int kChunk = 128;  // default block size of the tile kernels
// Largest block of the tile kernels.  The scatter kernels stage one particle
// per thread, so their shared memory grows with the block; k_g2p_t stays at
// kChunk threads at most (its register bound below is per 128-thread block).
constexpr int kMaxTileThreads = 256;

// Minimum resident blocks of 128 threads per SM requested for the tile kernels
// that run the return mapping; it bounds their registers per thread.  Four
// blocks of 128 threads (128 registers, some spilled to L1) measured 15-25%
// faster for k_defgrad_t than the unbounded two blocks (240 registers) on the
// 3D collapse.
// The FP32-storage form holds fewer live values and gains from a tighter bound:
// six blocks of 128 threads (80 registers) measured 6% faster for its
// k_defgrad_t on the 3D collapse than four.  The FP64 form keeps four: six
// measured 2% faster (0.295 -> 0.287 ms at step 300 of the 1M collapse) but
// spilled to DRAM, writing 378 MB per launch instead of 150 MB (ncu).
#ifndef MTR_DEFGRAD_MIN_BLOCKS
#define MTR_DEFGRAD_MIN_BLOCKS 4
#endif
#ifndef MTR_DEFGRAD_MIN_BLOCKS_F32
#define MTR_DEFGRAD_MIN_BLOCKS_F32 6
#endif
// Resident blocks of kChunk threads of k_g2p_t: with one plastic model compiled
// in, four in FP64 and five with FP32 storage (1.2M Cam-Clay incline FP64 0.505
// -> 0.488 ms, mixed 0.458 -> 0.392, 2M DP mixed 0.339 -> 0.299 against three);
// three for the generic kernel, which spills under more (150k elastic FP64
// 0.050 against 0.062).
template <typename R, int PM>
constexpr int g2p_min_blocks() {
  return PM < 0 ? 3 : (sizeof(R) == 4 ? 5 : 4);
}
// the same register bound for blocks of up to kMaxTileThreads threads (R is
// the storage type of the kernel the bound is written on)
// (the generic kernel spills 1.8 KB a thread under the FP32 form's bound: it takes the FP64 one's)
#define MTR_DEFGRAD_BOUNDS \
  kMaxTileThreads, ((sizeof(R) == 4 && PM >= 0 ? MTR_DEFGRAD_MIN_BLOCKS_F32 : MTR_DEFGRAD_MIN_BLOCKS) * kChunk / kMaxTileThreads)

#ifndef MTR_P2G_MIN_BLOCKS
#define MTR_P2G_MIN_BLOCKS 2
#endif
#ifndef MTR_P2G_MIN_BLOCKS_F32
#define MTR_P2G_MIN_BLOCKS_F32 3
#endif
#define MTR_P2G_BOUNDS kMaxTileThreads, (sizeof(R) == 4 ? MTR_P2G_MIN_BLOCKS_F32 : MTR_P2G_MIN_BLOCKS)
// A staged particle of the P2G: per axis the 4 weights and the second factor
// of each role, the channel factors V, X, Y, Z (2D: V, X, Z) of each role.
// Padded to an odd multiple of 16 bytes, so that the lanes that stage
// neighbouring slots store to different banks (a 512-byte stride made the
// FP64 stores 16-way conflicts, 65% of the kernel's shared-memory cycles).
template <int D, typename R, int ROLES>
struct PStageData {
  R w[D][4], a[ROLES][D][4];
  R q[ROLES][D][4];
  R mui;  // factor of role 1's fourth channel, the mu(I) deviation (role 0: 1, the mass)
};
constexpr size_t stage_stride(size_t n) {
  n = align16(n);
  return n % 32 ? n : n + 16;
}
template <int D, typename R, int ROLES>
struct __align__(16) PStage : PStageData<D, R, ROLES> {
  char pad[stage_stride(sizeof(PStageData<D, R, ROLES>)) - sizeof(PStageData<D, R, ROLES>)];
};
constexpr int kStage = 16;  // particles a warp stages at a time

// local stencil base along an axis, with the patch's first node n0, of the
// particles of the tile's cell c (the cell's floor, clamped at the grid's first
// node, p2g.cpp:21-24)
__device__ __forceinline__ int cell_base(int n0, int c) { return max(n0 + c, 0) - n0; }

// One step of a sum over the two halves of a warp's lanes that differ in the bit
// off: the half without the bit returns the sum of both halves' a, the other
// that of their b.  Half the exchanges of summing a and b in every lane.
template <typename R>
__device__ __forceinline__ R half_sum(R a, R b, int off) {
  const bool up = threadIdx.x & off;
  return (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, off);
}

// The sliding register window of a scatter: a lane's sums of NC channels on the
// 4 innermost nodes of one stencil column.  GR = 32 / LPP groups of a warp's
// lanes hold the same columns for different particles of a cell; their sums are
// taken together when a node leaves the window.  All lanes call together.
template <typename R, int NC, int LPP>
struct Window {
  static constexpr int GR = 32 / LPP;
  R acc[4][NC];
  __device__ __forceinline__ Window() {
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[h][c] = R(0.0);
  }
  static __device__ __forceinline__ R group_sum(R v, int from) {
#pragma unroll
    for (int off = from; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
  }
  // adds the first node to dst(channel)[node], and moves by one node
  template <typename Dst>
  __device__ __forceinline__ void advance(int grp, int& node, Dst&& dst) {
    if constexpr (GR == 1) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (acc[0][c] != R(0.0)) atomicAdd(dst(c) + node, acc[0][c]);
    } else {  // channels in pairs, one for each half of the groups
#pragma unroll
      for (int c = 0; c + 1 < NC; c += 2) {
        const R v = group_sum(half_sum(acc[0][c], acc[0][c + 1], LPP), 2 * LPP);
        if (grp < 2 && v != R(0.0)) atomicAdd((grp ? dst(c + 1) : dst(c)) + node, v);
      }
      if constexpr (NC % 2) {
        const R v = group_sum(acc[0][NC - 1], LPP);
        if (grp == 0 && v != R(0.0)) atomicAdd(dst(NC - 1) + node, v);
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
      for (int h = 0; h < 3; ++h) acc[h][c] = acc[h + 1][c];
      acc[3][c] = R(0.0);
    }
    ++node;
  }
  // adds all 4 nodes, each group its share of them, and clears the window
  template <typename Dst>
  __device__ __forceinline__ void flush(int grp, int node, Dst&& dst) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      if constexpr (GR == 1) {
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (acc[h][c] != R(0.0)) atomicAdd(dst(c) + node + h, acc[h][c]);
      } else {
        const R lo = half_sum(acc[0][c], acc[1][c], LPP), hi = half_sum(acc[2][c], acc[3][c], LPP);
        if constexpr (GR == 2) {
          if (lo != R(0.0)) atomicAdd(dst(c) + node + grp, lo);
          if (hi != R(0.0)) atomicAdd(dst(c) + node + 2 + grp, hi);
        } else {
          const R v = group_sum(half_sum(lo, hi, 2 * LPP), 4 * LPP);
          if (grp < 4 && v != R(0.0)) atomicAdd(dst(c) + node + grp, v);
        }
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) acc[h][c] = R(0.0);
    }
  }
};

// node of a lane's column (ix, iy) that a window at cell c of a tile starts at
template <int D>
__device__ __forceinline__ int window_node(const int (&n0)[3], int c, int ix, int iy) {
  constexpr int PN = Tiling<D>::PN;
  if constexpr (D == 3)
    return ((cell_base(n0[0], c >> 4) + ix) * PN + cell_base(n0[1], (c >> 2) & 3) + iy) * PN + cell_base(n0[2], c & 3);
  else
    return (cell_base(n0[0], c >> 3) + ix) * PN + cell_base(n0[1], c & 7);
}

// Nodes the window moves on by from a cell to a later one, 4 where it starts anew.
template <int D>
__device__ __forceinline__ int window_steps(const int (&n0)[3], int from, int to) {
  constexpr int TB = Tiling<D>::TB;
  if (from / TB != to / TB) return 4;
  return min(cell_base(n0[D - 1], to % TB) - cell_base(n0[D - 1], from % TB), 4);
}

// Largest block of the MUSL scatter and the resident blocks of that size its
// register bound asks for (FP64 and FP32 storage): what leaves the gather
// without spills (1M collapse, FP64 0.363 ms at 3, 0.380 at 4 and 0.382 at 5;
// mixed 0.230 at 5, 0.242 at 6).
#ifndef MTR_MUSL_MAX_THREADS
#define MTR_MUSL_MAX_THREADS 128
#endif
#ifndef MTR_MUSL_MIN_BLOCKS
#define MTR_MUSL_MIN_BLOCKS 3
#endif
#ifndef MTR_MUSL_MIN_BLOCKS_F32
#define MTR_MUSL_MIN_BLOCKS_F32 5
#endif
#define MTR_MUSL_BOUNDS MTR_MUSL_MAX_THREADS, (sizeof(R) == 4 ? MTR_MUSL_MIN_BLOCKS_F32 : MTR_MUSL_MIN_BLOCKS)

template <int D, typename R>
constexpr size_t p2g_crd_bytes() {
  return align16(sizeof(double) * 3 * Tiling<D>::PN);
}
// The patch's last channel (MIBF friction) is allocated only under MIBF: a
// block without it needs 2.7 KB (FP64, 3D) less shared memory, which lets
// five FP64 P2G blocks of 128 threads share an SM instead of four.
template <int D, typename R, bool FORCE = true>
__host__ __device__ constexpr size_t p2g_patch_bytes(bool mibf) {
  return align16(sizeof(R) * (FORCE ? Tiling<D>::NCH - (mibf ? 0 : 1) : 1 + D) * Tiling<D>::NODES);
}
template <int D, typename R, bool FORCE = true>
constexpr size_t p2g_smem_bytes(int threads, bool mibf = true) {
  return p2g_crd_bytes<D, R>() + p2g_patch_bytes<D, R, FORCE>(mibf) +
         kStage * sizeof(PStage<D, R, FORCE ? 2 : 1>) * (size_t)(threads / 32);
}

// FORCE: false for mass and momentum alone (no stress, no friction, no ids)
template <int D, int DEG, typename R, bool FORCE = true>
__device__ __forceinline__ void p2g_w_body(const StepArgsT<R>& A, const uint32_t* __restrict__ perm, const uint32_t bid,
                                                const uint32_t part, const uint32_t launched) {
  using TL = Tiling<D>;
  constexpr int PN = TL::PN, NODES = TL::NODES, NCH = FORCE ? TL::NCH : 1 + D, TB = TL::TB, Z = D - 1;
  // A lane sums NV vector components of a role and its scalar channel on one
  // stencil column (in 2D each component takes a lane, the first the scalar
  // too); GR groups of LPP lanes.
  constexpr int ROLES = FORCE ? 2 : 1, COLS = D == 3 ? 16 : 4, NV = D == 3 ? 3 : 1, NC = NV + 1;
  constexpr int LPP = COLS * ROLES * D / NV, GR = 32 / LPP;
  const StepHeader* H = A.H;
  const uint32_t t = bid;
  uint32_t lo, hi;
  even_run(A.cell_start + t * 64u, launched * (blockDim.x >> 5), lo, hi);
  if (step_inactive(H)) return;
  if (t >= H->ntiles) return;
  const int warp = threadIdx.x >> 5;
  uint32_t k0, wend;  // this warp's particles
  if (!warp_run<D, kStage, kFP64<R>, FORCE>(A.cell_start + t * 64u, part, launched, lo, hi, k0, wend)) return;
  const DevParams& P = *A.P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double(*crd)[PN] = reinterpret_cast<double(*)[PN]>(smem_raw);
  R(*patch)[NODES] = reinterpret_cast<R(*)[NODES]>(smem_raw + p2g_crd_bytes<D, R>());
  const bool mibf = FORCE && P.use_mibf;
  const int nch = !FORCE || mibf ? NCH : NCH - 1;  // channels the patch holds
  int tc[3];
  tile_coords<D>(H, t, tc);
  const int n0[3] = {tc[0] * TB - 1, tc[1] * TB - 1, D == 3 ? tc[2] * TB - 1 : 0};
  for (int i = threadIdx.x; i < nch * NODES; i += blockDim.x) (&patch[0][0])[i] = R(0.0);
  for (int i = threadIdx.x; i < D * PN; i += blockDim.x) {
    const int a = i / PN, o = i % PN;
    const int g = n0[a] + o;
    const double* ax = a == 0 ? A.gx : (a == 1 ? A.gy : A.gz);
    crd[a][o] = (g >= 0 && g < (int)H->N[a]) ? ax[g] : 0.0;
  }
  __shared__ uint32_t cstart[65];  // first particle of each cell of the tile
  for (int i = threadIdx.x; i < 65; i += blockDim.x) cstart[i] = A.cell_start[t * 64u + i];
  __syncthreads();
  const uint32_t Np = A.Np;
  const double ioh = P.one_over_dx;
  const R iohR = (R)ioh, apicD = (R)P.apicDinverse;
  const bool apic = P.flip_ratio < 0;
  const int lane = threadIdx.x & 31;
  const int grp = lane / LPP, role = lane / COLS % ROLES, col = lane % COLS;
  const int c0 = lane / (COLS * ROLES) % (D / NV);  // first component
  const int ix = D == 3 ? col >> 2 : col, iy = D == 3 ? col & 3 : 0;  // this lane's column
  using Stage = PStage<D, R, ROLES>;
  Stage* st = reinterpret_cast<Stage*>(smem_raw + p2g_crd_bytes<D, R>() + p2g_patch_bytes<D, R, FORCE>(mibf)) + warp * kStage;
  // patch channels of this role: c < D vector component, c == D mass or friction
  R* const vec = patch[role ? 1 + D : 1];
  R* const one = patch[role ? 1 + 2 * D : 0];
  auto dst = [&](int c) { return c < NV ? vec + (c0 + c) * NODES : one; };
  Window<R, NC, LPP> win;
  int node0 = 0;  // node of the window's first entry
  // adds a staged particle to the window; TINY: some node may fall under the
  // weight threshold of p2g.cpp:35 (mass and momentum of weights <= 1e-25 are
  // skipped, which is checked node by node for such a particle)
  auto add = [&](const Stage& S, auto tiny) {
    R f1[4], f2[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      f1[h] = S.w[Z][h];
      f2[h] = S.a[role][Z][h];
    }
    R u0 = S.w[0][ix], u1 = S.a[role][0][ix];
    [[maybe_unused]] R u2 = R(0.0);
    if constexpr (D == 3) {
      const R wy = S.w[1][iy], ay = S.a[role][1][iy];
      u2 = u0 * ay;
      u0 *= wy;
      u1 *= wy;
    }
    if constexpr (decltype(tiny)::value) {
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (role == 0 && !(f1[h] * u0 > R(1e-25))) f1[h] = f2[h] = R(0.0);
    }
#pragma unroll
    for (int c = 0; c < NV; ++c) {
      const R* f = S.q[role][c0 + c];
      R a1 = u0 * f[0] + u1 * f[1];
      if constexpr (D == 3) a1 += u2 * f[2];
      const R b1 = u0 * f[D];
#pragma unroll
      for (int h = 0; h < 4; ++h) win.acc[h][c] = f2[h] * b1 + (f1[h] * a1 + win.acc[h][c]);
    }
    const R a1 = c0 ? R(0.0) : u0 * (role ? S.mui : R(1.0));
#pragma unroll
    for (int h = 0; h < 4; ++h) win.acc[h][NV] += f1[h] * a1;
  };
  int cell = 0;
  if (k0 < wend) {
    cell = cell_of(cstart, k0);
    node0 = window_node<D>(n0, cell, ix, iy);
  }
  for (; k0 < wend; k0 += kStage) {
    __syncwarp();  // the last chunk has been read
    // Role 0 stores the weights, the weights times offsets, velocity and B,
    // role 1, in another lane, the weight derivatives, the stress and mu(I).
    // Both evaluate both second factors and keep theirs: a branch on the role
    // would run the two halves one after the other.
    bool tiny = false;
    const uint32_t s = k0 + lane % kStage;
    const int part = lane / kStage;  // the role this lane stages
    if (part < ROLES && s < wend) {
      Stage& S = st[lane % kStage];
      const uint32_t j = perm[s];
      double xp[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int a = 0; a < D; ++a) xp[a] = A.in.x[(size_t)a * Np + j];
      R qv[D][1 + D], mui = R(0.0);
      if (!FORCE || part == 0) {
#pragma unroll
        for (int a = 0; a < D; ++a) {
          qv[a][0] = A.in.v[(size_t)a * Np + j];
#pragma unroll
          for (int b = 0; b < D; ++b)
            qv[a][1 + b] = apic ? apicD * A.in.B[(size_t)(a * D + b) * Np + j] : R(0.0);
        }
      } else {
        R tau[Sym<D>::n];
#pragma unroll
        for (int i = 0; i < Sym<D>::n; ++i) tau[i] = iohR * A.in.tau[(size_t)i * Np + j];
#pragma unroll
        for (int a = 0; a < D; ++a) {
          qv[a][0] = R(0.0);
#pragma unroll
          for (int b = 0; b < D; ++b) qv[a][1 + b] = sym_at<D>(tau, a, b);
        }
        if (mibf) mui = (R)((double)A.in.sc[(size_t)MTR_SCALAR_MUI * Np + j] - P.mui0);
      }
      // The particle's cell, clamped at the first one; it must lie in the tile
      // and its stencil in the grid.  The sort sends a coordinate that is not
      // finite to the first cells, so the test is on the floor itself, which no
      // NaN passes; left of cell -2 every weight is zero.
      bool ok = true;
      int least = 0;
#pragma unroll
      for (int a = 0; a < D; ++a) {
        const double fl = floor((xp[a] - H->org[a]) * ioh);
        const int g = (int)fl, c = max(g, 0) - (n0[a] + 1);
        const bool in = fl >= -2.0 && (unsigned)c < (unsigned)TB;
        const int lb = cell_base(n0[a], in ? c : 0);
        ok = ok && in && lb + n0[a] + 3 < (int)H->N[a];
        R w[4], d[4], o[4];
        if constexpr (FORCE) {
          const double td = (xp[a] - crd[a][lb + 1]) * ioh;
          axis_weights<DEG, true, R>(td, w, d);
          if (g < 1) {  // clamped; through copies: w and d stay in registers otherwise
            R wc[4], dc[4];
            axis_weights_any<DEG, R>(td, wc, dc);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              w[h] = wc[h];
              d[h] = dc[h];
            }
          }
          axis_offsets<R>(td, P.dx, o);
        } else {  // a caller's axes: every node's own coordinate
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            o[h] = crd[a][lb + h] - xp[a];
            w[h] = bspline_N<DEG>((xp[a] - crd[a][lb + h]) * ioh);
            d[h] = R(0.0);
          }
        }
        least += FORCE && g >= 1 ? least_exponent<DEG, false>(w) : least_exponent<DEG, true>(w);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          if (part == 0) S.w[a][h] = w[h];
          S.a[part][a][h] = part ? d[h] : w[h] * o[h];
        }
      }
#pragma unroll
      for (int a = 0; a < D; ++a)
#pragma unroll
        for (int b = 0; b < 1 + D; ++b) S.q[part][a][b] = qv[a][b];
      if (part) S.mui = mui;
      tiny = least < -82;  // every product of weights is at least 2^least; 1e-25 < 2^-83
      if (!ok) {  // adds nothing
        if (part == 0) {
          if constexpr (FORCE)
            raise_status(A.H, MTR_STATUS_STENCIL_OOB, A.in.id[j]);
          else
            atomicOr(&A.H->status, MTR_STATUS_STENCIL_OOB);
#pragma unroll
          for (int a = 0; a < D; ++a)
#pragma unroll
            for (int h = 0; h < 4; ++h) S.w[a][h] = R(0.0);
        }
#pragma unroll
        for (int a = 0; a < D; ++a) {
#pragma unroll
          for (int h = 0; h < 4; ++h) S.a[part][a][h] = R(0.0);
#pragma unroll
          for (int b = 0; b < 1 + D; ++b) S.q[part][a][b] = R(0.0);
        }
        if (part) S.mui = R(0.0);
      }
    }
    const bool slow = __any_sync(0xffffffffu, tiny);  // (also orders the stage before its reads)
    __syncwarp();
    const uint32_t pend = min(k0 + kStage, wend);
    for (uint32_t k = k0;;) {
      const uint32_t e = min(cstart[cell + 1], pend);  // the cell's end within the chunk
      uint32_t i = k + grp;
      if (slow) {
#pragma unroll 1
        for (; i < e; i += GR) add(st[i - k0], std::true_type{});
      } else {
#pragma unroll (GR == 1 ? 2 : 1)
        for (; i < e; i += GR) add(st[i - k0], std::false_type{});
      }
      if constexpr (GR > 1) __syncwarp();
      k = e;
      if (k == pend) break;
      // the next cell that is not empty; the window moves there, or starts anew
      int next = cell + 1;
      while (cstart[next + 1] <= k) ++next;
      const int steps = window_steps<D>(n0, cell, next);
      cell = next;
      if (steps == 4) {
        win.flush(grp, node0, dst);
        node0 = window_node<D>(n0, cell, ix, iy);
      } else {
        for (int h = 0; h < steps; ++h) win.advance(grp, node0, dst);
      }
    }
  }
  win.flush(grp, node0, dst);
  __syncthreads();
  const uint32_t cap = A.cap_nodes;
  for (int n = threadIdx.x; n < NODES; n += blockDim.x) {
    uint32_t l;
    if (!patch_node<D>(H, n0, n, l)) continue;
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      if (ch >= nch) break;  // no friction channel without MIBF
      const R val = patch[ch][n];
      if (val != R(0.0)) atomicAdd(&A.acc[(size_t)ch * cap + l], val);
    }
  }
}

template <int D, int DEG, typename R>
__global__ void __launch_bounds__(MTR_P2G_BOUNDS) k_p2g_w(StepArgsT<R> A, const uint32_t* __restrict__ perm) {
  p2g_w_body<D, DEG, R>(A, perm, blockIdx.x, blockIdx.y, gridDim.y);
}

// ---------------------------------------------------------------------------
// 5b. periodic copies (pbc.cpp:37-85): a particle within 4 dx of x = Lx (else
// of x = 0) also scatters mass, momentum and force from x - Lx (else x + Lx),
// with the same stencil and formulas as P2G (p2g.cpp:6-100,
// explicit_euler_update.cpp:15-77).  Few particles have a copy; each one is a
// thread with global atomics.
// ---------------------------------------------------------------------------
template <int D, int DEG, typename R>
__global__ void __launch_bounds__(256) k_p2g_periodic(StepArgsT<R> A) {
  const StepHeader* H = A.H;
  if (step_inactive(H)) return;
  const DevParams& P = *A.P;
  constexpr int NS = Sym<D>::n, KN = D == 3 ? 4 : 1;
  const uint32_t Np = A.Np, cap = A.cap_nodes;
  const double ioh = P.one_over_dx, lim = 4.0 * P.dx, Lx = P.L[0], apicD = P.apicDinverse;
  const bool apic = P.flip_ratio < 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < Np; i += gridDim.x * blockDim.x) {
    double xp[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < D; ++a) xp[a] = A.in.x[(size_t)a * Np + i];
    double diff = Lx - xp[0];
    if (diff < lim && diff > 0) {
      xp[0] = -diff;
    } else {
      diff = xp[0];
      if (!(diff < lim && diff >= 0)) continue;
      xp[0] = Lx + diff;
    }
    double vp[3] = {0.0, 0.0, 0.0}, Bm[D][D], tau[NS];
#pragma unroll
    for (int a = 0; a < D; ++a) vp[a] = A.in.v[(size_t)a * Np + i];
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
      for (int c = 0; c < D; ++c) Bm[r][c] = apic ? (double)A.in.B[(size_t)(r * D + c) * Np + i] : 0.0;
#pragma unroll
    for (int q = 0; q < NS; ++q) tau[q] = A.in.tau[(size_t)q * Np + i];
    int base[3] = {0, 0, 0};
    bool oob = false;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const double fl = floor((xp[a] - H->org[a]) * ioh);
      const bool in = fl >= -2.0 && fl + 2.0 < (double)H->N[a];  // false for NaN; left of cell -2 no weight is left
      base[a] = in ? max((int)fl - 1, 0) : 0;                    // p2g.cpp:21-24 clamps at zero
      if (!in || base[a] + 3 >= (int)H->N[a]) oob = true;
    }
    if (oob) {
      raise_status(A.H, MTR_STATUS_STENCIL_OOB, A.in.id[i]);
      continue;
    }
    double w[3][4], dw[3][4], crd[3][4];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const double* ax = a == 0 ? A.gx : (a == 1 ? A.gy : A.gz);
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        crd[a][o] = ax[base[a] + o];
        const double u = (xp[a] - crd[a][o]) * ioh;
        w[a][o] = bspline_N<DEG>(u);
        dw[a][o] = bspline_dN<DEG>(u);
      }
    }
#pragma unroll
    for (int ii = 0; ii < 4; ++ii)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
#pragma unroll
        for (int kk = 0; kk < KN; ++kk) {
          const uint32_t l = node_index(H, base[0] + ii, base[1] + jj, D == 3 ? base[2] + kk : 0);
          const double wxy = w[0][ii] * w[1][jj];
          const double weight = D == 3 ? wxy * w[2][kk] : wxy;
          if (weight > 1e-25) {
            atomicAdd(&A.acc[l], (R)weight);
            const double pd[3] = {crd[0][ii] - xp[0], crd[1][jj] - xp[1], D == 3 ? crd[2][kk] - xp[2] : 0.0};
#pragma unroll
            for (int a = 0; a < D; ++a) {
              double bv = Bm[a][0] * pd[0];
#pragma unroll
              for (int c = 1; c < D; ++c) bv += Bm[a][c] * pd[c];
              atomicAdd(&A.acc[(size_t)(1 + a) * cap + l], (R)(weight * (vp[a] + apicD * bv)));
            }
          }
          double g[3];
          if constexpr (D == 3) {
            g[0] = dw[0][ii] * w[1][jj] * w[2][kk] * ioh;
            g[1] = w[0][ii] * dw[1][jj] * w[2][kk] * ioh;
            g[2] = w[0][ii] * w[1][jj] * dw[2][kk] * ioh;
          } else {
            g[0] = dw[0][ii] * w[1][jj] * ioh;
            g[1] = w[0][ii] * dw[1][jj] * ioh;
          }
#pragma unroll
          for (int a = 0; a < D; ++a) {
            double f = sym_at<D>(tau, a, 0) * g[0];
#pragma unroll
            for (int c = 1; c < D; ++c) f += sym_at<D>(tau, a, c) * g[c];
            if (f != 0.0) atomicAdd(&A.acc[(size_t)(1 + D + a) * cap + l], (R)f);
          }
        }
  }
}

// ---------------------------------------------------------------------------
// 6. grid update, one thread per node (arithmetic in FP64 on both paths)
// ---------------------------------------------------------------------------
template <int D, typename R>
__device__ __forceinline__ void grid_body(const StepArgsT<R>& A, const uint32_t bid, const uint32_t nblk) {
  StepHeader* H = A.H;
  if (step_inactive(H)) return;
  const DevParams& P = *A.P;
  const uint32_t G = H->G, cap = A.cap_nodes;
  const double dt = H->dt;
  const double dtpv_mp = dt * P.particle_volume / P.particle_mass;
  double dtg[3];
#pragma unroll
  for (int a = 0; a < D; ++a) dtg[a] = dt * H->gravity[a];
  __shared__ mtr_plate plates[MTR_MAXP];
  for (int i = threadIdx.x; i < P.nplates; i += blockDim.x) plates[i] = H->plates[i];
  __syncthreads();
  double sum_m = 0.0, sum_p[3] = {0.0, 0.0, 0.0};  // mass and momentum balance (simulation.cpp:292-333)
  for (uint32_t l = bid * blockDim.x + threadIdx.x; l < G; l += nblk * blockDim.x) {
    // every load of the node first, ahead of the branches on its mass: one
    // round of memory latency per node instead of several in a row
    const double mraw = A.acc[l];
    double pacc[3] = {0, 0, 0}, facc[3] = {0, 0, 0};
#pragma unroll
    for (int a = 0; a < D; ++a) {
      pacc[a] = A.acc[(size_t)(1 + a) * cap + l];
      facc[a] = A.acc[(size_t)(1 + D + a) * cap + l];
    }
    const double fracc = P.use_mibf ? (double)A.acc[(size_t)(1 + 2 * D) * cap + l] : 0.0;
    const uint32_t k = D == 3 ? l % H->N[2] : 0;
    const uint32_t r = D == 3 ? l / H->N[2] : l;
    const uint32_t jj = r % H->N[1], i = r / H->N[1];
    const double Xi0 = A.gx[i], Xi1 = A.gy[jj], Xi2 = D == 3 ? A.gz[k] : 0.0;
    double v[3] = {0, 0, 0}, vold[3] = {0, 0, 0};
    double fric = 0.0;
    sum_m += mraw;
    const double rm = 1.0 / mraw;  // one division for the node's six quotients
    if (mraw > 0) {
#pragma unroll
      for (int a = 0; a < D; ++a) {
        sum_p[a] += pacc[a];
        v[a] = pacc[a] * rm;
      }
    }
    if (P.use_mibf) fric = P.mui0 + fracc * rm;
    const double mi = mraw * P.particle_mass;
    double fl[3] = {0, 0, 0};
    if (mi > 0) {
#pragma unroll
      for (int a = 0; a < D; ++a) {
        double inc = -dtpv_mp * facc[a] * rm + dtg[a];
        vold[a] = v[a];
        v[a] = vold[a] + inc;
      }
      double Xi[3] = {Xi0, Xi1, Xi2};
      if (!boundary_collision<D>(P, plates, fric, Xi, dt, v)) raise_status(H, MTR_STATUS_BAD_BC, 0xffffffffu);
#pragma unroll
      for (int a = 0; a < D; ++a) fl[a] = v[a] - vold[a];
    }
#pragma unroll
    for (int a = 0; a < D; ++a) {
      A.nv[(size_t)a * cap + l] = v[a];
      A.nflip[(size_t)a * cap + l] = (R)fl[a];
    }
    A.nmass[l] = (R)mi;
    if (P.use_mibf) A.nfric[l] = (R)fric;
    if (P.use_musl) {
#pragma unroll
      for (int a = 0; a < D; ++a) A.v2[(size_t)a * cap + l] = 0.0;  // re-projection accumulator of this step
    }
#pragma unroll
    for (int ch = 0; ch < Tiling<D>::NCH; ++ch) A.acc[(size_t)ch * cap + l] = R(0.0);  // ready for the next step
  }
  double sums[1 + D];
  double* dst[1 + D];
  sums[0] = sum_m * P.particle_mass;
  dst[0] = &H->grid_mass;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    sums[1 + a] = sum_p[a] * P.particle_mass;
    dst[1 + a] = &H->grid_mom[a];
  }
  block_add<1 + D>(sums, dst);
}

template <int D, typename R>
__global__ void __launch_bounds__(256) k_grid(StepArgsT<R> A) {
  grid_body<D, R>(A, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// particle I/O helpers (the deformation update and return mapping are FP64)
// ---------------------------------------------------------------------------
template <int D>
struct PLoad {
  double x[3], v[3], F[D][D];
  PScalars s;
  uint32_t id;
};

template <int D, typename R>
__device__ __forceinline__ void load_particle(const PBufT<R>& b, uint32_t Np, uint32_t j, PLoad<D>& p) {
#pragma unroll
  for (int a = 0; a < 3; ++a) p.x[a] = p.v[a] = 0.0;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    p.x[a] = b.x[(size_t)a * Np + j];
    p.v[a] = b.v[(size_t)a * Np + j];
  }
#pragma unroll
  for (int r = 0; r < D; ++r)
#pragma unroll
    for (int c = 0; c < D; ++c) {
      if constexpr (kFP64<R>)
        p.F[r][c] = b.F[(size_t)(r * D + c) * Np + j];
      else
        p.F[r][c] = (double)b.F[(size_t)(r * D + c) * Np + j] + (r == c ? 1.0 : 0.0);
    }
  p.s.eps_pl_dev = b.sc[(size_t)MTR_SCALAR_EPS_PL_DEV * Np + j];
  p.s.eps_pl_vol = b.sc[(size_t)MTR_SCALAR_EPS_PL_VOL * Np + j];
  p.s.eps_pl_vol_pradhana = b.sc[(size_t)MTR_SCALAR_EPS_PL_VOL_PRADHANA * Np + j];
  p.s.delta_gamma = 0.0;  // deformation_update.cpp:13 zeroes it every step
  p.s.viscosity = b.sc[(size_t)MTR_SCALAR_VISCOSITY * Np + j];
  p.s.muI = b.sc[(size_t)MTR_SCALAR_MUI * Np + j];
  p.id = b.id[j];
}

template <int D, typename R>
__device__ __forceinline__ void store_defgrad(const PBufT<R>& b, uint32_t Np, uint32_t s, const double (&F)[D][D],
                                              const PScalars& sc, const double* tau) {
#pragma unroll
  for (int r = 0; r < D; ++r)
#pragma unroll
    for (int c = 0; c < D; ++c) {
      if constexpr (kFP64<R>)
        b.F[(size_t)(r * D + c) * Np + s] = F[r][c];
      else
        b.F[(size_t)(r * D + c) * Np + s] = (R)(F[r][c] - (r == c ? 1.0 : 0.0));
    }
  b.sc[(size_t)MTR_SCALAR_EPS_PL_DEV * Np + s] = (R)sc.eps_pl_dev;
  b.sc[(size_t)MTR_SCALAR_EPS_PL_VOL * Np + s] = (R)sc.eps_pl_vol;
  b.sc[(size_t)MTR_SCALAR_EPS_PL_VOL_PRADHANA * Np + s] = (R)sc.eps_pl_vol_pradhana;
  b.sc[(size_t)MTR_SCALAR_DELTA_GAMMA * Np + s] = (R)sc.delta_gamma;
  b.sc[(size_t)MTR_SCALAR_VISCOSITY * Np + s] = (R)sc.viscosity;
  b.sc[(size_t)MTR_SCALAR_MUI * Np + s] = (R)sc.muI;
#pragma unroll
  for (int q = 0; q < Sym<D>::n; ++q) b.tau[(size_t)q * Np + s] = (R)tau[q];
}

// the end of positionUpdate (position_update.cpp:26-41): periodic wrap in x,
// then the hard-coded teleport hook
__device__ __forceinline__ void wrap_and_teleport(const DevParams& P, double (&xn)[3]) {
  if (P.pbc) {
    if (xn[0] > P.L[0])
      xn[0] = xn[0] - P.L[0];
    else if (xn[0] < 0)
      xn[0] = P.L[0] + xn[0];
  }
  if (P.change_particle_positions && xn[0] > 0.8) {
    xn[0] = -0.1;
    xn[1] += 0.27;
  }
}

// velocity blend of position_update.cpp:14-24 / musl.cpp:15-22
__device__ __forceinline__ double blend_v(double fr, double v, double fl, double pic) {
  if (fr < -1) return pic;
  if (fr < 0) return (-fr) * (v + fl) + (1 - (-fr)) * pic;
  return fr * (v + fl) + (1 - fr) * pic;
}

// F_trial = F + dt * gradv * F (deformation_update.cpp:42-44), then the
// return mapping; writes F, scalars and tau into the out buffer at slot s.
template <int D, typename R, int PM>
__device__ __forceinline__ void defgrad_and_store(const StepArgsT<R>& A, uint32_t s, double dt, PLoad<D>& p,
                                                  const R (&gv)[D][D], uint32_t& flags, bool& plastic) {
  double T1[D][D], T2[D][D];
#pragma unroll
  for (int r = 0; r < D; ++r)
#pragma unroll
    for (int c = 0; c < D; ++c) T1[r][c] = dt * (double)gv[r][c];
  mat_mul<D>(T1, p.F, T2);
#pragma unroll
  for (int r = 0; r < D; ++r)
#pragma unroll
    for (int c = 0; c < D; ++c) p.F[r][c] = p.F[r][c] + T2[r][c];
  double tau[Sym<D>::n];
  plastic = return_map<D, PM>(*A.P, dt, p.F, p.s, tau, flags);
  store_defgrad<D, R>(A.out, A.Np, s, p.F, p.s, tau);
}

// ---------------------------------------------------------------------------
// Tile-structured gathers.  A tile block first copies the node values its
// particles' stencils can reach (the PN^D patch of the tile) from the node
// arrays into shared memory, then every particle gathers from there.
// ---------------------------------------------------------------------------

// Reference velocity of a tile: the FP64 node velocity at the patch node
// nearest the tile centre (zero outside the grid, and always zero on the FP64
// path, which gathers the node velocities themselves).
// NORM: src is the MUSL accumulator, divided by m_i / m_p (nmass, mp).
template <int D, typename R, bool NORM = false>
__device__ __forceinline__ void tile_vref(const StepCommon& A, const StepHeader* H, const int (&n0)[3],
                                          const double* src, double (&vref)[3], const R* nmass = nullptr,
                                          double mp = 0.0) {
  vref[0] = vref[1] = vref[2] = 0.0;
  if constexpr (!kFP64<R>) {
    constexpr int c = 1 + Tiling<D>::TB / 2;
    const int gi = n0[0] + c, gj = n0[1] + c, gk = D == 3 ? n0[2] + c : 0;
    if (gi < (int)H->N[0] && gj < (int)H->N[1] && gk < (int)H->N[2]) {
      const uint32_t l = node_index(H, gi, gj, gk);
      double f = 1.0;
      if constexpr (NORM) f = nmass[l] > R(0.0) ? mp / (double)nmass[l] : 0.0;
#pragma unroll
      for (int a = 0; a < D; ++a) vref[a] = src[(size_t)a * A.cap_nodes + l] * f;
    }
  }
}

// Node patch of the gathers, interleaved: values per node are the D velocity
// components (deviations from vref, rounded to R) and, with FLIP, the D flip
// components, padded so that a node is read with vector loads.
template <int D, bool FLIP, typename R>
struct NodePatch {
  static constexpr int STRIDE = D == 2 ? (FLIP ? 4 : 2) : (FLIP ? (sizeof(R) == 8 ? 6 : 8) : 4);
  static constexpr int SIZE = STRIDE * Tiling<D>::NODES;
};

template <typename R>
struct Vec2;
template <>
struct Vec2<double> {
  using T = double2;
};
template <>
struct Vec2<float> {
  using T = float2;
};

// v (and with WF flip) of one patch node
template <int D, bool WF, typename R>
__device__ __forceinline__ void load_node(const R* __restrict__ p, R (&v)[3], R (&f)[3]) {
  if constexpr (D == 2) {
    if constexpr (sizeof(R) == 4 && WF) {
      const float4 q = *reinterpret_cast<const float4*>(p);
      v[0] = q.x;
      v[1] = q.y;
      f[0] = q.z;
      f[1] = q.w;
    } else {
      const auto q = *reinterpret_cast<const typename Vec2<R>::T*>(p);
      v[0] = q.x;
      v[1] = q.y;
      if constexpr (WF) {
        const auto g = *reinterpret_cast<const typename Vec2<R>::T*>(p + 2);
        f[0] = g.x;
        f[1] = g.y;
      }
    }
  } else if constexpr (sizeof(R) == 8) {
    const double2 q = *reinterpret_cast<const double2*>(p);
    v[0] = q.x;
    v[1] = q.y;
    if constexpr (WF) {
      const double2 g = *reinterpret_cast<const double2*>(p + 2), h = *reinterpret_cast<const double2*>(p + 4);
      v[2] = g.x;
      f[0] = g.y;
      f[1] = h.x;
      f[2] = h.y;
    } else {
      v[2] = p[2];
    }
  } else {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    if constexpr (WF) {
      const float2 g = *reinterpret_cast<const float2*>(p + 4);
      f[0] = q.w;
      f[1] = g.x;
      f[2] = g.y;
    }
  }
}

// fills a node patch from the node velocities src (minus vref) and, with
// FLIP and want_flip, the node flips
template <int D, bool FLIP, typename R, bool NORM = false>
__device__ __forceinline__ void load_patch(const StepCommon& A, const StepHeader* H, const int (&n0)[3],
                                           const double* src, const double (&vref)[3], const R* flip, bool want_flip,
                                           R* dst, const R* nmass = nullptr, double mp = 0.0) {
  const uint32_t cap = A.cap_nodes;
  for (int n = threadIdx.x; n < Tiling<D>::NODES; n += blockDim.x) {
    uint32_t l = 0;
    const bool in = patch_node<D>(H, n0, n, l);
    R* q = dst + n * NodePatch<D, FLIP, R>::STRIDE;
    double v[D], f = 1.0;
#pragma unroll
    for (int a = 0; a < D; ++a) v[a] = in ? src[(size_t)a * cap + l] : 0.0;
    if constexpr (NORM) {
      const double mi = in ? (double)nmass[l] : 0.0;
      f = mi > 0 ? mp / mi : 0.0;
    }
#pragma unroll
    for (int a = 0; a < D; ++a) {
      if constexpr (NORM) v[a] *= f;
      if constexpr (kFP64<R>)
        q[a] = v[a];
      else
        q[a] = in ? (R)(v[a] - vref[a]) : R(0.0);
    }
    if constexpr (FLIP) {
#pragma unroll
      for (int a = 0; a < D; ++a) q[D + a] = in && want_flip ? flip[(size_t)a * cap + l] : R(0.0);
    }
  }
}

// G2P gather (g2p.cpp:24-77) and velocity gradient (deformation_update.cpp:17-40)
// from a shared node patch; lb = stencil base relative to the patch origin.
// The position in the cell is formed in FP64 from the FP64 position, then
// rounded to R.  The patch holds node velocities minus vref: B-spline weights
// sum to one and reproduce linears, so pic = vref + sum w dv, while B and
// grad v need the deviations only.
//
// The sums are factorised over the tensor-product stencil: per node of a row
// along the innermost axis only sum w_z v, sum w_z dz v, sum w_z' v and sum
// w_z flip are formed, and a row's sums are then added with its x and y
// factors.  USL in 3D takes 12 multiply-adds per node and 24 per row of 4
// instead of 32 per node, MUSL 9 and 15 instead of 20, the deformation update
// 6 and 9 instead of 12.  The rows are a loop whose x and y factors wait in
// shared memory (xf, `STRIDE` threads apart): what is live is the sums, the 4
// factors along the innermost axis and ROWS rows.  MUSL and the deformation
// update unroll all 4 rows of an x plane (1M collapse, FP64 0.375 -> 0.363 and
// 0.151 -> 0.147 ms against one row at a time, mixed 0.239 -> 0.230); USL, which
// also holds the particle for its return mapping, takes one (1.2M Cam-Clay
// incline, FP64 0.524 -> 0.488).
template <int D, int DEG, bool FLIP, bool WP, bool WB, bool WF, bool GV, int STRIDE, int ROWS, typename R>
__device__ __forceinline__ void gather_sums(const R* pv, const double (*crd)[Tiling<D>::PN], const int (&lb)[3],
                                            const double (&xp)[3], double ioh, double dx, R* xf, R (&ps)[3],
                                            R (&Bp)[D][D], R (&flp)[3], R (&gv)[D][D]) {
  constexpr int PN = Tiling<D>::PN, STR = NodePatch<D, FLIP, R>::STRIDE;
  constexpr int Z = D - 1;                  // innermost axis
  constexpr int NF = (1 + WB + GV) * 4;     // factors of an axis: w, w times offset, derivative
  constexpr int OP = 4, OD = WB ? 8 : 4;    // where the last two start
  R wz[4], dz[4], pz[4];
#pragma unroll
  for (int a = 0; a < D; ++a) {
    const double td = (xp[a] - crd[a][lb[a] + 1]) * ioh;
    axis_weights<DEG, GV, R>(td, wz, dz);
    if constexpr (WB) {
      axis_offsets<R>(td, dx, pz);
#pragma unroll
      for (int o = 0; o < 4; ++o) pz[o] *= wz[o];
    }
    if (a == Z) break;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      xf[(a * NF + o) * STRIDE] = wz[o];
      if constexpr (WB) xf[(a * NF + OP + o) * STRIDE] = pz[o];
      if constexpr (GV) xf[(a * NF + OD + o) * STRIDE] = dz[o];
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) ps[a] = flp[a] = R(0.0);
#pragma unroll
  for (int r = 0; r < D; ++r)
#pragma unroll
    for (int c = 0; c < D; ++c) Bp[r][c] = gv[r][c] = R(0.0);
  const R* plane = pv + (D == 3 ? (lb[0] * PN + lb[1]) * PN + lb[2] : lb[0] * PN + lb[1]) * STR;
#pragma unroll 1
  for (int ii = 0; ii < 4; ++ii, plane += (D == 3 ? PN * PN : PN) * STR) {
    const R* xi = xf + ii * STRIDE;
    const R* row = plane;
#pragma unroll ROWS
    for (int j = 0; j < (D == 3 ? 4 : 1); ++j, row += PN * STR) {
      R s0[3], s1[3], s2[3], f0[3];
#pragma unroll
      for (int a = 0; a < D; ++a) s0[a] = s1[a] = s2[a] = f0[a] = R(0.0);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        R v[3], f[3];
        load_node<D, WF, R>(row + k * STR, v, f);
#pragma unroll
        for (int a = 0; a < D; ++a) {
          s0[a] += wz[k] * v[a];
          if constexpr (WB) s1[a] += pz[k] * v[a];
          if constexpr (GV) s2[a] += dz[k] * v[a];
          if constexpr (WF) f0[a] += wz[k] * f[a];
        }
      }
      const R wx = xi[0];
      R w = wx, px, py, gx, gy;  // the row's factors of v, B and grad v
      if constexpr (WB) px = xi[OP * STRIDE];
      if constexpr (GV) gx = xi[OD * STRIDE];
      if constexpr (D == 3) {
        const R* yj = xf + (NF + j) * STRIDE;
        const R wy = yj[0];
        w = wx * wy;
        if constexpr (WB) {
          px *= wy;
          py = wx * yj[OP * STRIDE];
        }
        if constexpr (GV) {
          gx *= wy;
          gy = wx * yj[OD * STRIDE];
        }
      }
#pragma unroll
      for (int a = 0; a < D; ++a) {
        if constexpr (WP) ps[a] += w * s0[a];
        if constexpr (WB) {
          Bp[a][0] += px * s0[a];
          if constexpr (D == 3) Bp[a][1] += py * s0[a];
          Bp[a][Z] += w * s1[a];
        }
        if constexpr (GV) {
          gv[a][0] += gx * s0[a];
          if constexpr (D == 3) gv[a][1] += gy * s0[a];
          gv[a][Z] += w * s2[a];
        }
        if constexpr (WF) flp[a] += w * f0[a];
      }
    }
  }
}

// The sums a transfer scheme needs (B for APIC and AFLIP, flip for all but
// APIC), pic = vref + ps (the FP64 path gathers the velocities themselves) and
// grad v scaled by 1/dx.
template <int D, int DEG, bool GV, int STRIDE, int ROWS, typename R>
__device__ __forceinline__ void gather_patch(const R* pv, const double (*crd)[Tiling<D>::PN], const int (&lb)[3],
                                             const double (&xp)[3], double ioh, double dx, R* xf,
                                             const double (&vref)[3],
                                             double (&pic)[3], R (&Bp)[D][D], R (&flp)[3], R (&gv)[D][D], bool want_b,
                                             bool want_flip) {
  R ps[3];
  if (!want_flip)
    gather_sums<D, DEG, true, true, true, false, GV, STRIDE, ROWS, R>(pv, crd, lb, xp, ioh, dx, xf, ps, Bp, flp, gv);
  else if (want_b)
    gather_sums<D, DEG, true, true, true, true, GV, STRIDE, ROWS, R>(pv, crd, lb, xp, ioh, dx, xf, ps, Bp, flp, gv);
  else
    gather_sums<D, DEG, true, true, false, true, GV, STRIDE, ROWS, R>(pv, crd, lb, xp, ioh, dx, xf, ps, Bp, flp, gv);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if constexpr (kFP64<R>)
      pic[a] = ps[a];
    else
      pic[a] = vref[a] + (double)ps[a];
  }
  if (GV) {
    const R iohR = (R)ioh;
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
      for (int c = 0; c < D; ++c) gv[r][c] *= iohR;
  }
}

// grad v alone (MUSL deformation update), from a patch without flips
template <int D, int DEG, int STRIDE, int ROWS, typename R>
__device__ __forceinline__ void gather_gradv(const R* pv, const double (*crd)[Tiling<D>::PN], const int (&lb)[3],
                                             const double (&xp)[3], double ioh, double dx, R* xf, R (&gv)[D][D]) {
  R ps[3], Bp[D][D], flp[3];
  gather_sums<D, DEG, false, false, false, false, true, STRIDE, ROWS, R>(pv, crd, lb, xp, ioh, dx, xf, ps, Bp, flp, gv);
  const R iohR = (R)ioh;
#pragma unroll
  for (int r = 0; r < D; ++r)
#pragma unroll
    for (int c = 0; c < D; ++c) gv[r][c] *= iohR;
}

// ---------------------------------------------------------------------------
// 7a. USL: G2P + deformation update + return mapping + position update, one
// block per tile, node patch in shared memory.
// ---------------------------------------------------------------------------
template <int D, int DEG, typename R, int PM>
__device__ __forceinline__ void g2p_t_body(const StepArgsT<R>& A, const uint32_t* __restrict__ perm, const uint32_t bid,
                                                const uint32_t part, const uint32_t launched) {
  using TL = Tiling<D>;
  constexpr int PN = TL::PN;
  StepHeader* H = A.H;
  if (step_inactive(H)) return;
  const uint32_t t = bid;
  if (t >= H->ntiles) return;
  uint32_t pb, pe;
  tile_range(A, t, pb, pe);
  const uint32_t parts = tile_blocks<D>(pe - pb, launched);
  if (part >= parts) return;
  part_range(part, parts, pb, pe);
  if (pb >= pe) return;
  const DevParams& P = *A.P;
  __shared__ __align__(16) R pv[NodePatch<D, true, R>::SIZE];
  __shared__ R xfac[12 * (D - 1) * kChunk];  // x and y factors of each thread's gather
  __shared__ double crd[3][PN];
  int n0[3];
  load_tile_setup<D>(A, H, t, n0, crd);
  double vref[3];
  tile_vref<D, R>(A, H, n0, A.nv, vref);
  const double fr = P.flip_ratio;
  load_patch<D, true, R>(A, H, n0, A.nv, vref, A.nflip, fr >= -1, pv);
  __syncthreads();
  const uint32_t Np = A.Np;
  const double dt = H->dt, ioh = P.one_over_dx;
  unsigned nplastic = 0;
  for (uint32_t s = pb + threadIdx.x; s < pe; s += blockDim.x) {
    const uint32_t j = perm[s];
    PLoad<D> p;
    load_particle<D, R>(A.in, Np, j, p);
    double pic[3];
    R flp[3], Bp[D][D], gv[D][D];
    int lb[3];
    if (local_base<D>(H, p.x, ioh, n0, false, lb)) {
      gather_patch<D, DEG, true, kChunk, 1, R>(pv, crd, lb, p.x, ioh, P.dx, xfac + threadIdx.x, vref, pic, Bp, flp, gv, fr < 0, fr >= -1);
    } else {
      raise_status(H, MTR_STATUS_STENCIL_OOB, p.id);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        pic[a] = 0.0;
        flp[a] = R(0.0);
      }
#pragma unroll
      for (int r = 0; r < D; ++r)
#pragma unroll
        for (int c = 0; c < D; ++c) Bp[r][c] = gv[r][c] = R(0.0);
    }
    uint32_t f = 0;
    bool plastic = false;
    defgrad_and_store<D, R, PM>(A, s, dt, p, gv, f, plastic);
    if (f) raise_status(H, f, p.id);
    nplastic += plastic ? 1u : 0u;
    double xn[3], vn[3];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      xn[a] = p.x[a] + dt * pic[a];
      vn[a] = blend_v(fr, p.v[a], (double)flp[a], pic[a]);
    }
    wrap_and_teleport(P, xn);
#pragma unroll
    for (int a = 0; a < D; ++a) {
      A.out.x[(size_t)a * Np + s] = xn[a];
      A.out.v[(size_t)a * Np + s] = (R)vn[a];
    }
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
      for (int c = 0; c < D; ++c) A.out.B[(size_t)(r * D + c) * Np + s] = (fr < 0) ? Bp[r][c] : R(0.0);
    A.out.id[s] = p.id;
    if (P.store_pic_flip) {
#pragma unroll
      for (int a = 0; a < D; ++a) {
        A.pic[(size_t)a * Np + s] = (R)pic[a];
        A.flip[(size_t)a * Np + s] = (fr >= -1) ? flp[a] : R(0.0);
      }
    }
  }
  block_count(nplastic, &H->plastic_count);
}

template <int D, int DEG, typename R, int PM = -1>
__global__ void __launch_bounds__(kChunk, (g2p_min_blocks<R, PM>())) k_g2p_t(StepArgsT<R> A, const uint32_t* __restrict__ perm) {
  g2p_t_body<D, DEG, R, PM>(A, perm, blockIdx.x, blockIdx.y, gridDim.y);
}

// ---------------------------------------------------------------------------
// 7b. MUSL (musl.cpp:6-96), one block per tile (or part of one), each warp on
// its own run of cells as in P2G, 32 particles at a time.  Phase 1 (a lane per
// particle): gather pic/B/flip from the shared node patch, blend v, write
// x + dt pic, v, B.  Phase 2: the particles are staged in kMuslParts parts (half
// of the shared memory, so more blocks per SM) and v_p + B D^-1 (x_i - x_p) is
// summed in P2G's windows by two groups of lanes (2D: four, a lane for each
// component), whose sums meet by half_sum: half the exchanges, and half the
// shared adds (compare-and-swap loops in FP64) of every group for itself.
// Measured, ms per launch at 1,024,000 particles, cubic: FP64 0.393 -> 0.336,
// mixed 0.258 -> 0.217; 100,000 in 2D FP64 0.033 -> 0.027.  Each group on its
// own 16 particles took 0.362, 0.230 and 0.037; plain sums over both groups in
// every lane 0.376 and 0.242; two particles a turn (unrolled) 0.345 and 0.223.
// ---------------------------------------------------------------------------
constexpr int kMuslParts = 2;

template <int D, typename R>
struct MStageData {
  R w[D][4], a[D][4];  // weights and weights times offsets
  R q[D][4];           // V, X, Y, Z (2D: V, X, Z) of each component
};
template <int D, typename R>
struct __align__(16) MStage : MStageData<D, R> {
  char pad[stage_stride(sizeof(MStageData<D, R>)) - sizeof(MStageData<D, R>)];
};

template <int D, typename R>
constexpr size_t musl_crd_bytes() {
  return align16(sizeof(double) * 3 * Tiling<D>::PN);
}
template <int D, typename R>
constexpr size_t musl_patch_bytes() {
  return align16(sizeof(R) * NodePatch<D, true, R>::SIZE) + align16(sizeof(R) * D * Tiling<D>::NODES);
}
// a warp stages 32 / kMuslParts particles at a time
template <int D, typename R>
__host__ __device__ constexpr size_t musl_stage_bytes() {
  return 32 / kMuslParts * sizeof(MStage<D, R>);
}
template <int D, typename R>
constexpr size_t musl_smem_bytes(int threads) {
  return musl_crd_bytes<D, R>() + musl_patch_bytes<D, R>() +
         musl_stage_bytes<D, R>() * (size_t)(threads / 32);
}

template <int D, int DEG, typename R>
__device__ __forceinline__ void g2p_musl_w_body(const StepArgsT<R>& A, const uint32_t* __restrict__ perm, const uint32_t bid,
                                                const uint32_t part, const uint32_t launched) {
  using TL = Tiling<D>;
  constexpr int PN = TL::PN, NODES = TL::NODES, TB = TL::TB, Z = D - 1;
  // a lane sums NC components of one stencil column; GR groups of LPP lanes
  constexpr int NC = D == 3 ? 3 : 1, COLS = D == 3 ? 16 : 4, LPP = COLS * D / NC, GR = 32 / LPP, CH = 32 / kMuslParts;
  StepHeader* H = A.H;
  const uint32_t t = bid;
  uint32_t lo, hi;
  even_run(A.cell_start + t * 64u, launched * (blockDim.x >> 5), lo, hi);
  if (step_inactive(H)) return;
  if (t >= H->ntiles) return;
  const int warp = threadIdx.x >> 5;
  uint32_t k0, wend;  // this warp's particles
  if (!warp_run<D, 32, kFP64<R>>(A.cell_start + t * 64u, part, launched, lo, hi, k0, wend)) return;
  const DevParams& P = *A.P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double(*crd)[PN] = reinterpret_cast<double(*)[PN]>(smem_raw);
  R* pv = reinterpret_cast<R*>(smem_raw + musl_crd_bytes<D, R>());  // node v, flip
  R(*vsum)[NODES] = reinterpret_cast<R(*)[NODES]>(
      smem_raw + musl_crd_bytes<D, R>() + align16(sizeof(R) * NodePatch<D, true, R>::SIZE));  // [D][NODES]
  int n0[3];
  load_tile_setup<D>(A, H, t, n0, crd);
  double vref[3];
  tile_vref<D, R>(A, H, n0, A.nv, vref);
  const double fr = P.flip_ratio;
  load_patch<D, true, R>(A, H, n0, A.nv, vref, A.nflip, fr >= -1, pv);
  for (int i = threadIdx.x; i < D * NODES; i += blockDim.x) (&vsum[0][0])[i] = R(0.0);
  __shared__ uint32_t cstart[65];  // first particle of each cell of the tile
  for (int i = threadIdx.x; i < 65; i += blockDim.x) cstart[i] = A.cell_start[t * 64u + i];
  __syncthreads();
  const uint32_t Np = A.Np;
  const double dt = H->dt, ioh = P.one_over_dx;
  const double dx = P.dx;
  const R apicD = (R)P.apicDinverse;
  const bool apic = fr < 0;
  const int lane = threadIdx.x & 31;
  const int grp = lane / LPP, col = lane % COLS, c0 = NC == 1 ? lane % LPP / COLS : 0;
  const int ix = D == 3 ? col >> 2 : col, iy = D == 3 ? col & 3 : 0;  // this lane's column
  MStage<D, R>* st = reinterpret_cast<MStage<D, R>*>(smem_raw + musl_crd_bytes<D, R>() + musl_patch_bytes<D, R>() +
                                                     (size_t)warp * musl_stage_bytes<D, R>());
  // the gather's x and y factors use the warp's stage, which phase 1 does not
  R* xfac = reinterpret_cast<R*>(st) + lane;
  static_assert(8 * (D - 1) * 32 * sizeof(R) <= musl_stage_bytes<D, R>(), "x and y factors must fit the warp's stage");
  int cell = k0 < wend ? cell_of(cstart, k0) : 0;
  for (; k0 < wend; k0 += 32) {
    // phase 1
    __syncwarp();  // the stage has been read
    const uint32_t s = k0 + lane;
    bool ok = false;
    R vs[D], Bs[D][D];
    double td[3] = {0.0, 0.0, 0.0};
    if (s < wend) {
      const uint32_t j = perm[s];
      double xp[3] = {0, 0, 0};
#pragma unroll
      for (int a = 0; a < D; ++a) xp[a] = A.in.x[(size_t)a * Np + j];
      double pic[3];
      R flp[3], Bp[D][D], gv[D][D];
      int lb[3];
      ok = local_base<D>(H, xp, ioh, n0, false, lb);
      if (ok) {
        gather_patch<D, DEG, false, 32, 4, R>(pv, crd, lb, xp, ioh, dx, xfac, vref, pic, Bp, flp, gv, apic, fr >= -1);
#pragma unroll
        for (int a = 0; a < D; ++a) td[a] = (xp[a] - crd[a][lb[a] + 1]) * ioh;
      } else {
        raise_status(H, MTR_STATUS_STENCIL_OOB, A.in.id[j]);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          pic[a] = 0.0;
          flp[a] = R(0.0);
        }
#pragma unroll
        for (int r = 0; r < D; ++r)
#pragma unroll
          for (int c = 0; c < D; ++c) Bp[r][c] = R(0.0);
      }
      double xn[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int a = 0; a < D; ++a) {
        const double vn = blend_v(fr, (double)A.in.v[(size_t)a * Np + j], (double)flp[a], pic[a]);
        vs[a] = (R)vn;
        xn[a] = xp[a] + dt * pic[a];  // positionUpdate: x + dt pic
        A.out.v[(size_t)a * Np + s] = (R)vn;
      }
      wrap_and_teleport(P, xn);
#pragma unroll
      for (int a = 0; a < D; ++a) A.out.x[(size_t)a * Np + s] = xn[a];
#pragma unroll
      for (int r = 0; r < D; ++r)
#pragma unroll
        for (int c = 0; c < D; ++c) {
          const R b = apic ? Bp[r][c] : R(0.0);
          A.out.B[(size_t)(r * D + c) * Np + s] = b;
          Bs[r][c] = apicD * b;
        }
      A.out.id[s] = A.in.id[j];
      if (P.store_pic_flip) {
#pragma unroll
        for (int a = 0; a < D; ++a) {
          A.pic[(size_t)a * Np + s] = (R)pic[a];
          A.flip[(size_t)a * Np + s] = (fr >= -1) ? flp[a] : R(0.0);
        }
      }
    }
    // phase 2; the window starts and ends with the chunk, so that its registers
    // are free during the gather.  The re-scatter's base, clamped at zero like
    // P2G's (musl.cpp:35-40), is the gather's, which takes no particle left of
    // the first node, and so the cell's.
    Window<R, NC, LPP> win;
    auto dst = [&](int c) { return vsum[c0 + c]; };
    while (cstart[cell + 1] <= k0) ++cell;
    int node0 = window_node<D>(n0, cell, ix, iy);  // node of the window's first entry
#pragma unroll 1
    for (int part = 0; part < kMuslParts; ++part) {
      const uint32_t p0 = k0 + part * CH, pend = min(p0 + CH, wend);
      if (p0 >= wend) break;
      __syncwarp();  // the last part has been read
      bool tiny = false;
      if (lane / CH == part) {
        MStage<D, R>& S = st[lane % CH];
        int least = 0;
#pragma unroll
        for (int a = 0; a < D; ++a) {
          R w[4], d[4], o[4];
          axis_weights<DEG, false, R>(td[a], w, d);
          axis_offsets<R>(td[a], dx, o);
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            S.w[a][h] = ok ? w[h] : R(0.0);
            S.a[a][h] = ok ? w[h] * o[h] : R(0.0);
          }
          least += least_exponent<DEG, false>(w);
        }
#pragma unroll
        for (int r = 0; r < D; ++r) {
          S.q[r][0] = ok ? vs[r] : R(0.0);
#pragma unroll
          for (int c = 0; c < D; ++c) S.q[r][1 + c] = ok ? Bs[r][c] : R(0.0);
        }
        tiny = least < -82;
      }
      const bool slow = __any_sync(0xffffffffu, tiny);
      __syncwarp();
      auto add = [&](const MStage<D, R>& S, auto small) {
        R f1[4], f2[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          f1[h] = S.w[Z][h];
          f2[h] = S.a[Z][h];
        }
        R u0 = S.w[0][ix], u1 = S.a[0][ix];
        [[maybe_unused]] R u2 = R(0.0);
        if constexpr (D == 3) {
          const R wy = S.w[1][iy], ay = S.a[1][iy];
          u2 = u0 * ay;
          u0 *= wy;
          u1 *= wy;
        }
        if constexpr (decltype(small)::value) {  // musl.cpp:51 skips weights <= 1e-25
#pragma unroll
          for (int h = 0; h < 4; ++h)
            if (!(f1[h] * u0 > R(1e-25))) f1[h] = f2[h] = R(0.0);
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          R a1 = u0 * S.q[c0 + c][0] + u1 * S.q[c0 + c][1];
          if constexpr (D == 3) a1 += u2 * S.q[c0 + c][2];
          const R b1 = u0 * S.q[c0 + c][D];
#pragma unroll
          for (int h = 0; h < 4; ++h) win.acc[h][c] = f2[h] * b1 + (f1[h] * a1 + win.acc[h][c]);
        }
      };
      for (uint32_t k = p0;;) {
        const uint32_t e = min(cstart[cell + 1], pend);  // the cell's end within the part
        if (slow) {
#pragma unroll 1
          for (k += grp; k < e; k += GR) add(st[k - p0], std::true_type{});
        } else {
#pragma unroll 1
          for (k += grp; k < e; k += GR) add(st[k - p0], std::false_type{});
        }
        __syncwarp();
        k = e;
        if (k == pend) break;
        // the next cell that is not empty; the window moves there, or starts anew
        int next = cell + 1;
        while (cstart[next + 1] <= k) ++next;
        const int steps = window_steps<D>(n0, cell, next);
        cell = next;
        if (steps == 4) {
          win.flush(grp, node0, dst);
          node0 = window_node<D>(n0, cell, ix, iy);
        } else {
          for (int h = 0; h < steps; ++h) win.advance(grp, node0, dst);
        }
      }
    }
    win.flush(grp, node0, dst);
  }
  __syncthreads();
  const uint32_t cap = A.cap_nodes;
  for (int n = threadIdx.x; n < NODES; n += blockDim.x) {
    uint32_t l;
    if (!patch_node<D>(H, n0, n, l)) continue;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const R val = vsum[a][n];
      if (val != R(0.0)) atomicAdd(&A.v2[(size_t)a * cap + l], (double)val);
    }
  }
}

template <int D, int DEG, typename R>
__global__ void __launch_bounds__(MTR_MUSL_BOUNDS)
    k_g2p_musl_w(StepArgsT<R> A, const uint32_t* __restrict__ perm) {
  g2p_musl_w_body<D, DEG, R>(A, perm, blockIdx.x, blockIdx.y, gridDim.y);
}

// MUSL: deformation update from the re-projected velocity v2 and the old
// positions (deformation_update.cpp:6), then the return mapping.  v2 is divided
// by m_i / m_p (zero where m_i == 0, musl.cpp:80-95) as the patch is loaded: 1
// division a patch node, where a kernel of its own over the grid took 6 us at
// 172,000 nodes and a launch.
template <int D, int DEG, typename R, int PM>
__device__ __forceinline__ void defgrad_t_body(const StepArgsT<R>& A, const uint32_t* __restrict__ perm, const uint32_t bid,
                                                const uint32_t part, const uint32_t launched) {
  using TL = Tiling<D>;
  constexpr int PN = TL::PN;
  StepHeader* H = A.H;
  if (step_inactive(H)) return;
  const uint32_t t = bid;
  if (t >= H->ntiles) return;
  uint32_t pb, pe;
  tile_range(A, t, pb, pe);
  const uint32_t parts = tile_blocks<D>(pe - pb, launched);
  if (part >= parts) return;
  part_range(part, parts, pb, pe);
  if (pb >= pe) return;
  __shared__ __align__(16) R pv[NodePatch<D, false, R>::SIZE];
  __shared__ R xfac[8 * (D - 1) * kMaxTileThreads];  // x and y factors of each thread's gather
  __shared__ double crd[3][PN];
  int n0[3];
  load_tile_setup<D>(A, H, t, n0, crd);
  double vref[3];
  const double mp = A.P->particle_mass;
  tile_vref<D, R, true>(A, H, n0, A.v2, vref, A.nmass, mp);
  load_patch<D, false, R, true>(A, H, n0, A.v2, vref, (const R*)nullptr, false, pv, A.nmass, mp);
  __syncthreads();
  const uint32_t Np = A.Np;
  const double dt = H->dt, ioh = A.P->one_over_dx;
  unsigned nplastic = 0;
  for (uint32_t s = pb + threadIdx.x; s < pe; s += blockDim.x) {
    const uint32_t j = perm[s];
    PLoad<D> p;
    load_particle<D, R>(A.in, Np, j, p);
    R gv[D][D];
    int lb[3];
    if (local_base<D>(H, p.x, ioh, n0, false, lb)) {
      gather_gradv<D, DEG, kMaxTileThreads, 4, R>(pv, crd, lb, p.x, ioh, A.P->dx, xfac + threadIdx.x, gv);
    } else {
      raise_status(H, MTR_STATUS_STENCIL_OOB, p.id);
#pragma unroll
      for (int r = 0; r < D; ++r)
#pragma unroll
        for (int c = 0; c < D; ++c) gv[r][c] = R(0.0);
    }
    uint32_t f = 0;
    bool plastic = false;
    defgrad_and_store<D, R, PM>(A, s, dt, p, gv, f, plastic);
    if (f) raise_status(H, f, p.id);
    nplastic += plastic ? 1u : 0u;
  }
  block_count(nplastic, &H->plastic_count);
}

template <int D, int DEG, typename R, int PM = -1>
__global__ void __launch_bounds__(MTR_DEFGRAD_BOUNDS) k_defgrad_t(StepArgsT<R> A, const uint32_t* __restrict__ perm) {
  defgrad_t_body<D, DEG, R, PM>(A, perm, blockIdx.x, blockIdx.y, gridDim.y);
}

// ---------------------------------------------------------------------------
// 8. end of step: moveObjects and the clock of simulate()
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void tail_body(const StepCommon& A, int out_parity) {
  StepHeader* H = A.H;
  if (step_inactive(H)) return;
  const DevParams& P = *A.P;
  if (threadIdx.x != 0) return;
  const double dt = H->dt;
  for (int i = 0; i < P.nplates; ++i) {  // ObjectPlate::move, object_plate.hpp:136-162
    mtr_plate& o = H->plates[i];
    double factor = (H->time < o.load_factor * P.frame_dt) ? (1.0 / o.vmin_factor) : 1.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) o.v_object[a] = (a < D) ? o.v_object_original[a] * factor : 0.0;
    if (o.plate_type == MTR_PLATE_LEFT || o.plate_type == MTR_PLATE_RIGHT) {
      o.pos_object += dt * o.v_object[0];
      o.pos_upper += dt * o.v_object[1];
      o.pos_lower += dt * o.v_object[1];
    } else if (o.plate_type == MTR_PLATE_BOTTOM || o.plate_type == MTR_PLATE_TOP) {
      o.pos_object += dt * o.v_object[1];
      o.pos_upper += dt * o.v_object[0];
      o.pos_lower += dt * o.v_object[0];
    } else if (D == 3 && (o.plate_type == MTR_PLATE_BACK || o.plate_type == MTR_PLATE_FRONT)) {
      o.pos_object += dt * o.v_object[2];
    }
  }
  H->cur = out_parity;
  if (H->status & kExitMask) {  // simulation.cpp:176-177: return before time += dt
    H->done = 1;
    return;
  }
  H->time += dt;
  H->step += 1;
  if (__dsub_rn(__dmul_rn(P.frame_dt, (double)(H->frame + 1)), H->time) < 1e-15) H->frame += 1;
  if (fabs(__dsub_rn(P.final_time, H->time)) < 1e-15 || P.final_time < H->time || !(H->frame < P.end_frame)) H->done = 1;
}

template <int D>
__global__ void k_tail(StepCommon A, int out_parity) {
  tail_body<D>(A, out_parity);
}

// ---------------------------------------------------------------------------
// 9. batched steps: the scenes of one group (same dim, spline, precision and
// USL/MUSL) advance together, one launch per phase for all of them.  Each
// launch's blocks are laid out scene after scene; a block finds its scene in
// a per-launch-kind offset table and runs the same body as the single-scene
// kernel on that scene's arguments.  Both particle-buffer parities of every
// scene are in the table and the block picks the one its scene's header
// names, so one captured graph stays valid while scenes advance, stop or
// regrow independently.
// ---------------------------------------------------------------------------
enum BatchKind { kBK_BBOX = 0, kBK_SORT, kBK_SCAN, kBK_TILEK, kBK_NODES, kBK_ONE, kBK_KINDS };

template <typename R>
struct BatchView {
  const StepArgsT<R>* args;  // [2][n]: args[c * n + s] = scene s reading particle buffer c
  const uint32_t* off;       // [kBK_KINDS][n + 1]: first block of each scene, per launch kind
  int n;
};

// arguments of the scene that owns global block g, the block index b within
// the scene and the scene's block count nb; null past the last scene
template <typename R>
__device__ __forceinline__ const StepArgsT<R>* batch_locate_at(const BatchView<R>& B, int kind, uint32_t g,
                                                               uint32_t& b, uint32_t& nb) {
  const uint32_t* o = B.off + (size_t)kind * (B.n + 1);
  if (g >= o[B.n]) return nullptr;
  int lo = 0, hi = B.n - 1;  // last scene whose first block is <= g
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (o[mid] <= g)
      lo = mid;
    else
      hi = mid - 1;
  }
  b = g - o[lo];
  nb = o[lo + 1] - o[lo];
  const int cur = B.args[lo].H->cur;
  return B.args + (size_t)(cur & 1) * B.n + lo;
}

template <typename R>
__device__ __forceinline__ const StepArgsT<R>* batch_locate(const BatchView<R>& B, int kind, uint32_t& b,
                                                            uint32_t& nb) {
  return batch_locate_at(B, kind, blockIdx.x, b, nb);
}

// The tile kernels of a batch run one block per tile block of every scene;
// `body(A, b, nb)` runs this block's tile.
template <typename R, typename Body>
__device__ __forceinline__ void batch_tiles(const BatchView<R>& B, Body&& body) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_TILEK, b, nb);
  if (A) body(*A, b, nb);
}

template <int D, typename R>
__global__ void __launch_bounds__(256) kb_bbox(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_BBOX, b, nb);
  if (A) bbox_body<D, R>(*A, b, nb);
}

template <int D, typename R>
__global__ void __launch_bounds__(256) kb_header(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_ONE, b, nb);
  if (A) header_body<D>(*A);
}

template <int D, typename R>
__global__ void __launch_bounds__(kSortThreads) kb_sort_keys(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_SORT, b, nb);
  if (A) sort_keys_body<D>(*A, b);
}

template <typename R>
__global__ void __launch_bounds__(kSortThreads) kb_sort_scan(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_SCAN, b, nb);
  if (A) sort_scan_body(*A, b);
}

template <typename R>
__global__ void __launch_bounds__(kSortThreads) kb_sort_place(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_SORT, b, nb);
  if (A) sort_place_body(*A, b);
}

template <typename R>
__global__ void __launch_bounds__(kSortThreads) kb_sort_rank(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_SORT, b, nb);
  if (A) sort_rank_body(*A, b, nb);
}

template <int D, int DEG, typename R>
__global__ void __launch_bounds__(MTR_P2G_BOUNDS) kb_p2g_w(BatchView<R> B) {
  batch_tiles(B, [&](const StepArgsT<R>& A, uint32_t b, uint32_t nb) { p2g_w_body<D, DEG, R>(A, A.perm, b, 0u, 1u); });
}

template <int D, typename R>
__global__ void __launch_bounds__(256) kb_grid(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_NODES, b, nb);
  if (A) grid_body<D, R>(*A, b, nb);
}

template <int D, int DEG, typename R, int PM = -1>
__global__ void __launch_bounds__(kChunk, (g2p_min_blocks<R, PM>())) kb_g2p_t(BatchView<R> B) {
  batch_tiles(B, [&](const StepArgsT<R>& A, uint32_t b, uint32_t nb) { g2p_t_body<D, DEG, R, PM>(A, A.perm, b, 0u, 1u); });
}

template <int D, int DEG, typename R>
__global__ void __launch_bounds__(MTR_MUSL_BOUNDS) kb_g2p_musl_w(BatchView<R> B) {
  batch_tiles(B, [&](const StepArgsT<R>& A, uint32_t b, uint32_t nb) {
    g2p_musl_w_body<D, DEG, R>(A, A.perm, b, 0u, 1u);
  });
}

template <int D, int DEG, typename R, int PM = -1>
__global__ void __launch_bounds__(MTR_DEFGRAD_BOUNDS) kb_defgrad_t(BatchView<R> B) {
  batch_tiles(B, [&](const StepArgsT<R>& A, uint32_t b, uint32_t nb) {
    defgrad_t_body<D, DEG, R, PM>(A, A.perm, b, 0u, 1u);
  });
}

template <int D, typename R>
__global__ void __launch_bounds__(32) kb_tail(BatchView<R> B) {
  uint32_t b, nb;
  const StepArgsT<R>* A = batch_locate(B, kBK_ONE, b, nb);
  if (A) tail_body<D>(*A, A->out_parity);
}

// ---------------------------------------------------------------------------
// set-up and download
// ---------------------------------------------------------------------------
template <int D, typename R>
__global__ void k_init_state(StepCommon A, PBufT<R> b) {  // tau of the uploaded F, id = index
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.Np) return;
  PLoad<D> p;
  load_particle<D, R>(b, A.Np, i, p);
  double tau[Sym<D>::n];
  initial_tau<D>(*A.P, p.F, tau);
#pragma unroll
  for (int q = 0; q < Sym<D>::n; ++q) b.tau[(size_t)q * A.Np + i] = (R)tau[q];
  b.id[i] = i;
}

// AoS (host layout, column-major matrices) <-> SoA, in original particle order.
// kind 0: vector (D), 1: matrix (D*D, column-major AoS <-> (r*D+c) SoA),
// 2: scalars (6), 3: matrix stored as M - I (the FP32 deformation gradient).
// A null src stands for every particle's value being zero, or with eye set
// (matrices) the identity: absent inputs are filled here, not copied.
template <int D, typename R>
__global__ void k_aos_to_soa(uint32_t Np, const double* __restrict__ src, R* dst, int kind, bool eye = false) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Np) return;
  if (kind == 0) {
#pragma unroll
    for (int a = 0; a < D; ++a) dst[(size_t)a * Np + i] = src ? (R)src[(size_t)i * D + a] : (R)0;
  } else if (kind == 1 || kind == 3) {
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
      for (int c = 0; c < D; ++c) {
        const double m = src ? src[(size_t)i * D * D + c * D + r] : (eye && r == c ? 1.0 : 0.0);
        dst[(size_t)(r * D + c) * Np + i] = (R)(kind == 3 ? m - (r == c ? 1.0 : 0.0) : m);
      }
  } else {
#pragma unroll
    for (int q = 0; q < MTR_NUM_SCALARS; ++q)
      dst[(size_t)q * Np + i] = src ? (R)src[(size_t)i * MTR_NUM_SCALARS + q] : (R)0;
  }
}

template <int D, typename R>
__global__ void k_soa_to_aos(uint32_t Np, const R* __restrict__ src, const uint32_t* __restrict__ id, double* dst,
                             int kind) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= Np) return;
  const uint32_t i = id[s];
  if (kind == 0) {
#pragma unroll
    for (int a = 0; a < D; ++a) dst[(size_t)i * D + a] = src[(size_t)a * Np + s];
  } else if (kind == 1 || kind == 3) {
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
      for (int c = 0; c < D; ++c) {
        const double m = src[(size_t)(r * D + c) * Np + s];
        dst[(size_t)i * D * D + c * D + r] = kind == 3 ? m + (r == c ? 1.0 : 0.0) : m;
      }
  } else {
#pragma unroll
    for (int q = 0; q < MTR_NUM_SCALARS; ++q) dst[(size_t)i * MTR_NUM_SCALARS + q] = src[(size_t)q * Np + s];
  }
}

// ---------------------------------------------------------------------------
// Frame output (Simulation::saveParticleData, save_data.cpp:7-171): one row of
// FP64 columns per particle, in the original particle order, with the
// columns and their order of the reference's particle file:
//   x[D], v[D], p, q, Je,
//   eps_pl_vol, eps_pl_dev, delta_gamma   (kFrameCols & kFramePlastic)
//   muI                                    (kFrameCols & kFrameMuI)
//   viscosity                              (kFrameCols & kFrameViscosity)
// p = -tr(tau)/D, q = sqrt(c tau_dev : tau_dev) with c = 3/2 (use_mises_q) or
// 1/2, Je = det F (save_data.cpp:14-35).  tau is the particle's carried
// Kirchhoff stress, which the step computes from the final F exactly as
// HenckyPiola(F) F^T / NeoHookeanPiola(F) F^T.  The particle buffer read is
// the current one of the header (H->cur), so the kernel can be enqueued
// behind any number of steps.  The clock of the snapshot goes to clock[0..4]:
// time, dt, step, frame, done.
// ---------------------------------------------------------------------------
enum : unsigned { kFramePlastic = 1u, kFrameMuI = 2u, kFrameViscosity = 4u };

template <int D, typename R>
__global__ void __launch_bounds__(256) k_frame_rows(PBufT<R> b0, PBufT<R> b1, const StepHeader* __restrict__ H,
                                                    const DevParams* __restrict__ P, uint32_t Np, unsigned cols,
                                                    uint32_t ncols, double* __restrict__ rows,
                                                    double* __restrict__ clock) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) {
    clock[0] = H->time;
    clock[1] = H->dt;
    clock[2] = (double)H->step;
    clock[3] = (double)H->frame;
    clock[4] = (double)H->done;
  }
  if (s >= Np) return;
  const PBufT<R>& b = H->cur ? b1 : b0;
  constexpr int NS = Sym<D>::n;
  PLoad<D> p;
  load_particle<D, R>(b, Np, s, p);
  double tau[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) tau[q] = (double)b.tau[(size_t)q * Np + s];
  double tr = 0.0;
#pragma unroll
  for (int a = 0; a < D; ++a) tr += tau[a];
  const double pressure = -tr / D;
  double dd = 0.0;
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const double t = sym_at<D>(tau, i, j) + (i == j ? pressure : 0.0);
      dd += t * t;
    }
  const double q = sqrt((P->use_mises_q ? 1.5 : 0.5) * dd);
  const double(&F)[D][D] = p.F;
  double Je;
  if constexpr (D == 3)
    Je = F[0][0] * (F[1][1] * F[2][2] - F[2][1] * F[1][2]) - F[1][0] * (F[0][1] * F[2][2] - F[2][1] * F[0][2]) +
         F[2][0] * (F[0][1] * F[1][2] - F[1][1] * F[0][2]);
  else
    Je = F[0][0] * F[1][1] - F[1][0] * F[0][1];
  double* row = rows + (size_t)p.id * ncols;
  int c = 0;
#pragma unroll
  for (int a = 0; a < D; ++a) row[c++] = p.x[a];
#pragma unroll
  for (int a = 0; a < D; ++a) row[c++] = p.v[a];
  row[c++] = pressure;
  row[c++] = q;
  row[c++] = Je;
  if (cols & kFramePlastic) {
    row[c++] = p.s.eps_pl_vol;
    row[c++] = p.s.eps_pl_dev;
    row[c++] = (double)b.sc[(size_t)MTR_SCALAR_DELTA_GAMMA * Np + s];
  }
  if (cols & kFrameMuI) row[c++] = p.s.muI;
  if (cols & kFrameViscosity) row[c++] = p.s.viscosity;
}

// Gradient of a dense level set by second-order central differences,
// 0.5 (phi[i+1] - phi[i-1]) / h per axis, neighbours outside the lattice
// reading `background` (OpenVDB's Gradient with CD_2ND, tools/GridOperators.h,
// on a fully active grid).  Three floats per sample; unused axes are zero.
static __global__ void __launch_bounds__(256) k_levelset_grad(const float* __restrict__ phi, float* __restrict__ grad,
                                                       uint32_t n0, uint32_t n1, uint32_t n2, int dim,
                                                       float background, double half_inv_h) {
  const uint64_t total = (uint64_t)n0 * n1 * n2;
  for (uint64_t l = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; l < total; l += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t k = (uint32_t)(l % n2), j = (uint32_t)((l / n2) % n1), i = (uint32_t)(l / ((uint64_t)n1 * n2));
    const uint32_t n[3] = {n0, n1, n2}, c[3] = {i, j, k};
    const uint64_t step[3] = {(uint64_t)n1 * n2, n2, 1};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float g = 0.0f;
      if (a < dim) {
        const float plus = c[a] + 1 < n[a] ? phi[l + step[a]] : background;
        const float minus = c[a] >= 1 ? phi[l - step[a]] : background;
        g = (float)((double)__fsub_rn(plus, minus) * half_inv_h);
      }
      grad[l * 3 + a] = g;
    }
  }
}

// node array of type R -> FP64 (grid read-back of the FP32 path)
template <typename R>
__global__ void k_to_f64(uint64_t n, const R* __restrict__ src, double* dst) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

}  // namespace mtr
