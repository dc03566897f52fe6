// mtr_noalloc.cu — mtr_p2g_noalloc: the particle-to-grid transfer of one
// particle set onto a caller-described grid, without allocating any memory.
//
// Who needs it: callers that cannot call cudaMalloc at the point where they
// transfer particles to a grid.  A host loop being captured into a CUDA graph
// cannot allocate (allocation is not a capturable stream operation); a solver
// embedded in a framework that owns all device memory through its own pool
// (PyTorch's caching allocator, a game or VFX engine) may not allocate behind
// that pool's back; a real-time or fixed-budget caller must not pay for, or
// risk the failure of, an allocation inside its step.  Such callers pass
// device pointers they already own for the inputs and outputs, and this entry
// point keeps every intermediate (the cell-key sort, the tile ranges and the
// grid accumulators) in one file-scope device array of fixed size.
//
// Limits: at most MTR_NOALLOC_MAX_PARTICLES particles and
// MTR_NOALLOC_MAX_NODES grid nodes per call; larger requests are rejected
// with MTR_ERR_TOO_LARGE before anything is launched.  The array costs ~12 MB of device memory on every GPU
// that loads the library, until the process exits.
//
// Sharing: every call on a device uses the same array.  Each call clears
// what must start at zero (accumulators, tile ranges) at its start, so
// back-to-back calls are independent when they are ordered on the device;
// calls that overlap on the GPU (different streams without ordering, or
// several host threads) race on the array and give wrong results.
//
// Set-up: the first call on each device looks up the array's device address
// (cudaGetSymbolAddress) with that device current and raises the shared
// memory limit of the kernel; make that first call outside any stream
// capture.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "../../include/matter_gpu.h"
#include "mtr_kernels.cuh"

using namespace mtr;

namespace {

constexpr int kMaxDevices = 64;
constexpr size_t kMaxP = MTR_NOALLOC_MAX_PARTICLES;
constexpr size_t kMaxNodes = MTR_NOALLOC_MAX_NODES;
// Most tiles of a grid of kMaxNodes nodes with at least 4 per axis: an axis of n
// nodes has ceil(n / 4) tiles in 3D, at most 2/5 n (n = 5), so at most 0.064
// tiles per node; in 2D ceil(n / 8), at most n / 4 (n = 4), so at most 0.0625.
constexpr size_t kMaxTiles = kMaxNodes * 64 / 1000 + 1;
constexpr size_t kMaxSupers = (kMaxTiles * 64 + 1 + kSuperCells - 1) / kSuperCells;
constexpr size_t kMaxCells = kMaxSupers * kSuperCells;

constexpr size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

// scratch layout (byte offsets)
constexpr size_t kOffHeader = 0;
constexpr size_t kOffParams = kOffHeader + align256(sizeof(StepHeader));
constexpr size_t kOffKeys0 = kOffParams + align256(sizeof(DevParams));
constexpr size_t kOffRank = kOffKeys0 + align256(kMaxP * 4);
constexpr size_t kOffTmp = kOffRank + align256(kMaxP * 4);
constexpr size_t kOffBig = kOffTmp + align256(kMaxP * 4);
constexpr size_t kOffStart = kOffBig + align256((kMaxP / kBigCell + 1) * 4);
constexpr size_t kOffCount = kOffStart + align256((kMaxCells + 4) * 4);
constexpr size_t kOffSuper = kOffCount + align256(kMaxCells * 4);
constexpr size_t kOffAcc = kOffSuper + align256(kMaxSupers * 4);
constexpr size_t kScratchBytes = kOffAcc + align256(4 * kMaxNodes * sizeof(double));  // mass + momentum[3]

}  // namespace

// The scratch array.  In host code this name is a host-side stand-in, not a
// device address: host code must use the address returned by
// cudaGetSymbolAddress (scratch_for_current_device below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

namespace {

std::mutex g_setup_mutex;
void* g_scratch_ptr[kMaxDevices] = {};

// Scatter blocks: a call's tiles are few (64 for 4k particles, about 700 at
// capacity), so the chain of particles that each warp works through sets how
// long the launch takes.  While four blocks of a tile each fit the chip at once,
// a tile takes four of 256 threads, else two of 128 (whose shared memory lets
// more of them share an SM).  us per call, tiles as 1, 2, 4 blocks of 256, and 2,
// 4 of 128: 4k particles 49, 41, 38, 47, 41; 261k 94, 96, 111, 90, 94.  The
// scatter that staged a block's particles between barriers took 82 and 109.
constexpr int kScatterThreads = 256;
constexpr uint64_t kFewTiles = 148;

// The step's scatter, mass and momentum only, accumulating into the scratch
// grid.
template <int D, int DEG>
__global__ void __launch_bounds__(kScatterThreads, 2) k_p2g_noalloc(StepArgs A, const uint32_t* __restrict__ perm) {
  p2g_w_body<D, DEG, double, false>(A, perm, blockIdx.x, blockIdx.y, gridDim.y);
}

// Cell keys.  A particle whose cell lies outside the caller's grid (or whose
// position is not finite) gets the sentinel key ntiles * 64, one past every
// real tile: it sorts behind all real particles, no tile names it, and it is
// reported through the status word.  The test is written on the same
// expression cell_key floors, so a particle kept here has a tile index below
// ntiles.
template <int D>
__global__ void __launch_bounds__(kSortThreads) k_noalloc_keys(StepCommon A) {
  const StepHeader* H = A.H;
  const double ioh = A.P->one_over_dx;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < A.Np;
  uint32_t key = H->ntiles * 64u;
  if (valid) {
    double x[3] = {0.0, 0.0, 0.0};
    bool inside = true;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      x[a] = A.xin[(size_t)a * A.Np + i];
      const double u = (x[a] - H->org[a]) * ioh;
      if (!(u >= 0.0 && u < (double)H->N[a])) inside = false;
    }
    if (inside) {
      key = cell_key<D>(H, ioh, x);
    } else {
      atomicOr(&A.H->status, MTR_STATUS_STENCIL_OOB);
      atomicMin(&A.H->first_bad, i);
    }
    A.keys0[i] = key;
  }
  sort_count(A, i, valid, key);
}

template <int D>
constexpr size_t noalloc_smem_bytes(int threads = kScatterThreads) {
  return p2g_smem_bytes<D, double, false>(threads);
}

// Writes the grid description and the few constants the kernels read into
// the scratch header and parameter block (passed by value: no host copy), and
// clears the accumulators and the sort's counts.
__global__ void k_noalloc_setup(StepHeader* H, DevParams* P, const double* gx, const double* gy, const double* gz,
                                uint32_t nx, uint32_t ny, uint32_t nz, uint32_t tx, uint32_t ty, uint32_t tz,
                                double one_over_dx, double apicD, double flip_ratio, double particle_mass, uint32_t Np,
                                int dim, double* acc, uint32_t nacc, uint32_t* count, uint32_t ncount,
                                uint32_t* super, uint32_t nsuper) {
  const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (uint32_t i = i0; i < nacc; i += step) acc[i] = 0.0;
  for (uint32_t i = i0; i < ncount; i += step) count[i] = 0u;
  for (uint32_t i = i0; i < nsuper; i += step) super[i] = 0u;
  if (i0 != 0) return;
  H->done = 0;
  H->abort = 0;
  H->frame = 0;
  H->stop_frame = 0xffffffffu;
  H->step = 0;
  H->stop_step = 0xffffffffu;
  H->status = 0;
  H->first_bad = 0xffffffffu;
  H->org[0] = gx[0];
  H->org[1] = gy[0];
  H->org[2] = dim == 3 ? gz[0] : 0.0;
  H->N[0] = nx;
  H->N[1] = ny;
  H->N[2] = nz;
  H->G = nx * ny * nz;
  H->T[0] = tx;
  H->T[1] = ty;
  H->T[2] = tz;
  H->ntiles = tx * ty * tz;
  H->nbig = 0;
  P->one_over_dx = one_over_dx;
  P->apicDinverse = apicD;
  P->flip_ratio = flip_ratio;
  P->particle_mass = particle_mass;
  P->Np = Np;
  P->use_mibf = 0;
  P->dim = dim;
}

// p2g.cpp:84-98: v = momentum / (sum of weights), mass *= particle mass.
template <int D>
__global__ void k_noalloc_finalize(const double* __restrict__ acc, uint32_t cap, uint32_t G, double particle_mass,
                                   double* grid_mass, double* grid_v, const StepHeader* __restrict__ H,
                                   uint32_t* status) {
  if (status && blockIdx.x == 0 && threadIdx.x == 0) *status = H->status;
  for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < G; l += gridDim.x * blockDim.x) {
    const double m = acc[l];
#pragma unroll
    for (int a = 0; a < D; ++a) grid_v[(size_t)a * G + l] = (m > 0) ? acc[(size_t)(1 + a) * cap + l] / m : 0.0;
    grid_mass[l] = m * particle_mass;
  }
}

template <int D, int DEG>
bool set_attr() {
  return cudaFuncSetAttribute(k_p2g_noalloc<D, DEG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)noalloc_smem_bytes<D>()) == cudaSuccess;
}

// Once per device, with that device current: the device address of the
// scratch array.  Returns nullptr on failure.
unsigned char* scratch_for_current_device(int* rc_out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    *rc_out = MTR_ERR_NO_DEVICE;
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_ptr[dev]) {
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || !ptr) {
      *rc_out = MTR_ERR_CUDA;
      return nullptr;
    }
    if (!(set_attr<2, 2>() && set_attr<2, 3>() && set_attr<3, 2>() && set_attr<3, 3>())) {
      *rc_out = MTR_ERR_CUDA;  // the device stays unset: the next call tries again
      return nullptr;
    }
    g_scratch_ptr[dev] = ptr;
  }
  *rc_out = MTR_OK;
  return static_cast<unsigned char*>(g_scratch_ptr[dev]);
}

template <int D, int DEG>
int run_noalloc(unsigned char* base, const mtr_params& p, const double* x, const double* v, const double* B,
                uint32_t Np, const double* gx, const double* gy, const double* gz, const uint32_t dims[3],
                double* grid_mass, double* grid_v, uint32_t* status, cudaStream_t st) {
  constexpr int TB = Tiling<D>::TB;
  StepHeader* H = reinterpret_cast<StepHeader*>(base + kOffHeader);
  DevParams* P = reinterpret_cast<DevParams*>(base + kOffParams);
  const uint32_t nx = dims[0], ny = dims[1], nz = D == 3 ? dims[2] : 1;
  const uint32_t tx = (nx + TB - 1) / TB, ty = (ny + TB - 1) / TB, tz = D == 3 ? (nz + TB - 1) / TB : 1;
  const uint64_t G = (uint64_t)nx * ny * nz, ntiles = (uint64_t)tx * ty * tz;
  const double apicD = p.spline_deg == 3 ? 3.0 / (p.dx * p.dx) : 4.0 / (p.dx * p.dx);
  StepArgs A{};
  A.P = P;
  A.H = H;
  A.Np = Np;
  A.gx = const_cast<double*>(gx);
  A.gy = const_cast<double*>(gy);
  A.gz = const_cast<double*>(gz ? gz : gy);
  A.cap_nodes = (uint32_t)G;
  A.cap_tiles = (uint32_t)ntiles;
  A.acc = reinterpret_cast<double*>(base + kOffAcc);
  A.keys0 = reinterpret_cast<uint32_t*>(base + kOffKeys0);
  A.perm_rank = reinterpret_cast<uint32_t*>(base + kOffRank);
  A.perm = A.perm_rank;
  A.perm_tmp = reinterpret_cast<uint32_t*>(base + kOffTmp);
  A.big_cells = reinterpret_cast<uint32_t*>(base + kOffBig);
  A.cell_start = reinterpret_cast<uint32_t*>(base + kOffStart);
  A.cell_count = reinterpret_cast<uint32_t*>(base + kOffCount);
  A.super = reinterpret_cast<uint32_t*>(base + kOffSuper);
  A.in.x = const_cast<double*>(x);
  A.xin = x;
  A.in.v = const_cast<double*>(v);
  A.in.B = const_cast<double*>(B);
  if (ntiles > kMaxTiles) return MTR_ERR_TOO_LARGE;  // cannot happen (see kMaxTiles)
  const uint32_t supers = (uint32_t)((ntiles * 64 + 1 + kSuperCells - 1) / kSuperCells);
  const uint32_t pblocks = (Np + kSortThreads - 1) / kSortThreads;
  // sets the header up and clears what must start at zero: this grid's cell
  // counts and accumulators
  k_noalloc_setup<<<(uint32_t)std::min<uint64_t>((G * (1 + D) + 255) / 256, 148 * 4), 256, 0, st>>>(
      H, P, gx, gy, gz, nx, ny, nz, tx, ty, tz, 1.0 / p.dx, apicD, p.flip_ratio, p.particle_mass, Np, D, A.acc,
      (uint32_t)(G * (1 + D)), A.cell_count, supers * kSuperCells, A.super, supers);
  k_noalloc_keys<D><<<pblocks, kSortThreads, 0, st>>>(A);
  k_sort_scan<<<supers, kSortThreads, 0, st>>>(A);
  k_sort_place<<<pblocks, kSortThreads, 0, st>>>(A);
  k_sort_rank<<<pblocks, kSortThreads, 0, st>>>(A);
  const int parts = ntiles <= kFewTiles ? 4 : 2, threads = ntiles <= kFewTiles ? kScatterThreads : kScatterThreads / 2;
  k_p2g_noalloc<D, DEG><<<dim3((uint32_t)ntiles, parts), threads, noalloc_smem_bytes<D>(threads), st>>>(A, A.perm);
  k_noalloc_finalize<D><<<(uint32_t)std::min<uint64_t>((G + 255) / 256, 148 * 8), 256, 0, st>>>(
      A.acc, (uint32_t)G, (uint32_t)G, p.particle_mass, grid_mass, grid_v, H, status);
  return cudaGetLastError() == cudaSuccess ? MTR_OK : MTR_ERR_CUDA;
}

}  // namespace

extern "C" int mtr_p2g_noalloc(const mtr_params* params, const double* x, const double* v, const double* B,
                               uint32_t Np, const double* gx, const double* gy, const double* gz,
                               const uint32_t dims[3], double* grid_mass, double* grid_v, uint32_t* status,
                               void* stream) {
  // an error left by earlier, unrelated work of this thread is not this call's failure
  (void)cudaGetLastError();
  if (!params || !x || !v || !gx || !gy || !dims || !grid_mass || !grid_v || Np == 0) return MTR_ERR_INVALID;
  const mtr_params& p = *params;
  if ((p.dim != 2 && p.dim != 3) || (p.spline_deg != 2 && p.spline_deg != 3) || !(p.dx > 0)) return MTR_ERR_INVALID;
  if (p.dim == 3 && !gz) return MTR_ERR_INVALID;
  if (p.flip_ratio < 0 && !B) return MTR_ERR_INVALID;
  const uint64_t G = (uint64_t)dims[0] * dims[1] * (p.dim == 3 ? dims[2] : 1);
  if (dims[0] < 4 || dims[1] < 4 || (p.dim == 3 && dims[2] < 4)) return MTR_ERR_INVALID;
  if (Np > MTR_NOALLOC_MAX_PARTICLES || G > MTR_NOALLOC_MAX_NODES) return MTR_ERR_TOO_LARGE;
  int rc = MTR_OK;
  unsigned char* base = scratch_for_current_device(&rc);
  if (!base) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (p.dim == 3)
    return p.spline_deg == 3 ? run_noalloc<3, 3>(base, p, x, v, B, Np, gx, gy, gz, dims, grid_mass, grid_v, status, st)
                             : run_noalloc<3, 2>(base, p, x, v, B, Np, gx, gy, gz, dims, grid_mass, grid_v, status, st);
  return p.spline_deg == 3 ? run_noalloc<2, 3>(base, p, x, v, B, Np, gx, gy, gz, dims, grid_mass, grid_v, status, st)
                           : run_noalloc<2, 2>(base, p, x, v, B, Np, gx, gy, gz, dims, grid_mass, grid_v, status, st);
}
