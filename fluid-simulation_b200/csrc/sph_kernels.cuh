// CUDA kernels of the SPH step engine (sm_100a). Mostly one thread per particle;
// neighbor lists hold 16-bit positions in the block's halo and are stored
// warp-tiled (see nbr_slot): the 32 particles of a warp own one contiguous
// block, and each lane reads four consecutive neighbors with one 64-bit load, so
// a warp streams its lists as 256-byte coalesced reads. Gathered neighbor state
// comes from shared memory, where a block stages its halo's records.
//
// Reference functions each kernel restates (paths under simulation_lib/src/):
//   k_integrate_key      integration_schemes/euler_cromer.rs:12-25,
//                        take_predicted.rs:14-27, sph/mod.rs:674-699 (disable,
//                        max speed), spatial_hashing.rs:27-46 (cells)
//   k_scan_*, k_scatter, k_gather_particles
//                        spatial_hashing.rs:27-37 (populate) as a counting sort
//   k_neighbors_density  spatial_hashing.rs:75-158, neighbor_search/mod.rs:118-155,
//                        sph/quantities.rs:14-61 (get_volume's fluid sum)
//   k_volume             sph/quantities.rs:14-61 (get_volume), average density
//   k_sample_boundary    boundary_handling/static_sample_boundary.rs:157-168,
//                        sph/non_pressure_accelerations.rs (boundary viscosity)
//   k_vm_near, k_vm_sample
//                        boundary_handling/volume_map_boundary.rs:1259-1424,
//                        utilities/discretization.rs:437-557
//   k_accel              sph/non_pressure_accelerations.rs:19-185,
//                        pressure_solver/mod.rs:90-195, sesph.rs:31-67
//   k_body_react         the reactions of boundary viscosity and pressure
//   k_iisph_source_diag, k_sweep_*, k_solve
//                        pressure_solver/iisph.rs:117-560,
//                        iisph_optimized_source_term.rs:53-217
//   k_body_*             boundary_handling/rigid_body_motion.rs:135-201
//   k_quantity_at        sph/mod.rs:241-341, sph/quantities.rs:14-330
#pragma once

#include <cfloat>
#include <cmath>
#include <type_traits>

#include "sph_engine.cuh"

namespace sph {

// ---------------------------------------------------------------------------
// Reductions: fixed-order block reductions and last-block completion so the
// result does not depend on scheduling.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0;
  if (w == 0) {
    t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    t = warp_sum(t);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// Sum of per-block partials in a fixed order, run by the last block to finish.
// Returns true in thread 0 of that block with *total set.
__device__ __forceinline__ bool last_block_total(double block_value, double* partials,
                                                 unsigned int* counter, double* total,
                                                 double* sh) {
  __shared__ bool is_last;
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = block_value;
    __threadfence();
    unsigned t = atomicAdd(counter, 1u);
    is_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return false;
  __threadfence();
  double s = 0;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) s += ((volatile double*)partials)[b];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) {
    *total = s;
    *counter = 0;
  }
  return threadIdx.x == 0;
}

// Programmatic dependent launch: a kernel launched with programmatic stream
// serialization may start while the kernel before it finishes its last wave.
// grid_dep_wait() returns once that kernel has completed and its writes are
// visible; everything before it may read only data the earlier kernel does
// not write. grid_dep_release() lets the next kernel start launching (once
// every block of this grid has started). Both are no-ops in a plain launch.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_dep_release() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// Such a kernel's pointers carry no __restrict__: the kernel before may still write
// what they point to, so the promise does not hold, and with it the compiler may read
// through the non-coherent cache or move an access above the wait. (__ldg is for
// what nothing has written since the kernel before the last one ended: halo indices
// behind the volume pass, field nodes.)
// The start of a kernel that reads what the kernel before it wrote: its blocks
// are on their SMs by then, and the next kernel's may follow (small scenes, where
// a step is a dozen kernels of 3 to 30 us, save the launch latency between them).
__device__ __forceinline__ void grid_dep_begin() {
  grid_dep_wait();
  grid_dep_release();
}

// ---------------------------------------------------------------------------
// Rigid-body helpers (f64), nalgebra semantics (rigid_body_motion.rs)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void qrot(const double q[4], const double v[3], double out[3]) {
  // t = 2 (q.v x v); out = v + w t + q.v x t
  double tx = 2.0 * (q[2] * v[2] - q[3] * v[1]);
  double ty = 2.0 * (q[3] * v[0] - q[1] * v[2]);
  double tz = 2.0 * (q[1] * v[1] - q[2] * v[0]);
  double cx = q[2] * tz - q[3] * ty, cy = q[3] * tx - q[1] * tz, cz = q[1] * ty - q[2] * tx;
  out[0] = (tx * q[0] + cx) + v[0];
  out[1] = (ty * q[0] + cy) + v[1];
  out[2] = (tz * q[0] + cz) + v[2];
}
__device__ __forceinline__ void body_world_to_local(const Body& b, const double p[3], double out[3]) {
  double d[3] = {p[0] - b.com[0], p[1] - b.com[1], p[2] - b.com[2]};
  double qi[4] = {b.q[0], -b.q[1], -b.q[2], -b.q[3]};
  qrot(qi, d, out);
}
__device__ __forceinline__ void body_velocity_at(const Body& b, const double p[3], double out[3]) {
  double r[3] = {p[0] - b.com[0], p[1] - b.com[1], p[2] - b.com[2]};
  out[0] = b.v[0] + (b.omega[1] * r[2] - b.omega[2] * r[1]);
  out[1] = b.v[1] + (b.omega[2] * r[0] - b.omega[0] * r[2]);
  out[2] = b.v[2] + (b.omega[0] * r[1] - b.omega[1] * r[0]);
}

// ---------------------------------------------------------------------------
// 1. integrate + cell key + bucket histogram (+ disable test, max speed)
// ---------------------------------------------------------------------------
// mode: 0 EulerCromer, 1 TakePredicted, 2 no integration (initial update)
template <class R>
__global__ void __launch_bounds__(kBlock) k_integrate_key(
    Scalars* __restrict__ sc, R4<R>* __restrict__ pos, R4<R>* __restrict__ vel,
    const R4<R>* __restrict__ acc, const R4<R>* __restrict__ xint, const R4<R>* __restrict__ vint,
    int mode, uint32_t* __restrict__ key, uint32_t* __restrict__ slot,
    uint32_t* __restrict__ count, StepParams<R> P) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = sc->n;
  double speed = 0.0;
  if (i < n) {
    R4<R> x = pos[i], v = vel[i];
    if (mode == 0) {
      const R dt = (R)sc->dt;
      const R4<R> a = acc[i];
      v.x = v.x + dt * a.x; v.y = v.y + dt * a.y; v.z = v.z + dt * a.z;
      x.x = x.x + dt * v.x; x.y = x.y + dt * v.y; x.z = x.z + dt * v.z;
      vel[i] = v;
    } else if (mode == 1) {
      const R m = v.w;
      x = xint[i];
      v = vint[i];
      v.w = m;
      vel[i] = v;
    }
    uint32_t k;  // also kept in the position's spare lane, which the sort carries along
    if ((double)x.z < P.disable_below) {
      k = P.T;
      atomicAdd(&sc->n_below, 1);
    } else {
      k = morton_key(cell_coord((double)x.x, P.range), cell_coord((double)x.y, P.range),
                     cell_coord((double)x.z, P.range), P.mask);
      const double vx = v.x, vy = v.y, vz = v.z;
      speed = sqrt((vx * vx + vy * vy) + vz * vz);
    }
    x.w = key_lane<R>(k);
    pos[i] = x;
    key[i] = k;
    slot[i] = atomicAdd(&count[k], 1u);
  }
  // block max of the speed (non-negative doubles order like their bit patterns)
  unsigned long long bits = (unsigned long long)__double_as_longlong(speed);
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long ob = __shfl_down_sync(0xffffffffu, bits, o);
    bits = ob > bits ? ob : bits;
  }
  __shared__ unsigned long long smax[kBlock / 32];
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = bits;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long m = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = smax[w] > m ? smax[w] : m;
    if (m) atomicMax(&sc->max_speed, m);
  }
}

// Step prologue: active count and the CFL time increment (sph/mod.rs:825-829).
// One thread of the first scan kernel runs it: everything before it in the step
// has ended there, and nothing before the scan's end reads its results.
struct Prologue {
  Scalars* sc;  // null: no prologue (other scans)
  int cfl, accumulate_time;
  double cfl_number, spacing, dt_max;
};
__device__ __forceinline__ void run_prologue(const Prologue& P) {
  Scalars* sc = P.sc;
  sc->n_active = sc->n - sc->n_below;
  // simulated time of a CFL step advances by the increment it integrated with
  // (the one chosen by the previous update); graph-captured steps keep it here
  if (P.accumulate_time) sc->time_acc += sc->dt;
  if (P.cfl) {
    const double ms = __longlong_as_double((long long)sc->max_speed);
    const double c = P.cfl_number * P.spacing / ms;  // +inf at rest
    sc->dt = fmin(P.dt_max, c);
  }
  sc->max_nbrs = 0;
  sc->max_bnbrs = 0;
  sc->max_halo = 0;
  sc->n_wide = 0;
  sc->vm_near = 0;
  sc->n_touch = 0;
  sc->iterations = 0;
  sc->iterations_eqs1 = 0;
  sc->converged = 0;
  sc->err = INFINITY;
  sc->status = 0;
}

// ---------------------------------------------------------------------------
// 2. exclusive scan of bucket counts; clears the counts for reuse. Tile sums,
// then every block adds up the tiles before its own (DIRECT); from kScanDirect
// tiles on (2^22 buckets, large surface lattices) a kernel of its own scans the
// tile sums in between.
// ---------------------------------------------------------------------------
constexpr int kScanItems = 8;
constexpr int kScanTile = kBlock * kScanItems;

__device__ __forceinline__ uint32_t block_excl_scan_u32(uint32_t v, uint32_t* sh, uint32_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    uint32_t s = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    sh[lane] = s;
  }
  __syncthreads();
  uint32_t base = w > 0 ? sh[w - 1] : 0;
  if (total) *total = sh[(blockDim.x >> 5) - 1];
  __syncthreads();
  return base + x - v;
}

// A thread's kScanItems consecutive counts: two 16-byte loads when they lie
// inside [0, m) (the arrays are 16-byte aligned and base is a multiple of 8).
static_assert(kScanItems == 8, "two uint4 per thread");
__device__ __forceinline__ void scan_load8(const uint32_t* in, int base, int m, uint32_t v[8]) {
  if (base + 8 <= m) {
    const uint4 a = __ldcs(reinterpret_cast<const uint4*>(in + base));
    const uint4 b = __ldcs(reinterpret_cast<const uint4*>(in + base) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = base + k < m ? in[base + k] : 0u;
  }
}

constexpr int kScanDirect = 2048;
__global__ void __launch_bounds__(kBlock) k_scan_tiles(const uint32_t* in, int m,
                                                      uint32_t* tile_sums, Prologue prologue) {
  grid_dep_begin();
  __shared__ uint32_t sh[32];
  if (prologue.sc && blockIdx.x == 0 && threadIdx.x == 0) run_prologue(prologue);
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  scan_load8(in, base, m, v);
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += v[k];
  uint32_t total;
  block_excl_scan_u32(s, sh, &total);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_tile_sums(uint32_t* tile_sums, int ntiles) {
  grid_dep_begin();
  __shared__ uint32_t sh[32];
  // each thread owns a contiguous run of tiles
  const int per = (ntiles + blockDim.x - 1) / blockDim.x;
  const int b = threadIdx.x * per;
  uint32_t s = 0;
  for (int k = 0; k < per; ++k) s += b + k < ntiles ? tile_sums[b + k] : 0u;
  uint32_t run = block_excl_scan_u32(s, sh, nullptr);
  for (int k = 0; k < per; ++k)
    if (b + k < ntiles) {
      uint32_t t = tile_sums[b + k];
      tile_sums[b + k] = run;
      run += t;
    }
}

template <bool DIRECT>
__global__ void __launch_bounds__(kBlock) k_scan_apply(uint32_t* in, int m,
                                                      const uint32_t* tile_sums,
                                                      uint32_t* out) {
  grid_dep_begin();
  __shared__ uint32_t sh[32];
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  scan_load8(in, base, m, v);
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += v[k];
  uint32_t before = 0;
  if (DIRECT) {
    for (int t = threadIdx.x; t < (int)blockIdx.x; t += kBlock) before += tile_sums[t];
    block_excl_scan_u32(before, sh, &before);
  } else {
    before = tile_sums[blockIdx.x];
  }
  uint32_t run = block_excl_scan_u32(s, sh, nullptr) + before;
  if (base + 8 <= m) {
    uint32_t o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      o[k] = run;
      run += v[k];
    }
    uint4* po = reinterpret_cast<uint4*>(out + base);
    po[0] = make_uint4(o[0], o[1], o[2], o[3]);
    po[1] = make_uint4(o[4], o[5], o[6], o[7]);
    uint4* pz = reinterpret_cast<uint4*>(in + base);  // counts are rebuilt by the next histogram
    pz[0] = make_uint4(0u, 0u, 0u, 0u);
    pz[1] = make_uint4(0u, 0u, 0u, 0u);
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
      if (base + k < m) {
        out[base + k] = run;
        run += v[k];
        in[base + k] = 0u;
      }
  }
}

// ---------------------------------------------------------------------------
// 3. scatter, then gather with in-bucket ordering by reference index
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) k_scatter(const int* n_ptr,
                                                   const uint32_t* key,
                                                   const uint32_t* slot,
                                                   const uint32_t* start,
                                                   uint32_t* perm) {
  grid_dep_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= *n_ptr) return;
  perm[start[key[i]] + slot[i]] = (uint32_t)i;
}

// The place of sorted entry d in its bucket ordered by `order` (the reference
// index), which makes the sorted order independent of the atomic slot
// assignment: every entry counts the smaller ones of its bucket. (One thread
// per bucket sorting by insertion took 14 to 25 us where a sphere's samples
// crowd a bucket.)
__device__ __forceinline__ uint32_t ranked_place(uint32_t j, const uint32_t* key,
                                                 const uint32_t* start,
                                                 const uint32_t* order,
                                                 const uint32_t* perm) {
  const uint32_t k = key[j], b = start[k], e = start[k + 1], mine = order[j];
  uint32_t rank = 0;
#pragma unroll 4
  for (uint32_t t = b; t < e; ++t) rank += order[perm[t]] < mine ? 1u : 0u;
  return b + rank;
}

template <class R>
__global__ void __launch_bounds__(kBlock) k_gather_particles(
    const int* n_ptr, const uint32_t* perm, const uint32_t* key,
    const uint32_t* start, const R4<R>* pos, const R4<R>* vel,
    const uint32_t* ref, const uint32_t* fid, R4<R>* pos2,
    R4<R>* vel2, uint32_t* ref2, uint32_t* fid2) {
  grid_dep_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= *n_ptr) return;
  const uint32_t j = perm[t];
  const R4<R> x = pos[j], v = vel[j];
  const uint32_t r = ref[j], f = fid[j];
  const uint32_t d = ranked_place(j, key, start, ref, perm);
  pos2[d] = x;
  vel2[d] = v;
  ref2[d] = r;
  fid2[d] = f;
}

// boundary samples: key + histogram (no integration)
template <class R>
__global__ void __launch_bounds__(kBlock) k_sample_key(const int* __restrict__ n_ptr,
                                                      const R4<R>* __restrict__ xb,
                                                      uint32_t* __restrict__ key,
                                                      uint32_t* __restrict__ slot,
                                                      uint32_t* __restrict__ count, double range,
                                                      uint32_t mask) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= *n_ptr) return;
  const R4<R> x = xb[i];
  const uint32_t k = morton_key(cell_coord((double)x.x, range), cell_coord((double)x.y, range),
                                cell_coord((double)x.z, range), mask);
  key[i] = k;
  slot[i] = atomicAdd(&count[k], 1u);
}

template <class R>
__global__ void __launch_bounds__(kBlock) k_gather_samples(
    const int* __restrict__ n_ptr, const uint32_t* __restrict__ perm, const uint32_t* __restrict__ key,
    const uint32_t* __restrict__ start, const R4<R>* __restrict__ xb, const R4<R>* __restrict__ vb,
    const uint32_t* __restrict__ bid, const uint32_t* __restrict__ orig, R4<R>* __restrict__ xb2,
    R4<R>* __restrict__ vb2, uint32_t* __restrict__ bid2, uint32_t* __restrict__ orig2) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= *n_ptr) return;
  const uint32_t j = perm[t];
  const uint32_t d = ranked_place(j, key, start, orig, perm);
  xb2[d] = xb[j];
  vb2[d] = vb[j];
  bid2[d] = bid[j];
  orig2[d] = orig[j];
}

// ---------------------------------------------------------------------------
// 4. fluid neighbor lists + volume (fused), block halos
//
// The particles of one block (kBlock consecutive particles in bucket order)
// find their neighbors in the union of the 27-bucket stencils of their
// cells: the block's halo. Because buckets are contiguous in memory and the
// halo is kept cell by cell, rows of cells along x one after the other, the
// halo is a short list of runs of consecutive particle indices (halo_idx). Neighbor lists
// hold 16-bit positions in the block's halo. The passes over neighbors copy
// the halo's records into shared memory once per launch (ordered loads of
// those runs) and gather from there; a block whose halo does not fit the
// shared-memory capacity gathers through halo_idx from global memory.
//
// Neighbor-list layout: particle i = 32*t + lane keeps its k-th neighbor at
//   ((t * K/4 + k/4) * 32 + lane) * 4 + k % 4      (K a multiple of 4)
// i.e. tile-major, then groups of four neighbors, then lane, so a warp reads
// the next four neighbors of all its lanes as one 256-byte coalesced load.
__device__ __forceinline__ size_t nbr_slot(int i, int k, int K) {
  const size_t t = (size_t)(i >> 5), lane = (size_t)(i & 31);
  return ((t * (size_t)(K >> 2) + (size_t)(k >> 2)) * 32 + lane) * 4 + (size_t)(k & 3);
}

// Neighbor lists of one step and the block halos they index.
struct NbrArgs {
  const uint16_t* nbr;   // halo positions, layout of nbr_slot
  const uint32_t* ncnt;  // neighbors per particle (self excluded)
  const uint32_t* hidx;  // [blocks][hcap] halo particle indices
  const uint32_t* hn;    // [blocks] halo sizes
  int K;                 // list capacity per particle
  int hcap;              // halo table capacity per block
  int hs;                // halo records a launch stages in shared memory
  int ahead = 0;         // sweep passes: blocks resident at once (L2 prefetch distance), 0 = none
};

// L2 prefetch for the block one wave ahead (block b + ahead runs on the slot
// this block frees, about one block lifetime later): its particles' records,
// the first list groups of its warps and its halo indices, so that its start
// reads from L2 instead of DRAM.
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}
__device__ __forceinline__ void prefetch_lines(const void* p, size_t bytes) {
  const char* c = static_cast<const char*>(p);
  for (size_t o = (size_t)threadIdx.x * 128; o < bytes; o += (size_t)kBlock * 128) prefetch_l2(c + o);
}
constexpr int kPrefetchGroups = 10;     // list groups per warp (about 36 neighbors)
constexpr int kPrefetchHalo = 1408;     // halo indices (the typical halo of a block)
// (m: the block's particles; its warps beyond them hold no lists)
__device__ __forceinline__ void prefetch_block_lists(const NbrArgs& N, int b, int m) {
  const int G = min(N.K >> 2, kPrefetchGroups);
  const char* base = reinterpret_cast<const char*>(N.nbr + nbr_slot(b * kBlock, 0, N.K));
  const size_t warp_bytes = (size_t)(N.K >> 2) * 256;
  for (int q = threadIdx.x; q < ((m + 31) >> 5) * G * 2; q += kBlock)
    prefetch_l2(base + (size_t)(q / (2 * G)) * warp_bytes + (size_t)(q % (2 * G)) * 128);
  prefetch_lines(N.hidx + (size_t)b * N.hcap, (size_t)min(N.hcap, kPrefetchHalo) * sizeof(uint32_t));
}
// The prefetch of a neighbor pass: the per-particle streams it reads (and
// the neighbor counts) for block blockIdx.x + N.ahead, its lists and halo.
template <class... T>
__device__ __forceinline__ void prefetch_ahead(const NbrArgs& N, int n, const T*... streams) {
  if (N.ahead <= 0) return;
  const int b = blockIdx.x + N.ahead;
  if (b * kBlock >= n) return;
  const int i0 = b * kBlock, m = min(kBlock, n - i0);
  (prefetch_lines(streams + i0, (size_t)m * sizeof(T)), ...);
  prefetch_lines(N.ncnt + i0, (size_t)m * sizeof(uint32_t));
  prefetch_block_lists(N, b, m);
}

// The block's halo: its particle indices, its size and whether the launch
// copies its records to shared memory.
struct HaloView {
  const uint32_t* idx;
  int size;
  bool staged;
};
__device__ __forceinline__ HaloView halo_view(const NbrArgs& N) {
  HaloView h;
  h.idx = N.hidx + (size_t)blockIdx.x * (size_t)N.hcap;
  h.size = min((int)N.hn[blockIdx.x], N.hcap);
  h.staged = h.size <= N.hs;
  return h;
}

// Asynchronous global -> shared copies (cp.async): the records travel without
// passing through registers, so every copy a thread issues is in flight at
// once; stage_done() waits for this thread's copies and then for the block.
template <class T>
__device__ __forceinline__ void async_copy(T* smem_dst, const T* gsrc) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8 || sizeof(T) % 16 == 0, "cp.async moves 4, 8 or 16 bytes");
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  if constexpr (sizeof(T) % 16 == 0) {
#pragma unroll
    for (int o = 0; o < (int)sizeof(T); o += 16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + o),
                   "l"(reinterpret_cast<const char*>(gsrc) + o) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(gsrc), "n"(sizeof(T)) : "memory");
  }
}
__device__ __forceinline__ void stage_done() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
}

// Copies the block's halo records to shared memory: copy(l, g) moves the
// record of particle g to position l. Four halo indices per thread are read
// at a time, then their records are requested.
template <class F>
__device__ __forceinline__ void stage_halo(const HaloView& H, F&& copy) {
  for (int l0 = threadIdx.x; l0 < H.size; l0 += 4 * kBlock) {
    uint32_t g[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int l = l0 + u * kBlock;
      g[u] = l < H.size ? __ldg(H.idx + l) : 0u;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int l = l0 + u * kBlock;
      if (l < H.size) copy(l, g[u]);
    }
  }
}
// stage_halo in two steps for the sweep passes: halo_first() reads the
// first batch of halo indices (fixed during a solve, so before the grid
// dependency wait), stage_halo_from() requests the records and the rest.
struct HaloFirst {
  uint32_t g[4];
};
__device__ __forceinline__ HaloFirst halo_first(const HaloView& H) {
  HaloFirst f;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int l = threadIdx.x + u * kBlock;
    f.g[u] = H.staged && l < H.size ? __ldg(H.idx + l) : 0u;
  }
  return f;
}
template <class F>
__device__ __forceinline__ void stage_halo_from(const HaloView& H, const HaloFirst& f, F&& copy) {
  if (!H.staged) return;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int l = threadIdx.x + u * kBlock;
    if (l < H.size) copy(l, f.g[u]);
  }
  for (int l0 = threadIdx.x + 4 * kBlock; l0 < H.size; l0 += 4 * kBlock) {
    uint32_t g[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int l = l0 + u * kBlock;
      g[u] = l < H.size ? __ldg(H.idx + l) : 0u;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int l = l0 + u * kBlock;
      if (l < H.size) copy(l, g[u]);
    }
  }
}

template <class R>
__device__ __forceinline__ void kahan_add(R& s, R& c, R t) {
  const R y = t - c;
  const R u = s + y;
  c = (u - s) - y;
  s = u;
}

// The 27 stencil bucket keys of cell (cx,cy,cz) in stencil order.
__device__ __forceinline__ void stencil_keys(int cx, int cy, int cz, uint32_t mask, uint32_t keys[27]) {
#pragma unroll
  for (int q = 0; q < 27; ++q) keys[q] = morton_key(cx + (q % 3) - 1, cy + (q / 3) % 3 - 1, cz + q / 9 - 1, mask);
}

// Shared memory of the neighbor search. Region X holds the halo's positions
// (x, y and z each in an array of its own, so that a 16-byte load brings one
// coordinate of four f32 candidates), region L the lists under construction
// (entry k of thread t at [k * kBlock + t]) and, before them, the halo's
// construction; region W the candidate runs of the block's cells. Four blocks
// share an SM.
constexpr size_t kSearchX = 24576;       // 2048 f32 / 1024 f64 positions
constexpr int kListStage = 48;           // list entries per particle kept in shared memory
constexpr size_t kSearchL = (size_t)kListStage * kBlock * sizeof(uint16_t);
constexpr int kSearchCells = 184;        // cells of a block whose candidates are kept as runs
constexpr size_t kSearchW = (size_t)9 * kSearchCells * sizeof(uint32_t);
constexpr size_t kSearchSmem = kSearchX + kSearchL + kSearchW;
constexpr int kBoxCells = 16384;         // cells of the block's bounding boxes (one bit each)
constexpr int kBoxLevel = 12;            // key bit from which a block's cells get two boxes (16^3 cells)
constexpr int kHaloCells = 3064;         // distinct halo cells
constexpr int kHaloKeys = 8192;          // general path: >= 27 * kBlock stencil keys, a power of two
constexpr uint32_t kNoKey = 0xffffffffu;
static_assert(kHaloKeys >= 27 * kBlock, "the sort buffer must hold the stencil keys of a full block");
static_assert(kHaloKeys * (sizeof(uint32_t) + sizeof(uint16_t)) <= kSearchX + kSearchL, "general path buffers");
static_assert(kBoxCells / 32 * (sizeof(uint32_t) + sizeof(uint16_t)) + (kHaloCells + 2) * sizeof(uint16_t) +
                      kHaloCells * sizeof(uint32_t) + kBlock * sizeof(int3) <= kSearchL, "halo construction buffers");

// Distance tests of one particle against n staged candidates (n a multiple of
// four, px/py/pz 16-byte aligned): the sign bit of r^2 - limit of candidate c
// ends at bit n - 1 - c.
struct RangeTest32 {
  unsigned long long x, y, z, limit;
  __device__ __forceinline__ RangeTest32(const R4<float>& xi, float lim)
      : x(pack2(-xi.x, -xi.x)), y(pack2(-xi.y, -xi.y)), z(pack2(-xi.z, -xi.z)), limit(pack2(-lim, -lim)) {}
  __device__ __forceinline__ unsigned long long two(unsigned long long a, unsigned long long b,
                                                    unsigned long long c) const {
    const unsigned long long dx = add2(a, x), dy = add2(b, y), dz = add2(c, z);
    return fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, limit)));
  }
  __device__ __forceinline__ uint32_t run(const float* px, const float* py, const float* pz, int n) const {
    uint32_t hits = 0;
#pragma unroll 2
    for (int c = 0; c < n; c += 4) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(px + c);
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(py + c);
      const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(pz + c);
      const unsigned long long r0 = two(a.x, b.x, d.x), r1 = two(a.y, b.y, d.y);
      hits = __funnelshift_l((uint32_t)r0, hits, 1);
      hits = __funnelshift_l((uint32_t)(r0 >> 32), hits, 1);
      hits = __funnelshift_l((uint32_t)r1, hits, 1);
      hits = __funnelshift_l((uint32_t)(r1 >> 32), hits, 1);
    }
    return hits;
  }
};
// f64: NaN results keep a sign (inf - inf gives a negative one), so the test is on
// the magnitude of r^2: its upper word, the sign shifted out, minus the limit's,
// rounded up (a shell of 2^-18 more candidates, which the exact predicate decides).
struct RangeTest64 {
  double x, y, z;
  uint32_t limit;
  __device__ __forceinline__ RangeTest64(const R4<double>& xi, double lim) : x(xi.x), y(xi.y), z(xi.z) {
    limit = ((uint32_t)__double2hiint(lim) >> 1) + 1u;
  }
  __device__ __forceinline__ uint32_t one(double a, double b, double c) const {
    const double dx = a - x, dy = b - y, dz = c - z;
    return ((uint32_t)__double2hiint(dz * dz + (dy * dy + dx * dx)) >> 1) - limit;
  }
  __device__ __forceinline__ uint32_t run(const double* px, const double* py, const double* pz, int n) const {
    uint32_t hits = 0;
    for (int c = 0; c < n; c += 2) {
      const double2 a = *reinterpret_cast<const double2*>(px + c);
      const double2 b = *reinterpret_cast<const double2*>(py + c);
      const double2 d = *reinterpret_cast<const double2*>(pz + c);
      hits = __funnelshift_l(one(a.x, b.x, d.x), hits, 1);
      hits = __funnelshift_l(one(a.y, b.y, d.y), hits, 1);
    }
    return hits;
  }
};
template <class R>
using RangeTest = std::conditional_t<sizeof(R) == 4, RangeTest32, RangeTest64>;

// Compensated (Kahan) sum of W over the neighbors in list order, on top of the
// self term W(0) = alpha/h^3 / 2; add() takes the coordinates of four
// neighbors, of which the first n count, and keeps the largest squared
// distance. f32: two kernel values per packed instruction.
struct KernelSum32 {
  unsigned long long x, y, z;
  float ih, cw, s, c = 0.f, farthest = 0.f;
  __device__ __forceinline__ KernelSum32(const R4<float>& xi, const KernelConst<float>& k)
      : x(pack2(-xi.x, -xi.x)), y(pack2(-xi.y, -xi.y)), z(pack2(-xi.z, -xi.z)), ih(-k.inv_h),
        cw(k.cw), s(k.cw * 0.5f) {}
  __device__ __forceinline__ void one(float w) {
    const float v = fmaf(cw, w, -c), n = s + v;
    c = (n - s) - v;
    s = n;
  }
  __device__ __forceinline__ void two(const R4<float>& a, const R4<float>& b, int n) {
    const unsigned long long dx = add2(pack2(a.x, b.x), x), dy = add2(pack2(a.y, b.y), y),
                             dz = add2(pack2(a.z, b.z), z);
    const unsigned long long r2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));
    // (a coincident neighbor keeps a finite root)
    const float r0 = fmaxf(__uint_as_float((uint32_t)r2), 1e-35f);
    const float r1 = fmaxf(__uint_as_float((uint32_t)(r2 >> 32)), 1e-35f);
    farthest = fmaxf(farthest, r0);
    if (n > 1) farthest = fmaxf(farthest, r1);
    const unsigned long long half = pack2(0.5f, 0.5f), r = roots2(r0, r1);
    // -|r|/h, in scalar form: a packed product and the packed sums behind it
    // were measured to round once, and with them the volumes' last bits change
    const unsigned long long q = pack2(__fmul_rn(__uint_as_float((uint32_t)r), ih),
                                       __fmul_rn(__uint_as_float((uint32_t)(r >> 32)), ih));
    // (a neighbor is within the support up to rounding: 1 - q needs no clamp)
    const unsigned long long a1 = add2(pack2(1.f, 1.f), q), u = add2(half, q);
    const unsigned long long b1 = pack2(fmaxf(__uint_as_float((uint32_t)u), 0.f),
                                        fmaxf(__uint_as_float((uint32_t)(u >> 32)), 0.f));
    const unsigned long long w = fma2(mul2(a1, a1), a1, mul2(mul2(mul2(b1, b1), b1), pack2(-4.f, -4.f)));
    one(__uint_as_float((uint32_t)w));
    if (n > 1) one(__uint_as_float((uint32_t)(w >> 32)));
  }
  __device__ __forceinline__ void add(const R4<float> p[4], int n) {
    two(p[0], p[1], n);
    if (n > 2) two(p[2], p[3], n - 2);
  }
};
struct KernelSum64 {
  R4<double> xi;
  KernelConst<double> k;
  double s, c = 0, farthest = 0;
  __device__ __forceinline__ KernelSum64(const R4<double>& x, const KernelConst<double>& kc)
      : xi(x), k(kc), s(kc.cw * 0.5) {}
  __device__ __forceinline__ void add(const R4<double> p[4], int n) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (u >= n) break;
      const double rx = xi.x - p[u].x, ry = xi.y - p[u].y, rz = xi.z - p[u].z;
      const double r2 = rx * rx + ry * ry + rz * rz;
      farthest = fmax(farthest, r2);
      kahan_add(s, c, kernel_w_r2(r2, k));
    }
  }
};
template <class R>
using KernelSum = std::conditional_t<sizeof(R) == 4, KernelSum32, KernelSum64>;

// The neighbors one particle has found, before they are written out: up to
// kListStage halo positions in shared memory (entry k of thread t at
// [k * kBlock + t]), a longer list in its place in global memory.
struct FoundList {
  uint16_t* s;       // shared memory, this thread's entry 0
  uint16_t* list;    // global memory: entry k at list[(k >> 2) * 128 + (k & 3)]
  int cap;           // capacity of the global list
  int cnt = 0;
  bool global = false;
  __device__ __forceinline__ uint16_t& slot(int k) {
    return global ? list[(size_t)(k >> 2) * 128 + (k & 3)] : s[k * kBlock];
  }
  // hits: candidate p + c at bit 31 - c
  __device__ __forceinline__ void add(uint32_t hits, uint32_t p) {
    const int n = __popc(hits);
    if (!global && cnt + n > kListStage) {
      for (int k = 0; k < min(cnt, cap); ++k) list[(size_t)(k >> 2) * 128 + (k & 3)] = s[k * kBlock];
      global = true;
    }
    if (!global) {
      uint16_t* dst = s + cnt * kBlock;
      cnt += n;
      while (hits) {
        const int hb = __clz(hits);
        hits ^= 0x80000000u >> hb;
        *dst = (uint16_t)(p + (uint32_t)hb);
        dst += kBlock;
      }
    } else {
      while (hits) {
        const int hb = __clz(hits);
        hits ^= 0x80000000u >> hb;
        if (cnt < cap) slot(cnt) = (uint16_t)(p + (uint32_t)hb);
        ++cnt;
      }
    }
  }
};

// Writes a list in whole groups of four 16-bit halo positions, an 8-byte store each; the
// last group is completed with the particle's own position.
struct ListWriter {
  uint2* groups;  // this particle's group 0; group g sits 32 uint2 further
  int cap;        // list capacity (a multiple of four)
  uint32_t g0 = 0, g1 = 0;
  __device__ __forceinline__ void add(int k, uint32_t l) {
    const int q = k & 3;
    if (q < 2) g0 = q == 0 ? l : (g0 | (l << 16));
    else g1 = q == 2 ? l : (g1 | (l << 16));
    if (q == 3 && k < cap) groups[(size_t)(k >> 2) * 32] = make_uint2(g0, g1);
  }
  __device__ __forceinline__ void finish(int cnt, uint32_t self) {
    for (int k = cnt; (k & 3) != 0; ++k) add(k, self);
  }
};

// Bank-aware list order: a particle's entries in one queue per halo position
// modulo 8 (a full queue passes its entries on to the next); slot k of lane j
// takes from queue (j + k) mod 8, or the next one that has entries left. A
// 16-byte staged record at halo position l sits in shared-memory bank group
// l mod 8, so the eight lanes of one 16-byte load phase of a neighbor pass
// then mostly hit different groups.
constexpr int kOrderQueue = kListStage / 8;
struct OrderQueues {
  uint16_t* s;                   // shared memory, this thread's entry 0
  uint32_t fill = 0;             // entries per queue, four bits each
  uint32_t cur = 0, avail = 0;   // entries taken per queue; queues with entries left (the mask twice)
  __device__ __forceinline__ void push(uint32_t l) {
    uint32_t q = 4u * (l & 7u), f = (fill >> q) & 15u;
    while (f >= (uint32_t)kOrderQueue) {
      q = (q + 4u) & 31u;
      f = (fill >> q) & 15u;
    }
    fill += 1u << q;
    avail |= 0x101u << (q >> 2);
    s[((q >> 2) * kOrderQueue + f) * kBlock] = (uint16_t)l;
  }
  __device__ __forceinline__ uint32_t pop(uint32_t want) {
    const uint32_t r = (want + (uint32_t)__ffs((int)(avail >> want)) - 1u) & 7u, q = 4u * r;
    const uint32_t c = (cur >> q) & 15u;
    cur += 1u << q;
    if (c + 1u == ((fill >> q) & 15u)) avail &= ~(0x101u << r);
    return s[(r * kOrderQueue + c) * kBlock];
  }
};

// Neighbor search and kernel sum of one block of sorted particles.
//
// Halo: the block's cells are marked, each with its 26 neighbors, in a bitmap
// over their bounding box (rows along x), so the rank of a set bit is the
// cell's place in the halo and the three cells of a stencil row lie side by
// side: a cell's candidates are nine runs of halo positions. A block whose
// Morton keys cross a boundary of 16^3 cells, where the curve jumps, keeps
// one box on either side of it (a cell that both hold is in the halo twice, as is
// one on either end of a box that spans the bucket grid; it only costs room). A block whose boxes or cells are too many (sparse
// particles), or whose halo would outgrow 16-bit positions with such second
// copies, sorts the stencil keys instead and visits 27 buckets per particle.
//
// Candidates: each particle walks its cell's runs in pieces of up to 32
// positions, four at a time, two per packed f32 instruction. A test is
// branch-free: the sign bit of r^2 - h^2 (h^2 widened by the guard band) goes
// into a mask, and the mask's set bits to the particle's list in shared
// memory. A pass over the list sums the kernel; it decides the neighbors
// inside the guard band by the exact f64 predicate, and a particle that loses
// one there takes the pass again. The lists then go out in whole groups of
// four, for the IISPH sweeps (ORDER) in bank-aware order.
//
// A halo beyond the staged positions (a compressed scene; f64 at ordinary densities)
// goes through shared memory in pieces, by the same tests. Its lists are longer than
// the staged ones, so what a mask finds is summed at once and written group by group
// (the sweeps do not stage such halos either, so their order is of no use). 195 thousand
// SESPH particles after 500 steps, 187 to 363 neighbors at most: 273, 371 and 405 us for
// three stiffnesses; 661, 925 and 1052 us when every candidate was fetched through the
// halo's index and its list kept two bytes at a time in global memory, 472, 606 and
// 740 us with the test-and-append loop. f64, three steps of 64 thousand particles in a box:
// 1396 -> 1270 us.
//
// What bounds it: issue (about 216 candidates per particle; 74 % of the issue
// slots used, 211 M warp instructions for one million particles at spacing
// h/2). That scene took 470 us with a test-and-append loop per candidate over
// 27 hashed buckets, and 78 us more in a kernel of its own for the bank-aware
// order; in this form 269 us for both.
template <class R, bool ORDER>
__global__ void __launch_bounds__(kBlock, 4) k_neighbors_density(
    Scalars* sc, const R4<R>* pos, const uint32_t* start,
    R4<R>* xv, uint16_t* nbr, uint32_t* ncnt,
    uint32_t* halo_idx, uint32_t* halo_n, int hcap, int stage, StepParams<R> P) {
  grid_dep_begin();
  extern __shared__ __align__(32) unsigned char dsm[];
  __shared__ int s_own[kSearchCells];        // per cell: own bucket's halo offset - its first particle
  __shared__ uint8_t s_head[kSearchCells];   // per cell: its first thread
  __shared__ uint32_t s_scan[32];
  __shared__ int s_box[2][6];
  __shared__ uint32_t s_ends[2];        // keys of the block's first and last particle
  constexpr uint32_t kStage = (uint32_t)(kSearchX / (3 * sizeof(R)));
  R* s_px = reinterpret_cast<R*>(dsm);
  R* s_py = s_px + kStage;
  R* s_pz = s_py + kStage;
  int3* s_cell = reinterpret_cast<int3*>(dsm + kSearchX + kSearchL) - kBlock;  // the end of region L
  uint16_t* s_list = reinterpret_cast<uint16_t*>(dsm + kSearchX);
  uint32_t* s_row = reinterpret_cast<uint32_t*>(dsm + kSearchX + kSearchL);  // offset | length << 16, nine per cell
  const int tid = threadIdx.x;
  const int i = blockIdx.x * kBlock + tid;
  const bool active = i < sc->n_active;
  R4<R> xi = R4<R>{R(0), R(0), R(0), R(0)};
  uint32_t key = 0;
  int cx = 0, cy = 0, cz = 0;
  if (active) {
    xi = pos[i];
    key = lane_key(xi.w);
    // (the cell modulo the bucket grid, which is all that the stencil's buckets depend on)
    cx = (int)gather3(key);
    cy = (int)gather3(key >> 1);
    cz = (int)gather3(key >> 2);
  }
  s_cell[tid] = make_int3(cx, cy, cz);
  if (tid < 12) s_box[tid / 6][tid % 6] = tid % 6 < 3 ? 0x7fffffff : (int)0x80000000;
  if (tid == 0) s_ends[0] = key;
  if (i == min((int)(blockIdx.x + 1) * kBlock, sc->n_active) - 1) s_ends[1] = key;
  __syncthreads();
  // one head per run of particles in the same cell
  const int3 prev = tid > 0 ? s_cell[tid - 1] : make_int3(0, 0, 0);
  const bool head = active && (tid == 0 || prev.x != cx || prev.y != cy || prev.z != cz);
  const int jump = 31 - __clz((int)((s_ends[0] ^ s_ends[1]) | 1u));  // highest key bit the block's cells differ in
  const bool split = jump >= kBoxLevel;
  const int side = split ? (int)((key >> jump) & 1u) : 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int c = d == 0 ? cx : (d == 1 ? cy : cz);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (e == 1 && !split) break;
      const bool in = active && side == e;
      const int lo = __reduce_min_sync(0xffffffffu, in ? c : 0x7fffffff);
      const int hi = __reduce_max_sync(0xffffffffu, in ? c : (int)0x80000000);
      if ((tid & 31) == 0 && lo <= hi) {
        atomicMin(&s_box[e][d], lo);
        atomicMax(&s_box[e][3 + d], hi);
      }
    }
  }
  uint32_t nheads = 0;
  const uint32_t rank = block_excl_scan_u32(head ? 1u : 0u, s_scan, &nheads);
  const int hr = (int)rank - (head ? 0 : 1);  // this particle's cell
  if (head && rank < (uint32_t)kSearchCells) s_head[rank] = (uint8_t)tid;
  uint32_t* hidx = halo_idx + (size_t)blockIdx.x * (size_t)hcap;
  uint32_t H = 0;
  bool miss = false;
  int own_local = 0;
  uint32_t span[27];  // general path: the particle's buckets as offset | length << 16
  // the cells of each side and their neighbors as a box of nx x ny x nz cells,
  // the second box's bits behind the first's
  int nx[2] = {0, 0}, ny[2] = {0, 0}, bits[2] = {0, 0};
  bool boxed = nheads > 0 && nheads <= (uint32_t)kSearchCells;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if (s_box[e][0] > s_box[e][3]) continue;  // no cells on this side
    const long long bx = (long long)s_box[e][3] - s_box[e][0] + 3, by = (long long)s_box[e][4] - s_box[e][1] + 3,
                    bz = (long long)s_box[e][5] - s_box[e][2] + 3;
    boxed = boxed && bx <= kBoxCells && by <= kBoxCells && bz <= kBoxCells && bx * by <= kBoxCells &&
            bx * by * bz <= kBoxCells;
    if (!boxed) break;
    nx[e] = (int)bx; ny[e] = (int)by; bits[e] = (int)(bx * by * bz);
  }
  const int second = (bits[0] + 31) & ~31, nbits = bits[1] ? second + bits[1] : bits[0];
  boxed = boxed && nbits <= kBoxCells;
  if (boxed) {
    uint32_t* s_bits = reinterpret_cast<uint32_t*>(dsm + kSearchX);
    uint32_t* s_first = s_bits + kBoxCells / 32;                            // per halo cell: its bucket's first particle
    uint16_t* s_off = reinterpret_cast<uint16_t*>(s_first + kHaloCells);    // per halo cell: length, then halo offset
    uint16_t* s_pre = s_off + kHaloCells + 2;                               // set bits before each word
    const int nw = (nbits + 31) >> 5;
    for (int t = tid; t < nw; t += kBlock) s_bits[t] = 0u;
    __syncthreads();
    // bit of the cell at (-1, dy, dz) of the stencil around cell c of side e
    auto bit_of = [&](const int3& c, int e, int dy, int dz) {
      return (e ? second : 0) + ((c.z - s_box[e][2] + 1 + dz) * (e ? ny[1] : ny[0]) + (c.y - s_box[e][1] + 1 + dy)) *
                                    (e ? nx[1] : nx[0]) + (c.x - s_box[e][0]);
    };
    if (head) {
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const int b = bit_of(make_int3(cx, cy, cz), side, q % 3 - 1, q / 3 - 1), w = b >> 5, sh = b & 31;
        atomicOr(&s_bits[w], 7u << sh);
        if (sh > 29) atomicOr(&s_bits[w + 1], 7u >> (32 - sh));
      }
    }
    __syncthreads();
    uint32_t c0 = 0, c1 = 0, D = 0;
    if (2 * tid < nw) c0 = __popc(s_bits[2 * tid]);
    if (2 * tid + 1 < nw) c1 = __popc(s_bits[2 * tid + 1]);
    const uint32_t before = block_excl_scan_u32(c0 + c1, s_scan, &D);
    if (2 * tid < nw) s_pre[2 * tid] = (uint16_t)before;
    if (2 * tid + 1 < nw) s_pre[2 * tid + 1] = (uint16_t)(before + c0);
    __syncthreads();
    if (D > (uint32_t)kHaloCells) {
      boxed = false;
    } else {
      auto cell_rank = [&](int b) { return (int)s_pre[b >> 5] + __popc(s_bits[b >> 5] & ((1u << (b & 31)) - 1u)); };
      for (int b = tid; b < nbits; b += kBlock) {
        if (!((s_bits[b >> 5] >> (b & 31)) & 1u)) continue;
        const int r = cell_rank(b);
        const int e = bits[1] && b >= second ? 1 : 0;
        const int lx = e ? nx[1] : nx[0], lxy = lx * (e ? ny[1] : ny[0]), lb = e ? b - second : b;
        const int z = lb / lxy, y = (lb - z * lxy) / lx, x = lb - z * lxy - y * lx;
        const uint32_t k = morton_key(x + s_box[e][0] - 1, y + s_box[e][1] - 1, z + s_box[e][2] - 1, P.mask);
        const uint32_t f = start[k], len = start[k + 1] - f;
        miss |= len > 0xffffu;
        s_first[r] = f;
        s_off[r] = (uint16_t)min(len, 65535u);
      }
      __syncthreads();
      for (uint32_t r0 = 0; r0 < D; r0 += kBlock) {  // lengths to offsets
        const uint32_t r = r0 + tid;
        uint32_t total = 0;
        const uint32_t o = H + block_excl_scan_u32(r < D ? (uint32_t)s_off[r] : 0u, s_scan, &total);
        if (r < D) s_off[r] = (uint16_t)min(o, 65535u);
        H += total;
      }
      if (tid == 0) s_off[D] = (uint16_t)min(H, 65535u);
      // (buckets that are in it twice may take a halo over the 65535 positions that lists can
      // address: without the second copies it may fit)
      if (H > 65535u) boxed = false;
      __syncthreads();
      if (boxed) {
        // the halo's particle indices, and its positions where they fit: eight lanes per cell
        for (uint32_t r = tid >> 3; r < D; r += kBlock / 8) {
          const uint32_t o = s_off[r], e = s_off[r + 1], f = s_first[r];
          for (uint32_t l = o + (tid & 7); l < e; l += 8) {
            if (l < (uint32_t)hcap) hidx[l] = f + (l - o);
            if (l < kStage) {
              const R4<R>* p = &pos[f + (l - o)];
              async_copy(&s_px[l], &p->x);
              async_copy(&s_py[l], &p->y);
              async_copy(&s_pz[l], &p->z);
            }
          }
        }
        for (int e = tid; e < 9 * (int)nheads; e += kBlock) {
          const int h = e / 9, q = e - 9 * h;
          const int3 c = s_cell[s_head[h]];
          const int e1 = split ? (int)((morton_key(c.x, c.y, c.z, P.mask) >> jump) & 1u) : 0;
          const int r = cell_rank(bit_of(c, e1, q % 3 - 1, q / 3 - 1));
          const uint32_t o = s_off[r];
          s_row[e] = o | ((uint32_t)(s_off[r + 3] - o) << 16);
          if (q == 4) s_own[h] = (int)s_off[r + 1] - (int)s_first[r + 1];
        }
        stage_done();  // the construction buffers become the lists
        if (active) own_local = s_own[hr] + i;
      }
    }
  }
  if (!boxed) {
    // general path: bitonic-sorted stencil keys, halo offsets in key order,
    // per-particle lookups by binary search
    const int nk = 27 * (int)nheads;
    uint32_t* skey = reinterpret_cast<uint32_t*>(dsm);                 // sorted stencil keys
    uint16_t* soff = reinterpret_cast<uint16_t*>(skey + kHaloKeys);    // halo offset of each first key
    int S = 32;
    while (S < nk) S <<= 1;
    __syncthreads();
    if (head) {
      uint32_t keys[27];
      stencil_keys(cx, cy, cz, P.mask, keys);
#pragma unroll
      for (int q = 0; q < 27; ++q) skey[27 * rank + q] = keys[q];
    }
    for (int t = nk + tid; t < S; t += kBlock) skey[t] = kNoKey;
    __syncthreads();
    for (int k = 2; k <= S; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int t = tid; t < (S >> 1); t += kBlock) {
          const int a = 2 * t - (t & (j - 1)), b = a + j;
          const uint32_t ka = skey[a], kb = skey[b];
          if ((ka > kb) == ((a & k) == 0)) {
            skey[a] = kb;
            skey[b] = ka;
          }
        }
        __syncthreads();
      }
    const int per = S >= kBlock ? S / kBlock : 1;
    const int p0 = tid * per;
    uint32_t len = 0;
    for (int q = 0; q < per; ++q) {
      const int p = p0 + q;
      if (p >= S) break;
      const uint32_t k = skey[p];
      if (k != kNoKey && (p == 0 || skey[p - 1] != k)) len += start[k + 1] - start[k];
    }
    uint32_t run = block_excl_scan_u32(len, s_scan, &H);
    for (int q = 0; q < per; ++q) {
      const int p = p0 + q;
      if (p >= S) break;
      const uint32_t k = skey[p];
      if (k != kNoKey && (p == 0 || skey[p - 1] != k)) {
        const uint32_t b = start[k], e = start[k + 1];
        soff[p] = (uint16_t)min(run, 65535u);
        for (uint32_t j = b; j < e; ++j)
          if (run + (j - b) < (uint32_t)hcap) hidx[run + (j - b)] = j;
        run += e - b;
      }
    }
    __syncthreads();
    if (active) {
      uint32_t keys[27];
      stencil_keys(cx, cy, cz, P.mask, keys);
      const uint32_t own = morton_key(cx, cy, cz, P.mask);
#pragma unroll 1
      for (int q = 0; q < 27; ++q) {
        const uint32_t k = keys[q];
        int lo = 0, hi = S;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (skey[mid] < k) lo = mid + 1;
          else hi = mid;
        }
        const bool found = lo < S && skey[lo] == k;
        const uint32_t b = start[k], len2 = start[k + 1] - b;
        miss |= !found || len2 > 0xffffu;
        const uint32_t off = found ? (uint32_t)soff[lo] : 0u;
        span[q] = off | (found && len2 <= 0xffffu ? len2 << 16 : 0u);
        if (k == own) own_local = (int)off - (int)b + i;
      }
    }
    __syncthreads();  // spans, offsets and halo_idx are complete; the sort buffers are free
    if (H <= kStage && H <= (uint32_t)hcap)
      for (uint32_t l = tid; l < H; l += kBlock) {
        const R4<R> p = pos[hidx[l]];
        s_px[l] = p.x;
        s_py[l] = p.y;
        s_pz[l] = p.z;
      }
    __syncthreads();
  }
  if (tid == 0) {
    halo_n[blockIdx.x] = H;
    atomicMax(&sc->max_halo, (int)min(H, 0x7fffffffu));
    if (H > (uint32_t)stage) atomicAdd(&sc->n_wide, 1);
  }
  const uint32_t usable = min(H, (uint32_t)hcap);
  const bool staged = H <= usable && H <= kStage;
  FoundList found;
  const uint32_t pad = (uint32_t)own_local < usable ? (uint32_t)own_local : 0u;  // the unused slots of a list's last group
  found.s = s_list + tid;
  found.list = nbr + (active ? nbr_slot(i, 0, P.K) : 0);
  found.cap = P.K;
  const RangeTest<R> range(xi, P.range2_out);
  if (active && miss) atomicMax(&sc->max_halo, 0x7fffffff);  // a bucket beyond 65535 particles
  // Candidates of the particle among the staged positions [base, base + count) of the halo:
  // use(hits, p) with candidate p + c of those positions at bit 31 - c of hits.
  auto visit = [&](uint32_t base, uint32_t count, auto&& use) {
    auto test_run = [&](uint32_t row) {
      const uint32_t first = row & 0xffffu, last = first + (row >> 16);
      if (last <= base || first >= base + count) return;
      const uint32_t o = max(first, base) - base, end = min(last - base, count);
      for (uint32_t p = o & ~3u; p < end; p += 32) {
        const int n = min(32, (int)((end - p + 3u) & ~3u));
        uint32_t hits = range.run(s_px + p, s_py + p, s_pz + p, n) << (32 - n);
        if (p < o) hits &= 0xffffffffu >> (o - p);
        if (end - p < 32u) hits &= ~(0xffffffffu >> (end - p));
        const uint32_t self = (uint32_t)own_local - base - p;
        if (self < 32u) hits &= ~(0x80000000u >> self);
        use(hits, p);
      }
    };
    if (boxed) {
      const uint32_t* row = s_row + 9 * hr;
#pragma unroll 1
      for (int q = 0; q < 9; ++q) test_run(row[q]);
    } else {
#pragma unroll 1
      for (int q = 0; q < 27; ++q) test_run(span[q]);
    }
  };
  if (!staged) {
    // A larger halo goes through shared memory in pieces. What a particle finds in a mask of
    // candidates is summed at once, and its list goes out group by group.
    KernelSum<R> acc(xi, P.k);
    ListWriter list;
    list.groups = reinterpret_cast<uint2*>(found.list);
    list.cap = P.K;
    for (uint32_t base = 0; base < usable; base += kStage) {
      const uint32_t count = min(kStage, usable - base);
      if (base > 0 || !boxed) {  // (the first piece is there where the halo was built from boxes)
        __syncthreads();
        for (uint32_t l = tid; l < count; l += kBlock) {
          const R4<R>* p = &pos[hidx[base + l]];
          async_copy(&s_px[l], &p->x);
          async_copy(&s_py[l], &p->y);
          async_copy(&s_pz[l], &p->z);
        }
        stage_done();
      }
      if (active)
        visit(base, count, [&](uint32_t hits, uint32_t p) {
          auto position = [&](uint32_t l) { return R4<R>{s_px[l], s_py[l], s_pz[l], R(0)}; };
          for (;;) {
            KernelSum<R> next = acc;
            next.farthest = R(0);
            for (uint32_t left = hits; left;) {
              R4<R> xj[4];
              const int n = min(__popc(left), 4);
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int hb = left ? __clz(left) : 0;  // (beyond the last: any position)
                left &= ~(0x80000000u >> hb);
                xj[u] = position(p + (uint32_t)hb);
              }
              next.add(xj, n);
            }
            if (next.farthest >= P.range2_lo) {  // some lie inside the guard band
              uint32_t keep = 0;
              for (uint32_t left = hits; left;) {
                const int hb = __clz(left);
                left ^= 0x80000000u >> hb;
                if (in_range(xi, position(p + (uint32_t)hb), P.range, P.range2_lo, P.range2_hi)) keep |= 0x80000000u >> hb;
              }
              if (keep != hits) {
                hits = keep;
                continue;
              }
            }
            acc = next;
            break;
          }
          while (hits) {
            const int hb = __clz(hits);
            hits ^= 0x80000000u >> hb;
            list.add(found.cnt++, base + p + (uint32_t)hb);
          }
        });
    }
    if (active) {
      list.finish(found.cnt, pad);
      xv[i] = R4<R>{xi.x, xi.y, xi.z, acc.s};  // (k_volume puts the volume in its place)
      ncnt[i] = (uint32_t)found.cnt;
    }
  } else if (active) {
    visit(0, H, [&](uint32_t hits, uint32_t p) { found.add(hits, p); });
    auto position = [&](uint32_t l) { return R4<R>{s_px[l], s_py[l], s_pz[l], R(0)}; };
    // the kernel sum in list order
    R sum;
    for (;;) {
      const int stored = min(found.cnt, P.K);
      KernelSum<R> acc(xi, P.k);
      if (!found.global) {
        const uint16_t* e = found.s;
        int k = stored;
        for (; k >= 4; k -= 4, e += 4 * kBlock) {
          R4<R> xj[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t l = e[u * kBlock];
            xj[u] = R4<R>{s_px[l], s_py[l], s_pz[l], R(0)};
          }
          acc.add(xj, 4);
        }
        if (k > 0) {
          R4<R> xj[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t l = e[min(u, k - 1) * kBlock];
            xj[u] = R4<R>{s_px[l], s_py[l], s_pz[l], R(0)};
          }
          acc.add(xj, k);
        }
      } else {
        for (int k = 0; k < stored; ++k) {
          const R4<R> xj[4] = {position((uint32_t)found.slot(k))};
          acc.add(xj, 1);
        }
      }
      sum = acc.s;
      // (a list that is cut off at the capacity keeps its count, so that the update is redone with a larger one)
      if (!(acc.farthest >= P.range2_lo) || found.cnt > P.K) break;
      // some neighbor lies inside the guard band: keep those the exact predicate keeps
      int kept = 0;
      for (int k = 0; k < stored; ++k) {
        const uint32_t l = found.slot(k);
        if (in_range(xi, position(l), P.range, P.range2_lo, P.range2_hi)) found.slot(kept++) = (uint16_t)l;
      }
      if (kept == stored) break;  // all of them
      found.cnt -= stored - kept;
    }
    xv[i] = R4<R>{xi.x, xi.y, xi.z, sum};  // (k_volume puts the volume in its place)
    ncnt[i] = (uint32_t)found.cnt;
  }
  // The lists in whole groups of four. The unused slots of the last group hold
  // the particle's own halo position: the passes over neighbors read whole
  // groups, and the self pair adds zero.
  if (ORDER) __syncthreads();  // the queues take the place of the positions
  if (active && staged) {
    const int stored = min(found.cnt, P.K);
    uint2* groups = reinterpret_cast<uint2*>(found.list);
    OrderQueues queue;
    queue.s = reinterpret_cast<uint16_t*>(dsm) + tid;
    if (ORDER && !found.global)
      for (int k = 0; k < stored; ++k) queue.push(found.s[k * kBlock]);
    for (int k0 = 0; k0 < stored; k0 += 4) {
      uint32_t l[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        l[u] = k0 + u >= stored ? pad
               : ORDER && !found.global ? queue.pop((uint32_t)(i + k0 + u) & 7u)
                                        : (uint32_t)found.slot(k0 + u);
      groups[(size_t)(k0 >> 2) * 32] = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
    }
  }
  int cnt = found.cnt;
  // block max of the neighbor count
  for (int o = 16; o > 0; o >>= 1) cnt = max(cnt, __shfl_down_sync(0xffffffffu, cnt, o));
  if ((threadIdx.x & 31) == 0 && cnt > 0) atomicMax(&sc->max_nbrs, cnt);
}

// ---------------------------------------------------------------------------
// 5. boundary samples: sample boundaries (sorted sample grid) and volume maps
// ---------------------------------------------------------------------------
// Serendipity reference nodes (discretization.rs:267-300): lattice offsets in
// the reference's order.
__constant__ int c_ser_off[32][3];

// f64 arithmetic that the compiler may not contract into FMAs, so that the
// field evaluation rounds exactly like the reference's (discretization.rs:
// 437-557 is plain f64 without fused operations): threshold decisions such
// as sd < r, sd <= -r or 0.5 < |grad| < 2 then fall on the same side.
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double div_(double a, double b) { return __ddiv_rn(a, b); }

// The 32 nodes in the reference's order (discretization.rs:267-300): 8 corners,
// 8 nodes each on the edges along x, y and z. The partial products that nodes
// share are formed once, in the reference's order of multiplication, so every
// term keeps its bits. The nodes of a group are loaded together.
__device__ __forceinline__ bool ser_eval(const DevField& F, double px, double py, double pz, double& out) {
  const double p[3] = {px, py, pz};
  long long c[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double fi = floor(div_(sub_(p[d], F.xmin[d]), F.dx));
    if (p[d] < F.xmin[d] || p[d] > F.xmax[d]) return false;
    const long long idx = (long long)fi;
    c[d] = idx < (long long)F.n[d] - 1 ? idx : (long long)F.n[d] - 1;
  }
  const double xi = sub_(div_(mul_(2.0, sub_(p[0], add_(F.xmin[0], mul_((double)c[0], F.dx)))), F.dx), 1.0);
  const double eta = sub_(div_(mul_(2.0, sub_(p[1], add_(F.xmin[1], mul_((double)c[1], F.dx)))), F.dx), 1.0);
  const double zeta = sub_(div_(mul_(2.0, sub_(p[2], add_(F.xmin[2], mul_((double)c[2], F.dx)))), F.dx), 1.0);
  const long long ny = F.NX, nz = F.NX * F.NY;  // one step along y and z
  const double* base = F.nodes + ((3 * c[2] * F.NY + 3 * c[1]) * F.NX + 3 * c[0]);
  const double lx[2] = {sub_(1.0, xi), add_(1.0, xi)};
  const double ly[2] = {sub_(1.0, eta), add_(1.0, eta)};
  const double lz[2] = {sub_(1.0, zeta), add_(1.0, zeta)};
  const double third = 1.0 / 3.0;
  double s = 0.0;
  double v[8], w[4];
  auto load = [&](auto offset) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __ldg(base + offset(k));
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 8; ++k) ok = ok && v[k] == v[k];
    return ok;  // no pruned node
  };
  // corners: (1/64)(1+xi a)(1+eta b)(1+zeta c)(9 r^2 - 19)
  if (!load([&](int k) { return 3 * (k & 1) + 3 * ((k >> 1) & 1) * ny + 3 * (k >> 2) * nz; })) return false;
  const double e19 = sub_(mul_(9.0, add_(add_(mul_(xi, xi), mul_(eta, eta)), mul_(zeta, zeta))), 19.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = mul_(mul_(1.0 / 64.0, lx[k & 1]), ly[k >> 1]);
#pragma unroll
  for (int k = 0; k < 8; ++k) s = add_(s, mul_(v[k], mul_(mul_(w[k & 3], lz[k >> 2]), e19)));
  // edges along x: (9/64)(1-xi^2)(1+9 xi a)(1+eta b)(1+zeta c), a = -1/3, 1/3
  auto along = [&](double u, double e[2]) {
    const double f = mul_(9.0 / 64.0, sub_(1.0, mul_(u, u))), g = mul_(mul_(9.0, u), third);
    e[0] = mul_(f, sub_(1.0, g));
    e[1] = mul_(f, add_(1.0, g));
  };
  double e[2];
  if (!load([&](int k) { return 1 + (k & 1) + 3 * ((k >> 1) & 1) * ny + 3 * (k >> 2) * nz; })) return false;
  along(xi, e);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = mul_(e[k & 1], ly[k >> 1]);
#pragma unroll
  for (int k = 0; k < 8; ++k) s = add_(s, mul_(v[k], mul_(w[k & 3], lz[k >> 2])));
  // along y: z outer, x, then the node on the edge
  if (!load([&](int k) { return (1 + (k & 1)) * ny + 3 * ((k >> 1) & 1) + 3 * (k >> 2) * nz; })) return false;
  along(eta, e);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = mul_(e[k & 1], lx[k >> 1]);
#pragma unroll
  for (int k = 0; k < 8; ++k) s = add_(s, mul_(v[k], mul_(w[k & 3], lz[k >> 2])));
  // along z: y outer, x, then the node on the edge
  if (!load([&](int k) { return (1 + (k & 1)) * nz + 3 * ((k >> 1) & 1) + 3 * (k >> 2) * ny; })) return false;
  along(zeta, e);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = mul_(e[k & 1], lx[k >> 1]);
#pragma unroll
  for (int k = 0; k < 8; ++k) s = add_(s, mul_(v[k], mul_(w[k & 3], ly[k >> 2])));
  out = s;
  return true;
}
__device__ __noinline__ bool ser_function(const DevField& F, double px, double py, double pz, double& out) {
  return ser_eval(F, px, py, pz, out);
}

__device__ bool ser_gradient(const DevField& F, double px, double py, double pz, double g[3]) {
  const double h = div_(F.dx, 6.0);
  const double h2 = mul_(2.0, h);
  double fp, fm;
  if (!ser_function(F, add_(px, h), py, pz, fp) || !ser_function(F, sub_(px, h), py, pz, fm)) return false;
  g[0] = div_(sub_(fp, fm), h2);
  if (!ser_function(F, px, add_(py, h), pz, fp) || !ser_function(F, px, sub_(py, h), pz, fm)) return false;
  g[1] = div_(sub_(fp, fm), h2);
  if (!ser_function(F, px, py, add_(pz, h), fp) || !ser_function(F, px, py, sub_(pz, h), fm)) return false;
  g[2] = div_(sub_(fp, fm), h2);
  return true;
}

// One volume-map boundary sample per (particle, boundary): x_b = x - n d with
// vol = min(VM, 4/3 pi r^3); stored as vmx = {x_b, vol}, vmv = {v_b, kind}
// where kind 0 = none, 1 = tangent helper x-axis, 2 = helper y-axis.
// Volume-map samples in two kernels: k_vm_near evaluates every particle's
// signed distance (the cheap, light first test of find_boundary_samples) and
// lists the particles within the support radius of some boundary, writing
// the empty result for all others; k_vm_sample then does the full sampling
// for the listed particles only, eight lanes each, which evaluate the eight
// field values of a sample at once (one lane after the other took 77-87 us per
// update for scenes of 133 thousand to one million particles, 15-56 us now; both
// passes are bound by f64 issue and the latency of the node loads).
template <class R>
__global__ void __launch_bounds__(kBlock) k_vm_near(
    Scalars* sc, const R4<R>* pos, const VMDesc* vms, int nvm,
    const Body* bodies, uint32_t* near_list, R4<R>* vmx,
    R4<R>* vmv, R* bW, R4<R>* bG, R4<R>* bGu,
    R4<R>* bA, StepParams<R> P) {
  grid_dep_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= sc->n_active) return;
  const R4<R> xr = pos[i];
  const double p[3] = {(double)xr.x, (double)xr.y, (double)xr.z};
  bool near = false;
  for (int b = 0; b < nvm && !near; ++b) {
    const VMDesc& D = vms[b];
    double pl[3] = {p[0], p[1], p[2]};
    if (D.body >= 0) body_world_to_local(bodies[D.body], p, pl);
    double sd;
    near = ser_eval(D.sdf, pl[0], pl[1], pl[2], sd) && sd < P.range;
  }
  if (near) {
    near_list[atomicAdd(&sc->vm_near, 1u)] = (uint32_t)i;
    return;
  }
  for (int b = 0; b < nvm; ++b) vmv[(size_t)b * P.Np + i] = R4<R>{R(0), R(0), R(0), R(0)};  // kind 0: vmx is not read
  bW[i] = R(0);
  bG[i] = R4<R>{R(0), R(0), R(0), R(0)};
  if (bGu) bGu[i] = R4<R>{R(0), R(0), R(0), R(0)};
  bA[i] = R4<R>{R(0), R(0), R(0), R(0)};
}

// Normal-mode sample of volume map D for the world-frame point p
// (volume_map_boundary.rs:1287-1330): the signed distance (in the body frame
// for a dynamic map) must be below the search range, the gradient norm inside
// (0.5, 2) and the volume-map value positive (then clamped to the volume of
// the support ball); the sample sits at max(sd + spacing/4, spacing) against
// the normalized gradient, moving with the body's velocity there. Returns
// false, leaving the outputs untouched, when the point has no sample.
// vm_sample_from takes the field values: the signed distance, its gradient in
// the body frame, and the volume map.
__device__ __forceinline__ bool vm_sample_from(double sd, const double gl[3], double vm, const Body* body,
                                               const double p[3], double ball, double spacing, double xb[3],
                                               double vb[3], double& vol) {
  double g[3] = {gl[0], gl[1], gl[2]};
  if (body) qrot(body->q, gl, g);
  const double gn = __dsqrt_rn(add_(add_(mul_(g[0], g[0]), mul_(g[1], g[1])), mul_(g[2], g[2])));
  if (!(gn > 0.5 && gn < 2.0) || !(vm > 0.0)) return false;
  vol = vm < ball ? vm : ball;
  const double d = fmax(add_(sd, mul_(0.25, spacing)), spacing);
  for (int c = 0; c < 3; ++c) xb[c] = sub_(p[c], mul_(div_(g[c], gn), d));
  if (body) body_velocity_at(*body, xb, vb);
  return true;
}
__device__ __forceinline__ bool vm_normal_sample(const VMDesc& D, const Body* body, const double p[3],
                                                 double range, double ball, double spacing,
                                                 double xb[3], double vb[3], double& vol) {
  double pl[3] = {p[0], p[1], p[2]};
  if (body) body_world_to_local(*body, p, pl);
  double sd, g[3], vm;
  if (!ser_function(D.sdf, pl[0], pl[1], pl[2], sd) || !(sd < range)) return false;
  if (!ser_gradient(D.sdf, pl[0], pl[1], pl[2], g)) return false;
  if (!ser_function(D.vm, pl[0], pl[1], pl[2], vm)) return false;
  return vm_sample_from(sd, g, vm, body, p, ball, spacing, xb, vb, vol);
}

// The four tangential viscosity samples of a volume-map sample x_b of particle
// position xi: x_b +- r/2 t1, x_b +- r/2 t2 (volume_map_boundary.rs:1344-1377);
// kind as in vmv.w.
template <class R>
struct TangentSamples {
  V3<R> xb, d1, d2;
  __device__ __forceinline__ TangentSamples(const R4<R>& xi, const R4<R>& x, R kind, double range)
      : xb{x.x, x.y, x.z} {
    const V3<R> u = xb - V3<R>{xi.x, xi.y, xi.z};
    const V3<R> tmp = kind == R(1) ? V3<R>{1, 0, 0} : V3<R>{0, 1, 0};
    V3<R> t1 = cross(u, tmp);
    V3<R> t2 = cross(u, t1);
    t1 = (R(1) / sqrt(dot(t1, t1))) * t1;
    t2 = (R(1) / sqrt(dot(t2, t2))) * t2;
    const R d = R(0.5) * (R)range;
    d1 = d * t1;
    d2 = d * t2;
  }
  __device__ __forceinline__ V3<R> at(int k) const {
    return k == 0 ? xb + d1 : k == 1 ? xb - d1 : k == 2 ? xb + d2 : xb - d2;
  }
};
template <class R>
__device__ __forceinline__ V3<R> body_velocity_r(const Body* bodies, int body, const V3<R>& q) {
  if (body < 0) return V3<R>{0, 0, 0};
  const double p[3] = {(double)q.x, (double)q.y, (double)q.z};
  double v[3];
  body_velocity_at(bodies[body], p, v);
  return V3<R>{(R)v[0], (R)v[1], (R)v[2]};
}
// Boundary viscosity acceleration from one sample: its factor along r = xi - x.
template <class R>
__device__ __forceinline__ R boundary_viscosity(const V3<R>& r, const V3<R>& dv, R V, const StepParams<R>& P) {
  const R r2 = r.x * r.x + r.y * r.y + r.z * r.z;
  const R f = kernel_grad_factor(r2, P.k);
  const R vr = dv.x * r.x + dv.y * r.y + dv.z * r.z;
  return P.visc_b * V * vr / (r2 + P.eps_visc) * f;
}

template <class R>
__global__ void __launch_bounds__(kBlock, 3) k_vm_sample(
    Scalars* sc, const uint32_t* near_list, const R4<R>* pos,
    const R4<R>* vel, const VMDesc* vms, int nvm, const Body* bodies,
    R4<R>* vmx, R4<R>* vmv, R* bW, R4<R>* bG,
    R4<R>* bGu, R4<R>* bA, uint32_t* touch, StepParams<R> P) {
  grid_dep_begin();
  const int lane = threadIdx.x & 31, e = lane & 7;
  const unsigned group = 0xffu << (lane & ~7);
  const int t = (blockIdx.x * kBlock + threadIdx.x) >> 3;
  if (t >= (int)sc->vm_near) return;  // (a group of eight lanes stays together)
  const int i = (int)near_list[t];
  const R4<R> xr = pos[i], vi = vel[i];
  bool dyn = false;
  R sx = 0, sy = 0, sz = 0;  // viscosity
  const double p[3] = {(double)xr.x, (double)xr.y, (double)xr.z};
  const double range = P.range;
  const double ball = 4.0 / 3.0 * 3.14159265358979323846 * (range * range * range);
  R w = 0, gx = 0, gy = 0, gz = 0, gv = 0, ux = 0, uy = 0, uz = 0;
  for (int b = 0; b < nvm; ++b) {
    const VMDesc& D = vms[b];
    const Body* body = D.body >= 0 ? &bodies[D.body] : nullptr;
    int kind = 0;
    double xb[3] = {0, 0, 0}, vb[3] = {0, 0, 0}, vol = 0;
    double pl[3] = {p[0], p[1], p[2]};
    if (body) body_world_to_local(*body, p, pl);
    // lanes 0 to 5: the distance half a node step to either side along x, y
    // and z (ser_gradient); lane 6: the distance; lane 7: the volume map
    const double step = div_(D.sdf.dx, 6.0);
    const double off = e & 1 ? -step : step;
    double q[3] = {pl[0], pl[1], pl[2]};
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (e >> 1 == d) q[d] = add_(q[d], off);
    double f = 0.0;
    const bool ok = ser_eval(e == 7 ? D.vm : D.sdf, q[0], q[1], q[2], f);
    const bool all = __all_sync(group, ok);
    const double sd = __shfl_sync(group, f, 6, 8), vm = __shfl_sync(group, f, 7, 8);
    double g[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
      g[d] = div_(sub_(__shfl_sync(group, f, 2 * d, 8), __shfl_sync(group, f, 2 * d + 1, 8)), mul_(2.0, step));
    if (all && sd < range && vm_sample_from(sd, g, vm, body, p, ball, P.spacing, xb, vb, vol)) {
      const double u[3] = {xb[0] - p[0], xb[1] - p[1], xb[2] - p[2]};
      const double un = sqrt((u[0] * u[0] + u[1] * u[1]) + u[2] * u[2]);
      kind = fabs(u[0] / un) > 0.9 ? 2 : 1;
      // aggregates in f64 from the exact sample position
      const double rx = p[0] - xb[0], ry = p[1] - xb[1], rz = p[2] - xb[2];
      const double r2 = (rx * rx + ry * ry) + rz * rz;
      const double rn = sqrt(r2), q = rn / range;
      const double a1 = q < 1.0 ? 1.0 - q : 0.0, a2 = q < 0.5 ? 0.5 - q : 0.0;
      const double alpha = 16.0 / 3.14159265358979323846;
      const double kw = alpha / (range * range * range) * (a1 * a1 * a1 - 4.0 * (a2 * a2 * a2));
      const double f = rn > 0.0 ? alpha / (range * range * range * range) *
                                      (-3.0 * a1 * a1 + 12.0 * a2 * a2) / rn
                                : 0.0;
      w += (R)(vol * kw);
      const double vf = vol * f;
      gx += (R)(vf * rx); gy += (R)(vf * ry); gz += (R)(vf * rz);
      gv += (R)(vf * (vb[0] * rx + vb[1] * ry + vb[2] * rz));
      ux += (R)(f * rx); uy += (R)(f * ry); uz += (R)(f * rz);
    }
    const size_t o = (size_t)b * P.Np + i;
    const R4<R> xx{(R)xb[0], (R)xb[1], (R)xb[2], (R)vol};
    if (e == 0) {
      vmx[o] = xx;
      vmv[o] = R4<R>{(R)vb[0], (R)vb[1], (R)vb[2], (R)kind};
    }
    if (kind == 0) continue;
    // viscosity: four tangential samples of a quarter of the volume each, one per lane
    const TangentSamples<R> ts(xr, xx, (R)kind, range);
    dyn |= D.body >= 0 && bodies[D.body].dynamic;
    const V3<R> qt = ts.at(e & 3);
    const V3<R> vq = body_velocity_r(bodies, D.body, qt);
    const V3<R> r{xr.x - qt.x, xr.y - qt.y, xr.z - qt.z};
    const R c = boundary_viscosity(r, V3<R>{vi.x - vq.x, vi.y - vq.y, vi.z - vq.z}, R(0.25) * xx.w, P);
    const R tx = c * r.x, ty = c * r.y, tz = c * r.z;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sx += __shfl_sync(group, tx, k, 8);
      sy += __shfl_sync(group, ty, k, 8);
      sz += __shfl_sync(group, tz, k, 8);
    }
  }
  if (e != 0) return;
  bW[i] = w;
  bG[i] = R4<R>{gx, gy, gz, gv};
  if (bGu) bGu[i] = R4<R>{ux, uy, uz, R(0)};
  bA[i] = R4<R>{sx, sy, sz, R(0)};
  if (dyn) touch[atomicAdd(&sc->n_touch, 1u)] = (uint32_t)i;
}

// Visits the particles within h of p (f64, the reference's exact predicate) in
// bucket order: use(j, x, r2) with the sorted index, the record and the squared
// distance. An f32 distance test with a margin for the rounding of both
// positions and of the test itself first puts the candidates that may be in
// range (a sixth of about 216) on a list in shared memory, so the f64 work runs
// on those only, all lanes at once. (Lists of 24 to 40 entries measured alike. In a
// compressed fluid of 60 candidates a cell, where a list fills several times, a plane of
// 512 x 512 points takes 1396 us; 5987 us when each lane worked its own list off, 1877 us
// with the f64 test for every candidate.) (f64 positions are rounded to f32 for it.)
constexpr int kNearList = 32;  // entries per thread: kNearList * kBlock words of shared memory
template <class R, class Use>
__device__ __forceinline__ void for_each_within(const double p[3], double h, uint32_t mask,
                                                const uint32_t* __restrict__ start, const R4<R>* __restrict__ x,
                                                uint32_t* s_list, Use&& use) {
  const int cx = cell_coord(p[0], h), cy = cell_coord(p[1], h), cz = cell_coord(p[2], h);
  const float fx = (float)p[0], fy = (float)p[1], fz = (float)p[2];
  const float m = (float)h * 1.00001f + 4e-7f * (fabsf(fx) + fabsf(fy) + fabsf(fz) + (float)h);
  const float limit = m * m * 1.00001f;
  const double h2 = h * h, lo = h2 * (1.0 - 1e-14), hi = h2 * (1.0 + 1e-14);
  uint32_t* list = s_list + threadIdx.x;
  int cnt = 0;
  auto drain = [&]() {
    for (int k = 0; k < cnt; ++k) {
      const uint32_t j = list[k * kBlock];
      const R4<R> xj = x[j];
      const double qx = (double)xj.x, qy = (double)xj.y, qz = (double)xj.z;
      const double rx = p[0] - qx, ry = p[1] - qy, rz = p[2] - qz;
      const double r2 = (rx * rx + ry * ry) + rz * rz;
      if (r2 < lo || (!(r2 > hi) && in_range_exact(p[0], p[1], p[2], qx, qy, qz, h))) use(j, xj, r2);
    }
    cnt = 0;
  };
  // The lanes take four candidates at a time together, and when one's list is nearly full
  // all work theirs off: lanes that each did so on their own took turns.
  const unsigned lanes = __activemask();
  const uint32_t x0 = morton_key(cx - 1, 0, 0, mask), x1 = morton_key(cx, 0, 0, mask), x2 = morton_key(cx + 1, 0, 0, mask);
  uint32_t yz = 0;
#pragma unroll 1
  for (int q = 0; q < 27; ++q) {
    if (q % 3 == 0) yz = morton_key(0, cy + (q / 3) % 3 - 1, cz + q / 9 - 1, mask);
    const uint32_t k = yz | (q % 3 == 0 ? x0 : q % 3 == 1 ? x1 : x2);
    const uint32_t e = start[k + 1];
    for (uint32_t j = start[k]; __any_sync(lanes, j < e); j += 4) {
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
        if (j + u >= e) continue;
        const R4<R> xj = x[j + u];
        const float dx = fx - (float)xj.x, dy = fy - (float)xj.y, dz = fz - (float)xj.z;
        if (dx * dx + dy * dy + dz * dz > limit) continue;
        list[cnt * kBlock] = j + u;
        ++cnt;
      }
      if (__any_sync(lanes, cnt > kNearList - 4)) drain();
    }
  }
  drain();
}

// ScalarQuantity at evaluation positions (sph/mod.rs:241-341 with the sums
// of quantities.rs:14-330), for sensor planes: one thread per position walks
// the 27 buckets of the fluid grid of the last update (sorted positions and
// volumes `xv`, velocities and masses `vel`, pressures), keeps the
// reference's exact neighbor predicate and sums in f64 whatever the state
// precision. Speed and volume also take the position's boundary samples
// (RequestMode::Normal): the sorted sample grid, or one sample per volume
// map. Quantities: 0 speed |sum v V W|, 1 volume V0 / sum V0 W, 2 density
// sum m W, 3 density error 100 sum_{m < V0} (V0/m - 1) m W (the reference
// passes the masses where the sum takes volumes), 4 pressure sum p V W,
// 5 kinetic energy sum m |v|^2 V W / 2. The result is cast to f32.
template <class R>
__global__ void __launch_bounds__(kBlock) k_quantity_at(
    int quantity, int n_eval, const float* __restrict__ eval, float* __restrict__ out,
    const uint32_t* __restrict__ start, const R4<R>* __restrict__ xv, const R4<R>* __restrict__ vel,
    const R* __restrict__ press, SampleGrid<R> G, const VMDesc* __restrict__ vms, int nvm,
    const Body* __restrict__ bodies, KernelConst<double> kd, double V0, StepParams<R> P) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_eval) return;
  const double p[3] = {(double)eval[3 * t], (double)eval[3 * t + 1], (double)eval[3 * t + 2]};
  const double h = P.range;
  __shared__ uint32_t s_list[kNearList * kBlock];
  double s = 0, sx = 0, sy = 0, sz = 0;
  if (start)
    for_each_within(p, h, P.mask, start, xv, s_list, [&](uint32_t j, const R4<R>& xj, double r2) {
      const double w = kernel_w_r2<double>(r2, kd);
      const double V = (double)xj.w;
      if (quantity == 1) { s += V0 * w; return; }
      const R4<R> vj = vel[j];
      const double vx = (double)vj.x, vy = (double)vj.y, vz = (double)vj.z, m = (double)vj.w;
      switch (quantity) {
        case 0: sx += vx * V * w; sy += vy * V * w; sz += vz * V * w; break;
        case 2: s += m * w; break;
        case 3: if (m < V0) s += (V0 / m - 1.0) * m * w; break;
        case 4: s += (double)press[j] * V * w; break;
        default: s += 0.5 * m * ((vx * vx + vy * vy) + vz * vz) * V * w; break;
      }
    });
  if (quantity <= 1) {
    if (G.start)
      for_each_within(p, h, G.mask, G.start, G.xb, s_list, [&](uint32_t j, const R4<R>& xs, double r2) {
        const double vw = (double)xs.w * kernel_w_r2<double>(r2, kd);
        if (quantity == 1) {
          s += vw;
        } else {
          const R4<R> vs = G.vb[j];
          sx += (double)vs.x * vw; sy += (double)vs.y * vw; sz += (double)vs.z * vw;
        }
      });
    const double ball = 4.0 / 3.0 * 3.14159265358979323846 * (h * h * h);
    for (int b = 0; b < nvm; ++b) {
      const VMDesc& D = vms[b];
      double xb[3] = {0, 0, 0}, vb[3] = {0, 0, 0}, vol = 0;
      if (!vm_normal_sample(D, D.body >= 0 ? &bodies[D.body] : nullptr, p, h, ball, P.spacing, xb, vb, vol))
        continue;
      const double rx = p[0] - xb[0], ry = p[1] - xb[1], rz = p[2] - xb[2];
      const double vw = vol * kernel_w_r2<double>((rx * rx + ry * ry) + rz * rz, kd);
      if (quantity == 1) {
        s += vw;
      } else {
        sx += vb[0] * vw; sy += vb[1] * vw; sz += vb[2] * vw;
      }
    }
  }
  double val;
  switch (quantity) {
    case 0: val = sqrt((sx * sx + sy * sy) + sz * sz); break;
    case 1: val = V0 / s; break;
    case 3: val = 100.0 * s; break;
    default: val = s; break;
  }
  out[t] = (float)val;
}

// ---------------------------------------------------------------------------
// Boundary iteration helpers used by the acceleration passes
// ---------------------------------------------------------------------------
template <class R>
struct BoundaryArgs {
  int kind;  // 0 none, 1 sample boundaries, 2 volume maps
  SampleGrid<R> grid;
  const R4<R>* vmx;
  const R4<R>* vmv;
  const VMDesc* vms;
  int nvm;
  const Body* bodies;
  int any_dynamic;
  const R* bW;
  const R4<R>* bG;
  const R4<R>* bGu;
  const R4<R>* bA;
  double* body_partials;  // [gridDim][kMaxBodies][6] reaction force/torque partials
  const uint32_t* touch;  // particles with a neighbor on a dynamic body (sc->n_touch of them)
  int nbodies;
};

// Per-block rigid-body force/torque accumulation in f64 (shared memory),
// flushed to per-block partials that a fixed-order kernel reduces.
// A thread sums for one body at a time and adds to the block's sums when the
// next force is another body's, and at the end.
struct BodyAccum {
  double* sh;  // [kMaxBodies][6]
  int body = -1;
  double a[6] = {0, 0, 0, 0, 0, 0};
  __device__ __forceinline__ void add(const Body* bodies, int b, const double F[3], const double x[3]) {
    if (b != body) flush();
    body = b;
    const double* com = bodies[b].com;
    const double r[3] = {x[0] - com[0], x[1] - com[1], x[2] - com[2]};
    a[0] += F[0]; a[1] += F[1]; a[2] += F[2];
    a[3] += r[1] * F[2] - r[2] * F[1];
    a[4] += r[2] * F[0] - r[0] * F[2];
    a[5] += r[0] * F[1] - r[1] * F[0];
  }
  __device__ __forceinline__ void flush() {
    for (int k = 0; k < 6; ++k) {
      if (body >= 0) atomicAdd(&sh[body * 6 + k], a[k]);
      a[k] = 0.0;
    }
    body = -1;
  }
};

__device__ __forceinline__ void body_accum_init(double* sh, int nbodies) {
  for (int t = threadIdx.x; t < nbodies * 6; t += blockDim.x) sh[t] = 0.0;
  __syncthreads();
}
__device__ __forceinline__ void body_accum_flush(double* sh, int nbodies, double* partials) {
  __syncthreads();
  for (int t = threadIdx.x; t < nbodies * 6; t += blockDim.x)
    partials[(size_t)blockIdx.x * kMaxBodies * 6 + t] = sh[t];
}

// ---------------------------------------------------------------------------
// 5a. sample boundaries: everything a particle takes from its boundary
// samples, in one pass over them (all boundaries):
//   bW  = sum V_b W_ib                                  (volume)
//   bG  = {sum V_b gradW_ib, sum V_b (v_b . gradW_ib)}  (pressure, source, a_ii)
//   bGu = {sum gradW_ib, -}                             (SESPHwSplitting only)
//   bA  = {boundary viscosity acceleration, -}
// and the list of the particles with a neighbor on a dynamic body.
//
// A warp takes one cell at a time (a block holds eight warps for the cells of
// kSampleBlock particles, about as many): 27 lanes read the stencil's bucket
// bounds at once, and a cell without samples around it (most of them) is
// done. Otherwise its candidates are staged in shared memory, and 4 or 8 lanes
// share them for every particle of the cell. (A block with fewer cells than warps, as
// in a compressed scene, hands out its cells' groups of eight particles instead.) A lane first tests its
// candidates into a mask, then sums over the set bits. The kernel values go
// through shared memory to one lane, which sums them in sample order (the
// volume's compensated sum keeps its bits whatever the split).
//
// What bounds it: latency. With one thread per particle walking 27 buckets,
// in this pass and again for the viscosity, scenes of 5 to 195 thousand
// particles took 63-72 us here and 75-105 us more in the acceleration pass;
// in this form 23-36 us here and 11-36 us there.
// ---------------------------------------------------------------------------
constexpr int kSampleBlock = 64;   // particles per block of kBlock threads
constexpr int kSampleChunk = 96;   // candidates staged at a time
template <class R>
struct SampleStage {  // per warp
  R4<R> x[kSampleChunk], v[kSampleChunk];
  uint32_t s[kSampleChunk];
  R w[8][kSampleChunk];  // per particle: kernel values, -1 out of range
};

template <class R, bool SPLIT>
__global__ void __launch_bounds__(kBlock) k_sample_boundary(
    Scalars* sc, const R4<R>* pos, const R4<R>* vel, SampleGrid<R> G,
    const Body* bodies, int any_dynamic, R* bW, R4<R>* bG,
    R4<R>* bGu, R4<R>* bA, uint32_t* touch, StepParams<R> P) {
  grid_dep_begin();
  extern __shared__ __align__(32) unsigned char dsm[];
  __shared__ uint32_t s_key[kSampleBlock], s_heads[kSampleBlock / 32];
  __shared__ uint8_t s_head[kSampleBlock + 1], s_near[kSampleBlock];  // per cell: first particle; it has candidates
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = blockIdx.x * kSampleBlock, i = i0 + tid;
  const int m = min(kSampleBlock, sc->n_active - i0);  // this block's particles
  if (m <= 0) return;
  if (tid < kSampleBlock) s_key[tid] = tid < m ? lane_key(pos[i].w) : 0u;
  __syncthreads();
  const bool head = tid < m && (tid == 0 || s_key[tid - 1] != s_key[tid]);
  const uint32_t heads = __ballot_sync(0xffffffffu, head);
  if (lane == 0 && warp < kSampleBlock / 32) s_heads[warp] = heads;
  __syncthreads();
  const int nheads = __popc(s_heads[0]) + __popc(s_heads[1]);
  const int rank = (warp == 1 ? __popc(s_heads[0]) : 0) + __popc(heads & ((2u << lane) - 1u)) - 1;  // this particle's cell
  if (head) s_head[rank] = (uint8_t)tid;
  if (tid == 0) s_head[nheads] = (uint8_t)m;
  __syncthreads();
  SampleStage<R>& T = reinterpret_cast<SampleStage<R>*>(dsm)[warp];
  int most = 0;
  constexpr int kWarps = kBlock / 32;
  const bool spread = nheads < kWarps;  // fewer cells than warps: their groups of eight particles one by one
  for (int h = spread ? 0 : warp, units = 0; h < nheads; h += spread ? 1 : kWarps) {
    const int p0 = s_head[h], np = s_head[h + 1] - p0;
    const int S = np <= 4 ? 8 : 4;  // lanes per particle
    int g0 = 0, g_step = 32 / S;
    if (spread) {
      g0 = 8 * ((warp - units) & (kWarps - 1));
      g_step = 8 * kWarps;
      units += (np + 7) / 8;
      if (g0 >= np) continue;
    }
    const uint32_t ck = s_key[p0];
    uint32_t first = 0, len = 0;
    if (lane < 27) {
      const uint32_t k = morton_key((int)gather3(ck) + lane % 3 - 1, (int)gather3(ck >> 1) + (lane / 3) % 3 - 1,
                                    (int)gather3(ck >> 2) + lane / 9 - 1, G.mask);
      first = G.start[k];
      len = G.start[k + 1] - first;
    }
    const bool near = __any_sync(0xffffffffu, len != 0);
    if (lane == 0) s_near[h] = near;
    if (!near) continue;
    uint32_t end = len;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += y;
    }
    const uint32_t C = __shfl_sync(0xffffffffu, end, 31), begin = end - len;
    const int sub = lane & (S - 1), row = lane / S;
    for (int g = g0; g < np; g += g_step) {
      const int p = g + row;
      const bool mine = p < np;
      const int ip = i0 + p0 + (mine ? p : 0);
      const R4<R> xi = pos[ip], vi = vel[ip];
      R w = 0, wc = 0;
      R gx = 0, gy = 0, gz = 0, gv = 0, ux = 0, uy = 0, uz = 0, sx = 0, sy = 0, sz = 0;
      int cnt = 0;
      bool dyn = false;
      for (uint32_t c0 = 0; c0 < C; c0 += kSampleChunk) {
        const int nc = (int)min(C - c0, (uint32_t)kSampleChunk);
        __syncwarp();
        for (uint32_t c = max(begin, c0); c < min(end, c0 + (uint32_t)nc); ++c) T.s[c - c0] = first + (c - begin);
        __syncwarp();
        for (int c = lane; c < nc; c += 32) {
          const uint32_t s = T.s[c];
          T.x[c] = G.xb[s];
          T.v[c] = G.vb[s];
        }
        __syncwarp();
        uint32_t in = 0;  // candidate sub + S q at bit q
        for (int c = sub, q = 0; c < nc; c += S, ++q) {
          const bool hit = mine && in_range(xi, T.x[c], P.range, P.range2_lo, P.range2_hi);
          if (hit) in |= 1u << q;
          else T.w[row][c] = R(-1);
        }
        cnt += __popc(in);
        while (in) {
          const int q = __ffs((int)in) - 1;
          in &= in - 1;
          const int c = sub + S * q;
          const R4<R> xs = T.x[c], vs = T.v[c];
          const R rx = xi.x - xs.x, ry = xi.y - xs.y, rz = xi.z - xs.z;
          const R r2 = rx * rx + ry * ry + rz * rz;
          R kw, f;
          kernel_w_and_grad(r2, P.k, kw, f);
          T.w[row][c] = kw;
          const R vf = xs.w * f;
          gx += vf * rx; gy += vf * ry; gz += vf * rz;
          gv += vf * (vs.x * rx + vs.y * ry + vs.z * rz);
          if (SPLIT) { ux += f * rx; uy += f * ry; uz += f * rz; }
          const R vr = (vi.x - vs.x) * rx + (vi.y - vs.y) * ry + (vi.z - vs.z) * rz;
          const R s = P.visc_b * xs.w * vr / (r2 + P.eps_visc) * f;
          sx += s * rx; sy += s * ry; sz += s * rz;
          if (any_dynamic) dyn |= bodies[G.bid[T.s[c]]].dynamic != 0;
        }
        __syncwarp();
        if (sub == 0) {
#pragma unroll 8
          for (int c = 0; c < nc; ++c) {
            const R kw = T.w[row][c], V = T.x[c].w;
            R w2 = w, c2 = wc;
            kahan_add(w2, c2, V * kw);
            w = kw >= R(0) ? w2 : w;
            wc = kw >= R(0) ? c2 : wc;
          }
        }
      }
      for (int o = S >> 1; o > 0; o >>= 1) {
        gx += __shfl_xor_sync(0xffffffffu, gx, o); gy += __shfl_xor_sync(0xffffffffu, gy, o);
        gz += __shfl_xor_sync(0xffffffffu, gz, o); gv += __shfl_xor_sync(0xffffffffu, gv, o);
        if (SPLIT) {
          ux += __shfl_xor_sync(0xffffffffu, ux, o); uy += __shfl_xor_sync(0xffffffffu, uy, o);
          uz += __shfl_xor_sync(0xffffffffu, uz, o);
        }
        sx += __shfl_xor_sync(0xffffffffu, sx, o); sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sz += __shfl_xor_sync(0xffffffffu, sz, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (any_dynamic) dyn |= __shfl_xor_sync(0xffffffffu, (int)dyn, o) != 0;
      }
      most = max(most, cnt);
      if (mine && sub == 0) {
        bW[ip] = w;
        bG[ip] = R4<R>{gx, gy, gz, gv};
        if (SPLIT) bGu[ip] = R4<R>{ux, uy, uz, R(0)};
        bA[ip] = R4<R>{sx, sy, sz, R(0)};
        if (dyn) touch[atomicAdd(&sc->n_touch, 1u)] = (uint32_t)ip;
      }
    }
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0 && most > 0) atomicMax(&sc->max_bnbrs, most);
  __syncthreads();
  if (tid < m && !s_near[rank]) {
    bW[i] = R(0);
    bG[i] = R4<R>{R(0), R(0), R(0), R(0)};
    if (SPLIT) bGu[i] = R4<R>{R(0), R(0), R(0), R(0)};
    bA[i] = R4<R>{R(0), R(0), R(0), R(0)};
  }
}

// Reactions on dynamic bodies, once the pressures are known: for every
// particle of the touch list and each of its boundary neighbors on a dynamic
// body, the viscosity's F = -m_i a_ib (non_pressure_accelerations.rs) and the
// pressure's F = 2 gamma_p V_i V_b p_i gradW_ib (pressure_solver/mod.rs:
// 160-195). A warp per particle: its lanes take the stencil's buckets (sample
// boundaries) or the volume maps. (Inside the acceleration passes, which
// walked every particle's samples twice for it, a tank of 276 thousand
// particles with eight bodies took 591 us there, now 56 us and 21 us here.)
template <class R>
__global__ void __launch_bounds__(kBlock) k_body_react(const Scalars* __restrict__ sc, const R4<R>* __restrict__ xv,
                                                      const R4<R>* __restrict__ vel, const R* __restrict__ press,
                                                      BoundaryArgs<R> B, StepParams<R> P) {
  __shared__ double sh_body[kMaxBodies * 6];
  body_accum_init(sh_body, B.nbodies);
  BodyAccum acc_b{sh_body};
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (kBlock / 32);
  for (uint32_t t = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); t < sc->n_touch; t += warps) {
    const int i = (int)B.touch[t];
    const R4<R> xi = xv[i], vi = vel[i];
    const R pi = press[i];
    auto viscous = [&](const V3<R>& x, const V3<R>& v, R V, int body) {
      const V3<R> r{xi.x - x.x, xi.y - x.y, xi.z - x.z};
      const R s = boundary_viscosity(r, V3<R>{vi.x - v.x, vi.y - v.y, vi.z - v.z}, V, P);
      const double mi = (double)vi.w;
      const double F[3] = {-mi * (double)(s * r.x), -mi * (double)(s * r.y), -mi * (double)(s * r.z)};
      const double xl[3] = {(double)x.x, (double)x.y, (double)x.z};
      acc_b.add(B.bodies, body, F, xl);
    };
    auto pressure = [&](const V3<R>& x, R V, int body) {
      const R rx = xi.x - x.x, ry = xi.y - x.y, rz = xi.z - x.z;
      const R f = kernel_grad_factor(rx * rx + ry * ry + rz * rz, P.k);
      const double c2 = 2.0 * (double)P.gamma_p * (double)xi.w * (double)V * (double)pi * (double)f;
      const double F[3] = {c2 * rx, c2 * ry, c2 * rz};
      const double xl[3] = {(double)x.x, (double)x.y, (double)x.z};
      acc_b.add(B.bodies, body, F, xl);
    };
    if (B.kind == 1 && lane < 27) {
      const uint32_t k = morton_key(cell_coord((double)xi.x, P.range) + lane % 3 - 1,
                                    cell_coord((double)xi.y, P.range) + (lane / 3) % 3 - 1,
                                    cell_coord((double)xi.z, P.range) + lane / 9 - 1, B.grid.mask);
      const uint32_t e = B.grid.start[k + 1];
      for (uint32_t s = B.grid.start[k]; s < e; ++s) {
        const int body = (int)B.grid.bid[s];
        if (!B.bodies[body].dynamic) continue;
        const R4<R> xs = B.grid.xb[s], vs = B.grid.vb[s];
        if (!in_range(xi, xs, P.range, P.range2_lo, P.range2_hi)) continue;
        const V3<R> x{xs.x, xs.y, xs.z};
        viscous(x, V3<R>{vs.x, vs.y, vs.z}, xs.w, body);
        pressure(x, xs.w, body);
      }
    } else if (B.kind == 2 && lane < B.nvm) {
      const size_t o = (size_t)lane * P.Np + i;
      const int body = B.vms[lane].body;
      const R kind = B.vmv[o].w;
      if (body >= 0 && B.bodies[body].dynamic && kind != R(0)) {
        const R4<R> xs = B.vmx[o];
        const TangentSamples<R> ts(xi, xs, kind, P.range);
        for (int k = 0; k < 4; ++k) {
          const V3<R> q = ts.at(k);
          viscous(q, body_velocity_r(B.bodies, body, q), R(0.25) * xs.w, body);
        }
        pressure(V3<R>{xs.x, xs.y, xs.z}, xs.w, body);
      }
    }
  }
  acc_b.flush();
  body_accum_flush(sh_body, B.nbodies, B.body_partials);
}

// ---------------------------------------------------------------------------
// Neighbor gather loop. The halo positions of NB neighbors are fetched first
// (streaming, evict-first 64-bit loads of four 16-bit positions), then the NB
// records are loaded, then consumed, so NB loads are in flight per thread.
// Slots past the count read position 0, which every non-empty halo has.
// ---------------------------------------------------------------------------
// The first D batches of a particle's list, requested ahead of use (a kernel
// can issue them before it waits for its halo staging).
template <int NB, int D = 1>
struct ListHead {
  uint2 g[D][NB / 4];
};
template <int NB, int D = 1>
__device__ __forceinline__ ListHead<NB, D> list_head(const uint16_t* __restrict__ nbr, int K, int i, int cnt) {
  ListHead<NB, D> h;
  const uint2* base = reinterpret_cast<const uint2*>(nbr) + nbr_slot(i, 0, K) / 4;
  const int ngroups = (cnt + 3) >> 2;
#pragma unroll
  for (int d = 0; d < D; ++d)
#pragma unroll
    for (int g = 0; g < NB / 4; ++g) {
      const int gi = d * (NB / 4) + g;
      h.g[d][g] = gi < ngroups ? __ldcs(base + (size_t)gi * 32) : make_uint2(0u, 0u);
    }
  return h;
}

// Visits the neighbors of particle i in batches of NB: while a batch is
// consumed, the list words of the batch D ahead are in flight.
template <int NB, int D, class Load, class Use>
__device__ __forceinline__ void for_each_neighbor(const uint16_t* __restrict__ nbr, int K, int i, int cnt,
                                                  const ListHead<NB, D>& head, Load&& load, Use&& use) {
  static_assert(NB % 4 == 0, "neighbors are read in groups of four");
  // group g of this lane sits 32 uint2 after group g-1
  const uint2* base = reinterpret_cast<const uint2*>(nbr) + nbr_slot(i, 0, K) / 4;
  const int ngroups = (cnt + 3) >> 2;
  uint2 q[D][NB / 4];
#pragma unroll
  for (int d = 0; d < D; ++d)
#pragma unroll
    for (int g = 0; g < NB / 4; ++g) q[d][g] = head.g[d][g];
  for (int k0 = 0; k0 < cnt; k0 += NB) {
    uint2 nxt[NB / 4];
#pragma unroll
    for (int g = 0; g < NB / 4; ++g) {
      const int gi = (k0 + D * NB) / 4 + g;
      nxt[g] = gi < ngroups ? __ldcs(base + (size_t)gi * 32) : make_uint2(0u, 0u);
    }
    uint32_t l[NB];
#pragma unroll
    for (int g = 0; g < NB / 4; ++g) {
      const uint2 w = q[0][g];
      l[4 * g + 0] = k0 + 4 * g + 0 < cnt ? (w.x & 0xffffu) : 0u;
      l[4 * g + 1] = k0 + 4 * g + 1 < cnt ? (w.x >> 16) : 0u;
      l[4 * g + 2] = k0 + 4 * g + 2 < cnt ? (w.y & 0xffffu) : 0u;
      l[4 * g + 3] = k0 + 4 * g + 3 < cnt ? (w.y >> 16) : 0u;
    }
    decltype(load(0u)) d[NB];
#pragma unroll
    for (int u = 0; u < NB; ++u) d[u] = load(l[u]);
#pragma unroll
    for (int u = 0; u < NB; ++u)
      if (k0 + u < cnt) use(d[u]);
#pragma unroll
    for (int e = 0; e + 1 < D; ++e)
#pragma unroll
      for (int g = 0; g < NB / 4; ++g) q[e][g] = q[e + 1][g];
#pragma unroll
    for (int g = 0; g < NB / 4; ++g) q[D - 1][g] = nxt[g];
  }
}
template <int NB, class Load, class Use>
__device__ __forceinline__ void for_each_neighbor(const uint16_t* __restrict__ nbr, int K, int i, int cnt,
                                                  Load&& load, Use&& use) {
  for_each_neighbor<NB, 1>(nbr, K, i, cnt, list_head<NB, 1>(nbr, K, i, cnt), load, use);
}

// Shared-memory layout of staged halo records: arrays of R4 then arrays of R,
// each `hs` records long.
template <class R>
__device__ __forceinline__ R4<R>* staged_vec(unsigned char* dsm, int hs, int which) {
  return reinterpret_cast<R4<R>*>(dsm) + (size_t)which * hs;
}
template <class R>
__device__ __forceinline__ R* staged_scalar(unsigned char* dsm, int hs, int nvec, int which) {
  return reinterpret_cast<R*>(reinterpret_cast<R4<R>*>(dsm) + (size_t)nvec * hs) + (size_t)which * hs;
}

template <class R>
struct XP {  // position+volume and one scalar
  R4<R> x;
  R s;
};
template <class R>
struct XV {  // position+volume and one vector
  R4<R> x;
  R4<R> v;
};
template <class R>
struct SweepList {
  const uint2* p;  // this particle's first group of four; group g sits 32 uint2 further
  int ng;          // groups
  uint2 w0, w1;    // the next two groups, in flight
  __device__ __forceinline__ void begin(const NbrArgs& N, int i, int cnt) {
    p = reinterpret_cast<const uint2*>(N.nbr) + nbr_slot(i, 0, N.K) / 4;
    ng = (cnt + 3) >> 2;
    w0 = ng > 0 ? __ldcs(p) : make_uint2(0u, 0u);
    w1 = ng > 1 ? __ldcs(p + 32) : make_uint2(0u, 0u);
  }
  // the group to use now; requests the one two groups ahead
  __device__ __forceinline__ uint2 next(int g) {
    const uint2 w = w0;
    w0 = w1;
    w1 = g + 2 < ng ? __ldcs(p + (size_t)(g + 2) * 32) : make_uint2(0u, 0u);
    return w;
  }
};

// Visits every slot of a particle's neighbor list in whole groups of four,
// padding included: the unused slots of the last group repeat the particle's
// own halo position, so a pass whose pair term is zero at r = 0 needs no
// per-neighbor count test. The four records of a group are gathered before
// they are used.
template <class List, class Load, class Use>
__device__ __forceinline__ void sweep_groups(List& L, Load&& load, Use&& use) {
  for (int g = 0; g < L.ng; ++g) {
    const uint2 w = L.next(g);
    const auto d0 = load(w.x & 0xffffu);
    const auto d1 = load(w.x >> 16);
    const auto d2 = load(w.y & 0xffffu);
    const auto d3 = load(w.y >> 16);
    use(d0); use(d1); use(d2); use(d3);
  }
}

// ---------------------------------------------------------------------------
// 6. accelerations: gravity + viscosity (+ SESPH pressure) (+ v* = v + dt a)
// ---------------------------------------------------------------------------
// PRESS: 0 none, 1 SESPH state equation from the volume on the fly
template <class R, int PRESS>
__global__ void __launch_bounds__(kBlock) k_accel(
    const Scalars* sc, const R4<R>* xv, const R4<R>* vel,
    NbrArgs N, BoundaryArgs<R> B, R4<R>* acc, R4<R>* vstar,
    R* press, int write_vstar, StepParams<R> P) {
  grid_dep_begin();
  extern __shared__ __align__(32) unsigned char dsm[];
  const HaloView H = halo_view(N);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < sc->n_active;
  SweepList<R> L;  // the list head travels while the halo stages
  L.begin(N, act ? i : 0, act ? min((int)N.ncnt[i], N.K) : 0);
  R4<R> xi{}, vi{};
  if (act) {
    xi = xv[i];
    vi = vel[i];
  }
  R4<R>* s_x = staged_vec<R>(dsm, N.hs, 0);
  R4<R>* s_v = staged_vec<R>(dsm, N.hs, 1);
  if (H.staged)
    stage_halo(H, [&](int l, uint32_t g) {
      async_copy(&s_x[l], &xv[g]);
      async_copy(&s_v[l], &vel[g]);
    });
  stage_done();
  if (act) {
    const R mi = vi.w, Vi = xi.w;
    R ax, ay, az;
    if (P.gravity_mode == 0) {
      ax = 0; ay = 0; az = R(-9.81);
    } else {
      const R dx = P.gc[0] - xi.x, dy = P.gc[1] - xi.y, dz = P.gc[2] - xi.z;
      const R dist = sqrt(dx * dx + dy * dy + dz * dz + R(1e-4));
      ax = R(9.81) * dx / dist; ay = R(9.81) * dy / dist; az = R(9.81) * dz / dist;
    }
    R pi = 0;
    if (PRESS == 1) pi = P.stiffness * fmax(P.V0 / Vi - R(1), R(0));
    R sx = 0, sy = 0, sz = 0;   // viscosity
    R px = 0, py = 0, pz = 0;   // pressure
    // pair terms are zero at r = 0 (self padding adds nothing)
    auto pair = [&](const XV<R>& d) {
          const R4<R>& xj = d.x;
          const R4<R>& vj = d.v;
          const R rx = xi.x - xj.x, ry = xi.y - xj.y, rz = xi.z - xj.z;
          const R r2 = rx * rx + ry * ry + rz * rz;
          const R f = kernel_grad_factor(r2, P.k);
          const R vr = (vi.x - vj.x) * rx + (vi.y - vj.y) * ry + (vi.z - vj.z) * rz;
          const R s = quotient(P.visc_f * xj.w * vr, r2 + P.eps_visc) * f;
          sx += s * rx; sy += s * ry; sz += s * rz;
          if (PRESS == 1) {
            const R pj = P.stiffness * fmax(quotient(P.V0, xj.w) - R(1), R(0));
            const R t = xj.w * (pi + pj) * f;
            px += t * rx; py += t * ry; pz += t * rz;
          }
        };
    if (H.staged)
      sweep_groups(L, [&](uint32_t l) { return XV<R>{s_x[l], s_v[l]}; }, pair);
    else
      sweep_groups(L, [&](uint32_t l) { const uint32_t g = H.idx[l]; return XV<R>{xv[g], vel[g]}; }, pair);
    if (B.kind != 0) {
      const R4<R> bv = B.bA[i];
      sx += bv.x; sy += bv.y; sz += bv.z;
      if (PRESS == 1) {
        const R4<R> g = B.bG[i];
        const R c = R(2) * P.gamma_p * pi;  // boundary: 2 gamma V_i V_b p_i gradW / m_i
        px += c * g.x; py += c * g.y; pz += c * g.z;
      }
    }
    const R vm = Vi / mi;
    ax += sx - vm * px;
    ay += sy - vm * py;
    az += sz - vm * pz;
    acc[i] = R4<R>{ax, ay, az, R(0)};
    if (write_vstar) {
      const R dt = (R)sc->dt;
      // (the lane that the next pass needs rides along: the mass, or V^2 / m)
      vstar[i] = R4<R>{vi.x + dt * ax, vi.y + dt * ay, vi.z + dt * az, write_vstar == 2 ? Vi * Vi / mi : mi};
    }
    if (PRESS == 1) press[i] = pi;
  }
}

// ---------------------------------------------------------------------------
// 7. pressure acceleration from stored pressures (pressure_solver/mod.rs:121-195)
// ---------------------------------------------------------------------------
// acc += accel (the solvers with Jacobi sweeps take it from k_sweep_accel)
template <class R>
__global__ void __launch_bounds__(kBlock) k_pressure_accel(
    const Scalars* sc, const R4<R>* xv, const R4<R>* vel,
    const R* press, NbrArgs N, BoundaryArgs<R> B, R4<R>* out, StepParams<R> P) {
  grid_dep_begin();
  extern __shared__ __align__(32) unsigned char dsm[];
  const HaloView H = halo_view(N);
  // this particle's own data and first list batch travel while the halo stages
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < sc->n_active;
  SweepList<R> L;
  L.begin(N, act ? i : 0, act ? min((int)N.ncnt[i], N.K) : 0);
  R4<R> xi{};
  R mi = 1, pi = 0;
  if (act) {
    xi = xv[i];
    mi = vel[i].w;
    pi = press[i];
  }
  R4<R>* s_x = staged_vec<R>(dsm, N.hs, 0);
  R* s_p = staged_scalar<R>(dsm, N.hs, 1, 0);
  if (H.staged)
    stage_halo(H, [&](int l, uint32_t g) {
      async_copy(&s_x[l], &xv[g]);
      async_copy(&s_p[l], &press[g]);
    });
  stage_done();
  if (act) {
    const R Vi = xi.w;
    R px = 0, py = 0, pz = 0;
    auto pair = [&](const XP<R>& d) {  // zero at r = 0 (self padding)
      const R rx = xi.x - d.x.x, ry = xi.y - d.x.y, rz = xi.z - d.x.z;
      const R f = kernel_grad_factor(rx * rx + ry * ry + rz * rz, P.k);
      const R t = d.x.w * (pi + d.s) * f;
      px += t * rx; py += t * ry; pz += t * rz;
    };
    if (H.staged)
      sweep_groups(L, [&](uint32_t l) { return XP<R>{s_x[l], s_p[l]}; }, pair);
    else
      sweep_groups(L, [&](uint32_t l) { const uint32_t g = H.idx[l]; return XP<R>{xv[g], press[g]}; }, pair);
    if (B.kind != 0) {
      const R4<R> g = B.bG[i];
      const R c = R(2) * P.gamma_p * pi;
      px += c * g.x; py += c * g.y; pz += c * g.z;
    }
    const R vm = Vi / mi;
    R4<R> o = out[i];
    o.x += -vm * px; o.y += -vm * py; o.z += -vm * pz;
    out[i] = o;
  }
}

// ---------------------------------------------------------------------------
// 8. IISPH: source term + diagonal + initial pressure (iisph.rs:117-376)
// ---------------------------------------------------------------------------
// VP = 1: volume-preserving source s = 1 - V0/V - dt sum ..., VP = 0: the
// velocity-divergence source of IISPHwOST's first solve.
template <class R, int VP>
__global__ void __launch_bounds__(kBlock) k_iisph_source_diag(
    const Scalars* sc, const R4<R>* xv, const R4<R>* vel,
    const R4<R>* vstar, NbrArgs N, BoundaryArgs<R> B, R* s_out,
    R* aii_out, R* press, R4<R>* TA, R4<R>* TB,
    R2<R>* SA, R4<R>* xq_out, StepParams<R> P) {
  grid_dep_begin();
  extern __shared__ __align__(32) unsigned char dsm[];
  const HaloView H = halo_view(N);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < sc->n_active;
  SweepList<R> L;  // the list head travels while the halo stages
  L.begin(N, act ? i : 0, act ? min((int)N.ncnt[i], N.K) : 0);
  R4<R> xi{}, vsi{};
  R mi = 1;
  if (act) {
    xi = xv[i];
    vsi = vstar[i];
    mi = vel[i].w;
  }
  // records {x, V} and {v*, V^2/m} (the acceleration pass stores V^2/m in v*.w)
  R4<R>* s_x = staged_vec<R>(dsm, N.hs, 0);
  R4<R>* s_v = staged_vec<R>(dsm, N.hs, 1);
  if (H.staged)
    stage_halo(H, [&](int l, uint32_t g) {
      async_copy(&s_x[l], &xv[g]);
      async_copy(&s_v[l], &vstar[g]);
    });
  stage_done();
  if (!act) return;
  const R dt = (R)sc->dt;
  const R Vi = xi.w;
  R div = 0;                       // sum V_j (v*_i - v*_j) . gradW
  R sfx = 0, sfy = 0, sfz = 0;     // S_f = sum V_j gradW
  R s2 = 0;                        // sum V_j^2 / m_j |gradW|^2
  auto pair = [&](const XV<R>& d) {  // zero at r = 0 (self padding)
    const R4<R>& xj = d.x;
    const R4<R>& vsj = d.v;
    const R rx = xi.x - xj.x, ry = xi.y - xj.y, rz = xi.z - xj.z;
    const R r2 = rx * rx + ry * ry + rz * rz;
    const R f = kernel_grad_factor(r2, P.k);
    const R Vf = xj.w * f;
    div += Vf * ((vsi.x - vsj.x) * rx + (vsi.y - vsj.y) * ry + (vsi.z - vsj.z) * rz);
    sfx += Vf * rx; sfy += Vf * ry; sfz += Vf * rz;
    s2 += vsj.w * (f * f * r2);
  };
  if (H.staged)
    sweep_groups(L, [&](uint32_t l) { return XV<R>{s_x[l], s_v[l]}; }, pair);
  else
    sweep_groups(L, [&](uint32_t l) { const uint32_t g = H.idx[l]; return XV<R>{xv[g], vstar[g]}; }, pair);
  R bx = 0, by = 0, bz = 0, bdiv = 0;
  if (B.kind != 0) {
    const R4<R> g = B.bG[i];
    bx = g.x; by = g.y; bz = g.z;
    bdiv = vsi.x * g.x + vsi.y * g.y + vsi.z * g.z - g.w;  // sum V_b (v*_i - v_b) . gradW
  }
  R s = VP ? R(1) - P.V0 / Vi : R(0);
  s -= dt * (div + bdiv);
  const R dt2 = dt * dt;
  const R c = -Vi / mi;
  const R cx = c * (sfx + R(2) * P.gamma_p * bx), cy = c * (sfy + R(2) * P.gamma_p * by),
          cz = c * (sfz + R(2) * P.gamma_p * bz);
  const R aii = dt2 * (cx * (sfx + bx) + cy * (sfy + by) + cz * (sfz + bz)) - dt2 * Vi * s2;
  s_out[i] = s;
  aii_out[i] = aii;
  R p0 = 0;
  if (aii > P.min_diag || aii < -P.min_diag) p0 = fmax(P.omega * s / aii, R(0));
  press[i] = p0;
  // the Jacobi sweeps' per-solve constants (S_i = sum_j V_j gradW_ij with the
  // boundary terms folded in) and the first pass A record {x, V p}
  const R g2 = R(2) * P.gamma_p;
  TA[i] = R4<R>{sfx + g2 * bx, sfy + g2 * by, sfz + g2 * bz, -(Vi / mi) * Vi};
  TB[i] = R4<R>{sfx + bx, sfy + by, sfz + bz, Vi};
  SA[i] = R2<R>{s, aii};
  xq_out[i] = R4<R>{xi.x, xi.y, xi.z, Vi * p0};
}

// ---------------------------------------------------------------------------
// Jacobi sweep (iisph.rs:401-560): pass A, the pressure accelerations of the
// current pressures (pressure_solver/mod.rs:121-195, overwrite, no reaction
// forces), then pass B, A_i, the relaxed pressure update and the residual.
// Positions and volumes are fixed during a solve, so the pair sums split:
//   sum_j V_j (p_i + p_j) gradW_ij    = p_i S_i + sum_j (V_j p_j) gradW_ij
//   sum_j V_j (a_i - a_j) . gradW_ij  = a_i . S_i - sum_j (V_j a_j) . gradW_ij
// with S_i = sum_j V_j gradW_ij from the source pass (stored with the boundary
// terms and the particle's own constants: TA = {S_i + 2 gamma_p bG_i, -V_i^2/m_i},
// TB = {S_i + bG_i, V_i}, SA = {s_i, a_ii}). Each pass then gathers
// one record per neighbor from the block's halo in shared memory:
//   pass A: xq = {x, y, z, V p}            (written by pass B and the source pass)
//   pass B: xu = {x, y, z, V a_x}, uu = {V a_y, V a_z}   (written by pass A)
// A neighbor group of four always holds four valid halo positions (unused
// slots repeat the particle's own, whose pair adds zero), so the loops carry
// no per-neighbor test. The kernel constant cg (-3 cg for pass A's piecewise
// gradient factor) multiplies each pair sum once.
// ---------------------------------------------------------------------------

// pass A: a_i = -(V_i/m_i) [p_i (S_i + 2 gamma_p bG_i) + sum_j (V_j p_j) gradW_ij],
// stored as the records of pass B (V_i a_i).
// (f32: at most 48 registers, so five blocks share an SM; the records are
// gathered two at a time to fit)
// OUT 0: the records of pass B; OUT 1: acc += a_i, OUT 2: acc = a_i (the
// final pressure acceleration of a solve, pressure_solver/mod.rs:121-195; the
// reaction on dynamic bodies is k_body_react).
template <class R, int OUT = 0>
__global__ void __launch_bounds__(kBlock, sizeof(R) == 4 ? 5 : 1) k_sweep_accel(
    const Scalars* sc, const R* press, const R4<R>* TA,
    const R4<R>* xq, NbrArgs N, R4<R>* xu, R2<R>* uu, StepParams<R> P,
    R4<R>* acc, const R4<R>* TB) {
  grid_dep_release();
  extern __shared__ __align__(32) unsigned char dsm[];
  const HaloView H = halo_view(N);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < sc->n_active;
  // what is fixed during a solve (list head, constants, halo indices) is read
  // before the wait on the previous pass; p and the records after it
  SweepList<R> L;
  L.begin(N, act ? i : 0, act ? min((int)N.ncnt[i], N.K) : 0);
  R4<R> xi{}, Ti{};
  R pi = 0;
  if (act) Ti = TA[i];
  const HaloFirst hf = halo_first(H);
  grid_dep_wait();
  if (OUT == 0 && sc->converged) return;
  if (act) {
    xi = xq[i];
    pi = press[i];
  }
  R4<R>* s_r = reinterpret_cast<R4<R>*>(dsm);
  stage_halo_from(H, hf, [&](int l, uint32_t g) { async_copy(&s_r[l], &xq[g]); });
  prefetch_ahead(N, sc->n_active, xq, TA, press);
  stage_done();
  if (!act) return;
  const R ih = P.k.inv_h;
  R px = 0, py = 0, pz = 0;
  auto pair = [&](const R4<R>& r) {
    const R rx = xi.x - r.x, ry = xi.y - r.y, rz = xi.z - r.z;
    const R t = r.w * grad_third_close(rx, ry, rz, ih);
    px += t * rx; py += t * ry; pz += t * rz;
  };
  if (H.staged) {
    for (int g = 0; g < L.ng; ++g) {
      const uint2 w = L.next(g);
      {
        const R4<R> r0 = s_r[w.x & 0xffffu], r1 = s_r[w.x >> 16];
        pair(r0); pair(r1);
      }
      {
        const R4<R> r2 = s_r[w.y & 0xffffu], r3 = s_r[w.y >> 16];
        pair(r2); pair(r3);
      }
    }
  } else {
    for (int g = 0; g < L.ng; ++g) {
      const uint2 w = L.next(g);
      const R4<R> r0 = xq[H.idx[w.x & 0xffffu]], r1 = xq[H.idx[w.x >> 16]], r2 = xq[H.idx[w.y & 0xffffu]],
                  r3 = xq[H.idx[w.y >> 16]];
      pair(r0); pair(r1); pair(r2); pair(r3);
    }
  }
  const R cg = R(-3) * P.k.cg;  // gradW = -3 cg grad_third r
  const R fx = pi * Ti.x + cg * px, fy = pi * Ti.y + cg * py, fz = pi * Ti.z + cg * pz;
  const R c = Ti.w;  // V_i a_i = -(V_i^2 / m_i) F
  if (OUT == 0) {
    xu[i] = R4<R>{xi.x, xi.y, xi.z, c * fx};
    uu[i] = R2<R>{c * fy, c * fz};
  } else {
    const R m = c / TB[i].w;  // a_i = -(V_i / m_i) F, TB.w = V_i
    R4<R> o = OUT == 1 ? acc[i] : R4<R>{R(0), R(0), R(0), R(0)};
    o.x += m * fx; o.y += m * fy; o.z += m * fz;
    acc[i] = o;
  }
}

// End of a sweep (one thread): error, sweep count, stop test (iisph.rs:378-393).
__device__ __forceinline__ void end_sweep(Scalars* sc, double total, int n, int after, double tde, int cap) {
  const int it = sc->iterations + 1;  // (both loads at once: other blocks wait)
  const double before = sc->err;
  const double err = n > 0 ? total / (double)n * 100.0 : 0.0;
  sc->iterations = it;
  sc->err_before = before;
  sc->err = err;
  bool stop;
  if (after >= 0) {
    stop = it > after;
  } else {
    stop = it > 2 && err < tde;
    if (!stop && cap > 0 && it >= cap) {
      stop = true;
      sc->status = 2;  // not converged within the cap
    }
  }
  if (stop) sc->converged = 1;
}

// pass B: A_i = dt^2 [a_i . (S_i + bG_i) - sum_j (V_j a_j) . gradW_ij];
// p_i <- max(p_i + omega (s_i - A_i) / a_ii, 0) where a_ii < -eps; the
// residual e_i = |A_i - s_i| where s_i < 0, summed in f64 over all N (last
// block: error, sweep count and the stop test of iisph.rs:378-393).
// AFTER >= 0: stop after AFTER+1 sweeps; AFTER < 0: target density error.
template <class R>
__global__ void __launch_bounds__(kBlock, sizeof(R) == 4 ? 5 : 1) k_sweep_jacobi(
    Scalars* sc, const R4<R>* TB, const R2<R>* SA,
    const R4<R>* xu, const R2<R>* uu, NbrArgs N, R* press,
    R4<R>* xq, double* partials, int after, StepParams<R> P) {
  grid_dep_release();
  __shared__ double sh[32];
  extern __shared__ __align__(32) unsigned char dsm[];
  const HaloView H = halo_view(N);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = sc->n_active;
  const bool act = i < n;
  // fixed during a solve: read before the wait on pass A
  SweepList<R> L;
  L.begin(N, act ? i : 0, act ? min((int)N.ncnt[i], N.K) : 0);
  R4<R> Ti{}, u4{};
  R2<R> u2{}, sa{};
  R p0 = 0;
  if (act) {
    Ti = TB[i];
    sa = SA[i];
  }
  const HaloFirst hf = halo_first(H);
  grid_dep_wait();
  if (sc->converged) return;
  if (act) {
    u4 = xu[i];
    u2 = uu[i];
    p0 = press[i];
  }
  const R4<R> xi{u4.x, u4.y, u4.z, Ti.w};
  R4<R>* s_a = reinterpret_cast<R4<R>*>(dsm);
  R2<R>* s_b = reinterpret_cast<R2<R>*>(s_a + N.hs);
  stage_halo_from(H, hf, [&](int l, uint32_t g) {
    async_copy(&s_a[l], &xu[g]);
    async_copy(&s_b[l], &uu[g]);
  });
  prefetch_ahead(N, n, xu, uu, TB, SA, (const R*)press);
  stage_done();
  double e = 0.0;
  if (act) {
    const R ih = P.k.inv_h;
    R sum = 0;
    auto pair = [&](const R4<R>& a, const R2<R>& b) {
      const R rx = xi.x - a.x, ry = xi.y - a.y, rz = xi.z - a.z;
      sum += grad_third(rx, ry, rz, ih) * (a.w * rx + b.x * ry + b.y * rz);
    };
    if (H.staged) {
      for (int g = 0; g < L.ng; ++g) {
        const uint2 w = L.next(g);
        const uint32_t l0 = w.x & 0xffffu, l1 = w.x >> 16, l2 = w.y & 0xffffu, l3 = w.y >> 16;
        const R4<R> a0 = s_a[l0], a1 = s_a[l1], a2 = s_a[l2], a3 = s_a[l3];
        const R2<R> b0 = s_b[l0], b1 = s_b[l1], b2 = s_b[l2], b3 = s_b[l3];
        pair(a0, b0); pair(a1, b1); pair(a2, b2); pair(a3, b3);
      }
    } else {
      for (int g = 0; g < L.ng; ++g) {
        const uint2 w = L.next(g);
        const uint32_t g0 = H.idx[w.x & 0xffffu], g1 = H.idx[w.x >> 16], g2 = H.idx[w.y & 0xffffu],
                       g3 = H.idx[w.y >> 16];
        const R4<R> a0 = xu[g0], a1 = xu[g1], a2 = xu[g2], a3 = xu[g3];
        const R2<R> b0 = uu[g0], b1 = uu[g1], b2 = uu[g2], b3 = uu[g3];
        pair(a0, b0); pair(a1, b1); pair(a2, b2); pair(a3, b3);
      }
    }
    const R dt = (R)sc->dt;
    const R iV = R(1) / xi.w;
    const R ax = u4.w * iV, ay = u2.x * iV, az = u2.y * iV;
    const R tot = ax * Ti.x + ay * Ti.y + az * Ti.z + R(3) * P.k.cg * sum;  // gradW = -3 cg grad_third r
    const R A = dt * dt * tot;
    const R s = sa.x, aii = sa.y;
    R pn = p0;
    if (aii < -P.min_diag) pn = fmax(p0 + P.omega * (s - A) / aii, R(0));
    press[i] = pn;
    xq[i] = R4<R>{xi.x, xi.y, xi.z, xi.w * pn};
    if (s < R(0)) e = fabs((double)A - (double)s);
  }
  const double bs = block_sum(e, sh);
  double total;
  if (last_block_total(bs, partials, &sc->done_blocks, &total, sh)) end_sweep(sc, total, n, after, P.tde, P.iteration_cap);
}

// ---------------------------------------------------------------------------
// A whole solve in one cooperative launch, for scenes whose blocks are on the
// GPU all at once: the sweeps' passes A and B as above (same operations, same
// order), with a barrier over the grid between them. A particle's own data
// stay in registers; records that other blocks rewrite between two barriers are
// read past L1.
//
// What bounds it: latency (records, lists, barrier, reduction). A sweep as two
// launches takes the launches as well, and either a host that reads the error
// between batches of sweeps or a while-node. KEEP: the lists are copied to shared
// memory once (a warp alone on its scheduler waits for every group read from L2).
// 5 thousand particles: 15 us a sweep; per step of four sweeps against a launch per
// pass 431 -> 151 us stepped by calls and 138 -> 123 us in a graph (8 steps with the
// lists read every sweep 1171 us, kept 997 us, and with u's second records
// requested four at a time 984 us).
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T load_l2(const T* p) {
  T r;
  if constexpr (sizeof(T) == 8) {
    reinterpret_cast<int2&>(r) = __ldcg(reinterpret_cast<const int2*>(p));
  } else {
#pragma unroll
    for (int o = 0; o < (int)(sizeof(T) / 16); ++o)
      reinterpret_cast<int4*>(&r)[o] = __ldcg(reinterpret_cast<const int4*>(p) + o);
  }
  return r;
}

// Four records of a thread, requested before the first is stored.
template <class T>
__device__ __forceinline__ void stage_batch(const HaloView& H, const uint32_t (&g)[4], int l0, const T* src, T* dst) {
  T r[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) r[u] = load_l2(&src[g[u]]);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int l = l0 + u * kBlock + (int)threadIdx.x;
    if (l < H.size) dst[l] = r[u];
  }
}

// Barrier over a cooperative grid. The last block to arrive runs last() (all its
// threads) before it lets the others go. The wait is bounded: a block that gives
// up after `polls` looks sets barrier_timeout and returns false, and so do the
// others in turn. The arrival count is then left as it is, and no solve runs on it
// (k_solve looks at barrier_timeout first) until a restart sets the scalars anew.
constexpr int kBarrierPolls = 1 << 22;  // some seconds
template <class F>
__device__ __forceinline__ bool grid_barrier(Scalars* sc, int polls, F&& last) {
  __shared__ unsigned s_gen;
  __shared__ int s_last, s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    s_gen = *(volatile unsigned*)&sc->barrier_gen;  // (before the arrival: it cannot move on until then)
    __threadfence();
    s_last = atomicAdd(&sc->barrier_count, 1u) == gridDim.x - 1;
    s_ok = 1;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    last();
    __syncthreads();
    if (threadIdx.x == 0) {
      sc->barrier_count = 0;
      __threadfence();
      atomicAdd(&sc->barrier_gen, 1u);
    }
  } else if (threadIdx.x == 0) {
    int looks = 0;
    while (*(volatile unsigned*)&sc->barrier_gen == s_gen) {
      if (++looks >= polls) {
        sc->barrier_timeout = 1;
        s_ok = 0;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return s_ok != 0;
}

// The groups of a particle's neighbor list from shared memory, after SweepList.
struct KeptList {
  const uint2* p;
  int ng;
  __device__ __forceinline__ uint2 next(int g) const { return p[g * 32]; }
};

template <class R, bool KEEP>
__global__ void __launch_bounds__(kBlock, (sizeof(R) == 4 ? 4 : 2) / (KEEP ? 2 : 1)) k_solve(
    Scalars* sc, const R4<R>* __restrict__ TA, const R4<R>* __restrict__ TB, const R2<R>* __restrict__ SA,
    R4<R>* xq, R4<R>* xu, R2<R>* uu, R* press, NbrArgs N, double* partials, int after, int limit, int polls,
    StepParams<R> P) {
  __shared__ double sh[32];
  extern __shared__ __align__(32) unsigned char dsm[];
  // (converged is set between barriers only: every block sees the same. A timeout is an
  // earlier launch's, or another block's that gave up on this one: this one gives up too)
  if (*(volatile int*)&sc->converged || *(volatile int*)&sc->barrier_timeout) return;
  R4<R>* s_a = reinterpret_cast<R4<R>*>(dsm);
  R2<R>* s_b = reinterpret_cast<R2<R>*>(s_a + N.hs);
  const HaloView H = halo_view(N);
  const int i = blockIdx.x * kBlock + threadIdx.x;
  const int n = sc->n_active;
  const bool act = i < n;
  const int cnt = act ? min((int)N.ncnt[i], N.K) : 0;
  const HaloFirst hf = halo_first(H);
  const R dt = (R)sc->dt;
  R4<R> xi{}, Ti{}, Tb{};
  R2<R> sa{};
  R p = 0;
  if (act) {
    xi = xq[i];
    Ti = TA[i];
    Tb = TB[i];
    sa = SA[i];
    p = press[i];
  }
  uint2* s_nbr = reinterpret_cast<uint2*>(s_b + N.hs) + (threadIdx.x >> 5) * 8 * N.K + (threadIdx.x & 31);
  if (KEEP) {
    SweepList<R> L;
    L.begin(N, act ? i : 0, cnt);
    for (int g = 0; g < L.ng; ++g) s_nbr[g * 32] = L.next(g);
  }
  auto list = [&] {
    if constexpr (KEEP) {
      return KeptList{s_nbr, (cnt + 3) >> 2};
    } else {
      SweepList<R> L;
      L.begin(N, act ? i : 0, cnt);
      return L;
    }
  };
  const R ih = P.k.inv_h;
  for (int sweep = 0; sweep < limit; ++sweep) {
    // pass A
    R4<R> u4{};
    R2<R> u2{};
    {
      auto L = list();
      stage_halo_from(H, hf, [&](int l, uint32_t g) { async_copy(&s_a[l], &xq[g]); });
      stage_done();
      if (act) {
        R px = 0, py = 0, pz = 0;
        auto pair = [&](const R4<R>& r) {
          const R rx = xi.x - r.x, ry = xi.y - r.y, rz = xi.z - r.z;
          const R t = r.w * grad_third_close(rx, ry, rz, ih);
          px += t * rx; py += t * ry; pz += t * rz;
        };
        if (H.staged)
          sweep_groups(L, [&](uint32_t l) { return s_a[l]; }, pair);
        else
          sweep_groups(L, [&](uint32_t l) { return load_l2(&xq[H.idx[l]]); }, pair);
        const R cg = R(-3) * P.k.cg;
        const R fx = p * Ti.x + cg * px, fy = p * Ti.y + cg * py, fz = p * Ti.z + cg * pz;
        const R c = Ti.w;
        u4 = R4<R>{xi.x, xi.y, xi.z, c * fx};
        u2 = R2<R>{c * fy, c * fz};
        xu[i] = u4;
        uu[i] = u2;
      }
    }
    if (!grid_barrier(sc, polls, [] {})) return;
    // pass B
    double e = 0.0;
    {
      auto L = list();
      stage_halo_from(H, hf, [&](int l, uint32_t g) { async_copy(&s_a[l], &xu[g]); });
      // (f32: eight-byte records, for which cp.async has no form past L1)
      if constexpr (sizeof(R2<R>) == 16) {
        stage_halo_from(H, hf, [&](int l, uint32_t g) { async_copy(&s_b[l], &uu[g]); });
      } else if (H.staged) {
        stage_batch(H, hf.g, 0, uu, s_b);
        for (int l0 = 4 * kBlock; l0 < H.size; l0 += 4 * kBlock) {
          uint32_t g[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int l = l0 + u * kBlock + (int)threadIdx.x;
            g[u] = l < H.size ? __ldg(H.idx + l) : 0u;
          }
          stage_batch(H, g, l0, uu, s_b);
        }
      }
      stage_done();
      if (act) {
        R sum = 0;
        struct Rec {
          R4<R> a;
          R2<R> b;
        };
        auto pair = [&](const Rec& d) {
          const R rx = xi.x - d.a.x, ry = xi.y - d.a.y, rz = xi.z - d.a.z;
          sum += grad_third(rx, ry, rz, ih) * (d.a.w * rx + d.b.x * ry + d.b.y * rz);
        };
        if (H.staged)
          sweep_groups(L, [&](uint32_t l) { return Rec{s_a[l], s_b[l]}; }, pair);
        else
          sweep_groups(L, [&](uint32_t l) { const uint32_t g = H.idx[l]; return Rec{load_l2(&xu[g]), load_l2(&uu[g])}; }, pair);
        const R iV = R(1) / Tb.w;
        const R ax = u4.w * iV, ay = u2.x * iV, az = u2.y * iV;
        const R tot = ax * Tb.x + ay * Tb.y + az * Tb.z + R(3) * P.k.cg * sum;
        const R A = dt * dt * tot;
        const R s = sa.x, aii = sa.y;
        R pn = p;
        if (aii < -P.min_diag) pn = fmax(p + P.omega * (s - A) / aii, R(0));
        p = pn;
        xq[i] = R4<R>{xi.x, xi.y, xi.z, Tb.w * pn};
        if (s < R(0)) e = fabs((double)A - (double)s);
      }
    }
    const double bs = block_sum(e, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
    const bool ok = grid_barrier(sc, polls, [&] {  // (the sum of last_block_total)
      double t = 0;
      for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) t += ((volatile double*)partials)[b];
      t = block_sum(t, sh);
      if (threadIdx.x == 0) end_sweep(sc, t, n, after, P.tde, P.iteration_cap);
    });
    if (!ok) return;
    if (*(volatile int*)&sc->converged) break;
  }
  if (act) press[i] = p;
}

// IISPHwOST between the solves: v* += dt a_p1 (iisph_optimized_source_term.rs:97-110)
template <class R>
__global__ void __launch_bounds__(kBlock) k_ost_predict(Scalars* __restrict__ sc,
                                                       const R4<R>* __restrict__ acc,
                                                       R4<R>* __restrict__ vstar) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    sc->iterations_eqs1 = sc->iterations;
    sc->iterations = 0;
    sc->converged = 0;
    sc->err = INFINITY;
  }
  if (i >= sc->n_active) return;
  const R dt = (R)sc->dt;
  const R4<R> a = acc[i];
  R4<R> v = vstar[i];
  v.x += dt * a.x; v.y += dt * a.y; v.z += dt * a.z;
  vstar[i] = v;
}

// IISPHwOST commit: x_pred = x + dt v*, x_new = x_pred + dt^2 a, v_new = v* + dt a
// into the integrator slots (iisph_optimized_source_term.rs:139-216).
template <class R>
__global__ void __launch_bounds__(kBlock) k_ost_commit(const Scalars* __restrict__ sc,
                                                      const R4<R>* __restrict__ xv,
                                                      const R4<R>* __restrict__ vel,
                                                      const R4<R>* __restrict__ vstar,
                                                      const R4<R>* __restrict__ acc,
                                                      R4<R>* __restrict__ xint,
                                                      R4<R>* __restrict__ vint) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= sc->n_active) return;
  const R dt = (R)sc->dt;
  const R dt2 = dt * dt;
  const R4<R> x = xv[i], v = vstar[i], a = acc[i];
  const R xpx = x.x + dt * v.x, xpy = x.y + dt * v.y, xpz = x.z + dt * v.z;
  xint[i] = R4<R>{xpx + dt2 * a.x, xpy + dt2 * a.y, xpz + dt2 * a.z, R(0)};
  vint[i] = R4<R>{v.x + dt * a.x, v.y + dt * a.y, v.z + dt * a.z, vel[i].w};
}

// SESPHwSplitting predicted density (sesph_with_splitting.rs:90-152) and the
// state equation: rho* = sum_j [m_j W + dt (v*_i - v*_j) . gradW]
//                      + (m_i/V0) bW + dt v*_i . bGu, p = k max(V0/(m_i/rho*) - 1, 0)
template <class R, int NB>
__global__ void __launch_bounds__(kBlock) k_split_density(
    const Scalars* sc, const R4<R>* xv, const R4<R>* vel,
    const R4<R>* vstar, NbrArgs N, BoundaryArgs<R> B, R* press,
    R* rho_pred, StepParams<R> P) {
  grid_dep_begin();
  extern __shared__ __align__(32) unsigned char dsm[];
  const HaloView H = halo_view(N);
  // records {x, V} and {v*, m} (the acceleration pass stores m in v*.w)
  R4<R>* s_x = staged_vec<R>(dsm, N.hs, 0);
  R4<R>* s_v = staged_vec<R>(dsm, N.hs, 1);
  if (H.staged)
    stage_halo(H, [&](int l, uint32_t g) {
      async_copy(&s_x[l], &xv[g]);
      async_copy(&s_v[l], &vstar[g]);
    });
  stage_done();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= sc->n_active) return;
  const R dt = (R)sc->dt;
  const R4<R> xi = xv[i];
  const R4<R> vsi = vstar[i];
  const R mi = vsi.w;
  R rho = mi * P.k.cw * R(0.5), comp = 0;  // self term m_i W(0)
  const int cnt = min((int)N.ncnt[i], N.K);
  for_each_neighbor<NB>(
      N.nbr, N.K, i, cnt,
      [&](uint32_t l) {
        if (H.staged) return XV<R>{s_x[l], s_v[l]};
        const uint32_t g = H.idx[l];
        return XV<R>{xv[g], vstar[g]};
      },
      [&](const XV<R>& d) {
        const R4<R>& xj = d.x;
        const R4<R>& vsj = d.v;
        const R rx = xi.x - xj.x, ry = xi.y - xj.y, rz = xi.z - xj.z;
        R w, f;
        kernel_w_and_grad(rx * rx + ry * ry + rz * rz, P.k, w, f);
        const R t = vsj.w * w + dt * f * ((vsi.x - vsj.x) * rx + (vsi.y - vsj.y) * ry + (vsi.z - vsj.z) * rz);
        kahan_add(rho, comp, t);
      });
  if (B.kind != 0) {
    const R4<R> gu = B.bGu[i];
    rho += B.bW[i] * mi / P.V0 + dt * (vsi.x * gu.x + vsi.y * gu.y + vsi.z * gu.z);
  }
  rho_pred[i] = rho;
  const R vol = mi / rho;
  press[i] = P.stiffness * fmax(P.V0 / vol - R(1), R(0));
}

// ---------------------------------------------------------------------------
// 9. volumes (quantities.rs:14-61) from the kernel sums and the boundary's
//    share, with the average density after the update (sph/mod.rs:444-486);
//    measurement sums (density error, kinetic energy) in f64
// ---------------------------------------------------------------------------
// The last block also sets up the next update's scalars, leaving the particles
// that entered this one and those it disabled in n_in and n_disabled (nothing
// after the sort reads n, n_below or max_speed).
template <class R>
__global__ void __launch_bounds__(kBlock) k_volume(Scalars* sc, R4<R>* xv,
                                                  const R4<R>* vel, const R* bW,
                                                  int has_boundary, double* partials,
                                                  StepParams<R> P) {
  grid_dep_begin();
  __shared__ double sh[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = sc->n_active;
  double d = 0.0;
  if (i < n) {
    const R sum = xv[i].w;
    R denom = P.V0 * sum;
    if (has_boundary) denom += bW[i];
    const R Vr = P.V0 / denom;
    xv[i].w = Vr;
    const double V = (double)Vr, m = (double)vel[i].w, V0 = (double)P.V0;
    d = V < V0 ? m / V : m / V0;
  }
  double total;
  if (last_block_total(block_sum(d, sh), partials, &sc->done_blocks, &total, sh)) {
    sc->avg_density = n > 0 ? total / (double)n : 0.0;
    sc->n_in = sc->n;
    sc->n_disabled = sc->n_below;
    sc->n = n;
    sc->n_below = 0;
    sc->max_speed = 0;
  }
}

// out[0] = sum (V < V0 ? V0/V : 1), out[1] = sum 1/2 m |v|^2
template <class R>
__global__ void __launch_bounds__(kBlock) k_measure(Scalars* __restrict__ sc,
                                                   const R4<R>* __restrict__ xv,
                                                   const R4<R>* __restrict__ vel,
                                                   double* __restrict__ partials,
                                                   double* __restrict__ out, StepParams<R> P) {
  __shared__ double sh[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = sc->n_active;
  double de = 0.0, ke = 0.0;
  if (i < n) {
    const double V = (double)xv[i].w, V0 = (double)P.V0;
    de = V < V0 ? V0 / V : 1.0;
    const R4<R> v = vel[i];
    const double vx = v.x, vy = v.y, vz = v.z;
    ke = 0.5 * (double)v.w * ((vx * vx + vy * vy) + vz * vz);
  }
  const double b0 = block_sum(de, sh);
  const double b1 = block_sum(ke, sh);
  // one completion counter for both sums
  __shared__ bool is_last;
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = b0;
    partials[gridDim.x + blockIdx.x] = b1;
    __threadfence();
    is_last = atomicAdd(&sc->done_blocks, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  double s0 = 0, s1 = 0;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
    s0 += ((volatile double*)partials)[b];
    s1 += ((volatile double*)partials)[gridDim.x + b];
  }
  s0 = block_sum(s0, sh);
  s1 = block_sum(s1, sh);
  if (threadIdx.x == 0) {
    out[0] = s0;
    out[1] = s1;
    sc->done_blocks = 0;
  }
}

// ---------------------------------------------------------------------------
// 10. rigid bodies (f64)
// ---------------------------------------------------------------------------
// Gravity on dynamic bodies: F += m g at the center of mass
// (non_pressure_accelerations.rs:79-100, static_sample_boundary.rs:328-341).
__global__ void k_body_gravity(Body* bodies, int nb, int mode, double gx, double gy, double gz) {
  const int b = threadIdx.x;
  if (b >= nb || !bodies[b].dynamic) return;
  Body& B = bodies[b];
  double a[3];
  if (mode == 0) {
    a[0] = 0.0; a[1] = 0.0; a[2] = -9.81;
  } else {
    const double d[3] = {gx - B.com[0], gy - B.com[1], gz - B.com[2]};
    const double dist = sqrt(((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]) + 1e-4);
    for (int c = 0; c < 3; ++c) a[c] = 9.81 * d[c] / dist;
  }
  for (int c = 0; c < 3; ++c) B.F[c] += a[c] * B.mass;
}

// Fixed-order sum of per-block reaction partials into the body accumulators.
__global__ void k_body_reduce(Body* bodies, int nb, const double* partials, int nblocks) {
  const int b = blockIdx.x;
  if (b >= nb || !bodies[b].dynamic) return;
  __shared__ double sh[32];
  for (int c = 0; c < 6; ++c) {
    double s = 0.0;
    for (int k = threadIdx.x; k < nblocks; k += blockDim.x)
      s += partials[(size_t)k * kMaxBodies * 6 + b * 6 + c];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) {
      if (c < 3) bodies[b].F[c] += s;
      else bodies[b].T[c - 3] += s;
    }
    __syncthreads();
  }
}

__device__ void mat_rot(const double q[4], double R_[9]) {
  const double ww = q[0] * q[0], ii = q[1] * q[1], jj = q[2] * q[2], kk = q[3] * q[3];
  const double ij = q[1] * q[2] * 2.0, wk = q[0] * q[3] * 2.0, wj = q[0] * q[2] * 2.0;
  const double ik = q[1] * q[3] * 2.0, jk = q[2] * q[3] * 2.0, wi = q[0] * q[1] * 2.0;
  R_[0] = ww + ii - jj - kk; R_[1] = ij - wk; R_[2] = wj + ik;
  R_[3] = wk + ij; R_[4] = ww - ii + jj - kk; R_[5] = jk - wi;
  R_[6] = ik - wj; R_[7] = wi + jk; R_[8] = ww - ii - jj + kk;
}
__device__ void body_update_derived(Body& B) {
  double Rm[9], t[9];
  mat_rot(B.q, Rm);
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c)
      t[r * 3 + c] = (Rm[r * 3 + 0] * B.inv_inertia_body[0 * 3 + c] +
                      Rm[r * 3 + 1] * B.inv_inertia_body[1 * 3 + c]) +
                     Rm[r * 3 + 2] * B.inv_inertia_body[2 * 3 + c];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c)
      B.inv_inertia_world[r * 3 + c] =
          (t[r * 3 + 0] * Rm[c * 3 + 0] + t[r * 3 + 1] * Rm[c * 3 + 1]) + t[r * 3 + 2] * Rm[c * 3 + 2];
  for (int r = 0; r < 3; ++r)
    B.omega[r] = (B.inv_inertia_world[r * 3 + 0] * B.L[0] + B.inv_inertia_world[r * 3 + 1] * B.L[1]) +
                 B.inv_inertia_world[r * 3 + 2] * B.L[2];
}

// Euler-Cromer body step with q <- exp(omega dt / 2) q (rigid_body_motion.rs:183-201).
__global__ void k_body_step(Body* bodies, int nb, const Scalars* sc) {
  const int b = threadIdx.x;
  if (b >= nb || !bodies[b].dynamic) return;
  Body& B = bodies[b];
  const double dt = sc->dt;
  for (int c = 0; c < 3; ++c) {
    const double a = B.F[c] / B.mass;
    B.v[c] += a * dt;
  }
  for (int c = 0; c < 3; ++c) B.com[c] += B.v[c] * dt;
  for (int c = 0; c < 3; ++c) B.L[c] += B.T[c] * dt;
  for (int r = 0; r < 3; ++r)
    B.omega[r] = (B.inv_inertia_world[r * 3 + 0] * B.L[0] + B.inv_inertia_world[r * 3 + 1] * B.L[1]) +
                 B.inv_inertia_world[r * 3 + 2] * B.L[2];
  const double h[3] = {B.omega[0] * dt / 2.0, B.omega[1] * dt / 2.0, B.omega[2] * dt / 2.0};
  const double nn = (h[0] * h[0] + h[1] * h[1]) + h[2] * h[2];
  double e[4] = {1.0, 0.0, 0.0, 0.0};
  if (nn > DBL_EPSILON * DBL_EPSILON) {
    const double nrm = sqrt(nn), s = sin(nrm) / nrm;
    e[0] = cos(nrm); e[1] = h[0] * s; e[2] = h[1] * s; e[3] = h[2] * s;
  }
  const double* q = B.q;
  const double nq[4] = {e[0] * q[0] - e[1] * q[1] - e[2] * q[2] - e[3] * q[3],
                        e[0] * q[1] + e[1] * q[0] + e[2] * q[3] - e[3] * q[2],
                        e[0] * q[2] - e[1] * q[3] + e[2] * q[0] + e[3] * q[1],
                        e[0] * q[3] + e[1] * q[2] - e[2] * q[1] + e[3] * q[0]};
  for (int c = 0; c < 4; ++c) B.q[c] = nq[c];
  for (int c = 0; c < 3; ++c) { B.F[c] = 0.0; B.T[c] = 0.0; }
  body_update_derived(B);
}

// World positions/velocities of dynamic sample-boundary samples
// (static_sample_boundary.rs:392-412): x = R x_body + c, v = v + omega x (x - c).
template <class R>
__global__ void __launch_bounds__(kBlock) k_body_samples(const int* __restrict__ n_ptr,
                                                        const Body* __restrict__ bodies,
                                                        const R4<R>* __restrict__ x_body,
                                                        const uint32_t* __restrict__ orig,
                                                        const uint32_t* __restrict__ bid,
                                                        R4<R>* __restrict__ xb,
                                                        R4<R>* __restrict__ vb) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= *n_ptr) return;
  const Body& B = bodies[bid[d]];
  if (!B.dynamic) return;
  const R4<R> xl = x_body[orig[d]];
  const double pl[3] = {(double)xl.x, (double)xl.y, (double)xl.z};
  double pw[3];
  qrot(B.q, pl, pw);
  for (int c = 0; c < 3; ++c) pw[c] += B.com[c];
  double vw[3];
  body_velocity_at(B, pw, vw);
  const R V = xb[d].w;
  xb[d] = R4<R>{(R)pw[0], (R)pw[1], (R)pw[2], V};
  vb[d] = R4<R>{(R)vw[0], (R)vw[1], (R)vw[2], R(0)};
}

// Boundary pseudo-volumes V_b = gamma_V / sum_{b' same boundary} W_bb'
// (static_sample_boundary.rs:354-390), on the sorted sample grid.
template <class R>
__global__ void __launch_bounds__(kBlock) k_sample_volumes(const int* __restrict__ n_ptr,
                                                          SampleGrid<R> G, R4<R>* __restrict__ xb,
                                                          double gamma_v, StepParams<R> P) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= *n_ptr) return;
  const R4<R> xi = G.xb[d];
  const uint32_t myb = G.bid[d];
  const int cx = cell_coord((double)xi.x, P.range), cy = cell_coord((double)xi.y, P.range),
            cz = cell_coord((double)xi.z, P.range);
  R sum = 0, comp = 0;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const uint32_t k = morton_key(cx + dx, cy + dy, cz + dz, G.mask);
        const uint32_t b = G.start[k], e = G.start[k + 1];
        for (uint32_t s = b; s < e; ++s) {
          if (G.bid[s] != myb) continue;
          const R4<R> xs = G.xb[s];
          if (!in_range(xi, xs, P.range, P.range2_lo, P.range2_hi)) continue;
          const R rx = xi.x - xs.x, ry = xi.y - xs.y, rz = xi.z - xs.z;
          kahan_add(sum, comp, kernel_w_r2(rx * rx + ry * ry + rz * rz, P.k));
        }
      }
  R4<R> o = xi;
  o.w = (R)(gamma_v / (double)sum);
  xb[d] = o;
}

// ---------------------------------------------------------------------------
// graph-captured stepping
// ---------------------------------------------------------------------------
// Opens a chunk of graph launches: simulated time enters, flags clear.
__global__ void k_chunk_begin(Scalars* sc, double time) {
  sc->time_acc = time;
  sc->trouble = 0;
  sc->status_any = 0;
  sc->loop_sweeps = 0;
  sc->chunk_max_nbrs = 0;
  sc->chunk_max_halo = 0;
}

// Condition of the while-node that runs the Jacobi sweeps of one solve: go on
// until the sweep kernel sets `converged` or `limit` sweeps have run. Every
// body execution either finds `converged` set or adds one to `iterations`,
// so the loop ends after at most `limit` bodies.
__global__ void k_loop_cond(cudaGraphConditionalHandle h, const Scalars* sc, int limit) {
  grid_dep_wait();
  const unsigned int more = (!sc->converged && sc->iterations < limit) ? 1u : 0u;
  cudaGraphSetConditional(h, more);
}

// End of a graph-captured step: records what the per-step host check would
// have acted on (then the host replays the chunk on the per-step path).
__global__ void k_step_epilogue(Scalars* sc, int K, int hcap, int solver_loop) {
  unsigned int t = 0;
  if (sc->max_nbrs > K || sc->max_halo > hcap) t |= 1u;
  sc->chunk_max_nbrs = max(sc->chunk_max_nbrs, sc->max_nbrs);
  sc->chunk_max_halo = max(sc->chunk_max_halo, sc->max_halo);
  if (sc->n_disabled > 0) t |= 2u;
  if (solver_loop && !sc->converged) t |= 4u;
  sc->trouble |= t;
  if (sc->status == 2) sc->status_any = 2;
  if (solver_loop) sc->loop_sweeps += (unsigned long long)sc->iterations;
}

// ---------------------------------------------------------------------------
// Rigid-rigid contact of volume-map bodies (volume_map_boundary.rs:55-1102,
// 1440-1453), run before the body step. k_contact_tasks cuts the overlap of
// every pair of world bounding boxes (at least one body dynamic) into
// sub-cells; k_contact_build evaluates one sub-cell per block, one 8^3
// Gauss-Legendre point per thread, and reduces the contact cell's volume,
// center and unit force/torque sensitivities (build_contact_cell and
// compute_diagonal); k_contact_solve runs the NNCG-accelerated projected
// Jacobi iteration for all cells in one block and adds the contact forces
// and torques to the bodies. Everything is f64.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool vm_phi(const VMDesc& D, const Body* bodies, const double p[3], double& phi) {
  double pl[3] = {p[0], p[1], p[2]};
  if (D.body >= 0) body_world_to_local(bodies[D.body], p, pl);
  return ser_function(D.sdf, pl[0], pl[1], pl[2], phi);
}
__device__ __forceinline__ bool vm_phi_grad(const VMDesc& D, const Body* bodies, const double p[3], double g[3]) {
  double pl[3] = {p[0], p[1], p[2]};
  if (D.body >= 0) body_world_to_local(bodies[D.body], p, pl);
  if (!ser_gradient(D.sdf, pl[0], pl[1], pl[2], g)) return false;
  if (D.body >= 0) {
    double gw[3];
    qrot(bodies[D.body].q, g, gw);
    g[0] = gw[0]; g[1] = gw[1]; g[2] = gw[2];
  }
  return true;
}

// cubic_extension_fn and its derivative (:1717-1745): the cubic spline's
// W(x) / W(0) on (0, h), 1 below and 0 above.
__device__ __forceinline__ double cubic_ext(double x, double h) {
  if (x >= h) return 0.;
  if (x <= 0.) return 1.;
  const double q = x / h, a = fmax(1. - q, 0.), b = fmax(0.5 - q, 0.);
  const double c = 16. / 3.14159265358979323846 / (h * h * h);
  return (c * (a * a * a - 4. * (b * b * b))) / (c * 0.5);
}
__device__ __forceinline__ double cubic_ext_derivative(double x, double h) {
  if (x >= h || x <= 0.) return 0.;
  const double q = x / h, a = fmax(1. - q, 0.), b = fmax(0.5 - q, 0.);
  const double alpha = 16. / 3.14159265358979323846;
  const double c4 = alpha / (h * h * h * h);
  return (((c4 * x) / x) * (-3. * (a * a) + 12. * (b * b))) / (alpha / (h * h * h) * 0.5);
}

// World bounding box (BoundaryType::world_aabb, :2122-2151).
__device__ void vm_world_box(const VMDesc& D, const Body* bodies, double lo[3], double hi[3]) {
  if (D.body < 0) {
    for (int d = 0; d < 3; ++d) {
      lo[d] = D.aabb_c[d] - D.aabb_h[d];
      hi[d] = D.aabb_c[d] + D.aabb_h[d];
    }
    return;
  }
  const Body& B = bodies[D.body];
  double Rm[9], c[3];
  mat_rot(B.q, Rm);
  qrot(B.q, D.aabb_c, c);
  for (int d = 0; d < 3; ++d) {
    const double he = (fabs(Rm[d * 3]) * D.aabb_h[0] + fabs(Rm[d * 3 + 1]) * D.aabb_h[1]) +
                      fabs(Rm[d * 3 + 2]) * D.aabb_h[2];
    const double cw = c[d] + B.com[d];
    lo[d] = cw - he;
    hi[d] = cw + he;
  }
}

// broad_phase (:70-96) and the task list of generate_contact_cells
// (:98-117) with subdivide_overlap (:1813-1844); one thread.
__global__ void k_contact_tasks(const VMDesc* __restrict__ vms, const Body* __restrict__ bodies, int nb,
                                double target, ContactPair* __restrict__ pairs, ContactScalars* __restrict__ cs,
                                int task_cap) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int np = 0, nt = 0, overflow = 0;
  for (int i = 0; i < nb; ++i) {
    if (!vms[i].has_aabb) continue;
    double li[3], hi_[3];
    vm_world_box(vms[i], bodies, li, hi_);
    for (int j = i + 1; j < nb; ++j) {
      if (!vms[j].has_aabb) continue;
      if (vms[i].body < 0 && vms[j].body < 0) continue;
      double lj[3], hj[3];
      vm_world_box(vms[j], bodies, lj, hj);
      bool overlap = true;
      for (int d = 0; d < 3; ++d) overlap = overlap && li[d] <= hj[d] && hi_[d] >= lj[d];
      if (!overlap) continue;
      double mn[3], mx[3];
      bool inter = true;
      for (int d = 0; d < 3; ++d) {
        mn[d] = fmax(li[d], lj[d]);
        mx[d] = fmin(hi_[d], hj[d]);
        inter = inter && mn[d] <= mx[d];
      }
      if (!inter) continue;
      ContactPair P;
      P.a = i;
      P.b = j;
      double cnt = 1.0;
      for (int d = 0; d < 3; ++d) {
        const double ext = mx[d] - mn[d];
        const double nd = fmax(ceil(ext / target), 1.0);
        cnt *= nd;
        P.n[d] = nd < 1e7 ? (int)nd : 10000000;
        P.min[d] = mn[d];
      }
      if (cnt > (double)(task_cap - nt)) {
        overflow = 1;
        continue;
      }
      for (int d = 0; d < 3; ++d) P.cs[d] = (mx[d] - mn[d]) / (double)P.n[d];
      P.first = nt;
      pairs[np++] = P;
      nt += P.n[0] * P.n[1] * P.n[2];
    }
  }
  cs->npairs = np;
  cs->ntasks = nt;
  cs->ncells = 0;
  cs->iterations = 0;
  cs->overflow = overflow;
  cs->capped = 0;
}

// build_contact_cell (:700-782) and compute_diagonal (:835-926): block per
// sub-cell, thread per quadrature point (x slowest, z fastest as
// quadrature_points orders them).
constexpr int kContactThreads = kContactQuad * kContactQuad * kContactQuad;
__global__ void __launch_bounds__(kContactThreads) k_contact_build(
    const VMDesc* __restrict__ vms, const Body* __restrict__ bodies, const ContactPair* __restrict__ pairs,
    const ContactScalars* __restrict__ cs, ContactCell* __restrict__ cells, ContactGL gl, double h,
    const Scalars* __restrict__ sc) {
  __shared__ double red[kContactThreads / 32][17];
  __shared__ double tot[17];
  __shared__ int go;
  const int ntasks = cs->ntasks, npairs = cs->npairs;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
    int pi = 0;
    while (pi + 1 < npairs && pairs[pi + 1].first <= t) ++pi;
    const ContactPair P = pairs[pi];
    const int local = t - P.first;
    const int idx[3] = {local % P.n[0], (local / P.n[0]) % P.n[1], local / (P.n[0] * P.n[1])};
    double from[3], dd[3], half[3], center[3];
    for (int d = 0; d < 3; ++d) {
      from[d] = P.min[d] + (double)idx[d] * P.cs[d];
      dd[d] = (from[d] + P.cs[d]) - from[d];
      half[d] = dd[d] * 0.5;
      center[d] = from[d] + half[d];
    }
    const VMDesc& A = vms[P.a];
    const VMDesc& B = vms[P.b];
    if (threadIdx.x == 0) {
      // pruning (:128-159): both solids within twice the half diagonal
      const double bound = 2.0 * (sqrt((dd[0] * dd[0] + dd[1] * dd[1]) + dd[2] * dd[2]) * 0.5);
      double pa, pb;
      const bool oka = vm_phi(A, bodies, center, pa);
      const bool okb = vm_phi(B, bodies, center, pb);
      go = oka && okb && pa - bound < 0. && pb - bound < 0.;
      if (!go) cells[t].valid = 0;
    }
    __syncthreads();
    if (!go) {
      __syncthreads();
      continue;
    }
    const int q = threadIdx.x;
    const int i = q >> 6, j = (q >> 3) & 7, k = q & 7;
    const double pos[3] = {center[0] + gl.x[i] * half[0], center[1] + gl.x[j] * half[1],
                           center[2] + gl.x[k] * half[2]};
    const double w = gl.w[i] * gl.w[j] * gl.w[k] * half[0] * half[1] * half[2];
    // 0 count, 1 volume, 2-4 x V, 5-7 f_a, 8-10 tau_a, 11-13 f_b, 14-16 tau_b
    double v[17];
    for (int c = 0; c < 17; ++c) v[c] = 0.0;
    double pa, pb, ga[3], gb[3];
    if (vm_phi(A, bodies, pos, pa) && vm_phi(B, bodies, pos, pb)) {
      const double sa = cubic_ext(2.0 * pa + h, h), sb = cubic_ext(2.0 * pb + h, h);
      if (sa > 0.0 && sb > 0.0 && vm_phi_grad(A, bodies, pos, ga) && vm_phi_grad(B, bodies, pos, gb)) {
        const double spa = 2.0 * cubic_ext_derivative(2.0 * pa + h, h);
        const double spb = 2.0 * cubic_ext_derivative(2.0 * pb + h, h);
        const double wg = w * sa * sb, wa = w * spa * sb, wb = w * spb * sa;
        v[0] = 1.0;
        v[1] = wg;
        for (int d = 0; d < 3; ++d) {
          v[2 + d] = wg * pos[d];
          v[5 + d] = wa * ga[d];
          v[11 + d] = wb * gb[d];
        }
        if (A.body >= 0) {
          const double* c = bodies[A.body].com;
          const double r[3] = {pos[0] - c[0], pos[1] - c[1], pos[2] - c[2]};
          v[8] = wa * (r[1] * ga[2] - r[2] * ga[1]);
          v[9] = wa * (r[2] * ga[0] - r[0] * ga[2]);
          v[10] = wa * (r[0] * ga[1] - r[1] * ga[0]);
        }
        if (B.body >= 0) {
          const double* c = bodies[B.body].com;
          const double r[3] = {pos[0] - c[0], pos[1] - c[1], pos[2] - c[2]};
          v[14] = wb * (r[1] * gb[2] - r[2] * gb[1]);
          v[15] = wb * (r[2] * gb[0] - r[0] * gb[2]);
          v[16] = wb * (r[0] * gb[1] - r[1] * gb[0]);
        }
      }
    }
    for (int c = 0; c < 17; ++c) {
      const double s = warp_sum(v[c]);
      if (lane == 0) red[warp][c] = s;
    }
    __syncthreads();
    if (warp == 0) {
      for (int c = 0; c < 17; ++c) {
        double s = lane < kContactThreads / 32 ? red[lane][c] : 0.0;
        s = warp_sum(s);
        if (lane == 0) tot[c] = s;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      ContactCell& C = cells[t];
      const double vol = tot[1];
      if (!(vol > 0.0) || tot[0] == 0.0) {
        C.valid = 0;
      } else {
        const double dt = sc->dt;
        C.valid = 1;
        C.a = P.a;
        C.b = P.b;
        C.volume = vol;
        for (int d = 0; d < 3; ++d) {
          C.center[d] = tot[2 + d] / vol;
          C.f_a[d] = tot[5 + d];
          C.tau_a[d] = tot[8 + d];
          C.f_b[d] = tot[11 + d];
          C.tau_b[d] = tot[14 + d];
        }
        const double fn = fmax(sqrt((C.f_a[0] * C.f_a[0] + C.f_a[1] * C.f_a[1]) + C.f_a[2] * C.f_a[2]), 1e-15);
        const double nrm[3] = {C.f_a[0] / fn, C.f_a[1] / fn, C.f_a[2] / fn};
        for (int r = 0; r < 3; ++r)
          for (int c = 0; c < 3; ++c) C.tproj[r * 3 + c] = (r == c ? 1.0 : 0.0) - nrm[r] * nrm[c];
        double acc_p = 0.0, T[9];
        for (int e = 0; e < 9; ++e) T[e] = 0.0;
        for (int side = 0; side < 2; ++side) {
          const VMDesc& D = side ? B : A;
          if (D.body < 0) continue;
          const Body& M = bodies[D.body];
          const double* f = side ? C.f_b : C.f_a;
          const double* tq = side ? C.tau_b : C.tau_a;
          const double* I = M.inv_inertia_world;
          double It[3];
          for (int r = 0; r < 3; ++r) It[r] = (I[r * 3] * tq[0] + I[r * 3 + 1] * tq[1]) + I[r * 3 + 2] * tq[2];
          acc_p += ((f[0] * f[0] + f[1] * f[1]) + f[2] * f[2]) / M.mass + ((tq[0] * It[0] + tq[1] * It[1]) + tq[2] * It[2]);
          // I / m - [r]x I^-1 [r]x with r = center - com
          const double r[3] = {C.center[0] - M.com[0], C.center[1] - M.com[1], C.center[2] - M.com[2]};
          const double X[9] = {0.0, -r[2], r[1], r[2], 0.0, -r[0], -r[1], r[0], 0.0};
          double XI[9], XIX[9];
          for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b)
              XI[a * 3 + b] = (X[a * 3] * I[b] + X[a * 3 + 1] * I[3 + b]) + X[a * 3 + 2] * I[6 + b];
          for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b)
              XIX[a * 3 + b] = (XI[a * 3] * X[b] + XI[a * 3 + 1] * X[3 + b]) + XI[a * 3 + 2] * X[6 + b];
          for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) T[a * 3 + b] += (a == b ? 1.0 / M.mass : 0.0) - XIX[a * 3 + b];
        }
        C.acc_p = dt * dt * acc_p;
        double tr = 0.0;
        for (int a = 0; a < 3; ++a) {
          const double row = ((dt * C.tproj[a * 3]) * T[a] + (dt * C.tproj[a * 3 + 1]) * T[3 + a]) +
                             (dt * C.tproj[a * 3 + 2]) * T[6 + a];
          tr += row;
        }
        C.acc_f = 1. / 3. * tr;
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ double block_sum_all(double v, double* sh, double* out) {
  const double t = block_sum(v, sh);
  if (threadIdx.x == 0) *out = t;
  __syncthreads();
  const double r = *out;
  __syncthreads();
  return r;
}

// solve_for_p_c (:186-645) with accumulate_extra_forces (:928-965),
// compute_trial_velocities (:967-994), predicted_volume_error (:996-1009),
// predicted_tangential_velocity (:1011-1033), projected_jacobi (:1035-1102)
// and mean_fischer_burmeister (utilities/mod.rs:27-41); one block of 1024
// threads, warp b gathering body b's cells. The reference iterates until the
// merits converge; here at most `sweep_cap` sweeps run (`capped` is set).
constexpr int kContactSolveThreads = 1024;
__global__ void __launch_bounds__(kContactSolveThreads) k_contact_solve(
    Body* __restrict__ bodies, int nb, const ContactCell* __restrict__ cells, ContactScalars* __restrict__ cs,
    int* __restrict__ cell_idx, ContactState* __restrict__ st, const Scalars* __restrict__ sc, int sweep_cap,
    int fixed_sweeps) {
  constexpr double kMu = 0.5, kOmega = 0.5, kMinDiag = 1e-35, kTolP = 1e-6, kTolF = 1e-3;
  __shared__ double sh[32];
  __shared__ double bc;
  __shared__ int scan[32];
  __shared__ int base;
  __shared__ double ef[kMaxBodies][3], et[kMaxBodies][3], vt[kMaxBodies][3], wt[kMaxBodies][3];
  __shared__ int nact[kMaxBodies];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthreads = blockDim.x;
  const double dt = sc->dt;
  const int ntasks = cs->ntasks;
  // valid cells in task order
  if (tid == 0) base = 0;
  __syncthreads();
  for (int c0 = 0; c0 < ntasks; c0 += nthreads) {
    const int t = c0 + tid;
    const int f = (t < ntasks && cells[t].valid) ? 1 : 0;
    int x = f;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) scan[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int y = lane < nthreads / 32 ? scan[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int z = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += z;
      }
      scan[lane] = y;
    }
    __syncthreads();
    const int before = (warp ? scan[warp - 1] : 0) + x - f;
    if (f) cell_idx[base + before] = t;
    __syncthreads();
    if (tid == 0) base += scan[nthreads / 32 - 1];
    __syncthreads();
  }
  const int n = base;
  if (n == 0) {
    if (tid == 0) cs->ncells = 0;
    return;
  }
  for (int c = tid; c < n; c += nthreads) {
    ContactState& S = st[c];
    S.p = S.s_p = S.v_err = S.pj = S.gp = 0.0;
    for (int d = 0; d < 3; ++d) S.lambda[d] = S.s_l[d] = S.v_tang[d] = S.lj[d] = S.gl[d] = 0.0;
  }
  __syncthreads();

  auto accumulate = [&]() {
    if (warp < nb) {
      const int b = warp;
      const bool dyn = bodies[b].dynamic != 0;
      double f[3] = {0.0, 0.0, 0.0}, tq[3] = {0.0, 0.0, 0.0};
      for (int c = lane; c < n; c += 32) {
        const ContactCell& C = cells[cell_idx[c]];
        const ContactState& S = st[c];
        if (C.a != b && C.b != b) continue;
        const bool is_a = C.a == b;
        const double sgn = is_a ? 1.0 : -1.0;
        const double* fv = is_a ? C.f_a : C.f_b;
        const double* tv = is_a ? C.tau_a : C.tau_b;
        for (int d = 0; d < 3; ++d) f[d] += S.p * fv[d] + sgn * S.lambda[d];
        if (dyn) {
          const double* com = bodies[b].com;
          const double r[3] = {C.center[0] - com[0], C.center[1] - com[1], C.center[2] - com[2]};
          const double* l = S.lambda;
          const double cr[3] = {r[1] * l[2] - r[2] * l[1], r[2] * l[0] - r[0] * l[2], r[0] * l[1] - r[1] * l[0]};
          for (int d = 0; d < 3; ++d) tq[d] += S.p * tv[d] + sgn * cr[d];
        }
      }
      for (int d = 0; d < 3; ++d) {
        const double fs = warp_sum(f[d]), ts = warp_sum(tq[d]);
        if (lane == 0) {
          ef[b][d] = fs;
          et[b][d] = ts;
        }
      }
    }
    __syncthreads();
  };
  auto predict = [&]() {
    if (tid < nb) {
      const Body& M = bodies[tid];
      if (!M.dynamic) {
        for (int d = 0; d < 3; ++d) vt[tid][d] = wt[tid][d] = 0.0;
      } else {
        double l[3];
        for (int d = 0; d < 3; ++d) {
          vt[tid][d] = M.v[d] + dt / M.mass * (M.F[d] + ef[tid][d]);
          l[d] = M.L[d] + dt * (M.T[d] + et[tid][d]);
        }
        const double* I = M.inv_inertia_world;
        for (int r = 0; r < 3; ++r) wt[tid][r] = (I[r * 3] * l[0] + I[r * 3 + 1] * l[1]) + I[r * 3 + 2] * l[2];
      }
    }
    __syncthreads();
    for (int c = tid; c < n; c += nthreads) {
      const ContactCell& C = cells[cell_idx[c]];
      ContactState& S = st[c];
      const int a = C.a, b = C.b;
      auto dot3 = [](const double* x, const double* y) { return (x[0] * y[0] + x[1] * y[1]) + x[2] * y[2]; };
      S.v_err = -C.volume + dt * (((dot3(vt[a], C.f_a) + dot3(wt[a], C.tau_a)) + dot3(vt[b], C.f_b)) +
                                  dot3(wt[b], C.tau_b));
      if (bodies[a].dynamic && bodies[b].dynamic) {
        double vr[3];
        const double ra[3] = {C.center[0] - bodies[a].com[0], C.center[1] - bodies[a].com[1],
                              C.center[2] - bodies[a].com[2]};
        const double rb[3] = {C.center[0] - bodies[b].com[0], C.center[1] - bodies[b].com[1],
                              C.center[2] - bodies[b].com[2]};
        const double* wa = wt[a];
        const double* wb = wt[b];
        const double ca[3] = {wa[1] * ra[2] - wa[2] * ra[1], wa[2] * ra[0] - wa[0] * ra[2], wa[0] * ra[1] - wa[1] * ra[0]};
        const double cb[3] = {wb[1] * rb[2] - wb[2] * rb[1], wb[2] * rb[0] - wb[0] * rb[2], wb[0] * rb[1] - wb[1] * rb[0]};
        for (int d = 0; d < 3; ++d) vr[d] = ((vt[a][d] + ca[d]) - vt[b][d]) - cb[d];
        for (int r = 0; r < 3; ++r)
          S.v_tang[r] = (C.tproj[r * 3] * vr[0] + C.tproj[r * 3 + 1] * vr[1]) + C.tproj[r * 3 + 2] * vr[2];
      } else {
        S.v_tang[0] = S.v_tang[1] = S.v_tang[2] = 0.0;
      }
    }
    __syncthreads();
  };
  auto norm3 = [](const double* x) { return sqrt((x[0] * x[0] + x[1] * x[1]) + x[2] * x[2]); };
  auto jacobi = [&]() {
    if (warp < nb) {
      int cnt = 0;
      for (int c = lane; c < n; c += 32) {
        const ContactCell& C = cells[cell_idx[c]];
        if ((C.a == warp || C.b == warp) && (st[c].v_err < 0.0 || st[c].p > 0.0)) ++cnt;
      }
      for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
      if (lane == 0) nact[warp] = cnt;
    }
    __syncthreads();
    for (int c = tid; c < n; c += nthreads) {
      const ContactCell& C = cells[cell_idx[c]];
      ContactState& S = st[c];
      const double n_max = (double)max(max(nact[C.a], nact[C.b]), 1);
      const double alpha = kOmega / n_max / fmax(C.acc_p, kMinDiag);
      S.pj = fmax(S.p - alpha * S.v_err, 0.0);
      const double lmax = kMu * S.p * norm3(C.f_a);
      double star[3];
      const double af = fmax(C.acc_f, kMinDiag);
      for (int d = 0; d < 3; ++d) star[d] = -S.v_tang[d] / af;
      const double sn = norm3(star);
      if (sn > lmax)
        for (int d = 0; d < 3; ++d) star[d] = lmax * star[d] / sn;
      double ln[3];
      for (int d = 0; d < 3; ++d) ln[d] = S.lambda[d] + kOmega / n_max * star[d];
      const double lnn = norm3(ln);
      for (int d = 0; d < 3; ++d) S.lj[d] = lnn > lmax ? lmax * ln[d] / lnn : ln[d];
    }
    __syncthreads();
  };
  auto converged = [&]() {
    double fp = 0.0, ff = 0.0;
    for (int c = tid; c < n; c += nthreads) {
      const ContactCell& C = cells[cell_idx[c]];
      const ContactState& S = st[c];
      const double pp = S.p * fmax(C.acc_p, kMinDiag);
      fp += fabs(pp + S.v_err - sqrt(pp * pp + S.v_err * S.v_err));
      const double vtn = norm3(S.v_tang);
      const double dev = fmax(C.acc_f, kMinDiag) * (kMu * S.p * norm3(C.f_a) - norm3(S.lambda));
      ff += fabs(vtn + dev - sqrt(vtn * vtn + dev * dev));
    }
    fp = block_sum_all(fp, sh, &bc);
    ff = block_sum_all(ff, sh, &bc);
    return fp / (double)n < kTolP && ff / (double)n < kTolF;
  };

  accumulate();
  predict();
  jacobi();
  double prev = 0.0;
  {
    double g2 = 0.0;
    for (int c = tid; c < n; c += nthreads) {
      ContactState& S = st[c];
      S.gp = -(S.pj - S.p);
      S.s_p = -S.gp;
      g2 += S.gp * S.gp;
      double gl2 = 0.0;
      for (int d = 0; d < 3; ++d) {
        S.gl[d] = -(S.lj[d] - S.lambda[d]);
        S.s_l[d] = -S.gl[d];
      }
      gl2 = (S.gl[0] * S.gl[0] + S.gl[1] * S.gl[1]) + S.gl[2] * S.gl[2];
      g2 += gl2;
      S.p = S.pj;
      for (int d = 0; d < 3; ++d) S.lambda[d] = S.lj[d];
    }
    prev = block_sum_all(g2, sh, &bc);
  }
  accumulate();
  predict();
  int it = 0;
  // fixed_sweeps > 0: exactly that many sweeps, no merit test
  bool done = fixed_sweeps > 0 ? false : converged();
  while (fixed_sweeps > 0 ? it < fixed_sweeps : (!done && it < sweep_cap)) {
    jacobi();
    double g2 = 0.0;
    for (int c = tid; c < n; c += nthreads) {
      ContactState& S = st[c];
      S.gp = -(S.pj - S.p);
      g2 += S.gp * S.gp;
      for (int d = 0; d < 3; ++d) S.gl[d] = -(S.lj[d] - S.lambda[d]);
      g2 += (S.gl[0] * S.gl[0] + S.gl[1] * S.gl[1]) + S.gl[2] * S.gl[2];
    }
    const double gsum = block_sum_all(g2, sh, &bc);
    const double beta = gsum / fmax(prev, DBL_MIN);
    for (int c = tid; c < n; c += nthreads) {
      const ContactCell& C = cells[cell_idx[c]];
      ContactState& S = st[c];
      if (beta > 1.0) {
        S.s_p = 0.0;
        for (int d = 0; d < 3; ++d) S.s_l[d] = 0.0;
        S.p = S.pj;
        for (int d = 0; d < 3; ++d) S.lambda[d] = S.lj[d];
        continue;
      }
      // the friction cone of the iterate before this update (:452-467)
      const double lmax = kMu * S.p * norm3(C.f_a);
      const double p_nncg = S.pj + beta * S.s_p;
      if (p_nncg < 0.0) {
        S.p = S.pj;
        S.s_p = 0.0;
      } else {
        S.p = p_nncg;
        S.s_p = beta * S.s_p - S.gp;
      }
      double ln[3], tp[3];
      for (int d = 0; d < 3; ++d) ln[d] = S.lj[d] + beta * S.s_l[d];
      for (int r = 0; r < 3; ++r) tp[r] = (C.tproj[r * 3] * ln[0] + C.tproj[r * 3 + 1] * ln[1]) + C.tproj[r * 3 + 2] * ln[2];
      if (norm3(tp) > lmax) {
        for (int d = 0; d < 3; ++d) {
          S.lambda[d] = S.lj[d];
          S.s_l[d] = 0.0;
        }
      } else {
        for (int d = 0; d < 3; ++d) {
          S.lambda[d] = tp[d];
          S.s_l[d] = beta * S.s_l[d] - S.gl[d];
        }
      }
    }
    __syncthreads();
    prev = gsum;
    accumulate();
    predict();
    if (fixed_sweeps == 0) done = converged();
    ++it;
  }
  accumulate();
  if (tid < nb && bodies[tid].dynamic) {  // add_force_and_torque (rigid_body_motion.rs:156-159)
    for (int d = 0; d < 3; ++d) {
      bodies[tid].F[d] += ef[tid][d];
      bodies[tid].T[d] += et[tid][d];
    }
  }
  if (tid == 0) {
    cs->ncells = n;
    cs->iterations = it;
    cs->capped = (fixed_sweeps > 0 || done) ? 0 : 1;
  }
}

}  // namespace sph
