// pose_order.cuh -- poses sorted by where they put the ligand, for the exact kernel's chunks.
//
// A block of cull_kernel groups the positions of one ligand atom over one chunk of poses; the closer the
// chunk's poses are to each other, the smaller the boxes of its groups and the fewer protein atoms pass
// their tests.  So a large pose set is first put in the order of an 8 x 8 x 8 grid over the box of its
// translations (Hilbert order of the cells): a group of 64 of 4,096 poses meets 157 of 2,672 atoms at
// real density, 125 when the 4,096 are a 16th of 65,536 poses and 109 when they are a 256th of 1,048,576
// (58 interact with a pose).  Cells of the orientation as well as the translation gave 106 to 126.  An
// energy does not depend on the order (cull_kernel.cuh), and a ligand that turns about a far origin only
// loses the gain.
//
// Three kernels: the box, the cells (a counting sort: every block counts its tile in shared memory and
// takes its places in each cell by one atomic per cell), the transforms in sorted order.  Latency-bound
// at 65,536 poses (3, 6 and 7 us, pose_xform_kernel 5), by the scattered 48-byte rows at 1,048,576 (6, 11
// and 44 us).  Evaluations before | with them, end to end from the host: 4,096 x 64 x 1,048,576 3.64 |
// 3.01 ms, 2,672 x 48 x 400,003 streamed 2.77 | 2.39 ms, 938 x 26 x 65,536 155 | 147 us.
#pragma once
#include "cull_kernel.cuh"
#include "pose_xform.cuh"
#include "warp.cuh"

namespace bude {

constexpr int kOrderThreads = 512;
constexpr int kOrderBoxes = 128; // blocks of the box kernel, at most

// Cell of a translation in the 8 x 8 x 8 grid over the box from `lo` on with `s` cells per Angstrom, in Hilbert
// order.  Translations that are not regular go to a cell by the pose's index: their poses are irregular and
// are scored one after the other by the warp that finds them (cull_finish_kernel), so they have to stay as
// spread as they came.  One in ten of 65,536 poses against 938 x 26 not a number: 5.3 ms with all in one cell,
// 1.9 so.
__device__ __forceinline__ int order_cell(float3 t, float3 lo, float3 s, long long pose) {
  if (!(fabsf(t.x) + fabsf(t.y) + fabsf(t.z) < kPoseReach)) return (int)(pose % kBins);
  const int x = min(max((int)((t.x - lo.x) * s.x), 0), 7), y = min(max((int)((t.y - lo.y) * s.y), 0), 7),
            z = min(max((int)((t.z - lo.z) * s.z), 0), 7);
  return kHilbert.at[z * 64 + y * 8 + x];
}
__device__ __forceinline__ float order_scale(float lo, float hi) { return hi > lo ? 8.f / (hi - lo) : 0.f; }

// Scratch of a sort of n poses in `tiles` tiles.
struct PoseOrder {
  int *perm;     // [n] pose of each place
  unsigned *key; // [n] cell << 16 | rank among the tile's poses of the cell
  float *boxes;  // [kOrderBoxes][6]
  int *count;    // [cells] poses of each cell
  int *base;     // [tiles][cells] the tile's first place in each cell
  int tile;      // poses of a tile, a multiple of kOrderThreads, at most 65,536
  int coarse;    // 0: kBins cells; 1: 8 of them at a time
  __host__ __device__ int cells() const { return coarse ? kBins / 8 : kBins; }
};

// The box of the regular translations, one per block; the counts set to zero.
static __global__ void __launch_bounds__(kOrderThreads) pose_box_kernel(const float *__restrict__ poses,
                                                                        long long pstride, long long n, PoseOrder o) {
  __shared__ float red[6][kOrderThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (blockIdx.x == 0)
    for (int b = tid; b < o.cells(); b += kOrderThreads) o.count[b] = 0;
  float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (long long i = (long long)blockIdx.x * kOrderThreads + tid; i < n; i += (long long)gridDim.x * kOrderThreads) {
    const float x = poses[3 * pstride + i], y = poses[4 * pstride + i], z = poses[5 * pstride + i];
    if (!(fabsf(x) + fabsf(y) + fabsf(z) < kPoseReach)) continue;
    v[0] = fminf(v[0], x), v[1] = fminf(v[1], y), v[2] = fminf(v[2], z);
    v[3] = fmaxf(v[3], x), v[4] = fmaxf(v[4], y), v[5] = fmaxf(v[5], z);
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    const float m = d < 3 ? warp_min(v[d]) : warp_max(v[d]);
    if (lane == 0) red[d][warp] = m;
  }
  __syncthreads();
  if (warp < 6) {
    const float m = red[warp][lane % (kOrderThreads / 32)];
    const float r = warp < 3 ? warp_min(m) : warp_max(m);
    if (lane == 0) o.boxes[blockIdx.x * 6 + warp] = r;
  }
}

static __global__ void __launch_bounds__(kOrderThreads) pose_cell_kernel(const float *__restrict__ poses,
                                                                         long long pstride, long long n, int boxes,
                                                                         PoseOrder o, const RowOrder ro) {
  __shared__ int bins[kBins];
  __shared__ float box[6];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cells = o.cells(), shift = o.coarse ? 3 : 0;
  for (int b = tid; b < cells; b += kOrderThreads) bins[b] = 0;
  grid_dep_wait();
  if (ro.rows && blockIdx.x == gridDim.x - 1) {
    row_order(ro);
    return;
  }
  if (warp < 6) {
    float m = warp < 3 ? INFINITY : -INFINITY;
    for (int b = lane; b < boxes; b += 32)
      m = warp < 3 ? fminf(m, o.boxes[b * 6 + warp]) : fmaxf(m, o.boxes[b * 6 + warp]);
    m = warp < 3 ? warp_min(m) : warp_max(m);
    if (lane == 0) box[warp] = m;
  }
  __syncthreads();
  const float3 lo = make_float3(box[0], box[1], box[2]);
  const float3 s = make_float3(order_scale(box[0], box[3]), order_scale(box[1], box[4]), order_scale(box[2], box[5]));
  const long long first = (long long)blockIdx.x * o.tile, last = min(first + o.tile, n);
  for (long long i = first + tid; i < last; i += kOrderThreads) {
    const float3 t = make_float3(poses[3 * pstride + i], poses[4 * pstride + i], poses[5 * pstride + i]);
    const int cell = order_cell(t, lo, s, i) >> shift;
    o.key[i] = (unsigned)cell << 16 | (unsigned)atomicAdd(&bins[cell], 1);
  }
  __syncthreads();
  for (int b = tid; b < cells; b += kOrderThreads)
    o.base[(size_t)blockIdx.x * cells + b] = bins[b] ? atomicAdd(&o.count[b], bins[b]) : 0;
}

// The tile's transforms at their places; the irregular-pose bits in pose order (pose_xform_kernel).
static __global__ void __launch_bounds__(kOrderThreads) pose_place_kernel(const float *__restrict__ poses,
                                                                          long long pstride, long long n, PoseOrder o,
                                                                          float4 *__restrict__ xform,
                                                                          unsigned *__restrict__ edge_mask) {
  static_assert(kBins == kOrderThreads, "one cell per thread");
  __shared__ int start[kBins];
  __shared__ int warp_total[kOrderThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cells = o.cells();
  grid_dep_wait();
  {
    const int v = tid < cells ? o.count[tid] : 0;
    int sum = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += u;
    }
    if (lane == 31) warp_total[warp] = sum;
    __syncthreads();
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? warp_total[lane] : 0);
    if (tid < cells) start[tid] = before + sum - v + o.base[(size_t)blockIdx.x * cells + tid];
  }
  __syncthreads();
  const long long first = (long long)blockIdx.x * o.tile, last = min(first + o.tile, n);
  for (long long w = first + (tid & ~31); w < last; w += kOrderThreads) {
    const long long i = w + lane;
    bool irregular = false;
    if (i < last) {
      float4 r0, r1, r2;
      pose_rows(poses, pstride, i, r0, r1, r2);
      const unsigned k = o.key[i];
      const int at = start[k >> 16] + (int)(k & 0xffffu);
      xform[3ll * at + 0] = r0;
      xform[3ll * at + 1] = r1;
      xform[3ll * at + 2] = r2;
      o.perm[at] = (int)i;
      irregular = !pose_regular(r0, r1, r2);
    }
    const unsigned bits = __ballot_sync(0xffffffffu, irregular);
    if (lane == 0) edge_mask[w >> 5] = bits;
  }
}

// The same for a batch: every ligand's poses in the order of 64 cells over the box of their translations,
// within the ligand's own range of places.  The transforms and irregular-pose bits are there already
// (pose_xform_kernel); a tile is a finish item of the batch's plan, {first pose, poses, rows, ligand} of at
// most 256 poses.  Memory-bound (48 bytes read and written per pose) and short beside the kernel they
// serve: 256 ligands, 5.4 million poses 16.83 -> 15.02 ms in all.
constexpr int kBatchCells = kBins / 8;
struct BatchOrder {
  const long long *pose_off; // [ligands + 1]
  const int4 *tiles;
  const float4 *xform; // in pose order
  float4 *sorted;      // in the new order
  int *perm;           // [poses] pose of each place
  unsigned *key;       // [poses] cell << 16 | rank among the tile's poses of the cell
  unsigned *boxes;     // [ligands][6], zero at first: ~order_key of the lower corner, order_key of the upper; 0: none
  int *count;          // [ligands][kBatchCells], zero at first
  int *base;           // [tiles][kBatchCells]
};

// The boxes of the ligands' regular translations, one tile per block.  (One ligand per block read a ligand of
// 2,000,000 poses on one SM: against 100 x 2 atoms 1,385 us an evaluation, 413 so.)
static __global__ void __launch_bounds__(256) batch_box_kernel(const BatchOrder o) {
  __shared__ float red[6][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  grid_dep_wait();
  const int4 t = __ldg(&o.tiles[blockIdx.x]);
  float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (tid < t.y) {
    const long long i = (long long)t.x + tid;
    const float x = o.xform[3 * i].w, y = o.xform[3 * i + 1].w, z = o.xform[3 * i + 2].w;
    if (fabsf(x) + fabsf(y) + fabsf(z) < kPoseReach) v[0] = v[3] = x, v[1] = v[4] = y, v[2] = v[5] = z;
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    const float m = d < 3 ? warp_min(v[d]) : warp_max(v[d]);
    if (lane == 0) red[d][warp] = m;
  }
  __syncthreads();
  if (warp < 6) {
    const float m = red[warp][lane % 8];
    const float r = warp < 3 ? warp_min(m) : warp_max(m);
    if (lane == 0 && fabsf(r) < INFINITY) // a tile without a regular pose leaves the box as it is
      atomicMax(&o.boxes[t.w * 6 + warp], warp < 3 ? ~order_key(r) : order_key(r));
  }
}

// One tile per block, one pose per thread.
static __global__ void __launch_bounds__(256) batch_cell_kernel(const BatchOrder o) {
  __shared__ int bins[kBatchCells];
  __shared__ float b[6];
  const int tid = threadIdx.x;
  if (tid < kBatchCells) bins[tid] = 0;
  grid_dep_wait();
  const int4 t = __ldg(&o.tiles[blockIdx.x]);
  if (tid < 6) {
    const unsigned k = o.boxes[t.w * 6 + tid];
    b[tid] = k == 0 ? (tid < 3 ? INFINITY : -INFINITY) : key_float(tid < 3 ? ~k : k);
  }
  __syncthreads();
  if (tid < t.y) {
    const long long i = (long long)t.x + tid;
    const float3 at = make_float3(o.xform[3 * i].w, o.xform[3 * i + 1].w, o.xform[3 * i + 2].w);
    const float3 s = make_float3(order_scale(b[0], b[3]), order_scale(b[1], b[4]), order_scale(b[2], b[5]));
    const int cell = order_cell(at, make_float3(b[0], b[1], b[2]), s, i) >> 3;
    o.key[i] = (unsigned)cell << 16 | (unsigned)atomicAdd(&bins[cell], 1);
  }
  __syncthreads();
  if (tid < kBatchCells)
    o.base[(size_t)blockIdx.x * kBatchCells + tid] =
        bins[tid] ? atomicAdd(&o.count[t.w * kBatchCells + tid], bins[tid]) : 0;
}

static __global__ void __launch_bounds__(256) batch_place_kernel(const BatchOrder o) {
  __shared__ int start[kBatchCells], half;
  const int tid = threadIdx.x, lane = tid & 31;
  grid_dep_wait();
  const int4 t = __ldg(&o.tiles[blockIdx.x]);
  int v = 0, sum = 0;
  if (tid < kBatchCells) {
    v = sum = o.count[t.w * kBatchCells + tid];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += u;
    }
    if (tid == 31) half = sum;
  }
  __syncthreads();
  if (tid < kBatchCells)
    start[tid] = sum - v + (tid >= 32 ? half : 0) + o.base[(size_t)blockIdx.x * kBatchCells + tid];
  __syncthreads();
  if (tid >= t.y) return;
  const long long i = (long long)t.x + tid;
  const unsigned k = o.key[i];
  const long long at = o.pose_off[t.w] + start[k >> 16] + (int)(k & 0xffffu);
#pragma unroll
  for (int d = 0; d < 3; ++d) o.sorted[3 * at + d] = o.xform[3 * i + d];
  o.perm[at] = (int)i;
}
static_assert(kBatchCells == 64, "two warps scan a ligand's cells");

} // namespace bude
