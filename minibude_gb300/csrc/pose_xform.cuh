// pose_xform.cuh -- the 3x4 transforms of the poses.
#pragma once
#include "edge_pose.cuh"
#include "ptx.cuh"

namespace bude {

// Rows {r00, r01, r02, tx}, {r10, r11, r12, ty}, {r20, r21, r22, tz} of pose i.
__device__ __forceinline__ void pose_rows(const float *__restrict__ poses, long long pstride, long long i, float4 &r0,
                                          float4 &r1, float4 &r2) {
  float sx, cx, sy, cy, sz, cz;
  sincosf(poses[i], &sx, &cx);
  sincosf(poses[pstride + i], &sy, &cy);
  sincosf(poses[2 * pstride + i], &sz, &cz);
  r0 = make_float4(cy * cz, sx * sy * cz - cx * sz, cx * sy * cz + sx * sz, poses[3 * pstride + i]);
  r1 = make_float4(cy * sz, sx * sy * sz + cx * cz, cx * sy * sz - sx * cz, poses[4 * pstride + i]);
  r2 = make_float4(-sy, sx * cy, cx * cy, poses[5 * pstride + i]);
}

// The ligand atoms in the order in which the exact kernel's blocks take them, longest first: an atom's
// records go with the volume around its positions, so its weight is the sum over a sample of the protein of
// (reach of the pair + half its distance from the ligand's origin + 0.5)^3.  Written by one block of a
// transform kernel, beside the others (3 us, hidden); which atom a block takes changes no energy.  With the
// atoms as they come the last blocks of a launch of one to three waves left SMs idle: 1,237 x 37 x 12,345
// without allocation 162 -> 151 us, 938 x 26 x 65,536 135 -> 128, 2,672 x 48 x 400,003 streamed 1,685 ->
// 1,626.  By distance from the origin alone half of that was gained.
constexpr int kRowOrderMax = 1024;
struct RowOrder {
  const float4 *ligand;
  const float4 *reach; // CullArgs::reach
  int natlig, natpro, natpro_pad;
  int *rows;             // [natlig], or nullptr: no order (always above kRowOrderMax atoms)
  const unsigned *words; // as CullArgs::words
};

// The weight of ligand atom a, the whole warp's work; 0 where it is not a number.
__device__ __forceinline__ float atom_weight(const float4 a, const float4 *all_reach, int natpro, int natpro_pad) {
  constexpr int kPerLane = 8; // 256 protein atoms, evenly spread
  const float4 *reach = all_reach + (size_t)__float_as_int(a.w) * natpro_pad;
  const float wide = 0.5f * sqrtf(a.x * a.x + a.y * a.y + a.z * a.z) + 0.5f;
  float w = 0.f;
#pragma unroll
  for (int k = 0; k < kPerLane; ++k) {
    const int at = (int)((long long)(k * 32 + (int)(threadIdx.x & 31)) * natpro / (32 * kPerLane));
    const float x = (natpro > 0 ? sqrtf(reach[at].w) : 0.f) + wide;
    w += x * x * x;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) w += __shfl_xor_sync(0xffffffffu, w, d);
  return w >= 0.f ? w : 0.f;
}

__device__ __forceinline__ void row_order(const RowOrder &o) {
  __shared__ float weight[kRowOrderMax];
  if (o.words && deck_bad_type(o.words)) return;
  for (int i = threadIdx.x >> 5; i < o.natlig; i += blockDim.x >> 5) {
    const float w = atom_weight(o.ligand[i], o.reach, o.natpro, o.natpro_pad);
    if ((threadIdx.x & 31) == 0) weight[i] = w;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < o.natlig; i += blockDim.x) {
    const float w = weight[i];
    int rank = 0;
    for (int j = 0; j < o.natlig; ++j) rank += weight[j] > w || (weight[j] == w && j < i);
    o.rows[rank] = i;
  }
}

// Pose transforms: src/cuda/fasten.hpp:45-71 / serial/fasten.hpp:28-53, one thread per pose.
// Output: three float4 rows per pose (pose_rows).
// With edge_mask, bit (i & 31) of word i >> 5 is set when pose i is irregular and is rescored afterwards
// (edge_pose.cuh); blockDim must be a multiple of 32.  With ro.rows one more block
// than the poses take, for row_order.
// (Internal linkage, so several translation units may include this file.)
static __global__ void __launch_bounds__(256) pose_xform_kernel(const float *__restrict__ poses, long long pstride,
                                                         long long nposes, float4 *__restrict__ xform,
                                                         unsigned *__restrict__ edge_mask, const RowOrder ro) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  bool irregular = false;
  grid_dep_wait();
  if (ro.rows && blockIdx.x == gridDim.x - 1) {
    row_order(ro);
    return;
  }
  if (i < nposes) {
    float4 r0, r1, r2;
    pose_rows(poses, pstride, i, r0, r1, r2);
    xform[3 * i + 0] = r0;
    xform[3 * i + 1] = r1;
    xform[3 * i + 2] = r2;
    irregular = !pose_regular(r0, r1, r2);
  }
  if (edge_mask) {
    const unsigned bits = __ballot_sync(0xffffffffu, irregular);
    if ((threadIdx.x & 31) == 0 && i < nposes) edge_mask[i >> 5] = bits;
  }
}

} // namespace bude
