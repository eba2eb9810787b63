// direct_kernel.cuh -- the exact energies of many poses against a protein of a cluster or two: every pair.
//
// A thread takes up to four poses, keeps their transforms in registers and walks the ligand's atoms and all of
// the protein's records, which every lane reads from the same place (L1).  The pair terms, the order of a
// pose's sums (protein in cluster order, then the ligand's atoms) and so the bits of its energy are those of
// cull_kernel and cull_finish_kernel: a pair out of reach adds +0.
//
// What bounds it: the FMA pipe (12 cycles per warp and pair, Points::add), 67% busy at four poses per thread,
// 64 x 64 atoms and 524,288 poses (2.3e12 pairs/s); one pose per thread takes up to 2.4 times as long, for the
// records' loads.  8 | 32 | 64 protein atoms x 64 ligand atoms x 524,288 poses 153 | 496 | 953 us, culled 565 | 830 |
// 1,048.
#pragma once
#include "cull_kernel.cuh"

namespace bude {

constexpr int kDirectPoses = 4; // poses per thread, at most

struct DirectArgs {
  const float4 *ligand; // CullArgs::ligand; with folds the batch's atoms, from EdgeArgs::lig_off[ligand] on
  const float4 *slab;   // CullArgs::slab
  int natpro, natpro_pad;
  FinishArgs f; // n, folds, energies, edges, e; rows: the ligand's atoms (without folds)
};

template <int P> __global__ void __launch_bounds__(kMaxThreads, 1) direct_kernel(const DirectArgs a) {
  const int T = blockDim.x, tid = threadIdx.x;
  long long p0 = (long long)blockIdx.x * (P * T), p1 = min(p0 + P * T, a.f.n);
  const float4 *ligand = a.ligand;
  int rows = a.f.rows;
  bool all = a.f.e.all != 0;
  grid_dep_wait();
  if (a.f.folds) {
    const int4 f = __ldg(&a.f.folds[blockIdx.x]);
    p0 = f.x, p1 = (long long)f.x + f.y, rows = f.z;
    ligand += __ldg(&a.f.e.lig_off[f.w]);
    if (a.f.edges && *a.f.e.lig_any > 0) all = a.f.e.lig_all[f.w] != 0;
  }
  const float4 *xf = reinterpret_cast<const float4 *>(a.f.e.xform);
  float4 t[P][3];
  float acc[P];
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const long long p = min(p0 + k * T + tid, p1 - 1);
#pragma unroll
    for (int d = 0; d < 3; ++d) t[k][d] = __ldg(xf + 3 * p + d);
    acc[k] = 0.f;
  }
  for (int r = 0; r < rows; ++r) {
    const float4 la = __ldg(&ligand[r]);
    Points<P> pt;
#pragma unroll
    for (int k = 0; k < P; ++k) {
      float v[3];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        v[d] = t[k][d].w + la.x * t[k][d].x + la.y * t[k][d].y + la.z * t[k][d].z; // as in cull_kernel
      pt.set(k, make_float4(v[0], v[1], v[2], 0.f));
    }
    pt.clear();
    const float4 *rec = a.slab + (size_t)__float_as_int(la.w) * a.natpro_pad * kPairF4;
#pragma unroll 4
    for (int j = 0; j < a.natpro; ++j)
      pt.add(__ldg(rec + j * kPairF4), __ldg(rec + j * kPairF4 + 1),
             __ldg(reinterpret_cast<const float2 *>(rec + j * kPairF4 + 2)));
#pragma unroll
    for (int k = 0; k < P; ++k) acc[k] = __fadd_rn(acc[k], pt.energy(k));
  }
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const long long w = p0 + k * T + (tid & ~31), p = w + (tid & 31);
    bool irregular = false;
    if (p < p1) {
      a.f.energies[p] = 0.5f * acc[k];
      irregular = a.f.edges && (all || ((a.f.e.mask[p >> 5] >> (p & 31)) & 1u));
    }
    rescore_irregular(a.f, irregular, w, p);
  }
}

} // namespace bude
