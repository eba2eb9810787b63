// deck_tables.cuh -- the tables the exact kernel reads (cull_kernel.cuh: CullArgs), built on the device
// from the protein in cluster order and the forcefield.
//
// One warp takes one ligand type and one cluster of 32 protein atoms, one atom per lane: the pair's
// record and reach, the cluster's largest reach, and, for type 0, the cluster's box.  On the host the
// tables of 34 types x 938 atoms cost an upload 0.56 ms more and those of 34 x 4,096 are 9 MB to copy; here
// the copy is the protein, and 34 x 4,096 records take 6.6 us (1.35 TB/s of table from short warps).
#pragma once
#include <cstdint>

#include "../../include/minibude_gb300.h"
#include "exact_shape.h"
#include "pair_record.h"
#include "ptx.cuh"
#include "warp.cuh"

namespace bude {

// The squared distance past which the pair energy of ligand type L and protein type Pp is exactly zero:
// the cut-offs of pair_record's three terms (rec: the pair's record), with room for the rounding of the
// distance and of the constants (below 1e-5 of the distance, and 1e-6 A of the charge term's).
__device__ __forceinline__ float pair_reach2(const bude_ffparams &L, const bude_ffparams &Pp, const float *rec) {
  const float radij = Pp.radius + L.radius;
  float past = 0.f;
  if (rec[6] != 0.f) past = rec[11] == -0.25f ? 4.f : 2.f;
  if (rec[8] != 0.f) past = fmaxf(past, rec[13] == -1.f ? 1.f : 5.5f);
  const float reach = (radij + past) * (1.f + 2e-5f) + 1e-4f;
  return reach * reach * (1.f + 2e-6f);
}

// Rows of `stride` records (at least natpro, a multiple of 8) per type; grid: warps over types x clusters.
// A protein atom with a type outside the forcefield gets a padding record.
static __global__ void __launch_bounds__(256) deck_table_kernel(const bude_atom *__restrict__ protein, int natpro,
                                                                const bude_ffparams *__restrict__ ff, int ntypes,
                                                                int stride, int clusters, float4 *__restrict__ slab,
                                                                float4 *__restrict__ reach, float4 *__restrict__ box,
                                                                float *__restrict__ box_reach) {
  const int lane = threadIdx.x & 31;
  grid_dep_wait();
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long w = warp; w < (long long)ntypes * clusters; w += warps) {
    const int t = (int)(w / clusters), c = (int)(w - (long long)t * clusters);
    const int j = c * kClusterAtoms + lane;
    float rec[kRecFloats];
    float r2 = -1.f;
    bude_atom p{};
    bool real = j < natpro;
    if (real) {
      p = protein[j];
      real = p.type >= 0 && p.type < ntypes;
    }
    if (real) {
      pair_record(ff[t], ff[p.type], p.x, p.y, p.z, rec);
      r2 = pair_reach2(ff[t], ff[p.type], rec);
    } else {
      null_record(rec);
    }
    if (j < stride) {
      const size_t at = (size_t)t * stride + j;
      slab[at * kPairF4 + 0] = make_float4(rec[0], rec[2], rec[4], rec[6]);
      slab[at * kPairF4 + 1] = make_float4(rec[8], rec[10], rec[11], rec[12]);
      slab[at * kPairF4 + 2] = make_float4(rec[13], rec[14], 0.f, 0.f);
      reach[at] = make_float4(rec[0], rec[2], rec[4], r2);
    }
    // A reach that is not a number lets its cluster through (box_d2 > NaN is false).
    const float most = warp_max(r2);
    const unsigned odd = __ballot_sync(0xffffffffu, !(r2 == r2));
    if (lane == 0) box_reach[w] = odd ? NAN : most;
    if (t == 0) {
      const float lx = warp_min(real ? p.x : INFINITY), hx = warp_max(real ? p.x : -INFINITY);
      const float ly = warp_min(real ? p.y : INFINITY), hy = warp_max(real ? p.y : -INFINITY);
      const float lz = warp_min(real ? p.z : INFINITY), hz = warp_max(real ? p.z : -INFINITY);
      if (lane == 0) {
        box[2 * c] = make_float4(lx, ly, lz, 0.f);
        box[2 * c + 1] = make_float4(hx, hy, hz, 0.f);
      }
    }
  }
}

inline unsigned deck_table_grid(int ntypes, int clusters) {
  const long long blocks = ((long long)ntypes * clusters + 7) / 8;
  return (unsigned)(blocks < 4096 ? blocks : 4096);
}

} // namespace bude
