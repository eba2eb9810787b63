// cull_kernel.cuh -- the exact miniBUDE energy kernel for sm_103a: only the ligand-protein pairs that
// can interact are evaluated.
//
// Computes, for every pose, the energy of reference `fasten_main` (src/cuda/fasten.hpp:20-161,
// src/serial/fasten.hpp:18-132).
//
// Restatement of the pair energy.  For a ligand atom of type L and a protein atom of type P at
// distance r (radij = radius_L + radius_P), the reference's three terms are piecewise linear in r
// and each one is zero past its cut-off:
//   steric   76 * (1 - r/radij)                          for r < radij
//   charge   45*c * clamp(1 - (r - radij)/elcdst, 0, 1)  (c = elsc_L*elsc_P, sign forced negative
//                                                        when either type is 'E'; elcdst 4 or 2)
//   desolv   d * clamp(1 - (r - radij)/distdslv, 0, 1)   (d = signed hphb sum; zero unless the
//                                                        protein hphb is non-zero and distdslv > 0)
// The steric factor lies in [0, 1] as well (r >= 0), so all three are one `fma.rn.sat` each with
// per-type-pair constants (pair_record.h).  One interaction is 3 FADD + FMUL + 2 FFMA (distance^2),
// one MUFU square root, 3 FFMA.SAT and 3 FFMA: 12 FP32 operations against the reference's ~30.
//
// A pair past all three cut-offs adds +0, so leaving it out changes no bit of a sum.  Of the 4,096 x 64 pairs of a pose of the
// scaled-up workload 0.8% interact, of a 2,672-atom protein at real density 1.8%.
//
// What makes the pairs cheap to find: a rotated ligand atom of many poses fills a ball of a few
// Angstroms, so sorting the poses by where they put the atom gives groups of 64 whose positions share
// a box of 2-3 A, and a box is tested against 32 protein atoms by one warp instruction sequence.
//
//   * a block takes a chunk of poses (ppwi * wgsize of them) and one ligand atom: it transforms the atom
//     for every pose, bins the positions over an 8 x 8 x 8 grid of their bounding box in Hilbert order
//     (a counting sort in shared memory) and hands the sorted points out in groups of 32 * P, P per
//     lane, to its warps;
//   * a warp reduces its group to a box and walks the protein, which lies in clusters of 32 atoms near
//     each other (k-d order, ensure_slab): 32 clusters at a time are tested against the box with one
//     cluster per lane, then the 32 atoms of each cluster that is in reach with one atom per lane and
//     its own reach for this ligand type; the atoms left are evaluated for the group's points with the
//     48-byte records brought into shared memory, eight at a time, ahead of their use;
//   * a point's terms add up in protein order, and a pose's atoms in ligand order (cull_finish_kernel).
//     Nothing in that order depends on the other poses, so a pose's energy is the same bits for every
//     launch shape, chunk, batch or position.
//
//   * few points get a warp each (point_kernel), and many poses against a protein of a few dozen atoms every
//     pair (direct_kernel.cuh); both give the same bits;
//   * a large pose set comes in the order of its translations (pose_order.cuh), so that a chunk's poses
//     are near each other and the groups tighter still.
//
// What bounds it: instruction issue (75% of the slots on the 4,096 x 64 deck), 60 to 75% of the time the
// record loop (35 instructions per record and 64 points, 23 of them the pair arithmetic), the rest the
// sort, the boxes and the candidate lists.  Measured, all pairs evaluated (records broadcast to 16 poses
// per thread, TMA-staged) | this kernel, end to end from pinned host memory, over several GPUs: 4,096 x 64 x
// 1,048,576 101.5 | 2.5-2.8 ms, 938 x 26 x 65,536 0.750 | 0.124-0.133 ms, 2,672 x 48 x 400,003 streamed 21.2 |
// 1.5-1.8 ms; 64 ligands of 12-96 atoms x 1,024-16,384 poses against 2,672 atoms 67.0 | 2.1-2.3 ms.  What
// went into it, on 4,096 x 64 x 262,144 unsorted poses: records read through L1 one by one 1,140 us (and 64
// poses took 105 us for 41); 64-byte records with the packed instructions' operands twice, 1,250; 48 bytes
// 1,100 (the loads' register writes bound two points per lane); lists of 64 records 1,095, of 128 in stages
// of 10 1,067; no shared candidate lists 1,218.  One ligand atom per block instead of two, binned over the
// box of its own positions (no registers spill any more but 112 to 176 bytes with 16 poses per thread and 16
// with four per lane): the 4,096 x 64 x 1,048,576 deck 4.52 -> 3.30 ms;
// poses sorted 3.64 -> 3.01.
#pragma once
#include <cstdint>
#include <type_traits>

#include "edge_pose.cuh"
#include "exact_shape.h"
#include "ptx.cuh"
#include "warp.cuh"

namespace bude {

constexpr int kBins = 512;        // 8 x 8 x 8 cells

struct CullArgs {
  const float4 *ligand;  // atoms {x, y, z, __int_as_float(type)}
  const float4 *slab;    // [type][natpro_pad] 48-byte records (Points::add), protein in cluster order
  const float4 *reach;   // [type][natpro_pad] {x, y, z, squared reach of the pair}; padding: reach -1
  const float4 *box;     // [clusters][2]: lower and upper corner of the cluster's atoms
  const float *box_reach; // [type][clusters]: the largest squared reach in the cluster
  const float *xform;    // 12 floats per pose
  const int4 *items;     // {atom, row, first pose, poses} per block, or nullptr: block b = row b / chunks,
                         // chunk b % chunks of one ligand
  float *sums;           // [row][stride]: a ligand atom's sum over the protein, from pose `first` on
  long long stride, first;
  long long nposes;      // without items: poses of the ligand
  float3 lo, hi;         // protein atoms' bounding box, widened by the longest reach
  const unsigned *words; // optional: a deck checked on the device (edge_pose.cuh); nothing runs on a bad one
  const int *rows;       // optional, without items: the rows in the order in which the blocks take them (RowOrder)
  int atom0;             // without items: the atom of row 0
  int chunk, chunks;     // without items: poses of a chunk (at most K * blockDim.x) and chunks of the ligand
  int natpro_pad;        // records per type
  int clusters;          // of kClusterAtoms; the last may be short
  int supers;            // 2^supers groups share a list of candidates (protein indices below 65,536); 0: no lists
};

// Cell (x, y, z) of an 8 x 8 x 8 grid, at z * 64 + y * 8 + x, to its place on a Hilbert curve (Skilling,
// "Programming the Hilbert curve", AIP Conf. Proc. 707, 2004).
struct HilbertTable {
  unsigned short at[kBins];
  constexpr HilbertTable() : at() {
    for (int i = 0; i < kBins; ++i) {
      unsigned x[3] = {(unsigned)i & 7u, (unsigned)(i >> 3) & 7u, (unsigned)(i >> 6) & 7u};
      for (unsigned q = 4; q > 1; q >>= 1)
        for (int a = 0; a < 3; ++a) {
          const unsigned p = q - 1;
          if (x[a] & q) {
            x[0] ^= p;
          } else {
            const unsigned t = (x[0] ^ x[a]) & p;
            x[0] ^= t;
            x[a] ^= t;
          }
        }
      x[1] ^= x[0];
      x[2] ^= x[1];
      unsigned t = 0;
      for (unsigned q = 4; q > 1; q >>= 1)
        if (x[2] & q) t ^= q - 1;
      unsigned k = 0;
      for (int b = 2; b >= 0; --b)
        for (int a = 0; a < 3; ++a) k = (k << 1) | (((x[a] ^ t) >> b) & 1u);
      at[i] = (unsigned short)k;
    }
  }
};
static __device__ constexpr HilbertTable kHilbert{};

// Squared distance of the box [lo, hi] to the box [plo, phi].
__device__ __forceinline__ float box_d2(float3 lo, float3 hi, float4 plo, float4 phi) {
  const float dx = fmaxf(fmaxf(plo.x - hi.x, lo.x - phi.x), 0.f);
  const float dy = fmaxf(fmaxf(plo.y - hi.y, lo.y - phi.y), 0.f);
  const float dz = fmaxf(fmaxf(plo.z - hi.z, lo.z - phi.z), 0.f);
  return dx * dx + dy * dy + dz * dz;
}

// P points per lane, in pairs for the packed f32x2 instructions (P = 1: scalar, the same roundings).
template <int P> struct Points {
  static constexpr int NP = P / 2;
  float2 x[NP], y[NP], z[NP], e[NP];
  __device__ __forceinline__ void set(int i, float4 p) {
    float2 &a = x[i / 2], &b = y[i / 2], &c = z[i / 2];
    if (i & 1) a.y = p.x, b.y = p.y, c.y = p.z;
    else a.x = p.x, b.x = p.y, c.x = p.z;
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int j = 0; j < NP; ++j) e[j] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ float energy(int i) const { return (i & 1) ? e[i / 2].y : e[i / 2].x; }
  // The pair terms with the record {px, py, pz, kc | kd, -1/radij, -1/elcdst, b_c | -1/distdslv, b_d}.
  // A broadcast operand of a packed instruction takes a register pair, so with one pair of points the
  // differences and the accumulation are scalar (21 FP32 instructions, 24 cycles of the FMA pipe) and
  // from two pairs on packed (one move per pair operand and record).
  __device__ __forceinline__ void add(const float4 A, const float4 B, const float2 C) {
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      float2 dx, dy, dz;
      if (NP == 1) {
        dx = make_float2(__fsub_rn(x[j].x, A.x), __fsub_rn(x[j].y, A.x));
        dy = make_float2(__fsub_rn(y[j].x, A.y), __fsub_rn(y[j].y, A.y));
        dz = make_float2(__fsub_rn(z[j].x, A.z), __fsub_rn(z[j].y, A.z));
      } else {
        dx = sub2(x[j], make_float2(A.x, A.x));
        dy = sub2(y[j], make_float2(A.y, A.y));
        dz = sub2(z[j], make_float2(A.z, A.z));
      }
      float2 d2 = mul2(dx, dx);
      d2 = fma2(dy, dy, d2);
      d2 = fma2(dz, dz, d2);
      const float2 r = make_float2(sqrt_approx(d2.x), sqrt_approx(d2.y));
      const float2 fs = make_float2(fma_sat(r.x, B.y, 1.f), fma_sat(r.y, B.y, 1.f));
      const float2 fc = make_float2(fma_sat(r.x, B.z, B.w), fma_sat(r.y, B.z, B.w));
      const float2 fd = make_float2(fma_sat(r.x, C.x, C.y), fma_sat(r.y, C.x, C.y));
      if (NP == 1) {
        e[j].x = __fmaf_rn(fd.x, B.x, __fmaf_rn(fc.x, A.w, __fmaf_rn(fs.x, kSteric, e[j].x)));
        e[j].y = __fmaf_rn(fd.y, B.x, __fmaf_rn(fc.y, A.w, __fmaf_rn(fs.y, kSteric, e[j].y)));
      } else {
        e[j] = fma2(fs, make_float2(kSteric, kSteric), e[j]);
        e[j] = fma2(fc, make_float2(A.w, A.w), e[j]);
        e[j] = fma2(fd, make_float2(B.x, B.x), e[j]);
      }
    }
  }
};

template <> struct Points<1> {
  float x, y, z, e;
  __device__ __forceinline__ void set(int, float4 p) { x = p.x, y = p.y, z = p.z; }
  __device__ __forceinline__ void clear() { e = 0.f; }
  __device__ __forceinline__ float energy(int) const { return e; }
  __device__ __forceinline__ void add(const float4 A, const float4 B, const float2 C) {
    const float dx = __fsub_rn(x, A.x), dy = __fsub_rn(y, A.y), dz = __fsub_rn(z, A.z);
    const float r = sqrt_approx(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))));
    e = __fmaf_rn(fma_sat(r, B.y, 1.f), kSteric, e);
    e = __fmaf_rn(fma_sat(r, B.z, B.w), A.w, e);
    e = __fmaf_rn(fma_sat(r, C.x, C.y), B.x, e);
  }
};

// Per warp: the records found to be in reach, and the two stages they are copied through.
constexpr int kListCap = 256;      // room for the four clusters of one step past kListFull
constexpr int kListFull = 128;     // evaluated from here on
constexpr int kStageRecs = 10;     // 48-byte records per stage: one 16-byte copy per lane of the first 30
struct WarpList {
  float4 stage[2][kStageRecs * kPairF4];
  unsigned short at[kListCap]; // record indices, relative to the list's first cluster
};

__device__ __forceinline__ void copy16(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Evaluate the first `count` records of the list (indices from the record at `recs` on) for the warp's
// points, one stage of records in flight while the other is used.
template <int P>
__device__ __forceinline__ void list_eval(Points<P> &pt, WarpList &l, int count, const float4 *recs) {
  const int lane = threadIdx.x & 31;
  const float4 *mine = recs + lane % kPairF4;
  const int slot = lane < kStageRecs * kPairF4 ? lane / kPairF4 : kListCap; // record of the stage it copies
  auto fetch = [&](int first, int buf) {
    const int i = first + slot;
    if (i < count) copy16(&l.stage[buf][lane], mine + (int)l.at[i] * kPairF4);
    copy_commit();
  };
  __syncwarp();
  fetch(0, 0);
  for (int first = 0, buf = 0; first < count; first += kStageRecs, buf ^= 1) {
    fetch(first + kStageRecs, buf ^ 1);
    copy_wait<1>();
    __syncwarp();
    const float4 *r = l.stage[buf];
    auto add = [&](int i) {
      pt.add(r[i * kPairF4], r[i * kPairF4 + 1], *reinterpret_cast<const float2 *>(&r[i * kPairF4 + 2]));
    };
    if (first + kStageRecs <= count) {
#pragma unroll
      for (int i = 0; i < kStageRecs; ++i) add(i);
    } else {
      for (int i = 0; i < count - first; ++i) add(i);
    }
    __syncwarp();
  }
}

// One bit per cluster of [c0, c0 + 32) below k1: whether it is in reach of the box [lo, hi].
__device__ __forceinline__ unsigned near_clusters(float3 lo, float3 hi, int c0, int k1, const float *box_reach,
                                                  const float4 *box) {
  const int mine = c0 + (threadIdx.x & 31);
  bool near = false;
  if (mine < k1) near = !(box_d2(lo, hi, __ldg(&box[2 * mine]), __ldg(&box[2 * mine + 1])) > __ldg(&box_reach[mine]));
  return __ballot_sync(0xffffffffu, near);
}

// The next four clusters of `todo` (bits from cluster c0 on): this lane's atom of each, as an index from
// cluster `base` on, and its entry of `reach`; a reach of -1 where there is none.
__device__ __forceinline__ void next_clusters(unsigned &todo, int c0, int base, const float4 *reach, int (&at)[4],
                                              int atoms, float4 (&t)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int atom = (c0 + __ffs(todo) - 1) * kClusterAtoms + (threadIdx.x & 31);
    t[i] = todo && atom < atoms ? __ldg(&reach[atom]) : make_float4(0.f, 0.f, 0.f, -1.f);
    at[i] = atom - base * kClusterAtoms;
    todo &= todo - 1u;
  }
}

// Append the lanes' values whose atom t is in reach of the box to list[count...], in lane order.
__device__ __forceinline__ void push_hits(unsigned short *list, int &count, float3 lo, float3 hi, float4 t, int value) {
  const bool hit = !(box_d2(lo, hi, t, t) > t.w);
  const unsigned hits = __ballot_sync(0xffffffffu, hit);
  if (hit) list[count + __popc(hits & ((1u << (threadIdx.x & 31)) - 1u))] = (unsigned short)value;
  count += __popc(hits);
}

// The interactions of a warp's points (inside [lo, hi]) with the protein, for ligand type lt: the
// `ncand` candidates at `cand` (protein indices in order) or, without a list, every cluster.
template <int P>
__device__ __forceinline__ void cull_eval(Points<P> &pt, float3 lo, float3 hi, int lt, const unsigned short *cand,
                                          int ncand, WarpList &l, const CullArgs &a) {
  const int lane = threadIdx.x & 31;
  const float4 *reach = a.reach + (size_t)lt * a.natpro_pad;
  int pos = 0, c0 = 0; // next candidate; or next cluster block, and the one whose clusters are `todo`
  unsigned todo = 0;
  for (bool more = true; more;) {
    int count = 0, base = cand ? 0 : c0;
    while (count <= kListFull) {
      int at[4];
      float4 t[4];
      if (cand) {
        more = pos < ncand;
        if (!more) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int k = pos + i * 32 + lane;
          at[i] = k < ncand ? cand[k] : 0;
          t[i] = k < ncand ? __ldg(&reach[at[i]]) : make_float4(0.f, 0.f, 0.f, -1.f);
        }
        pos += 128;
      } else {
        // The list's indices are 16 bits wide: 2,048 clusters from `base` on.
        while (!todo && pos < a.clusters && (count == 0 || pos + 31 - base < 2048)) {
          c0 = pos;
          if (count == 0) base = c0;
          todo = near_clusters(lo, hi, c0, a.clusters, a.box_reach + (size_t)lt * a.clusters, a.box);
          pos += 32;
        }
        more = todo || pos < a.clusters;
        if (!todo) break;
        next_clusters(todo, c0, base, reach, at, a.natpro_pad, t);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) push_hits(l.at, count, lo, hi, t[i], at[i]);
    }
    list_eval<P>(pt, l, count, a.slab + ((size_t)lt * a.natpro_pad + (size_t)base * kClusterAtoms) * kPairF4);
  }
}

// Groups that follow each other share a list of candidates, found by one warp for their common box.
constexpr int kCandidates = 512; // of a list; a super group with more leaves its groups to the clusters
struct Candidates {
  int n; // -1: too many
  unsigned short at[kCandidates + 128];
};

// The box of the points [first, first + count) of the chunk (count >= 1), the whole warp's work.
__device__ __forceinline__ void points_box(const float4 *pts, int first, int count, float3 &lo, float3 &hi) {
  lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
  for (int i = threadIdx.x & 31; i < count; i += 32) {
    const float4 p = pts[first + i];
    lo = make_float3(fminf(lo.x, p.x), fminf(lo.y, p.y), fminf(lo.z, p.z));
    hi = make_float3(fmaxf(hi.x, p.x), fmaxf(hi.y, p.y), fmaxf(hi.z, p.z));
  }
  lo = make_float3(warp_min(lo.x), warp_min(lo.y), warp_min(lo.z));
  hi = make_float3(warp_max(hi.x), warp_max(hi.y), warp_max(hi.z));
}

// The points of the group at `first` (the last point in place of those past n) and their box.
template <int P>
__device__ __forceinline__ void group_points(Points<P> &pt, const float4 *pts, int first, int n, float3 &lo, float3 &hi) {
  lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const float4 p = pts[min(first + i * 32 + (int)(threadIdx.x & 31), n - 1)];
    pt.set(i, p);
    lo = make_float3(fminf(lo.x, p.x), fminf(lo.y, p.y), fminf(lo.z, p.z));
    hi = make_float3(fmaxf(hi.x, p.x), fmaxf(hi.y, p.y), fmaxf(hi.z, p.z));
  }
  lo = make_float3(warp_min(lo.x), warp_min(lo.y), warp_min(lo.z));
  hi = make_float3(warp_max(hi.x), warp_max(hi.y), warp_max(hi.z));
}

// Dynamic shared memory: the chunk's points, the warps' lists and the super groups' candidates.
inline size_t cull_smem_bytes(int chunk, int threads, int P, int supers) {
  return (size_t)chunk * sizeof(float4) + (size_t)(threads / 32) * sizeof(WarpList) +
         (size_t)(supers ? (chunk + (32 * P << supers) - 1) / (32 * P << supers) : 0) * sizeof(Candidates);
}

// K poses per thread (a chunk of K * blockDim.x poses per block), P points per lane of a group.
template <int K, int P> __global__ void __launch_bounds__(kMaxThreads, 2) cull_kernel(const CullArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  float4 *pts = reinterpret_cast<float4 *>(smem); // the chunk's points in sorted order, .w = pose of the chunk
  const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = T >> 5;
  WarpList &list = reinterpret_cast<WarpList *>(pts + K * T)[warp];
  Candidates *cand = reinterpret_cast<Candidates *>(reinterpret_cast<WarpList *>(pts + K * T) + warps);
  __shared__ int bins[kBins];
  __shared__ int warp_total[kMaxThreads / 32];
  __shared__ float red[6][kMaxThreads / 32];
  __shared__ int next_group;

  grid_dep_wait();
  int atom, row, n;
  long long pose0;
  if (a.items) {
    const int4 it = __ldg(&a.items[blockIdx.x]);
    atom = it.x, row = it.y, pose0 = it.z, n = it.w;
  } else {
    row = (int)(blockIdx.x / (unsigned)a.chunks);
    if (a.rows) row = __ldg(&a.rows[row]);
    atom = row + a.atom0;
    pose0 = (long long)(blockIdx.x % (unsigned)a.chunks) * a.chunk;
    n = (int)min((long long)a.chunk, a.nposes - pose0);
  }
  if (a.words && deck_bad_type(a.words)) return;
  const float4 *xf = reinterpret_cast<const float4 *>(a.xform) + pose0 * 3;

  // 1. positions, their box (of regular positions, edge_pose.cuh, where the protein is in reach) and cells
  const float4 la = __ldg(&a.ligand[atom]);
  float x[K], y[K], z[K];
  float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = tid + k * T;
    if (i >= n) continue;
    const float4 r0 = __ldg(xf + i * 3), r1 = __ldg(xf + i * 3 + 1), r2 = __ldg(xf + i * 3 + 2);
    // serial/fasten.hpp:66-73
    x[k] = r0.w + la.x * r0.x + la.y * r0.y + la.z * r0.z;
    y[k] = r1.w + la.x * r1.x + la.y * r1.y + la.z * r1.z;
    z[k] = r2.w + la.x * r2.x + la.y * r2.y + la.z * r2.z;
    if (fabsf(x[k]) + fabsf(y[k]) + fabsf(z[k]) < kPoseReach) {
      lo = make_float3(fminf(lo.x, x[k]), fminf(lo.y, y[k]), fminf(lo.z, z[k]));
      hi = make_float3(fmaxf(hi.x, x[k]), fmaxf(hi.y, y[k]), fmaxf(hi.z, z[k]));
    }
  }
  {
    const float v[6] = {warp_min(lo.x), warp_min(lo.y), warp_min(lo.z), warp_max(hi.x), warp_max(hi.y), warp_max(hi.z)};
#pragma unroll
    for (int d = 0; d < 6; ++d)
      if (lane == 0) red[d][warp] = v[d];
    for (int b = tid; b < kBins; b += T) bins[b] = 0;
    __syncthreads();
    const int w = lane < warps ? lane : 0;
    lo = make_float3(fmaxf(warp_min(red[0][w]), a.lo.x), fmaxf(warp_min(red[1][w]), a.lo.y),
                     fmaxf(warp_min(red[2][w]), a.lo.z));
    hi = make_float3(fminf(warp_max(red[3][w]), a.hi.x), fminf(warp_max(red[4][w]), a.hi.y),
                     fminf(warp_max(red[5][w]), a.hi.z));
  }
  const float ix = hi.x > lo.x ? 8.f / (hi.x - lo.x) : 0.f, iy = hi.y > lo.y ? 8.f / (hi.y - lo.y) : 0.f,
              iz = hi.z > lo.z ? 8.f / (hi.z - lo.z) : 0.f;
  int slot[K]; // cell << 16 | rank in the cell
#pragma unroll
  for (int k = 0; k < K; ++k) {
    slot[k] = -1;
    if (tid + k * T >= n) continue;
    const unsigned qx = min(__float2uint_rz((x[k] - lo.x) * ix), 7u), qy = min(__float2uint_rz((y[k] - lo.y) * iy), 7u),
                   qz = min(__float2uint_rz((z[k] - lo.z) * iz), 7u); // below the box, or not a number: 0
    const int cell = kHilbert.at[qz * 64 + qy * 8 + qx];
    slot[k] = cell << 16 | atomicAdd(&bins[cell], 1);
  }
  __syncthreads();
  // 2. first point of every cell: exclusive scan of the counts.  Scanning warp w owns `per` cells.
  const int scanners = 1 << (31 - __clz(min(warps, kBins / 32))), per = kBins / scanners;
  if (warp < scanners) {
    int run = 0;
    for (int b = warp * per; b < (warp + 1) * per; b += 32) {
      const int v = bins[b + lane];
      int s = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += u;
      }
      bins[b + lane] = run + s - v;
      run += __shfl_sync(0xffffffffu, s, 31);
    }
    if (lane == 0) warp_total[warp] = run;
  }
  if (tid == 0) next_group = 0;
  __syncthreads();
  if (warp > 0 && warp < scanners) {
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? warp_total[lane] : 0);
    for (int b = warp * per; b < (warp + 1) * per; b += 32) bins[b + lane] += before;
  }
  __syncthreads();
  // 3. scatter into sorted order
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (slot[k] >= 0)
      pts[bins[slot[k] >> 16] + (slot[k] & 0xffff)] = make_float4(x[k], y[k], z[k], __int_as_float(tid + k * T));
  __syncthreads();
  // 4. candidates of every super group
  const int lt = __float_as_int(la.w);
  if (a.supers) {
    const int points = 32 * P << a.supers;
    for (int sg = warp; sg * points < n; sg += warps) {
      float3 lo, hi;
      points_box(pts, sg * points, min(points, n - sg * points), lo, hi);
      const float4 *reach = a.reach + (size_t)lt * a.natpro_pad;
      int count = 0;
      for (int c0 = 0; c0 < a.clusters && count <= kCandidates; c0 += 32) {
        unsigned todo = near_clusters(lo, hi, c0, a.clusters, a.box_reach + (size_t)lt * a.clusters, a.box);
        while (todo && count <= kCandidates) {
          int at[4];
          float4 t[4];
          next_clusters(todo, c0, 0, reach, at, a.natpro_pad, t);
#pragma unroll
          for (int i = 0; i < 4; ++i) push_hits(cand[sg].at, count, lo, hi, t[i], at[i]);
        }
      }
      if (lane == 0) cand[sg].n = count <= kCandidates ? count : -1;
    }
    __syncthreads();
  }
  // 5. groups of 32 * P sorted points
  float *out = a.sums + (long long)row * a.stride + (pose0 - a.first);
  for (;;) {
    int g = 0;
    if (lane == 0) g = atomicAdd(&next_group, 1);
    g = __shfl_sync(0xffffffffu, g, 0);
    const int first = g * 32 * P;
    if (first >= n) break;
    Points<P> pt;
    float3 lo, hi;
    group_points(pt, pts, first, n, lo, hi);
    pt.clear();
    const int k = a.supers ? cand[g >> a.supers].n : -1;
    cull_eval<P>(pt, lo, hi, lt, k >= 0 ? cand[g >> a.supers].at : nullptr, k, list, a);
    // The energies to their poses, up to 32 sectors a store; a chunk's row stays in L2 until it is full.  Put
    // in order in shared memory first, three more barriers: 4,096 x 64 x 1,048,576 2,773 us, so 2,628.
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (first + i * 32 + lane < n) out[__float_as_int(pts[first + i * 32 + lane].w)] = pt.energy(i);
  }
}

// A warp for every point, all of whose lanes hold it: its own box, as tight as any.  For so few points that each
// has a warp of its own (points_pay, cull.cu), where latency is all: 64 poses of 938 x 26 16 -> 8 us of kernel.
inline size_t point_smem_bytes(int threads) { return (size_t)(threads / 32) * sizeof(WarpList); }

static __global__ void __launch_bounds__(kMaxThreads, 2) point_kernel(const CullArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  WarpList &list = reinterpret_cast<WarpList *>(smem)[warp];
  grid_dep_wait();
  int atom, row, n;
  long long pose0;
  if (a.items) {
    const int4 it = __ldg(&a.items[blockIdx.x]);
    atom = it.x, row = it.y, pose0 = it.z, n = it.w;
  } else {
    row = (int)(blockIdx.x / (unsigned)a.chunks);
    atom = row + a.atom0;
    pose0 = (long long)(blockIdx.x % (unsigned)a.chunks) * a.chunk;
    n = (int)min((long long)a.chunk, a.nposes - pose0);
  }
  if (a.words && deck_bad_type(a.words)) return;
  const float4 la = __ldg(&a.ligand[atom]);
  const float4 *xf = reinterpret_cast<const float4 *>(a.xform) + pose0 * 3;
  float *out = a.sums + (long long)row * a.stride + (pose0 - a.first);
  for (int i = warp; i < n; i += warps) {
    const float4 r0 = __ldg(xf + i * 3), r1 = __ldg(xf + i * 3 + 1), r2 = __ldg(xf + i * 3 + 2);
    const float4 p = make_float4(r0.w + la.x * r0.x + la.y * r0.y + la.z * r0.z,
                                 r1.w + la.x * r1.x + la.y * r1.y + la.z * r1.z,
                                 r2.w + la.x * r2.x + la.y * r2.y + la.z * r2.z, 0.f); // as in cull_kernel
    Points<1> pt;
    pt.set(0, p);
    pt.clear();
    const float3 at = make_float3(p.x, p.y, p.z);
    cull_eval<1>(pt, at, at, __float_as_int(la.w), nullptr, -1, list, a);
    if ((threadIdx.x & 31) == 0) out[i] = pt.energy(0);
  }
}

// energies[p] = 0.5 * the sum over pose p's ligand atoms in order (no atoms: 0), for the poses
// [first, first + n) of one ligand, or, with folds, for {first pose, poses, rows, ligand} per block.
// With `edges` the irregular poses among them (every pose of an irregular deck or ligand) then get the
// reference's arithmetic: edge_energy of edge_pose.cuh, one pose per warp at a time.
struct FinishArgs {
  const float *sums; // [row][stride], from pose `first` on
  long long stride, first, n;
  int rows;
  int more, last; // the sums add to what energies hold; these are the last rows
  const int4 *folds;
  float *energies;
  const int *perm;       // optional: the pose at each place of the sums and transforms (pose_order.cuh)
  const unsigned *words; // as CullArgs::words; its deck decides whether every pose is irregular
  int edges;
  EdgeArgs e;
};

// The irregular ones of a warp's 32 poses, at the places from w on; this lane's is at energies[q].
__device__ __forceinline__ void rescore_irregular(const FinishArgs &a, bool irregular, long long w, long long q) {
  unsigned bits = __ballot_sync(0xffffffffu, irregular);
  while (bits) {
    const int b = __ffs(bits) - 1;
    bits &= bits - 1u;
    const float e = __shfl_sync(0xffffffffu, edge_energy(a.e, w + b), 0);
    if ((threadIdx.x & 31) == b) a.energies[q] = e;
  }
}

static __global__ void __launch_bounds__(256) cull_finish_kernel(const FinishArgs a) {
  long long p0 = a.first + (long long)blockIdx.x * blockDim.x, p1 = min(p0 + blockDim.x, a.first + a.n);
  int rows = a.rows;
  bool all = a.e.all != 0;
  grid_dep_wait();
  if (a.words) {
    if (deck_bad_type(a.words)) return;
    all = deck_irregular(a.words, a.e.natpro, a.e.natlig);
  }
  if (a.folds) {
    const int4 f = __ldg(&a.folds[blockIdx.x]);
    p0 = f.x, p1 = (long long)f.x + f.y, rows = f.z;
    if (a.edges && *a.e.lig_any > 0) all = a.e.lig_all[f.w] != 0;
  }
  for (long long w = p0 + (threadIdx.x & ~31u); w < p1; w += blockDim.x) {
    const long long p = w + (threadIdx.x & 31);
    long long q = p;
    bool irregular = false;
    if (p < p1) {
      const float *s = a.sums + (p - a.first);
      if (a.perm) q = __ldg(&a.perm[p]);
      float acc = a.more ? a.energies[q] : 0.f;
      int r = 0;
      for (; r + 8 <= rows; r += 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = s[(long long)(r + j) * a.stride];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = __fadd_rn(acc, v[j]);
      }
      for (; r < rows; ++r) acc = __fadd_rn(acc, s[(long long)r * a.stride]);
      a.energies[q] = a.last ? 0.5f * acc : acc;
      irregular = a.edges && a.last && (all || ((a.e.mask[q >> 5] >> (q & 31)) & 1u));
    }
    rescore_irregular(a, irregular, w, q);
  }
}

} // namespace bude
