// cull.cu -- host side of the exact kernel (cull_kernel.cuh, cull.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <numeric>

#include "chain.h"
#include "cull.h"
#include "cull_kernel.cuh"
#include "direct_kernel.cuh"
#include "pose_order.cuh"
#include "pose_xform.cuh"

namespace bude {

// 16 poses per thread x 512 threads: 161, 171 or 191 KiB with lists; with one pose per lane and lists of four
// groups it would be 231, so those go without.
constexpr size_t kCullMaxSmem = 200 * 1024;

// Lists of candidates serve four groups, or the eight tighter ones of sorted poses (4,096 x 64 x 1,048,576
// 2,603 us with four, 2,519 with eight; 64 unsorted ligands 2,664 and 2,703).  A chunk of 256 poses has too
// few groups for them: 64 poses of 938 x 26 27.0 us with, 25.0 without, 205 of 2,672 x 48 45.9 and 41.5.
int cull_supers(int natpro_pad, const bude_launch_cfg &s, int chunk, bool sorted) {
  const int most = s.ppwi * s.wgsize, shift = sorted ? 3 : 2;
  return natpro_pad <= 65536 && chunk > 256 && cull_smem_bytes(most, s.wgsize, s.unroll, shift) <= kCullMaxSmem
             ? shift
             : 0;
}

static CullArgs cull_args(const Context &c, const bude_launch_cfg &s, int chunk, bool sorted) {
  CullArgs a{};
  a.supers = cull_supers(c.natpro_pad, s, chunk, sorted);
  a.slab = c.slab.as<float4>();
  a.reach = c.reach.as<float4>();
  a.box = c.box.as<float4>();
  a.box_reach = c.box_reach.as<float>();
  a.lo = make_float3(c.reach_lo[0], c.reach_lo[1], c.reach_lo[2]);
  a.hi = make_float3(c.reach_hi[0], c.reach_hi[1], c.reach_hi[2]);
  a.natpro_pad = c.natpro_pad;
  a.clusters = c.natpro_pad / kClusterAtoms;
  return a;
}

template <int K, int P>
static cudaError_t launch_kp(const CullArgs *a, unsigned grid, int threads, cudaStream_t st) {
  if (!a)
    return cudaFuncSetAttribute(cull_kernel<K, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCullMaxSmem);
  return launch_chained(cull_kernel<K, P>, grid, (unsigned)threads, cull_smem_bytes(K * threads, threads, P, a->supers),
                        st, *a);
}

template <int K>
static cudaError_t launch_k(const CullArgs *a, unsigned grid, const bude_launch_cfg &s, cudaStream_t st) {
  switch (s.unroll) {
  case 1: return launch_kp<K, 1>(a, grid, s.wgsize, st);
  case 2: return launch_kp<K, 2>(a, grid, s.wgsize, st);
  default: return launch_kp<K, 4>(a, grid, s.wgsize, st);
  }
}

// Launches the shape's kernel; a == nullptr: only sets its shared-memory limit.
static cudaError_t launch_shape(const CullArgs *a, unsigned grid, const bude_launch_cfg &s, cudaStream_t st) {
  switch (s.ppwi) {
  case 1: return launch_k<1>(a, grid, s, st);
  case 2: return launch_k<2>(a, grid, s, st);
  case 4: return launch_k<4>(a, grid, s, st);
  case 8: return launch_k<8>(a, grid, s, st);
  default: return launch_k<16>(a, grid, s, st);
  }
}

int prepare_shape(const bude_launch_cfg &shape) {
  const cudaError_t e = launch_shape(nullptr, 0, shape, nullptr);
  return e == cudaSuccess ? BUDE_OK : cuda_error(e, "launch shape");
}

static int launch(const CullArgs &a, long long grid, const bude_launch_cfg &s, bool points, cudaStream_t st,
                  long long &launches) {
  if (grid > 0x7fffffffLL) return set_error(BUDE_ERR_ARG, "too many poses for one launch");
  if (points) {
    const cudaError_t e =
        launch_chained(point_kernel, (unsigned)grid, (unsigned)s.wgsize, point_smem_bytes(s.wgsize), st, a);
    if (e != cudaSuccess) return cuda_error(e, "point_kernel launch");
    launches++;
    return BUDE_OK;
  }
  int rc = prepare_shape(s);
  if (rc) return rc;
  const cudaError_t e = launch_shape(&a, (unsigned)grid, s, st);
  if (e != cudaSuccess) return cuda_error(e, "cull_kernel launch");
  launches++;
  return BUDE_OK;
}

static int finish(const FinishArgs &f, long long grid, cudaStream_t st, long long &launches) {
  const cudaError_t e = launch_chained(cull_finish_kernel, (unsigned)grid, 256u, 0, st, f);
  if (e != cudaSuccess) return cuda_error(e, "cull_finish_kernel launch");
  launches++;
  return BUDE_OK;
}

// Against a protein of a few dozen atoms nearly every pair is in reach, and many poses leave no SM idle
// without the ligand's atoms spread over the blocks: then sorting positions, boxes, lists and atom sums cost
// more than the pairs they leave out.  The line is 64 natpro^2 poses (at least 16,384), where the two were
// equal or direct_kernel the faster for 1 to 64 ligand atoms, protein at the density of a real one (us culled
// | direct, 1 and 64 ligand atoms): 8 atoms x 16,384 poses 17 | 12 and 44 | 44, x 524,288 36 | 25 and 565 |
// 154; 32 atoms x 65,536 21 | 15 and 132 | 141, x 524,288 41 | 30 and 830 | 496; 64 atoms x 131,072 27 | 21
// and 290 | 361, x 262,144 33 | 27 and 540 | 547, x 524,288 48 | 37 and 1,048 | 953.  Above 64 atoms it takes
// ligands of few atoms, for which the culled path's launches weigh more (x 524,288, 1, 8 and 64 ligand atoms:
// 96 atoms 56 | 44, 208 | 198 and 1,288 | 1,408; 128 atoms 65 | 52, 229 | 255 and 1,415 | 1,864).
bool direct_pays(const Context &c, long long natlig, long long poses) {
  const long long most = 64 + std::min(64LL, 256 / std::max(natlig, 1LL));
  return c.natpro > 0 && c.natpro <= most && poses >= std::max(16384LL, 64LL * c.natpro * c.natpro);
}

// As above; ragged ligands leave a tail, so twice the poses: 64 ligands of 12 to 96 atoms, 321,818 poses, 8 |
// 32 | 64 atoms 292 | 472 | 606 us culled, 112 | 355 | 677 direct; 1,048,576 poses 964 | 1,401 | 1,793 and 253 |
// 865 | 1,636; 256 of 8 to 32, 36,368 poses, 8 | 32 atoms 32 | 42 and 24 | 59.
static bool direct_batch_pays(const Context &c, long long mean_natlig, long long poses) {
  return direct_pays(c, mean_natlig, poses / 2);
}

static int launch_direct(const Context &c, const FinishArgs &f, const float4 *ligand, long long grid,
                         const bude_launch_cfg &s, cudaStream_t st, long long &launches) {
  DirectArgs a{ligand, c.slab.as<float4>(), c.natpro, c.natpro_pad, f};
  cudaError_t e;
  switch (s.ppwi) {
  case 1: e = launch_chained(direct_kernel<1>, (unsigned)grid, (unsigned)s.wgsize, 0, st, a); break;
  case 2: e = launch_chained(direct_kernel<2>, (unsigned)grid, (unsigned)s.wgsize, 0, st, a); break;
  default: e = launch_chained(direct_kernel<4>, (unsigned)grid, (unsigned)s.wgsize, 0, st, a); break;
  }
  if (e != cudaSuccess) return cuda_error(e, "direct_kernel launch");
  launches++;
  return BUDE_OK;
}

// Poses of a direct_kernel block.
static int direct_chunk(const bude_launch_cfg &s) { return std::min(s.ppwi, kDirectPoses) * s.wgsize; }

constexpr double kFewPoints = 9e4; // cull_shape's first line

// Few points (poses x ligand atoms) get a warp each, point_kernel: the GPU has room for 4,864 warps at once,
// and groups of 32 would leave most of it idle and, of poses far apart, span the whole protein.  us culled |
// point_kernel, translations within 3 | 20 A: 4,096 atoms x 26 x 64 46 | 23 and 136 | 22, x 8 x 1,024 38 | 38 and
// 86 | 35; 938 x 26 x 64 38 | 22 and 44 | 21, x 26 x 256 36 | 34 and 40 | 25; 10,000 x 64 x 64 50 | 33 and 257 |
// 32.  Past the line the shared boxes of poses near each other win: 4,096 x 8 x 2,048 37 | 57; small proteins
// reach it sooner: 300 x 26 x 64 26 | 20, x 26 x 256 26 | 30; 100 x 64 x 64 20 | 21, x 26 x 256 20 | 25.
static bool points_pay(int natpro, long long points) { return points <= std::min(8192LL, 4096LL + 4LL * natpro); }

SumsWindow sums_window(int natpro, int natlig, long long nposes, const bude_launch_cfg &cfg, size_t most) {
  SumsWindow w;
  w.points = points_pay(natpro, nposes * natlig);
  // Of fewer points than cull_shape's first line a block takes at most 256 poses, whatever its shape could take:
  // more leave SMs idle (8 x 128 938 x 26 x 1,024 94 us with 1,024, 46 with 256).
  const int block = cfg.ppwi * cfg.wgsize;
  w.chunk = w.points ? cfg.wgsize / 32
                     : even_chunk(nposes, (double)nposes * natlig < kFewPoints ? std::min(block, 256) : block);
  const long long floats = std::max((long long)(most / sizeof(float)), (long long)w.chunk);
  w.atoms = (int)std::min<long long>(natlig, floats / w.chunk);
  w.poses = std::min(nposes, floats / std::max(w.atoms, 1) / w.chunk * w.chunk);
  return w;
}

int cull_range(CullArgs a, FinishArgs f, const bude_launch_cfg &cfg, const SumsWindow &w, int natlig, long long nposes,
               cudaStream_t st, long long &launches) {
  const float *xform = a.xform;
  a.chunk = w.chunk;
  if (w.atoms < natlig) a.rows = nullptr;
  f.sums = a.sums;
  for (long long w0 = 0; w0 < nposes; w0 += w.poses) {
    const long long n = std::min(w.poses, nposes - w0);
    a.nposes = f.n = n;
    a.xform = xform + 12 * w0;
    a.stride = f.stride = n;
    a.chunks = (int)((n + a.chunk - 1) / a.chunk);
    f.first = w0;
    int l = 0;
    do {
      a.atom0 = l;
      f.rows = std::min(w.atoms, natlig - l);
      f.more = l > 0;
      l += f.rows;
      f.last = l >= natlig;
      int rc = f.rows > 0 ? launch(a, (long long)f.rows * a.chunks, cfg, w.points, st, launches) : BUDE_OK;
      if (!rc) rc = finish(f, (n + 255) / 256, st, launches);
      if (rc) return rc;
    } while (l < natlig);
  }
  return BUDE_OK;
}

// Whether an evaluation puts its poses in order first: two launches more, and 8 us more than the plain
// transforms at 65,536 poses, 20 at 1,048,576, against groups with fewer records.  What that saves goes with
// the points and with the atoms near one, so the line is points x protein atoms per cubic Angstrom of their
// box (widened by the reach) = 3,300, where the two were equal or the sorted faster (6 to 96 ligand atoms;
// us plain, then sorted / plain): 400 atoms at 0.05 per cubic Angstrom 500k points 100, 0.98, 1.2M 167, 0.95;
// 1,237 300k 90, 0.91, 900k 176, 0.86; 3,500 220k 77, 0.89, 900k 151, 0.84; 3,500 at 0.015 400k 55, 1.00,
// 740k 82, 0.94.  Fewer than 4,096 poses are a few chunks.  And per pose the sort takes what it takes, so a
// ligand of few atoms does not pay for it, however many the poses: the second line is ligand atoms x density
// = 0.011 (2,000,000 poses, us plain | sorted: 65 x 1 atoms 0.002 134 | 199, 65 x 4 0.008 339 | 386, 100 x 4 0.0106
// 432 | 467, 400 x 2 0.0116 437 | 421, 100 x 8 0.021 762 | 757, 938 x 2 0.017 543 | 475).
static double density(const Context &c) {
  double volume = 1.0;
  for (int d = 0; d < 3; ++d) volume *= (double)c.reach_hi[d] - c.reach_lo[d];
  return c.natpro / volume;
}

bool sort_poses(const Context &c, long long nposes) {
  const double near = c.natlig * density(c); // of a pose
  return c.natpro > 0 && nposes >= 4096 && nposes * near >= 3300.0 && near >= 0.011 && nposes < (1LL << 31) &&
         !direct_pays(c, c.natlig, nposes);
}

// Blocks that all run at once have no last ones: below 100,000 points (one point per thread) there are fewer
// than a wave of them, and 938 x 26 x 64 takes 48 us with or without.
bool row_order_pays(long long n, int natlig) {
  return (double)n * natlig >= 1e5 && natlig > 1 && natlig <= kRowOrderMax;
}

static int order_tile(long long n) {
  const long long per = (n + 607) / 608; // four blocks per SM
  return (int)std::min<long long>((per + kOrderThreads - 1) / kOrderThreads * kOrderThreads, 65536);
}

static int order_coarse(long long n) { return n <= 262144; } // 64 chunks of 4,096: finer cells made none tighter

size_t pose_order_bytes(long long n) {
  const long long tiles = (n + order_tile(n) - 1) / order_tile(n), cells = order_coarse(n) ? kBins / 8 : kBins;
  return ((size_t)2 * n + 6 * kOrderBoxes + (size_t)(tiles + 1) * cells) * sizeof(int);
}

int enqueue_sorted(void *scratch, const float *poses, long long stride, long long n, float4 *xform, unsigned *mask,
                   const RowOrder &ro, const int **perm, cudaStream_t st) {
  PoseOrder o;
  o.perm = static_cast<int *>(scratch);
  o.key = static_cast<unsigned *>(scratch) + n;
  o.boxes = static_cast<float *>(scratch) + 2 * n;
  o.count = static_cast<int *>(scratch) + 2 * n + 6 * kOrderBoxes;
  o.coarse = order_coarse(n);
  o.base = o.count + o.cells();
  o.tile = order_tile(n);
  const unsigned tiles = (unsigned)((n + o.tile - 1) / o.tile);
  const int boxes = (int)std::min<long long>(kOrderBoxes, (n + kOrderThreads - 1) / kOrderThreads);
  pose_box_kernel<<<boxes, kOrderThreads, 0, st>>>(poses, stride, n, o);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = launch_chained(pose_cell_kernel, tiles + (ro.rows ? 1u : 0u), (unsigned)kOrderThreads, 0, st, poses, stride, n,
                       boxes, o, ro);
  if (e == cudaSuccess)
    e = launch_chained(pose_place_kernel, tiles, (unsigned)kOrderThreads, 0, st, poses, stride, n, o, xform, mask);
  if (e != cudaSuccess) return cuda_error(e, "pose order launch");
  *perm = o.perm;
  return BUDE_OK;
}

// As sort_poses, for the ligands of more than a chunk, with four launches instead of one: 64 ligands of 12
// to 96 atoms x 1,024 to 16,384 poses 2,217 us plain, 2,167 sorted, 256 x 4,096 to 65,536 16.83 and 15.02 ms.
// Ligands of a chunk or less gain nothing (24 of 20 to 40 atoms x 256 to 1,024 stay plain, 177 us).
// Its second line is 0.03 for the mean ligand of them (2,000,000 poses of one ligand, plain | sorted: 2,672 x 2
// atoms 0.026 441 | 525, 200 x 8 0.032 1,022 | 1,064, 938 x 4 0.035 696 | 720, 400 x 8 0.046 1,273 | 1,224; 524,288
// poses, 938 x 4 220 | 208).
bool sort_batch(const Context &c, int chunk) {
  double points = 0, poses = 0;
  for (int l = 0; l < c.nligands; ++l) {
    const long long n = c.pose_off[l + 1] - c.pose_off[l];
    if (n <= chunk) continue;
    points += (double)n * (c.lig_off[l + 1] - c.lig_off[l]);
    poses += (double)n;
  }
  return c.natpro > 0 && points * density(c) >= 10000.0 && points * density(c) >= 0.03 * poses;
}

size_t batch_order_bytes(const Context &c, size_t tiles) {
  return (size_t)c.batch_poses * (3 * sizeof(float4) + 2 * sizeof(int)) +
         ((size_t)c.nligands * (6 + kBatchCells) + tiles * kBatchCells) * sizeof(int);
}

int enqueue_batch_order(Context &c, const CullPlan &plan, const int4 *tiles, const float *xform, void *scratch,
                        const float **sorted, const int **perm) {
  BatchOrder o;
  o.pose_off = c.b_pose_off;
  o.tiles = tiles;
  o.xform = reinterpret_cast<const float4 *>(xform);
  o.sorted = static_cast<float4 *>(scratch);
  o.perm = reinterpret_cast<int *>(o.sorted + 3 * c.batch_poses);
  o.key = reinterpret_cast<unsigned *>(o.perm + c.batch_poses);
  o.boxes = o.key + c.batch_poses;
  o.count = reinterpret_cast<int *>(o.boxes + 6 * (size_t)c.nligands);
  o.base = o.count + kBatchCells * (size_t)c.nligands;
  const unsigned n = (unsigned)plan.folds.size();
  cudaError_t e = cudaMemsetAsync(o.boxes, 0, (6 + kBatchCells) * sizeof(int) * (size_t)c.nligands, c.stream);
  if (e == cudaSuccess) {
    batch_box_kernel<<<n, 256, 0, c.stream>>>(o);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = launch_chained(batch_cell_kernel, n, 256u, 0, c.stream, o);
  if (e == cudaSuccess) e = launch_chained(batch_place_kernel, n, 256u, 0, c.stream, o);
  if (e != cudaSuccess) return cuda_error(e, "batch pose order launch");
  c.launches += 3;
  *sorted = reinterpret_cast<const float *>(o.sorted);
  *perm = o.perm;
  return BUDE_OK;
}

int enqueue_poses(Context &c, const float *poses, long long stride, long long n, float *xform, unsigned *mask,
                  const int **perm) {
  *perm = nullptr;
  float4 *rows = reinterpret_cast<float4 *>(xform);
  int rc = c.rows.reserve(kRowOrderMax * sizeof(int), "row order");
  if (rc) return rc;
  const RowOrder ro{c.ligand.as<float4>(),
                    c.reach.as<float4>(),
                    c.natlig,
                    c.natpro,
                    c.natpro_pad,
                    row_order_pays(n, c.natlig) && !direct_pays(c, c.natlig, n) ? c.rows.as<int>() : nullptr,
                    nullptr};
  // In the order given where there is no memory for another: the same energies.
  if (sort_poses(c, n) && c.order.reserve(pose_order_bytes(n), "pose order") == BUDE_OK) {
    rc = enqueue_sorted(c.order.ptr, poses, stride, n, rows, mask, ro, perm, c.stream);
    c.launches += rc ? 0 : 3;
    return rc;
  }
  pose_xform_kernel<<<(unsigned)((n + 255) / 256 + (ro.rows ? 1 : 0)), 256, 0, c.stream>>>(poses, stride, n, rows, mask,
                                                                                         ro);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "pose_xform_kernel launch");
  c.launches++;
  return BUDE_OK;
}

int launch_exact_range(Context &c, const bude_launch_cfg &cfg, const float4 *ligand, int natlig, bool all_irregular,
                       const unsigned *mask, const float *xform, float *energies, long long nposes, bool ordered,
                       const int *perm) {
  if (nposes == 0) return BUDE_OK;
  FinishArgs f{};
  f.energies = energies;
  f.perm = perm;
  f.edges = mask != nullptr;
  f.e = edge_args_single(c, ligand, natlig, all_irregular, mask, xform);
  if (!perm && direct_pays(c, natlig, nposes)) {
    f.n = nposes;
    f.rows = natlig;
    return launch_direct(c, f, ligand, (nposes + direct_chunk(cfg) - 1) / direct_chunk(cfg), cfg, c.stream, c.launches);
  }
  SumsWindow w{};
  const int rc = reserve_sums(c.partial, [&](size_t most) {
    w = sums_window(c.natpro, natlig, nposes, cfg, most);
    return (size_t)w.atoms * w.poses * sizeof(float);
  });
  if (rc) return rc;
  CullArgs a = cull_args(c, cfg, w.chunk, perm != nullptr);
  a.ligand = ligand;
  a.xform = xform;
  a.sums = c.partial.as<float>();
  if (ordered && row_order_pays(nposes, natlig)) a.rows = c.rows.as<int>();
  return cull_range(a, f, cfg, w, natlig, nposes, c.stream, c.launches);
}

CullPlan plan_cull(const Context &c, const std::vector<int> &lig, const std::vector<long long> &first,
                   const std::vector<long long> &count, const bude_launch_cfg &shape, size_t most) {
  CullPlan plan;
  long long points = 0, poses = 0;
  for (size_t i = 0; i < lig.size(); ++i) {
    points += count[i] * (c.lig_off[lig[i] + 1] - c.lig_off[lig[i]]);
    poses += count[i];
  }
  plan.direct = direct_batch_pays(c, points / std::max(poses, 1LL), poses);
  if (plan.direct) {
    for (size_t i = 0; i < lig.size(); ++i)
      for_each_item(count[i], 1, direct_chunk(shape), [&](long long p, int n) {
        plan.folds.push_back(make_int4((int)(first[i] + p), n, c.lig_off[lig[i] + 1] - c.lig_off[lig[i]], lig[i]));
      });
    CullPlan::Window w{};
    w.folds = (int)plan.folds.size();
    plan.windows.push_back(w);
    return plan;
  }
  plan.points = points_pay(c.natpro, points);
  const int block = shape.wgsize / 32; // of point_kernel
  struct Chunk {
    int lig, n;
    long long pose;
  };
  std::vector<Chunk> chunks; // of the window being filled
  CullPlan::Window w{};
  auto natlig = [&](int l) { return c.lig_off[l + 1] - c.lig_off[l]; };
  auto close = [&]() {
    if (chunks.empty()) return;
    w.item0 = (int)plan.items.size();
    w.fold0 = (int)plan.folds.size();
    for (size_t i = 0, j = 0; i < chunks.size(); i = j) {
      long long n = 0; // of the chunks that one cut into folds takes: a ligand's small ones together
      do n += chunks[j++].n;
      while (plan.points && j < chunks.size() && chunks[j].lig == chunks[i].lig);
      for_each_item(n, 1, kFoldPoses, [&](long long p, int m) {
        plan.folds.push_back(make_int4((int)(chunks[i].pose + p), m, natlig(chunks[i].lig), chunks[i].lig));
      });
    }
    // Longest ligands first; the chunks of one ligand and atom next to each other (they read the same
    // records).
    std::stable_sort(chunks.begin(), chunks.end(),
                     [&](const Chunk &x, const Chunk &y) { return natlig(x.lig) > natlig(y.lig); });
    for (size_t i = 0, j = 0; i < chunks.size(); i = j) {
      while (j < chunks.size() && chunks[j].lig == chunks[i].lig) ++j;
      const int l = chunks[i].lig;
      for (int r = 0; r < natlig(l); ++r)
        for (size_t k = i; k < j; ++k)
          plan.items.push_back(make_int4(c.lig_off[l] + r, r, (int)chunks[k].pose, chunks[k].n));
    }
    w.items = (int)plan.items.size() - w.item0;
    w.folds = (int)plan.folds.size() - w.fold0;
    plan.sums_bytes = std::max(plan.sums_bytes, (size_t)w.n * w.atoms * sizeof(float));
    plan.windows.push_back(w);
    chunks.clear();
    w = CullPlan::Window{};
  };
  for (size_t i = 0; i < lig.size(); ++i) {
    const int per = plan.points && natlig(lig[i]) > 0 ? block : even_chunk(count[i], shape.ppwi * shape.wgsize);
    for (long long p = 0; p < count[i]; p += per) {
      const int n = (int)std::min<long long>(per, count[i] - p);
      const long long at = first[i] + p;
      if (!chunks.empty() &&
          (size_t)(at + n - w.first) * std::max(w.atoms, natlig(lig[i])) * sizeof(float) > most)
        close();
      if (chunks.empty()) w.first = at;
      w.n = at + n - w.first;
      w.atoms = std::max(w.atoms, natlig(lig[i]));
      chunks.push_back({lig[i], n, at});
    }
  }
  close();
  return plan;
}

int enqueue_plan(Context &c, const bude_launch_cfg &shape, const CullPlan &plan, const int4 *items, const int4 *folds,
                 const float *xform, float *energies, float *sums, bool edges, cudaStream_t st, const int *perm) {
  CullArgs a = cull_args(c, shape, shape.ppwi * shape.wgsize, perm != nullptr);
  a.ligand = c.b_ligands;
  a.xform = xform;
  a.sums = sums;
  FinishArgs f{};
  f.sums = sums;
  f.energies = energies;
  f.perm = perm;
  f.edges = edges;
  f.last = 1;
  f.e = edge_args_batch(c, xform);
  if (plan.direct) {
    int rc = BUDE_OK;
    for (const CullPlan::Window &w : plan.windows) {
      f.folds = folds + w.fold0;
      if (!rc && w.folds > 0) rc = launch_direct(c, f, c.b_ligands, w.folds, shape, st, c.launches);
    }
    return rc;
  }
  for (const CullPlan::Window &w : plan.windows) {
    a.items = items + w.item0;
    a.stride = f.stride = w.n;
    a.first = f.first = w.first;
    int rc = w.items > 0 ? launch(a, w.items, shape, plan.points, st, c.launches) : BUDE_OK;
    f.folds = folds + w.fold0;
    if (!rc && w.folds > 0) rc = finish(f, w.folds, st, c.launches);
    if (rc) return rc;
  }
  return BUDE_OK;
}

// A chunk wants to be large (its groups are tighter: 4,096 poses of the 4,096 x 64 deck leave 69 records
// per group of 64, 2,048 leave 82), but the launch wants several blocks per SM, one per chunk and ligand
// atom.  The lines lie where one shape overtook the next over 64 to 262,144 poses against 938 x 26,
// 2,672 x 48 and 4,096 x 64 atoms (us, smaller | larger shape): 1 x 256 | 2 x 512 at 65k points (poses x
// ligand atoms) 33 | 37, at 120k 94 | 78; 2 x 512 | 4 x 512 at 786k 190 | 200, at 1.05M 119 | 116; 4 x 512
// | 8 x 512 at 3.1M 480 | 491, at 6.3M 1,023 | 944.  One point per lane below the first line (latency:
// twice the warps), two above it; four lose to two nearly everywhere.  Ligands of fewer poses than a chunk
// take the smallest shape that holds them: 1,024 ligands of 410 poses 4 x 128 4.9 ms, 2 x 256 5.1, 4 x 64
// 6.2; 64 of 1,000 4 x 256 0.66 ms, 2 x 256 0.73; 128 of 205 2 x 128 0.45 ms, 1 x 256 0.49.
bude_launch_cfg cull_shape(long long n, int natlig, int ligands) {
  const double points = (double)n * natlig * ligands;
  bude_launch_cfg s{1, n <= 64 ? 64 : (n <= 128 ? 128 : 256), 1, 64, 1, 0};
  if (points < kFewPoints) return s;
  const int many[][2] = {{8, 512}, {4, 512}, {4, 256}, {4, 128}, {2, 128}}, few[][2] = {{2, 512}, {2, 256}, {2, 128}};
  const int(*shape)[2] = points < 9e5 ? few : (points < 3.8e6 ? many + 1 : many);
  const int(*last)[2] = points < 9e5 ? few + 2 : many + 4;
  while (shape < last && (long long)shape[1][0] * shape[1][1] >= n) ++shape;
  s.ppwi = (*shape)[0];
  s.wgsize = (*shape)[1];
  s.unroll = 2;
  return s;
}

// Of direct_kernel, one pose per thread where there are few, to have warps enough, four where there are many:
// 8 | 32 protein atoms x 26 ligand atoms x 32,768 poses 29 | 65 us with one, 29 | 64 with two, 35 | 88 with
// four; x 131,072 64 | 184, 37 | 94, 40 | 98; x 262,144 80 | 253, 63 | 180, 50 | 132.
bude_launch_cfg exact_shape(const Context &c, long long n, int natlig, int ligands) {
  const long long all = n * ligands;
  if (ligands > 1 ? !direct_batch_pays(c, natlig, all) : !direct_pays(c, natlig, all))
    return cull_shape(n, natlig, ligands);
  bude_launch_cfg s{all >= 200000 ? 4 : (all >= 32768 ? 2 : 1), 128, 1, 64, 1, 0};
  while (s.wgsize > 32 && (long long)s.ppwi * s.wgsize > n) s.wgsize /= 2;
  while (s.ppwi > 1 && (long long)s.ppwi * s.wgsize > n) s.ppwi /= 2;
  return s;
}

} // namespace bude
