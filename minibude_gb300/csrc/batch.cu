// batch.cu -- host side of batched ragged scoring: many ligands with uneven atom and pose counts
// against one protein, in one CUDA-graph-captured launch of the exact kernel over all of them, or, for
// comparison, one plain launch per ligand.
//
// The reference scores one ligand per run of its driver (src/main.cpp); a virtual screen runs it
// once per ligand.  Here the batch shares the protein's tables and the pose-transform pass, and one
// launch takes the (ligand, pose chunk, atom) items of all ligands, longest first.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "cull.h"
#include "pose_xform.cuh"

namespace bude {

void release_batch(Context &c) {
  if (c.graph) cudaGraphExecDestroy(c.graph);
  c.graph = nullptr;
  c.b_poses.release();
  c.b_xform.release();
  c.b_energies.release();
  c.b_items.release();
  c.b_folds.release();
  c.b_sums.release();
  c.b_order.release();
  c.b_edge_mask.release();
  c.b_meta.release();
  c.b_lig_all_host.clear();
  c.b_atoms_host.clear();
  c.have_batch = false;
  delete c.plan;
  c.plan = nullptr;
}

static void drop_graph(Context &c) {
  if (c.graph) cudaGraphExecDestroy(c.graph);
  c.graph = nullptr;
}

// A plan's blocks in the order of their work, longest first (RowOrder): the weights, one warp per item
// {atom, row, first pose, poses}, and the ranks, one thread per item; once per plan and set of ligands, 8 us.  24 ligands of 20 to
// 40 atoms x 256 to 1,024 poses (736 blocks) 179 -> 163 us an evaluation, 64 of 12 to 96 atoms x 1,024 to
// 16,384 (6,253 blocks) 2,197 -> 2,100.  Every item is compared with every other, so up to 16,384.
constexpr int kPlanOrderMax = 16384;
static __global__ void __launch_bounds__(256) item_weight_kernel(const int4 *items, int n, const float4 *ligands,
                                                                 const float4 *reach, int natpro, int natpro_pad,
                                                                 float *weight) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;
  const float w = (float)items[i].w * atom_weight(ligands[items[i].x], reach, natpro, natpro_pad);
  if ((threadIdx.x & 31) == 0) weight[i] = w;
}

static __global__ void __launch_bounds__(256) item_rank_kernel(const int4 *items, int n, const float *weight,
                                                               int4 *ranked) {
  __shared__ float tile[256];
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const float w = i < n ? weight[i] : 0.f;
  int rank = 0;
  for (int t = 0; t < n; t += 256) {
    const int j = t + (int)threadIdx.x;
    __syncthreads();
    tile[threadIdx.x] = j < n ? weight[j] : -1.f; // weights are at least 0
    __syncthreads();
    for (int k = 0; k < 256; ++k) rank += tile[k] > w || (tile[k] == w && t + k < i);
  }
  if (i < n) ranked[rank] = items[i];
}

// b_items: a ranked plan's items as they are run, as they were cut, their weights.
static int rank_items(Context &c, int n) {
  int4 *items = c.b_items.as<int4>(), *given = items + n;
  float *weight = reinterpret_cast<float *>(items + 2 * n);
  item_weight_kernel<<<(unsigned)(n + 7) / 8, 256, 0, c.stream>>>(given, n, c.b_ligands, c.reach.as<float4>(), c.natpro,
                                                                  c.natpro_pad, weight);
  item_rank_kernel<<<(unsigned)(n + 255) / 256, 256, 0, c.stream>>>(given, n, weight, items);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "batch item ranking");
  c.launches += 2;
  return BUDE_OK;
}

int upload_batch(Context &c, const bude_atom *protein, int natpro, const bude_ffparams *ff, int ntypes, int nligands,
                 const bude_atom *atoms, const int32_t *lig_off, const float *poses, long long pose_stride,
                 const int64_t *pose_off) {
  // A batch of the same shape as the uploaded one (same ligand sizes and pose counts, same protein
  // and forcefield) keeps its work items and captured graph: only the atoms and poses are copied.  Other
  // atoms rank the items anew and end the tuned launch shape.
  const bool same_shape = c.have_batch && nligands == c.nligands && lig_off && pose_off &&
                          std::equal(lig_off, lig_off + nligands + 1, c.lig_off.begin()) &&
                          std::equal(pose_off, pose_off + nligands + 1, c.pose_off.begin());
  c.have_batch = false;
  c.have_deck = false;
  if (nligands < 0 || !lig_off || !pose_off || ntypes <= 0 || !ff || natpro < 0 || (natpro > 0 && !protein))
    return set_error(BUDE_ERR_ARG, "bad batch sizes or pointers");
  if (lig_off[0] != 0 || pose_off[0] != 0) return set_error(BUDE_ERR_ARG, "batch offsets must start at 0");
  for (int l = 0; l < nligands; ++l)
    if (lig_off[l + 1] < lig_off[l] || pose_off[l + 1] < pose_off[l])
      return set_error(BUDE_ERR_ARG, "batch offsets must not decrease (ligand %d)", l);
  const int total_atoms = lig_off[nligands];
  const long long total_poses = pose_off[nligands];
  if ((total_atoms > 0 && !atoms) || (total_poses > 0 && (!poses || pose_stride < total_poses)))
    return set_error(BUDE_ERR_ARG, "bad batch atoms or poses");
  // Work items (batch, screen and surrogate) carry pose indices as 32-bit integers.
  if (total_poses > 0x7fffffffLL)
    return set_error(BUDE_ERR_ARG, "a batch holds at most 2^31 - 1 poses (got %lld)", total_poses);
  for (int i = 0; i < natpro; ++i)
    if (protein[i].type < 0 || protein[i].type >= ntypes)
      return set_error(BUDE_ERR_TYPE, "protein atom %d has type %d outside the forcefield (%d types)", i,
                       protein[i].type, ntypes);
  for (int i = 0; i < total_atoms; ++i)
    if (atoms[i].type < 0 || atoms[i].type >= ntypes)
      return set_error(BUDE_ERR_TYPE, "ligand atom %d of the batch has type %d outside the forcefield (%d types)", i,
                       atoms[i].type, ntypes);
  // Protein slab (shared with the single-deck path; rebuilt only for another protein/forcefield).
  bool rebuilt = false;
  int rc = ensure_slab(c, protein, natpro, ff, ntypes, &rebuilt);
  if (rc) return rc;
  const bool keep = same_shape && !rebuilt;
  if (!keep) drop_graph(c);
  const long long np = std::max(total_poses, 1LL);
  const size_t at_any = (size_t)(nligands + 1) * sizeof(long long), at_lig = at_any + 2 * sizeof(int),
               at_atoms = (at_lig + (size_t)(nligands + 1) * sizeof(int) + 15) / 16 * 16,
               at_all = at_atoms + (size_t)total_atoms * sizeof(bude_atom), meta_bytes = at_all + (size_t)nligands;
  rc = reserve_together({{&c.b_poses, (size_t)6 * np * sizeof(float)},
                         {&c.b_xform, (size_t)12 * np * sizeof(float)},
                         {&c.b_energies, (size_t)np * sizeof(float)},
                         {&c.b_edge_mask, (size_t)(np + 31) / 32 * sizeof(unsigned)},
                         {&c.b_meta, meta_bytes}},
                        "batch");
  if (rc) return rc;
  std::vector<unsigned char> meta(meta_bytes);
  std::memcpy(meta.data(), pose_off, at_any);
  std::memcpy(meta.data() + at_lig, lig_off, (size_t)(nligands + 1) * sizeof(int));
  if (total_atoms > 0) std::memcpy(meta.data() + at_atoms, atoms, (size_t)total_atoms * sizeof(bude_atom));
  // Ligands outside the regular-deck bounds (edge_pose.cuh): all their poses go to edge_energy.
  unsigned char *lig_all = meta.data() + at_all;
  int n_irregular = 0;
  for (int l = 0; l < nligands; ++l) {
    lig_all[l] = !ligand_regular(c, atoms + lig_off[l], lig_off[l + 1] - lig_off[l], ff);
    n_irregular += lig_all[l];
  }
  std::memcpy(meta.data() + at_any, &n_irregular, sizeof n_irregular);
  cudaError_t e = cudaMemcpyAsync(c.b_meta.ptr, meta.data(), meta_bytes, cudaMemcpyHostToDevice, c.stream);
  if (e == cudaSuccess && total_poses > 0)
    e = copy2d_sync(c, c.b_poses.ptr, (size_t)total_poses * sizeof(float), poses, (size_t)pose_stride * sizeof(float),
                    (size_t)total_poses * sizeof(float), 6, cudaMemcpyHostToDevice);
  else if (e == cudaSuccess)
    e = cudaStreamSynchronize(c.stream);
  if (e != cudaSuccess) return cuda_error(e, "batch upload");
  const unsigned char *dev = c.b_meta.as<unsigned char>();
  c.b_pose_off = reinterpret_cast<const long long *>(dev);
  c.b_lig_any = reinterpret_cast<const int *>(dev + at_any);
  c.b_lig_off = reinterpret_cast<const int *>(dev + at_lig);
  c.b_ligands = reinterpret_cast<const float4 *>(dev + at_atoms);
  c.b_lig_all = dev + at_all;
  c.b_lig_all_host.assign(lig_all, lig_all + nligands);
  const size_t atom_bytes = (size_t)total_atoms * sizeof(bude_atom);
  const bool same_atoms = c.b_atoms_host.size() == (size_t)total_atoms &&
                          (atom_bytes == 0 || std::memcmp(c.b_atoms_host.data(), atoms, atom_bytes) == 0);
  if (!same_atoms) {
    c.b_atoms_host.assign(atoms, atoms + total_atoms);
    c.batch_tuned_key = -1;
    if (keep && c.graph && c.plan->ranked) rc = rank_items(c, (int)c.plan->items.size());
    if (rc) return rc;
  }
  c.have_batch = true;
  ++c.batch_uploads;
  if (keep) return BUDE_OK;
  ++c.batch_gen;
  c.nligands = nligands;
  c.lig_off.assign(lig_off, lig_off + nligands + 1);
  c.pose_off.assign(pose_off, pose_off + nligands + 1);
  c.batch_poses = total_poses;
  c.batch_tuned_key = -1;
  return BUDE_OK;
}

bude_launch_cfg batch_shape(const Context &c) {
  const int nl = std::max(c.nligands, 1);
  return exact_shape(c, std::max(c.batch_poses / nl, 1LL), std::max(c.lig_off[c.nligands] / nl, 1), nl);
}

// Plan of the whole batch for a launch shape, on the device (b_items, b_folds, b_sums).
static int build_plan(Context &c, const bude_launch_cfg &cfg, CullPlan *out) {
  if (c.batch_poses > 0x7fffffffLL) return set_error(BUDE_ERR_ARG, "batch too large for 32-bit pose indices");
  std::vector<int> lig((size_t)c.nligands);
  std::iota(lig.begin(), lig.end(), 0);
  std::vector<long long> count((size_t)c.nligands);
  for (int l = 0; l < c.nligands; ++l) count[(size_t)l] = c.pose_off[l + 1] - c.pose_off[l];
  int rc = reserve_sums(c.b_sums, [&](size_t most) {
    *out = plan_cull(c, lig, c.pose_off, count, cfg, most);
    return out->sums_bytes;
  });
  if (rc) return rc;
  const int n = (int)out->items.size();
  out->ranked = n > 1 && n <= kPlanOrderMax && out->windows.size() == 1;
  rc = c.b_items.reserve((size_t)std::max(n, 1) * (out->ranked ? 2 * sizeof(int4) + sizeof(float) : sizeof(int4)),
                         "batch items");
  if (!rc) rc = c.b_folds.reserve(std::max<size_t>(out->folds.size(), 1) * sizeof(int4), "batch items");
  if (rc) return rc;
  // In the order given where there is no memory for another: the same energies.
  out->sorted = !out->direct && sort_batch(c, cfg.ppwi * cfg.wgsize) &&
                c.b_order.reserve(batch_order_bytes(c, out->folds.size()), "batch pose order") == BUDE_OK;
  int4 *items = c.b_items.as<int4>();
  cudaError_t e = copy_sync(c, out->ranked ? items + n : items, out->items.data(), out->items.size() * sizeof(int4),
                            cudaMemcpyHostToDevice);
  if (e == cudaSuccess && out->ranked) rc = rank_items(c, n);
  if (rc) return rc;
  if (e == cudaSuccess)
    e = copy_sync(c, c.b_folds.ptr, out->folds.data(), out->folds.size() * sizeof(int4), cudaMemcpyHostToDevice);
  return e == cudaSuccess ? BUDE_OK : cuda_error(e, "batch item upload");
}

static int enqueue_transforms(Context &c) {
  if (c.batch_poses == 0) return BUDE_OK;
  const int tb = 256;
  pose_xform_kernel<<<(unsigned)((c.batch_poses + tb - 1) / tb), tb, 0, c.stream>>>(
      c.b_poses.as<float>(), c.batch_poses, c.batch_poses, c.b_xform.as<float4>(), c.b_edge_mask.as<unsigned>(),
      RowOrder{});
  c.launches++;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? BUDE_OK : cuda_error(e, "pose transforms");
}

// Enqueue one evaluation of the whole batch: transforms, their order, then the plan's windows.
static int enqueue_whole(Context &c, const bude_launch_cfg &cfg, const CullPlan &plan) {
  int rc = enqueue_transforms(c);
  const float *xform = c.b_xform.as<float>();
  const int *perm = nullptr;
  if (!rc && plan.sorted)
    rc = enqueue_batch_order(c, plan, c.b_folds.as<int4>(), xform, c.b_order.ptr, &xform, &perm);
  if (rc) return rc;
  return enqueue_plan(c, cfg, plan, c.b_items.as<int4>(), c.b_folds.as<int4>(), xform, c.b_energies.as<float>(),
                      c.b_sums.as<float>(), true, c.stream, perm);
}

// The evaluation as a CUDA graph, captured once per launch shape.
static int ensure_graph(Context &c, const bude_launch_cfg &cfg) {
  const bool same = c.graph && c.graph_cfg.ppwi == cfg.ppwi && c.graph_cfg.wgsize == cfg.wgsize &&
                    c.graph_cfg.unroll == cfg.unroll;
  if (same) return BUDE_OK;
  drop_graph(c);
  if (!c.plan) c.plan = new CullPlan();
  int rc = build_plan(c, cfg, c.plan);
  // Kernel attributes are set, and errors of a launch shape come up, before the capture.
  if (!rc) rc = prepare_shape(cfg);
  if (rc) return rc;
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return cuda_error(e, "graph capture begin");
  const long long launches0 = c.launches;
  rc = enqueue_whole(c, cfg, *c.plan);
  c.graph_launches = c.launches - launches0;
  c.launches = launches0; // captured, not launched
  e = cudaStreamEndCapture(c.stream, &g);
  if (!rc && e != cudaSuccess) rc = cuda_error(e, "graph capture end");
  if (!rc) {
    e = cudaGraphInstantiate(&c.graph, g, 0);
    if (e != cudaSuccess) rc = cuda_error(e, "graph instantiate");
  }
  if (g) cudaGraphDestroy(g);
  if (rc) {
    c.graph = nullptr;
    return rc;
  }
  c.graph_cfg = cfg;
  return BUDE_OK;
}

int enqueue_batch(Context &c, const bude_launch_cfg &cfg, int per_ligand) {
  if (!c.have_batch) return set_error(BUDE_ERR_STATE, "no batch uploaded");
  bude_launch_cfg shape = cfg;
  shape.cluster = 0;
  int rc = check_cfg(c, shape);
  if (rc) return rc;
  if (!per_ligand) {
    rc = ensure_graph(c, shape);
    if (rc) return rc;
    cudaError_t e = cudaGraphLaunch(c.graph, c.stream);
    if (e != cudaSuccess) return cuda_error(e, "graph launch");
    c.launches += c.graph_launches;
    return BUDE_OK;
  }
  // One plain launch per ligand after one transform pass over all poses.
  rc = enqueue_transforms(c);
  for (int l = 0; l < c.nligands && !rc; ++l)
    rc = launch_exact_range(c, cfg, c.b_ligands + c.lig_off[l], c.lig_off[l + 1] - c.lig_off[l], false,
                            nullptr, c.b_xform.as<float>() + c.pose_off[l] * 12,
                            c.b_energies.as<float>() + c.pose_off[l], c.pose_off[l + 1] - c.pose_off[l]);
  return rc ? rc : enqueue_edge_batch(c, c.b_xform.as<float>(), c.b_energies.as<float>(), nullptr, c.stream);
}

int autotune_batch(Context &c, int max_ms, bude_launch_cfg &best, float *best_ms) {
  if (!c.have_batch) return set_error(BUDE_ERR_STATE, "no batch uploaded");
  if (c.batch_tuned_key == c.batch_poses) {
    best = c.batch_tuned;
    if (best_ms) *best_ms = c.batch_tuned_ms;
    return BUDE_OK;
  }
  // The rule's shape first, then its neighbours in chunk size and group width, each timed on the whole
  // batch after one untimed evaluation.
  std::vector<bude_launch_cfg> cands{batch_shape(c)};
  for (const bude_launch_cfg &s : {bude_launch_cfg{8, 512, 1, 64, 2, 0}, bude_launch_cfg{4, 512, 1, 64, 2, 0},
                                   bude_launch_cfg{4, 256, 1, 64, 2, 0}, bude_launch_cfg{2, 256, 1, 64, 2, 0},
                                   bude_launch_cfg{4, 128, 1, 64, 2, 0}, bude_launch_cfg{1, 256, 1, 64, 1, 0}})
    if (s.ppwi != cands[0].ppwi || s.wgsize != cands[0].wgsize || s.unroll != cands[0].unroll) cands.push_back(s);
  float best_t = 1e30f;
  float spent = 0.f;
  int rc = BUDE_OK;
  EventSet ev(2);
  if (!ev.ok()) return set_error(BUDE_ERR_CUDA, "could not create the autotuner's events");
  drop_graph(c); // its items and sums are overwritten
  for (const bude_launch_cfg &cfg : cands) {
    CullPlan plan;
    rc = build_plan(c, cfg, &plan);
    if (!rc) rc = enqueue_whole(c, cfg, plan); // warm-up
    cudaEventRecord(ev[0], c.stream);
    if (!rc) rc = enqueue_whole(c, cfg, plan);
    cudaEventRecord(ev[1], c.stream);
    const cudaError_t e = cudaStreamSynchronize(c.stream);
    if (!rc && e != cudaSuccess) rc = cuda_error(e, "batch autotune");
    if (rc) break;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev[0], ev[1]);
    spent += 2.f * ms;
    if (ms < best_t) {
      best_t = ms;
      best = cfg;
    }
    if (spent > (float)std::max(max_ms, 1)) break;
  }
  if (rc) return rc;
  if (best_t >= 1e30f) return set_error(BUDE_ERR_ARG, "no batch launch shape fits this device");
  c.batch_tuned = best;
  c.batch_tuned_ms = best_t;
  c.batch_tuned_key = c.batch_poses;
  if (best_ms) *best_ms = best_t;
  return BUDE_OK;
}

} // namespace bude

using namespace bude;

extern "C" {

int bude_gpu_upload_batch(bude_gpu_ctx *ctx, const bude_atom *protein, int32_t natpro,
                          const bude_ffparams *forcefield, int32_t ntypes, int32_t nligands,
                          const bude_atom *ligand_atoms, const int32_t *ligand_offsets, const float *poses,
                          int64_t pose_stride, const int64_t *pose_offsets) {
  if (!ctx) return set_error(BUDE_ERR_ARG, "ctx is NULL");
  cudaSetDevice(ctx->device);
  return upload_batch(*ctx, protein, natpro, forcefield, ntypes, nligands, ligand_atoms, ligand_offsets, poses,
                      pose_stride, pose_offsets);
}

int bude_gpu_autotune_batch(bude_gpu_ctx *ctx, int32_t max_ms, bude_launch_cfg *best, float *best_ms) {
  if (!ctx || !best) return set_error(BUDE_ERR_ARG, "NULL argument");
  cudaSetDevice(ctx->device);
  return autotune_batch(*ctx, max_ms, *best, best_ms);
}

int bude_gpu_run_batch(bude_gpu_ctx *ctx, const bude_launch_cfg *cfg, int32_t per_ligand, float *ms) {
  if (!ctx || !cfg) return set_error(BUDE_ERR_ARG, "NULL argument");
  cudaSetDevice(ctx->device);
  if (ctx->have_batch && !per_ligand) {
    // Capture (or re-capture) before timing so the first timed launch is the graph itself.
    bude_launch_cfg shape = *cfg;
    shape.cluster = 0;
    int rc = check_cfg(*ctx, shape);
    if (!rc) rc = ensure_graph(*ctx, shape);
    if (rc) return rc;
  }
  cudaEventRecord(ctx->ev0, ctx->stream);
  int rc = enqueue_batch(*ctx, *cfg, per_ligand);
  if (rc) return rc;
  cudaEventRecord(ctx->ev1, ctx->stream);
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cuda_error(e, "batch evaluation");
  if (ms) cudaEventElapsedTime(ms, ctx->ev0, ctx->ev1);
  return BUDE_OK;
}

int bude_gpu_download_batch(bude_gpu_ctx *ctx, float *energies, int64_t total_poses) {
  if (!ctx || (!energies && total_poses > 0)) return set_error(BUDE_ERR_ARG, "NULL argument");
  if (!ctx->have_batch || total_poses != ctx->batch_poses)
    return set_error(BUDE_ERR_ARG, "download of %lld energies but the batch has %lld poses", (long long)total_poses,
                     ctx->have_batch ? ctx->batch_poses : 0LL);
  if (total_poses == 0) return BUDE_OK;
  cudaSetDevice(ctx->device);
  cudaError_t e = cudaMemcpyAsync(energies, ctx->b_energies.ptr, (size_t)total_poses * sizeof(float),
                                  cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? BUDE_OK : cuda_error(e, "batch energy download");
}

} // extern "C"
