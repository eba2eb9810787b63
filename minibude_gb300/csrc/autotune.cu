// autotune.cu -- launch-shape selection for the exact kernel.
//
// Replaces the reference driver's brute-force PPWI x wgsize sweep (src/main.cpp:517-541) with a rule
// on the deck's size (cull_shape) and a short measured search around its pick, timed with CUDA events.
// The pick is cached in the context for the protein, forcefield, ligand and pose count that it was timed
// on: what an evaluation takes goes with the geometry, not with the sizes alone.  A sweep that is asked for runs: default_cfg takes
// the pair that it is given.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "cull.h"
#include "exact_shape.h"

namespace bude {

// The shape asked for, PPWI poses per thread and wgsize threads, each as near as the kernel takes it (a
// power of two up to 16; a multiple of 32 up to 512).  What is left open (ppwi below 1, wgsize below 32)
// follows the rule's chunk; both open is the rule.  A small pair is slow (small chunks, loose groups):
// 938 x 26 x 65,536 86 us an evaluation at 8 x 512, 96 at 8 x 128, 109 at 8 x 64, 235 at 1 x 32.
int default_cfg(const Context &c, int ppwi, int wgsize, bude_launch_cfg &cfg) {
  cfg = c.have_deck ? exact_shape(c, c.nposes, c.natlig, 1) : cull_shape(1LL << 20, 32, 1);
  const int chunk = cfg.ppwi * cfg.wgsize;
  const bool ask_p = ppwi >= 1, ask_w = wgsize >= 32;
  if (!ask_p && !ask_w) return BUDE_OK;
  auto pow2 = [](int most) { return most >= 16 ? 16 : (most >= 8 ? 8 : (most >= 4 ? 4 : (most >= 2 ? 2 : 1))); };
  auto warps = [](int threads) { return (std::max(32, std::min(threads, kMaxThreads)) + 31) / 32 * 32; };
  if (ask_w) cfg.wgsize = warps(wgsize);
  cfg.ppwi = pow2(ask_p ? ppwi : chunk / cfg.wgsize);
  if (!ask_w) cfg.wgsize = warps(chunk / cfg.ppwi);
  if (cfg.ppwi * cfg.wgsize < 32 * cfg.unroll) cfg.unroll = 1;
  return BUDE_OK;
}

// Time one shape: one untimed evaluation, then the mean of `reps` event-timed ones.
static int time_cfg(Context &c, const bude_launch_cfg &cfg, int reps, float *ms) {
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int rc = enqueue_eval(c, cfg);
  if (!rc) {
    cudaEventRecord(e0, c.stream);
    for (int i = 0; i < reps && !rc; ++i) rc = enqueue_eval(c, cfg);
    cudaEventRecord(e1, c.stream);
  }
  cudaError_t e = cudaStreamSynchronize(c.stream);
  if (!rc && e != cudaSuccess) rc = cuda_error(e, "autotune timing");
  if (!rc) {
    cudaEventElapsedTime(ms, e0, e1);
    *ms /= reps;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return rc;
}

int autotune(Context &c, int max_ms, bude_launch_cfg &best, float *best_ms) {
  if (!c.have_deck) return set_error(BUDE_ERR_STATE, "no deck uploaded");
  const long long key[3] = {c.natpro_pad, c.natlig, c.nposes};
  if (key[0] == c.tuned_key[0] && key[1] == c.tuned_key[1] && key[2] == c.tuned_key[2]) {
    best = c.tuned;
    if (best_ms) *best_ms = c.tuned_ms;
    return BUDE_OK;
  }
  // The rule's shape, then its neighbours in chunk size (poses per thread x threads) and group width.
  bude_launch_cfg first{};
  default_cfg(c, 0, 0, first);
  std::vector<bude_launch_cfg> cands{first};
  struct Shape { int p, w, u; };
  for (const Shape &s : {Shape{8, 512, 2}, Shape{4, 512, 2}, Shape{8, 384, 2}, Shape{4, 256, 2}, Shape{2, 256, 2},
                         Shape{2, 512, 2}, Shape{1, 256, 1}, Shape{1, 128, 1}, Shape{2, 128, 2}, Shape{8, 512, 4}})
    if (s.p != first.ppwi || s.w != first.wgsize || s.u != first.unroll)
      cands.push_back(bude_launch_cfg{s.p, s.w, 1, 64, s.u, 0});

  // Time on a ligand prefix of at most 2^27 (pose, atom) points: some ten milliseconds.
  const int natlig_full = c.natlig;
  int lig = natlig_full;
  if ((double)c.nposes * lig > double(1 << 27)) lig = std::max(1, (int)(double(1 << 27) / (double)c.nposes));
  c.natlig = lig;
  int rc = BUDE_OK;
  float best_t = 1e30f, spent = 0.f;
  for (const bude_launch_cfg &cfg : cands) {
    float ms = 0.f;
    rc = time_cfg(c, cfg, 2, &ms);
    if (rc) break;
    if (ms < best_t) {
      best_t = ms;
      best = cfg;
    }
    spent += 3.f * ms;
    if (spent > (float)std::max(max_ms, 1)) break;
  }
  c.natlig = natlig_full;
  if (rc) return rc;
  const float scale = float(natlig_full) / float(lig);
  c.tuned = best;
  c.tuned_ms = best_t * scale;
  for (int i = 0; i < 3; ++i) c.tuned_key[i] = key[i];
  if (best_ms) *best_ms = c.tuned_ms;
  return BUDE_OK;
}

} // namespace bude

extern "C" int bude_gpu_autotune(bude_gpu_ctx *ctx, int32_t max_ms, bude_launch_cfg *best, float *best_ms) {
  if (!ctx || !best) return bude::set_error(BUDE_ERR_ARG, "NULL argument");
  cudaSetDevice(ctx->device);
  return bude::autotune(*ctx, max_ms, *best, best_ms);
}
