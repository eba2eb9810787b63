// cull.h -- host side of the exact kernel (cull_kernel.cuh): launch shapes, the cut of poses into
// chunks, and the windows that bound the memory of the atom sums.
#pragma once
#include <algorithm>
#include <vector>

#include "internal.h"

namespace bude {

struct CullArgs;
struct FinishArgs;
struct RowOrder;

// A batch evaluation's work, cut for one launch shape: block items and finish items in windows of
// consecutive poses, with a bound on each window's atom sums.
struct CullPlan {
  struct Window {
    int item0, items, fold0, folds;
    long long first, n; // poses
    int atoms;          // the most of a ligand in the window
  };
  std::vector<int4> items, folds; // CullArgs::items, FinishArgs::folds
  std::vector<Window> windows;
  bool direct = false; // every pair, finish items of at most ppwi * wgsize poses alone (direct_kernel.cuh)
  bool points = false; // items of at most one pose per warp (point_kernel)
  bool sorted = false; // the batch's poses are put in order first (sort_batch)
  bool ranked = false; // the items are in the order of their work, which goes with the batch's atoms
  size_t sums_bytes = 0; // the largest window's
};

constexpr size_t kSumsBytes = (size_t)1 << 30, kSumsLeast = (size_t)1 << 20;

// Memory for atom sums: bytes_for(most) cuts the work into windows of at most `most` bytes and returns what
// the largest takes.  Where the device has no room for it, the windows get smaller; no energy changes.
template <class F> int reserve_sums(DevBuf &sums, F &&bytes_for) {
  for (size_t most = kSumsBytes;; most /= 4) {
    const int rc = sums.reserve(std::max<size_t>(bytes_for(most), 16), "atom sums");
    if (!rc || most <= kSumsLeast) return rc;
  }
}

// Poses of a finish block: with a chunk of 4,096 per block 64 ligands gave 108 blocks (89 us, so 17.5).
constexpr int kFoldPoses = 256;

// Poses of a chunk for n poses at `most` per block: as many chunks as that takes, evenly filled (a
// short last chunk would sort few poses into loose groups).
inline int even_chunk(long long n, int most) {
  const long long chunks = (n + most - 1) / most;
  const long long per = chunks > 0 ? (n + chunks - 1) / chunks : 1;
  return (int)((per + 31) / 32 * 32 < most ? (per + 31) / 32 * 32 : most);
}

// One ligand's poses, evaluated in windows whose atom sums, [atoms][poses], take at most `most` bytes (and
// room for one atom of a chunk).
struct SumsWindow {
  int chunk, atoms;
  long long poses;
  bool points; // of point_kernel
};
SumsWindow sums_window(int natpro, int natlig, long long nposes, const bude_launch_cfg &cfg, size_t most);
int cull_range(CullArgs a, FinishArgs f, const bude_launch_cfg &cfg, const SumsWindow &w, int natlig, long long nposes,
               cudaStream_t st, long long &launches);
// The transforms of n poses in the order of their translations, and that order, with pose_order_bytes(n) of
// scratch (internal.h; pose_order.cuh).
int enqueue_sorted(void *scratch, const float *poses, long long stride, long long n, float4 *xform, unsigned *mask,
                   const RowOrder &ro, const int **perm, cudaStream_t st);
// Whether the blocks of an evaluation take the ligand's atoms longest first (RowOrder).
bool row_order_pays(long long n, int natlig);
// Which groups of a launch in chunks of `chunk` poses share candidate lists (CullArgs::supers).
int cull_supers(int natpro_pad, const bude_launch_cfg &shape, int chunk, bool sorted);

// Plan of the poses [first[i], first[i] + count[i]) of ligand lig[i]; first ascending.  A window's sums take
// at most `most` bytes (and room for one chunk of a ligand).
CullPlan plan_cull(const Context &c, const std::vector<int> &lig, const std::vector<long long> &first,
                   const std::vector<long long> &count, const bude_launch_cfg &shape, size_t most);
// Whether evaluating the uploaded batch in chunks of `chunk` poses puts each ligand's poses in order first.
bool sort_batch(const Context &c, int chunk);
// Memory of that order for a batch of `poses` poses, and its kernels: the transforms at `xform` and their
// order in `scratch`.
size_t batch_order_bytes(const Context &c, size_t tiles);
int enqueue_batch_order(Context &c, const CullPlan &plan, const int4 *tiles, const float *xform, void *scratch,
                        const float **sorted, const int **perm);
// Enqueue the windows of a plan whose items and folds are on the device: energies of its poses from the
// transforms at `xform`; `sums` holds plan.sums_bytes.  edges: irregular poses of the uploaded batch
// get the reference's arithmetic.
int enqueue_plan(Context &c, const bude_launch_cfg &shape, const CullPlan &plan, const int4 *items, const int4 *folds,
                 const float *xform, float *energies, float *sums, bool edges, cudaStream_t st,
                 const int *perm = nullptr);
// Shared-memory limit of the shape's kernel (before a stream capture).
int prepare_shape(const bude_launch_cfg &shape);
// Whether an evaluation of `poses` poses of a ligand of natlig atoms evaluates every pair (direct_kernel.cuh).
bool direct_pays(const Context &c, long long natlig, long long poses);
// The launch shape for n poses of a ligand of natlig atoms, `ligands` such ligands at once; and that for the
// uploaded protein.
bude_launch_cfg cull_shape(long long n, int natlig, int ligands);
bude_launch_cfg exact_shape(const Context &c, long long n, int natlig, int ligands);
// The same for the uploaded batch (its mean ligand).
bude_launch_cfg batch_shape(const Context &c);

} // namespace bude
