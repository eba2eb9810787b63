// noalloc.cu -- bude_gpu_fasten_noalloc: one exact evaluation that allocates no device memory.
//
// Some callers of this library may not allocate GPU memory themselves: code running inside
// another framework whose allocator owns the whole device heap and must see every byte, plugin
// hosts that hand a plugin its buffers and forbid it to allocate, and latency-bound loops where
// cudaMalloc/cudaFree (which can synchronise the device) are not allowed.  They pass device
// buffers for the inputs and the output; the working memory the evaluation needs beyond those --
// the deck's tables, the pose transforms, sums and check words -- comes from one fixed file-scope
// array in device memory, `g_noalloc_scratch`, instead of the cudaMalloc'd buffers of a bude_gpu_ctx.
//
// Rules of the array:
//   * its size is fixed at build time (BUDE_NOALLOC_MAX_POSES transforms and
//     BUDE_NOALLOC_MAX_SLAB_RECORDS slab records, about 12 MiB), and every GPU that loads this
//     module holds it until the process exits;
//   * every call on a device shares it and it keeps the last call's contents: each call rewrites
//     what it reads;
//   * calls whose work overlaps on one GPU (two host threads, or two streams) race on it and
//     must be serialised by the caller;
//   * in host code the array's name is only a stand-in: its device address is looked up once per
//     device with cudaGetSymbolAddress, with that device current, by the first call made on the
//     device, and kept for the life of the process.  A cudaDeviceReset would leave that address
//     stale, so the entry point must not be used on a device after it has been reset.
// Each call reads its check word back and synchronises the stream before it returns; until then the
// kernels themselves leave a deck with a bad type alone.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "chain.h"
#include "cull.h"
#include "cull_kernel.cuh"
#include "deck_tables.cuh"
#include "pose_xform.cuh"
#include "internal.h"
#include "pair_record.h"

namespace bude {
namespace {

constexpr size_t kNaWordBytes = 256; // words [0..2]: the deck's checks (edge_pose.cuh)
// Poses and the bytes of their sort (pose_order_bytes: two words per pose, 128 tiles and the total of 64 cells,
// the boxes).
constexpr size_t kNaOrderBytes = ((size_t)2 * BUDE_NOALLOC_MAX_POSES + 129 * 64 + 1024) * sizeof(int);
constexpr size_t kNaXformBytes = (size_t)BUDE_NOALLOC_MAX_POSES * 3 * sizeof(float4);
constexpr size_t kNaMaskBytes = (size_t)BUDE_NOALLOC_MAX_POSES / 32 * sizeof(unsigned);
// Clusters of the largest protein (one type), and (type, cluster) pairs: a row of 8 records has one.
constexpr size_t kNaBoxBytes = (size_t)BUDE_NOALLOC_MAX_SLAB_RECORDS / kClusterAtoms * 2 * sizeof(float4);
constexpr size_t kNaBoxReachBytes = (size_t)BUDE_NOALLOC_MAX_SLAB_RECORDS / kAtomAlign * sizeof(float);
// Per record its pair constants and its reach; then the protein in cluster order, until the tables are
// built, and the group sums, which also take what the records leave.
constexpr size_t kNaRecordBytes = (kPairF4 + 1) * sizeof(float4);
constexpr size_t kNaTableBytes = (size_t)BUDE_NOALLOC_MAX_SLAB_RECORDS * kNaRecordBytes;
constexpr int kNaSortMax = 16384; // atoms one block sorts; a larger protein keeps its order
constexpr size_t kNaSumsBytes = 512 * 1024;
static_assert(kNaSumsBytes >= kNaSortMax * sizeof(bude_atom), "the protein in cluster order fits the sums");
constexpr size_t kNaScratchBytes =
    kNaWordBytes + kRowOrderMax * sizeof(int) + kNaOrderBytes + kNaXformBytes + kNaMaskBytes + kNaBoxBytes + kNaBoxReachBytes + kNaTableBytes +
    kNaSumsBytes;

// The working memory of bude_gpu_fasten_noalloc: [check words | row order | pose order | pose transforms |
// irregular-pose bits | cluster boxes | cluster reaches | tables | sums].
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaScratchBytes];

constexpr int kNaMaxDevices = 64;
std::mutex g_na_mutex;
unsigned char *g_na_scratch[kNaMaxDevices]; // device address of g_noalloc_scratch, per device

// Device address of the scratch array on `device` (the current device); looked up on first use.
int na_scratch(int device, unsigned char **out) {
  if (device < 0 || device >= kNaMaxDevices)
    return set_error(BUDE_ERR_ARG, "no-alloc entry point supports device ordinals below %d (got %d)", kNaMaxDevices,
                     device);
  std::lock_guard<std::mutex> lock(g_na_mutex);
  if (!g_na_scratch[device]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(no-alloc scratch)");
    g_na_scratch[device] = static_cast<unsigned char *>(p);
  }
  *out = g_na_scratch[device];
  return BUDE_OK;
}

// One block checks the deck (words, edge_pose.cuh) and writes the protein in cluster order: sorted by the
// cell of a 16 x 16 x 16 grid over its box (the 8 x 8 x 8 Hilbert cell, then the octant in it) and by
// index, a bitonic sort of 32-bit keys in shared memory.  Latency-bound, one block: 1,237 atoms take
// 19 us of a call.
__global__ void __launch_bounds__(1024) na_deck_kernel(const bude_atom *__restrict__ protein, int natpro,
                                                       const bude_atom *__restrict__ ligand, int natlig,
                                                       const bude_ffparams *__restrict__ ff, int ntypes, int sort,
                                                       unsigned *words, bude_atom *__restrict__ sorted) {
  extern __shared__ unsigned keys[];
  __shared__ unsigned flags, min_key[2];
  __shared__ float red[6][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) flags = 0, min_key[0] = min_key[1] = 0xffffffffu;
  __syncthreads();
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  unsigned bad = 0, least[2] = {0xffffffffu, 0xffffffffu};
  for (long long i = tid; i < (long long)natpro + natlig; i += blockDim.x) {
    const bool is_lig = i >= natpro;
    const bude_atom a = is_lig ? ligand[i - natpro] : protein[i];
    if (!is_lig) {
      lo[0] = fminf(lo[0], a.x), lo[1] = fminf(lo[1], a.y), lo[2] = fminf(lo[2], a.z);
      hi[0] = fmaxf(hi[0], a.x), hi[1] = fmaxf(hi[1], a.y), hi[2] = fmaxf(hi[2], a.z);
    }
    if (a.type < 0 || a.type >= ntypes) {
      bad |= is_lig ? kDeckBadLigand : kDeckBadProtein;
      continue;
    }
    const bude_ffparams f = ff[a.type];
    if (!param_regular(f) || !(is_lig ? ligand_atom_regular(a.x, a.y, a.z) : protein_atom_regular(a)))
      bad |= kDeckIrregular;
    unsigned &l = least[is_lig];
    l = min(l, order_key(f.radius));
  }
  if (bad) atomicOr(&flags, bad);
  for (int k = 0; k < 2; ++k) {
    const unsigned m = __reduce_min_sync(0xffffffffu, least[k]);
    if (lane == 0) atomicMin(&min_key[k], m);
  }
  for (int d = 0; d < 3; ++d) {
    const float l = warp_min(lo[d]), h = warp_max(hi[d]);
    if (lane == 0) red[d][warp] = l, red[3 + d][warp] = h;
  }
  __syncthreads();
  if (tid == 0) words[0] = flags, words[1] = min_key[0], words[2] = min_key[1];
  if (!sort) return;
  int n2 = 32;
  while (n2 < natpro) n2 <<= 1;
  float inv[3];
  for (int d = 0; d < 3; ++d) {
    lo[d] = warp_min(red[d][lane]);
    const float w = warp_max(red[3 + d][lane]) - lo[d];
    inv[d] = w > 0.f ? 16.f / w : 0.f;
  }
  for (int i = tid; i < n2; i += blockDim.x) {
    unsigned k = 0xffffffffu;
    if (i < natpro) {
      const bude_atom a = protein[i];
      const int x = min(max((int)((a.x - lo[0]) * inv[0]), 0), 15), y = min(max((int)((a.y - lo[1]) * inv[1]), 0), 15),
                z = min(max((int)((a.z - lo[2]) * inv[2]), 0), 15);
      const unsigned cell = (unsigned)kHilbert.at[(z >> 1) * 64 + (y >> 1) * 8 + (x >> 1)] * 8u +
                            (unsigned)((z & 1) * 4 + (y & 1) * 2 + (x & 1));
      k = cell << 14 | (unsigned)i;
    }
    keys[i] = k;
  }
  for (int size = 2; size <= n2; size <<= 1)
    for (int step = size >> 1; step > 0; step >>= 1) {
      __syncthreads();
      for (int t = tid; t < n2 / 2; t += blockDim.x) {
        const int i = 2 * t - (t & (step - 1)), j = i + step;
        const unsigned u = keys[i], v = keys[j];
        if ((u > v) == ((i & size) == 0)) keys[i] = v, keys[j] = u;
      }
    }
  __syncthreads();
  for (int i = tid; i < natpro; i += blockDim.x) sorted[i] = protein[keys[i] & 0x3fffu];
}

// Read n words from the device into a caller-provided host array (no allocation) and wait.
int na_read_words(const unsigned *words, int n, cudaStream_t st, unsigned *out) {
  cudaError_t e = cudaMemcpyAsync(out, words, (size_t)n * sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? BUDE_OK : cuda_error(e, "no-alloc error word");
}

// Device memory of `device` (the current device), or managed memory.  Another GPU's memory is
// refused: the kernels would read it over the interconnect or fault when peer access is off.
bool is_device_memory(const void *p, int device) {
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (at.type == cudaMemoryTypeDevice && at.device == device) || at.type == cudaMemoryTypeManaged;
}

} // namespace
} // namespace bude

extern "C" int bude_gpu_fasten_noalloc(const bude_atom *protein, int32_t natpro, const bude_atom *ligand,
                                       int32_t natlig, const bude_ffparams *forcefield, int32_t ntypes,
                                       const float *poses, int64_t pose_stride, int64_t nposes, float *energies,
                                       void *stream) {
  using namespace bude;
  // Sizes against the fixed scratch.
  if (natpro < 0 || natlig < 0 || ntypes <= 0 || nposes < 0 || pose_stride < nposes)
    return set_error(BUDE_ERR_ARG, "bad sizes (natpro %d, natlig %d, ntypes %d, nposes %lld, pose_stride %lld)",
                     natpro, natlig, ntypes, (long long)nposes, (long long)pose_stride);
  if (nposes > BUDE_NOALLOC_MAX_POSES)
    return set_error(BUDE_ERR_ARG, "no-alloc entry point takes at most %d poses per call (got %lld)",
                     BUDE_NOALLOC_MAX_POSES, (long long)nposes);
  const int natpro_pad = std::max((natpro + kAtomAlign - 1) / kAtomAlign * kAtomAlign, kAtomAlign);
  if ((long long)ntypes * natpro_pad > BUDE_NOALLOC_MAX_SLAB_RECORDS)
    return set_error(BUDE_ERR_ARG,
                     "no-alloc entry point holds at most %d slab records; forcefield types x padded protein atoms = "
                     "%d x %d",
                     BUDE_NOALLOC_MAX_SLAB_RECORDS, ntypes, natpro_pad);
  if (nposes == 0) return BUDE_OK;
  // Inputs and output must be device memory; the ligand is read as 16-byte vectors.
  if (!forcefield || !poses || !energies || (natpro > 0 && !protein) || (natlig > 0 && !ligand))
    return set_error(BUDE_ERR_ARG, "NULL input or output buffer");
  if (reinterpret_cast<uintptr_t>(ligand) % 16 != 0)
    return set_error(BUDE_ERR_ARG, "ligand must be 16-byte aligned");
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
  if (!is_device_memory(forcefield, device) || !is_device_memory(poses, device) ||
      !is_device_memory(energies, device) || (natpro > 0 && !is_device_memory(protein, device)) ||
      (natlig > 0 && !is_device_memory(ligand, device)))
    return set_error(BUDE_ERR_ARG, "no-alloc entry point takes buffers in the current device's memory only "
                                   "(device %d)", device);

  unsigned char *scratch = nullptr;
  int rc = na_scratch(device, &scratch);
  if (rc) return rc;
  unsigned char *at = scratch;
  auto take = [&at](size_t bytes) {
    unsigned char *p = at;
    at += bytes;
    return p;
  };
  unsigned *words = reinterpret_cast<unsigned *>(take(kNaWordBytes));
  int *rows = reinterpret_cast<int *>(take(kRowOrderMax * sizeof(int)));
  void *order = take(kNaOrderBytes);
  float4 *xform = reinterpret_cast<float4 *>(take(kNaXformBytes));
  unsigned *mask = reinterpret_cast<unsigned *>(take(kNaMaskBytes));
  float4 *box = reinterpret_cast<float4 *>(take(kNaBoxBytes));
  float *box_reach = reinterpret_cast<float *>(take(kNaBoxReachBytes));
  const size_t records = (size_t)ntypes * natpro_pad;
  float4 *slab = reinterpret_cast<float4 *>(take(records * kPairF4 * sizeof(float4)));
  float4 *reach = reinterpret_cast<float4 *>(take(records * sizeof(float4)));
  unsigned char *rest = at; // the sums, and before them the protein in cluster order
  const size_t rest_bytes = (size_t)(scratch + kNaScratchBytes - rest);
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  // 1. the deck: checks, cluster order and tables.  Nothing after them runs on a deck with a bad type.
  const int clusters = (natpro_pad + kClusterAtoms - 1) / kClusterAtoms;
  const bool sort = natpro > kClusterAtoms && natpro <= kNaSortMax;
  size_t keys = 0;
  if (sort)
    for (keys = 32 * sizeof(unsigned); keys < natpro * sizeof(unsigned);) keys *= 2;
  e = cudaFuncSetAttribute(na_deck_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(kNaSortMax * sizeof(unsigned)));
  if (e != cudaSuccess) return cuda_error(e, "no-alloc deck kernel");
  auto *sorted = reinterpret_cast<bude_atom *>(rest);
  na_deck_kernel<<<1, 1024, keys, st>>>(protein, natpro, ligand, natlig, forcefield, ntypes, sort, words, sorted);
  e = launch_chained(deck_table_kernel, deck_table_grid(ntypes, clusters), 256u, 0, st,
                     sort ? (const bude_atom *)sorted : protein, natpro, forcefield, ntypes, natpro_pad, clusters, slab,
                     reach, box, box_reach);
  // 2. pose transforms and the exact kernel; irregular poses (or every pose of an irregular deck) by the
  //    reference's arithmetic.
  // The protein's box is not known here: sorted from a number of points on that pays at the density of real
  // proteins (sort_poses; 1,237 x 37 x 12,345 190 us plain, 182 sorted).
  const int *perm = nullptr;
  const RowOrder ro{reinterpret_cast<const float4 *>(ligand), reach, natlig, natpro, natpro_pad,
                    row_order_pays(nposes, natlig) ? rows : nullptr, words};
  const bool order_poses = nposes >= 4096 && (double)nposes * natlig >= 4e5 && pose_order_bytes(nposes) <= kNaOrderBytes;
  if (e == cudaSuccess && order_poses) {
    rc = enqueue_sorted(order, poses, pose_stride, nposes, xform, mask, ro, &perm, st);
    if (rc) return rc;
  } else if (e == cudaSuccess)
    e = launch_chained(pose_xform_kernel, (unsigned)((nposes + 255) / 256 + (ro.rows ? 1 : 0)), 256u, 0, st, poses,
                       (long long)pose_stride, (long long)nposes, xform, mask, ro);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "no-alloc deck launch");
  const bude_launch_cfg cfg = cull_shape(nposes, natlig, 1);
  CullArgs a{};
  a.ligand = reinterpret_cast<const float4 *>(ligand);
  a.slab = slab;
  a.reach = reach;
  a.box = box;
  a.box_reach = box_reach;
  a.xform = reinterpret_cast<const float *>(xform);
  a.sums = reinterpret_cast<float *>(rest);
  a.lo = make_float3(-INFINITY, -INFINITY, -INFINITY); // the poses' own range bins them
  a.hi = make_float3(INFINITY, INFINITY, INFINITY);
  a.words = words;
  a.rows = ro.rows;
  a.natpro_pad = natpro_pad;
  a.clusters = clusters;
  const SumsWindow window = sums_window(natpro, natlig, nposes, cfg, rest_bytes);
  a.supers = cull_supers(natpro_pad, cfg, window.chunk, order_poses);
  FinishArgs f{};
  f.energies = energies;
  f.perm = perm;
  f.words = words;
  f.edges = 1;
  f.e.mask = mask;
  f.e.nlig = 1;
  f.e.ligand = a.ligand;
  f.e.natlig = natlig;
  f.e.protein = protein;
  f.e.natpro = natpro;
  f.e.ff = forcefield;
  f.e.xform = a.xform;
  long long launches = 0;
  rc = cull_range(a, f, cfg, window, natlig, nposes, st, launches);
  if (rc) return rc;
  unsigned h = 0;
  rc = na_read_words(words, 1, st, &h);
  if (rc) return rc;
  if (h & (kDeckBadProtein | kDeckBadLigand))
    return set_error(BUDE_ERR_TYPE, "%s atom type outside the forcefield (%d types)",
                     (h & kDeckBadLigand) ? "a ligand" : "a protein", ntypes);
  return BUDE_OK;
}
