// Host interface of the traversal kernels (trace.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "layout.h"

namespace bzr {

constexpr int kTraceThreads = 128;     // default threads per block of the trace kernels
constexpr int kMaxTraceThreads = 256;  // largest block the trace kernels are compiled for
constexpr uint32_t kRayChunk = 32;     // default rays a warp takes from the global counter
constexpr int kModeFp64 = 0;   // BZR_MODE_FP64
constexpr int kModeMixed = 1;  // BZR_MODE_MIXED
// Device words launch_trace takes per call.  First kTraceCounterWords zeroed words: the work
// counter of each kind's pass, then for each kind the work counter of the binary pass over the
// rays its wide walk handed on, the count of those it did not cover and the count of those whose
// walk ended without a result.  From kTraceListWord on, the first kUncoveredList and kRedoList
// of these rays' indices (the kinds' passes use them one after the other).  Words in between
// belong to the caller.
constexpr int kTraceCounterWords = 4 * kNumKinds;
constexpr int kTraceListWord = kTraceCounterWords + 4;
constexpr uint32_t kUncoveredList = 96, kRedoList = 32;
constexpr int kTraceWords = kTraceListWord + int(kUncoveredList + kRedoList);

// Device pointers of one batch.  tmin / tmax may be null (0 and DBL_MAX); each output except t
// may be null.  error_word collects kErr* bits.
struct RayIO {
  const double *org = nullptr;
  const double *dir = nullptr;
  const double *tmin = nullptr;
  const double *tmax = nullptr;
  double *t = nullptr;
  double *uv = nullptr;
  double *normal = nullptr;
  uint32_t *prim = nullptr;
  uint32_t *geom = nullptr;
  uint8_t *hit = nullptr;
  uint32_t n = 0;
  uint32_t *error_word = nullptr;
  const uint32_t *perm = nullptr;  // optional processing order (ray indices), see RaySort
  int any_hit = 0;                 // every ray is Ray::AnyHit::yes (blazert/ray.h:24-34)
  uint32_t chunk = kRayChunk;      // rays a warp takes per fetch: 32, 64, 128, or 0 for
                                   // exactly the lanes that are idle
  uint32_t top_nodes = 0;          // top-level nodes each block stages in shared memory
  // Wide passes: the rays that the first blocks leave to the walk but that the walk does not
  // cover (origins beyond its range), or whose walk ends without a result, are counted here
  // and the first of each noted in the lists, for the binary pass right after.  A batch has
  // hardly any: a short list needs no allocation, and past it the binary pass looks at every ray
  // again.  Set by launch_trace.
  uint32_t *uncovered_count = nullptr, *redo_count = nullptr;
  uint32_t *uncovered = nullptr, *redo = nullptr;
  int out_blocks = 0;  // a wide kernel's first blocks, which trace the rays its walk leaves out
  int wide_mode = 0;  // the mode whose wide pass handed the rays on (its cover test)
};

// Coherence sort of a batch: rays are processed in the order of a 32-bit key -- the direction
// octant (3 bits) over a Morton code of the origin quantised inside the scene bounds (9 bits
// per axis) -- bucketed on the key's top kSortBits bits by a device counting sort.  The order
// affects only speed: every ray's result is written to its own index.
struct RaySort {
  bool enabled = false;
  float lo[3] = {0, 0, 0};     // origin quantisation box
  float scale[3] = {0, 0, 0};  // 512 / extent per axis
};

// Grid of each per-kind persistent kernel: SMs x resident blocks per SM, and the launch
// shape the tuning knobs select (none of them changes results).
struct LaunchPlan {
  int sms = 0;
  int threads = kTraceThreads;     // threads per block: 64, 128 or 256
  bool shared_stack = false;       // traversal stack in shared memory even when it fits locally
  uint32_t chunk = kRayChunk;      // rays per warp fetch: 32, 64, 128 or 0 (exactly the idle lanes)
  uint32_t top_nodes = 0;          // top-level nodes each block stages in shared memory (0..256)
  // the trace kernels after a call's first one are launched with programmatic stream
  // serialisation: each is resident when its predecessor ends (it waits for it on the device)
  bool early_launch = true;
  int blocks[kNumKinds] = {0, 0, 0, 0};    // FP64 kernels
  int blocks32[kNumKinds] = {0, 0, 0, 0};  // mixed-precision kernels
  int blocks64w[kNumKinds] = {0, 0, 0, 0};  // the FP64 mode's wide kernels
  int blocks_rest[kNumKinds] = {0, 0, 0, 0};  // the binary passes after wide ones
  int small_blocks[kNumKinds] = {0, 0, 0, 0};  // resident blocks of the small kernel, by kinds
  RaySort sort;
  uint32_t sort_min_rays = 1u << 16;  // smaller batches are traced in their own order
  cudaMemPool_t pool = nullptr;       // stream-ordered scratch (keeps its memory mapped)
};

// Small batches (trace_small.cu): one launch for every kind.  done: for results in host memory,
// how the kernel tells the host that all of them are there: once every block has counted itself
// in *blocks (device, zero before and again after), the last one writes value, with the call's
// error word (zero again after) in the upper half, to *flag (host memory).
struct SmallDone {
  uint32_t *blocks = nullptr;
  unsigned long long *flag = nullptr;
  uint32_t value = 0;
};
cudaError_t small_prepare(LaunchPlan *plan);
// Whether a batch of n rays takes the small kernel.
bool small_batch(const SceneView &S, const LaunchPlan &plan, uint32_t n);
cudaError_t launch_small(const SceneView &S, const RayIO &io, const LaunchPlan &plan,
                         cudaStream_t stream, const SmallDone &done = SmallDone());

// Many scenes in one launch per kind (the batching form).  Rays of scene s occupy
// [ray_offset[s], ray_offset[s+1]) of the concatenated arrays in io.  Chunks of at most
// kBatchChunk rays never cross scenes.
constexpr uint32_t kBatchChunk = 64;
struct BatchChunk {
  uint32_t scene;
  uint32_t begin, end;  // ray range in the concatenated batch
};
struct BatchView {
  const SceneView *views = nullptr;    // n_scenes device copies of the scenes' views
  const BatchChunk *chunks = nullptr;  // n_chunks
  uint32_t n_chunks = 0;
  uint32_t n_scenes = 0;
  const int8_t *first_kind = nullptr;  // per scene: kind whose pass writes the whole record
  const int8_t *last_kind = nullptr;   // per scene: kind whose pass completes the scene
  const uint32_t *scene_rays = nullptr;  // per scene: ray count
  uint32_t *scene_left = nullptr;      // per scene: rays not yet completed (set to scene_rays)
  unsigned long long *scene_done_ns = nullptr;  // per scene completion time (%globaltimer), or null
  unsigned long long *start_ns = nullptr;       // batch start time, or null
  // coherence sort of each scene's rays (BatchPlan::sort): per scene the origin quantisation
  // box, and the bits of the sort key that hold the scene index
  const RaySort *scene_sort = nullptr;
  uint32_t scene_bits = 0;
};
// Scratch of the batch coherence sort: keys and permutation (one word per ray each) and the
// 2^kSortBits bucket counts.
struct BatchSortScratch {
  uint32_t *keys = nullptr, *perm = nullptr, *counts = nullptr;
};
constexpr uint32_t kBatchSortMaxScenes = 1u << 12;  // the key keeps at least 4 bits per scene
constexpr size_t kSortBuckets = size_t(1) << 16;     // buckets of the counting sort (kSortBits)
struct BatchPlan {
  int sms = 0;
  int threads = kTraceThreads;  // threads per block: 64, 128 or 256
  bool shared_stack = false;    // traversal stack in shared memory even when it fits locally
  uint32_t local_stack = 64;    // entries of the thread-local stack: 32 or 64 (kLocalStack)
  bool sort = false;            // coherence sort of each scene's rays before tracing
  uint32_t node_width = 8;      // mixed mode: 8 walks the wide nodes, 2 the binary FP64 nodes
  int blocks[kNumKinds] = {0, 0, 0, 0};
  int blocks32[kNumKinds] = {0, 0, 0, 0};
  uint32_t stack_cap = 32;
  int kinds_present = 0;  // bit k: some scene has kind k
};
// Fills plan's grids for stack_cap, plan->threads and plan->shared_stack.
cudaError_t batch_prepare(uint32_t stack_cap, BatchPlan *plan);
// counters: kNumKinds device words (chunk counters), zeroed here.
cudaError_t launch_batch(const BatchView &B, const RayIO &io, int mode, const BatchPlan &plan,
                         cudaStream_t stream, uint32_t *counters,
                         const BatchSortScratch &sort_scratch = BatchSortScratch());

// RayHit defaults for every ray of io (a scene without primitives).
cudaError_t launch_defaults(const RayIO &io, int sms, cudaStream_t stream);

// Fills K's leaf_box (device, 6 doubles per primitive position) from its nodes and root box.
cudaError_t fill_leaf_boxes(const KindView &K, double *leaf_box);

size_t trace_smem_bytes(uint32_t stack_cap, int threads);
// Dynamic shared memory of a trace_kind_kernel launch: the stack unless thread-local, then
// top_nodes staged 128-byte nodes.
size_t trace_kind_smem(uint32_t stack_cap, int threads, bool local, uint32_t top_nodes);
// Fills plan->sms and the per-kind grids for plan->threads and plan->shared_stack.
cudaError_t trace_prepare(const SceneView &S, LaunchPlan *plan);
// Number of per-kind passes a batch runs (kinds present with at least one primitive).
int trace_passes(const SceneView &S);
// Queues a batch on `stream`: one kernel per kind present, merged into io's outputs.  io.t must
// be non-null when trace_passes(S) > 1 (it carries the closest distance between passes).
// When plan.sort.enabled and the batch has at least plan.sort_min_rays rays, a coherence sort
// runs first (scratch from plan.pool, stream-ordered).
// counters: kTraceWords device words, zeroed here as far as needed.  totals (device, 8 x uint64,
// or null): when given, the counting kernels add per kind the box tests (totals[0..3]) and
// primitive tests (totals[4..7]) of every ray.
// A pass of a kind whose wide image exists is two kernels: one whose first blocks run the binary
// walk of the rays that the wide walk leaves out (FP32: a direction component of 0, below 2^-40 or
// above 2^100 in magnitude, a tmin beyond 1e18, NaN; FP64: RayD) and whose others run the wide walk
// of the rest, then the binary walk of those that the wide walk hands on.
cudaError_t launch_trace(const SceneView &S, const RayIO &io, int mode, const LaunchPlan &plan,
                         cudaStream_t stream, uint32_t *counters,
                         unsigned long long *totals = nullptr);

}  // namespace bzr
