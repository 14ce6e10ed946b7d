// Closest-hit traversal kernels for sm_100a.
//
// A batch runs as one persistent kernel per primitive kind present, in the reference's fixed
// order (triangles, spheres, planes, cylinders; blazert/scene.h:161-210).  Each pass merges its
// hits into the output record with the reference's rule (finalize_kind), so the result equals
// intersect1's.  Splitting by kind keeps each kernel small (registers, instruction cache) and
// keeps one kind's nodes and primitives hot in L1/L2 at a time.  (Batches that fit the GPU in one
// wave take the one launch of trace_small.cu instead.)
//
// Work distribution: each warp owns a pool of ray indices taken from a global counter in
// chunks of kChunk (one atomic per chunk).  A lane whose ray finishes takes the next index of
// its warp's pool at once, so lanes do not idle until the slowest ray of a fixed group of 32
// is done.  Within a ray the traversal alternates "walk internal nodes to the next leaf" and
// "test the leaf's primitives", so the lanes of a warp run their leaf tests together.
//
// Exactness.  The kernels reproduce the reference's visit order and arithmetic bit for bit:
//  * compiled with --fmad=false; every expression keeps the reference's evaluation order;
//  * the reference pushes both children of a node and tests a node's box when it is POPPED,
//    against the hit distance current at that moment (blazert/bvh/accel.h:89-113).  Here the
//    parent tests both children at once.  For each child the slab test splits into a part that
//    does not depend on the hit distance h (entry mn <= exit E, with E evaluated as if
//    h = +inf) and the comparison mn <= h, which is deferred to pop time (the stack stores mn
//    as the key).  When an exit distance is NaN (0 * inf on a slab plane) the reference's
//    std::min chain drops h entirely; the key is then -inf so that the pop test always passes.
//    The result is the reference's sequence of accepted nodes, including nodes re-accepted
//    after a cylinder hit moved h outward (cylinders do not test against h,
//    blazert/primitives/cylinder.h:181-495).
//  * the slab test keeps the reference's far-plane factor l1 = 1 + 4 eps and its std::max /
//    std::min argument order (blazert/bvh/intersect.h:33-51).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "alloc.h"
#include "layout.h"
#include "bucket_sort.cuh"
#include "trace.h"
#include "trace_core.cuh"

namespace bzr {
static_assert(kSortBuckets == (size_t(1) << kSortBits), "batch sort scratch size");
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

// Shared memory of the stack: none for a thread-local stack, else stack_cap entries of 12 bytes
// per thread, rounded up to 16 bytes (the staged top-level nodes follow).
template <bool LOCAL>
__device__ __forceinline__ size_t stack_smem_bytes(uint32_t stack_cap) {
  return LOCAL ? 0 : (size_t(stack_cap) * blockDim.x * 12 + 15) / 16 * 16;
}

// Traversal stack storage.  LOCAL: a thread-local array of kLocalStack entries (local memory,
// cached in L1; the host picks it when the tree's stack fits, and it leaves the SM's shared
// memory to L1 and the occupancy to the register count).  Otherwise shared memory sized from
// the tree, entry j of thread t at [j * blockDim.x + t].  The capacity is clamped to the
// storage, so a mismatch is reported as kErrStack, never written past.
template <bool LOCAL, uint32_t LCAP = kLocalStack>
__device__ __forceinline__ void init_stack(Stack &sk, uint32_t &tid, uint32_t cap,
                                           unsigned char *smem, double *lkey, uint32_t *lref) {
  if (LOCAL) {
    sk.stride = 1;
    sk.cap = cap < LCAP ? cap : LCAP;
    sk.key = lkey;
    sk.ref = lref;
    tid = 0;
  } else {
    sk.stride = blockDim.x;
    sk.cap = cap;
    sk.key = reinterpret_cast<double *>(smem);
    sk.ref = reinterpret_cast<uint32_t *>(sk.key + size_t(sk.cap) * sk.stride);
    tid = threadIdx.x;
  }
}

// Cold start: between batches the scene may have left L2 (other work, or the benchmark's L2
// flush), and then every dependent node fetch of the first rays waits for DRAM.  The grid
// first asks L2 for the breadth-first prefix of the node array (the top levels every ray
// visits) and for the leaf-ordered primitive data, at most kPrefetchBytes of each, one
// 128-byte line per thread per round.  A hint only: nothing waits for it.  A small batch's grid
// does not go round for more than kPrefetchRounds: its few rays need less than the loop costs
// (one block over 4 MB is 256 rounds before its first ray).
constexpr size_t kPrefetchBytes = size_t(4) << 20;
constexpr size_t kPrefetchRounds = 2;

__device__ __forceinline__ void prefetch_l2(const void *base, size_t bytes) {
  if (!base) return;
  bytes = bytes < kPrefetchBytes ? bytes : kPrefetchBytes;
  const size_t step = size_t(gridDim.x) * blockDim.x * 128;
  bytes = bytes < kPrefetchRounds * step ? bytes : kPrefetchRounds * step;
  for (size_t off = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) * 128; off < bytes;
       off += step)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char *>(base) + off));
}

template <int KIND, bool WIDE>
__device__ __forceinline__ void prefetch_kind(const KindView &K) {
  if (WIDE && K.mixed_ok)
    prefetch_l2(K.wide, size_t(K.n_wide) * kWideBytes);
  else
    prefetch_l2(K.nodes64, size_t(K.n_internal) * kNode64Doubles * sizeof(double));
  if (KIND == kMesh) {
    prefetch_l2(K.tri, size_t(K.n_prims) * 4 * sizeof(uint32_t));
    prefetch_l2(K.verts, size_t(K.n_verts) * kVertexDoubles * sizeof(double));
  } else {
    constexpr int kDoubles = KIND == kSpheres ? 4 : KIND == kPlanes ? 14 : 16;
    prefetch_l2(K.payload, size_t(K.n_prims) * kDoubles * sizeof(double));
    prefetch_l2(K.prim_ids, size_t(K.n_prims) * sizeof(uint32_t));
  }
}

// Programmatic dependent launch (sm_90 and later): a kernel launched with programmatic stream
// serialisation may start while the kernel before it on the stream still runs, once every
// block of that kernel has called griddep_launch_dependents (or exited); griddep_wait blocks
// until that kernel has completed and its writes are visible.  Both are no-ops for a kernel
// launched without the attribute.
__device__ __forceinline__ void griddep_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void griddep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One kind over the whole batch.  first: this pass writes the whole output record.
// COUNT: also sums the work counters into totals[16] (per kind: box tests, primitive tests,
// node fetches, leaf fetches; see Counts).  F: NoWalk, the binary FP64 traversal; RayW or RayD,
// the wide walk in FP32 or FP64, which hands on the rays that it does not cover (f.ok) or that
// end it without a result (kRedoLeaf); Rest, the binary traversal of those (cylinders always
// take the binary traversal).  Keeping the binary walk out of the wide walk's loop keeps its
// registers for the wide walk.
struct NoWalk {
  using Bound = float;
};
struct Rest {
  using Bound = float;
};

// The first io.out_blocks blocks of a wide kernel: each warp looks through its share of the batch
// for rays that the wide walk leaves out and traces them through the binary nodes, lanes refilled
// as they finish; the other blocks walk the wide nodes.  These rays start first because they can be
// the slowest: the middle row of an image of odd height has a zero direction component, and along a
// plane of box bounds the reference's 0 * inf accepts thousands of boxes.  Traced after the wide
// walk instead, they added their whole time to it: 541,501 pixels of a 20,480-triangle sphere
// 637 us, now 361; without that row 166.  (As a first phase, or a last one, of every block they
// cost the walk its registers: 8.4M bounce rays on a terrain 4,420 -> 4,560 to 4,850 us; a look
// through those takes about 10.  As a kernel of its own, which the wide one must run beside to gain
// anything, they have more registers, 420 us for that image where these then took 441, but the wide
// kernel then reads what earlier kernels wrote without a wait of its own; an acquire in its place
// empties the SM's L1 under the walks, 3 to 13 us a pass at 131,072 rays.)
constexpr uint32_t kScan = 8;  // runs of 32 rays a warp looks at together: independent loads

// Whether the wide walk covers hardly any ray of a large batch (an orthographic camera along an
// axis, a negative tmin in FP64 mode, far origins): at most 4 of 32 rays spread over it, twice.
// Such a batch is left to the binary pass as a whole, whose persistent kernel holds more warps than
// the blocks below and takes its rays in order; every block comes to the same answer.  1M / 4M
// rays, by the blocks below and so: raster rays straight down on a terrain 259 / 955 and 224 / 720
// us (the binary kernel alone 215 / 702), rays with tmin -1 in it 920 / 2,943 and 836 / 2,620.
// 524,288 of those 629 and 608, 400,000 476 and 484; with 10,000 spheres 1M 1,015 and 1,037, 4M
// 3,490 and 3,348.
constexpr uint32_t kWholeMinMesh = 1u << 19, kWholeMin = 1u << 21;
template <int KIND>
__host__ __device__ constexpr uint32_t whole_min() {
  return KIND == kMesh ? kWholeMinMesh : kWholeMin;
}
template <int KIND, class F>
__device__ __forceinline__ bool covers_hardly_any(const RayIO &io) {
  if (io.n < whole_min<KIND>()) return false;
  bool hardly = false;
  if (threadIdx.x < 32) {  // scattered loads: one warp of a block makes them
    auto covered = [&](uint32_t j) {
      const size_t i = (size_t(threadIdx.x) * 2 + j) * io.n / 64;
      const F *f = nullptr;
      const bool out = left_out(io.dir + 3 * i, io.tmin ? io.tmin[i] : 0.0,
                                io.tmax ? io.tmax[i] : kDblMax, f) ||
                       far_origin(io.org + 3 * i, f);
      return __popc(__ballot_sync(kFull, !out));
    };
    hardly = covered(0) <= 4 && covered(1) <= 4;
  }
  return __syncthreads_or(hardly);
}

template <int KIND, bool COUNT, class F, bool LOCAL>
__device__ __forceinline__ void trace_left_out_body(const SceneView &S, const RayIO &io, int first,
                                                    unsigned long long *totals) {
  griddep_launch_dependents();
  extern __shared__ __align__(16) unsigned char smem[];
  const KindView &K = S.k[KIND];
  double lkey[LOCAL ? kLocalStack : 1];
  uint32_t lref[LOCAL ? kLocalStack : 1];
  Stack sk;
  uint32_t tid;
  init_stack<LOCAL>(sk, tid, S.stack_cap, smem, lkey, lref);
  if (!COUNT) prefetch_kind<KIND, true>(K);
  Counts cnt = {};
  griddep_wait();
  const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  if (covers_hardly_any<KIND, F>(io)) return;
  const uint32_t warps = uint32_t(io.out_blocks) * (blockDim.x >> 5);
  const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  // Runs of 32 rays, dealt to the warps in turn (left-out rays tend to lie together), kScan runs
  // looked at together.  On a mesh a run is four pieces of 8 rays from the batch's four quarters, as
  // the slow rays of an image's middle row take the longer the more of them a warp has: 541,501
  // pixels of a 20,480-triangle sphere 445 us in whole runs, 361 so (mixed 480 and 387).  Elsewhere
  // rays rarely run along boxes, and whole runs are the better by 3 to 6 % where all are left out.
  constexpr uint32_t kPiece = KIND == kMesh ? 8 : 32;
  uint64_t run = warp;
  const uint64_t runs = (uint64_t(io.n) + 31) / 32;
  unsigned found[kScan] = {};  // warp-uniform: the left-out rays of the runs, not yet taken
  uint64_t at = 0;             // the first of these runs
  uint32_t i = 0;
  bool active = false;
  Ray r;
  KState st;
  Trav tv;
  auto ray_of = [&](uint64_t k, uint32_t b) {
    return (k + uint64_t(b / kPiece) * runs) * kPiece + b % kPiece;
  };
  auto any_found = [&] {
    unsigned m = 0;
#pragma unroll
    for (uint32_t j = 0; j < kScan; ++j) m |= found[j];
    return m != 0;
  };
  for (;;) {
    const unsigned idle = __ballot_sync(kFull, !active);
    while (idle && run < runs && !any_found()) {
#pragma unroll
      for (uint32_t j = 0; j < kScan; ++j) {
        const uint64_t idx = ray_of(run + uint64_t(j) * warps, lane);
        bool out = false;
        if (run + uint64_t(j) * warps < runs && idx < io.n) {
          const double w[3] = {io.dir[3 * idx], io.dir[3 * idx + 1], io.dir[3 * idx + 2]};
          out = left_out(w, io.tmin ? io.tmin[idx] : 0.0, io.tmax ? io.tmax[idx] : kDblMax,
                         static_cast<const F *>(nullptr));
        }
        found[j] = __ballot_sync(kFull, out);
      }
      at = run;
      run += uint64_t(kScan) * warps;
    }
    if (idle && any_found()) {  // the idle lanes take found rays in their order
      uint32_t rank = __popc(idle & below), left = __popc(idle);
      bool got = false;
#pragma unroll
      for (uint32_t j = 0; j < kScan; ++j) {
        const uint32_t have = __popc(found[j]);
        if (!active && !got && rank < have) {
          unsigned m = found[j];
          for (uint32_t k = 0; k < rank; ++k) m &= m - 1;
          i = uint32_t(ray_of(at + uint64_t(j) * warps, unsigned(__ffs(m)) - 1u));
          got = true;
        }
        if (!got) rank -= have < rank ? have : rank;
        const uint32_t taken = left < have ? left : have;
        for (uint32_t k = 0; k < taken; ++k) found[j] &= found[j] - 1;
        left -= taken;
      }
      if (got) {
        active = true;
        r = make_ray(io.org + 3 * size_t(i), io.dir + 3 * size_t(i), io.tmin ? io.tmin[i] : 0.0,
                     io.tmax ? io.tmax[i] : kDblMax);
        r.any_hit = io.any_hit != 0;
        trav_begin<KIND, COUNT>(K, r, st, tv, &cnt);
      }
    }
    if (!__any_sync(kFull, active)) {
      if (run >= runs && !any_found()) break;
      continue;
    }
    if (active) {
      if (tv.live) trav_to_leaf<KIND, COUNT>(K, r, st, tv, sk, tid, io.error_word, &cnt);
      if (tv.live) trav_leaf<KIND, COUNT>(K, r, st, tv, sk, tid, io.error_word, &cnt);
      if (!tv.live) {
        finalize_kind<KIND>(S, r, st, i, first != 0, io.t, io.uv, io.normal, io.prim, io.geom,
                            io.hit);
        active = false;
      }
    }
  }
  if (COUNT) {
    unsigned long long v[4] = {cnt.box[KIND], cnt.prim[KIND], cnt.node[KIND], cnt.leaf[KIND]};
    for (int j = 0; j < 4; ++j)
      if (v[j]) atomicAdd(totals + j * kNumKinds + KIND, v[j]);
  }
}

template <int KIND, bool COUNT, class F, bool LOCAL>
__device__ __forceinline__ void trace_kind_body(const SceneView &S, const RayIO &io, int first,
                                                uint32_t *work_counter,
                                                unsigned long long *totals) {
  constexpr bool kRest = std::is_same<F, Rest>::value;
  constexpr bool kWide = !std::is_same<F, NoWalk>::value && !kRest && KIND != kCylinders;
  // The next kernel on the stream may be scheduled now: it waits (griddep_wait) for this grid
  // to complete before it reads anything this grid writes.
  griddep_launch_dependents();
  extern __shared__ __align__(16) unsigned char smem[];
  double lkey[LOCAL ? kLocalStack : 1];
  uint32_t lref[LOCAL ? kLocalStack : 1];
  Stack sk;
  uint32_t tid;
  init_stack<LOCAL>(sk, tid, S.stack_cap, smem, lkey, lref);
  const KindView &K = S.k[KIND];
  // (the rays handed on are few as a rule: their pass leaves L2 to the rays)
  if (!COUNT && !kRest) prefetch_kind<KIND, kWide>(K);
  // The first io.top_nodes nodes of the array this kernel walks (the top levels every ray
  // visits) are staged in shared memory after the stack.
  {
    const uint32_t avail = kWide ? K.n_wide : K.n_internal;
    const uint32_t n_top = io.top_nodes < avail ? io.top_nodes : avail;
    uint4 *top = reinterpret_cast<uint4 *>(smem + stack_smem_bytes<LOCAL>(S.stack_cap));
    const uint4 *src = kWide ? reinterpret_cast<const uint4 *>(K.wide)
                             : reinterpret_cast<const uint4 *>(K.nodes64);
    for (uint32_t j = threadIdx.x; j < n_top * 8; j += blockDim.x) top[j] = ldg(src + j);
    if (n_top) __syncthreads();
    sk.top = top;
    sk.n_top = n_top;
  }
  // Up to here only the scene was read; the counters, the rays' closest distances and the
  // lists come from earlier kernels of the stream.
  griddep_wait();
  if constexpr (kWide)
    if (covers_hardly_any<KIND, F>(io)) return;
  // The rays of a Rest pass: the listed ones, or every ray that the wide walk does not cover
  // when they outgrew their list, or every ray when the wide kernel left it the whole batch or
  // those to redo outgrew theirs (a ray the wide walk has finished gives the same result again).
  uint32_t n = io.n, n_uncovered = 0;
  bool scan = false, all = false;
  if constexpr (kRest) {
    n_uncovered = __shfl_sync(kFull, *io.uncovered_count, 0);  // the same for every lane
    const uint32_t n_redo = __shfl_sync(kFull, *io.redo_count, 0);
    const bool whole = io.wide_mode == kModeMixed ? covers_hardly_any<KIND, RayW>(io)
                                                  : covers_hardly_any<KIND, RayD>(io);
    all = whole || n_redo > kRedoList;
    scan = all || n_uncovered > kUncoveredList;
    n = all ? io.n : scan ? io.n + n_redo : n_uncovered + n_redo;
    if (n == 0) return;
  }
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  uint32_t pool_next = 0, pool_end = 0;  // warp-uniform
  bool exhausted = false;                // warp-uniform
  bool list_full = false;                // warp-uniform: the list of uncovered rays is full
  bool active = false;
  uint32_t i = 0;
  Ray r;
  F f;
  typename F::Bound hl = 0;
  KState st;
  Trav tv;
  Counts cnt = {};
  for (;;) {
    for (;;) {  // refill the idle lanes; repeats only after a lane handed its ray on
      const unsigned idle = __ballot_sync(kFull, !active);
      bool deferred = false;
      bool skipped = false;
      if (idle && !exhausted) {
        const uint32_t want = __popc(idle), avail = pool_end - pool_next;
        // rays taken per fetch: io.chunk (>= 32, so one fetch serves every idle lane), or
        // with io.chunk == 0 exactly the number of idle lanes the pool cannot serve
        const uint32_t take = io.chunk ? io.chunk : want - avail;
        uint32_t base = 0;
        if (want > avail) {
          if (lane == 0) base = atomicAdd(work_counter, take);
          base = __shfl_sync(kFull, base, 0);
        }
        if (!active) {
          const uint32_t rank = __popc(idle & below);
          const uint32_t idx = rank < avail ? pool_next + rank : base + (rank - avail);
          if (idx < n) {
            active = true;
            if constexpr (kRest) {
              i = handed_on_ray(idx, scan ? io.n : n_uncovered, scan, io.uncovered, io.redo,
                                io.perm, io.n, io.error_word);
              if (i == kNoRay) active = false, skipped = true;
            } else {
              i = io.perm ? io.perm[idx] : idx;
            }
            if (!kRest || active) {
              r = make_ray(io.org + 3 * size_t(i), io.dir + 3 * size_t(i),
                           io.tmin ? io.tmin[i] : 0.0, io.tmax ? io.tmax[i] : kDblMax);
              r.any_hit = io.any_hit != 0;
            }
            if constexpr (kWide) {
              f = make_ray_f(r, static_cast<const F *>(nullptr));
              if (f.ok) {
                wtrav_begin<KIND, COUNT>(K, r, f, st, hl, tv, &cnt);
              } else {  // the pass's first blocks have it, or it is handed on
                active = false;
                skipped = true;
                deferred = !left_out(io.dir + 3 * size_t(i), r.tmin, r.tmax,
                                     static_cast<const F *>(nullptr));
              }
            } else {
              if constexpr (kRest) {  // the wide pass has traced the others
                const double *w = io.dir + 3 * size_t(i);
                if (active && scan && !all && idx < io.n &&
                    (io.wide_mode == kModeMixed
                         ? left_out(w, r.tmin, r.tmax, static_cast<const RayW *>(nullptr)) ||
                               make_ray_f(r, static_cast<const RayW *>(nullptr)).ok
                         : left_out(w, r.tmin, r.tmax, static_cast<const RayD *>(nullptr)) ||
                               make_ray_f(r, static_cast<const RayD *>(nullptr)).ok)) {
                  active = false;
                  skipped = true;
                }
              }
              if (active) trav_begin<KIND, COUNT>(K, r, st, tv, &cnt);
            }
          }
        }
        if (want > avail) {
          pool_next = base + (want - avail);
          pool_end = base + take;
          if (base >= n) exhausted = true;
        } else {
          pool_next += want;
        }
      }
      if constexpr (!kWide && !kRest) break;
      if (!__any_sync(kFull, skipped)) break;
      if constexpr (kWide) {
        const unsigned handed = __ballot_sync(kFull, deferred);
        if (handed && !list_full) {
          uint32_t at = 0;
          if (lane == 0) at = atomicAdd(io.uncovered_count, __popc(handed));
          at = __shfl_sync(kFull, at, 0);
          list_full = at + __popc(handed) > kUncoveredList;
          at += __popc(handed & below);
          if (deferred && at < kUncoveredList) io.uncovered[at] = i;
        }
      }
    }
    // every lane idle: the global counter has passed the end of the batch
    const unsigned stepping = __ballot_sync(kFull, active);
    if (!stepping) break;
    if (active) {
      if constexpr (kWide) {
        if (tv.live) wtrav_to_leaf<KIND, COUNT>(K, r, f, hl, tv, sk, tid, io.error_word, &cnt);
        // what only the leaf steps read of the ray is formed again here, so that no register
        // holds it through the walk (1 / w has w's sign for a covered ray)
        r.tmin = io.tmin ? ldg(io.tmin + i) : 0.0;
        r.any_hit = io.any_hit != 0;
        r.sx = f.oct & 1u, r.sy = (f.oct >> 1) & 1u, r.sz = f.oct >> 2;
        while (tv.live && tv.post != kNoLeaf)
          wtrav_leaf<KIND, COUNT>(K, r, f, st, hl, tv, io.error_word, &cnt);
        // The lanes that had a leaf meet the others here; the compiler otherwise keeps them apart
        // through the next walk.  10,000 spheres, 1M rays: 12.2 active lanes for 10.8, 586 -> 519 us
        // FP64 and 530 -> 472 mixed.  A mesh's leaves differ less and the wait costs as much: terrain
        // 4,550 -> 4,590 us, though 394 -> 381 mixed on 20,480 triangles.
        if constexpr (KIND != kMesh) __syncwarp(stepping);
      } else {
        if (tv.live) trav_to_leaf<KIND, COUNT>(K, r, st, tv, sk, tid, io.error_word, &cnt);
        if (tv.live) trav_leaf<KIND, COUNT>(K, r, st, tv, sk, tid, io.error_word, &cnt);
      }
      if (!tv.live) {
        if (kWide && tv.post == kRedoLeaf) {  // rare: the binary pass traces this ray
          const uint32_t at = atomicAdd(io.redo_count, 1u);
          if (at < kRedoList) io.redo[at] = i;
        } else {
          if constexpr (kWide) {
            r.tmax = io.tmax ? ldg(io.tmax + i) : kDblMax;
            wtrav_end<KIND>(K, r, st);
          }
          finalize_kind<KIND>(S, r, st, i, first != 0, io.t, io.uv, io.normal, io.prim, io.geom,
                              io.hit);
        }
        active = false;
      }
    }
  }
  if (COUNT) {
    for (int k = 0; k < kNumKinds; ++k) {
      unsigned long long v[4] = {cnt.box[k], cnt.prim[k], cnt.node[k], cnt.leaf[k]};
      for (int j = 0; j < 4; ++j) {
        for (int off = 16; off > 0; off >>= 1) v[j] += __shfl_down_sync(kFull, v[j], off);
        if (lane == 0 && v[j]) atomicAdd(totals + j * kNumKinds + k, v[j]);
      }
    }
  }
}

// The FP64 kernels, and the mixed-precision kernels with a register cap: the wide walk keeps
// the FP64 ray and hit state live beside its FP32 node state, and its latency-bound loop gains
// more from resident warps than it loses to the cap.
template <int KIND, bool COUNT, bool LOCAL>
__global__ void __launch_bounds__(kMaxTraceThreads)
    trace_kind_kernel(SceneView S, RayIO io, int first, uint32_t *work_counter,
                      unsigned long long *totals) {
  trace_kind_body<KIND, COUNT, NoWalk, LOCAL>(S, io, first, work_counter, totals);
}

#ifndef BZR_WIDE_REGS
#define BZR_WIDE_REGS 72
#endif
template <int KIND, bool COUNT, bool LOCAL>
__global__ void __maxnreg__(BZR_WIDE_REGS)
    trace_wide_kernel(SceneView S, RayIO io, int first, uint32_t *work_counter,
                      unsigned long long *totals) {
  if (int(blockIdx.x) < io.out_blocks)
    trace_left_out_body<KIND, COUNT, RayW, LOCAL>(S, io, first, totals);
  else
    trace_kind_body<KIND, COUNT, RayW, LOCAL>(S, io, first, work_counter, totals);
}

// The FP64 mode's wide walk, with the thread-local stack (other stacks take the binary walk).
// Its cap of 80 registers (6 blocks of 128 per SM) is the measured optimum over the workloads:
// terrain / mixed primitives / icosphere 4,415 / 1,394 / 99 us at 72, 4,606 / 1,387 / 94 at 80,
// 4,964 / 1,417 / 105 at 88, 4,943 / 1,407 / 104 at 96.
constexpr int kWide64Regs = 80;
template <int KIND>
__global__ void __maxnreg__(kWide64Regs)
    trace_wide64_kernel(SceneView S, RayIO io, int first, uint32_t *work_counter,
                      unsigned long long *totals) {
  if (int(blockIdx.x) < io.out_blocks)
    trace_left_out_body<KIND, false, RayD, true>(S, io, first, totals);
  else
    trace_kind_body<KIND, false, RayD, true>(S, io, first, work_counter, totals);
}

// The binary pass over the rays that a wide pass handed on.
template <int KIND, bool COUNT, bool LOCAL>
__global__ void __launch_bounds__(kMaxTraceThreads)
    trace_rest_kernel(SceneView S, RayIO io, int first, uint32_t *work_counter,
                      unsigned long long *totals) {
  trace_kind_body<KIND, COUNT, Rest, LOCAL>(S, io, first, work_counter, totals);
}

template <int KIND, bool COUNT, bool MIXED, bool LOCAL>
constexpr auto trace_kernel() {  // cylinders have no wide walk
  if constexpr (MIXED && KIND != kCylinders)
    return trace_wide_kernel<KIND, COUNT, LOCAL>;
  else
    return trace_kind_kernel<KIND, COUNT, LOCAL>;
}

// Batching form: one kind over many scenes.  Warps take chunks of one scene's rays; a lane
// keeps its own ray's scene, so a warp may finish rays of one scene while starting another's.
// The pass of a scene's first kind writes its whole record; the pass of its last kind
// completes it and stamps the scene's completion time.
// LCAP: entries of the thread-local stack (the batch's stack-depth knob: 32 or 64).  F: the walk,
// as in trace_kind_body; rays that a wide walk does not cover take the binary one in the same
// kernel.
template <int KIND, class F, bool LOCAL, uint32_t LCAP>
__device__ __forceinline__ void trace_batch_body(const BatchView &B, const RayIO &io,
                                                 uint32_t *chunk_counter, uint32_t stack_cap) {
  constexpr bool kWide = !std::is_same<F, NoWalk>::value && KIND != kCylinders;
  extern __shared__ __align__(16) unsigned char smem[];
  double lkey[LOCAL ? LCAP : 1];
  uint32_t lref[LOCAL ? LCAP : 1];
  Stack sk;
  uint32_t tid;
  init_stack<LOCAL, LCAP>(sk, tid, stack_cap, smem, lkey, lref);
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  uint32_t pool_next = 0, pool_end = 0, pool_scene = 0;  // warp-uniform
  bool exhausted = false;
  bool active = false;
  uint32_t i = 0, sc = 0;
  const KindView *K = nullptr;
  Ray r;
  F f;
  typename F::Bound hl = 0;
  bool wide = false;
  KState st;
  Trav tv;
  Counts cnt = {};
  for (;;) {
    const unsigned idle = __ballot_sync(kFull, !active);
    if (idle && !exhausted) {
      const uint32_t want = __popc(idle), avail = pool_end - pool_next;
      const uint32_t rank = __popc(idle & below);
      uint32_t base = 0, cbegin = 0, cend = 0, cscene = 0;
      bool got_chunk = false;
      if (want > avail) {  // next chunk that has this kind
        uint32_t c = 0;
        for (;;) {
          if (lane == 0) c = atomicAdd(chunk_counter, 1u);
          c = __shfl_sync(kFull, c, 0);
          if (c >= B.n_chunks) {
            exhausted = true;
            break;
          }
          const BatchChunk ch = B.chunks[c];
          if (B.views[ch.scene].k[KIND].present && B.views[ch.scene].k[KIND].n_prims) {
            cbegin = ch.begin;
            cend = ch.end;
            cscene = ch.scene;
            got_chunk = true;
            break;
          }
        }
        base = cbegin;
      }
      if (!active) {
        uint32_t idx = 0, s2 = 0;
        bool ok = false;
        if (rank < avail) {
          idx = pool_next + rank;
          s2 = pool_scene;
          ok = true;
        } else if (got_chunk && base + (rank - avail) < cend) {
          idx = base + (rank - avail);
          s2 = cscene;
          ok = true;
        }
        if (ok) {
          i = io.perm ? io.perm[idx] : idx;  // a sorted batch keeps each scene's range
          sc = s2;
          active = true;
          K = &B.views[sc].k[KIND];
          r = make_ray(io.org + 3 * size_t(i), io.dir + 3 * size_t(i), io.tmin ? io.tmin[i] : 0.0,
                       io.tmax ? io.tmax[i] : kDblMax);
          r.any_hit = io.any_hit != 0;
          if constexpr (kWide) {
            f = make_ray_f(r, static_cast<const F *>(nullptr));
            wide = K->mixed_ok && f.ok;
          }
          bool begun = false;
          if constexpr (kWide) {
            if (wide) {
              wtrav_begin<KIND, false>(*K, r, f, st, hl, tv, &cnt);
              begun = true;
            }
          }
          if (!begun) trav_begin<KIND, false>(*K, r, st, tv, &cnt);
        }
      }
      if (want > avail) {
        if (got_chunk) {
          const uint32_t used = want - avail;
          pool_next = cbegin + (used < cend - cbegin ? used : cend - cbegin);
          pool_end = cend;
          pool_scene = cscene;
        } else {
          pool_next = pool_end;
        }
      } else {
        pool_next += want;
      }
    }
    if (!__any_sync(kFull, active)) break;
    if (active) {
      bool stepped = false;
      if constexpr (kWide) {
        if (wide) {
          if (tv.live) wtrav_to_leaf<KIND, false>(*K, r, f, hl, tv, sk, tid, io.error_word, &cnt);
          // as in trace_kind_body: what only the leaf steps read is formed again here
          r.tmin = io.tmin ? ldg(io.tmin + i) : 0.0;
          r.any_hit = io.any_hit != 0;
          r.sx = f.oct & 1u, r.sy = (f.oct >> 1) & 1u, r.sz = f.oct >> 2;
          while (tv.live && tv.post != kNoLeaf)
            wtrav_leaf<KIND, false>(*K, r, f, st, hl, tv, io.error_word, &cnt);
          if (!tv.live && tv.post == kRedoLeaf) {  // rare: the binary walk, from the start
            wide = false;
            r.tmax = io.tmax ? ldg(io.tmax + i) : kDblMax;
            trav_begin<KIND, false>(*K, r, st, tv, &cnt);
          }
          stepped = true;
        }
      }
      if (!stepped) {
        if (tv.live) trav_to_leaf<KIND, false>(*K, r, st, tv, sk, tid, io.error_word, &cnt);
        if (tv.live) trav_leaf<KIND, false>(*K, r, st, tv, sk, tid, io.error_word, &cnt);
      }
      if (!tv.live) {
        if constexpr (kWide) {
          r.tmax = io.tmax ? ldg(io.tmax + i) : kDblMax;
          if (wide) wtrav_end<KIND>(*K, r, st);
        }
        finalize_kind<KIND>(B.views[sc], r, st, i, B.first_kind[sc] == KIND, io.t, io.uv,
                            io.normal, io.prim, io.geom, io.hit);
        // The count of a scene's unfinished rays serves the completion stamps only.  Most rays
        // in flight belong to one or two scenes, and an atomic per ray on their counters set the
        // pace of the whole batch (3M rays in 48 scenes, mixed:
        // 2,140 -> 1,514 us without them): without stamps nothing is counted, and with
        // them the lanes that finish together count once per scene.
        if (B.scene_done_ns && B.last_kind[sc] == KIND) {
          const unsigned same = __match_any_sync(__activemask(), sc);
          const uint32_t done = __popc(same);
          if (lane == unsigned(__ffs(same)) - 1u &&
              atomicSub(B.scene_left + sc, done) == done) {
            __threadfence();
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            B.scene_done_ns[sc] = now;
          }
        }
        active = false;
      }
    }
  }
}

// The batch's binary kernels, and its wide kernels under a register cap, as trace_wide_kernel.
// 3M rays in 48 icosphere scenes, mixed mode: 72 / 80 / 88 / 96 registers 1,560 / 1,514 / 1,621 /
// 1,599 us.
constexpr int kBatchWideRegs = 80;
template <int KIND, bool LOCAL, uint32_t LCAP>
__global__ void __launch_bounds__(kMaxTraceThreads)
    trace_batch_kernel(BatchView B, RayIO io, uint32_t *chunk_counter, uint32_t stack_cap) {
  trace_batch_body<KIND, NoWalk, LOCAL, LCAP>(B, io, chunk_counter, stack_cap);
}
template <int KIND, bool LOCAL, uint32_t LCAP>
__global__ void __maxnreg__(kBatchWideRegs)
    trace_batch_wide_kernel(BatchView B, RayIO io, uint32_t *chunk_counter, uint32_t stack_cap) {
  trace_batch_body<KIND, RayW, LOCAL, LCAP>(B, io, chunk_counter, stack_cap);
}
// FP64 mode, 3M rays in 48 icosphere scenes: the binary walk 2,163 us, the wide one with 80 /
// 88 / 96 / 112 registers 1,598 / 1,658 / 1,615 / 1,796 us.
constexpr int kBatchWide64Regs = 80;
template <int KIND, uint32_t LCAP>
__global__ void __maxnreg__(kBatchWide64Regs)
    trace_batch_wide64_kernel(BatchView B, RayIO io, uint32_t *chunk_counter, uint32_t stack_cap) {
  trace_batch_body<KIND, RayD, true, LCAP>(B, io, chunk_counter, stack_cap);
}
// The walk of a batch's pass: the binary one (cylinders; the FP64 mode with the stack in shared
// memory; node width 2), or the wide one in FP32 or FP64.
enum BatchWalk { kBinary, kWide32, kWide64 };
template <int KIND, int WALK, bool LOCAL, uint32_t LCAP>
constexpr auto batch_fn() {
  if constexpr (WALK == kWide32 && KIND != kCylinders)
    return trace_batch_wide_kernel<KIND, LOCAL, LCAP>;
  else if constexpr (WALK == kWide64 && LOCAL && KIND != kCylinders)
    return trace_batch_wide64_kernel<KIND, LCAP>;
  else
    return trace_batch_kernel<KIND, LOCAL, LCAP>;
}

__global__ void batch_start_kernel(BatchView B, uint32_t n_scenes) {
  for (uint32_t s = threadIdx.x; s < n_scenes; s += blockDim.x)
    if (B.scene_left) B.scene_left[s] = B.scene_rays[s];
  if (threadIdx.x == 0 && B.start_ns) {
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    *B.start_ns = now;
  }
}

// Output defaults for every ray of a scene without primitives (blazert/ray.h:80-84).
__global__ void fill_defaults_kernel(RayIO io) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < io.n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    if (io.t) io.t[i] = kDblMax;
    if (io.uv) io.uv[2 * i] = io.uv[2 * i + 1] = 0.0;
    if (io.normal) io.normal[3 * i] = io.normal[3 * i + 1] = io.normal[3 * i + 2] = 0.0;
    if (io.prim) io.prim[i] = 0xFFFFFFFFu;
    if (io.geom) io.geom[i] = 0xFFFFFFFFu;
    if (io.hit) io.hit[i] = 0;
  }
}

// -------------------------------------------------------------------------- coherence sort
// Sort keys of a batch of many scenes: the scene index in the top scene_bits bits, then the
// single-scene key (direction octant over the origin's Morton code in the scene's box), so
// that the counting sort keeps every scene's rays in the scene's own range.  One warp per
// chunk of the chunk table, which covers every ray of the batch when the batch is sorted
// (scenes with nothing to trace included).
__global__ void batch_sort_key_kernel(BatchView B, RayIO io, uint32_t *keys, uint32_t *counts) {
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < B.n_chunks;
       c += warps) {
    const BatchChunk ch = B.chunks[c];
    const RaySort rs = B.scene_sort[ch.scene];
    for (uint32_t p = ch.begin + lane; p < ch.end; p += 32) {
      const double *o = io.org + 3 * size_t(p), *d = io.dir + 3 * size_t(p);
      uint32_t q[3];
      for (int a = 0; a < 3; ++a) {
        float x = (float(o[a]) - rs.lo[a]) * rs.scale[a];
        x = fminf(fmaxf(x, 0.0f), 511.0f);  // NaN maps to 0
        q[a] = uint32_t(x);
      }
      const uint32_t oct = (d[0] < 0.0 ? 4u : 0u) | (d[1] < 0.0 ? 2u : 0u) | (d[2] < 0.0 ? 1u : 0u);
      const uint32_t low = (oct << 27) | (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
      const uint32_t k = B.scene_bits >= 2 ? (uint32_t(ch.scene) << (32 - B.scene_bits)) |
                                                 (low >> (B.scene_bits - 2))
                                           : (uint32_t(ch.scene) << 31) | (low << 1);
      keys[p] = k;
      atomicAdd(counts + (k >> (32 - kSortBits)), 1u);
    }
  }
}

__device__ __forceinline__ uint32_t ray_key(const RayIO &io, const RaySort &rs, uint32_t i) {
  const double *o = io.org + 3 * size_t(i), *d = io.dir + 3 * size_t(i);
  uint32_t q[3];
  for (int a = 0; a < 3; ++a) {
    float x = (float(o[a]) - rs.lo[a]) * rs.scale[a];
    x = fminf(fmaxf(x, 0.0f), 511.0f);  // NaN maps to 0
    q[a] = uint32_t(x);
  }
  const uint32_t oct = (d[0] < 0.0 ? 4u : 0u) | (d[1] < 0.0 ? 2u : 0u) | (d[2] < 0.0 ? 1u : 0u);
  return (oct << 27) | (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
}

__global__ void sort_histogram_kernel(RayIO io, RaySort rs, uint32_t *keys, uint32_t *counts) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < io.n; i += gridDim.x * blockDim.x) {
    const uint32_t k = ray_key(io, rs, i);
    keys[i] = k;
    atomicAdd(counts + (k >> (32 - kSortBits)), 1u);
  }
}

__global__ void leaf_box_kernel(KindView K, double *leaf_box) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < K.n_internal;
       i += gridDim.x * blockDim.x) {
    const double *nd = K.nodes64 + size_t(i) * kNode64Doubles;
    const uint32_t *ref = reinterpret_cast<const uint32_t *>(nd + 12);
    for (int c = 0; c < 2; ++c) {
      if (!(ref[c] & kLeafBit) || (ref[c] & kIdMask) >= K.n_prims) continue;
      double *out = leaf_box + size_t(ref[c] & kIdMask) * 6;
      for (int j = 0; j < 6; ++j) out[j] = nd[6 * c + j];
    }
  }
}

// The counting kernels (measurement only) always keep the stack in shared memory; the
// tracing kernels use the thread-local stack whenever the tree's stack fits it, unless the
// plan asks for shared memory.
inline bool use_local(const SceneView &S, const LaunchPlan &plan) {
  return !plan.shared_stack && S.stack_cap <= kLocalStack;
}

// Whether a pass of KIND in `mode` walks the wide image.  The FP64 mode does with the thread-local
// stack; its counting kernels count the binary walk.
//
// A mesh of less than kWideMinTriangles triangles keeps the binary walk: its nodes lie in L1 and
// a binary step is then the cheaper one.  543,004 / 91,204 pixels of a 320-triangle sphere 66 /
// 39 us binary, 76 / 48 wide; of a 1,280-triangle one 100 / 66 and 98 / 62.  (500 spheres and 100
// planes gain by the wide walk: 1M rays through spheres, planes and cylinders 1,380 against
// 1,359, a fitting step with 500 spheres 1,450 against 1,413.)
constexpr uint32_t kWideMinTriangles = 512;
template <int KIND>
bool walks_wide(const SceneView &S, int mode, const LaunchPlan &plan, bool count) {
  return KIND != kCylinders && S.k[KIND].present && S.k[KIND].n_prims && S.k[KIND].mixed_ok &&
         (mode == kModeMixed || (use_local(S, plan) && !count &&
                                 (KIND != kMesh || S.k[KIND].n_prims >= kWideMinTriangles)));
}

using TraceFn = void (*)(SceneView, RayIO, int, uint32_t *, unsigned long long *);

// One trace kernel on `stream`; early: launched with programmatic stream serialisation (the
// kernel before it on the stream is a trace kernel of the same call; see griddep_wait).
cudaError_t launch_one(TraceFn fn, int blocks, int threads, size_t smem, cudaStream_t stream,
                       bool early, const SceneView &S, const RayIO &io, int first,
                       uint32_t *counter, unsigned long long *totals) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, S, io, first, counter, totals);
}

// The pass of one kind: one kernel, or for a wide walk two: the wide kernel, then the binary walk of
// the rays that one handed on.  counters:
// the kTraceWords words of the call; after_trace: a trace kernel of this call precedes the pass on
// the stream.
template <int KIND, bool COUNT>
cudaError_t launch_kind(const SceneView &S, const RayIO &io, int mode, int first,
                        bool after_trace, const LaunchPlan &plan, cudaStream_t stream,
                        uint32_t *counters, unsigned long long *totals) {
  const int th = plan.threads;
  const bool local = !COUNT && use_local(S, plan);
  const size_t smem = trace_kind_smem(S.stack_cap, th, local, io.top_nodes);
  const bool early = after_trace && plan.early_launch;
  const TraceFn fp64 = local ? trace_kernel<KIND, false, false, true>()
                             : trace_kernel<KIND, COUNT, false, false>();
  // no more blocks than the batch fills
  auto grid = [&](int blocks) {
    return int(std::min<uint64_t>(uint64_t(blocks), (uint64_t(io.n) + th - 1) / th));
  };
  if constexpr (KIND != kCylinders) {
    if (walks_wide<KIND>(S, mode, plan, COUNT)) {
      const bool mixed = mode == kModeMixed;
      const TraceFn wide_fn = !mixed ? trace_wide64_kernel<KIND>
                              : local ? trace_kernel<KIND, false, true, true>()
                                      : trace_kernel<KIND, COUNT, true, false>();
      const TraceFn rest_fn = local ? trace_rest_kernel<KIND, false, true>
                                    : trace_rest_kernel<KIND, COUNT, false>;
      RayIO wide = io;
      wide.uncovered_count = counters + 2 * kNumKinds + KIND;
      wide.redo_count = counters + 3 * kNumKinds + KIND;
      wide.uncovered = counters + kTraceListWord;
      wide.redo = wide.uncovered + kUncoveredList;
      wide.wide_mode = mode;
      const int blocks = grid(mixed ? plan.blocks32[KIND] : plan.blocks64w[KIND]);
      wide.out_blocks = blocks;
      const cudaError_t e = launch_one(wide_fn, 2 * blocks, th, smem, stream, early, S, wide, first,
                                       counters + KIND, totals);
      if (e != cudaSuccess) return e;
      // Hardly ever any ray: a small grid, which leaves the SMs to the next pass, except where it
      // can be all of them, a large batch (covers_hardly_any) or one of far origins in mixed mode.
      const bool few = !mixed && io.n < whole_min<KIND>();
      const int rest_blocks = few ? std::min(plan.blocks_rest[KIND], plan.sms)
                                  : plan.blocks_rest[KIND];
      return launch_one(rest_fn, grid(rest_blocks), th, smem, stream, plan.early_launch, S, wide,
                        first, counters + kNumKinds + KIND, totals);
    }
  }
  return launch_one(fp64, grid(plan.blocks[KIND]), th, smem, stream, early, S, io, first,
                    counters + KIND, totals);
}

// Resident blocks per SM of `fn` with `threads` per block and `smem` bytes of dynamic shared
// memory, times the SMs.
cudaError_t grid_for(const void *fn, int threads, size_t smem, int sms, int *blocks) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  if (e != cudaSuccess) return e;
  *blocks = sms * (per_sm > 0 ? per_sm : 1);
  return cudaSuccess;
}

template <int KIND>
cudaError_t prepare_kind(const SceneView &S, LaunchPlan *plan) {
  const int th = plan->threads;
  const size_t smem = trace_kind_smem(S.stack_cap, th, false, plan->top_nodes);
  const size_t smem_local = trace_kind_smem(S.stack_cap, th, true, plan->top_nodes);
  const void *shared_fns[4] = {
      reinterpret_cast<const void *>(trace_kernel<KIND, false, false, false>()),
      reinterpret_cast<const void *>(trace_kernel<KIND, true, false, false>()),
      reinterpret_cast<const void *>(trace_kernel<KIND, false, true, false>()),
      reinterpret_cast<const void *>(trace_kernel<KIND, true, true, false>())};
  int ignored = 0;
  for (const void *fn : shared_fns) {
    const cudaError_t e = grid_for(fn, th, smem, plan->sms, &ignored);
    if (e != cudaSuccess) return e;
  }
  const bool local = use_local(S, *plan);
  const size_t bytes = local ? smem_local : smem;
  cudaError_t e = grid_for(
      local ? reinterpret_cast<const void *>(trace_kernel<KIND, false, false, true>())
            : shared_fns[0], th, bytes, plan->sms, &plan->blocks[KIND]);
  if (e != cudaSuccess) return e;
  e = grid_for(local ? reinterpret_cast<const void *>(trace_kernel<KIND, false, true, true>())
                     : shared_fns[2], th, bytes, plan->sms, &plan->blocks32[KIND]);
  if constexpr (KIND != kCylinders) {
    const void *rest_fns[2] = {reinterpret_cast<const void *>(trace_rest_kernel<KIND, true, false>),
                               reinterpret_cast<const void *>(trace_rest_kernel<KIND, false, false>)};
    for (const void *fn : rest_fns)
      if (e == cudaSuccess) e = grid_for(fn, th, smem, plan->sms, &plan->blocks_rest[KIND]);
    if (local && e == cudaSuccess)
      e = grid_for(reinterpret_cast<const void *>(trace_rest_kernel<KIND, false, true>), th, bytes,
                   plan->sms, &plan->blocks_rest[KIND]);
    if (local && e == cudaSuccess)
      e = grid_for(reinterpret_cast<const void *>(trace_wide64_kernel<KIND>), th,
                   bytes, plan->sms, &plan->blocks64w[KIND]);
  }
  return e;
}

}  // namespace

cudaError_t launch_defaults(const RayIO &io, int sms, cudaStream_t stream) {
  const int threads = 256;
  const uint64_t want = (uint64_t(io.n) + threads - 1) / threads;
  const int blocks = int(want < uint64_t(sms) * 8 ? (want ? want : 1) : uint64_t(sms) * 8);
  fill_defaults_kernel<<<blocks, threads, 0, stream>>>(io);
  return cudaGetLastError();
}

cudaError_t fill_leaf_boxes(const KindView &K, double *leaf_box) {
  if (K.root_ref & kLeafBit)
    return cudaMemcpy(leaf_box, K.root_box, sizeof K.root_box, cudaMemcpyHostToDevice);
  const uint32_t blocks = (K.n_internal + 255) / 256;
  leaf_box_kernel<<<blocks < 1184 ? blocks : 1184, 256>>>(K, leaf_box);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? cudaStreamSynchronize(nullptr) : e;
}

size_t trace_smem_bytes(uint32_t stack_cap, int threads) {
  return size_t(stack_cap) * threads * (sizeof(double) + sizeof(uint32_t));
}

size_t trace_kind_smem(uint32_t stack_cap, int threads, bool local, uint32_t top_nodes) {
  const size_t stack = local ? 0 : (trace_smem_bytes(stack_cap, threads) + 15) / 16 * 16;
  return stack + size_t(top_nodes) * 128;
}


cudaError_t trace_prepare(const SceneView &S, LaunchPlan *plan) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  plan->sms = sms;
  if ((e = prepare_kind<kMesh>(S, plan)) != cudaSuccess) return e;
  if ((e = prepare_kind<kSpheres>(S, plan)) != cudaSuccess) return e;
  if ((e = prepare_kind<kPlanes>(S, plan)) != cudaSuccess) return e;
  if ((e = small_prepare(plan)) != cudaSuccess) return e;
  return prepare_kind<kCylinders>(S, plan);
}

int trace_passes(const SceneView &S) {
  int n = 0;
  for (int k = 0; k < kNumKinds; ++k) n += (S.k[k].present && S.k[k].n_prims) ? 1 : 0;
  return n;
}

cudaError_t launch_trace(const SceneView &S, const RayIO &io, int mode, const LaunchPlan &plan,
                         cudaStream_t stream, uint32_t *counters, unsigned long long *totals) {
  if (!totals && small_batch(S, plan, io.n)) return launch_small(S, io, plan, stream);
  cudaError_t e = cudaMemsetAsync(counters, 0, kTraceCounterWords * sizeof(uint32_t), stream);
  if (e != cudaSuccess) return e;
  RayIO sorted = io;
  sorted.chunk = plan.chunk;
  sorted.top_nodes = plan.top_nodes;
  // scratch from the pool: the sort's keys, permutation and bucket counts
  const bool sort = plan.sort.enabled && io.n >= plan.sort_min_rays && trace_passes(S) > 0;
  const size_t nb = size_t(1) << kSortBits;
  uint32_t *scratch = nullptr;
  if (sort) {
    e = bzr::pool_malloc(&scratch, (2 * size_t(io.n) + nb) * sizeof(uint32_t), plan.pool, stream);
    if (e != cudaSuccess) return e;
  }
  if (sort) {
    uint32_t *keys = scratch, *perm = scratch + io.n, *counts = scratch + 2 * size_t(io.n);
    e = cudaMemsetAsync(counts, 0, nb * sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;
    const int blocks = plan.sms * 8;
    sort_histogram_kernel<<<blocks, 256, 0, stream>>>(io, plan.sort, keys, counts);
    bucket_scan_kernel<<<1, 1024, 0, stream>>>(counts);
    bucket_scatter_kernel<<<blocks, 256, 0, stream>>>(io.n, keys, counts, perm);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    sorted.perm = perm;
  }
  const RayIO &run = sorted;
  int first = 1;
  for (int k = 0; k < kNumKinds; ++k) {
    if (!S.k[k].present || S.k[k].n_prims == 0) continue;
    uint32_t *c = counters;
    const bool after = !first;
    switch (k) {
      case kMesh:
        e = totals ? launch_kind<kMesh, true>(S, run, mode, first, after, plan, stream, c, totals)
                   : launch_kind<kMesh, false>(S, run, mode, first, after, plan, stream, c,
                                               nullptr);
        break;
      case kSpheres:
        e = totals ? launch_kind<kSpheres, true>(S, run, mode, first, after, plan, stream, c,
                                                 totals)
                   : launch_kind<kSpheres, false>(S, run, mode, first, after, plan, stream, c,
                                                  nullptr);
        break;
      case kPlanes:
        e = totals ? launch_kind<kPlanes, true>(S, run, mode, first, after, plan, stream, c,
                                                totals)
                   : launch_kind<kPlanes, false>(S, run, mode, first, after, plan, stream, c,
                                                 nullptr);
        break;
      default:
        e = totals ? launch_kind<kCylinders, true>(S, run, mode, first, after, plan, stream, c,
                                                   totals)
                   : launch_kind<kCylinders, false>(S, run, mode, first, after, plan, stream, c,
                                                    nullptr);
        break;
    }
    if (e != cudaSuccess) break;  // the scratch is still released below
    first = 0;
  }
  if (first && e == cudaSuccess) {  // nothing to trace
    const int threads = 256;
    const uint64_t want = (uint64_t(io.n) + threads - 1) / threads;
    const int blocks = int(want < uint64_t(plan.sms) * 8 ? want : uint64_t(plan.sms) * 8);
    fill_defaults_kernel<<<blocks > 0 ? blocks : 1, threads, 0, stream>>>(io);
    e = cudaGetLastError();
  }
  if (scratch) {
    const cudaError_t f = cudaFreeAsync(scratch, stream);
    if (e == cudaSuccess) e = f;
  }
  return e;
}

namespace {
// The kernel a batch launch uses for one kind: stack storage (thread-local with 32 or 64
// entries, or shared) and mode.
using BatchFn = void (*)(BatchView, RayIO, uint32_t *, uint32_t);
template <int KIND, int WALK>
BatchFn batch_kernel(bool local, uint32_t lcap) {
  if (local && lcap == 32) return batch_fn<KIND, WALK, true, 32>();
  if (local) return batch_fn<KIND, WALK, true, kLocalStack>();
  return batch_fn<KIND, WALK, false, kLocalStack>();
}

inline bool batch_local(uint32_t stack_cap, const BatchPlan &plan) {
  return !plan.shared_stack && stack_cap <= plan.local_stack;
}

// The kernel of one kind's pass in `mode`.
template <int KIND>
BatchFn batch_pass(int mode, const BatchPlan &plan) {
  const bool local = batch_local(plan.stack_cap, plan);
  if (KIND == kCylinders || (mode == kModeMixed && plan.node_width != 8))
    return batch_kernel<KIND, kBinary>(local, plan.local_stack);
  if (mode == kModeMixed) return batch_kernel<KIND, kWide32>(local, plan.local_stack);
  return batch_kernel<KIND, kWide64>(local, plan.local_stack);
}

template <int KIND>
cudaError_t prepare_batch_kind(const BatchPlan &plan, int *blocks, int *blocks32) {
  const size_t smem = batch_local(plan.stack_cap, plan)
                          ? 0 : trace_smem_bytes(plan.stack_cap, plan.threads);
  const cudaError_t e = grid_for(reinterpret_cast<const void *>(batch_pass<KIND>(kModeFp64, plan)),
                                 plan.threads, smem, plan.sms, blocks);
  if (e != cudaSuccess) return e;
  return grid_for(reinterpret_cast<const void *>(batch_pass<KIND>(kModeMixed, plan)), plan.threads,
                  smem, plan.sms, blocks32);
}
}  // namespace

cudaError_t batch_prepare(uint32_t stack_cap, BatchPlan *plan) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  plan->sms = sms;
  plan->stack_cap = stack_cap;
  if ((e = prepare_batch_kind<kMesh>(*plan, &plan->blocks[kMesh], &plan->blocks32[kMesh])) !=
      cudaSuccess)
    return e;
  if ((e = prepare_batch_kind<kSpheres>(*plan, &plan->blocks[kSpheres],
                                        &plan->blocks32[kSpheres])) != cudaSuccess)
    return e;
  if ((e = prepare_batch_kind<kPlanes>(*plan, &plan->blocks[kPlanes],
                                       &plan->blocks32[kPlanes])) != cudaSuccess)
    return e;
  return prepare_batch_kind<kCylinders>(*plan, &plan->blocks[kCylinders],
                                        &plan->blocks32[kCylinders]);
}

cudaError_t launch_batch(const BatchView &B, const RayIO &io, int mode, const BatchPlan &plan,
                         cudaStream_t stream, uint32_t *counters,
                         const BatchSortScratch &sort_scratch) {
  cudaError_t e = cudaMemsetAsync(counters, 0, kNumKinds * sizeof(uint32_t), stream);
  if (e != cudaSuccess) return e;
  batch_start_kernel<<<1, 256, 0, stream>>>(B, B.n_scenes);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  RayIO run = io;
  if (plan.sort && sort_scratch.perm && B.n_chunks) {
    // every ray of the batch gets a scene-major key; rays of scenes without chunks are never
    // taken from the permutation, so their keys only need to land in their scene's range
    e = cudaMemsetAsync(sort_scratch.counts, 0, (size_t(1) << kSortBits) * sizeof(uint32_t),
                        stream);
    if (e != cudaSuccess) return e;
    const int blocks = plan.sms * 8;
    batch_sort_key_kernel<<<blocks, 256, 0, stream>>>(B, io, sort_scratch.keys,
                                                      sort_scratch.counts);
    bucket_scan_kernel<<<1, 1024, 0, stream>>>(sort_scratch.counts);
    bucket_scatter_kernel<<<blocks, 256, 0, stream>>>(io.n, sort_scratch.keys,
                                                      sort_scratch.counts, sort_scratch.perm);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    run.perm = sort_scratch.perm;
  }
  const size_t smem = batch_local(plan.stack_cap, plan)
                          ? 0 : trace_smem_bytes(plan.stack_cap, plan.threads);
  for (int k = 0; k < kNumKinds; ++k) {
    if (!(plan.kinds_present & (1 << k))) continue;
    const BatchFn fn = k == kMesh      ? batch_pass<kMesh>(mode, plan)
                       : k == kSpheres ? batch_pass<kSpheres>(mode, plan)
                       : k == kPlanes  ? batch_pass<kPlanes>(mode, plan)
                                       : batch_pass<kCylinders>(mode, plan);
    const int blocks = mode == kModeMixed ? plan.blocks32[k] : plan.blocks[k];
    fn<<<blocks, plan.threads, smem, stream>>>(B, run, counters + k, plan.stack_cap);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace bzr
