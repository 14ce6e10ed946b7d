// Closest-hit traversal of small batches (intersect1 included) for sm_100a: one launch for
// every kind, with the batch spread over the whole GPU.
//
// What bounds a small batch is the latency of its slowest warp, not throughput.  The persistent
// kernels of trace.cu give a warp 32 rays and run the kinds one after another: 3,001 rays fill
// 24 blocks on 148 SMs, each warp steps through the divergent walks of its 32 rays, and each
// kind waits for the slowest ray of the kind before it.  Here
//  * a block has one warp per kind present; all of them trace the same rays, each ray in the
//    same lane of every warp, and one of them merges the kinds' results from shared memory with
//    intersect1's rule (blazert/scene.h:161-210);
//  * a warp takes as few rays as fill the GPU once: lanes = ceil(n / resident blocks), so up to
//    resident blocks rays each walk alone in their warp.
// Triangles, spheres and planes walk the wide image in FP64 (RayD, trace_core.cuh) and rays
// that it does not cover, or whose walk ends without a result, the binary nodes in the same
// kernel; cylinders walk the binary nodes.  The results are the persistent kernels' bits.
// B200, device arrays, against the persistent kernels: 32 / 4,096 / 16,384 rays through spheres,
// cylinders and planes 130 / 168 / 172 -> 39 / 63 / 98 us, on a 5,120-triangle sphere 40 / 59 /
// 64 -> 23 / 39 / 50 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "layout.h"
#include "trace.h"
#include "trace_core.cuh"

namespace bzr {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
// Registers: 80 / 96 / 128 / 168 give 45.6 / 43.5 / 39.2 / 39.2 us for 32 rays through three
// kinds, 84 / 70 / 63 / 64 for 4,096 and 120 / 115 / 98 / 95 for 16,384 (fewer resident blocks
// against spills in the walks).
constexpr int kRegs = 128;

struct SmallArgs {
  int kind[kNumKinds];  // the kind of each warp of a block
  int n_kinds;
  uint32_t lanes;  // rays per block
  SmallDone done;
};

// A kind's result of one ray, as the merge reads it.
struct Partial {
  double hit, u, v, nx, ny, nz;
  uint32_t pos;
};

// One kind's traversal of the warp's rays; st holds the result on return.
template <int KIND>
__device__ __forceinline__ void trace_lanes(const SceneView &S, const Ray &r, bool mine,
                                            const Stack &sk, uint32_t *err, KState &st) {
  const KindView &K = S.k[KIND];
  constexpr bool kWide = KIND != kCylinders;
  Trav tv;
  bool binary = mine;
  if constexpr (kWide) {
    const RayD f = make_ray_f(r, static_cast<const RayD *>(nullptr));
    bool active = mine && K.mixed_ok && f.ok;
    binary = mine && !active;
    int32_t hl = 0;
    if (active) wtrav_begin<KIND, false>(K, r, f, st, hl, tv, nullptr);
    while (__any_sync(kFull, active)) {
      if (active) {
        if (tv.live) wtrav_to_leaf<KIND, false>(K, r, f, hl, tv, sk, 0, err, nullptr);
        while (tv.live && tv.post != kNoLeaf)
          wtrav_leaf<KIND, false>(K, r, f, st, hl, tv, err, nullptr);
        if (!tv.live) {
          active = false;
          binary = tv.post == kRedoLeaf;  // rare: the binary walk, from the start
          if (!binary) wtrav_end<KIND>(K, r, st);
        }
      }
    }
  }
  // A loop of its own: rays along a plane of box bounds take thousands of its steps.
  if (binary) trav_begin<KIND, false>(K, r, st, tv, nullptr);
  while (__any_sync(kFull, binary)) {
    if (binary) {
      if (tv.live) trav_to_leaf<KIND, false>(K, r, st, tv, sk, 0, err, nullptr);
      if (tv.live) trav_leaf<KIND, false>(K, r, st, tv, sk, 0, err, nullptr);
      binary = tv.live;
    }
  }
}

template <int KIND>
__device__ __forceinline__ void write_result(const SceneView &S, const RayIO &io, const Ray &r,
                                             const Partial &p, uint64_t i) {
  KState st;
  st.hit = p.hit;
  st.u = p.u;
  st.v = p.v;
  st.pos = p.pos;
  st.n = d3(p.nx, p.ny, p.nz);
  finalize_kind<KIND>(S, r, st, i, true, io.t, io.uv, io.normal, io.prim, io.geom, io.hit);
}

__global__ void __maxnreg__(kRegs)
    trace_small_kernel(SceneView S, RayIO io, const SmallArgs args) {
  __shared__ double rays[32 * 8];  // origin, direction, tmin, tmax of each lane's ray
  extern __shared__ Partial part[];  // the kinds' results, 32 each; none for a single kind
  double lkey[kLocalStack];
  uint32_t lref[kLocalStack];
  Stack sk;
  sk.key = lkey;
  sk.ref = lref;
  sk.cap = S.stack_cap < kLocalStack ? S.stack_cap : kLocalStack;
  sk.stride = 1;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t first = blockIdx.x * args.lanes;
  const uint32_t left = io.n - first;  // the grid has no block past the batch
  const uint32_t count = left < args.lanes ? left : args.lanes;
  // the rays are read once per block (they may lie in host memory), in whole rows
  for (uint32_t j = threadIdx.x; j < 3 * count; j += blockDim.x) {
    rays[(j / 3) * 8 + j % 3] = io.org[3 * size_t(first) + j];
    rays[(j / 3) * 8 + 3 + j % 3] = io.dir[3 * size_t(first) + j];
  }
  for (uint32_t j = threadIdx.x; j < count; j += blockDim.x) {
    rays[j * 8 + 6] = io.tmin ? io.tmin[first + j] : 0.0;
    rays[j * 8 + 7] = io.tmax ? io.tmax[first + j] : kDblMax;
  }
  __syncthreads();
  const bool mine = lane < count;
  const double *q = rays + 8 * (mine ? lane : 0);
  Ray r = make_ray(q, q + 3, q[6], q[7]);
  r.any_hit = io.any_hit != 0;
  KState st;
  st.hit = r.tmax;
  st.u = st.v = 0.0;
  st.pos = 0xFFFFFFFFu;
  st.n = d3(0.0, 0.0, 0.0);
  const int kind = args.kind[warp];
  switch (kind) {
    case kMesh: trace_lanes<kMesh>(S, r, mine, sk, io.error_word, st); break;
    case kSpheres: trace_lanes<kSpheres>(S, r, mine, sk, io.error_word, st); break;
    case kPlanes: trace_lanes<kPlanes>(S, r, mine, sk, io.error_word, st); break;
    default: trace_lanes<kCylinders>(S, r, mine, sk, io.error_word, st); break;
  }
  const Partial own = {st.hit, st.u, st.v, st.n.x, st.n.y, st.n.z, st.pos};
  if (args.n_kinds > 1) {
    part[32 * warp + lane] = own;
    __syncthreads();
  }
  // The merge of finalize_kind over the kinds in their order: a kind's hit replaces what was
  // there when it is strictly closer (triangles come first and always do).
  if (warp == 0 && mine) {
    int win = 0;
    double best = kDblMax;
    for (int k = 0; args.n_kinds > 1 && k < args.n_kinds; ++k) {
      const double h = part[32 * k + lane].hit;
      if (h < r.tmax && (args.kind[k] == kMesh || h < best)) {
        win = k;
        best = h;
      }
    }
    // without a hit, the first kind's record (a miss) writes the defaults
    const Partial p = args.n_kinds > 1 ? part[32 * win + lane] : own;
    const uint64_t i = uint64_t(first) + lane;
    switch (args.kind[win]) {
      case kMesh: write_result<kMesh>(S, io, r, p, i); break;
      case kSpheres: write_result<kSpheres>(S, io, r, p, i); break;
      case kPlanes: write_result<kPlanes>(S, io, r, p, i); break;
      default: write_result<kCylinders>(S, io, r, p, i); break;
    }
  }
  // Results in host memory: tell the host when all of them are there.  The barrier orders the
  // block's results and error bits, of every warp, before its thread 0; the fence there, for the
  // whole system, orders them before the block's count (or, for a lone block, the flag); and the
  // last block's fence after the counts orders every block's before the flag, which the host reads
  // with acquire.
  if (args.done.flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long err = gridDim.x == 1 ? atomicExch(io.error_word, 0u) : 0u;
      __threadfence_system();
      bool last = gridDim.x == 1;
      if (!last && atomicAdd(args.done.blocks, 1u) == gridDim.x - 1) {
        __threadfence_system();
        err = atomicExch(io.error_word, 0u);
        *args.done.blocks = 0;
        last = true;
      }
      if (last)
        asm volatile("st.relaxed.sys.u64 [%0], %1;" ::"l"(args.done.flag),
                     "l"(err << 32 | args.done.value)
                     : "memory");
    }
  }
}

}  // namespace

// Shared memory is L1 that the walks lack: a single kind's blocks take none for the merge.
static size_t small_smem(int kinds) { return kinds > 1 ? size_t(kinds) * 32 * sizeof(Partial) : 0; }

cudaError_t small_prepare(LaunchPlan *plan) {
  for (int k = 1; k <= kNumKinds; ++k) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, reinterpret_cast<const void *>(trace_small_kernel), 32 * k, small_smem(k));
    if (e != cudaSuccess) return e;
    plan->small_blocks[k - 1] = plan->sms * std::max(1, per_sm);
  }
  return cudaSuccess;
}

// The line lies where the batch no longer fits the GPU in one wave: as many blocks as are resident
// with a warp per kind, of 32 rays, or of 8 with a single kind.  B200, this kernel against the
// persistent ones: three kinds (23,680 rays) 97 / 172 us at 16,384, 131 / 176 at 24,000, 276 / 207
// at 65,536.  One kind (18,944 rays): 16,384 pixels of a 20,480-triangle sphere 69 / 102; up to
// 75,776 rays it would still gain on most images (68,510 pixels 62 / 82), but where a row of
// rays runs along a plane of box bounds (an odd number of rows) the persistent kernels' first
// pass is the faster one: 67,405 pixels 660 / 399, 32,761 pixels 718 / 573.
bool small_batch(const SceneView &S, const LaunchPlan &plan, uint32_t n) {
  const int kinds = trace_passes(S);
  return kinds > 0 && !plan.shared_stack && S.stack_cap <= kLocalStack &&
         !(plan.sort.enabled && n >= plan.sort_min_rays) &&
         n <= (kinds > 1 ? 32u : 8u) * uint32_t(plan.small_blocks[kinds - 1]);
}

cudaError_t launch_small(const SceneView &S, const RayIO &io, const LaunchPlan &plan,
                         cudaStream_t stream, const SmallDone &done) {
  SmallArgs a = {};
  for (int k = 0; k < kNumKinds; ++k)
    if (S.k[k].present && S.k[k].n_prims) a.kind[a.n_kinds++] = k;
  const uint32_t blocks = uint32_t(plan.small_blocks[a.n_kinds - 1]);
  a.lanes = std::min<uint32_t>(32u, (io.n + blocks - 1) / blocks);
  a.done = done;
  trace_small_kernel<<<(io.n + a.lanes - 1) / a.lanes, 32 * a.n_kinds, small_smem(a.n_kinds),
                       stream>>>(S, io, a);
  return cudaGetLastError();
}

}  // namespace bzr
