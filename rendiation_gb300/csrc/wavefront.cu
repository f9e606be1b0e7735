// Wavefront executor for the first bounce of the path tracer, sm_103a.
//
// The reference runs raygen -> trace -> closest-hit -> (shadow trace, bounce)
// as device tasks whose queues are compacted every round by a two-level
// Kogge-Stone prefix scan plus a shuffle move
// (shader/ray-tracing/src/backend/wavefront_compute/mod.rs:111-196,
// shader/task-graph/src/runtime/task_group.rs:176-278,
// shader/parallel-compute/src/stream_compaction.rs:3-45). Here the fixed
// pipeline of DeviceReferencePathTracingRenderer's first bounce
// (scene/rendering/gpu-ray-tracing/src/feature/path_tracing/{ray_gen.rs,ray_hit.rs})
// is two kernels:
//
//   primary_kernel: one thread per pixel, persistent warps that claim 4x8
//     pixel tiles (4 wide, 8 tall) from a counter. Pinhole ray -> closest hit -> geometric normal facing the ray ->
//     offset_ray_hit origin -> one shadow ray to the point light and one
//     cosine-weighted bounce ray. The shadow queue and the two bins of the
//     bounce queue (grazing rays at its front, steep rays at its back) are
//     filled through warp ballots and one 64-bit atomicAdd per warp, so the
//     queues come out compacted without a separate scan pass.
//   secondary_kernel: persistent warps that fetch 32 queue entries at a time
//     from a global work counter; the grazing bounce rays, then the steep
//     ones (closest hit, the long walks), occupy the first half of the index
//     space and shadow rays (first-hit search) the second, so warps stay
//     homogeneous and the kernel ends on short work. Results scatter to the
//     pixel records.
//
// Built with -fmad=false: all shading arithmetic is IEEE f32 in the same
// order as the oracle, so secondary rays are bit-identical.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "quad.cuh"
#include "shade.cuh"
#include "traverse.cuh"
#include "wavefront.h"

namespace rdn {
namespace {

using namespace dev;

// LOCAL: the traversal stack lives in the thread's local memory (L1-cached)
// instead of shared memory, so that the stack no longer limits occupancy.
// TIER picks the register budget through the launch bounds: 0 = the
// compiler's default for 128-thread blocks (64 registers, some spills),
// 1 = at least 7 blocks of 128 per SM (72 registers, no spills, 28 warps),
// 2 = at least 9 blocks (56 registers, 36 warps, more spills).
constexpr int min_blocks(int tier) { return tier == 1 ? 7 : (tier == 2 ? 9 : 0); }

// Bounce rays leaving their surface at a cosine of at least 1/2 (three
// quarters of a cosine-weighted sample) go to the back bin of the bounce
// queue; the grazing quarter, the longest walks, to its front.
constexpr float kSteepBounceCos = 0.5f;

// Queue entry of the j-th bounce ray of the secondary kernel's index space:
// the n_front grazing rays from the queue's front, then the steep ones from
// its back (entry cap - 1 down).
__device__ __forceinline__ uint32_t bounce_entry(uint32_t j, uint32_t n_front, uint32_t cap) {
  return j < n_front ? j : cap - 1u - (j - n_front);
}

// What a pixel's primary hit sends on: one shadow ray and one bounce ray.
struct NextRays {
  bool want;
  float3 org, ldir, bdir;
  float dist, bcos;
};

// Camera ray direction (pixel centre), the same f32 steps as the host generator.
__device__ __forceinline__ float3 camera_direction(const WavefrontParams& w, uint32_t px, uint32_t py) {
  const float sx = (((float)px + 0.5f) / (float)w.width * 2.0f - 1.0f) * w.tan_half * w.aspect;
  const float sy = (1.0f - ((float)(py + w.row0) + 0.5f) / (float)w.frame_height * 2.0f) * w.tan_half;
  return normalize3(make_float3((w.forward.x + sx * w.right.x) + sy * w.up.x,
                                (w.forward.y + sx * w.right.y) + sy * w.up.y,
                                (w.forward.z + sx * w.right.z) + sy * w.up.z));
}

__device__ __forceinline__ void primary_ray(const WavefrontParams& w, float3 d, RayCtx& R) {
  R.o = w.origin;
  R.d = d;
  R.tmin = 0.0f;
  R.tmax = __int_as_float(0x7f800000);
  R.cull_mask = 0xFFu;
  R.ray_flags = 0u;
}

// Writes the pixel's record and forms its secondary rays.
__device__ __forceinline__ NextRays shade_primary(const TraceParams& p, const WavefrontParams& w, uint32_t px,
                                                  uint32_t py, float3 d, const Best& best) {
  NextRays n;
  n.want = false;
  n.org = n.ldir = n.bdir = make_float3(0.f, 0.f, 0.f);
  n.dist = n.bcos = 0.0f;
  PixelResult out;
  out.primary_prim = INVALID_NEXT;
  out.primary_t = __int_as_float(0x7f800000);
  out.bounce_prim = INVALID_NEXT;
  out.bounce_t = F32_MAX;
  out.primary_flags = 0u;
  out.light = 0u;
  out.direct = 0.0f;
  out.primary_instance = INVALID_NEXT;
  if (best.have) {
    const uint4 gm = __ldg(reinterpret_cast<const uint4*>(p.tri_root + best.geom_slot));
    out.primary_prim = __ldg(p.redirect + best.k) - gm.z;
    out.primary_t = best.t;
    out.primary_flags = 1u;
    out.primary_instance = best.inst;
    // hit point and world geometric normal facing the incoming ray
    const float3 hp = w.origin + d * best.t;
    const float3 nf = facing_normal(p, best.k, best.inst, d);
    n.org = offset_ray_hit(hp, nf);
    const float3 L = w.light - n.org;
    const float dist2 = dot3(L, L);
    n.dist = sqrtf(dist2);
    n.ldir = normalize3(L);
    out.direct = fmaxf(0.0f, dot3(nf, n.ldir)) / dist2;  // kept only if the light is visible
    uint32_t state = xxhash32(px, py + w.row0, w.sample_index * 3u);
    const float s0 = sample_next(state);
    const float s1 = sample_next(state);
    n.bdir = cosine_sample_in_dir(nf, s0, s1);
    n.bcos = dot3(n.bdir, nf);
    n.want = true;
  }
  w.out[(size_t)py * w.width + px] = out;
  return n;
}

// Compacted appends: shadow rays to their queue; bounce rays to two bins of
// theirs, grazing ones (the longer walks) from its front and steep ones
// from its back, so that a warp of the secondary kernel traces rays of
// like walk lengths. One 64-bit atomic per warp counts both bins (low and
// high word); the shadow slot is the sum of the two bases plus the lane's
// rank, so the shadow queue stays dense. Every lane of the warp is here.
__device__ __forceinline__ void append_rays(const WavefrontParams& w, uint32_t px, uint32_t py, const NextRays& n) {
  const uint32_t lane = threadIdx.x & 31u;
  const bool steep = n.want && n.bcos >= kSteepBounceCos;
  const uint32_t m_want = __ballot_sync(0xffffffffu, n.want), m_steep = __ballot_sync(0xffffffffu, steep);
  const uint32_t m_front = m_want & ~m_steep;
  unsigned long long bases = 0ull;
  if (lane == 0 && m_want)
    bases = atomicAdd(w.bins, (unsigned long long)__popc(m_front) | ((unsigned long long)__popc(m_steep) << 32));
  bases = __shfl_sync(0xffffffffu, bases, 0);
  const uint32_t below = (1u << lane) - 1u;
  const uint32_t front = (uint32_t)bases + __popc(m_front & below);
  const uint32_t back = (uint32_t)(bases >> 32) + __popc(m_steep & below);
  const uint32_t slot = (uint32_t)bases + (uint32_t)(bases >> 32) + __popc(m_want & below);
  if (n.want) {
    const uint32_t pix = py * w.width + px;
    float4* sq = reinterpret_cast<float4*>(w.shadow_rays) + 2 * (size_t)slot;
    sq[0] = make_float4(n.org.x, n.org.y, n.org.z, F32_EPSILON);
    sq[1] = make_float4(n.ldir.x, n.ldir.y, n.ldir.z, n.dist);
    const uint32_t bslot = steep ? w.width * w.height - 1u - back : front;
    float4* bq = reinterpret_cast<float4*>(w.bounce_rays) + 2 * (size_t)bslot;
    bq[0] = make_float4(n.org.x, n.org.y, n.org.z, F32_EPSILON);
    bq[1] = make_float4(n.bdir.x, n.bdir.y, n.bdir.z, F32_MAX);
    w.shadow_pixel[slot] = pix;
    w.bounce_pixel[bslot] = pix;
  }
}

// persistent: each warp claims 4x8 pixel tiles from a counter until none is
// left, so that a warp that finishes early does not wait for its block
template <int MODE, bool LOCAL, int TIER, bool WT>
__global__ void __launch_bounds__(128, min_blocks(TIER)) primary_kernel(TraceParams p, WavefrontParams w) {
  extern __shared__ uint2 smem_stack[];
  uint2 local_stack[LOCAL ? kLocalStackEntries : 1];
  uint2* const stack = LOCAL ? local_stack : smem_stack + threadIdx.x;
  const uint32_t stride = LOCAL ? 1u : blockDim.x;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t tiles_x = (w.width + 3u) / 4u;
  const uint32_t tiles = tiles_x * ((w.height + 7u) / 8u);
  for (;;) {
    uint32_t tile = 0;
    if (lane == 0) tile = atomicAdd(w.tile_counter, 1u);
    tile = __shfl_sync(0xffffffffu, tile, 0);
    if (tile >= tiles) break;
    const uint32_t px = (tile % tiles_x) * 4u + (lane & 3u);
    const uint32_t py = (tile / tiles_x) * 8u + (lane >> 2);
    NextRays n;
    n.want = false;
    if (px < w.width && py < w.height) {
      const float3 d = camera_direction(w, px, py);
      RayCtx R;
      primary_ray(w, d, R);
      bool bad;
      traverse_ray<MODE, false, BuiltinAnyHit, WT, 3>(p, R, w.tlas, stack, stride, bad);
      n = shade_primary(p, w, px, py, d, R.best);
    }
    append_rays(w, px, py, n);
  }
}

// The same with four lanes per ray (quad.cuh): a warp claims `batch` pixels of
// a tile. For frames of up to kQuadPixels, whose slowest warps decide (us a
// frame on the 1024^2 field, one ray per lane -> quads: 64^2 pixels 236 -> 110,
// 256^2 393 -> 216, 400^2 464 -> 340, 512^2 482 -> 442, but 640x512 499 -> 525,
// 1280x720 899 -> 1246), and up to quad_limit where the trees are smaller:
// 160,000 primaries of the fields of 16^2, 64^2, 128^2, 256^2 take, of the time
// of two-child lanes, 2.04, 1.64, 1.24 and 0.86 by quads, 0.95, 0.84, 0.74 and
// 0.66 by lanes; their secondary rays 1.50, 1.17, 1.02, 0.96 and 0.93, 0.89,
// 0.83, 0.91. Those of soups, most of whose pixels hit nothing, are fewer and
// take 0.4 to 0.8 by quads, so the secondary rays go by their own number.
constexpr uint32_t kQuadPixelsLeast = 30000, kQuadPixels = 300000;
constexpr float kQuadPrimaries = 155.0f;
constexpr uint32_t kQuadSecondaryLeast = 100000;
constexpr float kQuadSecondary = 410.0f;
template <bool WT>
__global__ void __launch_bounds__(128, 8) primary_quad_kernel(TraceParams p, WavefrontParams w, uint32_t batch) {
  extern __shared__ __align__(16) unsigned char quad_smem[];
  const QuadWarp W = quad_warp(quad_smem, p.stack_depth4);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t tiles_x = (w.width + 3u) / 4u;
  const uint32_t parts = tiles_x * ((w.height + 7u) / 8u) * (32u / batch);
  for (;;) {
    uint32_t part = 0;
    if (lane == 0) part = atomicAdd(w.tile_counter, 1u);
    part = __shfl_sync(0xffffffffu, part, 0);
    if (part >= parts) break;
    const uint32_t at = part * batch + lane, tile = at >> 5, in = at & 31u;
    const uint32_t px = (tile % tiles_x) * 4u + (in & 3u);
    const uint32_t py = (tile / tiles_x) * 8u + (in >> 2);
    const bool valid = lane < batch && px < w.width && py < w.height;
    RayCtx R;
    primary_ray(w, valid ? camera_direction(w, px, py) : make_float3(0.f, 0.f, 0.f), R);
    bool bad;
    traverse_warp<WT>(p, R, w.tlas, valid, W, bad);
    NextRays n;
    n.want = false;
    if (valid) n = shade_primary(p, w, px, py, camera_direction(w, px, py), R.best);
    append_rays(w, px, py, n);
  }
}

// The result of queue entry q to its pixel's record.
__device__ __forceinline__ void store_secondary(const TraceParams& p, const WavefrontParams& w, bool shadow, uint32_t q,
                                                const Best& best) {
  if (shadow) {
    PixelResult* o = w.out + w.shadow_pixel[q];
    o->light = best.have ? 2u : 1u;
    if (best.have) o->direct = 0.0f;
  } else if (best.have) {
    PixelResult* o = w.out + w.bounce_pixel[q];
    const uint4 gm = __ldg(reinterpret_cast<const uint4*>(p.tri_root + best.geom_slot));
    o->bounce_prim = __ldg(p.redirect + best.k) - gm.z;
    o->bounce_t = best.t;
  }
}

template <int MODE, bool LOCAL, int TIER, bool WT>
__global__ void __launch_bounds__(128, min_blocks(TIER)) secondary_kernel(TraceParams p, WavefrontParams w) {
  extern __shared__ uint2 smem_stack[];
  uint2 local_stack[LOCAL ? kLocalStackEntries : 1];
  uint2* const stack = LOCAL ? local_stack : smem_stack + threadIdx.x;
  const uint32_t stride = LOCAL ? 1u : blockDim.x;
  const unsigned long long bins = *(volatile unsigned long long*)w.bins;
  const uint32_t n_front = (uint32_t)bins, n = n_front + (uint32_t)(bins >> 32);
  const uint32_t cap = w.width * w.height;
  const uint32_t total = 2u * n;
  if (w.least_rays && total < w.least_rays) return;
  const uint32_t lane = threadIdx.x & 31u;
  if (blockIdx.x == 0 && threadIdx.x == 0 && w.ray_counts) {
    w.ray_counts[0] = w.width * w.height;
    w.ray_counts[1] = n;
    w.ray_counts[2] = n;
  }
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(w.work_counter, 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= total) break;
    const uint32_t j = base + lane;
    if (j < total) {
      // bounce rays first: they are the longest walks, and a persistent kernel
      // that ends on short shadow rays leaves fewer warps waiting for a last
      // long batch (1.66 -> 1.54 ms on the 1080p frame)
      const bool shadow = j >= n;
      const uint32_t q = shadow ? j - n : bounce_entry(j, n_front, cap);
      const float4* rq = reinterpret_cast<const float4*>(shadow ? w.shadow_rays : w.bounce_rays) + 2 * (size_t)q;
      const float4 r0 = rq[0], r1 = rq[1];
      RayCtx R;
      R.o = make_float3(r0.x, r0.y, r0.z);
      R.tmin = r0.w;
      R.d = make_float3(r1.x, r1.y, r1.z);
      R.tmax = r1.w;
      R.cull_mask = 0xFFu;
      R.ray_flags = shadow ? TF_END_SEARCH : 0u;
      bool bad;
      traverse_ray<MODE, false, BuiltinAnyHit, WT, 3>(p, R, w.tlas, stack, stride, bad);
      store_secondary(p, w, shadow, q, R.best);
    }
  }
}

// The same with four lanes per ray (quad.cuh), a warp as many entries at a
// time as the queues give every resident warp.
template <bool WT, bool LIMIT>
__global__ void __launch_bounds__(128, 8) secondary_quad_kernel(TraceParams p, WavefrontParams w) {
  extern __shared__ __align__(16) unsigned char quad_smem[];
  const QuadWarp W = quad_warp(quad_smem, p.stack_depth4);
  const unsigned long long bins = *(volatile unsigned long long*)w.bins;
  const uint32_t n_front = (uint32_t)bins, n = n_front + (uint32_t)(bins >> 32);
  const uint32_t cap = w.width * w.height;
  const uint32_t total = 2u * n;
  if (LIMIT && total > w.most_rays) return;  // without a limit the first claim does not wait for the count
  // 131,072 rays took 104 us with 8 a warp, 127 with 16 and 152 with 32; 524,288 268, 242 and 230
  const uint32_t batch = total < 200000u ? 8u : (total < 400000u ? 16u : 32u);
  const uint32_t lane = threadIdx.x & 31u;
  if (blockIdx.x == 0 && threadIdx.x == 0 && w.ray_counts) {
    w.ray_counts[0] = w.width * w.height;
    w.ray_counts[1] = n;
    w.ray_counts[2] = n;
  }
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(w.work_counter, batch);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= total) break;
    const uint32_t j = base + lane;
    const bool valid = lane < batch && j < total;
    const bool shadow = j >= n;
    const uint32_t q = shadow ? j - n : bounce_entry(j, n_front, cap);
    RayCtx R;
    if (valid) {
      const float4* rq = reinterpret_cast<const float4*>(shadow ? w.shadow_rays : w.bounce_rays) + 2 * (size_t)q;
      const float4 r0 = rq[0], r1 = rq[1];
      R.o = make_float3(r0.x, r0.y, r0.z);
      R.tmin = r0.w;
      R.d = make_float3(r1.x, r1.y, r1.z);
      R.tmax = r1.w;
    }
    R.cull_mask = 0xFFu;
    R.ray_flags = shadow ? TF_END_SEARCH : 0u;
    bool bad;
    traverse_warp<WT>(p, R, w.tlas, valid, W, bad);
    if (valid) store_secondary(p, w, shadow, q, R.best);
  }
}

// Secondary rays with dynamic fetch (ordered walks only). In the batch
// schedule above a warp takes 32 rays and waits for the slowest of them:
// diffuse bounce rays differ several-fold in work, and most lanes idle while
// the last ray finishes. Here every lane keeps its own resumable traversal
// state (TLAS walk, instance, geometry, BLAS stack). Lanes walk their BLAS in
// the same speculative near-first loop as traverse_ray; a lane that finishes
// leaves the loop, and once at least `w.refill` lanes have left it the others
// pause at the end of their current round so that the warp can claim new queue
// entries for its idle lanes (one atomicAdd) and start them. Per ray the tests
// and their order are traverse_ray's, so every result equals the batch
// schedule's up to the order in which exact-distance ties are met. Iterations
// are capped far above any real traversal; a warp that reaches a cap sets bit
// 2 of the error word and stops.
constexpr uint32_t kMaxWarpIterations = 1u << 24;

template <int MODE, bool WT>
__global__ void __launch_bounds__(128, 8) secondary_dynamic_kernel(TraceParams p, WavefrontParams w) {
  extern __shared__ uint2 smem_stack[];
  constexpr int WIDTH = MODE == MODE_WIDE4 ? 4 : 2;
  const unsigned long long bins = *(volatile unsigned long long*)w.bins;
  const uint32_t n_front = (uint32_t)bins, n = n_front + (uint32_t)(bins >> 32);
  const uint32_t cap = w.width * w.height;
  const uint32_t total = 2u * n;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lanes_below = (1u << lane) - 1u;
  if (blockIdx.x == 0 && threadIdx.x == 0 && w.ray_counts) {
    w.ray_counts[0] = w.width * w.height;
    w.ray_counts[1] = n;
    w.ray_counts[2] = n;
  }
  uint2* stack = smem_stack + threadIdx.x;
  const uint32_t stride = blockDim.x;
  const uint32_t threshold = w.refill < 1u ? 1u : (w.refill > 32u ? 32u : w.refill);
  LaneWalk<WIDTH, WT> L;
  L.reset();
  uint32_t q = 0;
  bool exhausted = false;
  for (uint32_t iter = 0;; iter++) {
    if (iter >= (p.iteration_limit ? p.iteration_limit : kMaxWarpIterations)) {
      if (lane == 0) atomicOr(p.error_word, 4u);
      break;
    }
    // refill idle lanes from the queue
    const uint32_t idle = __ballot_sync(0xffffffffu, L.phase == WALK_IDLE);
    if (!exhausted && (__popc(idle) >= threshold || idle == 0xffffffffu)) {
      const uint32_t cnt = __popc(idle);
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(w.work_counter, cnt);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + cnt >= total) exhausted = true;
      if (L.phase == WALK_IDLE) {
        const uint32_t j = base + __popc(idle & lanes_below);
        if (j < total) {
          q = j;  // bounce rays first, as in the batch schedule
          const bool shadow = j >= n;
          const float4* rq = reinterpret_cast<const float4*>(shadow ? w.shadow_rays : w.bounce_rays) +
                             2 * (size_t)(shadow ? j - n : bounce_entry(j, n_front, cap));
          L.start(p, rq[0], rq[1], w.tlas, shadow ? TF_END_SEARCH : 0u);
        }
      }
    }
    if (exhausted && __ballot_sync(0xffffffffu, L.phase != WALK_IDLE) == 0u) break;
    if (L.phase != WALK_IDLE) L.advance(p, stack, stride, threshold);
    if (L.phase == WALK_DONE) {
      const RayCtx& R = L.R;
      if (q >= n) {
        PixelResult* o = w.out + w.shadow_pixel[q - n];
        o->light = R.best.have ? 2u : 1u;
        if (R.best.have) o->direct = 0.0f;
      } else if (R.best.have) {
        PixelResult* o = w.out + w.bounce_pixel[bounce_entry(q, n_front, cap)];
        const uint4 gm = __ldg(reinterpret_cast<const uint4*>(p.tri_root + R.best.geom_slot));
        o->bounce_prim = __ldg(p.redirect + R.best.k) - gm.z;
        o->bounce_t = R.best.t;
      }
      L.phase = WALK_IDLE;
    }
  }
}

}  // namespace

size_t wavefront_scratch_bytes(uint32_t width, uint32_t height) {
  const size_t n = (size_t)width * height;
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  return 256 + 2 * up(n * 32) + 2 * up(n * 4);
}

void wavefront_bind_scratch(WavefrontParams& w, void* scratch) {
  const size_t n = (size_t)w.width * w.height;
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  char* s = static_cast<char*>(scratch);
  w.queue_count = reinterpret_cast<uint32_t*>(s);
  w.bins = reinterpret_cast<unsigned long long*>(s + 8);
  w.tile_counter = reinterpret_cast<uint32_t*>(s + 16);
  w.work_counter = reinterpret_cast<uint32_t*>(s + 64);
  size_t off = 256;
  w.shadow_rays = s + off;
  off += up(n * 32);
  w.bounce_rays = s + off;
  off += up(n * 32);
  w.shadow_pixel = reinterpret_cast<uint32_t*>(s + off);
  off += up(n * 4);
  w.bounce_pixel = reinterpret_cast<uint32_t*>(s + off);
}

namespace {
template <int MODE, bool LOCAL, int TIER, bool WT>
cudaError_t launch_wavefront_mode(const TraceParams& p, const WavefrontParams& w, uint32_t block, int sm_count,
                                  uint32_t phases, cudaStream_t stream) {
  const size_t smem = MODE != MODE_THREADED && !LOCAL ? (size_t)p.stack_depth * block * sizeof(uint2) : 0;
  static std::atomic<uint64_t> attr_done{0};
  cudaError_t e = raise_smem_limit(
      attr_done, {(const void*)primary_kernel<MODE, LOCAL, TIER, WT>, (const void*)secondary_kernel<MODE, LOCAL, TIER, WT>,
                  (const void*)secondary_dynamic_kernel<MODE_WIDE4, WT>});
  if (e != cudaSuccess) return e;
  if (phases & 1u) {
    e = cudaMemsetAsync(w.queue_count, 0, 64, stream);
    if (e != cudaSuccess) return e;
    // persistent primary grid: as many resident blocks as fill every SM, or
    // fewer when the frame has fewer 4x8 tiles than resident warps
    int per_sm1 = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm1, primary_kernel<MODE, LOCAL, TIER, WT>, (int)block, smem);
    if (e != cudaSuccess) return e;
    if (per_sm1 < 1) per_sm1 = 1;
    const uint64_t tiles = (uint64_t)((w.width + 3) / 4) * ((w.height + 7) / 8);
    const uint64_t need = (tiles * 32 + block - 1) / block;
    const uint32_t grid1 = (uint32_t)std::min<uint64_t>((uint64_t)sm_count * per_sm1, need);
    primary_kernel<MODE, LOCAL, TIER, WT><<<grid1, block, smem, stream>>>(p, w);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (!(phases & 2u)) return cudaSuccess;
  if (w.least_rays == 0u) {  // else the quads' launch before this one has zeroed it, and has not used it if this one runs
    e = cudaMemsetAsync(w.work_counter, 0, 64, stream);
    if (e != cudaSuccess) return e;
  }
  // persistent secondary grid: enough resident blocks to fill every SM
  const bool dynamic = MODE != MODE_THREADED && w.refill != 0u && !LOCAL;
  int per_sm = 0;
  constexpr int DMODE = MODE_WIDE4;  // the threaded walk has no dynamic form
  if (dynamic)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, secondary_dynamic_kernel<DMODE, WT>, (int)block, smem);
  else
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, secondary_kernel<MODE, LOCAL, TIER, WT>, (int)block, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  const uint32_t grid2 = (uint32_t)(sm_count * per_sm);
  if (dynamic) secondary_dynamic_kernel<DMODE, WT><<<grid2, block, smem, stream>>>(p, w);
  else secondary_kernel<MODE, LOCAL, TIER, WT><<<grid2, block, smem, stream>>>(p, w);
  return cudaGetLastError();
}
}  // namespace

namespace {
template <bool WT>
cudaError_t launch_wavefront_quads(const TraceParams& p, const WavefrontParams& w, int sm_count, uint32_t phases,
                                   cudaStream_t stream) {
  constexpr uint32_t block = 64;
  const size_t smem = (size_t)quad_warp_bytes(p.stack_depth4) * (block / 32);
  static std::atomic<uint64_t> attr_done{0};
  const auto secondary = w.most_rays ? secondary_quad_kernel<WT, true> : secondary_quad_kernel<WT, false>;
  cudaError_t e = raise_smem_limit(attr_done, {(const void*)primary_quad_kernel<WT>, (const void*)secondary_quad_kernel<WT, true>,
                                               (const void*)secondary_quad_kernel<WT, false>});
  if (e != cudaSuccess) return e;
  const uint64_t pixels = (uint64_t)((w.width + 3) / 4) * ((w.height + 7) / 8) * 32;
  // persistent grids: as many resident blocks as fill every SM, or fewer when the rays are
  auto grid = [&](const void* fn, uint64_t rays, uint32_t batch, uint32_t& blocks) {
    int per_sm = 0;
    const cudaError_t r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, (int)block, smem);
    const uint64_t per = batch * (block / 32);
    blocks = (uint32_t)std::min<uint64_t>((uint64_t)sm_count * std::max(per_sm, 1), (rays + per - 1) / per);
    return r;
  };
  uint32_t blocks = 0;
  if (phases & 1u) {
    const uint32_t batch = pixels < 100000 ? 8u : 16u;
    e = cudaMemsetAsync(w.queue_count, 0, 64, stream);
    if (e == cudaSuccess) e = grid((const void*)primary_quad_kernel<WT>, pixels, batch, blocks);
    if (e != cudaSuccess) return e;
    primary_quad_kernel<WT><<<blocks, block, smem, stream>>>(p, w, batch);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (!(phases & 2u)) return cudaSuccess;
  e = cudaMemsetAsync(w.work_counter, 0, 64, stream);
  if (e == cudaSuccess) e = grid((const void*)secondary, 2 * pixels, 8u, blocks);
  if (e != cudaSuccess) return e;
  secondary<<<blocks, block, smem, stream>>>(p, w);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_wavefront(const TraceParams& params, const WavefrontParams& w, int mode, uint32_t block,
                             int sm_count, uint32_t phases, cudaStream_t stream) {
  if (phases == 0) phases = 3;
  if (block == 0) block = 64;
  const size_t n = (size_t)w.width * w.height;
  if (n == 0) return cudaSuccess;
#define RDN_WF(M, L, T)                                                                      \
  return p.watertight ? launch_wavefront_mode<M, L, T, true>(p, v, block, sm_count, phases, stream) \
                      : launch_wavefront_mode<M, L, T, false>(p, v, block, sm_count, phases, stream)
  WavefrontParams v = w;
  v.least_rays = v.most_rays = 0u;
  if (mode == MODE_THREADED) {
    const TraceParams& p = params;
    RDN_WF(MODE_THREADED, false, 0);
  }
  const TraceParams p = wide4_params(params);
  // dynamic fetch (w.refill) has its own secondary kernel, with stacks in shared memory
  const bool dynamic = w.refill != 0u && !(w.local_stack && p.local_stack);
  // Primaries by quads in small frames.
  const bool quads_ok = p.packed && !dynamic;
  const bool quads1 = quads_ok && n <= quad_limit(p, kQuadPrimaries, kQuadPixelsLeast, kQuadPixels);
  // Secondary rays by quads up to a number of rays that only the device knows: where the pixels leave it open both
  // kernels are launched, and one of them returns at once. Those of an instanced structure always, since one per lane
  // the lanes part at the first of a ray's BLASes (us, secondary rays of 640x480 and 1920x1080 pixels, lanes / quads: 512
  // instances of 300 triangles 900, 1130 / 178, 303; 64 of 5,000 1040, 1620 / 271, 638; 216 of 6 x 100 2260, 2640 /
  // 416, 925; the primaries are alike: 300, 500 / 525, 1450).
  const uint32_t limit2 = quad_limit(p, kQuadSecondary, kQuadSecondaryLeast, 2u * kQuadPixels);
  const bool quads2 = quads_ok && (p.instanced || n <= kQuadPixels);
  const bool open2 = quads2 && !p.instanced && 2 * n > limit2;
  const auto quads = [&](uint32_t phases) {
    return p.watertight ? launch_wavefront_quads<true>(p, v, sm_count, phases, stream)
                        : launch_wavefront_quads<false>(p, v, sm_count, phases, stream);
  };
  const auto lanes = [&](uint32_t phases) -> cudaError_t {
    if (!p.local_stack || dynamic) RDN_WF(MODE_WIDE4, false, 0);
    // register tiers apply to the local-stack kernels
    if (w.register_tier == 1) RDN_WF(MODE_WIDE4, true, 1);
    if (w.register_tier == 2) RDN_WF(MODE_WIDE4, true, 2);
    RDN_WF(MODE_WIDE4, true, 0);
  };
  cudaError_t e = cudaSuccess;
  if (phases & 1u) e = quads1 ? quads(1u) : lanes(1u);
  if (e != cudaSuccess || !(phases & 2u)) return e;
  if (open2) v.most_rays = limit2;
  if (quads2) e = quads(2u);
  if (e != cudaSuccess || (quads2 && !open2)) return e;
  if (open2) v.least_rays = limit2 + 1u;
  return lanes(2u);
#undef RDN_WF
}

}  // namespace rdn
