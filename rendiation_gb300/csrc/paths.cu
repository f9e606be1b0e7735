// Batched multi-scene path tracing, sm_103a.
//
// The reference's path tracer (scene/rendering/gpu-ray-tracing/src/feature/path_tracing/
// ray_gen.rs:89-211, ray_hit.rs:12-103) loops up to max_path_depth bounces per
// pixel through the task graph, one wavefront round per bounce. Here every ray
// of every scene goes through one persistent launch per bounce:
//
//   path_kernel: warps fetch 32 queue entries at a time from a global work
//   counter (load balance across scenes of very different size and across
//   paths of different length); each entry is a 32 B ray plus a 16 B path
//   state {output id, TLAS index, throughput, flags}. Closest hit in the
//   entry's own scene (the reference's per-ray tlas_idx, traverse_cpu.rs:63),
//   then one cosine-weighted diffuse bounce from an offset_ray_hit origin,
//   Russian roulette from the configured bounce on, and a warp-ballot /
//   one-atomic-per-warp append of the surviving path to the next queue.
//
// Path semantics (shared with the oracle): albedo a; a miss at bounce k
// writes radiance = throughput (sky = 1) and depth k; a hit at k == max_bounces
// or a path killed by roulette writes radiance 0. The sampler for bounce k of
// path i is xxhash32(i, k, seed) -> next() x3 (direction, roulette).
// Built with -fmad=false, like every traversal unit.
#include <cuda_runtime.h>

#include <cstdint>

#include "parallel.h"
#include "paths.h"
#include "quad.cuh"
#include "shade.cuh"
#include "traverse.cuh"

namespace rdn {
namespace {

using namespace dev;

struct PathRay {
  float4 r0, r1;
  uint32_t id, tlas;
  float throughput;
};

// Entry j of a bounce's queue: rays (2 float4) and states {id, tlas,
// throughput, 0}. from_user: bounce 0 reads the caller's primary rays instead.
__device__ __forceinline__ PathRay load_path(const PathParams& q, bool from_user, const float4* __restrict__ in_rays,
                                             const uint4* __restrict__ in_state, uint32_t j) {
  PathRay e;
  if (from_user) {
    const float4* rp = q.primary_rays + 2 * (size_t)j;
    e.r0 = __ldg(rp);
    e.r1 = __ldg(rp + 1);
    e.id = j;
    e.tlas = q.tlas_idx ? __ldg(q.tlas_idx + j) : q.tlas_uniform;
    e.throughput = 1.0f;
  } else {
    e.r0 = in_rays[2 * (size_t)j];
    e.r1 = in_rays[2 * (size_t)j + 1];
    const uint4 s = in_state[j];
    e.id = s.x;
    e.tlas = s.y;
    e.throughput = __uint_as_float(s.z);
  }
  return e;
}

// Ends or continues a path after its query; true when it goes on, with its
// next queue entry in (nr0, nr1, ns).
__device__ __forceinline__ bool shade_path(const TraceParams& p, const PathParams& q, uint32_t bounce, uint32_t id,
                                           uint32_t tlas, float throughput, float3 o, float3 d, const Best& best,
                                           float4& nr0, float4& nr1, uint4& ns) {
  if (!best.have) {
    q.out[id] = make_float2(throughput, __uint_as_float(bounce | RDN_PATH_ESCAPED));
    return false;
  }
  if (bounce == q.max_bounces) {
    q.out[id] = make_float2(0.0f, __uint_as_float(bounce));
    return false;
  }
  uint32_t st = xxhash32(id, bounce, q.seed);
  const float s0 = sample_next(st);
  const float s1 = sample_next(st);
  const float s2 = sample_next(st);
  float t_next = throughput * q.albedo;
  bool survive = true;
  if (bounce + 1 >= q.rr_start) {
    survive = s2 < q.rr_survive;
    t_next = t_next / q.rr_survive;
  }
  if (!survive) {
    q.out[id] = make_float2(0.0f, __uint_as_float(bounce | RDN_PATH_ROULETTE));
    return false;
  }
  const float3 hp = o + d * best.t;
  const float3 nf = facing_normal(p, best.k, best.inst, d);
  const float3 org = offset_ray_hit(hp, nf);
  const float3 dir = cosine_sample_in_dir(nf, s0, s1);
  nr0 = make_float4(org.x, org.y, org.z, 1.1920929e-7f);
  nr1 = make_float4(dir.x, dir.y, dir.z, 3.40282347e+38f);
  ns = make_uint4(id, tlas, __float_as_uint(t_next), 0u);
  return true;
}

// One bounce, a ray per lane: the reference order, and structures too large
// for packed_leaf.
template <int MODE, bool LOCAL, bool WT>
__global__ void __launch_bounds__(128) path_kernel(TraceParams p, PathParams q, uint32_t bounce, bool from_user,
                                                   const float4* __restrict__ in_rays,
                                                   const uint4* __restrict__ in_state, float4* __restrict__ out_rays,
                                                   uint4* __restrict__ out_state) {
  RDN_TRAVERSAL_STACK(LOCAL);
  const uint32_t n = bounce == 0 ? q.count : *(volatile uint32_t*)(q.queue_count + bounce - 1);
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t* work = q.work_counter + bounce;
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(work, 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n) break;
    const uint32_t j = base + lane;
    bool keep = false;
    float4 nr0 = make_float4(0.f, 0.f, 0.f, 0.f), nr1 = nr0;
    uint4 ns = make_uint4(0u, 0u, 0u, 0u);
    if (j < n) {
      const PathRay e = load_path(q, from_user, in_rays, in_state, j);
      RayCtx R;
      R.o = make_float3(e.r0.x, e.r0.y, e.r0.z);
      R.tmin = e.r0.w;
      R.d = make_float3(e.r1.x, e.r1.y, e.r1.z);
      R.tmax = e.r1.w;
      R.cull_mask = 0xFFu;
      R.ray_flags = 0u;
      bool bad;
      traverse_ray<MODE, false, BuiltinAnyHit, WT>(p, R, e.tlas, stack_ptr, stack_stride, bad);
      keep = shade_path(p, q, bounce, e.id, e.tlas, e.throughput, R.o, R.d, R.best, nr0, nr1, ns);
    }
    const uint32_t slot = warp_append(q.queue_count + bounce, keep);
    if (keep) {
      out_rays[2 * (size_t)slot] = nr0;
      out_rays[2 * (size_t)slot + 1] = nr1;
      out_state[slot] = ns;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && q.segment_counts) q.segment_counts[bounce] = n;
}

// Bounce 0 of large calls: a group of 32 primaries that are alike walks faster a
// ray per lane. A look at 128 groups, path_vote_kernel, says whether most are;
// if so path_alike_kernel goes through all, takes those that are and lists the
// others for the quads, and leaves the quads' usual launch nothing; else that
// takes all. (Both kernels over all groups, each with its own vote, cost the
// calls without alike rays 5 % of bounce 0; the quads' loop with a look at the
// list 0.6 %.)
// 2.07 M camera rays onto the 1024^2 field, no bounce: two-child lanes 787 us, all
// by quads 944, here 615; onto that of 64^2, up to two bounces: 1152, 1356, 1061.
// As many random rays: 592 and 717 by quads, 602 and 725 here.
enum { SPLIT_MOST_ALIKE = 0, SPLIT_LISTED = 1, SPLIT_CLAIMED = 2, SPLIT_TAKEN = 3 };  // words of PathParams::split

__device__ __forceinline__ void path_ray(const PathRay& e, RayCtx& R) {
  R.o = make_float3(e.r0.x, e.r0.y, e.r0.z);
  R.tmin = e.r0.w;
  R.d = make_float3(e.r1.x, e.r1.y, e.r1.z);
  R.tmax = e.r1.w;
  R.cull_mask = 0xFFu;
  R.ray_flags = 0u;
}

constexpr uint32_t kVoteThreads = 1024, kVotes = 4;
__global__ void __launch_bounds__(kVoteThreads) path_vote_kernel(PathParams q, bool from_user,
                                                                 const float4* __restrict__ in_rays,
                                                                 const uint4* __restrict__ in_state) {
  __shared__ uint32_t alike;
  if (threadIdx.x == 0) alike = 0u;
  __syncthreads();
  constexpr uint32_t samples = kVoteThreads / 32u * kVotes;
  const uint32_t groups = (uint32_t)(((uint64_t)q.count + 31u) / 32u);
  PathRay e[kVotes];
#pragma unroll
  for (uint32_t k = 0; k < kVotes; k++) {
    const uint32_t s = (threadIdx.x >> 5) * kVotes + k;
    const uint32_t j = (uint32_t)((uint64_t)s * groups / samples) * 32u + (threadIdx.x & 31u);
    e[k] = load_path(q, from_user, in_rays, in_state, j < q.count ? j : q.count - 1u);
  }
  uint32_t mine = 0;
#pragma unroll
  for (uint32_t k = 0; k < kVotes; k++) {
    RayCtx R;
    path_ray(e[k], R);
    mine += coherent_warp(R, e[k].tlas, true);
  }
  if ((threadIdx.x & 31u) == 0) atomicAdd(&alike, mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    const bool most = 2u * alike >= samples;
    q.split[SPLIT_MOST_ALIKE] = most;
    q.split[SPLIT_LISTED] = q.split[SPLIT_CLAIMED] = q.split[SPLIT_TAKEN] = 0u;
    if (most) q.work_counter[0] = q.count;  // all claimed: bounce 0 is path_alike_kernel's and the list's
  }
}

template <bool WT>
__global__ void __launch_bounds__(128) path_alike_kernel(TraceParams p, PathParams q, bool from_user,
                                                         const float4* __restrict__ in_rays,
                                                         const uint4* __restrict__ in_state,
                                                         float4* __restrict__ out_rays, uint4* __restrict__ out_state) {
  uint2 stack[kLocalStackEntries];
  if (!q.split[SPLIT_MOST_ALIKE]) return;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t groups = (uint32_t)(((uint64_t)q.count + 31u) / 32u);
  for (;;) {
    uint32_t g = 0;
    if (lane == 0) g = atomicAdd(q.split + SPLIT_CLAIMED, 1u);
    g = __shfl_sync(0xffffffffu, g, 0);
    if (g >= groups) break;
    const uint32_t j = g * 32u + lane;
    const bool valid = j < q.count;
    PathRay e{};
    if (valid) e = load_path(q, from_user, in_rays, in_state, j);
    RayCtx R;
    path_ray(e, R);
    if (!coherent_warp(R, e.tlas, valid)) {
      if (lane == 0) q.split_list[atomicAdd(q.split + SPLIT_LISTED, 1u)] = g;
      continue;
    }
    bool keep = false;
    float4 nr0 = make_float4(0.f, 0.f, 0.f, 0.f), nr1 = nr0;
    uint4 ns = make_uint4(0u, 0u, 0u, 0u);
    if (valid) {
      bool bad;
      traverse_ray<MODE_WIDE4, false, BuiltinAnyHit, WT, 2, WT>(p, R, e.tlas, stack, 1u, bad);
      keep = shade_path(p, q, 0u, e.id, e.tlas, e.throughput, R.o, R.d, R.best, nr0, nr1, ns);
    }
    const uint32_t slot = warp_append(q.queue_count, keep);
    if (keep) {
      out_rays[2 * (size_t)slot] = nr0;
      out_rays[2 * (size_t)slot + 1] = nr1;
      out_state[slot] = ns;
    }
  }
}

// One bounce with four lanes per ray (quad.cuh): the ordered walks. A warp
// claims 32 queue entries, or fewer of a queue that would not give every
// resident warp 32. The entry is read again for the shading, so that the walk
// holds no more than its ray. The rays of a bounce differ in scene and
// direction, the case the quads are for: 64 soups (2.4 M triangles, 3.7 M
// primaries, up to 4 bounces) 10151 us one ray per lane on two-child nodes,
// 5515 with quads; blocks of 32, 64 or 128 threads within 0.4 %.
// LISTED: bounce 0 of the groups that path_alike_kernel has listed.
template <bool WT, bool LISTED>
__global__ void __launch_bounds__(128, 8) path_quad_kernel(TraceParams p, PathParams q, uint32_t bounce, bool from_user,
                                                           const float4* __restrict__ in_rays,
                                                           const uint4* __restrict__ in_state,
                                                           float4* __restrict__ out_rays,
                                                           uint4* __restrict__ out_state) {
  extern __shared__ __align__(16) unsigned char quad_smem[];
  const uint32_t n = bounce == 0 ? q.count : *(volatile uint32_t*)(q.queue_count + bounce - 1);
  const uint32_t lane = threadIdx.x & 31u;
  if (LISTED && !q.split[SPLIT_MOST_ALIKE]) return;
  const uint32_t batch = LISTED ? 32u : quad_batch(n), end = LISTED ? 32u * q.split[SPLIT_LISTED] : n;
  uint32_t* work = LISTED ? q.split + SPLIT_TAKEN : q.work_counter + bounce;
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(work, batch);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= end) break;
    if (LISTED) base = 32u * q.split_list[base >> 5];
    const uint32_t j = base + lane;
    const bool valid = lane < batch && j < n;
    RayCtx R;
    uint32_t tlas = 0;
    if (valid) {
      const PathRay e = load_path(q, from_user, in_rays, in_state, j);
      R.o = make_float3(e.r0.x, e.r0.y, e.r0.z);
      R.tmin = e.r0.w;
      R.d = make_float3(e.r1.x, e.r1.y, e.r1.z);
      R.tmax = e.r1.w;
      tlas = e.tlas;
    }
    R.cull_mask = 0xFFu;
    R.ray_flags = 0u;
    bool bad;
    traverse_warp<WT>(p, R, tlas, valid, quad_warp(quad_smem, p.stack_depth4), bad);
    bool keep = false;
    float4 nr0 = make_float4(0.f, 0.f, 0.f, 0.f), nr1 = nr0;
    uint4 ns = make_uint4(0u, 0u, 0u, 0u);
    if (valid) {
      const PathRay e = load_path(q, from_user, in_rays, in_state, j);
      keep = shade_path(p, q, bounce, e.id, e.tlas, e.throughput, make_float3(e.r0.x, e.r0.y, e.r0.z),
                        make_float3(e.r1.x, e.r1.y, e.r1.z), R.best, nr0, nr1, ns);
    }
    const uint32_t slot = warp_append(q.queue_count + bounce, keep);
    if (keep) {
      out_rays[2 * (size_t)slot] = nr0;
      out_rays[2 * (size_t)slot + 1] = nr1;
      out_state[slot] = ns;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && q.segment_counts) q.segment_counts[bounce] = n;
}

// The same bounce with dynamic fetch (ordered walks only, q.refill > 0): every
// lane keeps its own resumable query (LaneWalk) and the warp claims new queue
// entries for its idle lanes whenever at least q.refill of them are idle, so
// that a few long paths do not hold a whole warp. Rays of different scenes and
// directions are mixed anyway, so no coherence is lost by refilling. The
// shading and the warp-aggregated append run for the lanes that finished in
// the round; iterations are capped (error-word bit 2).
template <int MODE, bool WT>
__global__ void __launch_bounds__(128, 8) path_dynamic_kernel(TraceParams p, PathParams q, uint32_t bounce,
                                                              bool from_user, const float4* __restrict__ in_rays,
                                                              const uint4* __restrict__ in_state,
                                                              float4* __restrict__ out_rays,
                                                              uint4* __restrict__ out_state) {
  extern __shared__ uint2 smem_stack[];
  constexpr int WIDTH = MODE == MODE_WIDE4 ? 4 : 2;
  const uint32_t n = bounce == 0 ? q.count : *(volatile uint32_t*)(q.queue_count + bounce - 1);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lanes_below = (1u << lane) - 1u;
  uint32_t* work = q.work_counter + bounce;
  uint2* stack = smem_stack + threadIdx.x;
  const uint32_t threshold = q.refill < 1u ? 1u : (q.refill > 32u ? 32u : q.refill);
  LaneWalk<WIDTH, WT> L;
  L.reset();
  uint32_t id = 0, tlas = 0;
  float throughput = 0.0f;
  bool exhausted = false;
  for (uint32_t iter = 0;; iter++) {
    if (iter >= walk_round_cap(p)) {
      if (lane == 0) atomicOr(p.error_word, 4u);
      break;
    }
    const uint32_t idle = __ballot_sync(0xffffffffu, L.phase == WALK_IDLE);
    if (!exhausted && (__popc(idle) >= threshold || idle == 0xffffffffu)) {
      const uint32_t cnt = __popc(idle);
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(work, cnt);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + cnt >= n) exhausted = true;
      if (L.phase == WALK_IDLE) {
        const uint32_t j = base + __popc(idle & lanes_below);
        if (j < n) {
          const PathRay e = load_path(q, from_user, in_rays, in_state, j);
          id = e.id;
          tlas = e.tlas;
          throughput = e.throughput;
          L.start(p, e.r0, e.r1, tlas, 0u);
        }
      }
    }
    if (exhausted && __ballot_sync(0xffffffffu, L.phase != WALK_IDLE) == 0u) break;
    if (L.phase != WALK_IDLE) L.advance(p, stack, blockDim.x, threshold);
    bool keep = false;
    float4 nr0 = make_float4(0.f, 0.f, 0.f, 0.f), nr1 = nr0;
    uint4 ns = make_uint4(0u, 0u, 0u, 0u);
    if (L.phase == WALK_DONE) {
      keep = shade_path(p, q, bounce, id, tlas, throughput, L.R.o, L.R.d, L.R.best, nr0, nr1, ns);
      L.phase = WALK_IDLE;
    }
    const uint32_t slot = warp_append(q.queue_count + bounce, keep);
    if (keep) {
      out_rays[2 * (size_t)slot] = nr0;
      out_rays[2 * (size_t)slot + 1] = nr1;
      out_state[slot] = ns;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && q.segment_counts) q.segment_counts[bounce] = n;
}

// Primary rays into queue form (only when the executor sorts rays).
__global__ void path_prime_kernel(PathParams q, float4* __restrict__ rays, uint4* __restrict__ state) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= q.count) return;
  rays[2 * (size_t)i] = __ldg(q.primary_rays + 2 * (size_t)i);
  rays[2 * (size_t)i + 1] = __ldg(q.primary_rays + 2 * (size_t)i + 1);
  state[i] = make_uint4(i, q.tlas_idx ? __ldg(q.tlas_idx + i) : q.tlas_uniform, __float_as_uint(1.0f), 0u);
}

__device__ __forceinline__ uint32_t spread4(uint32_t v) {  // 4 bits -> every third bit
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}

// Sort key of queue entry i (entries at or past the live count are skipped).
__global__ void path_key_kernel(TraceParams p, PathParams q, const float4* __restrict__ rays,
                                const uint4* __restrict__ state, const uint32_t* __restrict__ n_dev) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t n = n_dev ? *n_dev : q.count;
  if (i >= n) return;
  const float4 r0 = rays[2 * (size_t)i], r1 = rays[2 * (size_t)i + 1];
  const uint32_t tlas = state[i].y;
  const uint32_t oct = (r1.x < 0.0f ? 1u : 0u) | (r1.y < 0.0f ? 2u : 0u) | (r1.z < 0.0f ? 4u : 0u);
  uint32_t key = (tlas << 3) | oct;
  if (q.sort_key == 2) {
    uint32_t cell = 0;
    if (tlas < p.n_binding) {
      const uint32_t h = __ldg(p.tlas_binding + tlas);
      const uint32_t root = h < p.n_tlas_root ? __ldg(p.tlas_bvh_root + h) : INVALID_NEXT;
      if (root != INVALID_NEXT) {
        const float* b = reinterpret_cast<const float*>(p.tlas_forest + root);
        const float lo[3] = {__ldg(b), __ldg(b + 1), __ldg(b + 2)}, hi[3] = {__ldg(b + 4), __ldg(b + 5), __ldg(b + 6)};
        const float o[3] = {r0.x, r0.y, r0.z};
        uint32_t c[3];
        for (int a = 0; a < 3; a++) {
          const float ext = hi[a] - lo[a];
          const float f = ext > 0.0f ? (o[a] - lo[a]) / ext * 16.0f : 0.0f;
          c[a] = f <= 0.0f ? 0u : (f >= 15.0f ? 15u : (uint32_t)f);
        }
        cell = spread4(c[0]) | (spread4(c[1]) << 1) | (spread4(c[2]) << 2);
      }
    }
    key = (key << 12) | cell;
  }
  q.keys[i] = key;
  q.idx[i] = i;
}

__global__ void path_gather_kernel(PathParams q, const float4* __restrict__ in_rays, const uint4* __restrict__ in_state,
                                   float4* __restrict__ out_rays, uint4* __restrict__ out_state,
                                   const uint32_t* __restrict__ n_dev) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t n = n_dev ? *n_dev : q.count;
  if (i >= n) return;
  const uint32_t j = q.idx[i];
  out_rays[2 * (size_t)i] = in_rays[2 * (size_t)j];
  out_rays[2 * (size_t)i + 1] = in_rays[2 * (size_t)j + 1];
  out_state[i] = in_state[j];
}

}  // namespace

size_t paths_scratch_bytes(uint32_t count, uint32_t max_bounces, uint32_t sort_key) {
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t n = count;
  size_t bytes = 256 + up(sizeof(uint32_t) * 2 * (max_bounces + 1)) + 2 * up(n * 32) + 2 * up(n * 16);
  if (sort_key) bytes += 2 * up(n * 4) + sort_scratch_bytes(count);
  return bytes;
}

void paths_bind_scratch(PathParams& q, void* scratch) {
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t n = q.count;
  char* s = static_cast<char*>(scratch);
  q.queue_count = reinterpret_cast<uint32_t*>(s + 256);
  q.work_counter = q.queue_count + (q.max_bounces + 1);
  size_t off = 256 + up(sizeof(uint32_t) * 2 * (q.max_bounces + 1));
  q.rays_a = s + off;
  off += up(n * 32);
  q.rays_b = s + off;
  off += up(n * 32);
  q.state_a = s + off;
  off += up(n * 16);
  q.state_b = s + off;
  off += up(n * 16);
  // the words before the queue counts; the list in an array that is free when bounce 0 runs
  q.split = reinterpret_cast<uint32_t*>(s);
  q.split_list = static_cast<uint32_t*>(q.rays_a);
  if (q.sort_key) {
    q.keys = reinterpret_cast<uint32_t*>(s + off);
    off += up(n * 4);
    q.idx = reinterpret_cast<uint32_t*>(s + off);
    off += up(n * 4);
    q.sort_scratch = s + off;
    q.split_list = q.keys;
  }
}

namespace {
// kernel variant: a ray per lane (stacks in shared or local memory), dynamic
// fetch, four lanes per ray, and the same with alike primaries a ray per lane
enum PathVariant { PATH_LANES = 0, PATH_DYNAMIC = 1, PATH_QUADS = 2, PATH_LOCAL_LANES = 3, PATH_SPLIT = 4 };
// Primaries from which a call is large (see quad_limit). Small trees go by lanes
// in every bounce then (two bounces on the field of 16^2, us, quads / lanes /
// two-child lanes: 160,000 camera primaries 133 / 99 / 108, random ones 98 / 117 /
// 123; 2.07 M 965 / 533 / 614, 535 / 467 / 544; 65,536 85 / 85 / 89, 71 / 87 / 94).
constexpr uint32_t kSplitLeast = 100000, kSplitMost = 400000;
constexpr float kSplitRays = 260.0f;
int path_variant(int mode, const TraceParams& p, const PathParams& q) {
  if (mode == MODE_THREADED) return PATH_LANES;
  if (q.refill != 0) return PATH_DYNAMIC;
  if (!p.packed) return PATH_LANES;
  if (!wide4_params(p).local_stack || q.count < quad_limit(p, kSplitRays, kSplitLeast, kSplitMost)) return PATH_QUADS;
  return small_trees(p) ? PATH_LOCAL_LANES : PATH_SPLIT;
}
// shared memory of a block: the variant's stacks
size_t path_smem(int mode, int variant, const TraceParams& p, uint32_t block) {
  if (variant == PATH_QUADS || variant == PATH_SPLIT) return (size_t)quad_warp_bytes(p.stack_depth4) * (block / 32);
  if (variant == PATH_LOCAL_LANES) return 0;
  return mode == MODE_THREADED ? 0 : (size_t)p.stack_depth4 * block * sizeof(uint2);
}
using PathKernel = void (*)(TraceParams, PathParams, uint32_t, bool, const float4*, const uint4*, float4*, uint4*);
template <bool WT>
PathKernel path_fn_wt(int mode, int variant) {
  if (mode == MODE_THREADED) return path_kernel<MODE_THREADED, false, WT>;
  if (variant == PATH_QUADS || variant == PATH_SPLIT) return path_quad_kernel<WT, false>;
  if (variant == PATH_LOCAL_LANES) return path_kernel<MODE_WIDE4, true, WT>;
  return variant == PATH_DYNAMIC ? path_dynamic_kernel<MODE_WIDE4, WT> : path_kernel<MODE_WIDE4, false, WT>;
}
PathKernel path_fn(int mode, int variant, bool wt) {
  return wt ? path_fn_wt<true>(mode, variant) : path_fn_wt<false>(mode, variant);
}
}  // namespace

cudaError_t prepare_paths(const TraceParams& p, const PathParams& q, int mode, uint32_t block, int sm_count,
                          uint32_t* grid) {
  if (block == 0) block = 64;
  const int variant = path_variant(mode, p, q);
  const size_t smem = path_smem(mode, variant, p, block);
  static std::atomic<uint64_t> attr_done[2][5][3] = {}, split_done{0};
  const void* fn = (const void*)path_fn(mode, variant, p.watertight != 0);
  cudaError_t e = raise_smem_limit(attr_done[p.watertight ? 1 : 0][variant][mode], {fn});
  if (e != cudaSuccess) return e;
  if (variant == PATH_SPLIT)
    e = raise_smem_limit(split_done, {(const void*)path_quad_kernel<false, true>, (const void*)path_quad_kernel<true, true>});
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, (int)block, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  // persistent grid, never larger than the primary queue needs
  uint32_t g = (uint32_t)(sm_count * per_sm);
  const uint32_t per = variant == PATH_QUADS || variant == PATH_SPLIT ? quad_batch(q.count) * (block / 32) : block;  // rays a block takes at a time
  const uint32_t need = (q.count + per - 1) / per;
  *grid = g > need ? need : g;
  return cudaSuccess;
}

cudaError_t record_paths(const TraceParams& p, const PathParams& q, int mode, uint32_t block, uint32_t grid,
                         cudaStream_t stream) {
  if (block == 0) block = 64;
  if (q.count == 0 || grid == 0) return cudaSuccess;
  const int variant = path_variant(mode, p, q);
  const size_t smem = path_smem(mode, variant, p, block);
  const PathKernel fn = path_fn(mode, variant, p.watertight != 0);
  const TraceParams walk = mode == MODE_THREADED ? p : wide4_params(p);
  cudaError_t e = cudaMemsetAsync(q.queue_count, 0, sizeof(uint32_t) * 2 * (q.max_bounces + 1), stream);
  if (e != cudaSuccess) return e;
  float4* ra = static_cast<float4*>(q.rays_a);
  float4* rb = static_cast<float4*>(q.rays_b);
  uint4* sa = static_cast<uint4*>(q.state_a);
  uint4* sb = static_cast<uint4*>(q.state_b);
  const uint32_t eg = (q.count + 255) / 256;
  if (q.sort_key) {
    path_prime_kernel<<<eg, 256, 0, stream>>>(q, ra, sa);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  for (uint32_t b = 0; b <= q.max_bounces; b++) {
    const float4* in_r;
    const uint4* in_s;
    float4* out_r;
    uint4* out_s;
    bool from_user = false;
    if (q.sort_key) {
      // regroup the queue in A by key into B, trace B, append to A
      const uint32_t* n_dev = b == 0 ? nullptr : q.queue_count + b - 1;
      path_key_kernel<<<eg, 256, 0, stream>>>(p, q, ra, sa, n_dev);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = radix_sort_u32(q.keys, q.idx, q.count, q.key_bits, q.sort_scratch, stream, n_dev);
      if (e != cudaSuccess) return e;
      path_gather_kernel<<<eg, 256, 0, stream>>>(q, ra, sa, rb, sb, n_dev);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      in_r = rb;
      in_s = sb;
      out_r = ra;
      out_s = sa;
    } else {
      from_user = b == 0;
      in_r = (b & 1) ? rb : ra;
      in_s = (b & 1) ? sb : sa;
      out_r = (b & 1) ? ra : rb;
      out_s = (b & 1) ? sa : sb;
    }
    if (variant == PATH_SPLIT && b == 0) {
      path_vote_kernel<<<1, kVoteThreads, 0, stream>>>(q, from_user, in_r, in_s);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      const auto alike = p.watertight ? path_alike_kernel<true> : path_alike_kernel<false>;
      alike<<<grid, block, 0, stream>>>(walk, q, from_user, in_r, in_s, out_r, out_s);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      const PathKernel listed = p.watertight ? path_quad_kernel<true, true> : path_quad_kernel<false, true>;
      listed<<<grid, block, smem, stream>>>(walk, q, b, from_user, in_r, in_s, out_r, out_s);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    fn<<<grid, block, smem, stream>>>(walk, q, b, from_user, in_r, in_s, out_r, out_s);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace rdn
