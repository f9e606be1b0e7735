// Batch ray-query kernels for sm_103a (rdn_trace), one 16 B hit (+ optional
// 16 B context) out per ray: one thread per ray with the traversal of
// traverse.cuh, or four lanes per ray with that of quad.cuh.
// Built with -fmad=false: see traverse.cuh.
#include <cuda_runtime.h>

#include <cstdint>

#include "quad.cuh"
#include "traverse.cuh"

namespace rdn {
namespace {

using namespace dev;

__device__ __forceinline__ void load_ray(const TraceParams& p, uint32_t i, RayCtx& R) {
  const float4* rp = p.rays + 2 * (size_t)i;
  const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
  R.o = make_float3(r0.x, r0.y, r0.z);
  R.tmin = r0.w;
  R.d = make_float3(r1.x, r1.y, r1.z);
  R.tmax = r1.w;
}

__device__ __forceinline__ void store_hit(const TraceParams& p, uint32_t i, const RayCtx& R) {
  float4 out;
  uint4 ext;
  if (R.best.have) {
    const uint4 gm = __ldg(reinterpret_cast<const uint4*>(p.tri_root + R.best.geom_slot));
    const uint32_t prim = __ldg(p.redirect + R.best.k) - gm.z;
    out = make_float4(R.best.t, R.best.u, R.best.v, __uint_as_float(prim));
    ext = make_uint4(gm.y, R.best.inst, __ldg(&p.tlas_data[R.best.inst].instance_custom_index),
                     (R.best.s < 0.0f) ? 0xFFu : 0xFEu);
  } else {
    out = make_float4(R.tmax, 0.0f, 0.0f, __uint_as_float(INVALID_NEXT));
    ext = make_uint4(INVALID_NEXT, INVALID_NEXT, INVALID_NEXT, 0u);
  }
  reinterpret_cast<float4*>(p.hits)[i] = out;
  if (p.hits_ext) reinterpret_cast<uint4*>(p.hits_ext)[i] = ext;
}

// SPLIT: only the warps whose rays are alike (trace_quad_kernel takes the others).
template <int MODE, bool COUNT, bool LOCAL, bool WT, bool SPLIT>
__global__ void __launch_bounds__(256) trace_kernel(TraceParams p) {
  RDN_TRAVERSAL_STACK(LOCAL);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  // Lanes past the ray count stay alive (with zero counts) until the counter
  // reduction, which reads every lane of the warp: block sizes are multiples of 32.
  unsigned long long nv = 0, tt = 0, th = 0, bt = 0;
  const bool valid = i < p.count;
  RayCtx R;
  uint32_t tidx = p.tlas_uniform;
  if (valid) {
    load_ray(p, i, R);
    if (p.tlas_idx) tidx = __ldg(p.tlas_idx + i);
  }
  if (SPLIT && !coherent_warp(R, tidx, valid)) return;
  if (valid) {
    R.cull_mask = p.cull_mask;
    R.ray_flags = p.ray_flags;
    bool bad;
    traverse_ray<MODE, COUNT, BuiltinAnyHit, WT, 2, WT>(p, R, tidx, stack_ptr, stack_stride, bad);
    store_hit(p, i, R);
    if (bad) atomicOr(p.error_word, 2u);
    if (COUNT) {
      nv = R.node_visits;
      tt = R.tri_tests;
      th = R.tri_hits;
      bt = bad ? 1ull : 0ull;
    }
  }
  if (COUNT) {
    __syncwarp();
    for (int off = 16; off > 0; off >>= 1) {
      nv += __shfl_down_sync(0xffffffffu, nv, off);
      tt += __shfl_down_sync(0xffffffffu, tt, off);
      th += __shfl_down_sync(0xffffffffu, th, off);
      bt += __shfl_down_sync(0xffffffffu, bt, off);
    }
    if ((threadIdx.x & 31) == 0 && (nv | tt | th | bt)) {
      atomicAdd(p.counters + 0, nv);
      atomicAdd(p.counters + 1, tt);
      atomicAdd(p.counters + 2, th);
      atomicAdd(p.counters + 3, bt);
    }
  }
}

// Four lanes per ray, one warp per block. The first `differing` blocks take
// `batch` rays each; with split they leave out the groups of 32 rays that are
// alike, which the blocks after them (if there are any) take eight rays at a
// time: the quads of such a warp walk the same nodes in step, and four warps
// on a group finish sooner than one.
template <bool WT>
__global__ void __launch_bounds__(128, 8) trace_quad_kernel(TraceParams p, uint32_t batch, uint32_t differing, bool split) {
  extern __shared__ __align__(16) unsigned char quad_smem[];
  const uint32_t lane = threadIdx.x & 31u;
  const bool take_alike = blockIdx.x >= differing;
  if (take_alike) batch = 8;
  const uint32_t first = (blockIdx.x - (take_alike ? differing : 0u)) * batch;
  RayCtx R;
  uint32_t tidx = p.tlas_uniform;
  if (split) {
    const uint32_t g = (first & ~31u) + lane;
    if (g < p.count) {
      load_ray(p, g, R);
      if (p.tlas_idx) tidx = __ldg(p.tlas_idx + g);
    }
    if (coherent_warp(R, tidx, g < p.count) != take_alike) return;
  }
  const uint32_t i = first + lane;
  const bool valid = lane < batch && i < p.count;
  if (valid && !(split && batch == 32u)) {
    load_ray(p, i, R);
    if (p.tlas_idx) tidx = __ldg(p.tlas_idx + i);
  }
  R.cull_mask = p.cull_mask;
  R.ray_flags = p.ray_flags;
  bool bad;
  traverse_warp<WT>(p, R, tidx, valid, quad_warp(quad_smem, p.stack_depth4), bad);
  if (!valid) return;
  store_hit(p, i, R);
  if (bad) atomicOr(p.error_word, 2u);
}

}  // namespace

uint32_t stack_entries(int mode, uint32_t max_binary_depth, uint32_t max_wide4_depth) {
  uint32_t d = mode == MODE_WIDE4 ? 3 * max_wide4_depth + 1 : (mode == MODE_BINARY ? max_binary_depth + 1 : 0);
  d = (d + 3) & ~3u;
  return d < 8 ? 8 : d;
}

namespace {
// How a batch query is shared out, by its ray count (ordered walks; us on
// camera rays of the 1024^2 / 128^2 field and on random rays through a 10k soup):
//   below kQuadSplit    quads, eight rays a warp: too few rays to fill the
//                       chip, so the longest warp decides. 65,536 camera rays
//                       onto the soup: one ray per lane 85, 8 rays a warp 49,
//                       16 79, 32 119; 1,000 random rays: 84 -> 47
//   below kQuadBatch32  quads; rays that differ 16 a warp (48,000 random rays:
//                       8 a warp 100, 16 88, 32 120), alike ones still 8
//   below quad_limit    the same with 32 (131,072 random: 193 / 159 / 150;
//                       camera rays: 160,000 8 a warp 127 / 70, lanes 173 / 87;
//                       327,680 215 / 101, lanes 237 / 98)
//   from there on       alike rays one per lane (400,000: quads 259 / 102,
//                       lanes 273 / 99; 786,432: 431 / 187, 323 / 112), the
//                       rest quads (777,777 through a 150k soup: lanes 917,
//                       quads 835; watertight 1200, 943)
// quad_limit is 400,000 for these; 262,144 camera rays on fields of 16^2, 64^2
// and 128^2: quads 73, 90, 107 us, lanes 28, 43, 60, two-child lanes 32, 56, 88.
constexpr uint32_t kQuadSplit = 40000, kQuadBatch32 = 100000, kQuadMost = 400000;
constexpr float kQuadRays = 300.0f;

template <int MODE, bool COUNT, bool LOCAL, bool WT, bool SPLIT>
cudaError_t launch_lanes_wt(const TraceParams& p, uint32_t block, cudaStream_t stream) {
  const uint32_t grid = (uint32_t)(((uint64_t)p.count + block - 1) / block);
  const size_t smem = MODE != MODE_THREADED && !LOCAL ? (size_t)p.stack_depth * block * sizeof(uint2) : 0;
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = raise_smem_limit(attr_done, {(const void*)trace_kernel<MODE, COUNT, LOCAL, WT, SPLIT>});
  if (e != cudaSuccess) return e;
  trace_kernel<MODE, COUNT, LOCAL, WT, SPLIT><<<grid, block, smem, stream>>>(p);
  return cudaGetLastError();
}

template <int MODE, bool COUNT, bool LOCAL, bool SPLIT = false>
cudaError_t launch_lanes(const TraceParams& p, uint32_t block, cudaStream_t stream) {
  return p.watertight ? launch_lanes_wt<MODE, COUNT, LOCAL, true, SPLIT>(p, block, stream)
                      : launch_lanes_wt<MODE, COUNT, LOCAL, false, SPLIT>(p, block, stream);
}

// split: 0 every ray, 1 the groups of 32 that differ, 2 those and the others eight rays a warp
cudaError_t launch_quads(const TraceParams& p, uint32_t batch, int split, cudaStream_t stream) {
  const uint32_t differing = (uint32_t)(((uint64_t)p.count + batch - 1) / batch);
  const uint32_t grid = differing + (split == 2 ? (uint32_t)(((uint64_t)p.count + 7) / 8) : 0u);
  const size_t smem = quad_warp_bytes(p.stack_depth4);
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = raise_smem_limit(attr_done, {(const void*)trace_quad_kernel<false>, (const void*)trace_quad_kernel<true>});
  if (e != cudaSuccess) return e;
  if (p.watertight) trace_quad_kernel<true><<<grid, 32, smem, stream>>>(p, batch, differing, split != 0);
  else trace_quad_kernel<false><<<grid, 32, smem, stream>>>(p, batch, differing, split != 0);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_trace(const TraceParams& p, int mode, bool counted, uint32_t block, cudaStream_t stream) {
  if (p.count == 0) return cudaSuccess;
  if (block == 0) block = 64;
  if (mode == MODE_THREADED)
    return counted ? launch_lanes<MODE_THREADED, true, false>(p, block, stream)
                   : launch_lanes<MODE_THREADED, false, false>(p, block, stream);
  if (counted)
    return mode == MODE_WIDE4 ? launch_lanes<MODE_WIDE4, true, false>(p, block, stream)
                              : launch_lanes<MODE_BINARY, true, false>(p, block, stream);
  const TraceParams q = wide4_params(p);
  const bool local = q.local_stack != 0;
  if (!p.packed) return local ? launch_lanes<MODE_WIDE4, false, true>(q, block, stream)
                             : launch_lanes<MODE_WIDE4, false, false>(q, block, stream);
  if (p.count < kQuadSplit) return launch_quads(q, 8, 0, stream);
  const uint32_t batch = p.count < kQuadBatch32 ? 16 : 32;
  if (!local || p.count < quad_limit(p, kQuadRays, kQuadSplit, kQuadMost)) return launch_quads(q, batch, 2, stream);
  if (small_trees(p)) return launch_lanes<MODE_WIDE4, false, true>(q, block, stream);
  const cudaError_t e = launch_quads(q, batch, 1, stream);
  return e == cudaSuccess ? launch_lanes<MODE_WIDE4, false, true, true>(q, block, stream) : e;
}

}  // namespace rdn
