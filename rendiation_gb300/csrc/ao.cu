// Fused ambient-occlusion frame for sm_103a: the reference AO renderer's ray
// generation, primary closest hit, occlusion ray and miss shaders
// (feature/ao.rs:193-296) as one kernel, one thread per pixel over 4x8 pixel
// tiles, or four lanes per ray for frames that do not fill the chip. It computes what the task-graph form of the same pipeline
// computes, without the task pools. Built with -fmad=false: see ao.cuh.
#include <cuda_runtime.h>

#include <cstdint>

#include "ao.cuh"
#include "quad.cuh"
#include "traverse.cuh"

namespace rdn {
namespace {

using namespace dev;

template <int MODE, bool LOCAL, bool WT>
__global__ void __launch_bounds__(128) ao_kernel(TraceParams P, AoEnv A) {
  RDN_TRAVERSAL_STACK(LOCAL);
  uint32_t x, y;
  if (!ao_pixel(A, blockIdx.x * blockDim.x + threadIdx.x, x, y)) return;
  float3 o, d;
  ao_camera_ray(A, x, y, o, d);
  RayCtx R;
  R.o = o;
  R.d = d;
  R.tmin = F32_EPSILON;
  R.tmax = F32_MAX;
  R.ray_flags = RAY_FLAG_CULL_BACK;
  R.cull_mask = 0xFFFFFFFFu;
  bool bad;
  traverse_ray<MODE, false, BuiltinAnyHit, WT>(P, R, A.tlas, stack_ptr, stack_stride, bad);
  float payload = 1.0f;  // miss shader
  if (R.best.have) {
    const float3 hit = o + d * R.best.t;
    const float3 n =
        ao_shading_normal(A, P.tlas_data + R.best.inst, __ldg(P.redirect + R.best.k), R.best.u, R.best.v, o, hit);
    RayCtx S;
    S.o = hit;
    S.d = ao_direction(n, ao_sample(A));
    S.tmin = AO_TEST_MIN;
    S.tmax = AO_TEST_MAX;
    S.ray_flags = RAY_FLAG_END_SEARCH;
    S.cull_mask = 0xFFFFFFFFu;
    bool bad2;
    traverse_ray<MODE, false, BuiltinAnyHit, WT>(P, S, A.tlas, stack_ptr, stack_stride, bad2);
    bad |= bad2;
    payload = S.best.have ? 0.0f : 1.0f;  // secondary closest hit: occluded
  }
  if (bad) atomicOr(P.error_word, 2u);
  ao_count(A, 0, true);
  ao_count(A, 1, R.best.have);
  ao_accumulate(A, y * A.width + x, payload);
}

// Four lanes per ray (quad.cuh), a warp `batch` pixels, for frames of up to
// kQuadPixels: below that the slowest warps decide a frame's time, and a warp
// of eight or sixteen pixels is done in less than half the time of one of 32
// (us for four samples on the 1024^2 field: 128^2 pixels, one per thread 582,
// 8 a warp 303; 256^2 662, 8 487, 16 520; means of four cameras: 400x300 841,
// 760; 400^2 930, 890; 512^2 1030, 1180; 800x500 1370, 1710). Above it pixels that are alike share their
// nodes better one per lane. Smaller trees: up to quad_limit (160,000 pixels of
// the fields of 16^2, 64^2, 128^2, of two-child lanes: quads 2.08, 1.34, 0.91,
// lanes 0.90, 0.78, 0.67; soups of 100, 1000: 1.28, 1.02 and 0.90, 0.76).
constexpr uint32_t kQuadLeast = 40000, kQuadPixels = 200000;
constexpr float kQuadRays = 180.0f;
constexpr uint32_t ao_quad_batch(uint32_t pixels) { return pixels < 100000u ? 8u : 16u; }

template <bool WT>
__global__ void __launch_bounds__(128, 8) ao_quad_kernel(TraceParams P, AoEnv A, uint32_t batch) {
  extern __shared__ __align__(16) unsigned char quad_smem[];
  const QuadWarp W = quad_warp(quad_smem, P.stack_depth4);
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t x = 0, y = 0;
  const uint32_t idx = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * batch + lane;
  const bool valid = lane < batch && ao_pixel(A, idx, x, y);
  RayCtx R;
  if (valid) ao_camera_ray(A, x, y, R.o, R.d);
  R.tmin = F32_EPSILON;
  R.tmax = F32_MAX;
  R.ray_flags = RAY_FLAG_CULL_BACK;
  R.cull_mask = 0xFFFFFFFFu;
  bool bad;
  traverse_warp<WT>(P, R, A.tlas, valid, W, bad);
  const bool hit = valid && R.best.have;
  RayCtx S;
  if (hit) {
    float3 o, d;
    ao_camera_ray(A, x, y, o, d);
    S.o = o + d * R.best.t;
    const float3 n =
        ao_shading_normal(A, P.tlas_data + R.best.inst, __ldg(P.redirect + R.best.k), R.best.u, R.best.v, o, S.o);
    S.d = ao_direction(n, ao_sample(A));
  }
  S.tmin = AO_TEST_MIN;
  S.tmax = AO_TEST_MAX;
  S.ray_flags = RAY_FLAG_END_SEARCH;
  S.cull_mask = 0xFFFFFFFFu;
  bool bad2;
  traverse_warp<WT>(P, S, A.tlas, hit, W, bad2);
  if (!valid) return;
  if (bad || (hit && bad2)) atomicOr(P.error_word, 2u);
  ao_count(A, 0, true);
  ao_count(A, 1, hit);
  ao_accumulate(A, y * A.width + x, hit && S.best.have ? 0.0f : 1.0f);  // 1: the camera ray or the occlusion ray missed
}

template <bool WT>
cudaError_t launch_quads(const TraceParams& p, const AoEnv& a, uint32_t pixels, cudaStream_t st) {
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = raise_smem_limit(attr_done, {(const void*)ao_quad_kernel<WT>});
  if (e != cudaSuccess) return e;
  const uint32_t batch = ao_quad_batch(pixels);
  ao_quad_kernel<WT><<<(pixels + batch - 1) / batch, 32, quad_warp_bytes(p.stack_depth4), st>>>(p, a, batch);
  return cudaGetLastError();
}

template <int MODE, bool LOCAL, bool WT>
cudaError_t launch_variant_wt(const TraceParams& p, const AoEnv& a, cudaStream_t st) {
  const uint32_t block = a.block ? a.block : 128;
  const uint32_t grid = (ao_dispatch_count(a.width, a.height) + block - 1) / block;
  const size_t smem = MODE != MODE_THREADED && !LOCAL ? (size_t)p.stack_depth * block * sizeof(uint2) : 0;
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = raise_smem_limit(attr_done, {(const void*)ao_kernel<MODE, LOCAL, WT>});
  if (e != cudaSuccess) return e;
  ao_kernel<MODE, LOCAL, WT><<<grid, block, smem, st>>>(p, a);
  return cudaGetLastError();
}

template <int MODE, bool LOCAL>
cudaError_t launch_variant(const TraceParams& p, const AoEnv& a, cudaStream_t st) {
  return p.watertight ? launch_variant_wt<MODE, LOCAL, true>(p, a, st) : launch_variant_wt<MODE, LOCAL, false>(p, a, st);
}

__global__ void ao_advance_kernel(uint32_t* counter) { *counter += 1u; }

}  // namespace

cudaError_t launch_ao_advance(uint32_t* counter, cudaStream_t st) {
  ao_advance_kernel<<<1, 1, 0, st>>>(counter);
  return cudaGetLastError();
}

cudaError_t launch_ao(const TraceParams& p, const AoEnv& a, int mode, cudaStream_t st) {
  if (a.width == 0 || a.height == 0) return cudaSuccess;
  const uint32_t pixels = ao_dispatch_count(a.width, a.height);
  if (mode != MODE_THREADED && p.packed && pixels <= quad_limit(p, kQuadRays, kQuadLeast, kQuadPixels))
    return p.watertight ? launch_quads<true>(p, a, pixels, st) : launch_quads<false>(p, a, pixels, st);
  if (mode != MODE_THREADED) {
    const TraceParams q = wide4_params(p);
    return q.local_stack ? launch_variant<MODE_WIDE4, true>(q, a, st) : launch_variant<MODE_WIDE4, false>(q, a, st);
  }
  return launch_variant<MODE_THREADED, false>(p, a, st);
}

}  // namespace rdn
