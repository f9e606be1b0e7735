// Launch interface of the ray-query kernels (trace.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "rdn_core.h"

namespace rdn {

struct TraceParams {
  const float4* rays;  // 2 per ray (rdn_ray)
  rdn_hit* hits;
  rdn_hit_ext* hits_ext;
  const uint32_t* tlas_idx;
  uint32_t count, tlas_uniform, ray_flags, cull_mask, anyhit_mode, stack_depth;
  uint32_t stack_depth4;  // entries of a four-child walk's stack, whatever the traversal asked for
  uint32_t n_binding, n_tlas_root;
  const uint32_t* tlas_binding;
  const uint32_t* tlas_bvh_root;
  const DeviceBVHNode* tlas_forest;
  const DeviceInstance* tlas_data;
  const TlasBounding* tlas_bounding;
  const BlasMetaInfo* blas_meta;
  const GeometryMetaInfo* tri_root;
  const DeviceBVHNode* tri_forest;
  const uint32_t* redirect;
  const float4* tris;   // 4 per triangle (TriRecord)
  const float4* wide;   // 4 per node (WideNode)
  const uint2* leaves;
  const uint32_t* geom_root_code;
  const float4* wide4;  // 8 per node (Wide4Node)
  const uint32_t* geom_root_code4;
  unsigned long long* counters;  // 4 x u64, used by counted launches
  uint32_t* error_word;          // bit 0 stack overflow, bit 1 bad tlas index, bit 2 iteration cap
  // 1: per-thread traversal stacks in local memory (ordered walks whose stack
  // fits kLocalStackEntries), 0: in shared memory
  uint32_t local_stack;
  // speculative ordered walk: lanes holding a leaf keep descending while more
  // than this many lanes of the warp are still looking for one (0 = until all
  // have one)
  uint32_t spec_threshold;
  const uint32_t* anyhit_mask;  // RDN_ANYHIT_PRIMITIVE_MASK: one bit per built triangle
  // iteration cap of the dynamic-fetch loops (0 = the built-in cap); on
  // reaching it a warp sets bit 2 of the error word and stops
  uint32_t iteration_limit;
  // 1: launch the kernels built for the watertight test (over `verts`, with
  // conservative box tests) instead of the reference's formula over `tris`
  // (which still gives the shading normal); kernels take the choice as a
  // template argument, so the reference-formula kernels carry no cost for it
  uint32_t watertight;
  const float4* verts;  // 3 per triangle (VertexRecord), sorted order
  uint32_t packed;      // 1: the four-child tree holds packed_leaf codes (needed to walk it with quads)
  uint32_t instanced;   // 1: a TLAS holds more than one instance
  float line_nodes;     // HostBuilt::line_nodes: how much a ray walks, by which a launch is given its kind of walk
};

// 1 + 2 gamma_3 (gamma_n = n u / (1 - n u), u = 2^-24) rounded up to f32:
// 1 + 4 * 2^-23 (Ize, "Robust BVH Ray Traversal", JCGT 2013).
constexpr float kWatertightBoxFarScale = 1.000000476837158203125f;

// entries of a local-memory traversal stack
constexpr uint32_t kLocalStackEntries = 64;

// Traversal modes (template argument of every traversal kernel).
// MODE_WIDE4_TOGETHER is the walk of MODE_WIDE4 with the lanes of a warp
// entering their BLASes together (traverse_together).
enum TraversalMode : int { MODE_THREADED = 0, MODE_BINARY = 1, MODE_WIDE4 = 2, MODE_WIDE4_TOGETHER = 3 };

// Parameters of an ordered walk on the four-child tree, whichever node width
// was asked for (the results are the same and the four-child walk is the
// faster one: 2.07 M camera rays 917 us on two-child nodes, 789 on four-child
// ones of the same build), its stack in local memory where it fits.
inline TraceParams wide4_params(const TraceParams& p) {
  TraceParams q = p;
  q.stack_depth = p.stack_depth4;
  q.local_stack = q.stack_depth <= kLocalStackEntries;
  return q;
}

// Rays (pixels, paths) of a batch up to which four lanes per ray are its faster
// walk: `per_square` times the square of the nodes that a line meets, between
// `least` and `most`. Four lanes per ray finish a batch sooner that is bound by
// its longest walks, and cost more where the chip is full; the longest walk
// grows faster with the tree than the mean. Where the two met (camera queries):
//   field of 16^2, 64^2, 128^2, 256^2, 512^2, 1024^2   10.7, 19.6, 24.2, 28.8, 33.4, 37.9 nodes
//                                      40k, 65k, 95k, 150k, 240k, 400k rays
//   soup of 12, 100, 1000, 10000       2.9, 7.8, 21, 57 nodes; 10k, 65k, 160k, above 320k rays
// Neither the depth nor the triangles tell a field from a soup. The factors of
// the kernels lie between these lines and those where two-child walks, one ray
// per lane, were as fast.
inline uint32_t quad_limit(const TraceParams& p, float per_square, uint32_t least, uint32_t most) {
  const float n = per_square * p.line_nodes * p.line_nodes;
  return n >= (float)most ? most : (n > (float)least ? (uint32_t)n : least);
}
// Trees so small that a batch above quad_limit goes by lanes whole: the second
// kernel of a split batch costs more than its four lanes per ray gain (us,
// 1920x1080 camera rays, two-child lanes / split / lanes: soups of 12 triangles
// 32 / 69 / 32, of 300 58 / 86 / 47; 777,777 random rays 38 / 67 / 36, 175 /
// 151 / 119). Rays that enter many instances gain more.
inline bool small_trees(const TraceParams& p) { return p.line_nodes < (p.instanced ? 5.0f : 13.0f); }

// stack entries the mode needs per thread
uint32_t stack_entries(int mode, uint32_t max_binary_depth, uint32_t max_wide4_depth);

cudaError_t launch_trace(const TraceParams& p, int mode, bool counted, uint32_t block, cudaStream_t stream);

}  // namespace rdn
