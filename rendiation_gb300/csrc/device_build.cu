// Device build of the triangle BVH forest: the reference's binned SAH tree
// (content/space/src/bvh/strategy.rs:11-43,202-284 with SAH::new(4); degenerate
// binning falls back to BalanceTree's median split, strategy.rs:66-87 and
// apply.rs:19-45), flattened exactly as NaiveSahBvhSource::build flattens it
// (shader/ray-tracing/src/backend/wavefront_compute/geometry/naive/mod.rs:
// 122-260 for the geometry arrays, :338-386 for the forest, :611-632 for the
// threaded links), plus the two-child, four-child and triangle-record layouts
// of the traversal kernels. The arrays equal the host build's byte for byte.
//
// The reference builds one node at a time, depth first, on one thread. Here
// every geometry's tree is built together. Nodes of more than kSmall primitives
// go one tree level per round:
//   stats     per chunk: the 4 centroid buckets on the longest axis of the
//             node box, their counts and boxes, merged into the node;
//   decide    per node: the reference's 3-candidate SAH choice (or the median
//             fallback when 3 buckets are empty), each chunk's per-bucket
//             offset inside the node, and the two children, each a leaf or a
//             split (count > bin_size and depth < max_depth, utils.rs:35-37)
//             that claims warp tasks of 256 primitives ("chunks");
//   prefix    the chunk offsets of nodes with many chunks, a block per node;
//             median-split nodes run Rust's select_nth_unstable_by restatement
//             on one thread each;
//   scatter   SAH nodes write their primitives in bucket order, stable inside
//             a bucket (warp ballots), into the other of two order arrays;
//             median-split nodes copy theirs and reduce the children's boxes.
// Nodes of kSmall primitives and fewer are left to small_trees_kernel, which
// builds the whole subtree below each in shared memory, a block per subtree and
// a warp or a lane per node: a level of many small nodes is bound by the gaps
// between its launches and by reductions over empty lanes (2.1 M triangles,
// bin size 4: all by level rounds 5.2 ms a build, subtrees in blocks 3.35 ms;
// 8,000 triangles 1.58 and 0.75 ms; 1,000 triangles 1.19 and 0.63 ms; with the arrays
// kept and four launches a level now 2.04, 0.44 and 0.33 ms).
// Boxes are merged with integer atomics on an order-preserving key of the
// float, so a union does not depend on the order primitives arrive in. The
// reference's pre-order numbering is recovered afterwards from subtree sizes
// (bottom-up) and a top-down pass, and the two-child node / leaf numbering from
// one scan over the pre-order inner-node flags. Compiled with -fmad=false: the
// bucket, area and cost arithmetic must round exactly as the reference's.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "device_build.h"
#include "parallel.h"
#include "rust_select.h"

namespace rdn {
namespace {

constexpr uint32_t NONE = 0xFFFFFFFFu;
constexpr uint32_t kChunk = 256;
constexpr uint32_t kBlock = 256;
constexpr uint32_t kWarps = kBlock / 32;
constexpr uint32_t F_BOX_PENDING = 1u, F_ACTIVE = 2u, F_FALLBACK = 4u, F_IN_B = 8u;  // F_IN_B: primitives in the second order array
// Subtrees of at most this many primitives are built by one block each.
constexpr uint32_t kSmall = 256;

// Order-preserving int key of a float (no NaN reaches a box: boxes start
// empty and grow with NaN-ignoring min/max). -0.0 orders below +0.0.
__host__ __device__ __forceinline__ int key_of(float f) {
#ifdef __CUDA_ARCH__
  const int i = __float_as_int(f);
#else
  int i;
  std::memcpy(&i, &f, 4);
#endif
  return i >= 0 ? i : (i ^ 0x7FFFFFFF);
}
__host__ __device__ __forceinline__ float val_of(int k) {
  const int i = k >= 0 ? k : (k ^ 0x7FFFFFFF);
#ifdef __CUDA_ARCH__
  return __int_as_float(i);
#else
  float f;
  std::memcpy(&f, &i, 4);
  return f;
#endif
}

struct alignas(16) BNode {  // 64 B, one per tree node during the build
  int lo[3], hi[3];   // box as keys
  uint32_t start, end;  // range in the global primitive order
  uint32_t depth, left;  // left child id (right = left + 1), NONE for a leaf
  uint32_t tree, flags;
  uint32_t cbase, nchunks;  // a split's chunks; in the finished tree: subtree size, pre-order place below `sub`
  uint32_t sub;             // finished tree: root of the subtree that a block built, NONE for a node above those
  uint32_t pad;
};
static_assert(sizeof(BNode) == 64, "64 B build node");

struct LevelCounters {  // one per tree level, zeroed before the first level
  uint32_t chunks, children, big, pad;
};
struct BuildCounters {
  unsigned long long sah, fallback;
  uint32_t bad_index, max_depth;
  uint32_t ended;     // nodes that have left the level rounds
  uint32_t added;     // nodes that the subtrees added to the pool
  uint32_t unfit;     // a split had an empty child (the subtree blocks count on none)
  uint32_t overflow;  // a level had more children than the pool holds
};

struct F3 {
  float x, y, z;
};
struct NodeBox {
  F3 lo, hi;
};

__device__ __forceinline__ NodeBox box_of(const BNode& n) {
  return NodeBox{{val_of(n.lo[0]), val_of(n.lo[1]), val_of(n.lo[2])}, {val_of(n.hi[0]), val_of(n.hi[1]), val_of(n.hi[2])}};
}
__device__ __forceinline__ float comp(const F3& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }
__device__ __forceinline__ int split_axis(const NodeBox& b) {  // Box3::longest_axis
  const float x = b.hi.x - b.lo.x, y = b.hi.y - b.lo.y, z = b.hi.z - b.lo.z;
  if (x > y) return x > z ? 0 : 2;
  return y > z ? 1 : 2;
}
__device__ __forceinline__ uint32_t bucket_of(float value, float start, float step) {
  // ((value - start) / step).floor() as usize, clamped to the last bucket
  const float f = floorf((value - start) / step);
  const uint32_t b = (f > 0.0f) ? (f >= 4.0f ? 4u : (uint32_t)f) : 0u;
  return b >= 4 ? 3u : b;
}
__device__ __forceinline__ float sah_area(const NodeBox& b) {  // 2 * (w*h + w*d + h*d)
  const float w = b.hi.x - b.lo.x, h = b.hi.y - b.lo.y, d = b.hi.z - b.lo.z;
  return 2.0f * (w * h + w * d + h * d);
}
__device__ __forceinline__ float half_area(const NodeBox& b) {  // collapse order of the four-child layout
  const float w = b.hi.x - b.lo.x, h = b.hi.y - b.lo.y, d = b.hi.z - b.lo.z;
  return w * h + w * d + h * d;
}
__device__ __forceinline__ NodeBox empty_box() {
  return NodeBox{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
}
__device__ __forceinline__ void grow(NodeBox& b, const NodeBox& o) {
  b.lo = {fminf(b.lo.x, o.lo.x), fminf(b.lo.y, o.lo.y), fminf(b.lo.z, o.lo.z)};
  b.hi = {fmaxf(b.hi.x, o.hi.x), fmaxf(b.hi.y, o.hi.y), fmaxf(b.hi.z, o.hi.z)};
}
__device__ __forceinline__ void set_box(BNode& n, const NodeBox& b) {
  n.lo[0] = key_of(b.lo.x);
  n.lo[1] = key_of(b.lo.y);
  n.lo[2] = key_of(b.lo.z);
  n.hi[0] = key_of(b.hi.x);
  n.hi[1] = key_of(b.hi.y);
  n.hi[2] = key_of(b.hi.z);
}

// Centre keys of one axis with the reference's comparator
// (partial_cmp(..).unwrap_or(Less) on the centre coordinate).
struct CentreLess {
  const float* key;  // centres, or lower and upper corners `boxes` floats apart
  uint32_t boxes;
  __device__ float of(uint32_t p) const {
    return boxes ? (key[2 * boxes * (size_t)p] + key[2 * boxes * (size_t)p + boxes]) * 0.5f : key[p];
  }
  __device__ bool operator()(const uint32_t& a, const uint32_t& b) const {
    const float ka = of(a), kb = of(b);
    return ka != ka || kb != kb || ka < kb;  // a NaN on either side compares Less
  }
};

// ---- geometry preparation ----------------------------------------------

// Global vertex indices (BLAS concatenation, naive/mod.rs:155-186), the
// primitive boxes (BuildPrimitive::new, utils.rs:40-66: grow an empty box by
// the 3 vertices); their centres are computed where they are used.
__global__ void prepare_primitives_kernel(uint32_t N, uint32_t G, const uint32_t* __restrict__ g_prim_start,
                                          const uint32_t* __restrict__ g_vstart, const uint32_t* __restrict__ g_vcount,
                                          const uint32_t* __restrict__ g_indexed, uint32_t* __restrict__ idx,
                                          const float* __restrict__ vtx, float4* __restrict__ pbox,
                                          BuildCounters* ctr) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = G;  // last g with g_prim_start[g] <= p
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) / 2;
      if (g_prim_start[mid] <= p) lo = mid;
      else hi = mid;
    }
    const uint32_t g = lo, local = p - g_prim_start[g], vs = g_vstart[g], vc = g_vcount[g];
    NodeBox b = empty_box();
    for (int k = 0; k < 3; k++) {
      uint32_t raw = g_indexed[g] ? idx[3 * (size_t)p + k] : 3 * local + k;
      if (raw >= vc) {
        atomicAdd(&ctr->bad_index, 1u);
        raw = 0;
      }
      idx[3 * (size_t)p + k] = vs + raw;
      if (vc) {
        const float* v = vtx + 3 * (size_t)(vs + raw);
        const F3 q = {v[0], v[1], v[2]};
        grow(b, NodeBox{q, q});
      }
    }
    pbox[2 * (size_t)p] = make_float4(b.lo.x, b.lo.y, b.lo.z, 0.0f);
    pbox[2 * (size_t)p + 1] = make_float4(b.hi.x, b.hi.y, b.hi.z, 0.0f);
  }
}

// The start of a build: the primitives in their order, one root per geometry
// (its box pending), level 0, and cleared counters.
__global__ void start_kernel(uint32_t N, uint32_t G, const uint32_t* __restrict__ g_prim_start,
                             uint32_t* __restrict__ order, BNode* __restrict__ pool, uint32_t* __restrict__ lvl,
                             LevelCounters* __restrict__ lcs, uint32_t level_cap, BuildCounters* bc) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (uint32_t p = t; p < N; p += stride) order[p] = p;
  for (uint32_t l = t; l < level_cap; l += stride) lcs[l] = LevelCounters{};
  if (t == 0) {
    lvl[0] = 0;
    lvl[1] = G;
    *bc = BuildCounters{};
  }
  for (uint32_t g = t; g < G; g += stride) {
    BNode r{};
    set_box(r, empty_box());
    r.start = g_prim_start[g];
    r.end = g_prim_start[g + 1];
    r.left = r.sub = NONE;
    r.tree = g;
    r.flags = F_BOX_PENDING;
    pool[g] = r;
  }
}

// Area shares are summed as whole numbers, so that a sum does not depend on the
// order: a root's share is kShareUnit.
constexpr uint32_t kShareUnit = 1u << 24;

// What the host reads of the finished build, in one copy.
struct BuildRoot {
  int lo[3], hi[3];
  uint32_t left, nodes, code;
  float line_nodes;
};
struct BuildSummary {
  uint32_t wide4_nodes, wide4_depth;
};
__global__ void summary_kernel(uint32_t G, uint32_t T, const BNode* __restrict__ pool, const uint32_t* __restrict__ tree_nodes,
                               const uint32_t* __restrict__ root_code, const uint32_t* __restrict__ index4,
                               const uint32_t* __restrict__ croot, const uint32_t* __restrict__ max_level4,
                               const unsigned long long* __restrict__ tree_share, BuildSummary* __restrict__ summary, BuildRoot* __restrict__ roots) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) *summary = BuildSummary{index4[T - 1] + croot[T - 1], *max_level4};
  if (t >= G) return;
  const BNode n = pool[t];
  roots[t] = BuildRoot{{n.lo[0], n.lo[1], n.lo[2]}, {n.hi[0], n.hi[1], n.hi[2]}, n.left, tree_nodes[t], root_code[t],
                       (float)((double)tree_share[t] * (1.0 / kShareUnit))};
}

// ---- one tree level -----------------------------------------------------

__device__ __forceinline__ uint32_t warp_inclusive_u32(uint32_t v, uint32_t lane) {
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= (uint32_t)o) v += t;
  }
  return v;
}

// Warp-aggregated claim on a counter: all 32 lanes call, each with its own
// amount (0 allowed); one atomic per warp instead of one per lane (a level
// of 250 k nodes would otherwise serialise on the counter's address).
__device__ __forceinline__ uint32_t warp_claim(uint32_t* ctr, uint32_t amount, uint32_t lane) {
  const uint32_t inc = warp_inclusive_u32(amount, lane);
  const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
  uint32_t base = 0;
  if (lane == 31 && total) base = atomicAdd(ctr, total);
  base = __shfl_sync(0xffffffffu, base, 31);
  return base + inc - amount;
}

// Level L holds nodes [lvl[L], lvl[L+1]) of the pool. The bounds live on the
// device: level L's last kernel writes lvl[L+2], so that the host can queue
// several levels without reading anything back. Kernels of an empty level
// (past the last one) find no node and return. Node loops step a whole warp
// at a time (warp-uniform bounds) so that the lanes can aggregate atomics.
struct LevelBuffers {  // of the nodes of one level, by their place in it
  uint32_t* acc_cnt;
  int* acc_box;
  uint32_t* chunk_node;
};
struct SplitRule {
  uint32_t bin_size, max_depth, small;
};

// Leaf or split of node n (id, the i-th of level L): a split claims its chunks
// and clears its sums, any other node goes to the list of ended ones. All 32
// lanes call, those without a node with `valid` unset.
__device__ __forceinline__ void prepare_node(bool valid, BNode& n, uint32_t id, uint32_t i, uint32_t L, const SplitRule& rule,
                                             const LevelBuffers& B, LevelCounters* lcs, BuildCounters* bc,
                                             uint32_t* __restrict__ ended) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t count = n.end - n.start;
  const bool active = valid && n.depth < rule.max_depth && count > rule.bin_size && count > rule.small;
  const bool need = active || (valid && count > rule.small && (n.flags & F_BOX_PENDING));
  const uint32_t nch = need ? (count + kChunk - 1) / kChunk : 0;
  n.flags = (n.flags & F_BOX_PENDING) | (active ? F_ACTIVE : 0u) | ((L & 1u) ? F_IN_B : 0u);
  n.left = NONE;
  n.nchunks = nch;
  const bool ends = valid && !active;
  const uint32_t at = warp_claim(&bc->ended, ends ? 1u : 0u, lane);
  if (ends) ended[at] = id;
  const uint32_t base = warp_claim(&lcs[L].chunks, nch, lane);
  n.cbase = nch ? base : 0u;
  // chunk -> node map: small ranges by their own lane, long ones by the whole warp
  if (nch && nch <= 32)
    for (uint32_t j = 0; j < nch; j++) B.chunk_node[base + j] = id;
  uint32_t wide = __ballot_sync(0xffffffffu, nch > 32);
  while (wide) {
    const uint32_t src = __ffs(wide) - 1;
    wide &= wide - 1;
    const uint32_t b = __shfl_sync(0xffffffffu, base, src), c = __shfl_sync(0xffffffffu, nch, src),
                   node = __shfl_sync(0xffffffffu, id, src);
    for (uint32_t j = lane; j < c; j += 32) B.chunk_node[b + j] = node;
  }
  if (active) {
    for (int b = 0; b < 4; b++) B.acc_cnt[4 * (size_t)i + b] = 0;
    for (int b = 0; b < 4; b++)
      for (int k = 0; k < 3; k++) {
        B.acc_box[24 * (size_t)i + 6 * b + k] = key_of(INFINITY);
        B.acc_box[24 * (size_t)i + 6 * b + 3 + k] = key_of(-INFINITY);
      }
  }
}

__global__ void prepare_roots_kernel(uint32_t G, SplitRule rule, BNode* __restrict__ pool, LevelBuffers B, LevelCounters* lcs,
                                     BuildCounters* bc, uint32_t* __restrict__ ended) {
  const uint32_t lane = threadIdx.x & 31u, stride = gridDim.x * blockDim.x;
  for (uint32_t g0 = blockIdx.x * blockDim.x + threadIdx.x - lane; g0 < G; g0 += stride) {
    const uint32_t g = g0 + lane;
    BNode n{};
    if (g < G) n = pool[g];
    prepare_node(g < G, n, g, g, 0, rule, B, lcs, bc, ended);
    if (g < G) pool[g] = n;
  }
}

__device__ __forceinline__ void chunk_range(const BNode& n, uint32_t c, uint32_t& s, uint32_t& e) {
  s = n.start + (c - n.cbase) * kChunk;
  e = min(n.end, s + kChunk);
}

// Boxes of the roots: min/max of the primitive boxes.
__global__ void root_box_kernel(const LevelCounters* lcs, BNode* __restrict__ pool,
                                const uint32_t* __restrict__ chunk_node, const uint32_t* __restrict__ order,
                                const float4* __restrict__ pbox) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t total = lcs[0].chunks;
  for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < total; c += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t id = chunk_node[c];
    const BNode n = pool[id];
    if (!(n.flags & F_BOX_PENDING)) continue;
    uint32_t s, e;
    chunk_range(n, c, s, e);
    int lo[3] = {key_of(INFINITY), key_of(INFINITY), key_of(INFINITY)};
    int hi[3] = {key_of(-INFINITY), key_of(-INFINITY), key_of(-INFINITY)};
    for (uint32_t i = s + lane; i < e; i += 32) {
      const uint32_t p = order[i];
      const float4 a = pbox[2 * (size_t)p], b = pbox[2 * (size_t)p + 1];
      lo[0] = min(lo[0], key_of(a.x));
      lo[1] = min(lo[1], key_of(a.y));
      lo[2] = min(lo[2], key_of(a.z));
      hi[0] = max(hi[0], key_of(b.x));
      hi[1] = max(hi[1], key_of(b.y));
      hi[2] = max(hi[2], key_of(b.z));
    }
    for (int k = 0; k < 3; k++) {
      lo[k] = __reduce_min_sync(0xffffffffu, lo[k]);
      hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
    }
    if (lane < 3) {
      atomicMin(&pool[id].lo[lane], lo[lane]);
      atomicMax(&pool[id].hi[lane], hi[lane]);
    }
  }
}

struct SplitPlane {
  int axis;
  float a0, step;
};
__device__ __forceinline__ SplitPlane plane_of(const BNode& n) {
  const NodeBox nb = box_of(n);
  SplitPlane sp;
  sp.axis = split_axis(nb);
  sp.a0 = comp(nb.lo, sp.axis);
  const float a1 = comp(nb.hi, sp.axis);
  sp.step = (a1 - sp.a0) / 4.0f;
  return sp;
}

// Bucket counts and boxes of each chunk, merged into the node. Bound by the
// latency of the gathers: a lane loads four primitives' boxes (one sector each,
// their centres included) before it uses the first.
__global__ void level_stats_kernel(const uint32_t* __restrict__ lvl, uint32_t L, const LevelCounters* lcs,
                                   const BNode* __restrict__ pool, const uint32_t* __restrict__ chunk_node,
                                   const uint32_t* __restrict__ order, const float4* __restrict__ pbox,
                                   uint8_t* __restrict__ bucket, uint32_t* __restrict__ chunk_cnt,
                                   uint32_t* __restrict__ acc_cnt, int* __restrict__ acc_box) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lb = lvl[L];
  const uint32_t total = lcs[L].chunks;
  for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < total; c += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t id = chunk_node[c];
    const BNode n = pool[id];
    if (!(n.flags & F_ACTIVE)) continue;
    const SplitPlane sp = plane_of(n);
    uint32_t s, e;
    chunk_range(n, c, s, e);
    uint32_t cnt[4] = {0, 0, 0, 0};
    int bx[4][6];
#pragma unroll
    for (int b = 0; b < 4; b++) {
      bx[b][0] = bx[b][1] = bx[b][2] = key_of(INFINITY);
      bx[b][3] = bx[b][4] = bx[b][5] = key_of(-INFINITY);
    }
    constexpr int kAhead = 4;
    for (uint32_t i0 = s + lane; i0 < e; i0 += 32 * kAhead) {
      float4 a[kAhead], b[kAhead];
#pragma unroll
      for (int m = 0; m < kAhead; m++) {
        const uint32_t i = i0 + 32 * m;
        if (i < e) {
          const size_t p = order[i];
          a[m] = pbox[2 * p];
          b[m] = pbox[2 * p + 1];
        }
      }
#pragma unroll
      for (int m = 0; m < kAhead; m++) {
        const uint32_t i = i0 + 32 * m;
        if (i >= e) break;
        const float centre = sp.axis == 0 ? (a[m].x + b[m].x) * 0.5f
                             : sp.axis == 1 ? (a[m].y + b[m].y) * 0.5f
                                            : (a[m].z + b[m].z) * 0.5f;
        const uint32_t bk = bucket_of(centre, sp.a0, sp.step);
        bucket[i] = (uint8_t)bk;
        const int k[6] = {key_of(a[m].x), key_of(a[m].y), key_of(a[m].z), key_of(b[m].x), key_of(b[m].y), key_of(b[m].z)};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (bk == (uint32_t)q) {
            cnt[q]++;
            bx[q][0] = min(bx[q][0], k[0]);
            bx[q][1] = min(bx[q][1], k[1]);
            bx[q][2] = min(bx[q][2], k[2]);
            bx[q][3] = max(bx[q][3], k[3]);
            bx[q][4] = max(bx[q][4], k[4]);
            bx[q][5] = max(bx[q][5], k[5]);
          }
        }
      }
    }
    const uint32_t li = id - lb;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t tot = __reduce_add_sync(0xffffffffu, cnt[q]);
      int r[6];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        r[k] = __reduce_min_sync(0xffffffffu, bx[q][k]);
        r[3 + k] = __reduce_max_sync(0xffffffffu, bx[q][3 + k]);
      }
      if (lane == 0) chunk_cnt[4 * (size_t)c + q] = tot;
      if (tot) {
        if (lane == 0) atomicAdd(&acc_cnt[4 * (size_t)li + q], tot);
        if (lane < 3) atomicMin(&acc_box[24 * (size_t)li + 6 * q + lane], r[lane]);
        else if (lane < 6) atomicMax(&acc_box[24 * (size_t)li + 6 * q + lane], r[lane]);
      }
    }
  }
}

// Nodes with more chunks than this leave their chunk prefix to
// level_big_prefix_kernel (a block per node); smaller ones are scanned by
// their own thread.
constexpr uint32_t kBigChunks = 8;

// The reference's split decision (strategy.rs:202-284) from the 4 buckets'
// counts and boxes: BalanceTree's median split (3 empty buckets,
// strategy.rs:67-87; `left` is unset) or the first strictly cheaper of the 3
// SAH candidates, `left` primitives to the left.
struct Split {
  bool fallback;
  uint32_t left;
  NodeBox l, r;
};
__device__ __forceinline__ Split decide_split(const uint32_t (&cnt)[4], const NodeBox (&bb)[4]) {
  Split s;
  const int empties = (cnt[0] == 0) + (cnt[1] == 0) + (cnt[2] == 0) + (cnt[3] == 0);
  s.fallback = empties == 3;
  s.left = 0;
  s.l = s.r = empty_box();
  if (s.fallback) return s;  // child boxes come from their primitives
  // candidate j puts buckets 0..=j left; the first strictly cheaper
  // candidate wins, candidate 0 when no cost is below +inf
  float best_cost = INFINITY;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    NodeBox lb_ = empty_box(), rb_ = empty_box();
    uint32_t lc_ = 0, rc_ = 0;
#pragma unroll
    for (int p = 0; p <= j; p++) {
      grow(lb_, bb[p]);
      lc_ += cnt[p];
    }
#pragma unroll
    for (int p = j + 1; p < 4; p++) {
      grow(rb_, bb[p]);
      rc_ += cnt[p];
    }
    const float cost = sah_area(lb_) * (float)lc_ + sah_area(rb_) * (float)rc_;
    if (j == 0 || cost < best_cost) {
      s.l = lb_;
      s.r = rb_;
      s.left = lc_;
    }
    if (cost < best_cost) best_cost = cost;
  }
  return s;
}

// The two children of active node i of the level; true for the median split.
__device__ __forceinline__ bool split_node(const BNode& n, uint32_t i, const uint32_t* __restrict__ acc_cnt,
                                           const int* __restrict__ acc_box, BNode& l, BNode& r) {
  uint32_t cnt[4];
  NodeBox bb[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    cnt[q] = acc_cnt[4 * (size_t)i + q];
    const int* k = acc_box + 24 * (size_t)i + 6 * q;
    bb[q] = NodeBox{{val_of(k[0]), val_of(k[1]), val_of(k[2])}, {val_of(k[3]), val_of(k[4]), val_of(k[5])}};
  }
  const Split s = decide_split(cnt, bb);
  const uint32_t mid = s.fallback ? (n.end + n.start) / 2 : n.start + s.left;
  l.start = n.start;
  l.end = r.start = mid;
  r.end = n.end;
  l.flags = r.flags = 0u;  // the median split's boxes, empty so far, grow in level_scatter_kernel
  set_box(l, s.l);
  set_box(r, s.r);
  l.depth = r.depth = n.depth + 1;
  l.tree = r.tree = n.tree;
  l.left = r.left = NONE;
  l.sub = r.sub = NONE;
  return s.fallback;
}

// One thread per node of the level: the split decision, the two children
// (slots claimed per warp, prepared for the next level at once: a launch of
// their own cost 8 us a level), and the exclusive per-bucket prefix of the node's
// chunk counts (big nodes: appended to big_list for the block-wide scan).
__global__ void level_decide_kernel(const uint32_t* __restrict__ lvl, uint32_t L, BNode* __restrict__ pool,
                                    const uint32_t* __restrict__ acc_cnt, const int* __restrict__ acc_box,
                                    const uint4* __restrict__ chunk_cnt, uint4* __restrict__ chunk_prefix,
                                    LevelCounters* lcs, BuildCounters* bc, uint32_t* __restrict__ big_list,
                                    uint32_t big_cap, uint32_t pool_cap, SplitRule rule, LevelBuffers next,
                                    uint32_t* __restrict__ ended) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lb = lvl[L], next_base = lvl[L + 1], W = next_base - lb;
  LevelCounters* lc = lcs + L;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < W; i0 += stride) {
    const uint32_t i = i0 + lane;
    BNode n;
    bool active = false, fallback = false;
    BNode l{}, r{};
    if (i < W) {
      n = pool[lb + i];
      active = (n.flags & F_ACTIVE) != 0;
      if (active) fallback = split_node(n, i, acc_cnt, acc_box, l, r);
    }
    const uint32_t base = next_base + warp_claim(&lc->children, active ? 2u : 0u, lane);
    const uint32_t n_sah = __popc(__ballot_sync(0xffffffffu, active && !fallback));
    const uint32_t n_med = __popc(__ballot_sync(0xffffffffu, active && fallback));
    if (lane == 0 && n_sah) atomicAdd(&bc->sah, (unsigned long long)n_sah);
    if (lane == 0 && n_med) atomicAdd(&bc->fallback, (unsigned long long)n_med);
    const bool fits = active && base + 1 < pool_cap;
    const bool big = fits && !fallback && n.nchunks > kBigChunks;
    const uint32_t slot = warp_claim(&lc->big, big ? 1u : 0u, lane);
    if (active && !fits) {  // the host gives up on the build; no kernel may scatter this node
      bc->overflow = 1u;
      pool[lb + i].flags = n.flags & ~F_ACTIVE;
    }
    prepare_node(fits, l, base, base - next_base, L + 1, rule, next, lcs, bc, ended);
    prepare_node(fits, r, base + 1, base + 1 - next_base, L + 1, rule, next, lcs, bc, ended);
    if (!fits) continue;
    if (l.start == l.end || r.start == r.end) bc->unfit = 1u;
    pool[base] = l;
    pool[base + 1] = r;
    pool[lb + i].left = base;
    if (fallback) pool[lb + i].flags = n.flags | F_FALLBACK;
    if (fallback || n.nchunks == 0) continue;
    if (big && slot < big_cap) {
      big_list[slot] = lb + i;
      continue;
    }
    uint4 run = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t j = 0; j < n.nchunks; j++) {
      const uint4 v = chunk_cnt[n.cbase + j];
      chunk_prefix[n.cbase + j] = run;
      run.x += v.x;
      run.y += v.y;
      run.z += v.z;
      run.w += v.w;
    }
  }
}

// Exclusive per-bucket prefix of the chunk counts of the big nodes, one block
// per node: each thread takes kPerThread consecutive chunks of a tile, the
// block scans the thread totals (warp shuffles, then the warp totals).
constexpr uint32_t kPerThread = 4;
// The last blocks run the median splits meanwhile: Rust's
// select_nth_unstable_by on the node's range, one thread per node.
__global__ void __launch_bounds__(kBlock) level_prefix_select_kernel(
    const uint32_t* __restrict__ lvl, const LevelCounters* lcs, uint32_t L, const BNode* __restrict__ pool,
    const uint32_t* __restrict__ big_list, uint32_t big_cap, const uint4* __restrict__ chunk_cnt,
    uint4* __restrict__ chunk_prefix, const float4* __restrict__ pbox, uint32_t* __restrict__ order) {
  const uint32_t lb = lvl[L], W = lvl[L + 1] - lb;
  for (uint32_t i = (gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x; i < W; i += gridDim.x * blockDim.x) {
    const BNode n = pool[lb + i];
    if (!(n.flags & F_FALLBACK)) continue;
    const uint32_t count = n.end - n.start;
    if (count / 2 == 0) continue;
    const int axis = split_axis(box_of(n));
    RustSelectNth<uint32_t, CentreLess> sel(CentreLess{&pbox[0].x + axis, 4u});
    sel.run(order + n.start, count, count / 2);
  }
  __shared__ uint4 warp_total[kWarps];
  __shared__ uint4 carry_s;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t nbig = min(lcs[L].big, big_cap);
  for (uint32_t b = blockIdx.x; b < nbig; b += gridDim.x) {
    const BNode n = pool[big_list[b]];
    uint4 carry = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t t0 = 0; t0 < n.nchunks; t0 += kBlock * kPerThread) {
      const uint32_t j0 = t0 + threadIdx.x * kPerThread;
      uint4 v[kPerThread];
      uint4 sum = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (uint32_t k = 0; k < kPerThread; k++) {
        v[k] = j0 + k < n.nchunks ? chunk_cnt[n.cbase + j0 + k] : make_uint4(0u, 0u, 0u, 0u);
        sum.x += v[k].x;
        sum.y += v[k].y;
        sum.z += v[k].z;
        sum.w += v[k].w;
      }
      uint4 inc = sum;  // inclusive scan of the thread totals inside the warp
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, inc.x, o), y = __shfl_up_sync(0xffffffffu, inc.y, o);
        const uint32_t z = __shfl_up_sync(0xffffffffu, inc.z, o), w = __shfl_up_sync(0xffffffffu, inc.w, o);
        if (lane >= (uint32_t)o) {
          inc.x += x;
          inc.y += y;
          inc.z += z;
          inc.w += w;
        }
      }
      if (lane == 31) warp_total[warp] = inc;
      __syncthreads();
      uint4 before = carry;  // carry + earlier warps of the tile
      for (uint32_t q = 0; q < warp; q++) {
        const uint4 t = warp_total[q];
        before.x += t.x;
        before.y += t.y;
        before.z += t.z;
        before.w += t.w;
      }
      uint4 run = make_uint4(before.x + inc.x - sum.x, before.y + inc.y - sum.y, before.z + inc.z - sum.z,
                             before.w + inc.w - sum.w);
#pragma unroll
      for (uint32_t k = 0; k < kPerThread; k++) {
        if (j0 + k < n.nchunks) chunk_prefix[n.cbase + j0 + k] = run;
        run.x += v[k].x;
        run.y += v[k].y;
        run.z += v[k].z;
        run.w += v[k].w;
      }
      if (threadIdx.x == kBlock - 1) carry_s = run;  // the last thread's running total ends the tile
      __syncthreads();
      carry = carry_s;
      __syncthreads();
    }
  }
}

// End of the level whose first node is `first`: the children that were claimed,
// as far as the pool holds them. Children are claimed in pairs from `first` on
// and a pair is written when both of its slots lie below `cap`, so every node
// below the end that this returns has been written: the levels that are queued
// behind an overflow see no other node, and none of theirs fits any more.
__host__ __device__ constexpr uint32_t level_end(uint32_t first, uint32_t children, uint32_t cap) {
  const uint32_t room = (cap - first) & ~1u;
  return first + (children < room ? children : room);
}
static_assert(level_end(10, 4, 14) == 14 && level_end(10, 4, 13) == 12 && level_end(10, 4, 11) == 10 &&
                  level_end(10, 0, 64) == 10 && level_end(10, 6, 10) == 10,
              "whole pairs below the cap");

// SAH nodes: each chunk writes its primitives to their bucket-ordered slots of
// the other order array; a median-split node's are copied as they stand. Also
// closes the level: the next level's end, from the children that
// level_decide_kernel claimed (decide ran before this launch).
__global__ void level_scatter_kernel(uint32_t* __restrict__ lvl, uint32_t L, const LevelCounters* lcs, BNode* __restrict__ pool,
                                     const float4* __restrict__ pbox,
                                     const uint32_t* __restrict__ chunk_node, const uint32_t* __restrict__ order,
                                     const uint8_t* __restrict__ bucket, const uint32_t* __restrict__ acc_cnt,
                                     const uint32_t* __restrict__ chunk_prefix, uint32_t* __restrict__ scratch,
                                     uint32_t pool_cap) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t lb = lvl[L];
  const uint32_t total = lcs[L].chunks;
  if (blockIdx.x == 0 && threadIdx.x == 0) lvl[L + 2] = level_end(lvl[L + 1], lcs[L].children, pool_cap);
  for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < total; c += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t id = chunk_node[c];
    const BNode n = pool[id];
    if (!(n.flags & F_ACTIVE)) continue;
    if (n.flags & F_FALLBACK) {
      uint32_t s, e;
      chunk_range(n, c, s, e);
      const uint32_t mid = pool[n.left].end;
      int lo[2][3], hi[2][3];
      for (int c2 = 0; c2 < 2; c2++)
        for (int k = 0; k < 3; k++) {
          lo[c2][k] = key_of(INFINITY);
          hi[c2][k] = key_of(-INFINITY);
        }
      for (uint32_t i = s + lane; i < e; i += 32) {
        const uint32_t p = order[i];
        scratch[i] = p;
        const float4 a = pbox[2 * (size_t)p], b = pbox[2 * (size_t)p + 1];
        const int c2 = i >= mid;
        const int kl[3] = {key_of(a.x), key_of(a.y), key_of(a.z)}, kh[3] = {key_of(b.x), key_of(b.y), key_of(b.z)};
#pragma unroll
        for (int k = 0; k < 3; k++) {
          lo[0][k] = min(lo[0][k], c2 ? lo[0][k] : kl[k]);
          hi[0][k] = max(hi[0][k], c2 ? hi[0][k] : kh[k]);
          lo[1][k] = min(lo[1][k], c2 ? kl[k] : lo[1][k]);
          hi[1][k] = max(hi[1][k], c2 ? kh[k] : hi[1][k]);
        }
      }
#pragma unroll
      for (int c2 = 0; c2 < 2; c2++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const int l = __reduce_min_sync(0xffffffffu, lo[c2][k]), h = __reduce_max_sync(0xffffffffu, hi[c2][k]);
          if (lane == 0) {
            atomicMin(&pool[n.left + c2].lo[k], l);
            atomicMax(&pool[n.left + c2].hi[k], h);
          }
        }
      continue;
    }
    const uint32_t li = id - lb;
    uint32_t base[4];
    uint32_t run = n.start;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      base[q] = run + chunk_prefix[4 * (size_t)c + q];
      run += acc_cnt[4 * (size_t)li + q];
    }
    uint32_t s, e;
    chunk_range(n, c, s, e);
    for (uint32_t i0 = s; i0 < e; i0 += 32) {
      const uint32_t i = i0 + lane;
      const bool valid = i < e;
      const uint32_t p = valid ? order[i] : 0u;
      const uint32_t bk = valid ? bucket[i] : 4u;
      uint32_t dest = 0;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t m = __ballot_sync(0xffffffffu, bk == (uint32_t)q);
        if (bk == (uint32_t)q) dest = base[q] + __popc(m & lt_mask);
        base[q] += __popc(m);
      }
      if (valid) scratch[dest] = p;
    }
  }
}

// ---- subtrees -------------------------------------------------------------

struct SmallNode {
  int lo[3], hi[3];
  uint16_t start, end, left, size, pre;  // left: NO_CHILD for a leaf; pre: place in the subtree's pre-order
  uint16_t pending;
};
constexpr uint16_t NO_CHILD = 0xFFFF;
struct SmallTree {
  int lo[3][kSmall], hi[3][kSmall];  // boxes as keys
  float cen[3][kSmall];
  uint32_t prim[kSmall], order[kSmall], moved[kSmall];
  SmallNode node[2 * kSmall];
  uint16_t level[kSmall + 2];  // first node of each level
  uint32_t count, sah, fallback, base;
};
constexpr uint32_t kSmallThreads = 128, kSmallWarps = kSmallThreads / 32;

// The two children of a node that is split at mid, and the median split's order.
__device__ __forceinline__ void small_children(SmallTree& S, SmallNode& n, const Split& s, uint32_t mid, const float* cen) {
  const uint32_t child = atomicAdd(&S.count, 2u), start = n.start, end = n.end;
  n.left = (uint16_t)child;
  for (uint32_t c = 0; c < 2; c++) {
    SmallNode& q = S.node[child + c];
    const NodeBox& b = c ? s.r : s.l;
    q.lo[0] = key_of(b.lo.x);
    q.lo[1] = key_of(b.lo.y);
    q.lo[2] = key_of(b.lo.z);
    q.hi[0] = key_of(b.hi.x);
    q.hi[1] = key_of(b.hi.y);
    q.hi[2] = key_of(b.hi.z);
    q.start = (uint16_t)(c ? mid : start);
    q.end = (uint16_t)(c ? end : mid);
    q.pending = s.fallback ? 1 : 0;
  }
  atomicAdd(s.fallback ? &S.fallback : &S.sah, 1u);
  if (s.fallback) {
    RustSelectNth<uint32_t, CentreLess> sel(CentreLess{cen, 0u});
    sel.run(S.order + start, end - start, (end - start) / 2);
  }
}

// Nodes of at most this many primitives (16: their bucket numbers fit a word)
// are taken by a lane each: they are three of four nodes, and a warp each spends
// most of its instructions on reductions over empty lanes (2.1 M triangles: the
// kernel takes 520 us by warps alone, 365 with lanes).
constexpr uint32_t kLaneNode = 16;

__device__ __forceinline__ bool lane_node(SmallTree& S, uint32_t j, uint32_t bin_size, bool may_split) {
  SmallNode& n = S.node[j];
  const uint32_t start = n.start, end = n.end, count = end - start;
  if (n.pending) {
    int lo[3] = {key_of(INFINITY), key_of(INFINITY), key_of(INFINITY)};
    int hi[3] = {key_of(-INFINITY), key_of(-INFINITY), key_of(-INFINITY)};
    for (uint32_t i = start; i < end; i++) {
      const uint32_t p = S.order[i];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        lo[k] = min(lo[k], S.lo[k][p]);
        hi[k] = max(hi[k], S.hi[k][p]);
      }
    }
    for (int k = 0; k < 3; k++) {
      n.lo[k] = lo[k];
      n.hi[k] = hi[k];
    }
  }
  n.left = NO_CHILD;
  if (!(may_split && count > bin_size)) return true;
  const NodeBox nb{{val_of(n.lo[0]), val_of(n.lo[1]), val_of(n.lo[2])}, {val_of(n.hi[0]), val_of(n.hi[1]), val_of(n.hi[2])}};
  const int axis = split_axis(nb);
  const float a0 = comp(nb.lo, axis), step = (comp(nb.hi, axis) - a0) / 4.0f;
  const float* cen = S.cen[axis];
  uint32_t cnt[4] = {0, 0, 0, 0}, buckets = 0;
  int bx[4][6];
#pragma unroll
  for (int b = 0; b < 4; b++) {
    bx[b][0] = bx[b][1] = bx[b][2] = key_of(INFINITY);
    bx[b][3] = bx[b][4] = bx[b][5] = key_of(-INFINITY);
  }
  for (uint32_t i = 0; i < count; i++) {
    const uint32_t p = S.order[start + i];
    const uint32_t bk = bucket_of(cen[p], a0, step);
    buckets |= bk << (2 * i);
    const int k[6] = {S.lo[0][p], S.lo[1][p], S.lo[2][p], S.hi[0][p], S.hi[1][p], S.hi[2][p]};
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const bool in = bk == (uint32_t)q;
      cnt[q] += in;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        bx[q][c] = in ? min(bx[q][c], k[c]) : bx[q][c];
        bx[q][3 + c] = in ? max(bx[q][3 + c], k[3 + c]) : bx[q][3 + c];
      }
    }
  }
  NodeBox bb[4];
#pragma unroll
  for (int q = 0; q < 4; q++)
    bb[q] = NodeBox{{val_of(bx[q][0]), val_of(bx[q][1]), val_of(bx[q][2])}, {val_of(bx[q][3]), val_of(bx[q][4]), val_of(bx[q][5])}};
  const Split s = decide_split(cnt, bb);
  const uint32_t mid = s.fallback ? (start + end) / 2 : start + s.left;
  if (mid == start || mid == end) return false;
  small_children(S, n, s, mid, cen);
  if (s.fallback) return true;
  uint32_t base[4] = {start, start + cnt[0], start + cnt[0] + cnt[1], start + cnt[0] + cnt[1] + cnt[2]};
  for (uint32_t i = 0; i < count; i++) {
    const uint32_t bk = (buckets >> (2 * i)) & 3u;
    uint32_t dest = 0;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (bk == (uint32_t)q) dest = base[q]++;
    S.moved[dest] = S.order[start + i];
  }
  for (uint32_t i = start; i < end; i++) S.order[i] = S.moved[i];
  return true;
}

// One node by one warp: its box if it is not known, then leaf or split, as the
// level kernels do it. False, and a leaf, where a child would be empty.
__device__ __forceinline__ bool small_node(SmallTree& S, uint32_t j, uint32_t bin_size, bool may_split) {
  const uint32_t lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
  SmallNode& n = S.node[j];
  const uint32_t start = n.start, end = n.end, count = end - start;
  if (n.pending) {
    int lo[3] = {key_of(INFINITY), key_of(INFINITY), key_of(INFINITY)};
    int hi[3] = {key_of(-INFINITY), key_of(-INFINITY), key_of(-INFINITY)};
    for (uint32_t i = start + lane; i < end; i += 32) {
      const uint32_t p = S.order[i];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        lo[k] = min(lo[k], S.lo[k][p]);
        hi[k] = max(hi[k], S.hi[k][p]);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      lo[k] = __reduce_min_sync(0xffffffffu, lo[k]);
      hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
      if (lane == 0) {
        n.lo[k] = lo[k];
        n.hi[k] = hi[k];
      }
    }
    __syncwarp();
  }
  if (lane == 0) n.left = NO_CHILD;
  if (!(may_split && count > bin_size)) return true;
  const NodeBox nb{{val_of(n.lo[0]), val_of(n.lo[1]), val_of(n.lo[2])}, {val_of(n.hi[0]), val_of(n.hi[1]), val_of(n.hi[2])}};
  const int axis = split_axis(nb);
  const float a0 = comp(nb.lo, axis), step = (comp(nb.hi, axis) - a0) / 4.0f;
  const float* cen = S.cen[axis];
  uint32_t cnt[4] = {0, 0, 0, 0};
  int bx[4][6];
#pragma unroll
  for (int b = 0; b < 4; b++) {
    bx[b][0] = bx[b][1] = bx[b][2] = key_of(INFINITY);
    bx[b][3] = bx[b][4] = bx[b][5] = key_of(-INFINITY);
  }
  for (uint32_t i = start + lane; i < end; i += 32) {
    const uint32_t p = S.order[i];
    const uint32_t bk = bucket_of(cen[p], a0, step);
    const int k[6] = {S.lo[0][p], S.lo[1][p], S.lo[2][p], S.hi[0][p], S.hi[1][p], S.hi[2][p]};
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (bk == (uint32_t)q) {
        cnt[q]++;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          bx[q][c] = min(bx[q][c], k[c]);
          bx[q][3 + c] = max(bx[q][3 + c], k[3 + c]);
        }
      }
  }
  NodeBox bb[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    cnt[q] = __reduce_add_sync(0xffffffffu, cnt[q]);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      bx[q][c] = __reduce_min_sync(0xffffffffu, bx[q][c]);
      bx[q][3 + c] = __reduce_max_sync(0xffffffffu, bx[q][3 + c]);
    }
    bb[q] = NodeBox{{val_of(bx[q][0]), val_of(bx[q][1]), val_of(bx[q][2])}, {val_of(bx[q][3]), val_of(bx[q][4]), val_of(bx[q][5])}};
  }
  const Split s = decide_split(cnt, bb);
  const uint32_t mid = s.fallback ? (start + end) / 2 : start + s.left;  // the range starts at a whole number
  if (mid == start || mid == end) return false;
  if (lane == 0) small_children(S, n, s, mid, cen);
  __syncwarp();
  if (s.fallback) return true;
  uint32_t base[4] = {start, start + cnt[0], start + cnt[0] + cnt[1], start + cnt[0] + cnt[1] + cnt[2]};
  for (uint32_t i0 = start; i0 < end; i0 += 32) {
    const uint32_t i = i0 + lane;
    const bool valid = i < end;
    const uint32_t p = valid ? S.order[i] : 0u;
    const uint32_t bk = valid ? bucket_of(cen[p], a0, step) : 4u;
    uint32_t dest = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t m = __ballot_sync(0xffffffffu, bk == (uint32_t)q);
      if (bk == (uint32_t)q) dest = base[q] + __popc(m & lt_mask);
      base[q] += __popc(m);
    }
    if (valid) S.moved[dest] = p;
  }
  __syncwarp();
  for (uint32_t i = start + lane; i < end; i += 32) S.order[i] = S.moved[i];
  return true;
}

// Every node that left the level rounds: a subtree of at most `small`
// primitives is built in shared memory, level by level, and added to the pool
// in that order (children next to each other, behind their parents); a larger
// leaf is closed. Afterwards order_a holds the final order, and every node has
// its subtree's size and its place in that subtree's pre-order.
__global__ void __launch_bounds__(kSmallThreads) small_trees_kernel(uint32_t small, uint32_t top,
                                                                    const uint32_t* __restrict__ ended,
                                                                    uint32_t bin_size, uint32_t max_depth,
                                                                    BNode* __restrict__ pool, uint32_t* order_a,
                                                                    const uint32_t* order_b,
                                                                    const float4* __restrict__ pbox, BuildCounters* bc) {
  __shared__ SmallTree S;
  const uint32_t warp = threadIdx.x >> 5, total = bc->ended;
  for (uint32_t e = blockIdx.x; e < total; e += gridDim.x) {
    const uint32_t id = ended[e];
    const BNode root = pool[id];
    const uint32_t count = root.end - root.start;
    const uint32_t* src = (root.flags & F_IN_B ? order_b : order_a) + root.start;
    __syncthreads();  // the previous subtree has been written, and every thread has read this root
    if (count > small) {
      if (root.flags & F_IN_B)
        for (uint32_t i = threadIdx.x; i < count; i += kSmallThreads) order_a[root.start + i] = src[i];
      if (threadIdx.x == 0) {
        pool[id].cbase = 1;
        pool[id].nchunks = 0;
        pool[id].sub = id;
        atomicMax(&bc->max_depth, root.depth);
      }
      continue;
    }
    for (uint32_t i = threadIdx.x; i < count; i += kSmallThreads) {
      const uint32_t p = src[i];
      const float4 a = pbox[2 * (size_t)p], b = pbox[2 * (size_t)p + 1];
      S.prim[i] = p;
      S.order[i] = i;
      S.lo[0][i] = key_of(a.x);
      S.lo[1][i] = key_of(a.y);
      S.lo[2][i] = key_of(a.z);
      S.hi[0][i] = key_of(b.x);
      S.hi[1][i] = key_of(b.y);
      S.hi[2][i] = key_of(b.z);
      S.cen[0][i] = (a.x + b.x) * 0.5f;
      S.cen[1][i] = (a.y + b.y) * 0.5f;
      S.cen[2][i] = (a.z + b.z) * 0.5f;
    }
    if (threadIdx.x == 0) {
      SmallNode& n = S.node[0];
      for (int k = 0; k < 3; k++) {
        n.lo[k] = root.lo[k];
        n.hi[k] = root.hi[k];
      }
      n.start = 0;
      n.end = (uint16_t)count;
      n.pending = (root.flags & F_BOX_PENDING) ? 1 : 0;
      S.count = 1;
      S.sah = S.fallback = 0;
    }
    __syncthreads();
    uint32_t first = 0, last = 1, levels = 0;
    while (first < last) {
      if (threadIdx.x == 0) S.level[levels] = (uint16_t)first;
      const bool may_split = root.depth + levels < max_depth;
      for (uint32_t j = first + warp; j < last; j += kSmallWarps)
        if (S.node[j].end - S.node[j].start > (int)kLaneNode && !small_node(S, j, bin_size, may_split)) bc->unfit = 1u;
      for (uint32_t j = first + threadIdx.x; j < last; j += kSmallThreads)
        if (S.node[j].end - S.node[j].start <= (int)kLaneNode && !lane_node(S, j, bin_size, may_split)) bc->unfit = 1u;
      __syncthreads();
      levels++;
      first = last;
      last = S.count;
      __syncthreads();
    }
    if (threadIdx.x == 0) S.level[levels] = (uint16_t)last;
    __syncthreads();
    for (uint32_t l = levels; l-- > 0;) {
      for (uint32_t j = S.level[l] + threadIdx.x; j < S.level[l + 1]; j += kSmallThreads) {
        const uint32_t c = S.node[j].left;
        S.node[j].size = c == NO_CHILD ? 1 : (uint16_t)(1 + S.node[c].size + S.node[c + 1].size);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      S.node[0].pre = 0;
      S.base = last > 1 ? top + atomicAdd(&bc->added, last - 1) : 0u;
      if (S.sah) atomicAdd(&bc->sah, (unsigned long long)S.sah);
      if (S.fallback) atomicAdd(&bc->fallback, (unsigned long long)S.fallback);
      atomicMax(&bc->max_depth, root.depth + levels - 1);
    }
    __syncthreads();
    for (uint32_t l = 0; l < levels; l++) {
      for (uint32_t j = S.level[l] + threadIdx.x; j < S.level[l + 1]; j += kSmallThreads) {
        const uint32_t c = S.node[j].left, pre = S.node[j].pre;
        if (c != NO_CHILD) {
          S.node[c].pre = (uint16_t)(pre + 1);
          S.node[c + 1].pre = (uint16_t)(pre + 1 + S.node[c].size);
        }
        const SmallNode& n = S.node[j];
        BNode o;
        for (int k = 0; k < 3; k++) {
          o.lo[k] = n.lo[k];
          o.hi[k] = n.hi[k];
        }
        o.start = root.start + n.start;
        o.end = root.start + n.end;
        o.depth = root.depth + l;
        o.left = c == NO_CHILD ? NONE : S.base + c - 1;
        o.tree = root.tree;
        o.flags = 0;
        o.cbase = n.size;
        o.nchunks = pre;
        o.sub = id;
        o.pad = 0;
        pool[j == 0 ? id : S.base + j - 1] = o;
      }
      __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < count; i += kSmallThreads) order_a[root.start + i] = S.prim[S.order[i]];
  }
}

// ---- numbering and emission --------------------------------------------

// Adds the inner nodes' shares of their geometry's root area to tree_share
// (HostBuilt::geom_line_nodes). Every thread of the block calls; blocks whose
// nodes are one tree's add once (a build of 2.1 M triangles takes 2.01 ms with and
// without).
__device__ __forceinline__ void add_shares(bool inner, uint32_t tree, const NodeBox& box, const BNode* pool,
                                           unsigned long long* tree_share) {
  __shared__ uint32_t sums[kWarps];
  __shared__ uint32_t tree_s;
  uint32_t share = 0;
  if (inner) {
    const float a = half_area(box), b = half_area(box_of(pool[tree]));
    if (a > 0.0f && a <= b && b < INFINITY) share = (uint32_t)(a / b * (float)kShareUnit);
  }
  if (threadIdx.x == 0) tree_s = tree;
  __syncthreads();
  if (__syncthreads_and(tree == tree_s || share == 0u)) {
    const uint32_t sum = __reduce_add_sync(0xffffffffu, share);  // 32 shares of at most 2^24
    if ((threadIdx.x & 31u) == 0) sums[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long total = 0;
      for (uint32_t w = 0; w < kWarps; w++) total += sums[w];
      if (total) atomicAdd(tree_share + tree_s, total);
    }
  } else if (share) {
    atomicAdd(tree_share + tree, (unsigned long long)share);
  }
}

// Numbering above the subtrees, by one block: subtree sizes bottom-up (in
// cbase), the geometries' first nodes by a scan of their trees' sizes, and the
// reference's pre-order numbers top-down.
constexpr uint32_t kNumberThreads = 1024;
__global__ void __launch_bounds__(kNumberThreads) top_numbering_kernel(const uint32_t* __restrict__ lvl, uint32_t levels,
                                                                       uint32_t G, BNode* __restrict__ pool,
                                                                       uint32_t* __restrict__ tree_end,
                                                                       uint32_t* __restrict__ tree_nodes,
                                                                       uint32_t* __restrict__ pre,
                                                                       unsigned long long* __restrict__ tree_share) {
  __shared__ uint32_t warp_sums[kNumberThreads / 32], carry;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t l = levels; l-- > 0;) {
    for (uint32_t i = lvl[l] + threadIdx.x; i < lvl[l + 1]; i += kNumberThreads) {
      const uint32_t c = pool[i].left;
      if (pool[i].sub == NONE) pool[i].cbase = 1u + pool[c].cbase + pool[c + 1].cbase;  // nodes above are inner
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t g0 = 0; g0 < G; g0 += kNumberThreads) {
    const uint32_t g = g0 + threadIdx.x;
    const uint32_t size = g < G ? pool[g].cbase : 0u;
    const uint32_t inc = warp_inclusive_u32(size, lane);
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    uint32_t before = carry + inc - size, total = 0;
    for (uint32_t w = 0; w < kNumberThreads / 32; w++) {
      if (w < warp) before += warp_sums[w];
      total += warp_sums[w];
    }
    if (g < G) {
      pre[g] = before;
      tree_end[g] = before + size;
      tree_nodes[g] = size;
      tree_share[g] = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
  for (uint32_t l = 0; l < levels; l++) {
    for (uint32_t i = lvl[l] + threadIdx.x; i < lvl[l + 1]; i += kNumberThreads) {
      if (pool[i].sub != NONE) continue;
      const uint32_t c = pool[i].left, me = pre[i];
      pre[c] = me + 1;
      pre[c + 1] = me + 1 + pool[c].cbase;
    }
    __syncthreads();
  }
}

// Pre-order numbers of the subtrees' nodes, and which numbers are inner nodes.
__global__ void inner_flags_kernel(uint32_t T, const BNode* __restrict__ pool, uint32_t* __restrict__ pre,
                                   uint32_t* __restrict__ inner_at) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= T) return;
  const uint32_t sub = pool[id].sub;
  uint32_t g;
  if (sub == NONE || sub == id) {
    g = pre[id];
  } else {
    g = pre[sub] + pool[id].nchunks;
    pre[id] = g;
  }
  inner_at[g] = pool[id].left != NONE ? 1u : 0u;
}

__device__ __forceinline__ uint32_t code_of(uint32_t id, const BNode* pool, const uint32_t* pre, const uint32_t* rank) {
  const uint32_t g = pre[id];
  return pool[id].left != NONE ? rank[g] : (LEAF_BIT | (g - rank[g]));
}

__global__ void emit_nodes_kernel(uint32_t T, uint32_t G, const BNode* __restrict__ pool,
                                  const uint32_t* __restrict__ pre, const uint32_t* __restrict__ rank,
                                  const uint32_t* __restrict__ tree_end, DeviceBVHNode* __restrict__ forest,
                                  WideNode* __restrict__ wide, uint32_t* __restrict__ leaves,
                                  uint32_t* __restrict__ root_code, unsigned long long* __restrict__ tree_share) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  const BNode n = pool[id < T ? id : T - 1];
  const NodeBox b = box_of(n);
  const bool inner = n.left != NONE;
  add_shares(inner && id < T, n.tree, b, pool, tree_share);
  if (id >= T) return;
  const uint32_t g = pre[id];
  const uint32_t next = g + n.cbase;
  const uint32_t miss = next < tree_end[n.tree] ? next : INVALID_NEXT;
  float4* o = reinterpret_cast<float4*>(forest + g);  // DeviceBVHNode
  o[0] = make_float4(b.lo.x, b.lo.y, b.lo.z, __uint_as_float(inner ? g + 1 : miss));
  o[1] = make_float4(b.hi.x, b.hi.y, b.hi.z, __uint_as_float(miss));
  o[2] = make_float4(__uint_as_float(n.start), __uint_as_float(n.end), 0.0f, 0.0f);
  if (inner) {
    const NodeBox a = box_of(pool[n.left]), c = box_of(pool[n.left + 1]);
    float4* w = reinterpret_cast<float4*>(wide + rank[g]);  // WideNode
    w[0] = make_float4(a.lo.x, a.lo.y, a.lo.z, a.hi.x);
    w[1] = make_float4(a.hi.y, a.hi.z, c.lo.x, c.lo.y);
    w[2] = make_float4(c.lo.z, c.hi.x, c.hi.y, c.hi.z);
    w[3] = make_float4(__uint_as_float(code_of(n.left, pool, pre, rank)),
                       __uint_as_float(code_of(n.left + 1, pool, pre, rank)), 0.0f, 0.0f);
  } else {
    const uint32_t l = g - rank[g];
    leaves[2 * (size_t)l] = n.start;
    leaves[2 * (size_t)l + 1] = n.end;
  }
  if (id < G) root_code[id] = code_of(id, pool, pre, rank);
}

// indices_redirect and the 64 B triangle records in the sorted order.
// One thread per sorted triangle: its three vertices, copied (no arithmetic).
__global__ void emit_vertex_records_kernel(uint32_t N, const uint32_t* __restrict__ redirect,
                                           const uint32_t* __restrict__ idx, const float* __restrict__ vtx,
                                           VertexRecord* __restrict__ out) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < N; j += gridDim.x * blockDim.x) {
    const uint32_t p = __ldg(redirect + j);
    float v[9];
    for (int k = 0; k < 3; k++) {
      const float* q = vtx + 3 * (size_t)__ldg(idx + 3 * (size_t)p + k);
      v[3 * k] = __ldg(q);
      v[3 * k + 1] = __ldg(q + 1);
      v[3 * k + 2] = __ldg(q + 2);
    }
    float4* o = reinterpret_cast<float4*>(out + j);
    o[0] = make_float4(v[0], v[1], v[2], v[3]);
    o[1] = make_float4(v[4], v[5], v[6], v[7]);
    o[2] = make_float4(v[8], 0.0f, 0.0f, 0.0f);
  }
}

__global__ void emit_primitives_kernel(uint32_t N, const uint32_t* __restrict__ order, const uint32_t* __restrict__ idx,
                                       const float* __restrict__ vtx, uint32_t* __restrict__ redirect,
                                       TriRecord* __restrict__ tris) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < N; j += gridDim.x * blockDim.x) {
    const uint32_t p = order[j];
    redirect[j] = p;
    F3 v[3];
    for (int k = 0; k < 3; k++) {
      const float* q = vtx + 3 * (size_t)idx[3 * (size_t)p + k];
      v[k] = {q[0], q[1], q[2]};
    }
    const F3 e1 = {v[1].x - v[0].x, v[1].y - v[0].y, v[1].z - v[0].z};
    const F3 e2 = {v[2].x - v[0].x, v[2].y - v[0].y, v[2].z - v[0].z};
    F3 nrm = {e1.y * e2.z - e1.z * e2.y, e1.z * e2.x - e1.x * e2.z, e1.x * e2.y - e1.y * e2.x};
    const float mag_sq = nrm.x * nrm.x + nrm.y * nrm.y + nrm.z * nrm.z;
    if (mag_sq > 0.0f) {
      const float inv = 1.0f / sqrtf(mag_sq);
      nrm = {nrm.x * inv, nrm.y * inv, nrm.z * inv};
    }
    const float uu = e1.x * e1.x + e1.y * e1.y + e1.z * e1.z;
    const float uv = e1.x * e2.x + e1.y * e2.y + e1.z * e2.z;
    const float vv = e2.x * e2.x + e2.y * e2.y + e2.z * e2.z;
    const float inv_d = 1.0f / (uv * uv - uu * vv);
    float4* o = reinterpret_cast<float4*>(tris + j);
    o[0] = make_float4(v[0].x, v[0].y, v[0].z, nrm.x);
    o[1] = make_float4(e1.x, e1.y, e1.z, nrm.y);
    o[2] = make_float4(e2.x, e2.y, e2.z, nrm.z);
    o[3] = make_float4(uu, uv, vv, inv_d);
  }
}

// True when box s is flat on some axis and lies on a face plane of box a,
// which is not flat there (the host build's flat_on_boundary: a ray with a
// zero direction component and its origin in that plane fails a's slab test
// but passes s's, so the four-child walk, which skips the boxes of opened
// nodes, must not open a node above such a child).
__device__ __forceinline__ bool flat_on_boundary(const NodeBox& s, const NodeBox& a) {
  const float sl[3] = {s.lo.x, s.lo.y, s.lo.z}, sh[3] = {s.hi.x, s.hi.y, s.hi.z};
  const float al[3] = {a.lo.x, a.lo.y, a.lo.z}, ah[3] = {a.hi.x, a.hi.y, a.hi.z};
  for (int k = 0; k < 3; k++)
    if (sl[k] == sh[k] && al[k] != ah[k] && (al[k] == sl[k] || ah[k] == sl[k])) return true;
  return false;
}

__device__ __forceinline__ bool openable(uint32_t x, const uint32_t anc[2], const BNode* pool) {
  const NodeBox bx = box_of(pool[x]);
  for (uint32_t c = pool[x].left; c <= pool[x].left + 1; c++) {
    const NodeBox bc = box_of(pool[c]);
    if (flat_on_boundary(bc, bx)) return false;
    for (int a = 0; a < 2; a++)
      if (anc[a] != NONE && flat_on_boundary(bc, box_of(pool[anc[a]]))) return false;
  }
  return true;
}

// Four-child collapse of binary inner node b: open the inner slot with the
// largest surface area (first of equals) until 4 slots are used, skipping
// nodes that openable() refuses (the host build's emit_wide4).
__device__ __forceinline__ int collapse_slots(uint32_t b, const BNode* pool, uint32_t slot[4]) {
  uint32_t anc[4][2];
  int n = 0;
  slot[n++] = pool[b].left;
  slot[n++] = pool[b].left + 1;
  for (int k = 0; k < 4; k++) anc[k][0] = anc[k][1] = NONE;
  while (n < 4) {
    int best = -1;
    float best_area = -1.0f;
    for (int k = 0; k < n; k++) {
      if (pool[slot[k]].left == NONE || !openable(slot[k], anc[k], pool)) continue;
      const float a = half_area(box_of(pool[slot[k]]));
      if (best < 0 || a > best_area) {
        best = k;
        best_area = a;
      }
    }
    if (best < 0) break;
    const uint32_t open = slot[best];
    const uint32_t up0 = open, up1 = anc[best][0];
    for (int k = n; k > best + 1; k--) {
      slot[k] = slot[k - 1];
      anc[k][0] = anc[k - 1][0];
      anc[k][1] = anc[k - 1][1];
    }
    slot[best] = pool[open].left;
    slot[best + 1] = pool[open].left + 1;
    for (int k = best; k <= best + 1; k++) {
      anc[k][0] = up0;
      anc[k][1] = up1;
    }
    n++;
  }
  return n;
}

__device__ __forceinline__ uint4 collapse(uint32_t b, const BNode* pool) {
  uint32_t slot[4];
  const int n = collapse_slots(b, pool, slot);
  return make_uint4(slot[0], slot[1], n > 2 ? slot[2] : NONE, n > 3 ? slot[3] : NONE);
}

// Four-child layout: the binary nodes that root a four-child node ("collapse
// roots") are marked top-down, their slots are kept, one scan numbers the roots
// in pool order and one launch emits every node. A collapse is a chain of
// dependent loads, the marks only follow its result: above the subtrees every
// inner node is collapsed at once, root or not, and one block then walks the
// levels (2 M triangles: 200 us as a launch per level that collapses its roots).
__global__ void wide4_slots_kernel(uint32_t top, const BNode* __restrict__ pool, uint4* __restrict__ slots) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < top && pool[i].sub == NONE) slots[i] = collapse(i, pool);
}

// Marks the slots of collapse root b that are roots themselves.
__device__ __forceinline__ void mark_slots(const uint4& s, uint32_t level, const BNode* pool, volatile uint32_t* croot,
                                           volatile uint32_t* level4, uint32_t& deepest) {
  const uint32_t slot[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (slot[q] != NONE && pool[slot[q]].left != NONE) {
      croot[slot[q]] = 1u;
      level4[slot[q]] = level + 1u;
      deepest = max(deepest, level + 1u);
    }
}

__global__ void __launch_bounds__(kNumberThreads) wide4_top_kernel(const uint32_t* __restrict__ lvl, uint32_t levels,
                                                                   uint32_t G, const BNode* __restrict__ pool,
                                                                   const uint4* __restrict__ slots,
                                                                   volatile uint32_t* croot, volatile uint32_t* level4,
                                                                   uint32_t* __restrict__ max_level4) {
  uint32_t deepest = 0;
  for (uint32_t g = threadIdx.x; g < G; g += kNumberThreads)
    if (pool[g].left != NONE) {
      croot[g] = level4[g] = 1u;
      deepest = 1u;
    }
  __syncthreads();
  for (uint32_t l = 0; l < levels; l++) {
    for (uint32_t i = lvl[l] + threadIdx.x; i < lvl[l + 1]; i += kNumberThreads)
      if (croot[i] && pool[i].sub == NONE) mark_slots(slots[i], level4[i], pool, croot, level4, deepest);
    __syncthreads();
  }
  deepest = __reduce_max_sync(0xffffffffu, deepest);
  if ((threadIdx.x & 31u) == 0 && deepest) atomicMax(max_level4, deepest);
}

// The same below a subtree's root, a warp per subtree: its nodes lie behind the
// root's children in level order.
__global__ void wide4_mark_small_kernel(const uint32_t* __restrict__ ended, const BuildCounters* bc,
                                        const BNode* __restrict__ pool, uint4* __restrict__ slots,
                                        volatile uint32_t* croot, volatile uint32_t* level4,
                                        uint32_t* __restrict__ max_level4) {
  const uint32_t lane = threadIdx.x & 31u, total = bc->ended;
  for (uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < total; e += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t id = ended[e];
    const uint32_t m = pool[id].cbase, first = pool[id].left;  // node j > 0 of the subtree is pool[first + j - 1]
    if (m <= 1) continue;
    uint32_t depth = pool[id].depth, deepest = 0;
    for (uint32_t j = 0; j < m;) {
      // the nodes of one level, as far as a warp reaches
      const uint32_t k = j + lane, node = k == 0 ? id : first + k - 1;
      const bool in = k < m && pool[node].depth == depth;
      if (in && croot[node]) {
        const uint4 s = collapse(node, pool);
        slots[node] = s;
        mark_slots(s, level4[node], pool, croot, level4, deepest);
      }
      __syncwarp();
      const uint32_t taken = __popc(__ballot_sync(0xffffffffu, in));
      j += taken;
      if (taken < 32u) depth++;
    }
    deepest = __reduce_max_sync(0xffffffffu, deepest);
    if (lane == 0 && deepest) atomicMax(max_level4, deepest);
  }
}

__global__ void wide4_emit_kernel(uint32_t T, bool packed, const BNode* __restrict__ pool, const uint32_t* __restrict__ croot,
                                  const uint4* __restrict__ slots, const uint32_t* __restrict__ index4,
                                  const uint32_t* __restrict__ pre, const uint32_t* __restrict__ rank,
                                  Wide4Node* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T || !croot[i]) return;
  const uint4 s = slots[i];
  const uint32_t slot[4] = {s.x, s.y, s.z, s.w};
  float4* o = reinterpret_cast<float4*>(out + index4[i]);  // Wide4Child: lo_x lo_y hi_x hi_y lo_z hi_z code pad
#pragma unroll
  for (int k = 0; k < 4; k++) {
    NodeBox b{{NAN, NAN, NAN}, {NAN, NAN, NAN}};
    uint32_t code = EMPTY_SLOT;
    if (slot[k] != NONE) {
      const BNode c = pool[slot[k]];
      b = box_of(c);
      if (c.left != NONE) {
        code = index4[slot[k]];
      } else {
        const uint32_t g = pre[slot[k]], leaf = g - rank[g];
        code = packed ? packed_leaf(leaf, c.start, c.end) : (LEAF_BIT | leaf);
      }
    }
    o[2 * k] = make_float4(b.lo.x, b.lo.y, b.hi.x, b.hi.y);
    o[2 * k + 1] = make_float4(b.lo.z, b.hi.z, __uint_as_float(code), 0.0f);
  }
}

// ---- host side -------------------------------------------------------------

// Stream-ordered scratch: allocated from the context's pool on the build
// stream and returned to it (also stream-ordered) when the build returns, so
// that a rebuild takes no driver allocation and no implicit synchronisation.
struct Scratch {
  cudaMemPool_t pool;
  cudaStream_t st;
  std::vector<void*> ptrs;
  ~Scratch() {
    for (void* p : ptrs) cudaFreeAsync(p, st);
  }
  template <class T>
  cudaError_t alloc(T** out, size_t count) {
    void* p = nullptr;
    const size_t bytes = (count ? count : 1) * sizeof(T);
    cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, pool, st);
    if (e == cudaSuccess) ptrs.push_back(p);
    *out = static_cast<T*>(p);
    return e;
  }
};

// Device array owned by DeviceBuilt: at least one element, zeroed when empty
// (the reference uploads one zeroed element for an empty array).
template <class T>
cudaError_t alloc_out(DevBuf<T>& b, size_t count, uint64_t& bytes, cudaMemPool_t pool, cudaStream_t s) {
  const size_t n = count ? count : 1;
  const cudaError_t e = alloc_built(b, n, pool, s);
  if (e != cudaSuccess) return e;
  b.count = count;
  bytes += n * sizeof(T);
  if (!count) return cudaMemsetAsync(b.ptr, 0, sizeof(T), s);
  return cudaSuccess;
}

inline uint32_t blocks_for(uint64_t n, uint32_t per = kBlock) {
  const uint64_t b = (n + per - 1) / per;
  return (uint32_t)(b ? b : 1);
}

}  // namespace

std::string build_blas_device(const std::vector<DeviceGeometry>& geoms, uint32_t bin_size, uint32_t max_depth,
                              int sm_count, const DeviceBuildQueue& q, DeviceBuilt& d, DeviceBlasOut& out) {
  const uint32_t G = (uint32_t)geoms.size();
  uint64_t N64 = 0, V64 = 0;
  for (const auto& g : geoms) {
    N64 += g.triangle_count;
    V64 += g.vertex_count;
  }
  if (N64 >= (1ull << 31) || V64 >= (1ull << 31) / 3 || N64 * 3 >= (1ull << 32))
    return "too many triangles or vertices for one device build";
  const uint32_t N = (uint32_t)N64, V = (uint32_t)V64;
  out = DeviceBlasOut();
  out.triangles = N;
  out.vertices = V;
  const cudaStream_t st = q.stream;
  const cudaMemPool_t mem_pool = q.pool;
  Scratch S{mem_pool, st, {}};
  uint64_t& bytes = out.bytes;
#define CK(x)                                                                                  \
  do {                                                                                         \
    cudaError_t e_ = (x);                                                                      \
    if (e_ != cudaSuccess)                                                                     \
      return std::string(e_ == cudaErrorMemoryAllocation ? "CUDA OOM " : "CUDA ") + #x + ": " + \
             cudaGetErrorString(e_);                                                           \
  } while (0)

  // geometry arrays
  CK(alloc_out(d.vertices, 3 * (size_t)V, bytes, mem_pool, st));
  CK(alloc_out(d.indices, 3 * (size_t)N, bytes, mem_pool, st));
  // per geometry: first triangle (and their end), first vertex, vertex count, indexed
  std::vector<uint32_t> g_in(4 * (size_t)G + 1);
  uint32_t *g_prim = g_in.data(), *g_vs = g_prim + G + 1, *g_vc = g_vs + G, *g_ix = g_vc + G;
  {
    uint32_t ps = 0, vs = 0;
    for (uint32_t g = 0; g < G; g++) {
      const DeviceGeometry& q = geoms[g];
      g_prim[g] = ps;
      g_vs[g] = vs;
      g_vc[g] = q.vertex_count;
      g_ix[g] = q.indices ? 1u : 0u;
      if (q.vertex_count)
        CK(cudaMemcpyAsync(d.vertices.ptr + 3 * (size_t)vs, q.positions, 12 * (size_t)q.vertex_count,
                           cudaMemcpyHostToDevice, st));
      if (q.indices && q.triangle_count)
        CK(cudaMemcpyAsync(d.indices.ptr + 3 * (size_t)ps, q.indices, 12 * (size_t)q.triangle_count,
                           cudaMemcpyHostToDevice, st));
      ps += q.triangle_count;
      vs += q.vertex_count;
    }
    g_prim[G] = ps;
  }
  d.vertex_count = V;
  uint32_t* dg_prim;
  CK(S.alloc(&dg_prim, g_in.size()));
  CK(cudaMemcpyAsync(dg_prim, g_in.data(), 4 * g_in.size(), cudaMemcpyHostToDevice, st));
  const uint32_t *dg_vs = dg_prim + G + 1, *dg_vc = dg_vs + G, *dg_ix = dg_vc + G;

  float4* pbox;
  uint8_t* bucket;  // per primitive in the level's order
  uint32_t *order, *order_b;
  CK(S.alloc(&pbox, 2 * (size_t)N));
  CK(S.alloc(&bucket, N));
  CK(S.alloc(&order, N));
  CK(S.alloc(&order_b, N));
  const uint32_t persistent = (uint32_t)(sm_count > 0 ? sm_count : 1) * 8;
  CK(cudaEventRecord(q.begin, st));
  const size_t cap = 2 * (size_t)N + 2 * (size_t)G + 64;
  BNode* pool;
  CK(S.alloc(&pool, cap));
  const uint32_t pool_cap = (uint32_t)std::min<uint64_t>(cap, NONE);

  // level rounds. Every buffer is sized for the largest possible level (nodes
  // that are split hold more than `small` and more than bin_size primitives,
  // and their ranges are disjoint), so that no level waits for the host. The
  // host queues a batch of levels, then reads the level bounds back once to see
  // whether an empty level has been reached; levels queued past it do nothing.
  // A split with an empty child (areas beyond the float range) can repeat down
  // to max_depth, which the subtree blocks have no room for: such a forest is
  // built over, by level rounds alone.
  const uint32_t level_cap = (uint32_t)std::min<uint64_t>(max_depth, N) + 2;  // possible levels + one empty
  const uint32_t big_cap = N / (kBigChunks * kChunk) + 2;  // a big node holds > kBigChunks * kChunk primitives
  uint32_t *lvl, *chunk_cnt, *chunk_prefix, *big_list, *ended;
  LevelCounters* lcs;
  LevelBuffers buf[2];  // this level's and the next one's
  // the counters and the level bounds: one copy to the host
  constexpr size_t kBounds = sizeof(BuildCounters) / 4;
  CK(S.alloc(&lvl, kBounds + level_cap + 2));
  BuildCounters* bc = reinterpret_cast<BuildCounters*>(lvl);
  lvl += kBounds;
  CK(S.alloc(&lcs, (size_t)level_cap + 1));
  CK(S.alloc(&big_list, big_cap));
  CK(S.alloc(&ended, cap));
  std::vector<uint32_t> counters(kBounds + level_cap + 2);
  const uint32_t* h_lvl = counters.data() + kBounds;
  uint32_t levels = 0;
  BuildCounters hbc;
  for (uint32_t small = kSmall;; small = 0) {
    const size_t node_cap = 2 * (size_t)N / (std::max(bin_size, small) + 1ull) + G + 1;
    const size_t chunk_cap = (size_t)N / kChunk + node_cap + 1;
    for (LevelBuffers& b : buf) {
      CK(S.alloc(&b.acc_cnt, 4 * node_cap));
      CK(S.alloc(&b.acc_box, 24 * node_cap));
      CK(S.alloc(&b.chunk_node, chunk_cap));
    }
    const SplitRule rule{bin_size, max_depth, small};
    CK(S.alloc(&chunk_cnt, 4 * chunk_cap));
    CK(S.alloc(&chunk_prefix, 4 * chunk_cap));
    start_kernel<<<std::min(blocks_for(std::max(N, G)), persistent * 4), kBlock, 0, st>>>(N, G, dg_prim, order, pool, lvl, lcs,
                                                                                        level_cap + 1, bc);
    if (N && small)  // once: it makes the indices global
      prepare_primitives_kernel<<<std::min(blocks_for(N), persistent * 4), kBlock, 0, st>>>(
          N, G, dg_prim, dg_vs, dg_vc, dg_ix, d.indices.ptr, d.vertices.ptr, pbox, bc);
    if (G) {
      prepare_roots_kernel<<<std::min(blocks_for(G), persistent), kBlock, 0, st>>>(G, rule, pool, buf[0], lcs, bc, ended);
      root_box_kernel<<<persistent, kBlock, 0, st>>>(lcs, pool, buf[0].chunk_node, order, pbox);
    }
    uint32_t queued = 0;
    bool closed = false;
    // first batch: about the depth of a balanced tree, then a few levels at a time
    uint32_t batch = 2;
    for (uint64_t m = std::max<uint32_t>(std::max(bin_size, small), 1); m < N; m *= 2) batch++;
    while (!closed) {
      const uint32_t stop = std::min(queued + batch, level_cap);
      batch = 4;
      for (; queued < stop; queued++) {
        const uint32_t L = queued;
        uint32_t *from = L & 1 ? order_b : order, *to = L & 1 ? order : order_b;
        const LevelBuffers &B = buf[L & 1], &next = buf[(L + 1) & 1];
        level_stats_kernel<<<persistent, kBlock, 0, st>>>(lvl, L, lcs, pool, B.chunk_node, from, pbox, bucket, chunk_cnt,
                                                          B.acc_cnt, B.acc_box);
        level_decide_kernel<<<persistent, kBlock, 0, st>>>(lvl, L, pool, B.acc_cnt, B.acc_box,
                                                           reinterpret_cast<const uint4*>(chunk_cnt),
                                                           reinterpret_cast<uint4*>(chunk_prefix), lcs, bc, big_list,
                                                           big_cap, pool_cap, rule, next,
                                                           ended);
        level_prefix_select_kernel<<<persistent, kBlock, 0, st>>>(lvl, lcs, L, pool, big_list, big_cap,
                                                                  reinterpret_cast<const uint4*>(chunk_cnt),
                                                                  reinterpret_cast<uint4*>(chunk_prefix), pbox, from);
        level_scatter_kernel<<<persistent, kBlock, 0, st>>>(lvl, L, lcs, pool, pbox, B.chunk_node, from, bucket, B.acc_cnt,
                                                            chunk_prefix, to, pool_cap);
      }
      CK(cudaGetLastError());
      if (!d.tri_records.ptr) {  // while the levels run
        CK(alloc_out(d.indices_redirect, N, bytes, mem_pool, st));
        CK(alloc_out(d.tri_records, N, bytes, mem_pool, st));
      }
      CK(cudaMemcpyAsync(counters.data(), bc, 4 * (kBounds + queued + 2), cudaMemcpyDeviceToHost, st));
      CK(cudaStreamSynchronize(st));
      std::memcpy(&hbc, counters.data(), sizeof(hbc));
      if (hbc.bad_index) return "triangle index out of range";  // no kernel has read a vertex through the indices yet
      if (hbc.overflow) return "device build: more nodes than the build holds";
      for (uint32_t k = 0; k <= queued && !closed; k++)
        if (h_lvl[k + 1] == h_lvl[k]) {  // level k is empty: the tree has k levels
          levels = k;
          closed = true;
        }
      if (!closed && queued >= level_cap) return "device build: tree deeper than its level bound";
    }
    if (hbc.ended && !(small && hbc.unfit))
      small_trees_kernel<<<std::min(hbc.ended, 1u << 20), kSmallThreads, 0, st>>>(small, h_lvl[levels], ended, bin_size, max_depth,
                                                                  pool, order, order_b, pbox, bc);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&hbc, bc, sizeof(hbc), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (!(small && hbc.unfit)) break;
  }
  // the level rounds' nodes, then those of the subtrees
  const uint32_t T = h_lvl[levels] + hbc.added;
  out.max_depth = hbc.max_depth;
  out.nodes = T;

  // The four-child collapse reads only the finished binary tree: its marks
  // and numbering scan run on a side stream, overlapped with the
  // pre-order numbering and the allocations below; the emit waits for them.
  struct SideStream {
    cudaStream_t s;
    ~SideStream() {
      // before the scratch it reads is freed (on the main stream, by S's
      // destructor, which runs after this one), also on an early error return
      cudaStreamSynchronize(s);
    }
  } side{q.side};
  uint32_t *croot, *level4, *index4, *max_level4;
  CK(S.alloc(&croot, T));
  CK(S.alloc(&level4, T));
  CK(S.alloc(&index4, T));
  uint4* slots;
  CK(S.alloc(&slots, T));
  CK(S.alloc(&max_level4, 1));
  void* scan4 = nullptr;
  if (T) CK(S.alloc(reinterpret_cast<char**>(&scan4), scan_scratch_bytes(T) + 256));
  CK(cudaMemsetAsync(croot, 0, 4 * (size_t)(T ? T : 1), st));
  CK(cudaMemsetAsync(level4, 0, 4 * (size_t)(T ? T : 1), st));
  CK(cudaMemsetAsync(max_level4, 0, 4, st));
  CK(cudaEventRecord(q.fork, st));
  CK(cudaStreamWaitEvent(side.s, q.fork, 0));
  if (T) {
    wide4_slots_kernel<<<blocks_for(h_lvl[levels]), kBlock, 0, side.s>>>(h_lvl[levels], pool, slots);
    wide4_top_kernel<<<1, kNumberThreads, 0, side.s>>>(lvl, levels, G, pool, slots, croot, level4, max_level4);
    wide4_mark_small_kernel<<<std::min(blocks_for(hbc.ended, kWarps), 1u << 20), kBlock, 0, side.s>>>(
        ended, bc, pool, slots, croot, level4, max_level4);
    CK(scan_u32(croot, index4, T, false, 0, scan4, side.s));
    CK(cudaGetLastError());
  }
  CK(cudaEventRecord(q.join, side.s));

  uint32_t *pre, *inner_at, *rank, *tree_end, *tree_nodes, *root_code;
  CK(S.alloc(&pre, T));
  CK(S.alloc(&inner_at, T));
  CK(S.alloc(&rank, T));
  CK(S.alloc(&tree_end, G));
  CK(S.alloc(&tree_nodes, G));
  CK(S.alloc(&root_code, G));
  unsigned long long* tree_share;
  CK(S.alloc(&tree_share, G));
  if (T) {
    top_numbering_kernel<<<1, kNumberThreads, 0, st>>>(lvl, levels, G, pool, tree_end, tree_nodes, pre, tree_share);
    inner_flags_kernel<<<blocks_for(T), kBlock, 0, st>>>(T, pool, pre, inner_at);
    void* scan_tmp;
    CK(S.alloc(reinterpret_cast<char**>(&scan_tmp), scan_scratch_bytes(T) + 256));
    CK(scan_u32(inner_at, rank, T, false, 0, scan_tmp, st));
  }
  const uint32_t inner_total = (T - G) / 2;  // every inner node has two children
  const uint32_t leaf_total = T - inner_total;
  CK(alloc_out(d.tri_bvh_forest, T, bytes, mem_pool, st));
  CK(alloc_out(d.wide_nodes, inner_total, bytes, mem_pool, st));
  CK(alloc_out(d.leaf_ranges, 2 * (size_t)leaf_total, bytes, mem_pool, st));
  CK(alloc_out(d.wide4_nodes, inner_total, bytes, mem_pool, st));
  if (T)
    emit_nodes_kernel<<<blocks_for(T), kBlock, 0, st>>>(T, G, pool, pre, rank, tree_end, d.tri_bvh_forest.ptr,
                                                        d.wide_nodes.ptr, d.leaf_ranges.ptr, root_code,
                                                        tree_share);
  if (N)
    emit_primitives_kernel<<<std::min(blocks_for(N), persistent * 4), kBlock, 0, st>>>(
        N, order, d.indices.ptr, d.vertices.ptr, d.indices_redirect.ptr, d.tri_records.ptr);
  CK(cudaGetLastError());

  // four-child layout: collapse roots marked level by level, numbered by one
  // scan in pool order (inner geometry roots first, in geometry order), one emit
  out.root_code.resize(G);
  out.root_code4.resize(G);
  BuildSummary* summary;
  std::vector<char> h_summary(sizeof(BuildSummary) + sizeof(BuildRoot) * G);
  CK(S.alloc(reinterpret_cast<char**>(&summary), h_summary.size()));
  CK(cudaStreamWaitEvent(st, q.join, 0));
  if (T) {
    wide4_emit_kernel<<<blocks_for(T), kBlock, 0, st>>>(T, N < kPackedTriangles, pool, croot, slots, index4, pre, rank, d.wide4_nodes.ptr);
    CK(cudaGetLastError());
    summary_kernel<<<blocks_for(G), kBlock, 0, st>>>(G, T, pool, tree_nodes, root_code, index4, croot, max_level4,
                                                     tree_share, summary,
                                                     reinterpret_cast<BuildRoot*>(summary + 1));
    CK(cudaGetLastError());
  }
  CK(cudaEventRecord(q.end, st));

  out.tree_nodes.resize(G);
  out.root_box.resize(G);
  out.line_nodes.resize(G);
  BuildSummary hs{};
  if (T) CK(cudaMemcpyAsync(h_summary.data(), summary, h_summary.size(), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (T) std::memcpy(&hs, h_summary.data(), sizeof(hs));
  d.wide4_nodes.count = hs.wide4_nodes;
  out.max_wide4_depth = hs.wide4_depth;
  uint32_t inner_roots = 0;
  for (uint32_t g = 0; g < G; g++) {
    BuildRoot r;
    std::memcpy(&r, h_summary.data() + sizeof(BuildSummary) + sizeof(BuildRoot) * g, sizeof(r));
    out.tree_nodes[g] = r.nodes;
    out.root_code[g] = r.code;
    out.line_nodes[g] = r.line_nodes;
    out.root_code4[g] = r.left == NONE ? r.code : inner_roots++;  // a leaf root's code is the two-child one
    out.root_box[g] = Box{{val_of(r.lo[0]), val_of(r.lo[1]), val_of(r.lo[2])}, {val_of(r.hi[0]), val_of(r.hi[1]), val_of(r.hi[2])}};
  }
  float ms = 0.0f;
  CK(cudaEventElapsedTime(&ms, q.begin, q.end));
  out.kernel_seconds = ms / 1000.0;
  out.sah_splits = hbc.sah;
  out.median_fallbacks = hbc.fallback;
#undef CK
  return std::string();
}

cudaError_t emit_vertex_records(const DeviceBuilt& d, cudaStream_t st) {
  const uint32_t N = (uint32_t)d.indices_redirect.count;
  if (N == 0) return cudaSuccess;
  const uint32_t blocks = std::min<uint32_t>((N + kBlock - 1) / kBlock, 4096u);
  emit_vertex_records_kernel<<<blocks, kBlock, 0, st>>>(N, d.indices_redirect.ptr, d.indices.ptr, d.vertices.ptr,
                                                        d.vertex_records.ptr);
  return cudaGetLastError();
}

}  // namespace rdn
