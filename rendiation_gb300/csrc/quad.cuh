// Warp-cooperative ordered traversal: four lanes per ray.
//
// A warp holds up to 32 rays, one per lane. Each lane walks the TLAS of its
// own ray to the next BLAS entry (to_instance, culling: the code of
// traverse_ray); the BLAS walks themselves are shared out to the warp's eight
// quads. A quad walks one ray through the four-child nodes, one child box per
// lane and one triangle of a leaf per lane, and takes the warp's next ray when
// its own is done. (Several lanes per ray on a wide tree: Lier, Stamminger and
// Selgrad, "CPU-style SIMD Ray Traversal on GPUs", HPG 2018.)
//
// Why: the walk of one ray per lane is bound by instruction issue with
// divergent lanes (6.4 of 32 active for random rays through a 150k soup) and,
// below a few hundred thousand rays, by the latency of its chain of steps. A
// quad's four lanes never diverge, a step tests its four boxes in the time of
// one, reads its node as one 128 B line, and a warp's longest ray no longer
// holds 31 others: 24 of 32 lanes active, 0.70 of the issue slots.
// Measured (rdn_trace, us, one ray per lane -> quads): 777,777 random rays
// through a 150k soup 917 -> 835 (watertight 1200 -> 943), 1,000,000 through
// the 1024^2 field 407 -> 355, 1,000 rays through a 10k soup 84 -> 47, 65,536
// camera rays onto it 85 -> 49. Large batches of rays that are alike walk faster
// one per lane, where a warp's lanes share the nodes they read (2.07 M camera
// rays: 597 against 985), and on small trees batches from some 40,000 rays on
// (quad_limit). 64 registers a thread; 72 and 56 cost the random rays 3 and 6 %.
//
// Results: every child box and every triangle is tested with the operations of
// the per-lane walk, and a leaf's candidates are committed in the leaf's order
// against the shrinking far, so a ray keeps the hit of a near-first walk. Only
// the order in which subtrees are met differs, which decides exact-distance
// ties and which hit ends a first-hit search, as between the other ordered
// walks.
#pragma once
#include "traverse.cuh"

namespace rdn {
namespace dev {

constexpr uint32_t kFullWarp = 0xffffffffu;
constexpr uint32_t kQuads = 8;  // per warp
// Quads (in lanes) that may still look for a leaf when the others' leaves are
// tested: 64 soups' paths took 5667 us with 12, 5528 with 16, 5460 with 20,
// 5488 with 24 and 5635 with 28 (0 cost 777,777 rays a third more than 16).
constexpr uint32_t kQuadWait = 20;

// Rays a warp claims of a queue of n: as many as leave no resident warp
// without work (the sizes are rdn_trace's, trace.cu).
__host__ __device__ constexpr uint32_t quad_batch(uint32_t n) { return n < 40000u ? 8u : (n < 100000u ? 16u : 32u); }

// Rows a quad's stack needs: a step pops one entry and pushes at most the four
// children of its node, so every level of the four-child tree below the top
// one holds at most three entries and the top one four: 3 D + 1 for D levels
// (stack_entries(MODE_WIDE4), from the built depth). The steps therefore carry
// no bounds check (with one, 777,777 rays took 898 us instead of 831).

// One BLAS entry of a lane's ray, read by the quad that walks it; the quad
// writes the committed hit over it.
//   in:  a = (object-space origin, tmin)   b = (direction, scaling)
//        c = (root code, far, QB_* bits, 0)
//   out: a = (t, u, v, s)  b.x = sorted triangle  c.w = QS_* state
struct QuadSlot {
  float4 a, b;
  uint4 c;
};
constexpr uint32_t QB_OPAQUE = 1u, QB_CULL = 2u, QB_CULL_BACK = 4u, QB_END = 8u, QB_ODD_START = 16u;
constexpr uint32_t QS_HIT = 1u, QS_ENDED = 2u;

// Shared memory of one warp: 32 slots, the order of its entered rays, and the
// quads' stacks as rows of eight entries (row = depth, column = quad: quads
// reading rows of their own never share a bank). Row 0 is the empty stack's
// top: an entry at +inf, which no far reaches.
struct QuadWarp {
  QuadSlot* slots;
  uint32_t* order;
  uint2* stack;
};
__host__ __device__ constexpr uint32_t quad_warp_bytes(uint32_t stack_depth) {
  return 32u * (uint32_t)sizeof(QuadSlot) + 32u * 4u + (stack_depth + 1u) * kQuads * 8u;
}
__device__ __forceinline__ QuadWarp quad_warp(unsigned char* smem, uint32_t stack_depth) {
  unsigned char* base = smem + (threadIdx.x >> 5) * quad_warp_bytes(stack_depth);
  QuadWarp w;
  w.slots = reinterpret_cast<QuadSlot*>(base);
  w.order = reinterpret_cast<uint32_t*>(base + 32u * sizeof(QuadSlot));
  w.stack = reinterpret_cast<uint2*>(base + 32u * sizeof(QuadSlot) + 128u);
  return w;
}

// True when the warp's rays are alike: but for at most kSeams of them each ray
// points where the one before it does (within 30 degrees) in the same TLAS. A
// seam is the end of an image's row, or of a batch of the caller's: with every
// ray held against the first, the rows' ends of a 1000x524 image, one group in
// 31, went to the quads and made 305 us of camera rays 430. Which walk a ray
// takes decides only exact-distance ties and which hit ends a first-hit search;
// both kernels of a split query form the same vote.
constexpr float kAlikeCos2 = 0.75f;
constexpr int kSeams = 2;
__device__ __forceinline__ bool coherent_warp(const RayCtx& R, uint32_t tidx, bool valid) {
  const float dx = __shfl_up_sync(kFullWarp, R.d.x, 1), dy = __shfl_up_sync(kFullWarp, R.d.y, 1),
              dz = __shfl_up_sync(kFullWarp, R.d.z, 1);
  const uint32_t t0 = __shfl_up_sync(kFullWarp, tidx, 1);
  const bool follows = __shfl_up_sync(kFullWarp, valid, 1) && (threadIdx.x & 31u) != 0u;
  const float dot = R.d.x * dx + R.d.y * dy + R.d.z * dz;
  const float len2 = (R.d.x * R.d.x + R.d.y * R.d.y + R.d.z * R.d.z) * (dx * dx + dy * dy + dz * dz);
  const bool alike = tidx == t0 && dot > 0.0f && dot * dot > kAlikeCos2 * len2;
  return __popc(__ballot_sync(kFullWarp, valid && follows && !alike)) <= kSeams;
}

// Walks the n entered rays order[0..n) of the warp. Every lane calls it; all
// votes and shuffles are full-warp and stand outside divergent code.
template <bool WT>
__device__ __forceinline__ void quad_walk(const TraceParams& p, const QuadWarp& W, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u, l = lane & 3u, qb = lane & ~3u;
  uint2* const stack = W.stack + (lane >> 2);
  uint32_t next = 0;
  if (l == 0u) stack[0] = make_uint2(EMPTY_SLOT, 0x7f800000u);
  __syncwarp();
  // the quad's ray: object space
  float2 no_xy = make_float2(0.f, 0.f), no_z = no_xy, inv_xy = no_xy, inv_z = no_xy;
  float3 d = make_float3(0.f, 0.f, 0.f);
  float near_ = 0.f, far_ = 0.f, scaling = 1.f;
  uint32_t bits = 0, slot = 0;
  uint32_t leaf = EMPTY_SLOT, sp = 0;  // the ray is done when both are empty

  for (;;) {
    // idle quads take the next rays of the warp
    const bool idle = sp == 0u && leaf == EMPTY_SLOT;
    const uint32_t idle_lanes = __ballot_sync(kFullWarp, idle);
    if (idle_lanes && next < n) {
      const uint32_t leaders = idle_lanes & 0x11111111u;
      const uint32_t mine = next + __popc(leaders & ((1u << qb) - 1u));
      const bool take = idle && mine < n;
      next += __popc(leaders);
      float c = 1.f;
      if (take) {
        slot = W.order[mine];
        const float4 a = W.slots[slot].a, b = W.slots[slot].b;
        const uint4 e = W.slots[slot].c;
        no_xy = make_float2(-a.x, -a.y);
        no_z = make_float2(-a.z, -a.z);
        d = make_float3(b.x, b.y, b.z);
        scaling = b.w;
        near_ = a.w * scaling;
        far_ = __uint_as_float(e.y) * scaling;
        bits = e.z;
        if (l == 0u) stack[kQuads] = make_uint2(e.x, 0xff800000u);  // the root, entered at -inf
        sp = 1;
        c = 1.0f / (l == 0 ? d.x : (l == 1 ? d.y : d.z));
      }
      const float cx = __shfl_sync(kFullWarp, c, qb), cy = __shfl_sync(kFullWarp, c, qb + 1u),
                  cz = __shfl_sync(kFullWarp, c, qb + 2u);
      if (take) {
        inv_xy = make_float2(cx, cy);
        inv_z = make_float2(cz, cz);
      }
      __syncwarp();
    } else if (idle_lanes == kFullWarp) {
      break;
    }

    // inner nodes, until no more than kQuadWait lanes' quads still look for a leaf
    bool stuck;  // holds a leaf and the next entry is one too
    do {
#pragma unroll
      for (int rep = 0; rep < 2; rep++) {  // two steps between the votes: 835 us instead of 898 for 777,777 rays
        // the topmost entry, dropped when its box no longer lies before the far; a leaf goes to a quad that holds none
        const uint2 e = stack[sp * kQuads];
        const bool live = __uint_as_float(e.y) < far_;
        const bool is_leaf = live && (int)e.x < 0;
        stuck = is_leaf && leaf != EMPTY_SLOT;
        if (sp != 0u && !stuck) sp--;
        if (is_leaf && !stuck) leaf = e.x;
        const bool act = live && !is_leaf;
        const Wide4Load c = load_wide4_if(p.wide4 + 8 * (size_t)e.x + 2 * l, act);
        float tn;
        const bool hit = slab2<WT>(no_xy, no_z, inv_xy, inv_z, near_, far_, c, tn) && act;
        // near-first: the distance (negative ones equal), the lane in its lowest bits; -1 no hit
        const int key = hit ? ((__float_as_int(fmaxf(tn, 0.0f)) & ~3) | (int)l) : -1;
        const int k1 = __shfl_xor_sync(kFullWarp, key, 1), k2 = __shfl_xor_sync(kFullWarp, key, 2),
                  k3 = __shfl_xor_sync(kFullWarp, key, 3);
        const uint32_t hits = (__ballot_sync(kFullWarp, hit) >> qb) & 15u;
        // the farthest lowest
        const uint32_t row = sp + 1u + (uint32_t)(k1 > key) + (uint32_t)(k2 > key) + (uint32_t)(k3 > key);
        if (hit) stack[row * kQuads] = make_uint2(c.code, __float_as_uint(tn));
        sp += __popc(hits);
        __syncwarp();
      }
    } while ((uint32_t)__popc(__ballot_sync(kFullWarp, sp != 0u && !stuck)) > kQuadWait);

    // leaves: four triangles at a time, committed in order
    if (__any_sync(kFullWarp, leaf != EMPTY_SLOT)) {
      uint32_t k = 0, ke = 0;
      if (leaf != EMPTY_SLOT) {
        const uint2 lr = packed_range(p, leaf);
        k = lr.x;
        ke = lr.y;
      }
      leaf = EMPTY_SLOT;
      bool ended = false;
      do {
        TriOut h;
        h.t = 0.f;
        bool hit = false;
        uint32_t behavior = ANYHIT_ACCEPT;
        if (k + l < ke) {
          const uint32_t t = k + l;
          const bool ce = (bits & QB_CULL) != 0u, cb = (bits & QB_CULL_BACK) != 0u;
          const float3 o = make_float3(-no_xy.x, -no_xy.y, -no_z.x);
          if (WT)
            hit = tri_test_watertight(p.verts + 3 * (size_t)t, o, make_shear(d, make_float3(inv_xy.x, inv_xy.y, inv_z.x)),
                                      near_, far_, ce, cb, h);
          else
            hit = tri_test(p.tris + 4 * (size_t)t, o, d, near_, far_, ce, cb, h);
          if (hit && !(bits & QB_OPAQUE)) {
            // the built-in policies look at the triangle and the parity of its index in the geometry
            const uint32_t tri = __ldg(p.redirect + t);
            behavior = anyhit_policy(p.anyhit_mode, tri - ((bits & QB_ODD_START) ? 1u : 0u), tri, p.anyhit_mask);
          }
        }
        const uint32_t hit_lanes = __ballot_sync(kFullWarp, hit);
        if (hit_lanes) {
          uint32_t m = (hit_lanes >> qb) & 15u;
          const uint32_t accept = (__ballot_sync(kFullWarp, hit && (behavior & ANYHIT_ACCEPT)) >> qb) & 15u;
          const uint32_t stop = (__ballot_sync(kFullWarp, hit && (behavior & ANYHIT_END)) >> qb) & 15u;
          do {
            const uint32_t j = m ? (uint32_t)__ffs(m) - 1u : 0u;
            const float t = __shfl_sync(kFullWarp, h.t, qb + j);
            if (m) {
              m &= m - 1u;
              if (!(t > far_)) {  // the far may have shrunk since the test
                bool end = (stop >> j) & 1u;
                if ((accept >> j) & 1u) {
                  const float distance = t / scaling;
                  far_ = distance * scaling;
                  end |= (bits & QB_END) != 0u;
                  if (l == j) {
                    W.slots[slot].a = make_float4(distance, h.u, h.v, h.s);
                    W.slots[slot].b.x = __uint_as_float(k + l);
                    W.slots[slot].c.w = QS_HIT;
                  }
                }
                if (end) {
                  ended = true;
                  m = 0u;
                  ke = k;
                }
              }
            }
            __syncwarp();
          } while (__any_sync(kFullWarp, m != 0u));
        }
        k += 4u;
      } while (__any_sync(kFullWarp, k < ke));
      if (ended) {
        sp = 0;
        if (l == 0) W.slots[slot].c.w |= QS_ENDED;
      }
      __syncwarp();
    }
  }
}

// The ray's next BLAS entry, written to the slot; false when the query has none left.
template <bool WT>
__device__ __forceinline__ bool quad_enter(const TraceParams& p, const RayCtx& R, TlasCursor& c, QuadSlot& s,
                                           uint32_t& gslot) {
  BlasEntry e;
  if (!next_blas<WT>(p, R, c, e)) return false;
  s.a = make_float4(e.ir.o.x, e.ir.o.y, e.ir.o.z, R.tmin);
  s.b = make_float4(e.ir.d.x, e.ir.d.y, e.ir.d.z, e.ir.scaling);
  s.c = make_uint4(wide4_root(p, e.gslot), __float_as_uint(R.far_world),
                   (e.is_opaque ? QB_OPAQUE : 0u) | (e.cull_enable ? QB_CULL : 0u) | (e.cull_back ? QB_CULL_BACK : 0u) |
                       ((e.ir.flags & TF_END_SEARCH) ? QB_END : 0u) | ((e.gm.z & 1u) ? QB_ODD_START : 0u),
                   0u);
  gslot = e.gslot;
  return true;
}

// Full query of the warp's rays (traverse_cpu.rs:52-245): traverse_ray's
// result for every lane with `valid`. Every lane of the warp calls it.
template <bool WT>
__device__ __forceinline__ void traverse_warp(const TraceParams& p, RayCtx& R, uint32_t tidx, bool valid,
                                              const QuadWarp& W, bool& bad) {
  const uint32_t lane = threadIdx.x & 31u;
  R.best.have = false;
  bad = false;
  TlasCursor c{INVALID_NEXT, 0u, 0u, 0u, 0u, 0u};
  if (valid) c = start_query(p, R, tidx, bad);
  bool more = valid && !bad;
  for (;;) {
    uint32_t gslot = 0;
    const bool entered = more && quad_enter<WT>(p, R, c, W.slots[lane], gslot);
    more = entered;
    const uint32_t m = __ballot_sync(kFullWarp, entered);
    if (m == 0u) break;
    if (entered) W.order[__popc(m & ((1u << lane) - 1u))] = lane;
    __syncwarp();
    quad_walk<WT>(p, W, __popc(m));
    __syncwarp();
    if (entered) {
      const uint32_t state = W.slots[lane].c.w;
      if (state & QS_HIT) {
        const float4 a = W.slots[lane].a;
        R.best.t = R.far_world = a.x;
        R.best.u = a.y;
        R.best.v = a.z;
        R.best.s = a.w;
        R.best.k = __float_as_uint(W.slots[lane].b.x);
        R.best.geom_slot = gslot;
        R.best.inst = c.inst;
        R.best.have = true;
      }
      if (state & QS_ENDED) more = false;
    }
  }
}

// ---- batches of independent rays whose hits go on to per-ray work ----------
// Blocks of four warps. The first `differing` blocks take 128 rays, a warp 32
// of its own. The blocks after them take 32 rays each, a warp eight: a quarter
// of the walk's length for a batch that does not fill the chip, and quads in
// step on the same nodes where the 32 rays are alike; their hits are gathered
// so that one warp goes on with all 32. With `split` the former leave out the
// groups of 32 that are alike and the latter (or a kernel with a ray per lane)
// those that are not.
struct QuadShare {
  uint32_t differing;
  bool split;
};
struct QuadHits {
  float4 tuvs[32];
  uint4 where[32];  // sorted triangle, geometry slot, instance, hit
};
constexpr uint32_t kShareBlock = 128;
// From kShareSplit rays on, groups that differ are walked 32 a warp; from
// quad_limit on, groups that are alike one ray per lane (the hit query of
// 262,144 camera rays on a field of 64^2 98 us by quads, 51 by lanes), and all
// of them where the trees are small.
constexpr uint32_t kShareSplit = 48000, kShareMost = 400000;
constexpr float kShareRays = 255.0f;
__host__ __device__ constexpr uint32_t quad_share_bytes(uint32_t stack_depth) {
  return (uint32_t)sizeof(QuadHits) + 4u * quad_warp_bytes(stack_depth);
}

// Closest hits of the block's rays (ray i: two float4 at rays + 2 i). Returns
// whether this warp goes on, then with its lane's ray i, `valid`, and R.
template <bool WT>
__device__ __forceinline__ bool quad_share_query(const TraceParams& p, const QuadShare& S, const float4* rays,
                                                 uint32_t count, uint32_t tlas, unsigned char* smem, uint32_t& i,
                                                 bool& valid, RayCtx& R) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const bool gather = blockIdx.x >= S.differing;
  const uint32_t group = gather ? blockIdx.x - S.differing : blockIdx.x * 4u + warp;
  i = group * 32u + lane;
  valid = i < count;
  auto load = [&](uint32_t k) {
    const float4 r0 = __ldg(rays + 2 * (size_t)k), r1 = __ldg(rays + 2 * (size_t)k + 1);
    R.o = make_float3(r0.x, r0.y, r0.z);
    R.tmin = r0.w;
    R.d = make_float3(r1.x, r1.y, r1.z);
    R.tmax = r1.w;
  };
  if (valid) load(i);
  // every warp of a gathering block votes on the same 32 rays
  if (S.split && coherent_warp(R, tlas, valid) != gather) return false;
  const uint32_t mine = group * 32u + warp * 8u + lane;
  const bool walks = gather ? lane < 8u && mine < count : valid;
  if (gather && walks) load(mine);
  R.cull_mask = 0xFFu;
  R.ray_flags = 0u;
  bool bad;
  traverse_warp<WT>(p, R, tlas, walks, quad_warp(smem + sizeof(QuadHits), p.stack_depth4), bad);
  if (gather) {
    QuadHits& H = *reinterpret_cast<QuadHits*>(smem);
    if (lane < 8u) {
      const uint32_t at = warp * 8u + lane;
      H.tuvs[at] = make_float4(R.best.t, R.best.u, R.best.v, R.best.s);
      H.where[at] = make_uint4(R.best.k, R.best.geom_slot, R.best.inst, R.best.have ? 1u : 0u);
    }
    __syncthreads();
    if (warp != 0u) return false;
    const float4 t = H.tuvs[lane];
    const uint4 w = H.where[lane];
    R.best.t = t.x;
    R.best.u = t.y;
    R.best.v = t.z;
    R.best.s = t.w;
    R.best.k = w.x;
    R.best.geom_slot = w.y;
    R.best.inst = w.z;
    R.best.have = valid && w.w != 0u;
  }
  if (valid) load(i);
  return true;
}

}  // namespace dev

// The share of a batch of `count` rays (no blocks: none of it), and whether the
// groups that are alike, or all, are left to a kernel with a ray per lane.
struct QuadShareLaunch {
  dev::QuadShare share;
  uint32_t grid;
  bool lanes;
};
inline QuadShareLaunch quad_share(const TraceParams& p, uint32_t count) {
  const uint32_t differing = (uint32_t)(((uint64_t)count + 127) / 128), alike = (uint32_t)(((uint64_t)count + 31) / 32);
  if (count < dev::kShareSplit) return {{0u, false}, alike, false};
  if (!p.local_stack || count < quad_limit(p, dev::kShareRays, dev::kShareSplit, dev::kShareMost))
    return {{differing, true}, differing + alike, false};
  if (small_trees(p)) return {{0u, false}, 0u, true};
  return {{differing, true}, differing, true};
}

}  // namespace rdn
