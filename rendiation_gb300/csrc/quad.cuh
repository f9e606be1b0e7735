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
// through a 150k soup 1140 -> 898 (watertight 1387 -> 1026), 1,000,000 through
// the 1024^2 field 455 -> 380, 1,000 through a 10k soup 130 -> 52, 65,536
// camera rays onto it 121 -> 53. Only large batches of rays that are alike
// walk faster one per lane, where a warp's lanes share the nodes they read
// (2.07 M camera rays: 727 against 1082). 64 registers; with 72 the random
// rays took 910 us, with 56 938 us.
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
// tested: 777,777 rays through a 150k soup took 1326 us with 0, 986 with 8,
// 949 with 16 and 957 with 20.
constexpr uint32_t kQuadWait = 16;

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

// True when the warp's rays point the same way (within about 11 degrees of the
// first one's direction) in the same TLAS. Which walk a ray takes does not
// change its result; both kernels of a split query form the same vote.
__device__ __forceinline__ bool coherent_warp(const RayCtx& R, uint32_t tidx, bool valid) {
  const uint32_t m = __ballot_sync(kFullWarp, valid);
  const uint32_t src = m ? (uint32_t)__ffs(m) - 1u : 0u;
  const float dx = __shfl_sync(kFullWarp, R.d.x, src), dy = __shfl_sync(kFullWarp, R.d.y, src),
              dz = __shfl_sync(kFullWarp, R.d.z, src);
  const uint32_t t0 = __shfl_sync(kFullWarp, tidx, src);
  const float dot = R.d.x * dx + R.d.y * dy + R.d.z * dz;
  const float len2 = (R.d.x * R.d.x + R.d.y * R.d.y + R.d.z * R.d.z) * (dx * dx + dy * dy + dz * dz);
  return __all_sync(kFullWarp, !valid || (tidx == t0 && dot > 0.0f && dot * dot > 0.96f * len2));
}

// Walks the n entered rays order[0..n) of the warp. Every lane calls it; all
// votes and shuffles are full-warp and stand outside divergent code.
template <bool WT>
__device__ __forceinline__ void quad_walk(const TraceParams& p, const QuadWarp& W, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u, l = lane & 3u, qb = lane & ~3u;
  const uint32_t depth = p.stack_depth4;
  uint2* const stack = W.stack + (lane >> 2);
  uint32_t next = 0;
  if (l == 0u) stack[0] = make_uint2(EMPTY_SLOT, 0x7f800000u);
  __syncwarp();
  // the quad's ray: object space
  float2 no_xy = make_float2(0.f, 0.f), no_z = no_xy, inv_xy = no_xy, inv_z = no_xy;
  float3 d = make_float3(0.f, 0.f, 0.f);
  float near_ = 0.f, far_ = 0.f, scaling = 1.f;
  uint32_t bits = 0, slot = 0;
  bool over = false;
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
      if (over) atomicOr(p.error_word, 1u);
      break;
    }

    // inner nodes, until no more than kQuadWait lanes' quads still look for a leaf
    bool stuck;  // holds a leaf and the next entry is one too
    do {
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
      // the farthest lowest; the stack is sized from the tree depth, so no row is past it
      const uint32_t row = sp + 1u + (uint32_t)(k1 > key) + (uint32_t)(k2 > key) + (uint32_t)(k3 > key);
      if (hit && row <= depth) stack[row * kQuads] = make_uint2(c.quad, __float_as_uint(tn));
      sp += __popc(hits);
      over |= sp > depth;
      sp = min(sp, depth);
      __syncwarp();
    } while ((uint32_t)__popc(__ballot_sync(kFullWarp, sp != 0u && !stuck)) > kQuadWait);

    // leaves: four triangles at a time, committed in order
    if (__any_sync(kFullWarp, leaf != EMPTY_SLOT)) {
      uint32_t k = 0, ke = 0;
      if (leaf != EMPTY_SLOT) {
        const uint32_t count = (leaf >> kLeafCountShift) & kLeafCountMask;
        k = leaf & kLeafStartMask;
        ke = k + count;
        if (count == 0u) {  // a leaf of another size: by its range
          const uint2 lr = __ldg(p.leaves + k);
          k = lr.x;
          ke = lr.y;
        }
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

// Quad code of a geometry's root.
__device__ __forceinline__ uint32_t quad_root(const TraceParams& p, uint32_t g) {
  const uint32_t code = __ldg(p.geom_root_code4 + g);
  if (!(code & LEAF_BIT)) return code;
  const uint2 lr = __ldg(p.leaves + (code & ~LEAF_BIT));
  return quad_leaf_code(code & ~LEAF_BIT, lr.x, lr.y);
}

// Where a lane's ray stands in its TLAS walk.
struct TlasCursor {
  uint32_t node, ti, ti_end, inst, g, g_end;
};

// TLAS / instance / geometry steps of traverse_ray up to the next BLAS entry,
// written to the slot; false when the query has none left.
template <bool WT>
__device__ __forceinline__ bool quad_enter(const TraceParams& p, const RayCtx& R, TlasCursor& c, QuadSlot& s,
                                           uint32_t& gslot) {
  for (;;) {
    while (c.g < c.g_end) {
      const uint32_t g = c.g++;
      const InstanceRay ir = to_instance(p.tlas_data + c.inst, R.o, R.d, R.ray_flags);
      const uint4 gm = __ldg(reinterpret_cast<const uint4*>(p.tri_root + g));
      bool pass, is_opaque, cull_enable, cull_back;
      geometry_cull(ir.flags, gm.w, pass, is_opaque, cull_enable, cull_back);
      if (!pass) continue;
      const float4* nd = reinterpret_cast<const float4*>(p.tri_forest + gm.x);
      const float4 a = __ldg(nd), b = __ldg(nd + 1);
      float tn;
      if (!slab<WT>(ir.o, ir.inv_d, R.tmin * ir.scaling, R.far_world * ir.scaling, a.x, a.y, a.z, b.x, b.y, b.z, tn))
        continue;
      s.a = make_float4(ir.o.x, ir.o.y, ir.o.z, R.tmin);
      s.b = make_float4(ir.d.x, ir.d.y, ir.d.z, ir.scaling);
      s.c = make_uint4(quad_root(p, g), __float_as_uint(R.far_world),
                       (is_opaque ? QB_OPAQUE : 0u) | (cull_enable ? QB_CULL : 0u) | (cull_back ? QB_CULL_BACK : 0u) |
                           ((ir.flags & TF_END_SEARCH) ? QB_END : 0u) | ((gm.z & 1u) ? QB_ODD_START : 0u),
                       0u);
      gslot = g;
      return true;
    }
    bool entered = false;
    while (c.ti < c.ti_end) {
      const uint32_t cur = c.ti++;
      const float4* tb = reinterpret_cast<const float4*>(p.tlas_bounding + cur);
      const float4 ba = __ldg(tb), bb = __ldg(tb + 1);
      float tn;
      if (!slab<WT>(R.o, R.inv_d, R.tmin, R.tmax, ba.x, ba.y, ba.z, bb.x, bb.y, bb.z, tn)) continue;
      if ((R.cull_mask & __float_as_uint(ba.w)) == 0) continue;
      const DeviceInstance* inst = p.tlas_data + cur;
      if (merge_instance_flags(R.ray_flags, __ldg(&inst->flags)) & TF_SKIP_TRIANGLES) continue;
      const uint32_t blas = __ldg(&inst->acceleration_structure_handle);
      const uint2 range = __ldg(reinterpret_cast<const uint2*>(p.blas_meta + blas));
      c.g = range.x;
      c.g_end = range.y;
      c.inst = cur;
      entered = true;
      break;
    }
    if (entered) continue;
    bool found = false;
    while (c.node != INVALID_NEXT) {
      const float4* nd = reinterpret_cast<const float4*>(p.tlas_forest + c.node);
      const float4 a = __ldg(nd), b = __ldg(nd + 1);
      const uint32_t hit_next = __float_as_uint(a.w), miss_next = __float_as_uint(b.w);
      float tn;
      if (!slab<WT>(R.o, R.inv_d, R.tmin * 1.0f, R.far_world * 1.0f, a.x, a.y, a.z, b.x, b.y, b.z, tn)) {
        c.node = miss_next;
        continue;
      }
      c.node = hit_next;
      if (hit_next != miss_next) continue;
      const uint2 cr = __ldg(reinterpret_cast<const uint2*>(nd + 2));
      c.ti = cr.x;
      c.ti_end = cr.y;
      found = true;
      break;
    }
    if (!found) return false;
  }
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
  if (valid) {
    R.inv_d = make_float3(1.0f / R.d.x, 1.0f / R.d.y, 1.0f / R.d.z);
    R.far_world = R.tmax;
    if (tidx >= p.n_binding) {
      bad = true;
    } else {
      const uint32_t handle = __ldg(p.tlas_binding + tidx);
      if (handle >= p.n_tlas_root) bad = true;
      else c.node = __ldg(p.tlas_bvh_root + handle);
    }
  }
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

}  // namespace dev
}  // namespace rdn
