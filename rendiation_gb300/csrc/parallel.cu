// Device-wide scan, stream compaction and LSD radix sort for sm_103a: the
// parallel-compute primitives the reference's wavefront executor builds on
// (shader/parallel-compute/src/prefix_scan.rs:39-114 Kogge-Stone workgroup scan,
// lib.rs:398-429 two-level segmented scan, stream_compaction.rs:3-45,
// shuffle_move.rs:4-59, radix_sort.rs:29-74).
//
// The reference scans with one Kogge-Stone pass per workgroup and a second
// level over workgroup tails, which caps its length at WG^2 elements
// (lib.rs:395-397). Here every primitive reads its input once: blocks take
// tiles (8192 elements, 4096 in the sort) in order from a ticket counter,
// publish a tile's total and find what stands before it by looking back over
// the tiles before (decoupled look-back, Merrill and Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back", 2016).
//   scan     any length up to 2^32-1; an optional power-of-two segment length
//            restarts the sum (the reference's workgroup-scoped scan)
//   compact  the same scan over keep-flags, the kept values gathered in shared
//            memory and written in one run per tile; the tail of the output is
//            zero-filled, as the reference's test expects
//   sort     8-bit digits: the histograms of all passes in one read of the
//            keys, then one kernel per pass that ranks a tile's digits, looks
//            back per digit, and writes the tile from shared memory in digit
//            order (Adinets and Merrill, "Onesweep", 2022); up to 4096
//            elements sort in one block
// 4,000,003 elements, with three kernels a pass and tiles of 1024 or 2048 ->
// here: 32-bit pair sort 330 -> 168 us, compaction 54 -> 24, scan 31 -> 17;
// 10,000 elements: 99 -> 44, 21 -> 11, 15 -> 6.
//
// A tile's predecessors have taken their tickets before it, so they run and
// every wait ends; each wait is bounded all the same. A block whose wait runs
// out counts the missing tile in the input itself, so that every result is
// right whatever held the other block up.
#include <cuda_runtime.h>

#include <cstdint>

#include "parallel.h"

namespace rdn {
namespace {

constexpr uint32_t THREADS = 512, WARPS = THREADS / 32, ITEMS = 16, TILE = THREADS * ITEMS;
constexpr uint32_t SORT_TILE = 4096, HIST_THREADS = 256;
constexpr uint32_t FULL = 0xffffffffu;
constexpr uint32_t kMaxWait = 1u << 16;  // polls of one descriptor, some 40 ms: waits are of microseconds
constexpr uint32_t DIGITS = 256;
constexpr uint32_t kWindow = 4;

// Tile descriptor of a scan: the sum in the low word, how far it reaches above.
enum : uint32_t { TILE_EMPTY = 0, TILE_SUM = 1, TILE_PREFIX = 2 };
using TileState = unsigned long long;
__device__ __forceinline__ TileState tile_state(uint32_t status, uint32_t value) {
  return ((TileState)status << 32) | value;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v) {
  const uint32_t lane = threadIdx.x & 31u;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t n = __shfl_up_sync(FULL, v, o);
    if (lane >= (uint32_t)o) v += n;
  }
  return v;
}

// The next tile, in ticket order, to every thread of the block.
__device__ __forceinline__ uint32_t take_tile(uint32_t* ticket, uint32_t* shared) {
  if (threadIdx.x == 0) *shared = atomicAdd(ticket, 1u);
  __syncthreads();
  return *shared;
}

// The sum over one whole tile of `in`, by a warp, for a look-back whose wait
// ran out. `in` may be what the scan writes over: see look_back.
__device__ __forceinline__ uint32_t tile_sum(const uint32_t* in, uint32_t tile, bool as_flags) {
  const volatile uint32_t* p = in + (size_t)tile * TILE;
  uint32_t sum = 0;
#pragma unroll 1
  for (uint32_t k = threadIdx.x & 31u; k < TILE; k += 32u) sum += as_flags ? (uint32_t)(p[k] != 0u) : p[k];
  return __reduce_add_sync(FULL, sum);
}

// Publishes ahead of everything that the block writes after its next barrier:
// an exchange that acquires. 16,000,000 elements in place take 33.8 us with it,
// 46.7 with a plain store and a fence after the look-back, and took 43.2 with
// the store alone, which orders nothing.
__device__ __forceinline__ void publish_first(volatile TileState* at, TileState s) {
  TileState old;
  asm volatile("atom.acquire.gpu.global.exch.b64 %0, [%1], %2;" : "=l"(old) : "l"(const_cast<TileState*>(at)), "l"(s) : "memory");
}

// One warp: publishes the tile's total and returns the sum of the tiles
// [first, tile) before it. A tile that does not publish in time is summed here.
// That holds in place too: nothing of the block is written before its
// descriptor is (publish_first), so one that is still empty after the sum was
// read proves that the tile's input was whole.
__device__ __forceinline__ uint32_t look_back(volatile TileState* state, uint32_t tile, uint32_t first, uint32_t total,
                                              const uint32_t* in, bool as_flags, bool in_place) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t before = 0;
  if (lane == 0) {
    const TileState own = tile_state(tile == first ? TILE_PREFIX : TILE_SUM, total);
    if (in_place) publish_first(state + tile, own);
    else state[tile] = own;
  }
  if (tile == first) return 0;
  for (uint32_t behind = 1;; behind += 32) {
    // lane k reads the tile `behind + k` before; the first tile's prefix is its sum
    const uint32_t back = behind + lane;
    const bool known = back > tile - first;
    TileState s = 0;
    uint32_t stop = 0;
    for (uint32_t polls = 0;; polls++) {
      s = known ? tile_state(TILE_PREFIX, 0u) : state[tile - back];
      const uint32_t empty = __ballot_sync(FULL, (uint32_t)(s >> 32) == TILE_EMPTY);
      stop = __ballot_sync(FULL, (uint32_t)(s >> 32) == TILE_PREFIX);
      const uint32_t need = stop ? (stop & -stop) - 1u : FULL;  // lanes before the nearest prefix
      uint32_t missing = empty & need;
      if (missing == 0u) break;
      if (polls < kMaxWait) continue;
      for (; missing; missing &= missing - 1u) {
        const uint32_t k = (uint32_t)__ffs(missing) - 1u, at = tile - behind - k;
        const uint32_t sum = tile_sum(in, at, as_flags);
        __threadfence();
        const TileState now = state[at];
        if (lane == k) s = (uint32_t)(now >> 32) == TILE_EMPTY ? tile_state(at == first ? TILE_PREFIX : TILE_SUM, sum) : now;
      }
      stop = __ballot_sync(FULL, (uint32_t)(s >> 32) == TILE_PREFIX);
      break;
    }
    const uint32_t upto = stop ? (uint32_t)__ffs(stop) - 1u : 31u;
    before += __reduce_add_sync(FULL, lane <= upto ? (uint32_t)s : 0u);
    if (stop) break;
  }
  if (lane == 0) state[tile] = tile_state(TILE_PREFIX, before + total);
  return before;
}

// A warp's 512 elements of a tile, four consecutive ones per lane and round.
// (Tiles of 4096 took 18.4 us to scan 4,000,003 elements, of 8192 16.6, of
// 16384 14.6 but 1.5 us more below 100,000: fewer tiles shorten the look-back.)
__device__ __forceinline__ size_t striped(uint32_t tile, uint32_t round) {
  return (size_t)tile * TILE + (threadIdx.x >> 5) * (32u * ITEMS) + round * 128u + (threadIdx.x & 31u) * 4u;
}
template <bool VEC>
__device__ __forceinline__ uint4 load4(const uint32_t* __restrict__ p, size_t i, uint32_t n) {
  if (VEC && i + 4 <= n) return *reinterpret_cast<const uint4*>(p + i);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (i < n) v.x = p[i];
  if (i + 1 < n) v.y = p[i + 1];
  if (i + 2 < n) v.z = p[i + 2];
  if (i + 3 < n) v.w = p[i + 3];
  return v;
}
template <bool VEC>
__device__ __forceinline__ void store4(uint32_t* p, size_t i, uint32_t n, uint4 v) {
  if (VEC && i + 4 <= n) {
    *reinterpret_cast<uint4*>(p + i) = v;
    return;
  }
  if (i < n) p[i] = v.x;
  if (i + 1 < n) p[i + 1] = v.y;
  if (i + 2 < n) p[i + 2] = v.z;
  if (i + 3 < n) p[i + 3] = v.w;
}
__device__ __forceinline__ uint4 flags_of(uint4 v) {
  return make_uint4(v.x != 0u, v.y != 0u, v.z != 0u, v.w != 0u);
}

// Exclusive sums of the thread's four rounds inside the tile; the tile's total.
__device__ __forceinline__ uint32_t tile_exclusive(const uint4 (&v)[4], uint32_t (&base)[4], uint32_t* warp_sums) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint32_t s = v[r].x + v[r].y + v[r].z + v[r].w;
    const uint32_t inc = warp_inclusive(s);
    base[r] = carry + inc - s;
    carry += __shfl_sync(FULL, inc, 31);
  }
  if (lane == 31) warp_sums[warp] = carry;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (uint32_t w = 0; w < WARPS; w++) {
    const uint32_t s = warp_sums[w];
    if (w < warp) before += s;
    total += s;
  }
#pragma unroll
  for (int r = 0; r < 4; r++) base[r] += before;
  return total;
}

// segment_tiles: 0, or the tiles after which the sum restarts. A scan of one
// tile looks back at nothing and has no state to clear before it (null; 2048
// elements 4.2 us, 6.2 with the clearing and the ticket).
template <bool VEC>
__global__ void __launch_bounds__(THREADS, 3) scan_kernel(const uint32_t* in, uint32_t* out, uint32_t n, bool inclusive,
                                                       bool as_flags, uint32_t segment_tiles, TileState* state,
                                                       uint32_t* ticket) {
  __shared__ uint32_t warp_sums[WARPS], tile_s, before_s;
  const uint32_t tile = state ? take_tile(ticket, &tile_s) : 0u;
  uint4 v[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    v[r] = load4<VEC>(in, striped(tile, r), n);
    if (as_flags) v[r] = flags_of(v[r]);
  }
  uint32_t base[4];
  const uint32_t total = tile_exclusive(v, base, warp_sums);
  if (!state) {
    if (threadIdx.x == 0) before_s = 0;
  } else if (threadIdx.x < 32) {
    const uint32_t sum =
        look_back(state, tile, segment_tiles ? tile - tile % segment_tiles : 0u, total, in, as_flags, in == out);
    if (threadIdx.x == 0) before_s = sum;
  }
  __syncthreads();
  const uint32_t before = before_s;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint4 x = v[r];
    uint4 o;
    o.x = before + base[r];
    o.y = o.x + x.x;
    o.z = o.y + x.y;
    o.w = o.z + x.z;
    if (inclusive) o = make_uint4(o.y, o.z, o.w, o.w + x.w);
    store4<VEC>(out, striped(tile, r), n, o);
  }
}

// Inclusive scan that restarts every `segment` < TILE elements (a power of
// two): no tile looks at another.
__global__ void __launch_bounds__(THREADS) scan_segments_kernel(const uint32_t* in, uint32_t* out, uint32_t n,
                                                                bool as_flags, uint32_t segment) {
  __shared__ uint32_t warp_sums[WARPS], sums[TILE];
  uint4 v[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    v[r] = load4<false>(in, striped(blockIdx.x, r), n);
    if (as_flags) v[r] = flags_of(v[r]);
  }
  uint32_t base[4];
  tile_exclusive(v, base, warp_sums);
  const size_t tile0 = (size_t)blockIdx.x * TILE;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint32_t i = (uint32_t)(striped(blockIdx.x, r) - tile0);
    sums[i] = base[r] + v[r].x;
    sums[i + 1] = sums[i] + v[r].y;
    sums[i + 2] = sums[i + 1] + v[r].z;
    sums[i + 3] = sums[i + 2] + v[r].w;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < TILE && tile0 + i < n; i += THREADS) {
    const uint32_t s = i & ~(segment - 1u);
    out[tile0 + i] = sums[i] - (s ? sums[s - 1] : 0u);
  }
}

// Without state: one tile, which also zeroes the tail (33 elements 9.3 us with
// the clearing and the tail's kernel, 4.2 in one).
template <bool VEC>
__global__ void __launch_bounds__(THREADS) compact_kernel(const uint32_t* __restrict__ values,
                                                          const uint32_t* __restrict__ flags,
                                                          uint32_t* __restrict__ out, uint32_t n, uint32_t tiles,
                                                          uint32_t* __restrict__ count, TileState* state,
                                                          uint32_t* ticket) {
  __shared__ uint32_t warp_sums[WARPS], tile_s, before_s, kept[TILE];
  const uint32_t tile = state ? take_tile(ticket, &tile_s) : 0u;
  uint4 f[4], v[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    f[r] = flags_of(load4<VEC>(flags, striped(tile, r), n));
    v[r] = load4<VEC>(values, striped(tile, r), n);
  }
  uint32_t base[4];
  const uint32_t total = tile_exclusive(f, base, warp_sums);
#pragma unroll
  for (int r = 0; r < 4; r++) {
    uint32_t at = base[r];
    if (f[r].x) kept[at++] = v[r].x;
    if (f[r].y) kept[at++] = v[r].y;
    if (f[r].z) kept[at++] = v[r].z;
    if (f[r].w) kept[at++] = v[r].w;
  }
  if (threadIdx.x < 32) {
    const uint32_t before = state ? look_back(state, tile, 0u, total, flags, true, false) : 0u;
    if (threadIdx.x == 0) {
      before_s = before;
      if (tile == tiles - 1) *count = before + total;
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < total; i += THREADS) out[before_s + i] = kept[i];
  if (!state)
    for (uint32_t i = total + threadIdx.x; i < n; i += THREADS) out[i] = 0u;
}

__global__ void __launch_bounds__(THREADS) zero_tail_kernel(uint32_t* __restrict__ out, uint32_t n,
                                                            const uint32_t* __restrict__ count) {
  const uint32_t kept = *count;
  const size_t base = (size_t)blockIdx.x * TILE;
  if (base + TILE <= kept) return;
#pragma unroll
  for (uint32_t k = 0; k < ITEMS; k++) {
    const size_t i = base + k * THREADS + threadIdx.x;
    if (i >= kept && i < n) out[i] = 0u;
  }
}

// ---- radix sort ---------------------------------------------------------------

// n_dev (nullable): the element count lives on the device; n is the capacity
__device__ __forceinline__ uint32_t live_count(uint32_t n, const uint32_t* n_dev) {
  if (!n_dev) return n;
  const uint32_t d = *n_dev;
  return d < n ? d : n;
}

// Digit counts of every pass, and from them hist[pass][digit], the place where
// the digit's run starts in that pass's output.
__global__ void __launch_bounds__(HIST_THREADS) sort_histograms(const uint32_t* __restrict__ keys, uint32_t n_cap,
                                                           const uint32_t* __restrict__ n_dev, uint32_t passes,
                                                           uint32_t* __restrict__ hist, uint32_t* __restrict__ done) {
  __shared__ uint32_t h[4][DIGITS], warp_sums[HIST_THREADS / 32], last;
  const uint32_t n = live_count(n_cap, n_dev);
#pragma unroll
  for (uint32_t q = 0; q < 4; q++) h[q][threadIdx.x] = 0u;
  __syncthreads();
  const size_t stride = (size_t)gridDim.x * SORT_TILE;
  for (size_t base = (size_t)blockIdx.x * SORT_TILE; base < n; base += stride) {
    uint32_t k[ITEMS];
#pragma unroll
    for (uint32_t r = 0; r < ITEMS; r++) {
      const size_t i = base + r * HIST_THREADS + threadIdx.x;
      k[r] = i < n ? keys[i] : 0u;
    }
#pragma unroll
    for (uint32_t r = 0; r < ITEMS; r++) {
      if (base + r * HIST_THREADS + threadIdx.x >= n) continue;
#pragma unroll
      for (uint32_t q = 0; q < 4; q++)
        if (q < passes) atomicAdd(&h[q][(k[r] >> (8u * q)) & 0xFFu], 1u);
    }
  }
  __syncthreads();
  for (uint32_t q = 0; q < passes; q++) {
    const uint32_t c = h[q][threadIdx.x];
    if (c) atomicAdd(hist + q * DIGITS + threadIdx.x, c);
  }
  // the last block to finish turns the totals into each digit's first place
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t q = 0; q < passes; q++) {
    const uint32_t c = __ldcg(hist + q * DIGITS + threadIdx.x);
    const uint32_t inc = warp_inclusive(c);
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    uint32_t before = inc - c;
#pragma unroll
    for (uint32_t w = 0; w < HIST_THREADS / 32; w++)
      if (w < warp) before += warp_sums[w];
    hist[q * DIGITS + threadIdx.x] = before;
    __syncthreads();
  }
}

// A tile of the sort: 4096 elements on 512 threads, a warp 256 consecutive
// ones, 32 a round. The rounds of a warp count into one another, so that eight
// rounds on 16 warps are half the chain of 16 on 8 (43 -> 38 us a pass of
// 4,000,003 pairs). Tiles of 8192 took the same. A pass is bound by shared
// memory (ranking and staging: about 4000 wavefronts a tile) and, for a
// quarter of its time, by the look-back.
constexpr uint32_t SORT_THREADS = 512, SORT_WARPS = SORT_THREADS / 32, ROUNDS = SORT_TILE / SORT_THREADS;

struct SortShared {
  uint16_t count[SORT_WARPS][DIGITS];  // a warp's digit counts, then its offsets inside the digit
  union {
    uint32_t key[SORT_TILE];                 // in digit order
    // while ranking: the lanes of a warp's round with each digit, by atomic OR. 35 us a pass; eight ballots a
    // round 38 (bound by the ALU pipe), __match_any_sync 55
    uint32_t same[SORT_WARPS][DIGITS];
  };
  uint32_t val[SORT_TILE];
  uint32_t offset[DIGITS];             // where a digit's run goes, less where it stands in the tile
  uint32_t first[DIGITS];              // where a digit's run stands in the tile
  uint32_t warp_sums[DIGITS / 32];
  uint32_t tile;
};

// Ranks the tile's keys by digit, stably: on return place[r] is where the
// thread's r-th key stands in the tile's digit order; threads below 256 return
// the count of their digit.
__device__ __forceinline__ uint32_t rank_tile(SortShared& S, const uint32_t (&key)[ROUNDS], uint32_t valid_rounds,
                                              uint32_t shift, uint32_t (&place)[ROUNDS]) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t* clear = reinterpret_cast<uint32_t*>(S.count[warp]);
#pragma unroll
  for (uint32_t k = 0; k < DIGITS / 64; k++) clear[k * 32u + lane] = 0u;
#pragma unroll
  for (uint32_t k = 0; k < DIGITS / 32; k++) S.same[warp][k * 32u + lane] = 0u;
  __syncwarp();
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) {
    const uint32_t d = (key[r] >> shift) & 0xFFu;
    const bool valid = (valid_rounds >> r) & 1u;
    if (valid) atomicOr(&S.same[warp][d], 1u << lane);
    __syncwarp();
    const uint32_t peers = S.same[warp][d], below = peers & ((1u << lane) - 1u);
    const uint32_t before = S.count[warp][d];
    __syncwarp();
    if (valid && below == 0u) {
      S.count[warp][d] = (uint16_t)(before + __popc(peers));
      S.same[warp][d] = 0u;
    }
    __syncwarp();
    place[r] = before + __popc(below);
  }
  __syncthreads();
  uint32_t total = 0, inc = 0;
  if (threadIdx.x < DIGITS) {
    uint32_t c[SORT_WARPS];
#pragma unroll
    for (uint32_t w = 0; w < SORT_WARPS; w++) c[w] = S.count[w][threadIdx.x];
#pragma unroll
    for (uint32_t w = 0; w < SORT_WARPS; w++) {
      S.count[w][threadIdx.x] = (uint16_t)total;
      total += c[w];
    }
    inc = warp_inclusive(total);
    if (lane == 31) S.warp_sums[warp] = inc;
  }
  __syncthreads();
  if (threadIdx.x < DIGITS) {
    uint32_t before = inc - total;
#pragma unroll
    for (uint32_t w = 0; w < DIGITS / 32; w++)
      if (w < warp) before += S.warp_sums[w];
    S.first[threadIdx.x] = before;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) {
    const uint32_t d = (key[r] >> shift) & 0xFFu;
    place[r] += S.first[d] + S.count[warp][d];
  }
  return total;
}

// The keys of one whole tile with digit `digit`, by a thread whose wait for the
// tile's count ran out.
__device__ __forceinline__ uint32_t tile_digits(const uint32_t* __restrict__ keys, uint32_t tile, uint32_t shift,
                                             uint32_t digit) {
  const uint32_t* p = keys + (size_t)tile * SORT_TILE;
  uint32_t count = 0;
#pragma unroll 1
  for (uint32_t k = 0; k < SORT_TILE; k++) count += ((__ldg(p + k) >> shift) & 0xFFu) == digit;
  return count;
}

// One pass over the tile that this block takes. D: descriptor word, the count
// in its low bits, the status in its two top ones. first_of: where each
// digit's run starts in the output.
template <typename D>
__global__ void __launch_bounds__(SORT_THREADS, 3) sort_pass(const uint32_t* __restrict__ keys_in,
                                                             const uint32_t* __restrict__ vals_in,
                                                             uint32_t* __restrict__ keys_out,
                                                             uint32_t* __restrict__ vals_out, uint32_t n_cap,
                                                             const uint32_t* __restrict__ n_dev, uint32_t shift,
                                                             const uint32_t* __restrict__ first_of, volatile D* state,
                                                             uint32_t* ticket) {
  constexpr uint32_t STATUS = sizeof(D) * 8 - 2;
  constexpr D VALUE = ((D)1 << STATUS) - 1;
  __shared__ SortShared S;
  const uint32_t n = live_count(n_cap, n_dev);
  const uint32_t tile = take_tile(ticket, &S.tile);
  const size_t tile0 = (size_t)tile * SORT_TILE;
  if (tile0 >= n) return;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const size_t mine = tile0 + warp * (32u * ROUNDS) + lane;
  uint32_t key[ROUNDS], val[ROUNDS], place[ROUNDS], valid_rounds = 0;
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) {
    const bool valid = mine + 32u * r < n;
    key[r] = valid ? keys_in[mine + 32u * r] : 0u;
    valid_rounds |= (uint32_t)valid << r;
  }
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) val[r] = vals_in && ((valid_rounds >> r) & 1u) ? vals_in[mine + 32u * r] : 0u;
  const uint32_t digit_first = threadIdx.x < DIGITS ? first_of[threadIdx.x] : 0u;
  const uint32_t count = rank_tile(S, key, valid_rounds, shift, place);
  // thread d: what stands before this tile's run of digit d
  volatile D* own = state + (size_t)tile * DIGITS + threadIdx.x;
  if (threadIdx.x < DIGITS) *own = ((D)(tile == 0 ? TILE_PREFIX : TILE_SUM) << STATUS) | count;
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++)
    if ((valid_rounds >> r) & 1u) {
      S.key[place[r]] = key[r];
      if (vals_out) S.val[place[r]] = val[r];
    }
  if (threadIdx.x < DIGITS) {
    D before = 0;
    for (uint32_t back = 1; back <= tile;) {
      D d[kWindow];  // a few descriptors at a time, taken in order
#pragma unroll
      for (uint32_t k = 0; k < kWindow; k++)
        d[k] = back + k <= tile ? own[-(ptrdiff_t)((size_t)(back + k) * DIGITS)] : (D)0;
      bool done = false, missing = false;
      uint32_t polls = 0;
#pragma unroll
      for (uint32_t k = 0; k < kWindow; k++) {
        if (done || back > tile) break;
        while ((d[k] >> STATUS) == TILE_EMPTY && polls < kMaxWait) {
          d[k] = own[-(ptrdiff_t)((size_t)back * DIGITS)];
          polls++;
        }
        if ((d[k] >> STATUS) == TILE_EMPTY) {
          missing = true;
          break;
        }
        before += d[k] & VALUE;
        done = (d[k] >> STATUS) == TILE_PREFIX;
        back++;
      }
      if (done) break;
      if (missing) before += tile_digits(keys_in, tile - back++, shift, threadIdx.x);
    }
    if (tile) *own = ((D)TILE_PREFIX << STATUS) | (before + count);
    S.offset[threadIdx.x] = digit_first + (uint32_t)before - S.first[threadIdx.x];
  }
  __syncthreads();
  const uint32_t live = (uint32_t)(n - tile0 < SORT_TILE ? n - tile0 : SORT_TILE);
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) {
    const uint32_t j = r * SORT_THREADS + threadIdx.x;
    if (j < live) {
      const uint32_t k = S.key[j];
      const uint32_t dst = S.offset[(k >> shift) & 0xFFu] + j;
      keys_out[dst] = k;
      if (vals_out) vals_out[dst] = S.val[j];
    }
  }
}

// Up to one tile: every pass in one block, in place.
__global__ void __launch_bounds__(SORT_THREADS) sort_block(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                           uint32_t n_cap, const uint32_t* __restrict__ n_dev,
                                                           uint32_t passes) {
  __shared__ SortShared S;
  const uint32_t n = live_count(n_cap, n_dev);
  const uint32_t mine = (threadIdx.x >> 5) * (32u * ROUNDS) + (threadIdx.x & 31u);
  uint32_t key[ROUNDS], val[ROUNDS], place[ROUNDS], valid_rounds = 0;
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) {
    const bool valid = mine + 32u * r < n;
    key[r] = valid ? keys[mine + 32u * r] : 0u;
    val[r] = valid && vals ? vals[mine + 32u * r] : 0u;
    valid_rounds |= (uint32_t)valid << r;
  }
  for (uint32_t pass = 0; pass < passes; pass++) {
    rank_tile(S, key, valid_rounds, 8u * pass, place);
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; r++)
      if ((valid_rounds >> r) & 1u) {
        S.key[place[r]] = key[r];
        S.val[place[r]] = val[r];
      }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < ROUNDS; r++)
      if ((valid_rounds >> r) & 1u) {
        key[r] = S.key[mine + 32u * r];
        val[r] = S.val[mine + 32u * r];
      }
    __syncthreads();
  }
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++)
    if ((valid_rounds >> r) & 1u) {
      keys[mine + 32u * r] = key[r];
      if (vals) vals[mine + 32u * r] = val[r];
    }
}

// After an odd number of passes the sorted elements are in the alternate arrays
// (up to *n_dev; what lies past it stays as it is). One kernel for both arrays:
// 4097 pairs on 8 bits took 23.6 us with two copies in its place, 22.6 here.
__global__ void __launch_bounds__(SORT_THREADS) copy_back_kernel(const uint32_t* __restrict__ keys_alt,
                                                                 const uint32_t* __restrict__ vals_alt,
                                                                 uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                                 uint32_t n_cap, const uint32_t* __restrict__ n_dev) {
  const uint32_t n = live_count(n_cap, n_dev);
  const size_t first = (size_t)blockIdx.x * SORT_TILE + threadIdx.x;
  uint32_t k[ROUNDS], v[ROUNDS];
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) {
    const size_t i = first + r * SORT_THREADS;
    k[r] = i < n ? keys_alt[i] : 0u;
    v[r] = i < n && vals ? vals_alt[i] : 0u;
  }
#pragma unroll
  for (uint32_t r = 0; r < ROUNDS; r++) {
    const size_t i = first + r * SORT_THREADS;
    if (i >= n) break;
    keys[i] = k[r];
    if (vals) vals[i] = v[r];
  }
}

inline size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }
inline uint32_t tiles_of(uint32_t n, uint32_t tile) { return (uint32_t)(((uint64_t)n + tile - 1) / tile); }
inline bool aligned16(const void* a, const void* b) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}

// Scratch of a scan or a compaction: the ticket, then a descriptor per tile.
struct TileScratch {
  uint32_t* ticket;
  TileState* state;
};
cudaError_t clear_tiles(void* scratch, uint32_t tiles, cudaStream_t stream, TileScratch& t) {
  t.ticket = static_cast<uint32_t*>(scratch);
  t.state = reinterpret_cast<TileState*>(static_cast<char*>(scratch) + 64);
  return cudaMemsetAsync(scratch, 0, 64 + (size_t)tiles * sizeof(TileState), stream);
}

}  // namespace

// The sizes are those of the three-kernel scan that these scratch blocks were
// first laid out for; callers hold blocks of them. They cover what is used
// now: 64 B + 8 B per 8192 elements.
size_t scan_scratch_bytes(uint32_t n) {
  constexpr uint32_t OLD_TILE = 2048;
  size_t bytes = 0;
  uint32_t len = n;
  while (len > OLD_TILE) {
    len = (uint32_t)(((uint64_t)len + OLD_TILE - 1) / OLD_TILE);
    bytes += up256((size_t)len * 4);
  }
  return bytes + up256((size_t)n * 4) + 256;
}

cudaError_t scan_u32(const uint32_t* in, uint32_t* out, uint32_t n, bool inclusive, uint32_t segment, void* scratch,
                     cudaStream_t stream, bool as_flags) {
  if (n == 0) return cudaSuccess;
  const uint32_t tiles = tiles_of(n, TILE);
  if (segment && segment < TILE) {
    scan_segments_kernel<<<tiles, THREADS, 0, stream>>>(in, out, n, as_flags, segment);
    return cudaGetLastError();
  }
  TileScratch t{nullptr, nullptr};
  if (tiles > 1) {
    const cudaError_t e = clear_tiles(scratch, tiles, stream, t);
    if (e != cudaSuccess) return e;
  }
  const bool incl = inclusive || segment != 0;  // a segmented scan is inclusive
  if (aligned16(in, out)) scan_kernel<true><<<tiles, THREADS, 0, stream>>>(in, out, n, incl, as_flags, segment / TILE, t.state, t.ticket);
  else scan_kernel<false><<<tiles, THREADS, 0, stream>>>(in, out, n, incl, as_flags, segment / TILE, t.state, t.ticket);
  return cudaGetLastError();
}

size_t compact_scratch_bytes(uint32_t n) { return up256((size_t)n * 4) + scan_scratch_bytes(n); }

cudaError_t compact_u32(const uint32_t* values, const uint32_t* flags, uint32_t* out, uint32_t* count, uint32_t n,
                        void* scratch, cudaStream_t stream) {
  if (n == 0) return cudaMemsetAsync(count, 0, 4, stream);
  const uint32_t tiles = tiles_of(n, TILE);
  TileScratch t{nullptr, nullptr};
  cudaError_t e = cudaSuccess;
  if (tiles > 1) e = clear_tiles(scratch, tiles, stream, t);
  if (e != cudaSuccess) return e;
  if (aligned16(values, flags)) compact_kernel<true><<<tiles, THREADS, 0, stream>>>(values, flags, out, n, tiles, count, t.state, t.ticket);
  else compact_kernel<false><<<tiles, THREADS, 0, stream>>>(values, flags, out, n, tiles, count, t.state, t.ticket);
  e = cudaGetLastError();
  if (e != cudaSuccess || tiles == 1) return e;
  zero_tail_kernel<<<tiles, THREADS, 0, stream>>>(out, n, count);
  return cudaGetLastError();
}

// As above: the size that callers hold blocks of (a 256-entry histogram per
// 1024 elements, twice, and its scan). Used now: the two alternate arrays, 4 KB
// of digit counts and 256 B, and per pass and 4096 elements 256 descriptors.
size_t sort_scratch_bytes(uint32_t n) {
  constexpr uint32_t OLD_TILE = 1024;
  const size_t hist = ((size_t)n + OLD_TILE - 1) / OLD_TILE * DIGITS;
  return 2 * up256((size_t)n * 4) + 2 * up256(hist * 4) + scan_scratch_bytes((uint32_t)hist);
}

namespace {
template <typename D>
cudaError_t sort_passes(uint32_t* keys, uint32_t* vals, uint32_t n, uint32_t passes, char* scratch, cudaStream_t stream,
                        const uint32_t* n_dev) {
  const uint32_t tiles = tiles_of(n, SORT_TILE);
  uint32_t* k_alt = reinterpret_cast<uint32_t*>(scratch);
  uint32_t* v_alt = reinterpret_cast<uint32_t*>(scratch + up256((size_t)n * 4));
  char* s = scratch + 2 * up256((size_t)n * 4);
  uint32_t* hist = reinterpret_cast<uint32_t*>(s);
  uint32_t* tickets = hist + 4 * DIGITS;
  D* state = reinterpret_cast<D*>(s + 4 * DIGITS * 4 + 256);
  cudaError_t e =
      cudaMemsetAsync(s, 0, 4 * DIGITS * 4 + 256 + (size_t)passes * tiles * DIGITS * sizeof(D), stream);
  if (e != cudaSuccess) return e;
  // a few tiles a block: the counts of a block are added to the totals once
  sort_histograms<<<tiles < 512u ? tiles : 512u, HIST_THREADS, 0, stream>>>(keys, n, n_dev, passes, hist, tickets + 4);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  uint32_t *k_src = keys, *v_src = vals, *k_dst = k_alt, *v_dst = vals ? v_alt : nullptr;
  for (uint32_t pass = 0; pass < passes; pass++) {
    sort_pass<D><<<tiles, SORT_THREADS, 0, stream>>>(k_src, v_src, k_dst, v_dst, n, n_dev, 8 * pass, hist + pass * DIGITS,
                                                state + (size_t)pass * tiles * DIGITS, tickets + pass);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    uint32_t* t = k_src;
    k_src = k_dst;
    k_dst = t;
    t = v_src;
    v_src = v_dst;
    v_dst = vals ? t : nullptr;
  }
  if (k_src == keys) return cudaSuccess;
  copy_back_kernel<<<tiles, SORT_THREADS, 0, stream>>>(k_src, v_src, keys, vals, n, n_dev);
  return cudaGetLastError();
}
}  // namespace

cudaError_t radix_sort_u32(uint32_t* keys, uint32_t* vals, uint32_t n, uint32_t key_bits, void* scratch,
                           cudaStream_t stream, const uint32_t* n_dev) {
  if (n <= 1) return cudaSuccess;
  const uint32_t passes = (key_bits + 7) / 8;
  if (n <= SORT_TILE) {
    sort_block<<<1, SORT_THREADS, 0, stream>>>(keys, vals, n, n_dev, passes);
    return cudaGetLastError();
  }
  // a 32-bit descriptor counts to 2^30
  return n < (1u << 30) ? sort_passes<uint32_t>(keys, vals, n, passes, static_cast<char*>(scratch), stream, n_dev)
                        : sort_passes<unsigned long long>(keys, vals, n, passes, static_cast<char*>(scratch), stream, n_dev);
}

}  // namespace rdn
