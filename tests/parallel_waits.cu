// Launches of the look-back kernels of parallel.cu with the first `skip` tiles
// left out (the ticket counter starts at `skip`): their descriptors stay empty,
// so the blocks of the tiles after them wait until their limit. Used by
// tests/test_parallel_waits.py.
#include "parallel.cu"

namespace rdn {
static int done(cudaError_t e) { return e == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess ? 0 : -1; }

extern "C" uint32_t waits_tile(int sort) { return sort ? SORT_TILE : TILE; }

extern "C" int waits_scan(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t skip, int inclusive, int as_flags,
                          uint32_t segment_tiles, void* scratch) {
  TileScratch t;
  const uint32_t tiles = tiles_of(n, TILE);
  cudaError_t e = clear_tiles(scratch, tiles, 0, t);
  if (e == cudaSuccess) e = cudaMemset(t.ticket, (int)skip, 1);
  if (e != cudaSuccess) return -1;
  if (aligned16(in, out)) scan_kernel<true><<<tiles - skip, THREADS>>>(in, out, n, inclusive, as_flags, segment_tiles, t.state, t.ticket);
  else scan_kernel<false><<<tiles - skip, THREADS>>>(in, out, n, inclusive, as_flags, segment_tiles, t.state, t.ticket);
  return done(cudaGetLastError());
}

extern "C" int waits_compact(const uint32_t* values, const uint32_t* flags, uint32_t* out, uint32_t* count, uint32_t n,
                             uint32_t skip, void* scratch) {
  TileScratch t;
  const uint32_t tiles = tiles_of(n, TILE);
  cudaError_t e = clear_tiles(scratch, tiles, 0, t);
  if (e == cudaSuccess) e = cudaMemset(t.ticket, (int)skip, 1);
  if (e != cudaSuccess) return -1;
  compact_kernel<true><<<tiles - skip, THREADS>>>(values, flags, out, n, tiles, count, t.state, t.ticket);
  return done(cudaGetLastError());
}

// One pass on the digit at `shift` (a multiple of 8). scratch: 4 KB of counts, 256 B, a descriptor per tile and digit.
template <typename D>
static int sort_digit(const uint32_t* keys, const uint32_t* vals, uint32_t* keys_out, uint32_t* vals_out, uint32_t n,
                      uint32_t shift, uint32_t skip, char* scratch) {
  const uint32_t tiles = tiles_of(n, SORT_TILE);
  uint32_t* hist = reinterpret_cast<uint32_t*>(scratch);
  uint32_t* ticket = hist + 4 * DIGITS;
  D* state = reinterpret_cast<D*>(scratch + 16 * DIGITS + 256);
  cudaError_t e = cudaMemset(scratch, 0, 16 * DIGITS + 256 + (size_t)tiles * DIGITS * sizeof(D));
  if (e == cudaSuccess) e = cudaMemset(ticket, (int)skip, 1);
  if (e != cudaSuccess) return -1;
  sort_histograms<<<tiles, HIST_THREADS>>>(keys, n, nullptr, shift / 8 + 1, hist, ticket + 4);
  sort_pass<D><<<tiles - skip, SORT_THREADS>>>(keys, vals, keys_out, vals_out, n, nullptr, shift, hist + shift / 8 * DIGITS,
                                               state, ticket);
  return done(cudaGetLastError());
}
extern "C" int waits_sort(const uint32_t* keys, const uint32_t* vals, uint32_t* keys_out, uint32_t* vals_out, uint32_t n,
                          uint32_t shift, uint32_t skip, int wide, void* scratch) {
  char* s = static_cast<char*>(scratch);
  return wide ? sort_digit<unsigned long long>(keys, vals, keys_out, vals_out, n, shift, skip, s)
              : sort_digit<uint32_t>(keys, vals, keys_out, vals_out, n, shift, skip, s);
}
}  // namespace rdn
