// Stable LSD radix sort of (u32 key, u32 value) pairs: one read of the keys
// for every pass's digit counts, then one kernel per digit that reads and
// writes each pair once (the single-pass scheme of Merrill and Garland's
// decoupled look-back, as used for radix sorting by Adinets and Merrill,
// "Onesweep", 2022).
//
// Per pass and tile (RX_TILE consecutive pairs, taken in ticket order, so
// every earlier tile is already running or done):
//   1. each warp ranks its own run of keys by digit, 32 at a time, on
//      counters of its own in shared memory (no block barrier per step);
//   2. the tile's digit counts are published, and the threads of the first
//      256 walk back over earlier tiles' words, one digit each, adding counts
//      until they meet an inclusive prefix; then they publish theirs.  A
//      thread that has polled in vain RX_POLLS times takes the missing counts
//      from the earlier tiles' keys, which stay as they are during a pass: a
//      wait ends in any case, and with the right sum;
//   3. keys, then values, are staged in shared memory in digit order and
//      written as runs of consecutive addresses.
// Bound: 16 B per pair and pass over HBM; what it spends is issue slots (8
// votes and ~90 other instructions per 32 pairs).  64 M pairs (R-MAT scale 22
// edge list), one pass: ~0.41 ms; the tile-histogram + scan + scatter form
// of three kernels before took 0.79 ms (132 + 33 + 630 us), its scatter two
// block barriers per 256 keys.  Tiles of 4096 to 9216 pairs in blocks of 256
// to 512 threads at 2 to 4 per SM: build_csr of that list 2.91 to 3.46 ms,
// flat (2.91 to 2.97) over 384 x 16..24 and 512 x 16..18.
//
// Used by the device transpose (CSC build), the edge-list -> CSR build, the
// RGG generator, the residual pieces and the batch plan.
#include "prim.cuh"

namespace kspn {

namespace {

constexpr int RX_THREADS = 384;
constexpr int RX_ITEMS   = 16;
constexpr int RX_BLOCKS  = 3; // resident per SM
constexpr int RX_WARPS   = RX_THREADS / 32;
constexpr int RX_TILE    = RX_THREADS * RX_ITEMS;
constexpr int RX_PASSES  = 4; // 32 key bits, at most 8 per pass
constexpr int RX_BINS    = 256;

// Scratch of one sort, in u32 words: digit counts of every pass, a ticket
// per pass, then a u64 look-back word per (tile, digit).  A look-back word
// is pass + 1 in bits 34.., RX_SUM or RX_PREFIX in bits 32..33 and a count
// below, so the words of earlier passes read as "not there yet" and one
// clear per sort is enough.
constexpr size_t             RX_HEAD   = RX_PASSES * RX_BINS + 64;
constexpr unsigned long long RX_SUM    = 1ull << 32; // the tile's own count
constexpr unsigned long long RX_PREFIX = 2ull << 32; // the count of all tiles up to it
constexpr uint32_t           RX_LOOK   = 4;          // look-back words a thread loads at once
constexpr uint32_t           RX_POLLS  = 1u << 20;   // polls in vain (some tenths of a second) before a look-back counts keys instead

struct rx_digits
{
  int      shift[RX_PASSES];
  uint32_t mask[RX_PASSES];
  int      passes;
};

// Passes over key bits [begin, end): as few as 8 bits each allow, of equal
// width (fewer bins per pass make longer runs in the write-out).
rx_digits
rx_plan(int begin, int end)
{
  rx_digits d{};
  int const bits = end - begin;
  d.passes       = (bits + 7) / 8;
  for (int p = 0, at = begin; p < d.passes; ++p) {
    int const w = (end - at + (d.passes - p) - 1) / (d.passes - p);
    d.shift[p]  = at;
    d.mask[p]   = (1u << w) - 1u;
    at += w;
  }
  return d;
}

// Digit counts of all passes from one read of the keys.  Four counter sets
// per block spread the shared-memory atomics of frequent digits.
constexpr int RH_SETS = 4;

__global__ void __launch_bounds__(RX_THREADS)
k_radix_hist(uint32_t const* __restrict__ keys, uint64_t count, rx_digits d, uint32_t* __restrict__ hist)
{
  __shared__ uint32_t cnt[RH_SETS][RX_PASSES * RX_BINS];
  for (int i = threadIdx.x; i < RH_SETS * RX_PASSES * RX_BINS; i += RX_THREADS) (&cnt[0][0])[i] = 0;
  __syncthreads();
  uint32_t* const mine   = cnt[(threadIdx.x >> 5) % RH_SETS];
  uint64_t const  stride = static_cast<uint64_t>(gridDim.x) * RX_THREADS;
  for (uint64_t i0 = static_cast<uint64_t>(blockIdx.x) * RX_THREADS + threadIdx.x; i0 < count; i0 += 4 * stride) {
    uint32_t k[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j] = i0 + j * stride < count ? keys[i0 + j * stride] : 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + j * stride < count)
#pragma unroll
        for (int p = 0; p < RX_PASSES; ++p)
          if (p < d.passes) atomicAdd(mine + p * RX_BINS + ((k[j] >> d.shift[p]) & d.mask[p]), 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < d.passes * RX_BINS; i += RX_THREADS) {
    uint32_t s = 0;
#pragma unroll
    for (int c = 0; c < RH_SETS; ++c) s += cnt[c][i];
    if (s) atomicAdd(hist + i, s);
  }
}

// Exclusive prefix of x over the block's first 256 threads (eight warps);
// every thread of the block calls it.
__device__ __forceinline__ uint32_t
rx_scan_bins(uint32_t x, uint32_t* wsum)
{
  unsigned const t = threadIdx.x, lane = t & 31u, w = t >> 5;
  uint32_t       incl = x;
#pragma unroll
  for (int dd = 1; dd < 32; dd <<= 1) {
    uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, dd);
    if (lane >= static_cast<unsigned>(dd)) incl += y;
  }
  if (lane == 31 && w < 8) wsum[w] = incl;
  __syncthreads();
  uint32_t carry = 0;
  for (unsigned k = 0; k < w && k < 8; ++k) carry += wsum[k];
  __syncthreads(); // wsum reusable
  return carry + incl - x;
}

// Lanes of the warp holding the same 8-bit digit: one vote per bit.  (A
// match instruction takes a step per distinct value: with it a pass over
// random digits took 692 us, one over clustered digits 412 us.)
__device__ __forceinline__ unsigned
rx_peers(uint32_t d)
{
  unsigned peers = 0xFFFFFFFFu;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    bool const     set = (d >> b) & 1u;
    unsigned const bal = __ballot_sync(0xFFFFFFFFu, set);
    peers &= set ? bal : ~bal;
  }
  return peers;
}

struct rx_smem
{
  uint16_t wcnt[RX_WARPS][RX_BINS]; // per warp: running counts, then the warp's offset within the digit
  uint32_t buf[RX_TILE];
  uint32_t off[RX_BINS];  // the digit's first slot in the staged tile
  uint32_t base[RX_BINS]; // global position of the digit's first slot, minus off
  uint32_t wsum[8], tile;
};

struct rx_args
{
  uint32_t const*     kin;
  uint32_t const*     vin;
  uint32_t*           kout;
  uint32_t*           vout;
  uint64_t            count;
  int                 shift;
  uint32_t            mask;
  int                 pass;
  uint32_t const*     hist;   // this pass's digit counts
  uint32_t*           ticket; // this pass's
  unsigned long long* look;   // RX_BINS words per tile
  uint32_t            polls;  // RX_POLLS
};

// One tile of n pairs (FULL: all RX_TILE of them, no bounds checks).
template<bool FULL>
__device__ __forceinline__ void
rx_tile(rx_args const& a, rx_smem& sm, uint32_t tile, uint32_t n)
{
  unsigned const           t = threadIdx.x, w = t >> 5, lane = t & 31u;
  unsigned const           lt    = (1u << lane) - 1u;
  uint64_t const           base  = static_cast<uint64_t>(tile) * RX_TILE;
  unsigned long long const tag   = static_cast<unsigned long long>(a.pass + 1) << 34;
  uint32_t const           first = w * (32 * RX_ITEMS) + lane;
  uint32_t const* const    kin   = a.kin + base + first;
  uint32_t const* const    vin   = a.vin + base + first;

  // 1. ranks inside the warp's run; slots past the end (last tile only) take
  // the largest digit, so they sort behind every pair of the tile
  uint32_t key[RX_ITEMS], pos[RX_ITEMS / 2]; // pos: two 16-bit values per register, ranks first
#pragma unroll
  for (int r = 0; r < RX_ITEMS; ++r) key[r] = FULL || first + r * 32 < n ? kin[r * 32] : 0xFFFFFFFFu;
#pragma unroll
  for (int r = 0; r < RX_ITEMS; ++r) {
    uint32_t const d     = (key[r] >> a.shift) & a.mask;
    unsigned const peers = rx_peers(d);
    uint32_t const seen  = sm.wcnt[w][d];
    __syncwarp();
    if ((peers & lt) == 0) sm.wcnt[w][d] = static_cast<uint16_t>(seen + __popc(peers));
    __syncwarp();
    uint32_t const rank = seen + __popc(peers & lt);
    if (r % 2 == 0) pos[r / 2] = rank;
    else pos[r / 2] |= rank << 16;
  }
  __syncthreads();
  // 2. the tile's counts, published before anything else waits
  uint32_t c = 0;
  if (t < RX_BINS) {
#pragma unroll
    for (int ww = 0; ww < RX_WARPS; ++ww) {
      uint32_t const x  = sm.wcnt[ww][t];
      sm.wcnt[ww][t]    = static_cast<uint16_t>(c);
      c += x;
    }
    if (tile) st_relaxed64(a.look + static_cast<uint64_t>(tile) * RX_BINS + t, tag | RX_SUM | c);
  }
  uint32_t const off = rx_scan_bins(c, sm.wsum);
  if (tile == 0) {
    // the first tile's prefix holds the digits below as well
    uint32_t const g     = t < RX_BINS ? a.hist[t] : 0u;
    uint32_t const start = rx_scan_bins(g, sm.wsum);
    if (t < RX_BINS) {
      sm.base[t] = start - off;
      st_relaxed64(a.look + t, tag | RX_PREFIX | static_cast<uint32_t>(start + c));
    }
  }
  if (t < RX_BINS) sm.off[t] = off;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RX_ITEMS; ++r) {
    uint32_t const d    = (key[r] >> a.shift) & a.mask;
    uint32_t const slot = sm.off[d] + sm.wcnt[w][d]; // + rank < RX_TILE: no carry between the halves
    pos[r / 2] += r % 2 ? slot << 16 : slot;
    sm.buf[r % 2 ? pos[r / 2] >> 16 : pos[r / 2] & 0xFFFFu] = key[r];
  }
  uint32_t val[RX_ITEMS];
#pragma unroll
  for (int r = 0; r < RX_ITEMS; ++r) val[r] = FULL || first + r * 32 < n ? vin[r * 32] : 0u;
  if (tile && t < RX_BINS) {
    uint32_t sum = 0, polls = 0, j = tile;
    bool     done = false;
    while (j > 0 && !done) {
      // RX_LOOK earlier tiles' words in flight at once
      unsigned long long x[RX_LOOK];
#pragma unroll
      for (uint32_t q = 0; q < RX_LOOK; ++q) x[q] = j > q ? ld_relaxed64(a.look + static_cast<uint64_t>(j - 1 - q) * RX_BINS + t) : 0ull;
      uint32_t taken = 0;
#pragma unroll
      for (uint32_t q = 0; q < RX_LOOK; ++q)
        if (!done && taken == q && (x[q] >> 34) == static_cast<unsigned long long>(a.pass + 1)) {
          sum += static_cast<uint32_t>(x[q]);
          done = (x[q] & RX_PREFIX) != 0;
          ++taken;
        }
      j -= taken;
      if (taken == 0 && ++polls > a.polls) break;
    }
    if (!done) {
      // waited for tile j - 1 in vain: its count and all before it from the
      // keys, and the digits below
#pragma unroll 4
      for (uint64_t i = 0, end = static_cast<uint64_t>(j) * RX_TILE; i < end; ++i) sum += ((a.kin[i] >> a.shift) & a.mask) == t;
#pragma unroll 1
      for (uint32_t d = 0; d < t; ++d) sum += a.hist[d];
    }
    sm.base[t] = sum - off;
    st_relaxed64(a.look + static_cast<uint64_t>(tile) * RX_BINS + t, tag | RX_PREFIX | static_cast<uint32_t>(sum + c));
  }
  __syncthreads();
  // 3. keys, then values, out in digit order
  uint32_t out[RX_ITEMS];
#pragma unroll
  for (int r = 0; r < RX_ITEMS; ++r) {
    uint32_t const p = r * RX_THREADS + t;
    uint32_t const k = sm.buf[p];
    out[r]           = sm.base[(k >> a.shift) & a.mask] + p;
    if (FULL || p < n) a.kout[out[r]] = k;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RX_ITEMS; ++r) sm.buf[r % 2 ? pos[r / 2] >> 16 : pos[r / 2] & 0xFFFFu] = val[r];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RX_ITEMS; ++r) {
    uint32_t const p = r * RX_THREADS + t;
    if (FULL || p < n) a.vout[out[r]] = sm.buf[p];
  }
}

__global__ void __launch_bounds__(RX_THREADS, RX_BLOCKS)
k_radix_pass(rx_args const __grid_constant__ a)
{
  __shared__ rx_smem sm;
  if (threadIdx.x == 0) sm.tile = atomicAdd(a.ticket, 1u);
  for (unsigned i = threadIdx.x; i < RX_WARPS * RX_BINS / 2; i += RX_THREADS) reinterpret_cast<uint32_t*>(&sm.wcnt[0][0])[i] = 0;
  __syncthreads();
  uint32_t const tile = sm.tile;
  uint64_t const left = a.count - static_cast<uint64_t>(tile) * RX_TILE;
  if (left >= RX_TILE) rx_tile<true>(a, sm, tile, RX_TILE);
  else rx_tile<false>(a, sm, tile, static_cast<uint32_t>(left));
}

// Clears the scratch and counts every pass's digits.
void
rx_begin(kspn_context* ctx, rx_digits const& d, uint32_t const* keys, uint64_t count, uint32_t* scratch)
{
  cudaStream_t const s = ctx->stream;
  KSPN_CUDA(cudaMemsetAsync(scratch, 0, radix_hist_entries(count) * sizeof(uint32_t), s));
  uint64_t const blocks = (count + 4 * RX_THREADS - 1) / (4 * RX_THREADS);
  k_radix_hist<<<static_cast<unsigned>(blocks < 148ull * 4 ? blocks : 148ull * 4), RX_THREADS, 0, s>>>(keys, count, d, scratch);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 1;
}

void
rx_pass(kspn_context* ctx, rx_digits const& d, int p, uint32_t const* kin, uint32_t const* vin, uint32_t* kout, uint32_t* vout, uint64_t count, uint32_t* scratch)
{
  k_radix_pass<<<div_up(count, RX_TILE), RX_THREADS, 0, ctx->stream>>>(rx_args{ kin, vin, kout, vout, count, d.shift[p], d.mask[p], p, scratch + p * RX_BINS, scratch + RX_PASSES * RX_BINS + p,
                                                                              reinterpret_cast<unsigned long long*>(scratch + RX_HEAD), RX_POLLS });
  KSPN_CHECK_LAUNCH();
  ctx->launches += 1;
}

} // namespace

size_t
radix_hist_entries(uint64_t count)
{
  return RX_HEAD + 2 * static_cast<size_t>(RX_BINS) * div_up(count ? count : 1, RX_TILE);
}

int
radix_passes(int begin_bit, int end_bit)
{
  return end_bit > begin_bit ? (end_bit - begin_bit + 7) / 8 : 0;
}

bool
radix_sort_alternate(kspn_context* ctx, uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint64_t count, int begin_bit, int end_bit, uint32_t* hist)
{
  if (count <= 1 || end_bit <= begin_bit) return false;
  rx_digits const d = rx_plan(begin_bit, end_bit);
  rx_begin(ctx, d, keys, count, hist);
  uint32_t *ki = keys, *vi = vals, *ko = keys_alt, *vo = vals_alt;
  for (int p = 0; p < d.passes; ++p) {
    rx_pass(ctx, d, p, ki, vi, ko, vo, count, hist);
    std::swap(ki, ko);
    std::swap(vi, vo);
  }
  return ki != keys;
}

void
radix_sort_pairs(kspn_context* ctx, uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint64_t count, int begin_bit, int end_bit, uint32_t* hist)
{
  if (!radix_sort_alternate(ctx, keys, vals, keys_alt, vals_alt, count, begin_bit, end_bit, hist)) return;
  KSPN_CUDA(cudaMemcpyAsync(keys, keys_alt, count * sizeof(uint32_t), cudaMemcpyDeviceToDevice, ctx->stream));
  KSPN_CUDA(cudaMemcpyAsync(vals, vals_alt, count * sizeof(uint32_t), cudaMemcpyDeviceToDevice, ctx->stream));
}

void
radix_sort_pairs_to(kspn_context* ctx, uint32_t const* kin, uint32_t const* vin, uint32_t* kout, uint32_t* vout, uint32_t* ka, uint32_t* va, uint32_t* kb, uint32_t* vb, uint64_t count, int end_bit, uint32_t* hist)
{
  if (count == 0) return;
  if (end_bit <= 0 || count == 1) {
    KSPN_CUDA(cudaMemcpyAsync(kout, kin, count * sizeof(uint32_t), cudaMemcpyDeviceToDevice, ctx->stream));
    if (vout != vin) KSPN_CUDA(cudaMemcpyAsync(vout, vin, count * sizeof(uint32_t), cudaMemcpyDeviceToDevice, ctx->stream));
    return;
  }
  rx_digits const d = rx_plan(0, end_bit);
  rx_begin(ctx, d, kin, count, hist);
  uint32_t const *ki = kin, *vi = vin;
  for (int p = 0; p < d.passes; ++p) {
    // the last pass lands in (kout, vout); the ones before alternate A / B
    // so that no pass reads and writes one buffer
    bool const last = p == d.passes - 1;
    uint32_t*  ko   = last ? kout : (((d.passes - 1 - p) & 1) ? ka : kb);
    uint32_t*  vo   = last ? vout : (((d.passes - 1 - p) & 1) ? va : vb);
    rx_pass(ctx, d, p, ki, vi, ko, vo, count, hist);
    ki = ko;
    vi = vo;
  }
}

} // namespace kspn
