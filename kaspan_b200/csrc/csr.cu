// Graph construction on the device:
//  * transpose (CSC build): the reference's backward_complement_graph
//    (kaspan/scc/backward_complement.hpp:22-68) is a counting sort that
//    leaves each in-row ascending; here a stable radix sort of the
//    (target, source) pairs, taken in CSR order, gives the same rows.
//  * build_csr: edge list -> CSR with self-loops and duplicates removed and
//    rows ascending (two stable sorts, then an adjacent-difference compact).
//  * validate: monotone offsets, head[0] == 0, head[n] == m, ids < n.
#include "prim.cuh"

#include <algorithm>

namespace kspn {

namespace {

// src[e] = u for every edge e of row u.  Small rows by their own lane,
// rows of 64+ entries by the whole warp.  The offsets may not have been
// checked yet: nothing past src[m) is written.
__global__ void
k_expand_rows(uint32_t n, uint64_t m, uint64_t const* __restrict__ head, uint32_t* __restrict__ src)
{
  uint64_t const tid  = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  unsigned const lane = threadIdx.x & 31u;
  uint64_t const wbase = tid - lane; // first vertex of this warp's group
  if (wbase >= n) return;
  uint32_t const u   = static_cast<uint32_t>(tid);
  bool const     ok  = tid < n;
  uint64_t const end = ok ? min(head[u + 1], m) : 0, beg = ok ? min(head[u], end) : 0;
  bool const     big = (end - beg) >= 64;
  if (!big)
    for (uint64_t e = beg; e < end; ++e) src[e] = u;
  unsigned todo = __ballot_sync(0xFFFFFFFFu, big);
  while (todo) {
    unsigned const l  = __ffs(todo) - 1;
    todo &= todo - 1;
    uint64_t const b  = __shfl_sync(0xFFFFFFFFu, beg, l);
    uint64_t const e_ = __shfl_sync(0xFFFFFFFFu, end, l);
    uint32_t const uu = static_cast<uint32_t>(wbase + l);
    for (uint64_t e = b + lane; e < e_; e += 32) src[e] = uu;
  }
}

// head[v] = first index of key v in the ascending keys[0, m) (= m past the
// last key): every boundary between two different keys writes the heads of
// the ids it spans, so each head is written exactly once, without atomics.
// A stream of 4 m + 8 n bytes: four keys per 16-byte load (keys starts on a
// 16-byte boundary), the one before them from the lane below.
__global__ void __launch_bounds__(256)
k_heads_from_sorted(uint32_t n, uint64_t m, uint32_t const* __restrict__ keys, uint64_t* __restrict__ head)
{
  unsigned const lane   = threadIdx.x & 31u;
  uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  uint64_t const quads  = m / 4 + 1; // quad q: the boundaries before entries 4q .. 4q + 3, up to the one after the last entry
  for (uint64_t qb = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x - lane; qb < quads; qb += stride) {
    uint64_t const q  = qb + lane;
    uint64_t const i0 = q * 4;
    // ids >= n (an invalid graph, reported by validation afterwards) are
    // clamped so that no head beyond n is written; past the end: n
    uint32_t k[4] = { n, n, n, n };
    if (i0 + 4 <= m) {
      uint4 const x = *reinterpret_cast<uint4 const*>(keys + i0);
      k[0] = min(x.x, n), k[1] = min(x.y, n), k[2] = min(x.z, n), k[3] = min(x.w, n);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i0 + j < m) k[j] = min(keys[i0 + j], n);
    }
    uint32_t const below = __shfl_up_sync(0xFFFFFFFFu, k[3], 1);
    int64_t        lo    = lane ? below : (i0 == 0 ? -1 : static_cast<int64_t>(i0 <= m ? min(keys[i0 - 1], n) : n));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i0 + j <= m)
        for (int64_t v = lo + 1; v <= static_cast<int64_t>(k[j]); ++v) head[v] = i0 + j;
      lo = k[j];
    }
  }
}

// ---------------------------------------------------------------- sorted edges -> CSR
// (s, d)[0, m_raw) sorted by (s, d): self-loops and repeats are dropped, the
// rest become csr, and head[v] = edges kept before v's first edge.  Chunk c
// of the list belongs to block c of both kernels: k_edges_count counts its
// kept edges, k_edges_to_csr adds up the counts before its own (at most
// ET_CHUNKS of them, in L2) and writes.  Two reads of the list (16 B per raw
// edge) instead of one, but no chunk waits for another: with a decoupled
// look-back the one-pass form took 580 us on the scale-22 R-MAT edge list
// (64 M edges), and a scan of the keep flags into positions, a compaction
// and a pass over the kept sources 1,085 us.  build_csr of that list, both
// sorts included: 6.1 -> 2.95 ms; its transpose 2.8 -> 1.39 ms.
constexpr int      ET_THREADS = 256, ET_ITEMS = 4, ET_TILE = ET_THREADS * ET_ITEMS, ET_WARPS = ET_THREADS / 32;
constexpr uint32_t ET_CHUNKS  = 148 * 8;

// Edge i = (sv, dv) (all lanes of the warp call it, lane l with edge i0 + l):
// is it kept, and the source before it in ps (~0 for the first edge).
__device__ __forceinline__ bool
edge_kept(uint32_t const* s, uint32_t const* d, uint64_t i, uint32_t sv, uint32_t dv, uint32_t& ps)
{
  uint32_t pd = __shfl_up_sync(0xFFFFFFFFu, dv, 1);
  ps          = __shfl_up_sync(0xFFFFFFFFu, sv, 1);
  if ((threadIdx.x & 31u) == 0 && i > 0) ps = s[i - 1], pd = d[i - 1];
  if (i == 0) ps = 0xFFFFFFFFu;
  return sv != dv && !(i > 0 && ps == sv && pd == dv);
}

__global__ void __launch_bounds__(ET_THREADS, 8)
k_edges_count(uint64_t m_raw, uint64_t chunk, uint32_t const* __restrict__ s, uint32_t const* __restrict__ d, uint32_t* __restrict__ cnt)
{
  uint64_t const lo = blockIdx.x * chunk, hi = min(m_raw, lo + chunk);
  uint32_t       c = 0;
  for (uint64_t base = lo; base < hi; base += ET_TILE) {
    uint32_t sv[ET_ITEMS], dv[ET_ITEMS], ps;
#pragma unroll
    for (int r = 0; r < ET_ITEMS; ++r) {
      uint64_t const i = base + r * ET_THREADS + threadIdx.x;
      sv[r] = dv[r] = 0; // not kept
      if (i < hi) sv[r] = s[i], dv[r] = d[i];
    }
#pragma unroll
    for (int r = 0; r < ET_ITEMS; ++r) {
      uint64_t const i = base + r * ET_THREADS + threadIdx.x;
      c += edge_kept(s, d, i < hi ? i : 0, sv[r], dv[r], ps);
    }
  }
  uint32_t total;
  block_exclusive_scan<uint32_t, ET_THREADS>(c, &total);
  if (threadIdx.x == 0) cnt[blockIdx.x] = total;
}

__global__ void __launch_bounds__(ET_THREADS, 8)
k_edges_to_csr(uint32_t n, uint64_t m_raw, uint64_t chunk, uint32_t const* __restrict__ s, uint32_t const* __restrict__ d, uint32_t const* __restrict__ cnt, uint32_t* __restrict__ csr,
               uint64_t* __restrict__ head, uint32_t* __restrict__ m_out)
{
  __shared__ uint32_t s_cnt[2][ET_ITEMS * ET_WARPS]; // kept edges per (row of ET_THREADS edges, warp); tiles alternate
  static_assert(ET_ITEMS * ET_WARPS == 32, "one count per lane");
  unsigned const t = threadIdx.x, w = t >> 5, lane = t & 31u, lt = (1u << lane) - 1u;
  uint64_t const lo = blockIdx.x * chunk, hi = min(m_raw, lo + chunk);
  uint32_t       sum = 0, before; // kept edges before the tile: below m_raw < 2^32
  for (uint32_t k = t; k < blockIdx.x; k += ET_THREADS) sum += cnt[k];
  block_exclusive_scan<uint32_t, ET_THREADS>(sum, &before);
  int flip = 0;
  for (uint64_t base = lo; base < hi; base += ET_TILE, flip ^= 1) {
    uint32_t sv[ET_ITEMS], dv[ET_ITEMS], ps[ET_ITEMS];
    unsigned keep[ET_ITEMS];
#pragma unroll
    for (int r = 0; r < ET_ITEMS; ++r) {
      uint64_t const i = base + r * ET_THREADS + t;
      sv[r] = dv[r] = 0;
      if (i < hi) sv[r] = s[i], dv[r] = d[i];
    }
#pragma unroll
    for (int r = 0; r < ET_ITEMS; ++r) {
      uint64_t const i = base + r * ET_THREADS + t;
      keep[r]          = __ballot_sync(0xFFFFFFFFu, edge_kept(s, d, i < hi ? i : 0, sv[r], dv[r], ps[r]));
      if (lane == 0) s_cnt[flip][r * ET_WARPS + w] = __popc(keep[r]);
    }
    __syncthreads();
    uint32_t const mine = s_cnt[flip][lane]; // every warp scans the counts for itself
    uint32_t       incl = mine;
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
      uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, dd);
      if (lane >= static_cast<unsigned>(dd)) incl += y;
    }
#pragma unroll
    for (int r = 0; r < ET_ITEMS; ++r) {
      uint64_t const i   = base + r * ET_THREADS + t;
      uint32_t const pos = before + __shfl_sync(0xFFFFFFFFu, incl - mine, r * ET_WARPS + w) + __popc(keep[r] & lt);
      uint32_t const k   = (keep[r] >> lane) & 1u;
      if (k) csr[pos] = dv[r];
      if (i < hi && (ps[r] != sv[r] || i == 0 || i + 1 == m_raw)) {
        // the rows that start at this edge (ids >= n, an invalid list, are
        // clamped), and after the last edge the rows past it
        uint32_t const up = min(sv[r], n);
        for (uint64_t v = i == 0 ? 0 : static_cast<uint64_t>(min(ps[r], n)) + 1; v <= up; ++v) head[v] = pos;
        if (i + 1 == m_raw) {
          for (uint64_t v = static_cast<uint64_t>(up) + 1; v <= n; ++v) head[v] = pos + k;
          *m_out = pos + k;
        }
      }
    }
    before += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
}

// One direction's checks per grid row (blockIdx.y: CSR, transpose), both in
// one launch.  A pure stream of 4m bytes per direction, and 8(n+1) more with
// `heads` (false: k_trim_first, which reads every offset next, checks them).
// The ids are read 16 bytes at a time with VA_ILP loads in flight per thread
// (the rows' array may start at any 4-byte address: the ids before the first
// and after the last 16-byte boundary are read one by one).  R-MAT scale 24
// (n 16.8 M, m 263 M), both directions: 886 us with one 4-byte load per
// thread and step, 490 us with 4 x 16 bytes and the offsets; ids alone 470 us
// with 4 x 16 bytes, 345 us with 8 (6.1 TB/s; 16: 340 us), which need the
// grid of 4 blocks per SM and row or more (2: 470 us, 3: 365 us).
constexpr int VA_THREADS = 256, VA_ILP = 8;
struct graph_rows
{
  uint64_t const* head;
  uint32_t const* csr;
};

__global__ void __launch_bounds__(VA_THREADS)
k_validate(uint32_t n, uint64_t m, graph_rows fw, graph_rows bw, bool heads, uint32_t* __restrict__ err)
{
  graph_rows const g      = blockIdx.y ? bw : fw;
  uint64_t const   stride = static_cast<uint64_t>(gridDim.x) * VA_THREADS;
  uint64_t const   tid    = static_cast<uint64_t>(blockIdx.x) * VA_THREADS + threadIdx.x;
  uint32_t         bad    = 0;
  for (uint64_t i0 = heads ? tid : n; i0 < n; i0 += VA_ILP * stride) {
    uint64_t a[VA_ILP], b[VA_ILP];
#pragma unroll
    for (int k = 0; k < VA_ILP; ++k) {
      uint64_t const i = i0 + k * stride;
      a[k] = b[k] = 0;
      if (i < n) a[k] = g.head[i], b[k] = g.head[i + 1];
    }
#pragma unroll
    for (int k = 0; k < VA_ILP; ++k) bad |= a[k] > b[k] ? 1u : 0u;
  }
  if (heads && tid == 0 && (g.head[0] != 0 || g.head[n] != m)) bad |= 2u;
  uint64_t const lead = min(m, ((16u - (reinterpret_cast<uintptr_t>(g.csr) & 15u)) & 15u) / 4u);
  uint64_t const nv   = (m - lead) / 4;
  auto const*    v    = reinterpret_cast<uint4 const*>(g.csr + lead);
  uint32_t       most = 0; // largest id seen
  for (uint64_t i0 = tid; i0 < nv; i0 += VA_ILP * stride) {
    uint4 x[VA_ILP];
#pragma unroll
    for (int k = 0; k < VA_ILP; ++k) x[k] = i0 + k * stride < nv ? v[i0 + k * stride] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < VA_ILP; ++k) most = max(most, max(max(x[k].x, x[k].y), max(x[k].z, x[k].w)));
  }
  uint64_t const rest = m - lead - nv * 4; // at most 3 ids past the last boundary
  if (tid < lead) most = max(most, g.csr[tid]);
  if (tid < rest) most = max(most, g.csr[lead + nv * 4 + tid]);
  if (m && most >= n) bad |= 4u;
  if (bad) atomicOr(err, bad);
}

// src[e - e0] = u for the edges e in [e0, e1) of rows [u_lo, u_hi) (rows
// clipped to the range).  Small rows by their own lane, rows of 64+
// entries by the whole warp.
__global__ void
k_expand_range(uint32_t u_lo, uint32_t u_hi, uint64_t const* __restrict__ head, uint64_t e0, uint64_t e1, uint32_t* __restrict__ src)
{
  uint64_t const tid   = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  unsigned const lane  = threadIdx.x & 31u;
  uint64_t const wbase = u_lo + tid - lane;
  if (wbase >= u_hi) return;
  uint64_t const uu  = u_lo + tid;
  bool const     ok  = uu < u_hi;
  uint64_t       beg = ok ? head[uu] : 0, end = ok ? head[uu + 1] : 0;
  beg                = beg < e0 ? e0 : beg;
  end                = end > e1 ? e1 : end;
  end                = end < beg ? beg : end;
  bool const big = (end - beg) >= 64;
  if (!big)
    for (uint64_t e = beg; e < end; ++e) src[e - e0] = static_cast<uint32_t>(uu);
  for (unsigned todo = __ballot_sync(0xFFFFFFFFu, big); todo; todo &= todo - 1) {
    unsigned const l  = __ffs(todo) - 1;
    uint64_t const b  = __shfl_sync(0xFFFFFFFFu, beg, l);
    uint64_t const e_ = __shfl_sync(0xFFFFFFFFu, end, l);
    uint32_t const u  = static_cast<uint32_t>(wbase + l);
    for (uint64_t e = b + lane; e < e_; e += 32) src[e - e0] = u;
  }
}

// Offsets of one sorted chunk's entries inside their CSC rows, one block per
// RO_THREADS * RO_ITEMS consecutive entries (each thread RO_ITEMS of them):
// an entry's run of equal keys (one target) starts at the largest run start
// at or before it (a block-wide max-scan; a run that began in an earlier
// block is found by a binary search over the sorted keys), the run's start
// reads the target's placed count once and shares it in shared memory, and
// off[i] = that count + i's rank in the run.  One random read per run
// instead of two per entry.
constexpr int RO_THREADS = 256, RO_ITEMS = 8;
__global__ void __launch_bounds__(RO_THREADS)
k_run_offsets(uint32_t n, uint32_t const* __restrict__ keys, uint32_t cnt, uint32_t const* __restrict__ indeg, uint32_t* __restrict__ off)
{
  __shared__ uint32_t s_base[RO_THREADS * RO_ITEMS];
  __shared__ uint32_t s_wmax[RO_THREADS / 32];
  __shared__ uint32_t s_pre, s_prebase;
  uint32_t const b0 = blockIdx.x * (RO_THREADS * RO_ITEMS);
  if (b0 >= cnt) return;
  uint32_t const i0 = b0 + threadIdx.x * RO_ITEMS;
  uint32_t       key[RO_ITEMS];
  uint32_t       last = 0; // largest run start among this thread's items (0: none)
  bool           has  = false;
#pragma unroll
  for (int k = 0; k < RO_ITEMS; ++k) {
    uint32_t const i = i0 + k;
    key[k]           = i < cnt ? keys[i] : UNDECIDED;
    bool const start = i < cnt && (i == 0 || keys[i - 1] != key[k]);
    if (start) last = i, has = true;
  }
  if (threadIdx.x == 0) {
    // the run holding the block's first entry may have started earlier
    uint32_t const v = keys[b0];
    uint32_t       lo = 0, hi = b0; // first index in [0, b0] whose key is v
    if (b0 > 0 && keys[b0 - 1] == v) {
      while (lo < hi) {
        uint32_t const mid = lo + (hi - lo) / 2;
        if (keys[mid] >= v) hi = mid;
        else lo = mid + 1;
      }
    } else lo = b0;
    s_pre     = lo;
    s_prebase = v < n ? indeg[v] : 0u;
  }
  // block-wide inclusive max-scan of the threads' last run starts
  uint32_t incl = has ? last : 0u;
  unsigned const lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= static_cast<unsigned>(d)) incl = max(incl, y);
  }
  if (lane == 31) s_wmax[wid] = incl;
  __syncthreads();
  uint32_t prev = s_pre; // starts before this thread's first item
  for (uint32_t w = 0; w < wid; ++w) prev = max(prev, s_wmax[w]);
  uint32_t const wexcl = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
  if (lane > 0) prev = max(prev, wexcl);
  // run starts in this block publish their target's placed count
  uint32_t gstart[RO_ITEMS];
  uint32_t cur = prev;
#pragma unroll
  for (int k = 0; k < RO_ITEMS; ++k) {
    uint32_t const i = i0 + k;
    if (i < cnt && (i == 0 || keys[i - 1] != key[k])) {
      cur                = i;
      s_base[i - b0]     = key[k] < n ? indeg[key[k]] : 0u;
    }
    gstart[k] = cur;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < RO_ITEMS; ++k) {
    uint32_t const i = i0 + k;
    if (i >= cnt || key[k] >= n) continue;
    uint32_t const base = gstart[k] >= b0 ? s_base[gstart[k] - b0] : s_prebase;
    off[i]              = base + (i - gstart[k]);
  }
}

// placed count of each run's target, after the chunk: its last entry's
// offset + 1
__global__ void
k_run_ends(uint32_t n, uint32_t const* __restrict__ keys, uint32_t cnt, uint32_t const* __restrict__ off, uint32_t* __restrict__ indeg)
{
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
    uint32_t const v = keys[i];
    if (v < n && (i + 1 == cnt || keys[i + 1] != v)) indeg[v] = off[i] + 1;
  }
}

// Placement in bands: band b holds the vertices [bv[b], bv[b+1]) whose CSC
// rows fill about 1/nb of bc; bv[b] = first vertex whose head reaches
// b * m / nb.
__global__ void
k_band_vertices(uint32_t n, uint64_t m, uint64_t const* __restrict__ head, uint32_t nb, uint32_t* __restrict__ bv)
{
  uint32_t const b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > nb) return;
  uint64_t const target = b == nb ? m + 1 : (m / nb) * b + (m % nb) * b / nb;
  uint32_t       lo = 0, hi = n; // first v in [0, n] with head[v] >= target (n if none)
  while (lo < hi) {
    uint32_t const mid = lo + (hi - lo) / 2;
    if (head[mid] >= target) hi = mid;
    else lo = mid + 1;
  }
  bv[b] = b == 0 ? 0u : (b == nb ? n : lo);
}

// seg[b * nc + c] = first entry of sorted chunk c with key >= bv[b]
__global__ void
k_band_segments(uint32_t const* __restrict__ skeys, uint64_t m, uint64_t chunk, uint32_t nc, uint32_t nb, uint32_t const* __restrict__ bv, uint32_t* __restrict__ seg)
{
  uint32_t const t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (nb + 1) * nc) return;
  uint32_t const  b = t / nc, c = t % nc;
  uint64_t const  e0  = c * chunk;
  uint32_t const  cnt = static_cast<uint32_t>((e0 + chunk < m ? e0 + chunk : m) - e0);
  uint32_t const* k   = skeys + e0;
  uint32_t const  key = bv[b];
  uint32_t        lo = 0, hi = cnt;
  while (lo < hi) {
    uint32_t const mid = lo + (hi - lo) / 2;
    if (k[mid] >= key) hi = mid;
    else lo = mid + 1;
  }
  seg[t] = b == nb ? cnt : lo;
}

// bc[head[v] + off[i]] = source of entry i.  A neighbour id >= n (an
// invalid graph, which validation reports afterwards) splits runs, so
// positions are bounded here instead of trusted.
__global__ void
k_place(uint32_t n, uint64_t m, uint32_t const* __restrict__ keys, uint32_t const* __restrict__ off, uint32_t const* __restrict__ vals, uint64_t const* __restrict__ head, uint32_t* __restrict__ bc)
{
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    uint32_t const v = keys[i];
    if (v >= n) continue;
    uint64_t const p = head[v] + off[i];
    if (p < m) bc[p] = vals[i];
  }
}

// The same placement, band by band: block x of the grid works on band
// x / (nc * per) and chunk (x / per) % nc, so the blocks resident at one
// time write into one or two bands' rows and L2 merges their sectors.
__global__ void
k_place_banded(uint32_t n, uint64_t m, uint64_t chunk, uint32_t nc, uint32_t per, uint32_t const* __restrict__ seg, uint32_t const* __restrict__ keys, uint32_t const* __restrict__ off, uint32_t const* __restrict__ vals, uint64_t const* __restrict__ head, uint32_t* __restrict__ bc)
{
  uint32_t const b = blockIdx.x / (nc * per), c = (blockIdx.x / per) % nc, part = blockIdx.x % per;
  uint32_t const lo = seg[b * nc + c], hi = seg[(b + 1) * nc + c];
  uint64_t const e0 = c * chunk;
  for (uint32_t j = lo + part * blockDim.x + threadIdx.x; j < hi; j += per * blockDim.x) {
    uint64_t const i = e0 + j;
    uint32_t const v = keys[i];
    if (v >= n) continue;
    uint64_t const p = head[v] + off[i];
    if (p < m) bc[p] = vals[i];
  }
}

unsigned
grid_for(uint64_t items, int threads)
{
  uint64_t const b = (items + threads - 1) / threads;
  return static_cast<unsigned>(b < 148ull * 32 ? (b ? b : 1) : 148ull * 32);
}

struct scratch
{
  void*  p     = nullptr;
  size_t bytes = 0;
  template<typename T>
  T* carve(size_t& off, size_t count)
  {
    off      = (off + 255) & ~size_t(255);
    T* ptr   = reinterpret_cast<T*>(static_cast<char*>(p) + off);
    off += count * sizeof(T);
    return ptr;
  }
};

void
alloc_scratch(kspn_context* ctx, scratch& s, size_t bytes)
{
  s.p     = context_buffer(ctx, BUF_BUILD, bytes);
  s.bytes = bytes;
}

} // namespace

void
transpose(kspn_context* ctx, uint32_t n, uint64_t m, uint64_t const* fh, uint32_t const* fc, uint64_t* bh, uint32_t* bc)
{
  cudaStream_t const s = ctx->stream;
  if (n == 0) {
    KSPN_CUDA(cudaMemsetAsync(bh, 0, sizeof(uint64_t), s));
    return;
  }
  size_t const hist_n = radix_hist_entries(m);
  scratch      sc;
  alloc_scratch(ctx, sc, (3 * (m + 64) + hist_n) * sizeof(uint32_t) + 4096);
  size_t    off  = 0;
  uint32_t* ka   = sc.carve<uint32_t>(off, m + 1);
  uint32_t* kb   = sc.carve<uint32_t>(off, m + 1);
  uint32_t* va   = sc.carve<uint32_t>(off, m + 1);
  uint32_t* hist = sc.carve<uint32_t>(off, hist_n);

  // (target, source) pairs sorted by target, read where the targets lie,
  // through A = (ka, va) and B = (kb, bc); the last pass writes B, so the
  // sources start in the value buffer that the first pass does not write
  int const passes = m ? radix_passes(0, bits_for(n)) : 0;
  if (m) {
    uint32_t* const src = passes % 2 ? va : bc;
    k_expand_rows<<<div_up(n, 256), 256, 0, s>>>(n, m, fh, src);
    KSPN_CHECK_LAUNCH();
    radix_sort_pairs_to(ctx, fc, src, kb, bc, ka, va, kb, bc, m, bits_for(n), hist);
  }
  k_heads_from_sorted<<<grid_for(m / 4 + 1, 256), 256, 0, s>>>(n, m, kb, bh);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 2;
}

namespace {
constexpr uint64_t PLACE_BAND_BYTES = 32ull << 20; // a quarter of L2
constexpr uint64_t BAND_MAX         = 4096;
} // namespace

void
upload_transpose(kspn_context* ctx, uint32_t n, uint64_t m, uint64_t const* h_fh, uint32_t const* h_fc, uint64_t* dfh, uint32_t* dfc, uint64_t* dbh, uint32_t* dbc, uint64_t chunk)
{
  cudaStream_t const s = ctx->stream;
  if (!ctx->copy_stream) {
    KSPN_CUDA(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
    KSPN_CUDA(cudaEventCreateWithFlags(&ctx->copy_ev, cudaEventDisableTiming));
  }
  cudaStream_t const cs = ctx->copy_stream;
  if (chunk == 0) chunk = UPLOAD_CHUNK;
  chunk = chunk < m ? chunk : (m ? m : 1);
  // the copies start after the work already queued on the context's stream
  KSPN_CUDA(cudaEventRecord(ctx->copy_ev, s));
  KSPN_CUDA(cudaStreamWaitEvent(cs, ctx->copy_ev, 0));
  KSPN_CUDA(cudaMemcpyAsync(dfh, h_fh, (static_cast<size_t>(n) + 1) * 8, cudaMemcpyHostToDevice, cs));
  if (n == 0 || m == 0) {
    KSPN_CUDA(cudaMemsetAsync(dbh, 0, (static_cast<size_t>(n) + 1) * 8, s));
    KSPN_CUDA(cudaEventRecord(ctx->copy_ev, cs));
    KSPN_CUDA(cudaStreamWaitEvent(s, ctx->copy_ev, 0));
    return;
  }
  if (m >= 0xFFFFFFFFull) throw error{ KSPN_ERR_INVALID_ARGUMENT, "upload_transpose: 2^32-1 or more edges are not supported" };
  // the chunk row ranges come from binary searches over the host offsets
  if (h_fh[0] != 0 || h_fh[n] != m) throw error{ KSPN_ERR_INVALID_GRAPH, "invalid graph: head[0] != 0 or head[n] != m;" };
  size_t const hist_n = radix_hist_entries(chunk);
  size_t const part_n = scan_partial_entries(static_cast<uint64_t>(n) + 1);
  scratch      sc;
  size_t const band_cap = (BAND_MAX + 1) * ((m + chunk - 1) / chunk);
  alloc_scratch(ctx, sc, (3 * (m + 64) + 5 * (chunk + 64) + (static_cast<size_t>(n) + 64) + BAND_MAX + 64 + band_cap + 64 + hist_n) * sizeof(uint32_t) + part_n * sizeof(uint64_t) + 16384);
  size_t    off    = 0;
  uint32_t* skeys  = sc.carve<uint32_t>(off, m);     // chunk-sorted targets
  uint32_t* svals  = sc.carve<uint32_t>(off, m);     // their sources
  uint32_t* roff   = sc.carve<uint32_t>(off, m);     // offset inside the CSC row
  uint32_t* src    = sc.carve<uint32_t>(off, chunk); // sources of the chunk, CSR order
  uint32_t* ka     = sc.carve<uint32_t>(off, chunk);
  uint32_t* va     = sc.carve<uint32_t>(off, chunk);
  uint32_t* kb     = sc.carve<uint32_t>(off, chunk);
  uint32_t* vb     = sc.carve<uint32_t>(off, chunk);
  uint32_t* indeg  = sc.carve<uint32_t>(off, n);
  uint32_t* hist   = sc.carve<uint32_t>(off, hist_n);
  uint64_t* part64 = sc.carve<uint64_t>(off, part_n);
  uint32_t* bv     = sc.carve<uint32_t>(off, BAND_MAX + 1);
  uint32_t* seg    = sc.carve<uint32_t>(off, band_cap);
  KSPN_CUDA(cudaMemsetAsync(indeg, 0, static_cast<size_t>(n) * 4, s));
  int const bits = bits_for(n);
  for (uint64_t e0 = 0; e0 < m; e0 += chunk) {
    uint64_t const e1  = e0 + chunk < m ? e0 + chunk : m;
    uint32_t const cnt = static_cast<uint32_t>(e1 - e0);
    KSPN_CUDA(cudaMemcpyAsync(dfc + e0, h_fc + e0, static_cast<size_t>(cnt) * 4, cudaMemcpyHostToDevice, cs));
    KSPN_CUDA(cudaEventRecord(ctx->copy_ev, cs));
    KSPN_CUDA(cudaStreamWaitEvent(s, ctx->copy_ev, 0)); // the wait binds this record
    // rows holding [e0, e1): the host has the offsets
    uint32_t const u_lo = static_cast<uint32_t>(std::upper_bound(h_fh, h_fh + n + 1, e0) - h_fh - 1);
    uint32_t const u_hi = static_cast<uint32_t>(std::lower_bound(h_fh + u_lo, h_fh + n + 1, e1) - h_fh);
    k_expand_range<<<div_up(static_cast<uint64_t>(u_hi - u_lo), 256), 256, 0, s>>>(u_lo, u_hi, dfh, e0, e1, src);
    KSPN_CHECK_LAUNCH();
    radix_sort_pairs_to(ctx, dfc + e0, src, skeys + e0, svals + e0, ka, va, kb, vb, cnt, bits, hist);
    unsigned const g = grid_for(cnt, 256);
    k_run_offsets<<<div_up(cnt, RO_THREADS * RO_ITEMS), RO_THREADS, 0, s>>>(n, skeys + e0, cnt, indeg, roff + e0);
    k_run_ends<<<g, 256, 0, s>>>(n, skeys + e0, cnt, roff + e0, indeg);
    KSPN_CHECK_LAUNCH();
    ctx->launches += 3;
  }
  exclusive_scan<uint64_t>(s, f_array_u32{ indeg }, n, dbh, part64, &ctx->launches);
  // bands of about PLACE_BAND_BYTES of CSC rows; `per` blocks per (band, chunk)
  uint64_t const nc  = (m + chunk - 1) / chunk;
  uint64_t const nb  = std::max<uint64_t>(1, std::min<uint64_t>((m * 4 + PLACE_BAND_BYTES - 1) / PLACE_BAND_BYTES, n));
  uint32_t const per = static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>(64, m / (nb * nc * 8192))));
  if ((nb + 1) * nc > band_cap || nb * nc * per > 0x7FFFFFFFull) {
    k_place<<<grid_for(m, 256), 256, 0, s>>>(n, m, skeys, roff, svals, dbh, dbc);
    KSPN_CHECK_LAUNCH();
    ctx->launches += 1;
    return;
  }
  k_band_vertices<<<div_up(nb + 1, 256), 256, 0, s>>>(n, m, dbh, static_cast<uint32_t>(nb), bv);
  k_band_segments<<<div_up((nb + 1) * nc, 256), 256, 0, s>>>(skeys, m, chunk, static_cast<uint32_t>(nc), static_cast<uint32_t>(nb), bv, seg);
  k_place_banded<<<static_cast<unsigned>(nb * nc * per), 256, 0, s>>>(n, m, chunk, static_cast<uint32_t>(nc), per, seg, skeys, roff, svals, dbh, dbc);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 3;
}

uint64_t
build_csr(kspn_context* ctx, uint32_t n, uint64_t m_raw, uint32_t* src, uint32_t* dst, uint64_t* head, uint32_t* csr)
{
  cudaStream_t const s = ctx->stream;
  if (m_raw >= 0xFFFFFFFFull) throw error{ KSPN_ERR_INVALID_ARGUMENT, "build_csr: edge lists of 2^32-1 or more entries are not supported" };
  if (m_raw == 0) {
    KSPN_CUDA(cudaMemsetAsync(head, 0, (static_cast<size_t>(n) + 1) * sizeof(uint64_t), s));
    KSPN_CUDA(cudaStreamSynchronize(s));
    return 0;
  }
  size_t const hist_n = radix_hist_entries(m_raw);
  scratch      sc;
  // a third edge array that only the transpose needs: a caller who goes on
  // with it finds its scratch there, instead of freeing this one for a larger
  // one after the caller's own allocations have taken what is left
  alloc_scratch(ctx, sc, (3 * (m_raw + 64) + hist_n) * sizeof(uint32_t) + 4096);
  size_t    off  = 0;
  uint32_t* dalt = sc.carve<uint32_t>(off, m_raw + 1);
  uint32_t* salt = sc.carve<uint32_t>(off, m_raw + 1);
  uint32_t* hist = sc.carve<uint32_t>(off, hist_n);

  // (dst, src) stably by dst, then (src, dst) stably by src => sorted by
  // (src, dst); each sort goes on from the buffers the last pass wrote
  int const b = bits_for(n);
  if (radix_sort_alternate(ctx, dst, src, dalt, salt, m_raw, 0, b, hist)) std::swap(dst, dalt), std::swap(src, salt);
  if (radix_sort_alternate(ctx, src, dst, salt, dalt, m_raw, 0, b, hist)) std::swap(dst, dalt), std::swap(src, salt);
  // chunks of whole tiles, one block each
  uint64_t const chunk  = (div_up(m_raw, ET_TILE) + ET_CHUNKS - 1) / ET_CHUNKS * ET_TILE;
  unsigned const chunks = div_up(m_raw, chunk);
  uint32_t*      cnt    = hist; // ET_CHUNKS counts and the total (the sort's scratch is larger)
  static_assert(ET_CHUNKS + 1 <= 1500, "counts must fit the smallest sort scratch");
  k_edges_count<<<chunks, ET_THREADS, 0, s>>>(m_raw, chunk, src, dst, cnt);
  k_edges_to_csr<<<chunks, ET_THREADS, 0, s>>>(n, m_raw, chunk, src, dst, cnt, csr, head, cnt + ET_CHUNKS);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 2;
  uint32_t m = 0;
  KSPN_CUDA(cudaMemcpyAsync(&m, cnt + ET_CHUNKS, sizeof(m), cudaMemcpyDeviceToHost, s));
  KSPN_CUDA(cudaStreamSynchronize(s));
  return m;
}

void
validate_async(kspn_context* ctx, dgraph const& g, bool transpose_too, bool heads)
{
  uint64_t const items = std::max<uint64_t>(g.m / (4 * VA_ILP), g.n / VA_ILP) + 1;
  unsigned const gx    = static_cast<unsigned>(std::min<uint64_t>(div_up(items, VA_THREADS), 148ull * 8)); // both directions resident at once
  k_validate<<<dim3(gx, transpose_too && g.bh != g.fh ? 2 : 1), VA_THREADS, 0, ctx->stream>>>(g.n, g.m, graph_rows{ g.fh, g.fc }, graph_rows{ g.bh, g.bc }, heads, ctx->ws.ctr + CTR_ERR);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 1;
}

void
validate_check(uint32_t e)
{
  if (!e) return;
  std::string what = "invalid graph:";
  if (e & 1u) what += " offsets decrease;";
  if (e & 2u) what += " head[0] != 0 or head[n] != m;";
  if (e & 4u) what += " neighbour id >= n;";
  throw error{ KSPN_ERR_INVALID_GRAPH, what };
}

void
validate(kspn_context* ctx, dgraph const& g, bool transpose_too)
{
  KSPN_CUDA(cudaMemsetAsync(ctx->ws.ctr + CTR_ERR, 0, sizeof(uint32_t), ctx->stream));
  validate_async(ctx, g, transpose_too, true);
  read_counters(ctx);
  validate_check(ctx->h_ctr[CTR_ERR]);
}

} // namespace kspn
