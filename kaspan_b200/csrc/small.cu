// One decomposition in one block: graphs whose rows, offsets and search state
// fit one SM's shared memory.
//
// A graph of a few thousand vertices has no work to share out: on the
// grid-wide path every search level costs three or four grid barriers and two
// dependent global loads, about 12 us, whatever it holds.  Here a level is
// one block barrier between shared-memory accesses (about 0.4 us when thin),
// and checks, searches, peeling and ids are one launch whose counts the
// kernel writes to pinned host memory itself.
//
// The steps are the FAST pipeline's: trim-1 with the pivot (largest in * out,
// lowest id on ties), forward and backward search from it, the trim fixpoint;
// what is left then goes through rounds of a min-label search from every
// vertex at once and the trim fixpoint.  The labels carry a priority that is
// a new permutation of the ids each round, so a chain of components takes
// O(log n) rounds in expectation, not one round per component.
//
// Whole call, grid-wide -> here: G(n, m) n 1,000, degree 4: 188 -> 32 us;
// n 8,000, degree 4 (228 of 231 KB): 262 -> 86 us; n 300, degree 2: 409 (at
// its slowest) -> 32 us; random geometric graphs n 1,000 / 3,000 / 8,000:
// 1240 / 586 / 866 -> 71 / 117 / 199 us; R-MAT scale 10, degree 16 and scale
// 13, degree 4: 134, 169 -> 36, 71 us.  So the line is what fits: at the
// limit the block is still at least twice as fast.  About 12 us of each call
// are the launch and the wait; the rest is the levels' chain of dependent
// shared-memory accesses.  Forward and backward search one after the other
// instead of side by side: 37, 90, 144 us for n 1,000, 8,000 and the 3,000
// random geometric one.  512 threads: 34, 120, 119 us.
#include "small.cuh"

namespace kspn {

namespace {

struct sm_layout // byte offsets of the arrays in dynamic shared memory
{
  uint32_t lab, und, open, vis, inq, q0, q1, fh, bh, fc, bc, bytes;
};

__host__ __device__ constexpr sm_layout
sm_layout_of(uint32_t n, uint32_t m)
{
  uint32_t const words = (n + 31) / 32 * 4, half = (n + 2) / 2 * 4, row = (m + 1) / 2 * 4;
  sm_layout      l{};
  l.lab   = 0;
  l.und   = l.lab + 4 * n;
  l.open  = l.und + words;
  l.vis   = l.open + words;
  l.inq   = l.vis + words;
  l.q0    = l.inq + words;
  l.q1    = l.q0 + half;
  l.fh    = l.q1 + half;
  l.bh    = l.fh + half;
  l.fc    = l.bh + half;
  l.bc    = l.fc + row;
  l.bytes = l.bc + row;
  return l;
}

// Forward and backward search from the pivot side by side (even and odd
// warps), so that the levels are the longer search's, not both's; then the
// ids of what both reached.  Returns the component's size.
template<int T>
__device__ uint32_t
sm_fwbw(sm_graph& G, uint32_t pivot, uint32_t* __restrict__ ids, uint32_t& levels_fw, uint32_t& levels_bw, uint32_t& edges)
{
  unsigned const lane = threadIdx.x & 31u;
  bool const     odd  = (threadIdx.x >> 5) & 1u;
  uint32_t const tid  = (threadIdx.x >> 6) * 32 + lane;
  if (threadIdx.x < 2) {
    (threadIdx.x ? G.q1 : G.q0)[0] = static_cast<uint16_t>(pivot);
    sm_take(threadIdx.x ? G.vis : G.open, pivot);
  }
  __syncthreads();
  uint32_t* const       open = odd ? G.vis : G.open;
  uint16_t* const       list = odd ? G.q1 : G.q0;
  uint16_t const* const head = odd ? G.bh : G.fh;
  uint16_t const* const rows = odd ? G.bc : G.fc;
  uint2                 lo = make_uint2(0, 0), hi = make_uint2(1, 1);
  while (lo.x < hi.x || lo.y < hi.y) {
    uint32_t const a = odd ? lo.y : lo.x, b = odd ? hi.y : hi.x;
    edges += sm_expand<T / 2>(
      G, tid, odd, list + a, b - a, head, rows, list + b, [](uint32_t) {}, [&](uint32_t, uint32_t w) { return sm_bit(open, w) && sm_take(open, w); });
    levels_fw += lo.x < hi.x;
    levels_bw += lo.y < hi.y;
    uint2 const c = sm_level_end(G);
    lo            = hi;
    hi.x += c.x, hi.y += c.y;
  }
  // the members, a bitmap word at a time; the smallest one names them
  uint32_t mn = 0xFFFFFFFFu, size = 0;
  for (uint32_t w = threadIdx.x; w < G.words; w += T) {
    uint32_t const x = G.und[w] & ~(G.open[w] | G.vis[w]);
    G.open[w]        = x;
    G.und[w] &= ~x;
    size += __popc(x);
    if (x) mn = min(mn, w * 32 + __ffs(x) - 1);
  }
  mn   = __reduce_min_sync(0xFFFFFFFFu, mn);
  size = __reduce_add_sync(0xFFFFFFFFu, size);
  if (lane == 0 && size) atomicMin(&G.S->minid, mn), atomicAdd(&G.S->size, size);
  __syncthreads();
  mn = G.S->minid;
  for (uint32_t v = threadIdx.x; v < G.n; v += T)
    if (sm_bit(G.open, v)) ids[v] = mn;
  return G.S->size;
}

template<int T>
__global__ void __launch_bounds__(T, 1)
k_scc_small(uint32_t n, uint32_t m, uint64_t const* __restrict__ fh, uint32_t const* __restrict__ fc, uint64_t const* __restrict__ bh, uint32_t const* __restrict__ bc, uint32_t* __restrict__ ids,
            small_result* __restrict__ res)
{
  extern __shared__ __align__(16) unsigned char sm_dyn[];
  __shared__ sm_shared                          S;
  sm_layout const                               l    = sm_layout_of(n, m);
  unsigned const                                lane = threadIdx.x & 31u;
  auto const                                    u16  = [&](uint32_t at) { return reinterpret_cast<uint16_t*>(sm_dyn + at); };
  auto const                                    u32  = [&](uint32_t at) { return reinterpret_cast<uint32_t*>(sm_dyn + at); };
  sm_graph G{ n, (n + 31) / 32, u32(l.lab), u32(l.und), u32(l.open), u32(l.vis), u32(l.inq), u16(l.q0), u16(l.q1), u16(l.fh), u16(l.bh), u16(l.fc), u16(l.bc), &S, 0 };
  if (threadIdx.x == 0) S.best = S.edges = 0, S.bad = 0, S.minid = 0xFFFFFFFFu, S.decided = S.size = 0;
  if (threadIdx.x < 6) S.cnt[threadIdx.x >> 1][threadIdx.x & 1] = 0;
  // the graph into shared memory, 16-bit; every value is checked on the way
  uint32_t       bad = 0;
  uint16_t* const wfh = u16(l.fh); uint16_t* const wbh = u16(l.bh); uint16_t* const wfc = u16(l.fc); uint16_t* const wbc = u16(l.bc);
  constexpr int ILP = 4;
  for (uint32_t i0 = threadIdx.x; i0 <= n; i0 += ILP * T) {
    uint64_t a[ILP], b[ILP];
#pragma unroll
    for (int k = 0; k < ILP; ++k) {
      uint32_t const i = i0 + k * T;
      a[k] = b[k] = 0;
      if (i <= n) a[k] = fh[i], b[k] = bh[i];
    }
#pragma unroll
    for (int k = 0; k < ILP; ++k) {
      uint32_t const i = i0 + k * T;
      if (i > n) continue;
      if (a[k] > m || b[k] > m) bad |= 1u;
      if ((i == 0 && (a[k] | b[k])) || (i == n && (a[k] != m || b[k] != m))) bad |= 2u;
      wfh[i] = static_cast<uint16_t>(a[k]);
      wbh[i] = static_cast<uint16_t>(b[k]);
    }
  }
  for (uint32_t e0 = threadIdx.x; e0 < m; e0 += ILP * T) {
    uint32_t a[ILP], b[ILP];
#pragma unroll
    for (int k = 0; k < ILP; ++k) {
      uint32_t const e = e0 + k * T;
      a[k] = b[k] = 0;
      if (e < m) a[k] = fc[e], b[k] = bc[e];
    }
#pragma unroll
    for (int k = 0; k < ILP; ++k) {
      uint32_t const e = e0 + k * T;
      if (e >= m) continue;
      if (a[k] >= n || b[k] >= n) bad |= 4u;
      wfc[e] = static_cast<uint16_t>(a[k]);
      wbc[e] = static_cast<uint16_t>(b[k]);
    }
  }
  __syncthreads();
  // trim-1, pivot, ids; offsets that decrease are a fault
  unsigned long long best = 0;
  uint32_t           dead = 0;
  for (uint32_t v = threadIdx.x; v < G.words * 32; v += T) {
    bool live = false;
    if (v < n) {
      uint32_t const f0 = G.fh[v], f1 = G.fh[v + 1], b0 = G.bh[v], b1 = G.bh[v + 1];
      if (f0 > f1 || b0 > b1) bad |= 1u;
      live = f1 != f0 && b1 != b0;
      dead += !live;
      if (live) {
        unsigned long long const key = static_cast<unsigned long long>((f1 - f0) * (b1 - b0)) << 32 | (0xFFFFFFFFu - v);
        best                         = key > best ? key : best;
      }
    }
    unsigned const word = __ballot_sync(0xFFFFFFFFu, live);
    if (lane == 0) G.und[v >> 5] = G.open[v >> 5] = G.vis[v >> 5] = word;
  }
  dead = __reduce_add_sync(0xFFFFFFFFu, dead);
#pragma unroll
  for (int sh = 16; sh; sh >>= 1) {
    unsigned long long const o = __shfl_xor_sync(0xFFFFFFFFu, best, sh);
    best                       = o > best ? o : best;
  }
  if (lane == 0 && best) atomicMax(&S.best, best);
  if (lane == 0 && dead) atomicAdd(&S.decided, dead);
  if (bad) atomicOr(&S.bad, bad);
  __syncthreads();
  if (S.bad) { // before any use of a row
    if (threadIdx.x == 0) res->bad = S.bad;
    return;
  }
  for (uint32_t v = threadIdx.x; v < n; v += T) ids[v] = v;
  uint32_t const trim_first = S.decided, pivot = S.best ? 0xFFFFFFFFu - static_cast<uint32_t>(S.best) : n;
  uint32_t       rem = n - trim_first, fwbw = 0, trim = 0, rest = 0, rounds = 0, levels_fw = 0, levels_bw = 0, edges = 0;
  if (rem) {
    fwbw = sm_fwbw<T>(G, pivot, ids, levels_fw, levels_bw, edges);
    rem -= fwbw;
    if (rem) {
      trim = sm_trim<T>(G);
      rem -= trim;
    }
    while (rem) { // a round decides at least one component
      uint32_t d = sm_label_round<T>(G, rounds++, ids, [](uint32_t v) { return v; }, edges);
      if (d < rem) d += sm_trim<T>(G);
      rest += d;
      rem -= d;
    }
  }
  edges = __reduce_add_sync(0xFFFFFFFFu, edges);
  if (lane == 0) atomicAdd(&S.edges, static_cast<unsigned long long>(edges));
  __syncthreads();
  if (threadIdx.x == 0) {
    res->bad        = 0;
    res->trim_first = trim_first;
    res->fwbw       = fwbw;
    res->trim       = trim;
    res->rest       = rest;
    res->rounds     = rounds;
    res->pivot      = pivot;
    res->levels_fw  = levels_fw;
    res->levels_bw  = levels_bw;
    res->edges      = S.edges;
  }
}

constexpr int      SM_T     = 1024;
constexpr uint32_t SM_BYTES = 226 * 1024; // of the 227 KB a block may have; the rest is sm_shared's

} // namespace

bool
small_fits(dgraph const& g)
{
  return g.n != 0 && g.n <= 0xFFFFu && g.m <= 0xFFFFu && sm_layout_of(g.n, static_cast<uint32_t>(g.m)).bytes <= SM_BYTES;
}

void
scc_small_async(kspn_context* ctx, dgraph const& g, uint32_t* scc_id, small_result* res)
{
  uint32_t const m = static_cast<uint32_t>(g.m), bytes = sm_layout_of(g.n, m).bytes;
  if (!ctx->small_ready) {
    KSPN_CUDA(cudaFuncSetAttribute(k_scc_small<SM_T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SM_BYTES)));
    ctx->small_ready = true;
  }
  k_scc_small<SM_T><<<1, SM_T, bytes, ctx->stream>>>(g.n, m, g.fh, g.fc, g.bh, g.bc, scc_id, res);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 1;
}

} // namespace kspn
