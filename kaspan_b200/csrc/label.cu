// Multi-pivot label ("colour") search on the device.
//
// Reference: cache_label_search_pull (kaspan/scc/cache_multi_pivot_search_pull.hpp:40-244)
// with map = rotr(., rotation), unmap = rotl(., rotation)
// (cache_rot_label_search_pull, :246-266).  At one rank it computes:
//   FW    label[k] = min map(u) over k's undecided ancestors u (k included),
//         the fixpoint of pulling the minimum over undecided in-neighbours;
//   roots undecided k with label[k] == map(k): decided, id = k;
//   BW    an undecided k is decided (id = unmap(label[k])) when an
//         out-neighbour was decided with the same label.
// The fixpoint is unique, so the device may reach it in any order: here a
// push form over a worklist — every vertex whose label dropped offers it to
// its undecided out-neighbours with atomicMin, and joins the next level's
// worklist (a per-level claim bitmap keeps each vertex once per level).
// The backward closure pushes from newly decided vertices over in-edges.
//
// Learned seed order (kspn_options.learned_seeds, no reference
// counterpart): map(v) = bucket(v) << s | (v ^ mask), where s bits hold a
// vertex id, bucket(v) ranks the pivot model's score (a higher score, a
// smaller bucket, so the vertex wins the min-label propagation) and mask
// varies the order inside a bucket from call to call as the rotation does.
// map is injective on [0, n) and never UNDECIDED, so the fixpoint, the
// roots and the partition are those of any other seed order.
#include "expand.cuh"
#include "mlp.cuh"

namespace kspn {

namespace {

constexpr int L_THREADS  = 256;
constexpr int CTR_NTILES = 8;

unsigned
l_grid(uint64_t items)
{
  uint64_t const b = (items + L_THREADS - 1) / L_THREADS;
  return static_cast<unsigned>(b < 148ull * 8 ? (b ? b : 1) : 148ull * 8);
}

// A search's seed order: the reference's rotated ids, or the learned order.
struct seed_map
{
  uint32_t const* bucket; // null: rotr(v, rot)
  int             rot;
  uint32_t        shift;  // id bits of a learned label
  uint32_t        mask;   // xor of the id bits (this call's order inside a bucket)
  __device__ __forceinline__ uint32_t map(uint32_t v) const { return bucket ? (__ldg(bucket + v) << shift) | (v ^ mask) : rotr32(v, rot); }
  __device__ __forceinline__ uint32_t unmap(uint32_t l) const { return bucket ? (l & ((1u << shift) - 1u)) ^ mask : rotl32(l, rot); }
};

// The pivot model's score of every undecided vertex as a bucket in
// [0, nbuckets - 1): sigmoid(logit) high -> bucket low.  One warp per vertex
// (the features sample its rows); the top bucket stays unused, so no label
// is UNDECIDED.
__global__ void __launch_bounds__(L_THREADS)
k_seed_buckets(uint32_t n, uint32_t const* __restrict__ und, uint64_t const* __restrict__ fh, uint32_t const* __restrict__ fc, uint64_t const* __restrict__ bh,
               uint32_t const* __restrict__ bc, float const* __restrict__ params, uint32_t nbuckets, uint32_t* __restrict__ bucket)
{
  unsigned const lane  = threadIdx.x & 31u;
  uint32_t const words = (n + 31) / 32;
  uint32_t const gw    = (blockIdx.x * L_THREADS + threadIdx.x) >> 5;
  uint32_t const nw    = (gridDim.x * L_THREADS) >> 5;
  // a warp takes 32 words at once (one per lane, one coalesced load), then
  // scores the set bits of the non-empty ones, one vertex at a time
  for (uint32_t wb = gw * 32; wb < words; wb += nw * 32) {
    uint32_t const w  = wb + lane;
    uint32_t       mw = w < words ? und[w] : 0u;
    if (w == words - 1 && (n & 31)) mw &= (1u << (n & 31)) - 1u;
    for (unsigned todo = __ballot_sync(0xFFFFFFFFu, mw != 0); todo; todo &= todo - 1) {
      unsigned const src  = __ffs(todo) - 1;
      uint32_t       word = __shfl_sync(0xFFFFFFFFu, mw, src);
      while (word) {
        uint32_t const v = (wb + src) * 32 + (__ffs(word) - 1);
        word &= word - 1;
        float f[MLP_IN], h1, h2;
        mlp_features(v, fh, fc, bh, bc, f);
        float const z = mlp_forward_w(mlp_weights_global{ params }, f, h1, h2);
        if (lane == 0) {
          float const    p = 1.f / (1.f + expf(-z));
          float const    q = (1.f - p) * static_cast<float>(nbuckets - 1);
          uint32_t const b = q >= static_cast<float>(nbuckets - 2) ? nbuckets - 2 : (q > 0.f ? static_cast<uint32_t>(q) : 0u);
          bucket[v]        = b;
        }
      }
    }
  }
}

// label = map(v) for undecided v (all queued), UNDECIDED otherwise.
__global__ void __launch_bounds__(L_THREADS)
k_label_init(uint32_t n, uint32_t const* __restrict__ und, uint32_t* __restrict__ label, seed_map sm, uint32_t* __restrict__ q, uint32_t* __restrict__ qn)
{
  __shared__ uint32_t s_buf[DENSE_BUF];
  __shared__ uint32_t s_n, s_base;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  block_queue    bq{ s_buf, &s_n };
  uint64_t const span = (static_cast<uint64_t>(n) + L_THREADS - 1) / L_THREADS * L_THREADS;
  for (uint64_t base = static_cast<uint64_t>(blockIdx.x) * L_THREADS; base < span; base += static_cast<uint64_t>(gridDim.x) * L_THREADS) {
    uint64_t const t    = base + threadIdx.x;
    uint32_t const v    = static_cast<uint32_t>(t);
    bool const     live = t < n && bit_get(und, v);
    if (t < n) label[v] = live ? sm.map(v) : UNDECIDED;
    bq.push(live, v);
    __syncthreads();
    if (s_n > DENSE_BUF - L_THREADS) bq.flush(q, qn, &s_base);
  }
  bq.flush(q, qn, &s_base);
}

struct label_fw_op
{
  uint32_t const* und;
  uint32_t*       label;
  uint32_t*       claim_next;
  __device__ __forceinline__ uint32_t probe(uint32_t v) const { return und[v >> 5]; }
  __device__ __forceinline__ bool     operator()(uint32_t u, uint32_t v, bool valid, uint32_t word) const
  {
    if (!valid || !((word >> (v & 31)) & 1u)) return false;
    uint32_t const lu = __ldcg(label + u);
    if (lu >= __ldcg(label + v)) return false;
    uint32_t const old = atomicMin(label + v, lu);
    return lu < old && bit_claim(claim_next, v);
  }
};

// Clears the claim bits of the queue about to be expanded (they were set
// when its entries were pushed); runs before the level that pushes into the
// other bitmap, so no push races with the clearing.
__global__ void
k_unclaim(uint32_t const* __restrict__ q, uint32_t const* __restrict__ qn_ptr, uint32_t* __restrict__ claim)
{
  uint32_t const qn = *qn_ptr;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < qn; i += gridDim.x * blockDim.x) {
    uint32_t const v = q[i];
    atomicAnd(claim + (v >> 5), ~(1u << (v & 31)));
  }
}

__global__ void __launch_bounds__(L_THREADS)
k_label_roots(uint32_t n, uint32_t* __restrict__ und, uint32_t const* __restrict__ label, uint32_t* __restrict__ scc_id, seed_map sm, uint32_t* __restrict__ q, uint32_t* __restrict__ qn, uint32_t* __restrict__ decided)
{
  __shared__ uint32_t s_buf[DENSE_BUF];
  __shared__ uint32_t s_n, s_base;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  block_queue    bq{ s_buf, &s_n };
  uint64_t const span = (static_cast<uint64_t>(n) + L_THREADS - 1) / L_THREADS * L_THREADS;
  uint32_t       dec  = 0;
  for (uint64_t base = static_cast<uint64_t>(blockIdx.x) * L_THREADS; base < span; base += static_cast<uint64_t>(gridDim.x) * L_THREADS) {
    uint64_t const t    = base + threadIdx.x;
    uint32_t const v    = static_cast<uint32_t>(t);
    bool const     root = t < n && bit_get(und, v) && label[v] == sm.map(v);
    bool const     won  = root && bit_take(und, v);
    if (won) {
      scc_id[v] = v;
      ++dec;
    }
    bq.push(won, v);
    __syncthreads();
    if (s_n > DENSE_BUF - L_THREADS) bq.flush(q, qn, &s_base);
  }
  bq.flush(q, qn, &s_base);
  if (dec) atomicAdd(decided, dec);
}

struct label_bw_op
{
  uint32_t*       und;
  uint32_t const* label;
  uint32_t*       scc_id;
  seed_map        sm;
  // u = decided vertex, v = one of its in-neighbours; every push is a decision
  __device__ __forceinline__ uint32_t probe(uint32_t v) const { return und[v >> 5]; }
  __device__ __forceinline__ bool     operator()(uint32_t u, uint32_t v, bool valid, uint32_t word) const
  {
    if (!valid || !((word >> (v & 31)) & 1u)) return false;
    uint32_t const lu = label[u];
    if (label[v] != lu || !bit_take(und, v)) return false;
    scc_id[v] = sm.unmap(lu);
    return true;
  }
};

// ---------------------------------------------------------------- few undecided vertices
// A search over at most LS_VERTICES undecided vertices with at most LS_EDGES
// row entries runs in one block after one listing pass: level after level
// behind block barriers, instead of four launches, a memset and a host round
// trip per level (about 35 us each; a near-critical random graph of 10^6
// vertices left 10,248 vertices and ~490 levels: 17.2 ms).  A level costs
// its chain of dependent accesses, 3 to 4 us.
constexpr int      LS_THREADS  = 1024;
constexpr uint32_t LS_VERTICES = 1u << 15;
constexpr uint64_t LS_EDGES    = 1u << 20;
constexpr uint32_t LS_ROW      = 8192; // longest row one warp walks

struct ls_counts
{
  uint32_t           list_n, longest;
  unsigned long long entries; // out- and in-row entries of the listed vertices
  uint32_t           ran;     // 0: over the limits, nothing done
  uint32_t           err;     // 1: propagation cap, 2: closure cap
  uint32_t           decided;
  uint32_t           pad;
  unsigned long long edges;   // row entries walked
};

// The undecided vertices with their first labels, and the size of their rows.
__global__ void __launch_bounds__(L_THREADS)
k_label_list(uint32_t n, uint32_t const* __restrict__ und, uint64_t const* __restrict__ fh, uint64_t const* __restrict__ bh, uint32_t* __restrict__ label, uint32_t* __restrict__ stamp, seed_map sm,
             uint32_t* __restrict__ list, ls_counts* lc)
{
  unsigned const lane  = threadIdx.x & 31u;
  uint32_t const words = (n + 31) / 32, span = (words + 31) & ~31u;
  for (uint32_t w = blockIdx.x * L_THREADS + threadIdx.x; w < span; w += gridDim.x * L_THREADS) {
    uint32_t x = w < words ? und[w] : 0u;
    if (w == words - 1 && (n & 31)) x &= (1u << (n & 31)) - 1u;
    uint32_t const c    = __popc(x);
    uint32_t       incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= static_cast<unsigned>(d)) incl += y;
    }
    uint32_t const tot = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (!tot) continue; // warp-uniform
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&lc->list_n, tot);
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + incl - c;
    unsigned long long entries = 0;
    uint32_t           longest = 0;
    for (; x; x &= x - 1) {
      uint32_t const v = w * 32 + __ffs(x) - 1;
      uint64_t const o = fh[v + 1] - fh[v], i = bh[v + 1] - bh[v];
      list[at++]       = v;
      label[v]         = sm.map(v);
      stamp[v]         = 0;
      entries += o + i;
      longest = max(longest, static_cast<uint32_t>(min(max(o, i), static_cast<uint64_t>(UNDECIDED))));
    }
    if (entries) atomicAdd(&lc->entries, entries), atomicMax(&lc->longest, longest);
  }
}

// hit(u, w) for every neighbour w of list[0, cnt)'s rows; the accepted ones
// are appended to out.  A warp takes 32 listed vertices; its lanes share the
// entries of their rows.
template<class F>
__device__ __forceinline__ void
ls_expand(uint32_t const* list, uint32_t cnt, uint64_t const* __restrict__ head, uint32_t const* __restrict__ adj, uint32_t* out, uint32_t* counter, unsigned long long& edges, F&& hit)
{
  unsigned const lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  for (uint32_t i0 = threadIdx.x & ~31u; i0 < cnt; i0 += LS_THREADS) {
    bool const     ok   = i0 + lane < cnt;
    uint32_t const u    = ok ? __ldcg(list + i0 + lane) : 0u;
    uint64_t const b    = ok ? head[u] : 0ull;
    uint32_t const len  = ok ? static_cast<uint32_t>(head[u + 1] - b) : 0u;
    uint32_t       incl = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= static_cast<unsigned>(d)) incl += y;
    }
    uint32_t const tot = __shfl_sync(0xFFFFFFFFu, incl, 31), excl = incl - len;
    edges += len;
    for (uint32_t e0 = 0; e0 < tot; e0 += 32) {
      uint32_t const e = e0 + lane;
      uint32_t       j = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, excl, j + step) <= e) j += step;
      uint64_t const bj = __shfl_sync(0xFFFFFFFFu, b, j);
      uint32_t const xj = __shfl_sync(0xFFFFFFFFu, excl, j), uj = __shfl_sync(0xFFFFFFFFu, u, j);
      uint32_t const w  = e < tot ? adj[bj + (e - xj)] : 0u;
      bool const     f  = e < tot && hit(uj, w);
      unsigned const m  = __ballot_sync(0xFFFFFFFFu, f);
      if (!m) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(counter, static_cast<uint32_t>(__popc(m)));
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
      if (f) __stcg(out + at + __popc(m & lt), w);
    }
  }
}

__global__ void __launch_bounds__(LS_THREADS)
k_label_small(uint64_t const* __restrict__ fh, uint32_t const* __restrict__ fc, uint64_t const* __restrict__ bh, uint32_t const* __restrict__ bc, uint32_t* und, uint32_t* label, uint32_t* stamp,
              uint32_t* __restrict__ scc_id, seed_map sm, uint32_t const* list, uint32_t* q0, uint32_t* q1, uint32_t cap, ls_counts* lc)
{
  __shared__ uint32_t           s_n[3]; // append counters by level: used, next, being cleared
  __shared__ unsigned long long s_edges;
  uint32_t const k = lc->list_n;
  if (k > LS_VERTICES || lc->entries > LS_EDGES || lc->longest > LS_ROW) return;
  if (threadIdx.x < 3) s_n[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_edges = 0;
  __syncthreads();
  unsigned long long edges = 0;
  uint32_t           level = 0, err = 0;
  uint32_t*          q[2]  = { q0, q1 };
  // ends a level: its appended count (one barrier; see the counters)
  auto const close = [&]() {
    __syncthreads();
    uint32_t const c = s_n[level % 3];
    if (threadIdx.x == 0) s_n[(level + 2) % 3] = 0;
    ++level;
    return c;
  };
  // forward: the min-label fixpoint
  uint32_t const* cur = list;
  for (uint32_t cnt = k; cnt;) {
    if (level >= cap) {
      err = 1;
      break;
    }
    uint32_t* const nxt = q[level & 1];
    ls_expand(cur, cnt, fh, fc, nxt, &s_n[level % 3], edges, [&](uint32_t u, uint32_t v) {
      if (!((__ldcg(und + (v >> 5)) >> (v & 31)) & 1u)) return false;
      uint32_t const lu = __ldcg(label + u);
      if (lu >= __ldcg(label + v) || lu >= atomicMin(label + v, lu)) return false;
      return atomicExch(stamp + v, level + 1) != level + 1; // once per level
    });
    cnt = close();
    cur = nxt;
  }
  // roots, then the backward closure inside each label class
  uint32_t decided = 0, base = level;
  if (!err) {
    uint32_t* const nxt = q[level & 1];
    for (uint32_t i0 = threadIdx.x & ~31u; i0 < k; i0 += LS_THREADS) {
      unsigned const lane = threadIdx.x & 31u;
      uint32_t const v    = i0 + lane < k ? __ldcg(list + i0 + lane) : UNDECIDED;
      bool const     root = v != UNDECIDED && __ldcg(label + v) == sm.map(v);
      if (root) {
        bit_take(und, v);
        scc_id[v] = v;
      }
      unsigned const m  = __ballot_sync(0xFFFFFFFFu, root);
      uint32_t       at = 0;
      if (lane == 0 && m) at = atomicAdd(&s_n[level % 3], static_cast<uint32_t>(__popc(m)));
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
      if (root) __stcg(nxt + at + __popc(m & ((1u << lane) - 1u)), v);
    }
    uint32_t cnt = close();
    decided      = cnt;
    cur          = nxt;
    base         = level;
    while (cnt) {
      if (level - base >= cap) {
        err = 2;
        break;
      }
      uint32_t* const to = q[level & 1];
      ls_expand(cur, cnt, bh, bc, to, &s_n[level % 3], edges, [&](uint32_t u, uint32_t v) {
        if (!((__ldcg(und + (v >> 5)) >> (v & 31)) & 1u)) return false;
        uint32_t const lu = __ldcg(label + u);
        if (__ldcg(label + v) != lu || !bit_take(und, v)) return false;
        scc_id[v] = sm.unmap(lu);
        return true;
      });
      cnt = close();
      decided += cnt;
      cur = to;
    }
  }
  if (edges) atomicAdd(&s_edges, edges);
  __syncthreads();
  if (threadIdx.x == 0) lc->ran = 1, lc->err = err, lc->decided = decided, lc->edges = s_edges;
}

} // namespace

uint32_t
label_search(kspn_context* ctx, dgraph const& g, uint32_t* und, uint32_t* scc_id, int rotation, kspn_options const& opt, kspn_stats* st, uint64_t undecided)
{
  auto&          ws    = ctx->ws;
  size_t const   words = (static_cast<size_t>(g.n) + 31) / 32;
  uint32_t*      q[2]  = { ws.q0, ws.q1 };
  uint32_t*      qc[2] = { ws.ctr + CTR_Q0, ws.ctr + CTR_Q1 };
  uint32_t*      claim[2] = { ws.vis_a, ws.vis_b };
  auto*          edges = reinterpret_cast<unsigned long long*>(ws.ctr64);
  uint32_t const cap   = opt.max_label_iters ? opt.max_label_iters : g.n + 2;

  seed_map sm{ nullptr, rotation, 0, 0 };
  if (opt.learned_seeds && ctx->pivot_model && g.n > 0 && g.n <= (1u << 31)) {
    // the learned order: every undecided vertex scored once per call
    uint32_t const shift = std::max<uint32_t>(1u, static_cast<uint32_t>(32 - __builtin_clz(g.n - 1 | 1u)));
    auto* const    bk    = static_cast<uint32_t*>(context_buffer(ctx, BUF_SEEDS, static_cast<size_t>(g.n) * 4));
    k_seed_buckets<<<l_grid(g.n / 8 + 1), L_THREADS, 0, ctx->stream>>>(g.n, und, g.fh, g.fc, g.bh, g.bc, ctx->pivot_model, 1u << (32 - shift), bk);
    KSPN_CHECK_LAUNCH();
    ctx->launches += 1;
    sm = seed_map{ bk, rotation, shift, (static_cast<uint32_t>(rotation) * 0x9E3779B9u) & ((1u << shift) - 1u) };
  }
  if (undecided <= LS_VERTICES && !ctx->prof) {
    // few vertices: one block, unless their rows are too many or too long
    auto* const lc = reinterpret_cast<ls_counts*>(ws.links);
    ls_counts   h{};
    KSPN_CUDA(cudaMemsetAsync(lc, 0, sizeof(ls_counts), ctx->stream));
    k_label_list<<<l_grid((g.n + 31) / 32), L_THREADS, 0, ctx->stream>>>(g.n, und, g.fh, g.bh, ws.label, ws.indeg, sm, ws.q2, lc);
    k_label_small<<<1, LS_THREADS, 0, ctx->stream>>>(g.fh, g.fc, g.bh, g.bc, und, ws.label, ws.indeg, scc_id, sm, ws.q2, ws.q0, ws.q1, cap, lc);
    KSPN_CHECK_LAUNCH();
    ctx->launches += 2;
    KSPN_CUDA(cudaMemcpyAsync(&h, lc, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    KSPN_CUDA(cudaStreamSynchronize(ctx->stream));
    if (h.ran) {
      if (h.err == 1) throw error{ KSPN_ERR_TIMEOUT, "label search: propagation cap exceeded" };
      if (h.err == 2) throw error{ KSPN_ERR_TIMEOUT, "label search: closure cap exceeded" };
      ctx->td_edges += h.edges;
      if (st) st->label_calls += 1;
      return h.decided;
    }
  }
  zero_counters(ctx);
  KSPN_CUDA(cudaMemsetAsync(ws.vis_a, 0, words * 4, ctx->stream));
  KSPN_CUDA(cudaMemsetAsync(ws.vis_b, 0, words * 4, ctx->stream));
  k_label_init<<<l_grid(g.n), L_THREADS, 0, ctx->stream>>>(g.n, und, ws.label, sm, q[0], qc[0]);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 1;

  // forward: min-label fixpoint
  read_counters(ctx);
  uint32_t qn_cur = ctx->h_ctr[CTR_Q0];
  uint64_t e0     = ctx->h_ctr64[0];
  int      cur    = 0;
  for (uint32_t level = 0;; ++level) {
    if (level >= cap) throw error{ KSPN_ERR_TIMEOUT, "label search: propagation cap exceeded" };
    int const nxt = cur ^ 1;
    KSPN_CUDA(cudaMemsetAsync(qc[nxt], 0, sizeof(uint32_t), ctx->stream));
    if (level > 0) {
      k_unclaim<<<l_grid(g.n), L_THREADS, 0, ctx->stream>>>(q[cur], qc[cur], claim[cur]);
      ctx->launches += 1;
    }
    expand_level(ctx, g.fh, g.fc, q[cur], qc[cur], ws.ctr + CTR_NTILES, edges, ws.tile_start, q[nxt], qc[nxt], label_fw_op{ und, ws.label, claim[nxt] });
    read_counters(ctx);
    uint32_t const qn = ctx->h_ctr[CTR_Q0 + nxt];
    prof_add(ctx, 0, KSPN_KERNEL_EXPAND, expand_bytes(qn_cur, ctx->h_ctr64[0] - e0, qn, 4)); // + label[u] read per row
    e0     = ctx->h_ctr64[0];
    qn_cur = qn;
    if (qn == 0) break;
    cur = nxt;
  }

  // roots, then the backward closure inside each label class
  KSPN_CUDA(cudaMemsetAsync(ws.ctr + CTR_Q0, 0, 2 * sizeof(uint32_t), ctx->stream));
  KSPN_CUDA(cudaMemsetAsync(ws.ctr + CTR_DECIDED, 0, sizeof(uint32_t), ctx->stream));
  k_label_roots<<<l_grid(g.n), L_THREADS, 0, ctx->stream>>>(g.n, und, ws.label, scc_id, sm, q[0], qc[0], ws.ctr + CTR_DECIDED);
  KSPN_CHECK_LAUNCH();
  ctx->launches += 1;
  read_counters(ctx);
  uint32_t decided = ctx->h_ctr[CTR_DECIDED];
  cur              = 0;
  for (uint32_t level = 0; ctx->h_ctr[CTR_Q0 + cur] > 0; ++level) {
    if (level >= cap) throw error{ KSPN_ERR_TIMEOUT, "label search: closure cap exceeded" };
    int const nxt = cur ^ 1;
    KSPN_CUDA(cudaMemsetAsync(qc[nxt], 0, sizeof(uint32_t), ctx->stream));
    uint32_t const fq = ctx->h_ctr[CTR_Q0 + cur];
    uint64_t const eb = ctx->h_ctr64[0];
    expand_level(ctx, g.bh, g.bc, q[cur], qc[cur], ws.ctr + CTR_NTILES, edges, ws.tile_start, q[nxt], qc[nxt], label_bw_op{ und, ws.label, scc_id, sm });
    read_counters(ctx);
    uint32_t const pushed = ctx->h_ctr[CTR_Q0 + nxt];
    decided += pushed;
    prof_add(ctx, 0, KSPN_KERNEL_EXPAND, expand_bytes(fq, ctx->h_ctr64[0] - eb, pushed, 4));
    cur = nxt;
  }
  if (st) st->label_calls += 1;
  return decided;
}

} // namespace kspn
