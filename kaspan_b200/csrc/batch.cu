// Batched path: thousands of independent small graphs of uneven size in one
// captured launch sequence (no reference counterpart: the reference
// decomposes one graph per call; each graph here gets the same partition
// its `scc` would, named by the smallest member).
//
// Layout (kspn_scc_batched): graph g owns vertices [vtx_off[g],
// vtx_off[g+1]) of one concatenated CSR and CSC whose heads hold global edge
// positions (head[vtx_off[g]] = edge_off[g]) and whose rows hold LOCAL ids
// (0 .. n_g - 1); scc_id[vtx_off[g] + v] = the local id of the smallest
// member of v's SCC.
//
// Plan (device, captured): per graph its size class -- a graph of at most
// BT_WARP_N vertices and RS_MAXE edges is "small" -- and its bitmap word
// offset (each graph owns whole bitmap words); the large graphs sorted by
// n + m, largest first (a work queue in that order balances the tail).
// Solve (kernels on parallel branches of the same CUDA graph, so they
// overlap):
//  * k_batch_small: one warp per small graph builds its CSR in shared
//    memory and runs the explicit-stack Tarjan of tarjan_smem.cuh;
//  * k_batch_block: one block per larger graph, its vertex bitmaps in shared
//    memory (up to 2^18 vertices, two block sizes): init (degrees, in/out = 0
//    decided), then rounds of {trim-1 push levels, FW-BW from the largest
//    in*out (SCC named by its smallest member), live degrees recounted} until
//    the remainder has at most `rem_tarjan` vertices (64 before the first
//    FW-BW) -- then Tarjan in shared memory -- or the round cap is reached --
//    then one thread's Tarjan in global memory;
//  * k_batch_group: the same rounds with bitmaps in global memory, for larger
//    graphs, the joint searches (option search = 1) and thread-block clusters
//    (up to 8 blocks, distributed shared memory, the cluster barrier) for
//    graphs of n + m >= cluster_min (option cluster_size > 1).
// Every loop is bounded; a round / level cap sets the error word.
#include "kspn_internal.cuh"
#include "prim.cuh"
#include "tarjan_smem.cuh"

#include <cooperative_groups.h>
#include <cstring>

namespace cg = cooperative_groups;

namespace kspn {

namespace {

constexpr int      BT_THREADS = 512;
constexpr int      BS_WARPS   = 4; // warps per block of k_batch_small
constexpr uint32_t BT_NONE    = 0xFFFFFFFFu;

struct bt_args
{
  uint32_t        G;
  uint64_t const* vtx_off;  // G + 1
  uint64_t const* word_off; // G + 1: bitmap words of graph g start at word_off[g]
  uint64_t const* fh;
  uint32_t const* fc;
  uint64_t const* bh;
  uint32_t const* bc;
  uint32_t*       scc_id;
  uint32_t*       und; // bitmaps, word_off-indexed
  uint32_t*       vis_a;
  uint32_t*       vis_b;
  uint32_t*       indeg; // N each, vtx_off-indexed
  uint32_t*       outdeg;
  uint32_t*       q0;
  uint32_t*       q1;
  uint32_t*       q2;
  uint64_t*       pos;   // N: serial Tarjan's edge cursors
  uint32_t const* order; // graphs sorted by class (bt_class), largest first inside a class
  uint32_t*       ctr;   // [4] err, [5] FW-BW rounds, [6] shared-memory Tarjans, [7] serial Tarjans, [8] trim levels,
                         // [BT_COUNT + c] graphs of class c, [BT_CLAIM + c] of them claimed
  uint32_t        max_rounds; // FW-BW rounds per graph before the serial Tarjan
  uint32_t        rem_tarjan; // remainder size that goes to the shared-memory Tarjan (<= RS_MAXV)
  uint32_t        joint;      // FW and BW searches at the same time (bt_reach_joint)
};

constexpr uint32_t BT_WARP_N = 32; // vertices up to which a warp's Tarjan solves a graph (2500 graphs of 2^6 .. 2^9: 0.26 ms; 64: 0.28, 128: 0.32, 512: 0.59)
constexpr uint32_t BT_COUNT = 16, BT_CLAIM = 24;

// How a graph is solved (the work queue's classes, in queue order).
enum bt_class : uint32_t
{
  BT_CLUSTER  = 0, // thread-block cluster, bitmaps in global memory (option cluster_size > 1)
  BT_GLOBAL   = 1, // one block, bitmaps in global memory: too many vertices for shared memory, or joint searches
  BT_BLOCK_L  = 2, // one block, bitmaps in shared memory (k_batch_block)
  BT_BLOCK_M  = 3, // the same, a smaller block
  BT_WARP     = 4, // one warp's Tarjan
  BT_CLASSES  = 5
};

__device__ __forceinline__ uint32_t
bt_first(uint32_t const* ctr, uint32_t cls)
{
  uint32_t first = 0;
  for (uint32_t c = 0; c < cls; ++c) first += __ldcg(ctr + BT_COUNT + c);
  return first;
}

__device__ __forceinline__ bool
bt_get(uint32_t const* bm, uint32_t v)
{
  return (__ldcg(bm + (v >> 5)) >> (v & 31)) & 1u;
}

// ---------------------------------------------------------------- plan
// Per graph: its class as the sort key's top bits, ~(n + m) below them
// (largest first inside a class), and its bitmap word count.
__global__ void
k_bt_classify(uint32_t G, uint64_t const* __restrict__ vtx_off, uint64_t const* __restrict__ fh, uint64_t cluster_min, uint32_t joint, uint32_t l_max, uint32_t m_max, uint32_t* keys, uint32_t* vals,
              uint32_t* words, uint32_t* ctr)
{
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < G; g += gridDim.x * blockDim.x) {
    uint64_t const vo = vtx_off[g], n = vtx_off[g + 1] - vo;
    uint64_t const m  = fh[vo + n] - fh[vo];
    uint64_t const size  = n + m;
    uint32_t const cls   = n <= BT_WARP_N && m <= RS_MAXE ? BT_WARP : (size >= cluster_min ? BT_CLUSTER : (joint || n > l_max || m >= 0xFFFFFFFFull ? BT_GLOBAL : (n > m_max ? BT_BLOCK_L : BT_BLOCK_M)));
    keys[g]  = (cls << 29) | (0x1FFFFFFFu - static_cast<uint32_t>(size < 0x1FFFFFFFull ? size : 0x1FFFFFFFull));
    vals[g]  = g;
    words[g] = static_cast<uint32_t>((n + 31) / 32);
    atomicAdd(ctr + BT_COUNT + cls, 1u);
  }
}

struct f_words
{
  uint32_t const* w;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const { return w[i]; }
};

// ---------------------------------------------------------------- small graphs
__global__ void __launch_bounds__(BS_WARPS * 32)
k_batch_small(bt_args a)
{
  extern __shared__ __align__(16) unsigned char bs_smem[];
  unsigned const lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  rs_piece&      p    = reinterpret_cast<rs_piece*>(bs_smem)[wid];
  uint32_t const nb   = bt_first(a.ctr, BT_WARP), ns = __ldcg(a.ctr + BT_COUNT + BT_WARP);
  for (;;) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(a.ctr + BT_CLAIM + BT_WARP, 1u);
    i = __shfl_sync(0xFFFFFFFFu, i, 0);
    if (i >= ns) break;
    uint32_t const g  = a.order[nb + i];
    uint64_t const vo = a.vtx_off[g];
    uint32_t const n  = static_cast<uint32_t>(a.vtx_off[g + 1] - vo);
    uint64_t const e0 = a.fh[vo];
    // local CSR straight from the rows (ids are local already)
    for (uint32_t v = lane; v <= n; v += 32) p.off[v] = static_cast<uint16_t>(a.fh[vo + v] - e0);
    uint32_t const m = static_cast<uint32_t>(a.fh[vo + n] - e0);
    for (uint32_t e = lane; e < m; e += 32) p.adj[e] = static_cast<uint16_t>(a.fc[e0 + e]);
    for (uint32_t v = lane; v < n; v += 32) p.vid[v] = v;
    __syncwarp();
    if (lane == 0) rs_tarjan(p, n);
    __syncwarp();
    for (uint32_t v = lane; v < n; v += 32) a.scc_id[vo + v] = p.comp[v];
    __syncwarp();
  }
}

// ---------------------------------------------------------------- larger graphs
// A graph goes to a GROUP: one block (medium graphs) or a thread-block
// cluster of up to 8 blocks on different SMs (large graphs).  The group's
// counters live in the shared memory of its rank-0 block and the others
// reach them as distributed shared memory; group barriers are the
// hardware cluster barrier (release / acquire at cluster scope); data other
// blocks of the group write is read through L2.
struct bt_smem
{
  uint32_t           g, rem, cnt, minid, lo, hi, flag, pad;
  uint32_t           lo2, hi2, cnt2, pad2;
  unsigned long long best;
};

struct bt_group
{
  cg::cluster_group cl;
  bt_smem*          S;   // rank 0's counters (local or distributed shared memory)
  uint32_t          gt;  // thread index in the group
  uint32_t          GT;  // threads in the group
  bool              one; // a single block: block barriers suffice
  __device__ __forceinline__ void sync() const
  {
    if (one) __syncthreads();
    else cl.sync();
  }
  __device__ __forceinline__ bool leader() const { return gt == 0; }
};

// warp-aggregated slot from a group counter (lanes that may be inactive)
__device__ __forceinline__ uint32_t
bt_slot(uint32_t* counter)
{
  unsigned const mask = __activemask();
  unsigned const lane = threadIdx.x & 31u, leader = __ffs(mask) - 1;
  uint32_t       base = 0;
  if (lane == leader) base = atomicAdd(counter, static_cast<uint32_t>(__popc(mask)));
  base = __shfl_sync(mask, base, leader);
  return base + __popc(mask & ((1u << lane) - 1u));
}

// fn(u, e) for every edge e of every row of list[lo, hi): a warp takes 32
// listed vertices at a time and its lanes split their edges evenly (a
// warp-wide scan of the row lengths; each lane finds its row by a binary
// search over the lanes' exclusive prefixes), so 32 independent loads are
// in flight per instruction instead of one dependent row walk per thread.
// All lanes of every warp of the group call it; fn is called by the active
// lanes only.
template<class F>
__device__ __forceinline__ void
bt_warp_edges(bt_group const& g, uint32_t const* list, uint32_t lo, uint32_t hi, uint64_t const* head, F&& fn)
{
  unsigned const lane = threadIdx.x & 31u;
  uint32_t const gw = g.gt >> 5, GW = g.GT >> 5;
  for (uint32_t base = lo + gw * 32; base < hi; base += GW * 32) {
    uint32_t const i  = base + lane;
    bool const     ok = i < hi;
    uint32_t const u  = ok ? __ldcg(list + i) : 0u;
    uint64_t const b  = ok ? head[u] : 0;
    uint32_t const d  = ok ? static_cast<uint32_t>(head[u + 1] - b) : 0u;
    uint32_t       incl = d;
#pragma unroll
    for (int sh = 1; sh < 32; sh <<= 1) {
      uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, sh);
      if (lane >= static_cast<unsigned>(sh)) incl += y;
    }
    uint32_t const total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    uint32_t const excl  = incl - d;
    for (uint32_t kb = 0; kb < total; kb += 32) {
      uint32_t const k = kb + lane;
      uint32_t       j = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        uint32_t const ex = __shfl_sync(0xFFFFFFFFu, excl, j + step);
        if (ex <= k) j += step;
      }
      uint64_t const bj = __shfl_sync(0xFFFFFFFFu, b, j);
      uint32_t const xj = __shfl_sync(0xFFFFFFFFu, excl, j);
      uint32_t const uj = __shfl_sync(0xFFFFFFFFu, u, j);
      if (k < total) fn(uj, bj + (k - xj));
    }
  }
}

// Group-leader clock of the phases of the larger graphs (init, trim,
// pivot, searches, remainder): %globaltimer deltas summed over all groups
// into the u64 counters after the u32 ones.
__device__ __forceinline__ uint64_t
bt_now()
{
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void
bt_phase(bt_args const& a, bt_group const& g, int k, uint64_t& t)
{
  if (!g.leader()) return;
  uint64_t const now = bt_now();
  atomicAdd(reinterpret_cast<unsigned long long*>(a.ctr + 32) + k, static_cast<unsigned long long>(now - t));
  t = now;
}

// One graph's view for the group.
struct bt_graph
{
  uint64_t        vo;
  uint32_t        n, words;
  uint64_t const* fh; // rows of local v: fc[fh[v] .. fh[v+1])
  uint64_t const* bh;
  uint32_t*       und;
  uint32_t*       va;
  uint32_t*       vb;
  uint32_t*       indeg;
  uint32_t*       outdeg;
  uint32_t*       ids;
  uint32_t*       q0;
  uint32_t*       q1;
  uint32_t*       q2;
};

// Trim-1 push levels from qin[0, qn): every queued (just decided) vertex
// lowers its undecided out-neighbours' live in-degree and in-neighbours'
// live out-degree; a count reaching 0 decides that neighbour (id = itself)
// and queues it.  Queues alternate between the two buffers that are not
// qin; rows are walked warp-cooperatively (bt_warp_edges).  Returns the
// vertices decided.
__device__ uint32_t
bt_trim(bt_args const& a, bt_graph const& G, bt_group const& g, uint32_t* qin, uint32_t qn)
{
  uint32_t  total = 0;
  uint32_t* bufs[2];
  if (qin == G.q0) bufs[0] = G.q1, bufs[1] = G.q2;
  else if (qin == G.q1) bufs[0] = G.q0, bufs[1] = G.q2;
  else bufs[0] = G.q0, bufs[1] = G.q1;
  uint32_t levels = 0;
  for (uint32_t lvl = 0; qn > 0; ++lvl) {
    if (lvl > G.n + 1) {
      if (g.leader()) atomicExch(a.ctr + 4, 1u);
      break;
    }
    uint32_t* const qout = bufs[lvl & 1];
    if (g.leader()) g.S->cnt = 0;
    g.sync();
    auto const hit = [&](uint32_t w, uint32_t* deg) {
      if (bt_get(G.und, w) && atomicSub(deg + w, 1u) == 1u && bit_take(G.und, w)) {
        G.ids[w]                 = w;
        qout[bt_slot(&g.S->cnt)] = w;
      }
    };
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      uint32_t const* adj = dir ? a.bc : a.fc;
      uint32_t*       deg = dir ? G.outdeg : G.indeg;
      bt_warp_edges(g, qin, 0, qn, dir ? G.bh : G.fh, [&](uint32_t, uint64_t e) { hit(adj[e], deg); });
    }
    g.sync();
    qn = g.S->cnt;
    total += qn;
    qin = qout;
    ++levels;
    g.sync();
  }
  if (g.leader() && levels) atomicAdd(a.ctr + 8, levels);
  return total;
}

// Level-synchronous reach from `root` over head/adj rows, among vertices
// whose bit is set in `cand` (nullptr: among undecided vertices, n_und of
// them), claiming bits of `mark`; every reached vertex is appended to
// `list`.  Returns how many were reached.
// A level whose frontier holds more than 1/BT_BU_DIV of the undecided
// vertices runs bottom-up: every unreached candidate walks its
// opposite-direction row (bu_head / bu_adj) until a neighbour in `mark`
// (reached so far, this level's finds included: reachability does not
// need BFS levels), and joins.
constexpr int      BT_BU_ILP = 2; // candidates a thread walks side by side in a bottom-up level
constexpr uint32_t BT_BU_DIV = 5; // measured on C5: 1/2 23.1 ms, 1/3 19.2, 1/4 17.7, 1/6 17.7, 1/16 19.6, none 23.3

__device__ uint32_t
bt_reach(bt_args const& a, bt_graph const& G, bt_group const& g, uint64_t const* head, uint32_t const* adj, uint64_t const* bu_head, uint32_t const* bu_adj, uint32_t const* cand,
         uint32_t* mark, uint32_t* list, uint32_t root, uint32_t n_und)
{
  if (g.leader()) {
    list[0] = root;
    atomicOr(mark + (root >> 5), 1u << (root & 31));
    g.S->lo  = 0;
    g.S->hi  = 1;
    g.S->cnt = 1;
  }
  g.sync();
  for (uint32_t lvl = 0;; ++lvl) {
    uint32_t const lo = g.S->lo, hi = g.S->hi;
    if (lo == hi) break;
    if (lvl > G.n + 1) {
      if (g.leader()) atomicExch(a.ctr + 4, 1u);
      break;
    }
    if (static_cast<uint64_t>(hi - lo) * BT_BU_DIV > n_und) {
      // a thread walks up to BT_BU_ILP candidates of its word side by side
      // (their offset loads, then their neighbour loads, then their probes
      // in flight together) instead of one dependent row walk at a time
      for (uint32_t wd = g.gt; wd < G.words; wd += g.GT) {
        uint32_t cw = (cand ? __ldcg(cand + wd) : __ldcg(G.und + wd)) & ~__ldcg(mark + wd);
        while (cw) {
          uint32_t v[BT_BU_ILP];
          uint64_t b[BT_BU_ILP], e[BT_BU_ILP];
#pragma unroll
          for (int k = 0; k < BT_BU_ILP; ++k) {
            v[k] = UNDECIDED;
            b[k] = e[k] = 0;
            if (cw) {
              v[k] = wd * 32 + __ffs(cw) - 1;
              cw &= cw - 1;
            }
          }
#pragma unroll
          for (int k = 0; k < BT_BU_ILP; ++k)
            if (v[k] != UNDECIDED) b[k] = bu_head[v[k]], e[k] = bu_head[v[k] + 1];
          for (bool more = true; more;) {
            uint32_t x[BT_BU_ILP];
#pragma unroll
            for (int k = 0; k < BT_BU_ILP; ++k) x[k] = b[k] < e[k] ? bu_adj[b[k]] : 0u;
            more = false;
#pragma unroll
            for (int k = 0; k < BT_BU_ILP; ++k) {
              if (b[k] >= e[k]) continue;
              if (bt_get(mark, x[k])) {
                if (bit_claim(mark, v[k])) list[bt_slot(&g.S->cnt)] = v[k];
                e[k] = b[k]; // done
              } else if (++b[k] < e[k])
                more = true;
            }
          }
        }
      }
    } else
      bt_warp_edges(g, list, lo, hi, head, [&](uint32_t, uint64_t e) {
        uint32_t const w = adj[e];
        if ((cand ? bt_get(cand, w) : bt_get(G.und, w)) && bit_claim(mark, w)) list[bt_slot(&g.S->cnt)] = w;
      });
    g.sync();
    if (g.leader()) g.S->lo = hi, g.S->hi = g.S->cnt;
    g.sync();
  }
  uint32_t const c = g.S->cnt;
  g.sync();
  return c;
}

// FW and BW reach from `root` at the same time, both among the undecided
// vertices (FW over out-rows claiming vis_a into q1, BW over in-rows
// claiming vis_b into q2), one group barrier per joint level: the SCC is
// their intersection.  Half the levels of FW then BW on a graph's
// critical path, for BW also walking vertices outside the FW set.
// Returns (FW count, BW count).
__device__ uint2
bt_reach_joint(bt_args const& a, bt_graph const& G, bt_group const& g, uint32_t root)
{
  if (g.leader()) {
    G.q1[0] = G.q2[0] = root;
    atomicOr(G.va + (root >> 5), 1u << (root & 31));
    atomicOr(G.vb + (root >> 5), 1u << (root & 31));
    g.S->lo = g.S->lo2 = 0;
    g.S->hi = g.S->hi2 = 1;
    g.S->cnt = g.S->cnt2 = 1;
  }
  g.sync();
  for (uint32_t lvl = 0;; ++lvl) {
    uint32_t const lo = g.S->lo, hi = g.S->hi, lo2 = g.S->lo2, hi2 = g.S->hi2;
    if (lo == hi && lo2 == hi2) break;
    if (lvl > G.n + 1) {
      if (g.leader()) atomicExch(a.ctr + 4, 1u);
      break;
    }
    bt_warp_edges(g, G.q1, lo, hi, G.fh, [&](uint32_t, uint64_t e) {
      uint32_t const w = a.fc[e];
      if (bt_get(G.und, w) && bit_claim(G.va, w)) G.q1[bt_slot(&g.S->cnt)] = w;
    });
    bt_warp_edges(g, G.q2, lo2, hi2, G.bh, [&](uint32_t, uint64_t e) {
      uint32_t const w = a.bc[e];
      if (bt_get(G.und, w) && bit_claim(G.vb, w)) G.q2[bt_slot(&g.S->cnt2)] = w;
    });
    g.sync();
    if (g.leader()) g.S->lo = hi, g.S->hi = g.S->cnt, g.S->lo2 = hi2, g.S->hi2 = g.S->cnt2;
    g.sync();
  }
  uint2 const c = make_uint2(g.S->cnt, g.S->cnt2);
  g.sync();
  return c;
}

// argmax over undecided v of live in * out (lowest id on ties), as
// (saturated prod << 32 | ~id); BT_NONE when nothing is undecided
__device__ uint32_t
bt_pivot(bt_graph const& G, bt_group const& g)
{
  if (g.leader()) g.S->best = 0;
  g.sync();
  unsigned long long best = 0;
  for (uint32_t v = g.gt; v < G.n; v += g.GT) {
    if (!bt_get(G.und, v)) continue;
    uint64_t const           p   = static_cast<uint64_t>(__ldcg(G.indeg + v)) * __ldcg(G.outdeg + v);
    unsigned long long const key = (static_cast<unsigned long long>(p < 0xFFFFFFFFull ? p : 0xFFFFFFFFull) << 32) | (0xFFFFFFFFu - v);
    best                         = key > best ? key : best;
  }
#pragma unroll
  for (int sh = 16; sh; sh >>= 1) {
    unsigned long long const o = __shfl_xor_sync(0xFFFFFFFFu, best, sh);
    best                       = o > best ? o : best;
  }
  if ((threadIdx.x & 31) == 0 && best) atomicMax(&g.S->best, best);
  g.sync();
  unsigned long long const b = g.S->best;
  g.sync();
  return b ? 0xFFFFFFFFu - static_cast<uint32_t>(b & 0xFFFFFFFFu) : BT_NONE;
}

// The remaining (undecided) vertices of a graph in id order into the
// piece (rank 0's warp 0), if there are at most RS_MAXV of them with at
// most RS_MAXE edges among them; then Tarjan and the ids.  Returns false
// (and changes nothing) when they do not fit.
__device__ bool
bt_tarjan_smem(bt_args const& a, bt_graph const& G, bt_group const& g, rs_piece& p)
{
  unsigned const lane = threadIdx.x & 31u;
  if (g.gt < 32) {
    uint32_t k = 0;
    for (uint32_t wb = 0; wb < G.words; wb += 32) {
      uint32_t const w    = wb + lane;
      uint32_t       word = w < G.words ? __ldcg(G.und + w) : 0u;
      uint32_t const c    = __popc(word);
      uint32_t       incl = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= static_cast<unsigned>(d)) incl += y;
      }
      uint32_t j = k + incl - c;
      for (; word; word &= word - 1, ++j)
        if (j < RS_MAXV) p.vid[j] = w * 32 + __ffs(word) - 1;
      k += __shfl_sync(0xFFFFFFFFu, incl, 31);
      if (k > RS_MAXV) break;
    }
    __syncwarp();
    bool           fits = k <= RS_MAXV;
    uint32_t const per  = (k + 31) / 32;
    uint32_t       cnt  = 0;
    if (fits)
      for (uint32_t i = lane * per; i < k && i < lane * per + per; ++i) {
        uint32_t const v = p.vid[i];
        uint32_t       c = 0;
        for (uint64_t e = G.fh[v], end = G.fh[v + 1]; e < end; ++e) c += bt_get(G.und, a.fc[e]) ? 1u : 0u;
        p.comp[i] = static_cast<uint16_t>(c < RS_MAXE ? c : RS_MAXE);
        cnt += c;
      }
    uint32_t incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= static_cast<unsigned>(d)) incl += y;
    }
    uint32_t const total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    fits                 = fits && total <= RS_MAXE;
    if (fits) {
      uint32_t run = incl - cnt;
      for (uint32_t i = lane * per; i < k && i < lane * per + per; ++i) {
        p.off[i] = static_cast<uint16_t>(run);
        run += p.comp[i];
      }
      if (lane == 0) p.off[k] = static_cast<uint16_t>(total);
      __syncwarp();
      for (uint32_t i = lane * per; i < k && i < lane * per + per; ++i) {
        uint32_t const v = p.vid[i];
        uint32_t       o = p.off[i];
        for (uint64_t e = G.fh[v], end = G.fh[v + 1]; e < end; ++e) {
          uint32_t const w = a.fc[e];
          if (bt_get(G.und, w)) p.adj[o++] = static_cast<uint16_t>(rs_local(p, k, w));
        }
      }
      __syncwarp();
      if (lane == 0) rs_tarjan(p, k);
      __syncwarp();
      for (uint32_t i = lane; i < k; i += 32) {
        uint32_t const v = p.vid[i];
        G.ids[v]         = p.vid[p.comp[i]];
        atomicAnd(G.und + (v >> 5), ~(1u << (v & 31)));
      }
      if (lane == 0) atomicAdd(a.ctr + 6, 1u);
    }
    if (lane == 0) g.S->flag = fits ? 1u : 0u;
  }
  g.sync();
  bool const ok = g.S->flag != 0;
  g.sync();
  return ok;
}

// One thread's iterative Tarjan (tarjan.hpp:20-136) over the undecided
// sub-graph in global memory: index in indeg, low in outdeg, the SCC stack
// in q0, the call stack's vertices in q1 and edge cursors in pos; on-stack
// flags in vis_a.  The last resort after the round cap; n + m steps.
__device__ void
bt_tarjan_serial(bt_args const& a, bt_graph const& G, bt_group const& g, uint64_t* pos)
{
  g.sync();
  for (uint32_t v = g.gt; v < G.n; v += g.GT) G.indeg[v] = BT_NONE;
  for (uint32_t w = g.gt; w < G.words; w += g.GT) G.va[w] = 0;
  g.sync();
  if (g.leader()) {
    atomicAdd(a.ctr + 7, 1u);
    uint32_t idx = 0, sp = 0, cp = 0;
    for (uint32_t r = 0; r < G.n; ++r) {
      if (!bt_get(G.und, r) || __ldcg(G.indeg + r) != BT_NONE) continue;
      G.indeg[r] = G.outdeg[r] = idx++;
      G.q0[sp++]               = r;
      G.va[r >> 5] |= 1u << (r & 31);
      G.q1[cp]  = r;
      pos[cp++] = G.fh[r];
      while (cp > 0) {
        uint32_t const v = G.q1[cp - 1];
        uint64_t const e = pos[cp - 1];
        if (e < G.fh[v + 1]) {
          pos[cp - 1]      = e + 1;
          uint32_t const w = a.fc[e];
          if (!bt_get(G.und, w)) continue;
          if (G.indeg[w] == BT_NONE) {
            G.indeg[w] = G.outdeg[w] = idx++;
            G.q0[sp++]               = w;
            G.va[w >> 5] |= 1u << (w & 31);
            G.q1[cp]  = w;
            pos[cp++] = G.fh[w];
          } else if (((G.va[w >> 5] >> (w & 31)) & 1u) && G.indeg[w] < G.outdeg[v]) G.outdeg[v] = G.indeg[w];
        } else {
          --cp;
          if (cp > 0) {
            uint32_t const u = G.q1[cp - 1];
            if (G.outdeg[v] < G.outdeg[u]) G.outdeg[u] = G.outdeg[v];
          }
          if (G.outdeg[v] == G.indeg[v]) {
            uint32_t j = sp, mn = v;
            do {
              --j;
              if (G.q0[j] < mn) mn = G.q0[j];
            } while (G.q0[j] != v);
            for (uint32_t t = j; t < sp; ++t) {
              uint32_t const x = G.q0[t];
              G.va[x >> 5] &= ~(1u << (x & 31));
              G.ids[x] = mn;
              G.und[x >> 5] &= ~(1u << (x & 31));
            }
            sp = j;
          }
        }
      }
    }
  }
  g.sync();
}

__device__ void
bt_solve(bt_args const& a, uint32_t gi, bt_group const& g, rs_piece& piece)
{
  bt_graph G;
  G.vo     = a.vtx_off[gi];
  G.n      = static_cast<uint32_t>(a.vtx_off[gi + 1] - G.vo);
  G.words  = (G.n + 31) / 32;
  G.fh     = a.fh + G.vo;
  G.bh     = a.bh + G.vo;
  G.und    = a.und + a.word_off[gi];
  G.va     = a.vis_a + a.word_off[gi];
  G.vb     = a.vis_b + a.word_off[gi];
  G.indeg  = a.indeg + G.vo;
  G.outdeg = a.outdeg + G.vo;
  G.ids    = a.scc_id + G.vo;
  G.q0     = a.q0 + G.vo;
  G.q1     = a.q1 + G.vo;
  G.q2     = a.q2 + G.vo;
  uint64_t* const pos = a.pos + G.vo;

  uint64_t t = g.leader() ? bt_now() : 0;
  // init: all undecided, live degrees = raw degrees, in/out = 0 decided
  for (uint32_t w = g.gt; w < G.words; w += g.GT) {
    uint32_t const tail = G.n - w * 32;
    G.und[w]            = tail >= 32 ? 0xFFFFFFFFu : (1u << tail) - 1u;
    G.va[w] = G.vb[w] = 0;
  }
  if (g.leader()) g.S->cnt = 0;
  g.sync();
  for (uint32_t v = g.gt; v < G.n; v += g.GT) {
    uint32_t const o = static_cast<uint32_t>(G.fh[v + 1] - G.fh[v]);
    uint32_t const i = static_cast<uint32_t>(G.bh[v + 1] - G.bh[v]);
    G.outdeg[v]      = o;
    G.indeg[v]       = i;
    if (o == 0 || i == 0) {
      G.ids[v] = v;
      atomicAnd(G.und + (v >> 5), ~(1u << (v & 31)));
      G.q0[bt_slot(&g.S->cnt)] = v;
    } else G.ids[v] = UNDECIDED;
  }
  g.sync();
  uint32_t  qn   = g.S->cnt;
  uint32_t  rem  = G.n - qn;
  uint32_t* seed = G.q0;
  g.sync();
  bt_phase(a, g, 0, t);
  for (uint32_t round = 0;; ++round) {
    rem -= bt_trim(a, G, g, seed, qn);
    bt_phase(a, g, 1, t);
    if (rem == 0) break;
    if (rem <= a.rem_tarjan && bt_tarjan_smem(a, G, g, piece)) {
      bt_phase(a, g, 4, t);
      break;
    }
    if (round >= a.max_rounds) {
      bt_tarjan_serial(a, G, g, pos);
      bt_phase(a, g, 4, t);
      break;
    }
    // FW-BW from the largest live in * out
    uint32_t const p = bt_pivot(G, g);
    bt_phase(a, g, 2, t);
    if (p == BT_NONE) {
      if (g.leader()) atomicExch(a.ctr + 4, 1u);
      break;
    }
    uint32_t nf, nb;
    uint32_t* scc = G.q2; // the SCC's members
    if (a.joint) {
      uint2 const c = bt_reach_joint(a, G, g, p);
      nf            = c.x;
      // members: BW-reached vertices also FW-reached, compacted into q0
      if (g.leader()) g.S->cnt = 0;
      g.sync();
      for (uint32_t i = g.gt; i < c.y; i += g.GT) {
        uint32_t const v = __ldcg(G.q2 + i);
        if (bt_get(G.va, v)) G.q0[bt_slot(&g.S->cnt)] = v;
        atomicAnd(G.vb + (v >> 5), ~(1u << (v & 31))); // vis_b cleared through its own list
      }
      g.sync();
      nb  = g.S->cnt;
      scc = G.q0;
      g.sync();
    } else {
      nf = bt_reach(a, G, g, G.fh, a.fc, G.bh, a.bc, nullptr, G.va, G.q1, p, rem);
      nb = bt_reach(a, G, g, G.bh, a.bc, G.fh, a.fc, G.va, G.vb, G.q2, p, nf);
    }
    // the SCC: smallest member, ids, und; vis_a cleared through q1
    if (g.leader()) g.S->minid = 0xFFFFFFFFu;
    g.sync();
    uint32_t mn = 0xFFFFFFFFu;
    for (uint32_t i = g.gt; i < nb; i += g.GT) mn = min(mn, __ldcg(scc + i));
    mn = __reduce_min_sync(0xFFFFFFFFu, mn);
    if ((threadIdx.x & 31) == 0 && mn != 0xFFFFFFFFu) atomicMin(&g.S->minid, mn);
    g.sync();
    uint32_t const id = g.S->minid;
    for (uint32_t i = g.gt; i < nb; i += g.GT) {
      uint32_t const v = __ldcg(scc + i);
      G.ids[v]         = id;
      atomicAnd(G.und + (v >> 5), ~(1u << (v & 31)));
      atomicAnd(G.vb + (v >> 5), ~(1u << (v & 31)));
    }
    for (uint32_t i = g.gt; i < nf; i += g.GT) {
      uint32_t const v = __ldcg(G.q1 + i);
      atomicAnd(G.va + (v >> 5), ~(1u << (v & 31)));
    }
    if (g.leader()) atomicAdd(a.ctr + 5, 1u);
    g.sync();
    bt_phase(a, g, 3, t);
    rem -= nb;
    if (rem == 0) break;
    // the SCC's members seed the next trim
    seed = scc;
    qn   = nb;
  }
  g.sync();
}

// ---------------------------------------------------------------- graphs whose bitmaps fit shared memory
// One block per graph, its three vertex bitmaps (undecided, FW-reached,
// BW-reached) in shared memory: a probe or a claim costs a shared-memory
// access instead of a trip to L2, and a level needs one block barrier (its
// append counter rotates over three slots, so no thread waits for a reset).
// What then bounds it is DRAM: a few hundred graphs in flight overflow L2,
// and a row read at random costs a 128-byte line per access.  So the wide passes
// (bottom-up levels, the recount after an SCC) go through the vertices in id
// order, 32 lanes on neighbouring vertices; live degrees take one byte per
// direction (graphs with a row of BB_DEG8 or more entries: 32 bits); and
// after an SCC larger than the rest the rest is recounted instead of every
// SCC member's rows being walked.
// Every id is its vertex's own from the start (trimmed vertices keep it);
// only SCC members are written again, from the bitmap.
// Two sizes: BB_L (up to BB_L_WORDS bitmap words: 2^18 vertices, 96 KB, one
// block of BB_L_THREADS per SM) and BB_M (2^15 vertices, four blocks of
// BB_M_THREADS).  With at most two graphs per SM every graph above BB_M_FEW
// vertices gets the larger block: no other graph waits for the threads, and
// the slowest graph is the call's time (120 graphs of 2^8 .. 2^16 vertices:
// 0.69 -> 0.50 ms, 30 of 2^10 .. 2^13: 0.35 -> 0.32).
// Measured on the 4096-graph mix (157 M vertices, 533 M edges): 17.1 ms with
// bitmaps in global memory (k_batch_group), 14.3 with 1536 threads of 40
// registers per SM (spills), 10.8 with two BB_L blocks of 512 threads, 8.5
// with one of 1024 (half the graphs in flight leave each twice the L1 and
// L2; 296 graphs of 2^17 and 2^18 vertices: 6.7 -> 4.3, 120 of 2^18: 6.7 ->
// 2.9).  The line between the two at 2^16, 2^15, 2^14, 2^13: 8.50, 8.53,
// 8.77, 9.00; 2000 graphs of 2^10 .. 2^15: 1.45, 1.46, 1.58, 1.76; 16 graphs
// of 2^16: 1.37 at the first, 0.82 otherwise; BB_M of 512 threads: 8.86.
// Not kept: prefetching a find's offsets into L2 (+10%), walking the SCC
// members' rows instead of the recount (+3%), 4 neighbours at once (+1%), 1
// or 4 vertices per round (+12%, +2%).
constexpr int      BB_ILP       = 2; // neighbours of a row a lane reads at once
constexpr int      BB_CAND      = 2; // vertices a lane takes per round of a pass in id order
constexpr int      BB_L_THREADS = 1024, BB_M_THREADS = 256;
constexpr int      BB_L_BLOCKS = 1, BB_M_BLOCKS = 4; // per SM: 1024 threads of 64 registers either way
constexpr uint32_t BB_L_WORDS = 8192, BB_M_WORDS = 1024;
constexpr uint32_t BB_LONG   = 32; // neighbours a lane walks alone; longer rows go to the whole warp
constexpr uint32_t BB_BU_DIV = 10; // bottom-up when the frontier holds more than 1/10 of the candidates (4096 graphs: 8.46 ms, 1/16 the same, 1/8 8.59, 1/5 9.02; 200 graphs: 1.82, 1/16 1.96)
constexpr uint32_t BB_M_FEW = 512;
// A remainder goes to one lane's Tarjan (0.25 us per vertex and edge) from
// rem_tarjan on, but not a whole graph before its first FW-BW round: that
// leaves little in most.  30 graphs of 2^6 .. 2^9 vertices: 0.48 -> 0.13 ms,
// 2000 of 2^8 .. 2^11: 0.70 -> 0.37 (limit 32, 128: the same within 5%).
constexpr uint32_t BB_TARJAN_0 = 64;
constexpr uint32_t BB_DEG8   = 255;

constexpr uint32_t BB_ROUND = 32 * BB_CAND;    // vertices a warp takes per round
constexpr uint32_t BB_PACK  = BB_ROUND + 256;  // packed vertices a warp buffers

struct bb_smem
{
  uint32_t           claim;
  uint32_t           cnt[3]; // append counters by level
  uint32_t           minid, flag;
  unsigned long long best;
};

// A block's view of its graph.
struct bb_block
{
  uint32_t  n, words;
  bb_smem*  S;
  uint32_t* und; // shared memory
  uint32_t* va;
  uint32_t* vb;
  uint16_t* pack;  // this warp's buffer
  uint32_t  level; // levels run by the block: picks the append counter
};

// One direction's rows.  A graph of this path has fewer than 2^32 edges, so
// a row's place within the graph is the difference of the offsets' low
// words: half the registers of the 64-bit offsets.
struct bb_rows
{
  uint32_t const* low; // low word of vertex v's offset at low[2 v]
  uint32_t const* adj; // the graph's first entry
  uint32_t        e0;  // low word of its offset
  __device__ __forceinline__ uint32_t begin(uint32_t v) const { return __ldg(low + 2 * v) - e0; }
  __device__ __forceinline__ uint32_t length(uint32_t v, uint32_t b) const { return __ldg(low + 2 * v + 2) - e0 - b; }
  __device__ __forceinline__ uint32_t at(uint32_t e) const { return __ldg(adj + e); }
};
__device__ __forceinline__ bb_rows
bb_rows_of(uint64_t const* head, uint32_t const* adj)
{
  uint64_t const e0 = head[0];
  return bb_rows{ reinterpret_cast<uint32_t const*>(head), adj + e0, static_cast<uint32_t>(e0) };
}

// Live degrees: a byte per direction (vertex v: byte 2 v in-degree, 2 v + 1
// out-degree of deg8), or 32 bits each when the graph has a row of BB_DEG8
// or more entries.
struct bb_degrees
{
  uint32_t* deg8;
  uint32_t* in;
  uint32_t* out;
  bool      wide;
  __device__ __forceinline__ void set(uint32_t v, uint32_t i, uint32_t o) const
  {
    if (wide) in[v] = i, out[v] = o;
    else reinterpret_cast<uint16_t*>(deg8)[v] = static_cast<uint16_t>(i | o << 8);
  }
  // one fewer in direction dir (0: in, 1: out); the count before
  __device__ __forceinline__ uint32_t drop(uint32_t v, int dir) const
  {
    if (wide) return atomicSub((dir ? out : in) + v, 1u);
    uint32_t const sh = (v & 1u) * 16 + (dir ? 8 : 0);
    return (atomicSub(deg8 + (v >> 1), 1u << sh) >> sh) & 255u; // a live count is at least 1: no borrow
  }
  __device__ __forceinline__ uint2 get(uint32_t v) const
  {
    if (wide) return make_uint2(__ldcg(in + v), __ldcg(out + v));
    uint32_t const x = __ldcg(deg8 + (v >> 1)) >> ((v & 1u) * 16);
    return make_uint2(x & 255u, (x >> 8) & 255u);
  }
};

__device__ __forceinline__ bool
bb_bit(uint32_t const* bm, uint32_t v)
{
  return (bm[v >> 5] >> (v & 31)) & 1u;
}

__device__ __forceinline__ uint32_t
bb_warp_scan(uint32_t x) // inclusive
{
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if ((threadIdx.x & 31u) >= static_cast<unsigned>(d)) x += y;
  }
  return x;
}

// Appends the lanes' finds (bit k of `found`: vertex v[k]) to list[base..):
// one counter update per warp.  All lanes call it.
template<int N>
__device__ __forceinline__ void
bb_append(uint32_t found, uint32_t const (&v)[N], uint32_t* list, uint32_t base, uint32_t* counter)
{
  unsigned const lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  unsigned       bal[N];
  uint32_t       tot = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) bal[k] = __ballot_sync(0xFFFFFFFFu, (found >> k) & 1u), tot += __popc(bal[k]);
  if (!tot) return;
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(counter, tot);
  at = base + __shfl_sync(0xFFFFFFFFu, at, 0);
#pragma unroll
  for (int k = 0; k < N; ++k) {
    if ((found >> k) & 1u) list[at + __popc(bal[k] & lt)] = v[k];
    at += __popc(bal[k]);
  }
}

// round(v) for the set bits of word(w), w in [0, B.words), BB_ROUND vertices
// per call and warp (v[k] = UNDECIDED past the end): a warp takes groups of
// up to 8 neighbouring words in turn, packs their vertices in its buffer
// and hands out neighbouring ones to neighbouring lanes.  All lanes of every
// warp call it.
template<int T, class W, class F>
__device__ __forceinline__ void
bb_in_order(bb_block const& B, W&& word, F&& round)
{
  constexpr uint32_t NW   = T / 32;
  unsigned const     lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t           gw   = 8; // words per group: fewer on a graph that would leave warps idle
  while (gw > 1 && B.words < gw * NW) gw /= 2;
  uint32_t const bits = (1u << gw) - 1u; // a lane packs gw bits of a group
  uint32_t const lw = lane * gw / 32, ls = lane * gw % 32;
  uint32_t       held = 0;
  auto const     take = [&](uint32_t from, uint32_t cnt) {
    uint32_t v[BB_CAND];
#pragma unroll
    for (int k = 0; k < BB_CAND; ++k) {
      uint32_t const j = k * 32 + lane;
      uint32_t const e = j < cnt ? B.pack[from + j] : 0u;
      v[k]             = j < cnt ? (warp + (e >> 8) * NW) * gw * 32 + (e & 255u) : UNDECIDED;
    }
    __syncwarp();
    round(v);
  };
  for (uint32_t it = 0, w0 = warp * gw; w0 < B.words; ++it, w0 += NW * gw) {
    uint32_t       x    = w0 + lw < B.words ? (word(w0 + lw) >> ls) & bits : 0u;
    uint32_t const c    = __popc(x);
    uint32_t const incl = bb_warp_scan(c), tot = __shfl_sync(0xFFFFFFFFu, incl, 31);
    for (uint32_t at = held + incl - c; x; x &= x - 1) B.pack[at++] = static_cast<uint16_t>(it << 8 | (lane * gw + __ffs(x) - 1));
    __syncwarp();
    for (held += tot; held >= BB_ROUND;) {
      held -= BB_ROUND;
      take(held, BB_ROUND);
    }
  }
  if (held) take(0, held);
}

// hit(w) for the neighbours w of list[lo, hi)'s rows in each of D directions
// (w[d * BB_ILP + k]: direction d; UNDECIDED: none); the vertices it accepts
// are appended to out[base..).  A warp takes 32 listed vertices and its lanes
// share their rows' entries, BB_ILP per direction and step (a scan of the
// lengths; each lane finds its entries' rows by a binary search over the
// lanes' prefixes): sparse rows take one step, however uneven they are, and
// both directions' loads are in flight together.  Rows longer than BB_LONG
// are walked one by one.
template<int T, int D, class F>
__device__ __forceinline__ void
bb_expand(uint32_t const* list, uint32_t lo, uint32_t hi, bb_rows const (&r)[D], uint32_t* out, uint32_t base, uint32_t* counter, F&& hit)
{
  unsigned const lane = threadIdx.x & 31u;
  for (uint32_t i0 = lo + (threadIdx.x & ~31u); i0 < hi; i0 += T) {
    bool const     ok = i0 + lane < hi;
    uint32_t const u  = ok ? list[i0 + lane] : 0u;
    uint32_t       b[D], len[D], excl[D], tot[D];
#pragma unroll
    for (int d = 0; d < D; ++d) b[d] = ok ? r[d].begin(u) : 0u, len[d] = ok ? r[d].length(u, b[d]) : 0u;
    uint32_t most = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      uint32_t const own  = len[d] > BB_LONG ? 0u : len[d];
      uint32_t const incl = bb_warp_scan(own);
      tot[d]  = __shfl_sync(0xFFFFFFFFu, incl, 31);
      excl[d] = incl - own;
      most    = max(most, tot[d]);
    }
    for (uint32_t e0 = 0; e0 < most; e0 += 32 * BB_ILP) {
      uint32_t w[D * BB_ILP];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        uint32_t j[BB_ILP];
#pragma unroll
        for (int k = 0; k < BB_ILP; ++k) j[k] = 0;
#pragma unroll
        for (int step = 16; step; step >>= 1)
#pragma unroll
          for (int k = 0; k < BB_ILP; ++k)
            if (__shfl_sync(0xFFFFFFFFu, excl[d], j[k] + step) <= e0 + k * 32 + lane) j[k] += step;
#pragma unroll
        for (int k = 0; k < BB_ILP; ++k) {
          uint32_t const e  = e0 + k * 32 + lane;
          uint32_t const p  = __shfl_sync(0xFFFFFFFFu, b[d], j[k]) + e - __shfl_sync(0xFFFFFFFFu, excl[d], j[k]);
          w[d * BB_ILP + k] = e < tot[d] ? r[d].at(p) : UNDECIDED;
        }
      }
      bb_append(hit(w), w, out, base, counter);
    }
#pragma unroll
    for (int d = 0; d < D; ++d)
      for (unsigned todo = __ballot_sync(0xFFFFFFFFu, len[d] > BB_LONG); todo; todo &= todo - 1) {
        unsigned const l  = __ffs(todo) - 1;
        uint32_t const b0 = __shfl_sync(0xFFFFFFFFu, b[d], l);
        uint32_t const n0 = __shfl_sync(0xFFFFFFFFu, len[d], l);
#pragma unroll 1
        for (uint32_t x = 0; x < n0; x += 32 * BB_ILP) {
          uint32_t w[D * BB_ILP];
#pragma unroll
          for (int k = 0; k < D * BB_ILP; ++k) {
            uint32_t const y = x + (k % BB_ILP) * 32 + lane;
            w[k]             = k / BB_ILP == d && y < n0 ? r[d].at(b0 + y) : UNDECIDED;
          }
          bb_append(hit(w), w, out, base, counter);
        }
      }
  }
}

// End of a level: the vertices it appended.  One barrier; the counter of the
// level after next is cleared (no thread reads or adds to it before the next
// barrier).
__device__ __forceinline__ uint32_t
bb_level_end(bb_block& B)
{
  __syncthreads();
  uint32_t const c = B.S->cnt[B.level % 3];
  if (threadIdx.x == 0) B.S->cnt[(B.level + 2) % 3] = 0;
  ++B.level;
  return c;
}

// Trim-1 push levels from the decided vertices seed[0, qn): live degrees of
// undecided neighbours fall, the ones that reach 0 are decided and queued in
// q0[at..).  Returns q0's new length.
template<int T>
__device__ __forceinline__ uint32_t
bb_trim(uint32_t* err, bb_block& B, uint32_t* q0, bb_degrees const deg, bb_rows const fw, bb_rows const bw, uint32_t const* seed, uint32_t qn, uint32_t at, uint32_t& levels)
{
  uint32_t        lo = 0, hi = qn;
  uint32_t const* list = seed;
  for (uint32_t lvl = 0; lo < hi; ++lvl) {
    if (lvl > B.n + 1) {
      if (threadIdx.x == 0) atomicExch(err, 1u);
      break;
    }
    uint32_t* const counter = &B.S->cnt[B.level % 3];
    bb_rows const   rows[2] = { fw, bw }; // out-rows lower in-degrees, in-rows out-degrees
    bb_expand<T>(list, lo, hi, rows, q0, at, counter, [&](uint32_t const (&w)[2 * BB_ILP]) {
      uint32_t left[2 * BB_ILP], found = 0;
#pragma unroll
      for (int k = 0; k < 2 * BB_ILP; ++k) left[k] = w[k] != UNDECIDED && bb_bit(B.und, w[k]) ? deg.drop(w[k], k / BB_ILP) : 0u;
#pragma unroll
      for (int k = 0; k < 2 * BB_ILP; ++k)
        if (left[k] == 1u && bit_take(B.und, w[k])) found |= 1u << k;
      return found;
    });
    uint32_t const c = bb_level_end(B);
    list             = q0;
    lo               = at;
    hi               = at + c;
    at += c;
    ++levels;
  }
  return at;
}

// BB_ILP neighbours of each of the lane's vertices, from place x of their
// rows on (UNDECIDED past a row's end): all loads in flight together.
__device__ __forceinline__ void
bb_some(bb_rows const r, uint32_t const (&b)[BB_CAND], uint32_t const (&len)[BB_CAND], uint32_t x, uint32_t (&w)[BB_CAND][BB_ILP])
{
#pragma unroll
  for (int k = 0; k < BB_CAND; ++k)
#pragma unroll
    for (int j = 0; j < BB_ILP; ++j) w[k][j] = x + j < len[k] ? r.at(b[k] + x + j) : UNDECIDED;
}

// Undecided neighbours in the rows of v (UNDECIDED: none) into c[k].  All
// lanes call it.
__device__ __forceinline__ void
bb_count_live(bb_block const& B, bb_rows const r, uint32_t const (&v)[BB_CAND], uint32_t (&c)[BB_CAND])
{
  unsigned const lane = threadIdx.x & 31u;
  uint32_t       b[BB_CAND], len[BB_CAND], own[BB_CAND], most = 0;
#pragma unroll
  for (int k = 0; k < BB_CAND; ++k) {
    b[k]   = v[k] != UNDECIDED ? r.begin(v[k]) : 0u;
    len[k] = v[k] != UNDECIDED ? r.length(v[k], b[k]) : 0u;
    c[k]   = 0;
  }
#pragma unroll
  for (int k = 0; k < BB_CAND; ++k) own[k] = len[k] > BB_LONG ? 0u : len[k], most = max(most, own[k]);
  for (uint32_t x = 0; __any_sync(0xFFFFFFFFu, x < most); x += BB_ILP) {
    uint32_t w[BB_CAND][BB_ILP];
    bb_some(r, b, own, x, w);
#pragma unroll
    for (int k = 0; k < BB_CAND; ++k)
#pragma unroll
      for (int j = 0; j < BB_ILP; ++j) c[k] += w[k][j] != UNDECIDED && bb_bit(B.und, w[k][j]) ? 1u : 0u;
  }
#pragma unroll
  for (int k = 0; k < BB_CAND; ++k)
    for (unsigned todo = __ballot_sync(0xFFFFFFFFu, len[k] > BB_LONG); todo; todo &= todo - 1) {
      unsigned const l  = __ffs(todo) - 1;
      uint32_t const b0 = __shfl_sync(0xFFFFFFFFu, b[k], l), n0 = __shfl_sync(0xFFFFFFFFu, len[k], l);
      uint32_t       s  = 0;
      for (uint32_t x = lane; x < n0; x += 32) s += bb_bit(B.und, r.at(b0 + x)) ? 1u : 0u;
      s = __reduce_add_sync(0xFFFFFFFFu, s);
      if (lane == l) c[k] = s;
    }
}

// The live degrees of every undecided vertex counted anew; the ones without
// a live in- or out-neighbour are decided and queued in q0[at..).  Returns
// how many.  va is clear before and after (it holds the dead between the
// count and the decisions, so that every count sees the same set).
template<int T>
__device__ __forceinline__ uint32_t
bb_recount(bb_block& B, uint32_t* q0, bb_degrees const deg, bb_rows const fw, bb_rows const bw, uint32_t at)
{
  bb_in_order<T>(B, [&](uint32_t w) { return B.und[w]; }, [&](uint32_t const (&v)[BB_CAND]) {
    uint32_t o[BB_CAND], i[BB_CAND];
    bb_count_live(B, fw, v, o);
    bb_count_live(B, bw, v, i);
#pragma unroll
    for (int k = 0; k < BB_CAND; ++k)
      if (v[k] != UNDECIDED) {
        deg.set(v[k], i[k], o[k]);
        if (!i[k] || !o[k]) atomicOr(B.va + (v[k] >> 5), 1u << (v[k] & 31));
      }
  });
  __syncthreads();
  uint32_t* const counter = &B.S->cnt[B.level % 3];
  uint32_t const  span    = (B.words + 31) & ~31u;
  for (uint32_t w = threadIdx.x; w < span; w += T) {
    uint32_t dead = w < B.words ? B.va[w] : 0u;
    if (dead) B.und[w] &= ~dead, B.va[w] = 0;
    uint32_t const c    = __popc(dead);
    uint32_t const incl = bb_warp_scan(c), tot = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (!tot) continue; // warp-uniform
    uint32_t base = 0;
    if ((threadIdx.x & 31u) == 0) base = atomicAdd(counter, tot);
    base = at + __shfl_sync(0xFFFFFFFFu, base, 0) + incl - c;
    for (; dead; dead &= dead - 1) q0[base++] = w * 32 + __ffs(dead) - 1;
  }
  return bb_level_end(B);
}

// Vertices reachable from `root` inside `cand` along the rows td, claimed in
// `mark` and appended to `list`; a level whose frontier holds more than
// 1 / BB_BU_DIV of the n_cand candidates runs bottom-up along the rows bu
// (each unreached candidate walks its row until a reached neighbour, this
// level's finds included).  Returns how many were reached.
template<int T>
__device__ __forceinline__ uint32_t
bb_reach(uint32_t* err, bb_block& B, bb_rows const td, bb_rows const bu, uint32_t const* cand, uint32_t* mark, uint32_t* list, uint32_t root, uint32_t n_cand)
{
  unsigned const lane = threadIdx.x & 31u;
  if (threadIdx.x == 0) {
    list[0] = root;
    mark[root >> 5] |= 1u << (root & 31);
  }
  __syncthreads();
  uint32_t lo = 0, hi = 1;
  for (uint32_t lvl = 0; lo < hi; ++lvl) {
    if (lvl > B.n + 1) {
      if (threadIdx.x == 0) atomicExch(err, 1u);
      break;
    }
    uint32_t* const counter = &B.S->cnt[B.level % 3];
    if (static_cast<uint64_t>(hi - lo) * BB_BU_DIV > n_cand)
      bb_in_order<T>(B, [&](uint32_t w) { return cand[w] & ~mark[w]; }, [&](uint32_t const (&v)[BB_CAND]) {
        uint32_t b[BB_CAND], len[BB_CAND], found = 0, open = 0;
#pragma unroll
        for (int k = 0; k < BB_CAND; ++k) {
          b[k]   = v[k] != UNDECIDED ? bu.begin(v[k]) : 0u;
          len[k] = v[k] != UNDECIDED ? bu.length(v[k], b[k]) : 0u;
          open |= len[k] ? 1u << k : 0u;
        }
        for (uint32_t x = 0; x < BB_LONG && __any_sync(0xFFFFFFFFu, open != 0); x += BB_ILP) {
          uint32_t w[BB_CAND][BB_ILP], own[BB_CAND];
#pragma unroll
          for (int k = 0; k < BB_CAND; ++k) own[k] = (open >> k) & 1u ? len[k] : 0u;
          bb_some(bu, b, own, x, w);
#pragma unroll
          for (int k = 0; k < BB_CAND; ++k) {
            bool h = false;
#pragma unroll
            for (int j = 0; j < BB_ILP; ++j) h |= w[k][j] != UNDECIDED && bb_bit(mark, w[k][j]);
            if (h) found |= 1u << k;
            if (h || x + BB_ILP >= own[k]) open &= ~(1u << k);
          }
        }
        // rows still open: the whole warp, with early exit
#pragma unroll
        for (int k = 0; k < BB_CAND; ++k)
          for (unsigned todo = __ballot_sync(0xFFFFFFFFu, (open >> k) & 1u); todo; todo &= todo - 1) {
            unsigned const l  = __ffs(todo) - 1;
            uint32_t const b0 = __shfl_sync(0xFFFFFFFFu, b[k], l);
            uint32_t const n0 = __shfl_sync(0xFFFFFFFFu, len[k], l);
            bool           h  = false;
            for (uint32_t x = BB_LONG; x < n0 && !h; x += 32) h = __any_sync(0xFFFFFFFFu, x + lane < n0 && bb_bit(mark, bu.at(b0 + x + lane)));
            if (h && lane == l) found |= 1u << k;
          }
#pragma unroll
        for (int k = 0; k < BB_CAND; ++k)
          if ((found >> k) & 1u) atomicOr(mark + (v[k] >> 5), 1u << (v[k] & 31));
        bb_append(found, v, list, hi, counter);
      });
    else {
      bb_rows const rows[1] = { td };
      bb_expand<T>(list, lo, hi, rows, list, hi, counter, [&](uint32_t const (&w)[BB_ILP]) {
        uint32_t found = 0;
#pragma unroll
        for (int k = 0; k < BB_ILP; ++k)
          if (w[k] != UNDECIDED && ((cand[w[k] >> 5] & ~mark[w[k] >> 5]) >> (w[k] & 31)) & 1u && bit_claim(mark, w[k])) found |= 1u << k;
        return found;
      });
    }
    uint32_t const c = bb_level_end(B);
    lo               = hi;
    hi += c;
  }
  return hi;
}

// argmax of live in * out over the undecided vertices, lowest id on ties
// (as bt_pivot); BT_NONE when there is none
template<int T>
__device__ __forceinline__ uint32_t
bb_best(bb_block& B, unsigned long long best)
{
#pragma unroll
  for (int sh = 16; sh; sh >>= 1) {
    unsigned long long const o = __shfl_xor_sync(0xFFFFFFFFu, best, sh);
    best                       = o > best ? o : best;
  }
  if ((threadIdx.x & 31) == 0 && best) atomicMax(&B.S->best, best);
  __syncthreads();
  unsigned long long const b = B.S->best;
  __syncthreads();
  if (threadIdx.x == 0) B.S->best = 0;
  return b ? 0xFFFFFFFFu - static_cast<uint32_t>(b & 0xFFFFFFFFu) : BT_NONE;
}
__device__ __forceinline__ unsigned long long
bb_key(uint32_t in, uint32_t out, uint32_t v)
{
  uint64_t const p = static_cast<uint64_t>(in) * out;
  return (static_cast<unsigned long long>(p < 0xFFFFFFFFull ? p : 0xFFFFFFFFull) << 32) | (0xFFFFFFFFu - v);
}

// The undecided vertices through the shared-memory Tarjan, if they fit it
// (warp 0; the piece lies over the two reach bitmaps, unused by then).
__device__ __noinline__ bool
bb_tarjan(bt_args const& a, bt_graph const& G, bb_block const& B, rs_piece& p)
{
  unsigned const  lane = threadIdx.x & 31u;
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t k = 0;
    for (uint32_t wb = 0; wb < G.words && k <= RS_MAXV; wb += 32) {
      uint32_t const w    = wb + lane;
      uint32_t       word = w < G.words ? B.und[w] : 0u;
      uint32_t const c    = __popc(word);
      uint32_t       incl = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= static_cast<unsigned>(d)) incl += y;
      }
      uint32_t j = k + incl - c;
      for (; word; word &= word - 1, ++j)
        if (j < RS_MAXV) p.vid[j] = w * 32 + __ffs(word) - 1;
      k += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    __syncwarp();
    bool           fits = k <= RS_MAXV;
    uint32_t const per  = (k + 31) / 32;
    uint32_t       cnt  = 0;
    if (fits)
      for (uint32_t i = lane * per; i < k && i < lane * per + per; ++i) {
        uint32_t const v = p.vid[i];
        uint32_t       c = 0;
        for (uint64_t e = G.fh[v], end = G.fh[v + 1]; e < end; ++e) c += bb_bit(B.und, a.fc[e]) ? 1u : 0u;
        p.comp[i] = static_cast<uint16_t>(c < RS_MAXE ? c : RS_MAXE);
        cnt += c;
      }
    uint32_t incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= static_cast<unsigned>(d)) incl += y;
    }
    uint32_t const total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    fits                 = fits && total <= RS_MAXE;
    if (fits) {
      uint32_t run = incl - cnt;
      for (uint32_t i = lane * per; i < k && i < lane * per + per; ++i) {
        p.off[i] = static_cast<uint16_t>(run);
        run += p.comp[i];
      }
      if (lane == 0) p.off[k] = static_cast<uint16_t>(total);
      __syncwarp();
      for (uint32_t i = lane * per; i < k && i < lane * per + per; ++i) {
        uint32_t const v = p.vid[i];
        uint32_t       o = p.off[i];
        for (uint64_t e = G.fh[v], end = G.fh[v + 1]; e < end; ++e) {
          uint32_t const w = a.fc[e];
          if (bb_bit(B.und, w)) p.adj[o++] = static_cast<uint16_t>(rs_local(p, k, w));
        }
      }
      __syncwarp();
      if (lane == 0) rs_tarjan(p, k);
      __syncwarp();
      for (uint32_t i = lane; i < k; i += 32) G.ids[p.vid[i]] = p.vid[p.comp[i]];
      if (lane == 0) atomicAdd(a.ctr + 6, 1u);
    }
    if (lane == 0) B.S->flag = fits ? 1u : 0u;
  }
  __syncthreads();
  return B.S->flag != 0;
}

template<int T>
__device__ void
bb_solve(bt_args const& a, uint32_t gi, bb_block& B, rs_piece& piece, uint32_t scratch_words)
{
  bt_graph G;
  G.vo     = a.vtx_off[gi];
  G.n      = static_cast<uint32_t>(a.vtx_off[gi + 1] - G.vo);
  G.words  = (G.n + 31) / 32;
  G.fh     = a.fh + G.vo;
  G.bh     = a.bh + G.vo;
  G.und    = a.und + a.word_off[gi];
  G.va     = a.vis_a + a.word_off[gi];
  G.vb     = a.vis_b + a.word_off[gi];
  G.indeg  = a.indeg + G.vo;
  G.outdeg = a.outdeg + G.vo;
  G.ids    = a.scc_id + G.vo;
  G.q0     = a.q0 + G.vo;
  G.q1     = a.q1 + G.vo;
  G.q2     = a.q2 + G.vo;
  B.n     = G.n;
  B.words = G.words;
  bb_rows const  fw = bb_rows_of(G.fh, a.fc), bw = bb_rows_of(G.bh, a.bc);
  bb_degrees     deg{ G.indeg, G.indeg, G.outdeg, false };
  uint32_t* const err  = a.ctr + 4;
  unsigned const  lane = threadIdx.x & 31u;
  bt_group const  g{ cg::this_cluster(), nullptr, threadIdx.x, T, true }; // phase clock and the serial Tarjan

  uint64_t t = threadIdx.x == 0 ? bt_now() : 0;
  if (threadIdx.x < 3) B.S->cnt[threadIdx.x] = 0;
  if (threadIdx.x == 0) B.S->best = 0;
  B.level = 0;
  for (uint32_t w = threadIdx.x; w < scratch_words; w += T) B.va[w] = 0; // both reach bitmaps, whatever the last graph left
  __syncthreads();
  // init: a warp takes 32 vertices (one bitmap word) at a time; live degrees
  // = raw degrees, in or out = 0 decided and queued, every id = itself
  unsigned long long best = 0;
  uint32_t           over = 0;
  uint32_t const     span = (G.n + 31) & ~31u;
  for (uint32_t v0 = threadIdx.x; v0 < span; v0 += T * BB_ILP) {
    uint32_t o[BB_ILP], i[BB_ILP];
#pragma unroll
    for (int k = 0; k < BB_ILP; ++k) {
      uint32_t const v = v0 + k * T;
      o[k] = i[k] = 0;
      if (v < G.n) o[k] = fw.length(v, fw.begin(v)), i[k] = bw.length(v, bw.begin(v));
    }
    uint32_t dead[BB_ILP], found = 0;
#pragma unroll
    for (int k = 0; k < BB_ILP; ++k) {
      uint32_t const v  = v0 + k * T;
      bool const     in = v < G.n, live = in && o[k] && i[k];
      unsigned const word = __ballot_sync(0xFFFFFFFFu, live);
      if (lane == 0 && v < G.n) B.und[v >> 5] = word;
      dead[k] = v;
      if (in) {
        G.ids[v] = v;
        deg.set(v, i[k], o[k]);
        if (!live) found |= 1u << k;
      }
      over |= i[k] >= BB_DEG8 || o[k] >= BB_DEG8 ? 1u : 0u;
      if (live) {
        unsigned long long const key = bb_key(i[k], o[k], v);
        best                         = key > best ? key : best;
      }
    }
    bb_append(found, dead, G.q0, 0, &B.S->cnt[0]);
  }
  if (__syncthreads_or(over)) {
    // a degree does not fit a byte: 32-bit degrees for this graph
    deg.wide = true;
    for (uint32_t v = threadIdx.x; v < G.n; v += T) deg.set(v, bw.length(v, bw.begin(v)), fw.length(v, fw.begin(v)));
  }
  uint32_t qn   = bb_level_end(B);
  uint32_t done = qn; // q0's length: vertices decided by trimming
  uint32_t pv   = bb_best<T>(B, best);
  uint32_t rem  = G.n - qn, levels = 0;
  uint32_t* seed = G.q0;
  if (threadIdx.x == 0) bt_phase(a, g, 0, t);
  for (uint32_t round = 0;; ++round) {
    uint32_t const before = done;
    done                  = bb_trim<T>(err, B, G.q0, deg, fw, bw, seed, qn, done, levels);
    rem -= done - before;
    if (threadIdx.x == 0) bt_phase(a, g, 1, t);
    if (rem == 0) break;
    if (rem <= (round ? a.rem_tarjan : min(a.rem_tarjan, BB_TARJAN_0))) {
      if (bb_tarjan(a, G, B, piece)) {
        if (threadIdx.x == 0) bt_phase(a, g, 4, t);
        break;
      }
      // it did not fit: the bitmaps under the piece are cleared again
      for (uint32_t w = threadIdx.x; w < scratch_words; w += T) B.va[w] = 0;
      __syncthreads();
    }
    if (round >= a.max_rounds) {
      for (uint32_t w = threadIdx.x; w < G.words; w += T) G.und[w] = B.und[w];
      bt_tarjan_serial(a, G, g, a.pos + G.vo);
      if (threadIdx.x == 0) bt_phase(a, g, 4, t);
      break;
    }
    // FW-BW from the largest live in * out; in the first round from the
    // largest raw in * out, found on the way, if the trim left it
    uint32_t p = pv;
    pv         = BT_NONE;
    if (p == BT_NONE || !bb_bit(B.und, p)) {
      unsigned long long bk = 0;
      for (uint32_t v = threadIdx.x; v < G.n; v += T)
        if (bb_bit(B.und, v)) {
          uint2 const              d   = deg.get(v);
          unsigned long long const key = bb_key(d.x, d.y, v);
          bk                           = key > bk ? key : bk;
        }
      p = bb_best<T>(B, bk);
      if (threadIdx.x == 0) bt_phase(a, g, 2, t);
    }
    if (p == BT_NONE) {
      if (threadIdx.x == 0) atomicExch(err, 1u);
      break;
    }
    if (threadIdx.x == 0) B.S->minid = 0xFFFFFFFFu;
    uint32_t nb = rem; // candidates, then reached: FW among the undecided, BW among FW's
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) nb = bb_reach<T>(err, B, dir ? bw : fw, dir ? fw : bw, dir ? B.va : B.und, dir ? B.vb : B.va, dir ? G.q2 : G.q1, p, nb);
    // the SCC (vb): smallest member, then ids a word at a time; both reach
    // bitmaps are cleared on the way
    uint32_t mn = 0xFFFFFFFFu;
    for (uint32_t w = threadIdx.x; w < G.words; w += T)
      if (B.vb[w]) {
        mn = w * 32 + __ffs(B.vb[w]) - 1;
        break; // later words of this thread hold larger ids
      }
    mn = __reduce_min_sync(0xFFFFFFFFu, mn);
    if (lane == 0 && mn != 0xFFFFFFFFu) atomicMin(&B.S->minid, mn);
    __syncthreads();
    uint32_t const id = B.S->minid;
    for (uint32_t w0 = threadIdx.x & ~31u; w0 < G.words; w0 += T) {
      uint32_t const w = w0 + lane;
      uint32_t const s = w < G.words ? B.vb[w] : 0u;
      if (w < G.words) {
        B.und[w] &= ~s;
        B.va[w] = 0;
        B.vb[w] = 0;
      }
      for (unsigned todo = __ballot_sync(0xFFFFFFFFu, s != 0); todo; todo &= todo - 1) {
        unsigned const j = __ffs(todo) - 1;
        if ((__shfl_sync(0xFFFFFFFFu, s, j) >> lane) & 1u) G.ids[(w0 + j) * 32 + lane] = id;
      }
    }
    if (threadIdx.x == 0) atomicAdd(a.ctr + 5, 1u);
    __syncthreads();
    if (threadIdx.x == 0) bt_phase(a, g, 3, t);
    rem -= nb;
    if (rem == 0) break;
    if (rem <= nb) {
      // fewer vertices are left than the SCC took: their live degrees are
      // counted anew, and the ones that have none seed the next trim
      seed = G.q0 + done;
      qn   = bb_recount<T>(B, G.q0, deg, fw, bw, done);
      done += qn;
      rem -= qn;
    } else {
      seed = G.q2; // the SCC's members seed the next trim
      qn   = nb;
    }
  }
  if (threadIdx.x == 0 && levels) atomicAdd(a.ctr + 8, levels);
  __syncthreads();
}

// Persistent blocks over class `cls` of the queue.  Dynamic shared memory:
// und | va, vb (or the Tarjan piece over them) | the warps' pack buffers.
template<uint32_t WORDS>
constexpr uint32_t bb_scratch = std::max<uint32_t>(2 * WORDS, (sizeof(rs_piece) + 3) / 4); // va and vb, or the piece
template<int T, uint32_t WORDS>
constexpr size_t bb_dyn_bytes = (WORDS + bb_scratch<WORDS>) * sizeof(uint32_t) + T / 32 * BB_PACK * sizeof(uint16_t);

template<int T, int BLOCKS, uint32_t WORDS>
__global__ void __launch_bounds__(T, BLOCKS)
k_batch_block(bt_args a, uint32_t cls)
{
  extern __shared__ __align__(16) uint32_t bb_dyn[];
  __shared__ bb_smem s;
  static_assert(WORDS / 8 / (T / 32) <= 256, "a packed vertex is 8 bits of group, 8 of place");
  bb_block B;
  B.S    = &s;
  B.und  = bb_dyn;
  B.va   = bb_dyn + WORDS;
  B.vb   = bb_dyn + 2 * WORDS;
  B.pack = reinterpret_cast<uint16_t*>(bb_dyn + WORDS + bb_scratch<WORDS>) + (threadIdx.x >> 5) * BB_PACK;
  uint32_t const first = bt_first(a.ctr, cls), count = __ldcg(a.ctr + BT_COUNT + cls);
  for (;;) {
    if (threadIdx.x == 0) s.claim = atomicAdd(a.ctr + BT_CLAIM + cls, 1u);
    __syncthreads();
    uint32_t const i = s.claim;
    __syncthreads();
    if (i >= count) break;
    bb_solve<T>(a, a.order[first + i], B, *reinterpret_cast<rs_piece*>(B.va), 2 * WORDS);
  }
}

// Persistent groups over the graphs of one class.  Launched with a cluster dimension (or none: a
// group of one block).
__global__ void __launch_bounds__(BT_THREADS, 3) // 3 blocks per SM: the path is latency-bound, graphs in flight count most
k_batch_group(bt_args a, uint32_t cls)
{
  extern __shared__ __align__(16) unsigned char bt_dyn[];
  rs_piece&          piece = *reinterpret_cast<rs_piece*>(bt_dyn);
  __shared__ bt_smem s;
  bt_group           g{ cg::this_cluster(), nullptr, 0, 0, false };
  uint32_t const     csize = g.cl.num_blocks();
  g.one                    = csize == 1;
  g.S                      = g.one ? &s : g.cl.map_shared_rank(&s, 0);
  g.gt                     = g.cl.block_rank() * BT_THREADS + threadIdx.x;
  g.GT                     = csize * BT_THREADS;
  uint32_t const first     = bt_first(a.ctr, cls);
  uint32_t const count     = __ldcg(a.ctr + BT_COUNT + cls);
  g.sync(); // every block of the cluster has started (its shared memory exists)
  for (;;) {
    if (g.leader()) g.S->g = atomicAdd(a.ctr + BT_CLAIM + cls, 1u);
    g.sync();
    uint32_t const i = g.S->g;
    g.sync();
    if (i >= count) break;
    bt_solve(a, a.order[first + i], g, piece);
  }
  g.sync(); // no block leaves while another may still reach its shared memory
}

} // namespace

// ---------------------------------------------------------------- host
namespace {

struct batch_plan
{
  void*     base = nullptr; // one allocation: keys, vals, alt, words, word_off, hist, partials
  size_t    bytes = 0;
  uint32_t* keys = nullptr;
  uint32_t* order = nullptr;
  uint32_t* kalt = nullptr;
  uint32_t* valt = nullptr;
  uint32_t* words = nullptr;
  uint64_t* word_off = nullptr;
  uint32_t* hist = nullptr;
  uint64_t* part64 = nullptr;
  uint32_t* und = nullptr;
  uint32_t* vis_a = nullptr;
  uint32_t* vis_b = nullptr;
  uint32_t* indeg = nullptr;
  uint32_t* outdeg = nullptr;
  uint32_t* q0 = nullptr;
  uint32_t* q1 = nullptr;
  uint32_t* q2 = nullptr;
  uint64_t* pos = nullptr;
  uint32_t* ctr = nullptr; // 32 words
};

} // namespace

struct batch_cache
{
  batch_plan      plan;
  cudaGraph_t     graph = nullptr;
  cudaGraphExec_t exec  = nullptr;
  void const*     key[6] = {};
  uint32_t        G = 0;
  uint64_t        N = 0;
  uint32_t        max_rounds = 0, rem_tarjan = 0, block_blocks = 0, cluster_size = 0, cluster_blocks = 0;
  uint64_t        cluster_min = 0;
  uint32_t        joint       = 0;
  cudaStream_t    cap_stream = nullptr;
  cudaStream_t    side[3]    = {}; // the classes' branches of the captured call
  cudaEvent_t     fork = nullptr, join[3] = {};
  uint32_t        l_blocks = 0, m_blocks = 0;
};

void
batch_release(kspn_context* ctx)
{
  batch_cache* c = ctx->batch;
  if (!c) return;
  if (c->exec) cudaGraphExecDestroy(c->exec);
  if (c->graph) cudaGraphDestroy(c->graph);
  if (c->plan.base) cudaFree(c->plan.base);
  if (c->cap_stream) cudaStreamDestroy(c->cap_stream);
  for (cudaStream_t x : c->side)
    if (x) cudaStreamDestroy(x);
  for (cudaEvent_t x : { c->fork, c->join[0], c->join[1], c->join[2] })
    if (x) cudaEventDestroy(x);
  delete c;
  ctx->batch = nullptr;
}

namespace {

void
carve_plan(batch_plan& p, char* base, uint32_t G, uint64_t N, size_t* bytes_out)
{
  size_t off  = 0;
  auto   take = [&](size_t bytes) {
    off           = (off + 255) & ~size_t(255);
    char* const q = base ? base + off : nullptr;
    off += bytes;
    return q;
  };
  size_t const hist_n = radix_hist_entries(G);
  size_t const part_n = scan_partial_entries(hist_n > G + 1 ? hist_n : G + 1);
  size_t const words  = N / 32 + G + 2; // every graph rounds up to whole words
  p.keys     = reinterpret_cast<uint32_t*>(take(4 * (G + 1)));
  p.order    = reinterpret_cast<uint32_t*>(take(4 * (G + 1)));
  p.kalt     = reinterpret_cast<uint32_t*>(take(4 * (G + 1)));
  p.valt     = reinterpret_cast<uint32_t*>(take(4 * (G + 1)));
  p.words    = reinterpret_cast<uint32_t*>(take(4 * (G + 1)));
  p.word_off = reinterpret_cast<uint64_t*>(take(8 * (G + 1)));
  p.hist     = reinterpret_cast<uint32_t*>(take(4 * hist_n));
  p.part64   = reinterpret_cast<uint64_t*>(take(8 * part_n));
  p.und      = reinterpret_cast<uint32_t*>(take(4 * words));
  p.vis_a    = reinterpret_cast<uint32_t*>(take(4 * words));
  p.vis_b    = reinterpret_cast<uint32_t*>(take(4 * words));
  p.indeg    = reinterpret_cast<uint32_t*>(take(4 * (N + 1)));
  p.outdeg   = reinterpret_cast<uint32_t*>(take(4 * (N + 1)));
  p.q0       = reinterpret_cast<uint32_t*>(take(4 * (N + 1)));
  p.q1       = reinterpret_cast<uint32_t*>(take(4 * (N + 1)));
  p.q2       = reinterpret_cast<uint32_t*>(take(4 * (N + 1)));
  p.pos      = reinterpret_cast<uint64_t*>(take(8 * (N + 1)));
  p.ctr      = reinterpret_cast<uint32_t*>(take(4 * 64)); // [32..64): u64 phase times (bt_phase)
  *bytes_out = (off + 255) & ~size_t(255);
}

// The whole call as stream work (captured once per batch and settings).
void
enqueue_batch(kspn_context* ctx, batch_cache& c, bt_args const& a0)
{
  cudaStream_t const s = ctx->stream;
  batch_plan&        p = c.plan;
  uint32_t const     G = c.G;
  KSPN_CUDA(cudaMemsetAsync(p.ctr, 0, 64 * sizeof(uint32_t), s));
  unsigned const cgrid = div_up(G, 256);
  k_bt_classify<<<cgrid < 1 ? 1 : cgrid, 256, 0, s>>>(G, a0.vtx_off, a0.fh, c.cluster_min, c.joint, BB_L_WORDS * 32, G <= 2 * c.l_blocks ? BB_M_FEW : BB_M_WORDS * 32, p.keys, p.order, p.words, p.ctr);
  KSPN_CHECK_LAUNCH();
  exclusive_scan<uint64_t>(s, f_words{ p.words }, G, p.word_off, p.part64, nullptr);
  radix_sort_pairs(ctx, p.keys, p.order, p.kalt, p.valt, G, 0, 32, p.hist);
  bt_args a    = a0;
  a.word_off   = p.word_off;
  a.und        = p.und;
  a.vis_a      = p.vis_a;
  a.vis_b      = p.vis_b;
  a.indeg      = p.indeg;
  a.outdeg     = p.outdeg;
  a.q0         = p.q0;
  a.q1         = p.q1;
  a.q2         = p.q2;
  a.pos        = p.pos;
  a.order      = p.order;
  a.ctr        = p.ctr;
  a.max_rounds = c.max_rounds;
  a.rem_tarjan = c.rem_tarjan;
  a.joint      = c.joint;
  // the classes' kernels side by side: blocks of the smaller classes move in
  // as the larger graphs' blocks leave
  KSPN_CUDA(cudaEventRecord(c.fork, s));
  for (cudaStream_t side : c.side) KSPN_CUDA(cudaStreamWaitEvent(side, c.fork, 0));
  k_batch_block<BB_L_THREADS, BB_L_BLOCKS, BB_L_WORDS><<<c.l_blocks, BB_L_THREADS, bb_dyn_bytes<BB_L_THREADS, BB_L_WORDS>, s>>>(a, BT_BLOCK_L);
  k_batch_block<BB_M_THREADS, BB_M_BLOCKS, BB_M_WORDS><<<c.m_blocks, BB_M_THREADS, bb_dyn_bytes<BB_M_THREADS, BB_M_WORDS>, c.side[0]>>>(a, BT_BLOCK_M);
  k_batch_small<<<148 * 4, BS_WARPS * 32, BS_WARPS * sizeof(rs_piece), c.side[1]>>>(a);
  KSPN_CHECK_LAUNCH();
  if (c.cluster_size > 1) {
    cudaLaunchConfig_t   cfg{};
    cudaLaunchAttribute  attr[1];
    attr[0].id               = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c.cluster_size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim              = dim3(c.cluster_blocks);
    cfg.blockDim             = dim3(BT_THREADS);
    cfg.dynamicSmemBytes     = sizeof(rs_piece);
    cfg.stream               = c.side[2];
    cfg.attrs                = attr;
    cfg.numAttrs             = 1;
    KSPN_CUDA(cudaLaunchKernelEx(&cfg, k_batch_group, a, static_cast<uint32_t>(BT_CLUSTER)));
  }
  k_batch_group<<<c.block_blocks, BT_THREADS, sizeof(rs_piece), c.side[2]>>>(a, BT_GLOBAL);
  KSPN_CHECK_LAUNCH();
  for (int k = 0; k < 3; ++k) {
    KSPN_CUDA(cudaEventRecord(c.join[k], c.side[k]));
    KSPN_CUDA(cudaStreamWaitEvent(s, c.join[k], 0));
  }
}

} // namespace

void
scc_batched(kspn_context* ctx, uint32_t G, uint64_t N, uint64_t const* vtx_off, uint64_t const* fh, uint32_t const* fc, uint64_t const* bh, uint32_t const* bc, uint32_t* scc_id,
            kspn_batch_options const& opt, kspn_batch_stats* st)
{
  if (G == 0) return;
  uint32_t const rem = opt.rem_tarjan ? opt.rem_tarjan : RS_MAXV;
  if (rem > RS_MAXV) throw error{ KSPN_ERR_INVALID_ARGUMENT, "scc_batched: rem_tarjan > 512" };
  uint32_t const rounds = opt.max_rounds ? opt.max_rounds : 64;
  uint32_t const csize  = opt.cluster_size ? opt.cluster_size : 1;
  uint64_t const cmin   = csize == 1 ? ~0ull : (opt.cluster_min ? opt.cluster_min : (1ull << 16));
  if (csize > 8) throw error{ KSPN_ERR_INVALID_ARGUMENT, "scc_batched: cluster_size > 8" };
  uint32_t const joint = opt.search == 1 ? 1u : 0u; // 1: joint searches; 0 (default), 2: FW then BW
  batch_cache*&  cp     = ctx->batch;
  if (!cp) cp = new batch_cache{};
  batch_cache&      c   = *cp;
  void const* const key[6] = { vtx_off, fh, fc, bh, bc, scc_id };
  bool              same   = c.exec && c.G == G && c.N == N && c.max_rounds == rounds && c.rem_tarjan == rem && c.cluster_size == csize && c.cluster_min == cmin && c.joint == joint;
  for (int i = 0; i < 6 && same; ++i) same = c.key[i] == key[i];
  if (!same) {
    if (c.exec) cudaGraphExecDestroy(c.exec), c.exec = nullptr;
    if (c.graph) cudaGraphDestroy(c.graph), c.graph = nullptr;
    size_t bytes = 0;
    carve_plan(c.plan, nullptr, G, N, &bytes);
    if (bytes > c.plan.bytes) {
      if (c.plan.base) {
        KSPN_CUDA(cudaStreamSynchronize(ctx->stream));
        cudaFree(c.plan.base);
        c.plan = {};
      }
      void* b = nullptr;
      if (cudaMalloc(&b, bytes) != cudaSuccess) {
        cudaGetLastError();
        throw error{ KSPN_ERR_OOM, "batched workspace of " + std::to_string(bytes) + " bytes" };
      }
      c.plan.base  = b;
      c.plan.bytes = bytes;
    }
    size_t const keep = c.plan.bytes;
    void* const  base = c.plan.base;
    carve_plan(c.plan, static_cast<char*>(base), G, N, &bytes);
    c.plan.base  = base;
    c.plan.bytes = keep;
    c.G = G, c.N = N, c.max_rounds = rounds, c.rem_tarjan = rem, c.cluster_size = csize, c.cluster_min = cmin, c.joint = joint;
    for (int i = 0; i < 6; ++i) c.key[i] = key[i];
    int bps = 0, sms = 0;
    KSPN_CUDA(cudaFuncSetAttribute(k_batch_small, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(BS_WARPS * sizeof(rs_piece))));
    KSPN_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_batch_group, BT_THREADS, sizeof(rs_piece)));
    KSPN_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    c.block_blocks = static_cast<uint32_t>(std::max(1, bps) * sms);
    c.cluster_blocks = c.block_blocks;
    auto* const kl = &k_batch_block<BB_L_THREADS, BB_L_BLOCKS, BB_L_WORDS>;
    auto* const km = &k_batch_block<BB_M_THREADS, BB_M_BLOCKS, BB_M_WORDS>;
    KSPN_CUDA(cudaFuncSetAttribute(kl, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bb_dyn_bytes<BB_L_THREADS, BB_L_WORDS>)));
    KSPN_CUDA(cudaFuncSetAttribute(km, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bb_dyn_bytes<BB_M_THREADS, BB_M_WORDS>)));
    KSPN_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kl, BB_L_THREADS, bb_dyn_bytes<BB_L_THREADS, BB_L_WORDS>));
    c.l_blocks = static_cast<uint32_t>(std::max(1, bps) * sms);
    KSPN_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, km, BB_M_THREADS, bb_dyn_bytes<BB_M_THREADS, BB_M_WORDS>));
    c.m_blocks = static_cast<uint32_t>(std::max(1, bps) * sms);
    if (csize > 1) {
      cudaLaunchConfig_t  cfg{};
      cudaLaunchAttribute attr[1];
      attr[0].id               = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = csize;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.gridDim              = dim3(c.block_blocks / csize * csize);
      cfg.blockDim             = dim3(BT_THREADS);
      cfg.dynamicSmemBytes     = sizeof(rs_piece);
      cfg.attrs                = attr;
      cfg.numAttrs             = 1;
      int clusters             = 0;
      KSPN_CUDA(cudaOccupancyMaxActiveClusters(&clusters, k_batch_group, &cfg));
      if (clusters < 1) throw error{ KSPN_ERR_CUDA, "scc_batched: no cluster of that size fits" };
      c.cluster_blocks = static_cast<uint32_t>(clusters) * csize;
    }
    bt_args a{};
    a.G       = G;
    a.vtx_off = vtx_off;
    a.fh = fh, a.fc = fc, a.bh = bh, a.bc = bc;
    a.scc_id = scc_id;
    // capture the call (plan + solve) once, on a private stream (the
    // context's stream may be the legacy default stream, which cannot be
    // captured); later calls replay it on the context's stream
    if (!c.cap_stream) KSPN_CUDA(cudaStreamCreateWithFlags(&c.cap_stream, cudaStreamNonBlocking));
    if (!c.fork) KSPN_CUDA(cudaEventCreateWithFlags(&c.fork, cudaEventDisableTiming));
    for (int k = 0; k < 3; ++k) {
      if (!c.side[k]) KSPN_CUDA(cudaStreamCreateWithFlags(&c.side[k], cudaStreamNonBlocking));
      if (!c.join[k]) KSPN_CUDA(cudaEventCreateWithFlags(&c.join[k], cudaEventDisableTiming));
    }
    cudaStream_t const user = ctx->stream;
    KSPN_CUDA(cudaStreamSynchronize(user));
    ctx->stream = c.cap_stream;
    KSPN_CUDA(cudaStreamBeginCapture(c.cap_stream, cudaStreamCaptureModeThreadLocal));
    try {
      enqueue_batch(ctx, c, a);
    } catch (...) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(c.cap_stream, &g);
      if (g) cudaGraphDestroy(g);
      ctx->stream = user;
      throw;
    }
    cudaError_t const ec = cudaStreamEndCapture(c.cap_stream, &c.graph);
    ctx->stream          = user;
    KSPN_CUDA(ec);
    KSPN_CUDA(cudaGraphInstantiate(&c.exec, c.graph, 0));
  }
  KSPN_CUDA(cudaGraphLaunch(c.exec, ctx->stream));
  ctx->launches += 1;
  uint32_t h[64];
  KSPN_CUDA(cudaMemcpyAsync(h, c.plan.ctr, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  KSPN_CUDA(cudaStreamSynchronize(ctx->stream));
  if (h[4]) throw error{ KSPN_ERR_TIMEOUT, "scc_batched: a level or round bound was reached" };
  if (st) {
    st->graphs_small     = h[BT_COUNT + BT_WARP];
    st->graphs_large     = h[BT_COUNT + BT_CLUSTER] + h[BT_COUNT + BT_GLOBAL] + h[BT_COUNT + BT_BLOCK_L] + h[BT_COUNT + BT_BLOCK_M];
    st->graphs_cluster   = h[BT_COUNT + BT_CLUSTER];
    st->cluster_size     = csize;
    st->fwbw_rounds      = h[5];
    st->tarjan_smem      = h[6];
    st->tarjan_serial    = h[7];
    st->trim_levels      = h[8];
    uint64_t ph[5];
    std::memcpy(ph, h + 32, sizeof(ph));
    for (int k = 0; k < 5; ++k) st->phase_ms[k] = static_cast<float>(ph[k] * 1e-6);
  }
}

} // namespace kspn
