// Residual device finish: the undecided sub-graph, piece by piece.
//
// Reference: the residual step of variant/scc_trim_ex_residual.hpp:110-127
// (also scc_ispan_like.hpp, scc_trim_ex_light_residual.hpp):
// allgather_fw_sub_graph (kaspan/scc/allgather_sub_graph.hpp:253-301)
// gathers the sub-graph induced by the undecided vertices, tarjan
// (kaspan/scc/tarjan.hpp:20-136) decomposes it on one core, and each SCC is
// named by its smallest original vertex id.
//
// On the device the sub-graph splits into weakly connected pieces (an SCC
// never spans two), and one warp or block decomposes each small piece:
//   1. the undecided vertices are listed (every later pass runs over the
//      list), and union-find over their out-edges to undecided vertices joins
//      them (hooking the larger root under the smaller with atomicCAS, path
//      halving); then every entry is set to its root by a pass in which only
//      v's own thread writes parent[v]; every loop bounded;
//   2. in that pass each vertex takes a place in its piece (an atomic count at
//      the root); a pass over the roots gives each piece a range of one member
//      array, and each vertex enters its place;
//   3. a piece of up to 32 vertices goes to a warp, lane = vertex: rows become
//      bit masks, Warshall's closure takes one shuffle per vertex, and an SCC is
//      the closure and its transpose (one ballot per vertex); a piece of up to
//      RS_MAXV vertices and RS_MAXE internal edges goes to a block, trim and
//      label rounds in shared memory.  Either way each member gets its SCC's
//      smallest vertex and leaves und.
// Larger pieces stay undecided; the pipeline's label rounds finish them.
// Bound: launches and the latency of a few dependent loads each.  RGG of 10^6
// vertices (29,636 undecided, whole step): 390 us with ordered compaction,
// a radix sort by root and every piece through one lane's Tarjan.
#include "prim.cuh"
#include "small.cuh"
#include "tarjan_smem.cuh"

#include <algorithm>

namespace kspn {

namespace {

constexpr int      RS_THREADS = 256;
constexpr uint32_t RS_FIND    = 1u << 20; // bound on one find / unite loop

unsigned
rs_grid(uint64_t items)
{
  uint64_t const b = (items + RS_THREADS - 1) / RS_THREADS;
  return static_cast<unsigned>(b < 148ull * 16 ? (b ? b : 1) : 148ull * 16);
}

__device__ __forceinline__ bool
und_has(uint32_t const* und, uint32_t v)
{
  return (und[v >> 5] >> (v & 31)) & 1u;
}

// root of x with path halving; UNDECIDED when the bound was reached
__device__ __forceinline__ uint32_t
rs_find(uint32_t* parent, uint32_t x)
{
  for (uint32_t it = 0; it < RS_FIND; ++it) {
    uint32_t const p = __ldcg(parent + x);
    if (p == x) return x;
    uint32_t const gp = __ldcg(parent + p);
    if (gp != p) parent[x] = gp; // halving (a lost race only skips a shortcut)
    x = gp;
  }
  return UNDECIDED;
}

// The undecided vertices (in no particular order), each a root of its own
// with an empty piece.
__global__ void __launch_bounds__(RS_THREADS)
k_res_list(uint32_t n, uint32_t const* __restrict__ und, uint32_t* __restrict__ parent, uint32_t* __restrict__ count, uint32_t* __restrict__ list, uint32_t* list_n)
{
  unsigned const lane  = threadIdx.x & 31u;
  uint32_t const words = (n + 31) / 32, span = (words + 31) & ~31u;
  for (uint32_t w = blockIdx.x * RS_THREADS + threadIdx.x; w < span; w += gridDim.x * RS_THREADS) {
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
    if (lane == 0) at = atomicAdd(list_n, tot);
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + incl - c;
    for (; x; x &= x - 1) {
      uint32_t const v = w * 32 + __ffs(x) - 1;
      list[at++]       = v;
      parent[v]        = v;
      count[v]         = 0;
    }
  }
}

// u ~ v (both undecided); false when a loop bound was reached
__device__ __forceinline__ bool
rs_unite(uint32_t* parent, uint32_t u, uint32_t v)
{
  uint32_t a = u, b = v;
  for (uint32_t it = 0; it < RS_FIND; ++it) {
    a = rs_find(parent, a);
    b = rs_find(parent, b);
    if (a == UNDECIDED || b == UNDECIDED) return false;
    if (a == b) return true;
    if (a < b) {
      uint32_t const s = a;
      a = b, b = s;
    }
    // hook the larger root under the smaller
    if (atomicCAS(parent + a, a, b) == a) return true;
  }
  return false;
}

__device__ __forceinline__ void
rs_edge(uint32_t const* und, uint32_t* parent, uint32_t* err, uint32_t u, uint32_t v)
{
  if (v != u && und_has(und, v) && !rs_unite(parent, u, v)) atomicExch(err, 1u);
}

// u ~ v for every edge between undecided vertices.  A lane walks a row of
// up to 32 edges, the warp one of up to HEAVY_ROW; longer rows are listed
// for k_res_hook_heavy.
__global__ void __launch_bounds__(RS_THREADS)
k_res_hook(uint32_t const* __restrict__ list, uint32_t const* __restrict__ list_n, uint32_t const* __restrict__ und, uint64_t const* __restrict__ fh, uint32_t const* __restrict__ fc,
           uint32_t* parent, uint32_t* err, uint32_t* heavy, uint32_t* heavy_n)
{
  unsigned const lane = threadIdx.x & 31u;
  uint32_t const k    = *list_n;
  for (uint32_t t0 = blockIdx.x * RS_THREADS + (threadIdx.x & ~31u); t0 < k; t0 += gridDim.x * RS_THREADS) {
    bool const     have = t0 + lane < k;
    uint32_t const u    = have ? list[t0 + lane] : 0u;
    uint64_t       b = 0, e = 0;
    if (have) b = fh[u], e = fh[u + 1];
    uint64_t const len = e - b;
    if (have && len <= 32)
      for (uint64_t x = b; x < e; ++x) rs_edge(und, parent, err, u, fc[x]);
    for (unsigned todo = __ballot_sync(0xFFFFFFFFu, have && len > 32 && len <= HEAVY_ROW); todo; todo &= todo - 1) {
      unsigned const l  = __ffs(todo) - 1;
      uint32_t const ul = __shfl_sync(0xFFFFFFFFu, u, l);
      uint64_t const b0 = __shfl_sync(0xFFFFFFFFu, b, l), e0 = __shfl_sync(0xFFFFFFFFu, e, l);
      for (uint64_t x = b0 + lane; x < e0; x += 32) rs_edge(und, parent, err, ul, fc[x]);
    }
    warp_push(have && len > HEAVY_ROW, u, heavy, heavy_n);
  }
}

// The listed rows, in slices over every warp of the grid.
__global__ void __launch_bounds__(RS_THREADS)
k_res_hook_heavy(uint32_t const* __restrict__ und, uint64_t const* __restrict__ fh, uint32_t const* __restrict__ fc, uint32_t* parent, uint32_t* err, uint32_t const* heavy, uint32_t const* heavy_n)
{
  unsigned const lane = threadIdx.x & 31u;
  heavy_slices(heavy, *heavy_n, fh, [&](uint32_t, uint32_t u, uint64_t b, uint64_t e) {
    for (uint64_t x = b + lane; x < e; x += 32) rs_edge(und, parent, err, u, fc[x]);
  });
}

// parent[v] = root of v, each entry written only by v's own thread (the
// walk itself writes nothing), so every entry ends at its root; and v's
// place in its piece.
__global__ void __launch_bounds__(RS_THREADS)
k_res_flatten(uint32_t const* __restrict__ list, uint32_t const* __restrict__ list_n, uint32_t* parent, uint32_t* count, uint32_t* __restrict__ place, uint32_t* err)
{
  uint32_t const k = *list_n;
  for (uint32_t i = blockIdx.x * RS_THREADS + threadIdx.x; i < k; i += gridDim.x * RS_THREADS) {
    uint32_t const v = list[i];
    uint32_t       x = v;
    bool           ok = false;
    for (uint32_t it = 0; it < RS_FIND; ++it) {
      uint32_t const p = __ldcg(parent + x);
      if (p == x) {
        ok = true;
        break;
      }
      x = p;
    }
    if (!ok) atomicExch(err, 1u);
    else {
      parent[v] = x;
      place[v]  = atomicAdd(count + x, 1u);
    }
  }
}

// Device counters of the pieces.
struct rs_counts
{
  uint32_t list_n;  // undecided vertices
  uint32_t members; // handed-out places of the member array
  uint32_t small, mid; // pieces of at most 32 and of at most RS_MAXV vertices
};

// Every piece's range of the member array, and its list: small pieces from
// the front of `pieces`, the others from its end (an entry per vertex holds
// both).  Pieces of more than RS_MAXV vertices get none.
__global__ void __launch_bounds__(RS_THREADS)
k_res_ranges(uint32_t const* __restrict__ list, uint32_t const* __restrict__ parent, uint32_t const* __restrict__ count, uint32_t* __restrict__ start, uint32_t* __restrict__ pieces, uint32_t cap,
             rs_counts* rc, uint32_t* big)
{
  unsigned const lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  uint32_t const k    = rc->list_n;
  for (uint32_t t0 = blockIdx.x * RS_THREADS + (threadIdx.x & ~31u); t0 < k; t0 += gridDim.x * RS_THREADS) {
    uint32_t const v    = t0 + lane < k ? list[t0 + lane] : UNDECIDED;
    bool const     root = v != UNDECIDED && parent[v] == v;
    uint32_t const c    = root ? count[v] : 0u;
    uint32_t const take = c <= RS_MAXV ? c : 0u;
    if (root && c > RS_MAXV) start[v] = UNDECIDED, atomicAdd(big, 1u);
    uint32_t incl = take;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= static_cast<unsigned>(d)) incl += y;
    }
    unsigned const sm = __ballot_sync(0xFFFFFFFFu, take && take <= 32), md = __ballot_sync(0xFFFFFFFFu, take > 32);
    uint32_t       m0 = 0, s0 = 0, d0 = 0;
    if (lane == 31 && incl) m0 = atomicAdd(&rc->members, incl);
    if (lane == 0 && sm) s0 = atomicAdd(&rc->small, static_cast<uint32_t>(__popc(sm)));
    if (lane == 0 && md) d0 = atomicAdd(&rc->mid, static_cast<uint32_t>(__popc(md)));
    m0 = __shfl_sync(0xFFFFFFFFu, m0, 31), s0 = __shfl_sync(0xFFFFFFFFu, s0, 0), d0 = __shfl_sync(0xFFFFFFFFu, d0, 0);
    if (take) {
      start[v] = m0 + incl - take;
      if (take <= 32) pieces[s0 + __popc(sm & lt)] = v;
      else pieces[cap - 1 - (d0 + __popc(md & lt))] = v;
    }
  }
}

__global__ void __launch_bounds__(RS_THREADS)
k_res_members(uint32_t const* __restrict__ list, uint32_t const* __restrict__ list_n, uint32_t const* __restrict__ parent, uint32_t const* __restrict__ start, uint32_t const* __restrict__ place,
              uint32_t* __restrict__ members)
{
  uint32_t const k = *list_n;
  for (uint32_t i = blockIdx.x * RS_THREADS + threadIdx.x; i < k; i += gridDim.x * RS_THREADS) {
    uint32_t const v = list[i], b = start[parent[v]];
    if (b != UNDECIDED) members[b + place[v]] = v;
  }
}

// One warp per piece of at most 32 vertices, lane = place in the piece.
// und_in is the undecided set as the step found it (a vertex decided here
// still counts as its own piece's).
__global__ void __launch_bounds__(RS_THREADS)
k_res_small(rs_counts const* __restrict__ rc, uint32_t const* __restrict__ pieces, uint32_t const* __restrict__ count, uint32_t const* __restrict__ start, uint32_t const* __restrict__ place,
            uint32_t const* __restrict__ members, uint64_t const* __restrict__ fh, uint32_t const* __restrict__ fc, uint32_t* und, uint32_t* __restrict__ scc_id, uint32_t* decided, uint32_t* big)
{
  unsigned const lane = threadIdx.x & 31u;
  uint32_t const P    = rc->small;
  uint32_t       dec  = 0;
  for (uint32_t p = blockIdx.x * (RS_THREADS / 32) + (threadIdx.x >> 5); p < P; p += gridDim.x * (RS_THREADS / 32)) {
    uint32_t const root = pieces[p], k = count[root], b = start[root];
    bool const     have = lane < k;
    uint32_t const v    = have ? members[b + lane] : UNDECIDED;
    uint64_t const e0   = have ? fh[v] : 0;
    uint32_t const len  = have ? static_cast<uint32_t>(min(fh[v + 1] - e0, static_cast<uint64_t>(HEAVY_ROW) + 1)) : 0u;
    bool           left = __any_sync(0xFFFFFFFFu, len > HEAVY_ROW); // a row too long for one lane: left to the later rounds
    uint32_t       reach = have ? 1u << lane : 0u, edges = 0;
    // the row's members of the piece (undecided neighbours all are): four
    // neighbours' ids, state words and places in flight at once
    uint32_t const most = __reduce_max_sync(0xFFFFFFFFu, len);
    for (uint32_t x = 0; x < most && !left; x += 4) {
      uint32_t w[4], u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = x + j < len ? fc[e0 + x + j] : UNDECIDED;
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = w[j] != UNDECIDED ? (__ldcg(und + (w[j] >> 5)) >> (w[j] & 31)) & 1u : 0u;
      // another piece's vertex may just have been decided; one of this piece
      // has not: the piece is this warp's
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (u[j]) reach |= 1u << (place[w[j]] & 31u), ++edges;
    }
    left = left || __reduce_add_sync(0xFFFFFFFFu, edges) > RS_MAXE;
    if (left) {
      if (lane == 0) atomicAdd(big, 1u);
      continue;
    }
    // Warshall: after step j every path through places <= j counts
    for (uint32_t j = 0; j < k; ++j) {
      uint32_t const rj = __shfl_sync(0xFFFFFFFFu, reach, j);
      if ((reach >> j) & 1u) reach |= rj;
    }
    uint32_t back = 0; // who reaches this lane's vertex
    for (uint32_t j = 0; j < k; ++j) {
      unsigned const col = __ballot_sync(0xFFFFFFFFu, (reach >> j) & 1u);
      if (lane == j) back = col;
    }
    uint32_t const scc = reach & back;
    uint32_t       id  = v;
    for (uint32_t j = 0; j < k; ++j) {
      uint32_t const vj = __shfl_sync(0xFFFFFFFFu, v, j);
      if ((scc >> j) & 1u) id = min(id, vj);
    }
    if (have) {
      scc_id[v] = id;
      atomicAnd(und + (v >> 5), ~(1u << (v & 31)));
    }
    dec += lane == 0 ? k : 0u;
  }
  if (lane == 0 && dec) atomicAdd(decided, dec);
}

// One block per piece of 33 to RS_MAXV vertices and at most RS_MAXE internal
// edges, in shared memory: local index = place in the piece, the rows of both
// directions built from the out-rows' undecided neighbours, then trim and
// label rounds (small.cuh).  One lane's Tarjan of such a piece took 0.25 us
// per vertex and edge, 300 us and more for the largest; a level here takes
// about 0.25 us.  Whole call, random geometric graphs of 250,000 / 10^6 / 4 M
// vertices: 1,051 / 1,025 / 2,154 -> 919 / 933 / 1,887 us; 128 threads 934 /
// 936 / 1,930, 512 threads the same within 2%.
constexpr int RB_T = 256;
struct rb_piece
{
  uint32_t vid[RS_MAXV], edge[RS_MAXE], lab[RS_MAXV], out_at[RS_MAXV], in_at[RS_MAXV];
  uint32_t und[RS_MAXV / 32], open[RS_MAXV / 32], vis[RS_MAXV / 32], inq[RS_MAXV / 32];
  uint16_t q0[RS_MAXV], q1[RS_MAXV], fh[RS_MAXV + 2], bh[RS_MAXV + 2], fc[RS_MAXE], bc[RS_MAXE];
  uint32_t edges;
};

__global__ void __launch_bounds__(RB_T)
k_res_block(rs_counts const* __restrict__ rc, uint32_t const* __restrict__ pieces, uint32_t cap, uint32_t const* __restrict__ count, uint32_t const* __restrict__ start,
            uint32_t const* __restrict__ place, uint32_t const* __restrict__ members, uint64_t const* __restrict__ fh, uint32_t const* __restrict__ fc, uint32_t* und,
            uint32_t* scc_id, uint32_t* decided, uint32_t* big)
{
  __shared__ rb_piece  p;
  __shared__ sm_shared S;
  unsigned const       lane = threadIdx.x & 31u;
  uint32_t const       P    = rc->mid;
  uint32_t             dec  = 0;
  for (uint32_t pi = blockIdx.x; pi < P; pi += gridDim.x) {
    uint32_t const root = pieces[cap - 1 - pi], k = count[root], b = start[root];
    if (threadIdx.x == 0) p.edges = 0;
    if (threadIdx.x < 6) S.cnt[threadIdx.x >> 1][threadIdx.x & 1] = 0;
    bool heavy_row = false;
    for (uint32_t i = threadIdx.x; i < k; i += RB_T) {
      uint32_t const v = members[b + i];
      p.vid[i]         = v;
      p.out_at[i] = p.in_at[i] = 0;
      heavy_row |= fh[v + 1] - fh[v] > HEAVY_ROW;
    }
    // a member's row is too long for a few lanes: left to the later rounds
    bool left = __syncthreads_or(heavy_row);
    // internal edges, four lanes per vertex (undecided neighbours lie in this
    // piece, and nobody else decides them)
    for (uint32_t i = threadIdx.x >> 2; i < k && !left; i += RB_T / 4) {
      uint32_t const v = p.vid[i];
      uint64_t const end = fh[v + 1];
      for (uint64_t e = fh[v] + (lane & 3u); e < end; e += 4) {
        uint32_t const w = fc[e];
        if (!und_has(und, w)) continue;
        uint32_t const at = atomicAdd(&p.edges, 1u);
        if (at >= RS_MAXE) break;
        uint32_t const j = place[w];
        p.edge[at]       = i << 16 | j;
        atomicAdd(p.out_at + i, 1u);
        atomicAdd(p.in_at + j, 1u);
      }
    }
    __syncthreads();
    uint32_t const m = p.edges;
    if (left || m > RS_MAXE) {
      if (threadIdx.x == 0) atomicAdd(big, 1u);
      __syncthreads();
      continue;
    }
    // offsets: warp 0 the out-rows', warp 1 the in-rows'
    if (threadIdx.x < 64) {
      uint32_t* const at  = threadIdx.x < 32 ? p.out_at : p.in_at;
      uint16_t* const hd  = threadIdx.x < 32 ? p.fh : p.bh;
      uint32_t        run = 0;
      for (uint32_t i0 = 0; i0 < k; i0 += 32) {
        uint32_t const i = i0 + lane, c = i < k ? at[i] : 0u;
        uint32_t       incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
          if (lane >= static_cast<unsigned>(d)) incl += y;
        }
        if (i < k) at[i] = run + incl - c, hd[i] = static_cast<uint16_t>(run + incl - c);
        run += __shfl_sync(0xFFFFFFFFu, incl, 31);
      }
      if (lane == 0) hd[k] = static_cast<uint16_t>(run);
    }
    for (uint32_t w = threadIdx.x; w < (k + 31) / 32; w += RB_T) p.und[w] = k - w * 32 >= 32 ? 0xFFFFFFFFu : (1u << (k & 31)) - 1u;
    for (uint32_t i = threadIdx.x; i < k; i += RB_T) scc_id[p.vid[i]] = p.vid[i];
    __syncthreads();
    for (uint32_t x = threadIdx.x; x < m; x += RB_T) {
      uint32_t const i = p.edge[x] >> 16, j = p.edge[x] & 0xFFFFu;
      p.fc[atomicAdd(p.out_at + i, 1u)] = static_cast<uint16_t>(j);
      p.bc[atomicAdd(p.in_at + j, 1u)]  = static_cast<uint16_t>(i);
    }
    __syncthreads();
    sm_graph G{ k, (k + 31) / 32, p.lab, p.und, p.open, p.vis, p.inq, p.q0, p.q1, p.fh, p.bh, p.fc, p.bc, &S, 0 };
    auto const name  = [&](uint32_t v) { return p.vid[v]; };
    uint32_t   rem   = k - sm_trim<RB_T>(G), edges = 0;
    for (uint32_t round = 0; rem; ++round) { // a round decides at least one component
      uint32_t d = sm_label_round<RB_T>(G, round, scc_id, name, edges);
      if (d < rem) d += sm_trim<RB_T>(G);
      rem -= d;
    }
    // each vertex's word cleared by an atomic (pieces share words)
    for (uint32_t i = threadIdx.x; i < k; i += RB_T) atomicAnd(und + (p.vid[i] >> 5), ~(1u << (p.vid[i] & 31)));
    dec += threadIdx.x == 0 ? k : 0u;
    __syncthreads();
  }
  if (threadIdx.x == 0 && dec) atomicAdd(decided, dec);
}

} // namespace

// Decides every undecided piece (weakly connected component of the
// undecided sub-graph) of at most RS_MAXV vertices and RS_MAXE internal edges;
// returns the vertices decided.  `undecided` (n when not known) sizes the
// launches.  *pieces_left (nullable) = pieces left undecided.
uint32_t
residual(kspn_context* ctx, dgraph const& g, uint32_t* und, uint32_t* scc_id, uint32_t* pieces_left, uint64_t undecided)
{
  cudaStream_t const s = ctx->stream;
  auto&              ws = ctx->ws;
  if (pieces_left) *pieces_left = 0;
  if (g.n == 0) return 0;
  size_t const hcap  = heavy_capacity(g.n, g.m);
  size_t const each  = static_cast<size_t>(g.n) + 64;
  size_t const bytes = (6 * each + hcap) * sizeof(uint32_t) + 16 * 256;
  char*        base  = static_cast<char*>(context_buffer(ctx, BUF_BUILD, bytes));
  size_t       off   = 0;
  auto         take  = [&](size_t count) {
    off          = (off + 255) & ~size_t(255);
    auto* const p = reinterpret_cast<uint32_t*>(base + off);
    off += count * sizeof(uint32_t);
    return p;
  };
  uint32_t* list    = take(each);
  uint32_t* count   = take(each); // by vertex: members of the piece whose root it is
  uint32_t* start   = take(each); // by vertex: a root's range of `members`
  uint32_t* place   = take(each); // by vertex: its place in its piece
  uint32_t* members = take(each);
  uint32_t* pieces  = take(each);
  uint32_t* hlist   = take(hcap);
  auto* const rc    = reinterpret_cast<rs_counts*>(take(64));
  uint32_t* parent  = ws.label;

  zero_counters(ctx);
  KSPN_CUDA(cudaMemsetAsync(rc, 0, sizeof(rs_counts), s));
  uint32_t const words = (g.n + 31) / 32;
  unsigned const grid  = rs_grid(undecided); // passes over the list
  k_res_list<<<rs_grid(words), RS_THREADS, 0, s>>>(g.n, und, parent, count, list, &rc->list_n);
  k_res_hook<<<grid, RS_THREADS, 0, s>>>(list, &rc->list_n, und, g.fh, g.fc, parent, ws.ctr + CTR_ERR, hlist, ws.ctr + CTR_RES_HEAVY);
  if (g.m > HEAVY_ROW) {
    k_res_hook_heavy<<<std::min<unsigned>(148 * 8, grid * 8), RS_THREADS, 0, s>>>(und, g.fh, g.fc, parent, ws.ctr + CTR_ERR, hlist, ws.ctr + CTR_RES_HEAVY);
    ctx->launches += 1;
  }
  k_res_flatten<<<grid, RS_THREADS, 0, s>>>(list, &rc->list_n, parent, count, place, ws.ctr + CTR_ERR);
  k_res_ranges<<<grid, RS_THREADS, 0, s>>>(list, parent, count, start, pieces, static_cast<uint32_t>(each), rc, ws.ctr + CTR_AUX);
  k_res_members<<<grid, RS_THREADS, 0, s>>>(list, &rc->list_n, parent, start, place, members);
  k_res_small<<<std::min<unsigned>(148 * 8, rs_grid(undecided * 16)), RS_THREADS, 0, s>>>(rc, pieces, count, start, place, members, g.fh, g.fc, und, scc_id, ws.ctr + CTR_DECIDED, ws.ctr + CTR_AUX);
  if (undecided > 32) {
    k_res_block<<<static_cast<unsigned>(std::min<uint64_t>(148 * 6, undecided / 33 + 1)), RB_T, 0, s>>>(rc, pieces, static_cast<uint32_t>(each), count, start, place, members, g.fh, g.fc, und, scc_id,
                                                                                                       ws.ctr + CTR_DECIDED, ws.ctr + CTR_AUX);
    ctx->launches += 1;
  }
  KSPN_CHECK_LAUNCH();
  ctx->launches += 6;
  read_counters(ctx);
  if (ctx->h_ctr[CTR_ERR]) throw error{ KSPN_ERR_INTERNAL, "residual: union-find loop bound reached" };
  if (pieces_left) *pieces_left = ctx->h_ctr[CTR_AUX];
  return ctx->h_ctr[CTR_DECIDED];
}

} // namespace kspn
