// Searches of one block over a graph in its shared memory (16-bit ids, rows
// in both directions, state bitmaps): graphs that fit one SM (small.cu) and
// the residual step's pieces (residual.cu).
#pragma once

#include "kspn_internal.cuh"

namespace kspn {

namespace {

struct sm_shared
{
  unsigned long long best, edges;
  uint32_t           cnt[3][2]; // vertices appended by a level (in turn), per list
  uint32_t           bad, minid, decided, size; // size: the pivot's component
};

struct sm_graph
{
  uint32_t        n, words;
  uint32_t*       lab; // live degrees (in << 16 | out) while trimming, labels (priority << 16 | root) in a label round
  uint32_t *      und, *open, *vis, *inq;
  uint16_t *      q0, *q1;
  uint16_t const *fh, *bh, *fc, *bc;
  sm_shared*      S;
  uint32_t        level; // levels ended so far, modulo 3: S->cnt[level] counts the running one
};

__device__ __forceinline__ uint32_t
sm_bit(uint32_t const* map, uint32_t v)
{
  return (map[v >> 5] >> (v & 31)) & 1u;
}
__device__ __forceinline__ bool
sm_take(uint32_t* map, uint32_t v) // clears v's bit; true when this call cleared it
{
  uint32_t const b = 1u << (v & 31);
  return (atomicAnd(map + (v >> 5), ~b) & b) != 0;
}

// End of a level: the vertices it appended to either list.  One barrier: the
// counters of the level after next are zeroed once every thread has read them.
__device__ __forceinline__ uint2
sm_level_end(sm_graph& G)
{
  __syncthreads();
  uint2 const c = make_uint2(G.S->cnt[G.level][0], G.S->cnt[G.level][1]);
  if (threadIdx.x < 2) G.S->cnt[G.level ? G.level - 1 : 2][threadIdx.x] = 0;
  G.level = G.level == 2 ? 0 : G.level + 1;
  return c;
}

__device__ __forceinline__ void
sm_append(sm_graph const& G, uint32_t which, bool take, uint32_t v, uint16_t* out)
{
  unsigned const b = __ballot_sync(0xFFFFFFFFu, take);
  if (!b) return;
  unsigned const lane = threadIdx.x & 31u;
  uint32_t       at   = 0;
  if (lane == 0) at = atomicAdd(&G.S->cnt[G.level][which], __popc(b));
  at = __shfl_sync(0xFFFFFFFFu, at, 0);
  if (take) out[at + __popc(b & ((1u << lane) - 1))] = static_cast<uint16_t>(v);
}

// One list's share of a level, by the THREADS threads that tid numbers:
// prep(v) once for each of the cnt listed vertices, then visit(v, w) for every
// neighbour w; the w it takes are appended to out and counted in `which`.  A
// vertex gets 32 lanes in a thin level, down to four in a wide one, so that a
// thin level's rows are read side by side; a row too long for its lanes is
// read by the whole warp, so that a hub does not hold up a wide level.
constexpr uint32_t SM_LONG = 4; // entries per lane from which on a row is the warp's (R-MAT scale 13: 32: 85 us, 16: 76, 8: 74, 4: 71; never: 121)

template<int THREADS, class P, class F>
__device__ __forceinline__ uint32_t
sm_expand(sm_graph const& G, uint32_t tid, uint32_t which, uint16_t const* list, uint32_t cnt, uint16_t const* head, uint16_t const* rows, uint16_t* out, P prep, F visit)
{
  uint32_t s = 5;
  while (s > 2 && (cnt << s) > THREADS) --s; // (at least eight lanes: 97 instead of 86 us at n 8,000)
  unsigned const lane = threadIdx.x & 31u;
  uint32_t const sub = lane & ((1u << s) - 1), step = 1u << s;
  uint32_t       edges = 0;
  for (uint32_t i = tid >> s; __any_sync(0xFFFFFFFFu, i < cnt); i += THREADS >> s) {
    uint32_t v = 0, e = 0, end = 0;
    if (i < cnt) {
      v = list[i], e = head[v], end = head[v + 1];
      if (sub == 0) prep(v);
    }
    __syncwarp();
    unsigned wide = __ballot_sync(0xFFFFFFFFu, sub == 0 && end - e > (SM_LONG << s) && s < 5);
    bool const mine = !((wide >> (lane - sub)) & 1u);
    for (uint32_t x = e + sub; __any_sync(0xFFFFFFFFu, mine && x < end); x += step) {
      uint32_t w    = 0;
      bool     take = false;
      if (mine && x < end) {
        w    = rows[x];
        take = visit(v, w);
        ++edges;
      }
      sm_append(G, which, take, w, out);
    }
    for (; wide; wide &= wide - 1) {
      unsigned const l  = __ffs(wide) - 1;
      uint32_t const vl = __shfl_sync(0xFFFFFFFFu, v, l), x1 = __shfl_sync(0xFFFFFFFFu, end, l);
      for (uint32_t x = __shfl_sync(0xFFFFFFFFu, e, l) + lane; __any_sync(0xFFFFFFFFu, x < x1); x += 32) {
        uint32_t w    = 0;
        bool     take = false;
        if (x < x1) {
          w    = rows[x];
          take = visit(vl, w);
          ++edges;
        }
        sm_append(G, which, take, w, out);
      }
    }
  }
  return edges;
}

// The trim fixpoint over G.und: vertices decided (their id is set already).
template<int T>
__device__ uint32_t
sm_trim(sm_graph& G)
{
  // live degrees, four lanes per vertex
  unsigned const sub  = threadIdx.x & 3u;
  uint32_t const span = (G.n + 7) & ~7u;
  for (uint32_t i = threadIdx.x >> 2; i < span; i += T / 4) {
    bool const on  = i < G.n && sm_bit(G.und, i);
    uint32_t   deg = 0;
    if (!__any_sync(0xFFFFFFFFu, on)) continue;
    if (on) {
      for (uint32_t e = G.fh[i] + sub; e < G.fh[i + 1]; e += 4) deg += sm_bit(G.und, G.fc[e]);
      for (uint32_t e = G.bh[i] + sub; e < G.bh[i + 1]; e += 4) deg += sm_bit(G.und, G.bc[e]) << 16;
    }
    deg += __shfl_xor_sync(0xFFFFFFFFu, deg, 1);
    deg += __shfl_xor_sync(0xFFFFFFFFu, deg, 2);
    bool const first = on && sub == 0;
    if (first) G.lab[i] = deg;
    sm_append(G, 0, first && (!(deg & 0xFFFFu) || !(deg >> 16)), i, G.q0);
  }
  uint32_t lo = 0, hi = sm_level_end(G).x;
  for (uint32_t i = threadIdx.x; i < hi; i += T) sm_take(G.und, G.q0[i]); // (und does not change while degrees are counted)
  __syncthreads();
  // a level takes one degree from every undecided neighbour: out-rows by the
  // even warps, in-rows by the odd ones
  bool const     odd  = (threadIdx.x >> 5) & 1u;
  uint32_t const tid  = (threadIdx.x >> 6) * 32 + (threadIdx.x & 31u);
  uint32_t const unit = odd ? 1u : 1u << 16, part = odd ? 0xFFFFu : 0xFFFF0000u;
  while (lo < hi) {
    sm_expand<T / 2>(
      G, tid, 0, G.q0 + lo, hi - lo, odd ? G.bh : G.fh, odd ? G.bc : G.fc, G.q0 + hi, [](uint32_t) {},
      [&](uint32_t, uint32_t w) { return sm_bit(G.und, w) && (atomicSub(G.lab + w, unit) & part) == unit && sm_take(G.und, w); });
    lo = hi;
    hi += sm_level_end(G).x;
  }
  return hi;
}

// v's rank in round r: a permutation of the 16-bit ids
__device__ __forceinline__ uint32_t
sm_priority(uint32_t v, uint32_t r)
{
  uint32_t x = (v + r * 0x3D4Du) & 0xFFFFu;
  x          = (x * 0x9E3Bu) & 0xFFFFu;
  x ^= x >> 7;
  x = (x * 0xC2B3u) & 0xFFFFu;
  return x ^ (x >> 9);
}

// One min-label search from every undecided vertex; decides at least the
// component of the least priority.  name(v): v's vertex id in ids, where every
// vertex's id is its own name so far.
template<int T, class N>
__device__ uint32_t
sm_label_round(sm_graph& G, uint32_t round, uint32_t* __restrict__ ids, N name, uint32_t& edges)
{
  unsigned const lane = threadIdx.x & 31u;
  uint32_t const span = G.words * 32;
  for (uint32_t v = threadIdx.x; v < span; v += T) {
    uint32_t const word = G.und[v >> 5];
    bool const     on   = (word >> (v & 31)) & 1u;
    if (lane == 0) G.inq[v >> 5] = word, G.open[v >> 5] = word;
    if (on) G.lab[v] = sm_priority(v, round) << 16 | v;
    sm_append(G, 0, on, v, G.q0);
  }
  uint32_t  cnt = sm_level_end(G).x;
  uint16_t *in = G.q0, *out = G.q1;
  while (cnt) {
    // a vertex leaves the queue before its label is read: a label that drops
    // later queues it again
    edges += sm_expand<T>(
      G, threadIdx.x, 0, in, cnt, G.fh, G.fc, out,
      [&](uint32_t v) {
        sm_take(G.inq, v);
        __threadfence_block();
      },
      [&](uint32_t v, uint32_t w) {
        if (!sm_bit(G.und, w)) return false;
        uint32_t const label = *static_cast<uint32_t volatile*>(G.lab + v);
        if (atomicMin(G.lab + w, label) <= label) return false;
        __threadfence_block();
        uint32_t const b = 1u << (w & 31);
        return !(atomicOr(G.inq + (w >> 5), b) & b);
      });
    cnt               = sm_level_end(G).x;
    uint16_t* const t = in;
    in                = out;
    out               = t;
  }
  // roots keep their own label; backward from all of them inside their label
  for (uint32_t v = threadIdx.x; v < span; v += T) {
    bool const root = v < G.n && sm_bit(G.und, v) && (G.lab[v] & 0xFFFFu) == v;
    if (root) sm_take(G.open, v);
    sm_append(G, 0, root, v, G.q0);
  }
  uint32_t const roots = sm_level_end(G).x;
  uint32_t       lo = 0, members = roots;
  while (lo < members) {
    edges += sm_expand<T>(
      G, threadIdx.x, 0, G.q0 + lo, members - lo, G.bh, G.bc, G.q0 + members, [](uint32_t) {},
      [&](uint32_t v, uint32_t w) { return sm_bit(G.open, w) && G.lab[v] == G.lab[w] && sm_take(G.open, w); });
    lo = members;
    members += sm_level_end(G).x;
  }
  // the smallest member names a component; the root's id holds the minimum
  for (uint32_t i = roots + threadIdx.x; i < members; i += T) atomicMin(ids + name(G.lab[G.q0[i]] & 0xFFFFu), name(G.q0[i]));
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < members; i += T) {
    uint32_t const v = G.q0[i];
    if (i >= roots) ids[name(v)] = __ldcg(ids + name(G.lab[v] & 0xFFFFu));
    sm_take(G.und, v);
  }
  __syncthreads();
  return members;
}

} // namespace

} // namespace kspn
