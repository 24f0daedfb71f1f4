// cm_match.cuh -- device side of the deterministic matching: candidates and their
// order, proposals, row scans (cm_match.cu describes the scheme).
#pragma once

#include <climits>

#include "cm_ctx.h"

// Rows of at most kSerialDeg entries are scanned by one lane, longer rows in
// kMatchChunk-entry warp work items (tuning parameters, set through the build).
#ifndef CM_SERIAL_DEG
#define CM_SERIAL_DEG 16
#endif
#ifndef CM_MATCH_CHUNK
#define CM_MATCH_CHUNK 256
#endif
namespace cm {
namespace {

constexpr int kSerialDeg = CM_SERIAL_DEG;
constexpr int kMatchChunk = CM_MATCH_CHUNK;
static_assert(kSerialDeg == 8 || kSerialDeg == 16, "CM_SERIAL_DEG: 8 or 16");
static_assert(kMatchChunk == 128 || kMatchChunk == 256 || kMatchChunk == 512, "CM_MATCH_CHUNK: 128, 256 or 512");
constexpr int kTop = 4;          // listed candidates per vertex
constexpr int kNone = -1;        // list slot: no further candidate
constexpr int kUnknown = -3;     // list slot not computed (more candidates may exist)

struct Slot {      // rows to scan in one round
  int *big_base, *big_done;  // per row: first chunk, chunks done
  int4 *desc;      // per chunk: (vertex, first entry, end entry, row index or -1 if one chunk)
};

struct MatchArgs {
  int n, span;                   // span: vertices a warp takes at a time (multiple of 32, at most kSpan)
  const int *xadj, *adjncy, *adjwgt, *vwgt;
  long long maxvwgt;
  int *m2;                       // the matching (output)
  unsigned long long *best;      // best proposal received: (weight, proposer), 0 = none (best_key)
  int *top, *topw;               // kTop listed candidates per vertex: ids, weights
  Slot slot[2];
  unsigned long long *big;       // [3] = (rows << 32 | chunks) of the slots, by round
  int *tick;                     // [3] work tickets of the round kernel, by round
  int *vmax;                     // largest vertex weight (zeroed before the launch)
  int *odd;                      // [8]: an offer was not returned; blocks of k_match_finish done; handshake_rounds' counters
  int *part;                     // per chunk: kTop x (w, h, k)
  long long max_rounds;
  DevStatus *st;
  unsigned long long *trace;     // optional: row 0 header, row r+1 = round r
  int trace_rows;
  // Several independent graphs side by side (a batch): vgid[v] = v's graph,
  // whose weight cap is gcap[g] and whose first vertex is gbase[g] (the edge
  // hash of the tie rule is taken on graph-local ids, so a graph matches the
  // same alone and in a batch).  Null for one graph.
  const int *vgid, *gbase, *gcap;
};

// Candidates.  Lex mode (ties to the lower id) packs (weight, ~id) into one
// 64-bit key, larger = better, 0 = none.  Hash mode has (weight desc, edge hash
// asc) in the key and the id, which decides between equal keys, beside it.
template <bool H> struct Cand;
template <> struct Cand<false> {
  unsigned long long key = 0ull;
  __device__ __forceinline__ static Cand make(int v, int k, int w, int hb) {
    (void)v;
    (void)hb;
    Cand c;
    c.key = ((unsigned long long)((unsigned)w ^ 0x80000000u) << 32) | (unsigned)(~(unsigned)k);
    return c;
  }
  __device__ __forceinline__ bool valid() const { return key != 0ull; }
  __device__ __forceinline__ int id() const { return valid() ? (int)~(unsigned)key : -1; }
  __device__ __forceinline__ int weight() const { return (int)((unsigned)(key >> 32) ^ 0x80000000u); }
  __device__ __forceinline__ bool better(const Cand &o) const { return key > o.key; }
  __device__ __forceinline__ bool same(const Cand &o) const { return key == o.key; }
  __device__ __forceinline__ Cand warp_best() const {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
    Cand r;
    r.key = ((unsigned long long)hi << 32) | lo;
    return r;
  }
  // p: 16-byte aligned slot of kPartInts ints
  __device__ __forceinline__ void store(int *p) const { *reinterpret_cast<unsigned long long *>(p) = key; }
  __device__ __forceinline__ static Cand load(const int *p) {
    Cand c;
    c.key = __ldcg(reinterpret_cast<const unsigned long long *>(p));
    return c;
  }
};
template <> struct Cand<true> {
  unsigned long long key = 0ull;  // (weight, ~hash), larger = better
  int k = INT_MAX;                // INT_MAX = none
  __device__ __forceinline__ static Cand make(int v, int k, int w, int hb) {
    Cand c;
    const unsigned h = edge_hash((unsigned)(min(v, k) - hb), (unsigned)(max(v, k) - hb));
    c.key = ((unsigned long long)((unsigned)w ^ 0x80000000u) << 32) | (unsigned)~h;
    c.k = k;
    return c;
  }
  __device__ __forceinline__ bool valid() const { return k != INT_MAX; }
  __device__ __forceinline__ int id() const { return valid() ? k : -1; }
  __device__ __forceinline__ int weight() const { return (int)((unsigned)(key >> 32) ^ 0x80000000u); }
  __device__ __forceinline__ bool better(const Cand &o) const { return key > o.key || (key == o.key && k < o.k); }
  __device__ __forceinline__ bool same(const Cand &o) const { return key == o.key && k == o.k; }
  __device__ __forceinline__ Cand warp_best() const {
    const unsigned full = 0xffffffffu;
    const unsigned hi = __reduce_max_sync(full, (unsigned)(key >> 32));
    const bool top = (unsigned)(key >> 32) == hi;
    const unsigned lo = __reduce_max_sync(full, top ? (unsigned)key : 0u);
    Cand r;
    r.key = ((unsigned long long)hi << 32) | lo;
    r.k = __reduce_min_sync(full, key == r.key ? k : INT_MAX);
    return r;
  }
  __device__ __forceinline__ void store(int *p) const {
    *reinterpret_cast<int4 *>(p) = make_int4((int)(unsigned)(key >> 32), (int)(unsigned)key, k, 0);
  }
  __device__ __forceinline__ static Cand load(const int *p) {
    const int4 x = __ldcg(reinterpret_cast<const int4 *>(p));
    Cand c;
    c.key = ((unsigned long long)(unsigned)x.x << 32) | (unsigned)x.y;
    c.k = x.z;
    return c;
  }
};
constexpr int kPartInts = 4;  // ints per stored candidate slot (16 bytes, one vector access)

// Sorted (best first) list of up to KK candidates held in registers.
template <bool H, int KK>
struct TopK {
  Cand<H> c[KK];
  __device__ __forceinline__ void insert(const Cand<H> &x) {
    if (!x.better(c[KK - 1])) return;
    Cand<H> cur = x;
#pragma unroll
    for (int i = 0; i < KK; ++i) {
      if (cur.better(c[i])) { Cand<H> t = c[i]; c[i] = cur; cur = t; }
    }
  }
  // Edge (v, k) of weight w.  In hash mode the edge hash is computed only when
  // the weight can still enter the list (a lighter edge loses to the last
  // entry whatever its hash); the result is that of insert(make(v, k, w, hb)).
  // hb: the first vertex of v's graph (0 for one graph).
  __device__ __forceinline__ void insert_edge(int v, int k, int w, int hb) {
    if constexpr (H) {
      if (c[KK - 1].valid() && w < c[KK - 1].weight()) return;
    }
    insert(Cand<H>::make(v, k, w, hb));
  }
};

// First vertex of v's graph (the hash base of the tie rule) and its weight cap.
__device__ __forceinline__ int hash_base(const MatchArgs &a, int v) { return a.vgid ? __ldg(a.gbase + __ldg(a.vgid + v)) : 0; }
__device__ __forceinline__ long long weight_cap(const MatchArgs &a, int v) {
  return a.vgid ? (long long)__ldg(a.gcap + __ldg(a.vgid + v)) : a.maxvwgt;
}

// The pair (v, k) may match: both fit the cap and one of them is light.
__device__ __forceinline__ bool pair_fits(long long cap, long long vw, long long vk) {
  return vw + vk <= cap && (3 * vw < cap || 3 * vk < cap);
}

// Even the two heaviest vertices may pair and are light: every edge is
// eligible, and the scans skip the neighbours' weights.
__device__ __forceinline__ bool all_eligible(const MatchArgs &a) {
  const long long vmax = __ldcg(a.vmax);
  return 2 * vmax <= a.maxvwgt && 3 * vmax < a.maxvwgt;
}

// A proposal by v over an edge of weight w, as best[] holds it: 0 is none (the
// low half, ~v, is never 0).  Between different weights, and among equal
// weights with ties to the lower id, the larger key is the better proposal.
__device__ __forceinline__ unsigned long long best_key(int v, int w) {
  return ((unsigned long long)((unsigned)w ^ 0x80000000u) << 32) | (unsigned)~(unsigned)v;
}
__device__ __forceinline__ int best_holder(unsigned long long b) { return b == 0ull ? -1 : (int)~(unsigned)b; }
// Whether v and h hold each other's proposals, over entries of equal weight.  With
// every pair so, no two vertices prefer each other to their partners, each by its
// own row: v's proposal was refused for a better one, whose weight the row of the
// vertex that refused holds too.  The matching is then that of mutual proposals,
// whatever the other entries are.
__device__ __forceinline__ bool best_mutual(unsigned long long bv, unsigned long long bh, int v) {
  return best_holder(bh) == v && (bv >> 32) == (bh >> 32);
}
__device__ __forceinline__ unsigned long long ld_best(const MatchArgs &a, int k) { return ld_fresh(a.best + k); }

// v's proposal (key) to c beats the proposal b that c holds.
template <bool H>
__device__ __forceinline__ bool beats(unsigned long long key, unsigned long long b, int v, int c, int hb) {
  if constexpr (H) {
    if (b == 0ull) return true;
    if ((key >> 32) != (b >> 32)) return key > b;
    const int s = best_holder(b);
    const unsigned hv = edge_hash((unsigned)(min(v, c) - hb), (unsigned)(max(v, c) - hb));
    const unsigned hs = edge_hash((unsigned)(min(s, c) - hb), (unsigned)(max(s, c) - hb));
    return hv != hs ? hv < hs : v < s;
  } else {
    return key > b;
  }
}

// v offers itself to c over an edge of weight w.  Returns whether c took it;
// *out = the vertex c gave up for it (-1: none).  `seen`: a recent value of
// best[c] (any value is allowed; a right one saves a memory trip).
template <bool H>
__device__ __forceinline__ bool offer(const MatchArgs &a, int v, int c, int w, unsigned long long seen, int hb,
                                      int *out) {
  const unsigned long long key = best_key(v, w);
  if constexpr (H) {
    for (;;) {  // every turn best[c] has improved since the last
      const unsigned long long old = atomicCAS(a.best + c, seen, key);
      if (old == seen) break;
      if (!beats<H>(key, old, v, c, hb)) return false;
      seen = old;
    }
    *out = best_holder(seen);
  } else {
    const unsigned long long old = atomicMax(a.best + c, key);
    if (old >= key) return false;
    *out = best_holder(old);
  }
  return true;
}

// Merges the lanes' sorted lists into the warp's best KK (all lanes get it).
template <bool H, int KK>
__device__ __forceinline__ TopK<H, KK> warp_topk(const TopK<H, KK> &t) {
  TopK<H, KK> out;
  int head = 0;
#pragma unroll
  for (int i = 0; i < KK; ++i) {
    Cand<H> mine;
#pragma unroll
    for (int j = 0; j < KK; ++j)
      if (j == head) mine = t.c[j];
    const Cand<H> win = mine.warp_best();
    out.c[i] = win;
    if (win.valid() && mine.same(win)) ++head;
  }
  return out;
}

// The warp's best KK of the cnt candidates stored at slots slot(t), t < cnt,
// of the chunk partial lists (four loads in flight per lane).
template <bool H, int KK, typename F>
__device__ __forceinline__ TopK<H, KK> merge_parts(const MatchArgs &a, int cnt, F slot) {
  const int lane = threadIdx.x & 31;
  TopK<H, KK> acc;
  for (int t0 = lane; t0 < cnt; t0 += 128) {
    Cand<H> c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = t0 + 32 * i;
      if (t < cnt) c[i] = Cand<H>::load(a.part + slot(t) * kPartInts);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) acc.insert(c[i]);
  }
  return warp_topk(acc);
}

// Loads entries [b, e) (e - b <= kMatchChunk) of v's row, slot u of a lane entry
// b + lane + 32 u, all loads issued before any is used, and marks with
// k[u] = -1 those that are no candidates: the vertex itself, pairs that do not
// fit (`all`: every pair fits), and neighbours that hold a proposal v cannot
// beat: by its weight alone (kWeak), or at all (kExact); or those matched (kOpen,
// for the handshakes).
enum : int { kStatic = 0, kWeak = 1, kExact = 2, kOpen = 3 };
template <bool H, int FILTER>
__device__ __forceinline__ void load_entries(const MatchArgs &a, int v, int b, int e, bool all, int hb,
                                             int (&k)[kMatchChunk / 32], int (&w)[kMatchChunk / 32]) {
  const int lane = threadIdx.x & 31;
  constexpr int U = kMatchChunk / 32;
  const int nu = (e - b + 31) >> 5;  // slots holding entries (warp-uniform): the others are skipped
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int j = b + lane + 32 * u;
    k[u] = -1;
    w[u] = 0;
    if (u < nu && j < e) {
      k[u] = a.adjncy[j];
      w[u] = a.adjwgt[j];
    }
  }
  if (!all) {
    const long long vw = a.vwgt[v], cap = weight_cap(a, v);
    int vk[U];
#pragma unroll
    for (int u = 0; u < U; ++u) vk[u] = (u < nu && k[u] >= 0) ? a.vwgt[k[u]] : 0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (!pair_fits(cap, vw, vk[u])) k[u] = -1;
  }
  if constexpr (FILTER == kWeak) {
    unsigned bw[U];  // the weight half of best[]; 0 for none
#pragma unroll
    for (int u = 0; u < U; ++u)
      bw[u] = (u < nu && k[u] >= 0) ? ld_fresh(reinterpret_cast<const unsigned *>(a.best + k[u]) + 1) : 0u;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (((unsigned)w[u] ^ 0x80000000u) < bw[u]) k[u] = -1;
  }
  if constexpr (FILTER == kOpen) {
    int mk[U];
#pragma unroll
    for (int u = 0; u < U; ++u) mk[u] = (u < nu && k[u] >= 0) ? ld_fresh(a.m2 + k[u]) : 0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (mk[u] >= 0) k[u] = -1;
  }
  if constexpr (FILTER == kExact) {
    unsigned long long bk[U];
#pragma unroll
    for (int u = 0; u < U; ++u) bk[u] = (u < nu && k[u] >= 0) ? ld_best(a, k[u]) : 0ull;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < nu && k[u] >= 0 && !beats<H>(best_key(v, w[u]), bk[u], v, k[u], hb)) k[u] = -1;
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (k[u] == v) k[u] = -1;
}

// How a chain, or a span's chains, ended.
enum ChainEnd : int {
  kChainDone = 0,
  kChainFailed = 1,  // CM_ERR_LIMIT recorded
  kChainLong = 2,    // the steps allowed are used up (k_levels)
};

// Chains end by themselves: every accepted offer improves some best[], at most once
// for every entry of the graph.  A path whose weights grow from one end to the other
// makes one chain of n / 2 dependent steps (8 M vertices: 3 s), so a chain has no
// limit on its length.  What could only be a fault has one: a refusal means that
// the neighbour holds a better proposal for good, so a vertex is refused at most
// once per entry of its row before it is taken or has no candidate left.
constexpr int kLaneRefusals = kSerialDeg + kTop, kWarpRefusals = kMatchChunk + kTop;

// Where other warps wait for a chain at a grid barrier, whose wait has a limit, a
// warp takes at most kChainSteps accepted offers a round (about 0.1 s) and queues
// the vertex that is free then for the next round.
#ifndef CM_CHAIN_STEPS
#define CM_CHAIN_STEPS 65536
#endif
constexpr unsigned kChainSteps = CM_CHAIN_STEPS;

// The warp's best KK candidates over entries [b, e), e - b <= 64, of v's row, among
// those that FILTER leaves (kWeak: as kExact); every lane gets the list.
template <bool H, int KK, int FILTER>
__device__ __forceinline__ TopK<H, KK> pair_best(const MatchArgs &a, int v, int b, int e, bool all, int hb) {
  const int lane = threadIdx.x & 31, j0 = b + lane, j1 = j0 + 32;
  int k0 = -1, k1 = -1, w0 = 0, w1 = 0;
  if (j0 < e) {
    k0 = a.adjncy[j0];
    w0 = a.adjwgt[j0];
  }
  if (j1 < e) {
    k1 = a.adjncy[j1];
    w1 = a.adjwgt[j1];
  }
  if (k0 == v) k0 = -1;
  if (k1 == v) k1 = -1;
  if (!all) {
    const long long vw = a.vwgt[v], cap = weight_cap(a, v);
    const int x0 = k0 >= 0 ? a.vwgt[k0] : 0, x1 = k1 >= 0 ? a.vwgt[k1] : 0;
    if (!pair_fits(cap, vw, x0)) k0 = -1;
    if (!pair_fits(cap, vw, x1)) k1 = -1;
  }
  if (FILTER == kOpen) {
    if (k0 >= 0 && ld_fresh(a.m2 + k0) >= 0) k0 = -1;
    if (k1 >= 0 && ld_fresh(a.m2 + k1) >= 0) k1 = -1;
  } else if (FILTER != kStatic) {
    const unsigned long long y0 = k0 >= 0 ? ld_best(a, k0) : 0ull, y1 = k1 >= 0 ? ld_best(a, k1) : 0ull;
    if (k0 >= 0 && !beats<H>(best_key(v, w0), y0, v, k0, hb)) k0 = -1;
    if (k1 >= 0 && !beats<H>(best_key(v, w1), y1, v, k1, hb)) k1 = -1;
  }
  Cand<H> c0, c1;
  if (k0 >= 0) c0 = Cand<H>::make(v, k0, w0, hb);
  if (k1 >= 0) c1 = Cand<H>::make(v, k1, w1, hb);
  if (c1.better(c0)) {
    const Cand<H> t = c0;
    c0 = c1;
    c1 = t;
  }
  TopK<H, KK> out;
#pragma unroll
  for (int i = 0; i < KK; ++i) {
    const Cand<H> win = c0.warp_best();
    out.c[i] = win;
    if (!win.valid()) break;
    if (c0.same(win)) {
      c0 = c1;
      c1 = Cand<H>();
    }
    if (c0.same(win)) c0 = Cand<H>();  // the lane's second entry is the same parallel edge
  }
  return out;
}

// The warp's best KK candidates over entries [b, e) (e - b <= kMatchChunk) of v's
// row; every lane gets the list.  Hash order: most entries are lighter than the
// chunk's KK-th heaviest eligible entry and can never enter the list, so a
// weight threshold W is found first and only entries of weight >= W get an edge
// hash and a full comparison.  W is the KK-th largest of the lanes' heaviest
// eligible weights, so at least KK entries weigh >= W and the chunk's best KK
// are all among them (a list of the KK heaviest weights per lane gives a slightly
// higher W for eight times the instructions: R-MAT 22's matching 1937 against
// 1891 us).  The
// qualifying entries (usually KK, a few more and the ties at W) are packed one
// per lane through the warp's 32-entry buffer wbuf; more than 32 of them (many
// equal weights) take the per-lane lists instead.
template <bool H, int KK, int FILTER>
__device__ __forceinline__ TopK<H, KK> chunk_best(const MatchArgs &a, int v, int b, int e, bool all, int2 *wbuf) {
  constexpr int U = kMatchChunk / 32;
  const int nu = (e - b + 31) >> 5;
  const int hb = hash_base(a, v);
  // Rows and last chunks of up to 64 entries (most of a skewed graph's): two
  // entries a lane, every one compared in full, against a proposal too.
  if (nu <= 2) return pair_best<H, KK, FILTER>(a, v, b, e, all, hb);
  int k[U], w[U];
  load_entries<H, FILTER>(a, v, b, e, all, hb, k, w);
  if constexpr (!H) {
    (void)wbuf;
    TopK<H, KK> t;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < nu && k[u] >= 0) t.insert_edge(v, k[u], w[u], hb);
    return warp_topk(t);
  } else {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int top = INT_MIN;
    bool has = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;
      if (k[u] >= 0) {
        top = max(top, w[u]);
        has = true;
      }
    }
    // the lanes' heaviest in descending order until KK are taken; with fewer
    // lanes than that every eligible entry qualifies
    int W = INT_MIN, taken = 0;
#pragma unroll
    for (int r = 0; r < KK; ++r) {
      if (!__ballot_sync(full, has)) {
        W = INT_MIN;
        break;
      }
      W = __reduce_max_sync(full, has ? top : INT_MIN);
      const bool pop = has && top == W;
      taken += __popc(__ballot_sync(full, pop));
      has = has && !pop;
      if (taken >= KK) break;
    }
    int total = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;
      total += __popc(__ballot_sync(full, k[u] >= 0 && w[u] >= W));
    }
    TopK<H, KK> out;
    if (total > 32) {
      TopK<H, KK> t;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < nu && k[u] >= 0 && w[u] >= W) t.insert_edge(v, k[u], w[u], hb);
      out = warp_topk(t);
    } else {
      const unsigned below = (1u << lane) - 1u;
      int base = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (u >= nu) break;
        const bool q = k[u] >= 0 && w[u] >= W;
        const unsigned bal = __ballot_sync(full, q);
        if (q) wbuf[base + __popc(bal & below)] = make_int2(k[u], w[u]);
        base += __popc(bal);
      }
      __syncwarp();
      Cand<H> mine;
      if (lane < total) {
        const int2 x = wbuf[lane];
        mine = Cand<H>::make(v, x.x, x.y, hb);
      }
      __syncwarp();  // the buffer is free for the warp's next chunk
#pragma unroll
      for (int i = 0; i < KK; ++i) {
        const Cand<H> win = mine.warp_best();
        out.c[i] = win;
        if (win.valid() && mine.same(win)) mine = Cand<H>();
      }
    }
    // Identical entries (parallel edges of equal weight) count once in the
    // list but each in `taken`: a list left short although lighter entries
    // may exist is recomputed over every eligible entry, so that a short list
    // still means "no other candidate".
    if (W != INT_MIN && !out.c[KK - 1].valid()) {
      TopK<H, KK> t;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < nu && k[u] >= 0) t.insert_edge(v, k[u], w[u], hb);
      out = warp_topk(t);
    }
    return out;
  }
}

// Writes v's list.  A list of fewer than KK candidates holds them all; a full
// one of fewer than kTop slots ends with kUnknown.
template <bool H, int KK>
__device__ __forceinline__ void store_top(const MatchArgs &a, int v, const TopK<H, KK> &t) {
  int q[kTop], w[kTop];
#pragma unroll
  for (int i = 0; i < kTop; ++i) {
    const Cand<H> &c = t.c[i < KK ? i : KK - 1];
    q[i] = i < KK ? c.id() : (c.valid() ? kUnknown : kNone);
    w[i] = c.weight();
  }
  reinterpret_cast<int4 *>(a.top)[v] = make_int4(q[0], q[1], q[2], q[3]);
  reinterpret_cast<int4 *>(a.topw)[v] = make_int4(w[0], w[1], w[2], w[3]);
}

// A vertex's candidates, most preferred first, and the next one to offer to.
// Two of three candidates have a better proposal by the time they are reached,
// so the proposals that all of them hold are read together (check) and the
// first candidate that would take the vertex is offered to with one atomic.
struct List {
  int id[kTop], w[kTop];          // slot 0 is next; kNone: no other candidate, kUnknown: the list is used up
  unsigned long long seen[kTop];  // recent best[id]
  __device__ __forceinline__ void load(const MatchArgs &a, int v) {
    const int4 q = reinterpret_cast<const int4 *>(a.top)[v], x = reinterpret_cast<const int4 *>(a.topw)[v];
    id[0] = q.x; id[1] = q.y; id[2] = q.z; id[3] = q.w;
    w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
  }
  __device__ __forceinline__ void drop() {  // the next candidate
#pragma unroll
    for (int t = 0; t + 1 < kTop; ++t) {
      id[t] = id[t + 1];
      w[t] = w[t + 1];
      seen[t] = seen[t + 1];
    }
    id[kTop - 1] = kUnknown;
  }
  // Drops the candidates up to c: all when c is not listed (it came from a rescan).
  __device__ __forceinline__ void after(int c) {
    bool found = false;
#pragma unroll
    for (int t = 0; t < kTop; ++t)
      if (!found) {
        found = id[0] == c;
        drop();
      }
  }
  // Reads the candidates' proposals and drops those v does not beat up to the first that it does.
  template <bool H>
  __device__ __forceinline__ void check(const MatchArgs &a, int v, int hb) {
#pragma unroll
    for (int t = 0; t < kTop; ++t) seen[t] = id[t] >= 0 ? ld_best(a, id[t]) : 0ull;
    bool go = true;
#pragma unroll
    for (int t = 0; t < kTop; ++t) {
      go = go && id[0] >= 0 && !beats<H>(best_key(v, w[0]), seen[0], v, id[0], hb);
      if (go) drop();
    }
  }
};

__device__ __forceinline__ unsigned long long warp_excl_scan_u64(unsigned long long v, unsigned long long *total) {
  const unsigned long long inc = warp_inclusive_scan_u64(v);
  *total = __shfl_sync(0xffffffffu, inc, 31);
  return inc - v;
}

// Chunk descriptors of the rows queued by the lanes with `take` set (row x of
// deg entries from xs, nch chunks from desc[cb], row index idx): a one-chunk
// row's lane writes its descriptor, and the warp writes each longer row's
// descriptors together.  Convergent.
__device__ __forceinline__ void write_descs(int4 *desc, bool take, int x, int xs, int deg, int nch, int idx, int cb) {
  const int lane = threadIdx.x & 31;
  if (take && nch == 1) desc[cb] = make_int4(x, xs, xs + deg, -1);
  unsigned bm = __ballot_sync(0xffffffffu, take && nch > 1);
  while (bm) {
    const int src = __ffs(bm) - 1;
    bm &= bm - 1;
    const int rx = __shfl_sync(0xffffffffu, x, src), rs = __shfl_sync(0xffffffffu, xs, src);
    const int rd = __shfl_sync(0xffffffffu, deg, src), rn = __shfl_sync(0xffffffffu, nch, src);
    const int ri = __shfl_sync(0xffffffffu, idx, src), rc = __shfl_sync(0xffffffffu, cb, src);
    for (int j = lane; j < rn; j += 32)
      desc[rc + j] = make_int4(rx, rs + j * kMatchChunk, min(rs + rd, rs + (j + 1) * kMatchChunk), ri);
  }
}

// Queues x (row of deg > 0 entries starting at xs) for a scan: slot `par`,
// counter `ctr`; convergent.
__device__ __forceinline__ void append_scan(const MatchArgs &a, int par, int ctr, bool take, int x, int xs, int deg) {
  if (!__any_sync(0xffffffffu, take)) return;
  const Slot &S = a.slot[par];
  const int lane = threadIdx.x & 31;
  const int nch = take ? (deg + kMatchChunk - 1) / kMatchChunk : 0;
  const unsigned long long mine = take ? ((1ull << 32) | (unsigned long long)nch) : 0ull;
  unsigned long long tot;
  const unsigned long long ex = warp_excl_scan_u64(mine, &tot);
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(a.big + ctr, tot);
  base = __shfl_sync(0xffffffffu, base, 0) + ex;
  const int idx = (int)(base >> 32), cb = (int)(base & 0xffffffffu);
  if (take) {
    S.big_base[idx] = cb;
    S.big_done[idx] = 0;
  }
  write_descs(S.desc, take, x, xs, deg, nch, idx, cb);
}

// Stores a chunk's list among the row's partial lists; true for the warp of
// the row's last chunk (d: the chunk's descriptor, q its index).
template <bool H, int KK>
__device__ __forceinline__ bool part_done(const MatchArgs &a, const Slot &S, int q, const int4 &d, int nch,
                                          const TopK<H, KK> &r) {
  const int lane = threadIdx.x & 31;
  if (lane < KK) {
    Cand<H> mine = r.c[0];
#pragma unroll
    for (int t = 1; t < KK; ++t)
      if (lane == t) mine = r.c[t];
    mine.store(a.part + ((size_t)q * kTop + lane) * kPartInts);
    __threadfence();
  }
  __syncwarp();
  int last = 0;
  if (lane == 0) last = atomicAdd(S.big_done + d.w, 1) == nch - 1;
  last = __shfl_sync(0xffffffffu, last, 0);
  if (last) __threadfence();
  return last != 0;
}

// The list of a short row (deg <= kSerialDeg), by one lane: from the weights and
// the cap alone.
template <bool H>
__device__ __forceinline__ void short_list(const MatchArgs &a, int v, int xs, int deg) {
  constexpr int kHalf = 8;
  const int hb = hash_base(a, v);
  const long long vw = a.vwgt[v], cap = weight_cap(a, v);
  TopK<H, kTop> tk;
#pragma unroll 1
  for (int t0 = 0; t0 < deg; t0 += kHalf) {  // 8 entries in flight
    int k[kHalf], w[kHalf], vk[kHalf];
#pragma unroll
    for (int t = 0; t < kHalf; ++t) {
      k[t] = t0 + t < deg ? a.adjncy[xs + t0 + t] : -1;
      w[t] = t0 + t < deg ? a.adjwgt[xs + t0 + t] : 0;
    }
#pragma unroll
    for (int t = 0; t < kHalf; ++t) vk[t] = k[t] >= 0 ? a.vwgt[k[t]] : 0;
#pragma unroll
    for (int t = 0; t < kHalf; ++t)
      if (k[t] >= 0 && k[t] != v && pair_fits(cap, vw, vk[t])) tk.insert_edge(v, k[t], w[t], hb);
  }
  store_top(a, v, tk);
}

// Best candidate of a short row (deg <= kSerialDeg) that takes v now, by one
// lane, AHEAD entries at a time; *seen = the proposal it holds.  -1: none.
template <bool H, int AHEAD>
__device__ __forceinline__ int rescan_short(const MatchArgs &a, int v, int xs, int deg, bool all, int hb, int *weight,
                                            unsigned long long *seen) {
  constexpr int kHalf = AHEAD;
  const long long vw = all ? 0 : a.vwgt[v], cap = all ? 0 : weight_cap(a, v);
  TopK<H, 1> t1;
  *seen = 0ull;
#pragma unroll 1
  for (int t0 = 0; t0 < deg; t0 += kHalf) {
    int k[kHalf], w[kHalf];
    unsigned long long b[kHalf];
#pragma unroll
    for (int t = 0; t < kHalf; ++t) {
      k[t] = t0 + t < deg ? a.adjncy[xs + t0 + t] : -1;
      w[t] = t0 + t < deg ? a.adjwgt[xs + t0 + t] : 0;
    }
#pragma unroll
    for (int t = 0; t < kHalf; ++t) b[t] = k[t] >= 0 ? ld_best(a, k[t]) : 0ull;
    if (!all) {
      int vk[kHalf];
#pragma unroll
      for (int t = 0; t < kHalf; ++t) vk[t] = k[t] >= 0 ? a.vwgt[k[t]] : 0;
#pragma unroll
      for (int t = 0; t < kHalf; ++t)
        if (!pair_fits(cap, vw, vk[t])) k[t] = -1;
    }
#pragma unroll
    for (int t = 0; t < kHalf; ++t) {
      if (k[t] < 0 || k[t] == v || (t1.c[0].valid() && w[t] < t1.c[0].weight())) continue;
      const Cand<H> c = Cand<H>::make(v, k[t], w[t], hb);
      if (c.better(t1.c[0]) && beats<H>(best_key(v, w[t]), b[t], v, k[t], hb)) {
        t1.c[0] = c;
        *seen = b[t];
      }
    }
  }
  *weight = t1.c[0].weight();
  return t1.c[0].id();
}

// One warp, one lane a vertex of [b0, b0 + span): offers the vertex to its
// candidates in order and goes on with whomever a taker gives up, until nobody
// is left without a proposal or the free vertex needs a scan of a long row: the
// lane then hands it to queue(v, row start, entries), which all lanes call (v =
// -1: nothing).  A lane whose chain has ended takes the span's next vertex.
// list: span ints of the warp's shared memory.  AHEAD: a candidate most likely
// gives up the vertex it was seen to hold, and that one's list is read while the
// offer is under way: it pays where chains are long (low-id ties on a 700 x 700
// triangulation 3.21 -> 2.95 ms), and costs reads and registers where the chip is
// full (hashed ties, R-MAT 22: +0.08 ms).  SCAN: entries of a rescan in flight.
// BOUNDED: every turn takes one of *steps, and without any left the warp gives up
// (kChainLong).
template <bool H, bool AHEAD, int SCAN, bool BOUNDED, typename Q>
__device__ __forceinline__ ChainEnd propose_span(const MatchArgs &a, long long b0, int span, bool all, int *list,
                                                 unsigned *steps, Q queue) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int n = a.n;
  int cnt = 0, taken = 0;
  for (int i = 0; i < span; i += 32) {
    const int v = (int)(b0 + i + lane);
    const bool has = v < n && a.xadj[v + 1] > a.xadj[v];
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (has) list[cnt + __popc(m & below)] = v;
    cnt += __popc(m);
  }
  __syncwarp();
  int cur = -1, hb = 0;
  List L;
  int refused = 0;  // offers of cur in a row
  bool failed = false;
  for (;;) {
    if (BOUNDED) {
      if (*steps == 0) return kChainLong;
      --*steps;
    }
    const unsigned idle = __ballot_sync(0xffffffffu, cur < 0);
    const bool first = taken == 0;
    if (taken < cnt && idle) {
      const int at = taken + __popc(idle & below);
      if (cur < 0 && at < cnt) {
        cur = list[at];
        hb = hash_base(a, cur);  // a chain stays in its graph
        L.load(a, cur);
      }
      taken += __popc(idle);
    } else if (idle == 0xffffffffu) {
      break;
    }
    if (first) {
      // A hub's leaves all want the hub: of a warp's first vertices only the best offers
      // itself, the others are refused by it or with it (a star of 1 M leaves: the
      // matching 171 -> 143 us with ties to the lower id, 243 -> 200 with hashed ones).
      const int c = cur >= 0 ? L.id[0] : kNone, hub = __shfl_sync(0xffffffffu, c, 0);
      if (__all_sync(0xffffffffu, c >= 0 && c == hub) &&
          Cand<H>::make(hub, cur, L.w[0], hb).warp_best().id() != cur)
        L.drop();
    }
    int qv = -1, qx = 0, qdeg = 0;
    if (cur >= 0) {
      L.check<H>(a, cur, hb);
      int c = L.id[0], w = L.w[0];
      unsigned long long held = L.seen[0];
      if (c == kUnknown) {
        qx = a.xadj[cur];
        qdeg = a.xadj[cur + 1] - qx;
        if (qdeg > kSerialDeg) qv = cur;
        else c = rescan_short<H, SCAN>(a, cur, qx, qdeg, all, hb, &w, &held);
      }
      if (c < 0) {  // queued, or no candidate is left
        cur = -1;
        refused = 0;
      } else {
        int out = -1;
        const int guess = AHEAD ? best_holder(held) : -1;
        List N;
        if (AHEAD && guess >= 0) N.load(a, guess);
        if (offer<H>(a, cur, c, w, held, hb, &out)) {
          cur = out;
          refused = 0;
          if (cur >= 0) {
            if (AHEAD && cur == guess) L = N;
            else L.load(a, cur);
            L.after(c);
          }
        } else if (++refused > kLaneRefusals) {  // c holds a better proposal now, which the next check sees
          record_error(a.st, CM_ERR_LIMIT, ERR_SITE_ROUNDS);
          failed = true;
          cur = -1;
        }
      }
    }
    __syncwarp();
    queue(qv, qx, qdeg);
  }
  // (the list is free for the next span)
  return __any_sync(0xffffffffu, failed) ? kChainFailed : kChainDone;
}

// A warp's chain, starting with v (free): its row is scanned, or `r` holds the
// candidates of a scan already made (rows of several chunks).  With hashed ties
// a scan first filters by weight alone -- the hash of every entry that ties
// with its neighbour's proposal costs more than the scan -- and only when all
// the candidates so found turn out to be refused is the row scanned again with
// the full test.  A free vertex whose row has several chunks is queued for the
// next round (slot par, counter ctr).  Every accepted offer takes one of *steps;
// without any left the free vertex is queued too (kQueue) or the warp gives up
// (kGiveUp: kChainLong).  Convergent.
//
// The candidates lie in the lanes: lane t < kTop holds the t-th, reads the proposal
// that this neighbour holds and compares.  best[] changes while the warp looks at
// it, so every decision comes from a ballot or a shuffle: lanes that each read
// best[] for themselves can see different proposals, take different branches and
// wait for one another in the scans' collectives for good.
enum : int { kEndless = 0, kQueue = 1, kGiveUp = 2 };
template <bool H, int LIMIT>
__device__ __forceinline__ ChainEnd warp_chain(const MatchArgs &a, int v, int xs, int xe, bool scanned,
                                               const TopK<H, kTop> &r, bool all, int par, int ctr, unsigned *steps,
                                               int2 *wbuf) {
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int hb = hash_base(a, v);
  int cur = v;
  int id = kUnknown, w = 0, from = kTop;  // this lane's candidate; lanes before `from` are done with
  unsigned long long seen = 0ull;         // the proposal it holds
  auto take = [&](const TopK<H, kTop> &t) {  // a scan's candidates
#pragma unroll
    for (int i = 0; i < kTop; ++i)
      if (lane == i) {
        id = t.c[i].id();
        w = t.c[i].weight();
      }
    from = 0;
  };
  // The lane of the first candidate that would take cur; kNone: there is none,
  // kUnknown: the list is used up.
  auto next = [&]() -> int {
    const bool live = lane >= from && lane < kTop, cand = live && id >= 0;
    seen = cand ? ld_best(a, id) : 0ull;
    const unsigned yes = __ballot_sync(full, cand && beats<H>(best_key(cur, w), seen, cur, id, hb));
    const unsigned end = __ballot_sync(full, live && id < 0);  // nothing behind the first of these
    const int y = yes ? __ffs(yes) - 1 : kTop, e = end ? __ffs(end) - 1 : kTop;
    if (y < e) return y;
    return e < kTop && __shfl_sync(full, id, e) == kNone ? kNone : kUnknown;
  };
  if (scanned) take(r);
  for (int refused = 0;;) {  // offers and scans of cur in a row that came to nothing
    if (refused > kWarpRefusals) {
      if (lane == 0) record_error(a.st, CM_ERR_LIMIT, ERR_SITE_ROUNDS);
      return kChainFailed;
    }
    int at = next();
    if (at == kUnknown) {
      if (cur != v || scanned) {
        xs = a.xadj[cur];
        xe = a.xadj[cur + 1];
      }
      if (xe - xs > kMatchChunk) {
        append_scan(a, par, ctr, lane == 0, cur, xs, xe - xs);
        return kChainDone;
      }
      if constexpr (H) {
        take(chunk_best<H, kTop, kWeak>(a, cur, xs, xe, all, wbuf));
        at = next();
      }
      if (!H || at == kUnknown) {
        take(chunk_best<H, kTop, kExact>(a, cur, xs, xe, all, wbuf));
        at = next();
      }
      if (at == kUnknown) {  // others took all of them meanwhile
        from = kTop;
        ++refused;
        continue;
      }
    }
    if (at == kNone) return kChainDone;
    const int c = __shfl_sync(full, id, at);
    int res = -2;  // -2: refused, else the vertex given up (-1: none)
    if (lane == at) {
      int out = -1;
      if (offer<H>(a, cur, id, w, seen, hb, &out)) res = out;
    }
    res = __shfl_sync(full, res, at);
    if (res == -2) {
      from = at + 1;
      ++refused;
      continue;
    }
    if (res < 0) return kChainDone;
    cur = res;
    refused = 0;
    scanned = true;  // xs, xe are another row's
    if (LIMIT != kEndless && *steps > 0) --*steps;
    if (LIMIT != kEndless && *steps == 0) {
      if (LIMIT == kGiveUp) return kChainLong;
      xs = a.xadj[cur];
      append_scan(a, par, ctr, lane == 0, cur, xs, a.xadj[cur + 1] - xs);
      return kChainDone;
    }
    if (lane < kTop) {
      id = a.top[(size_t)cur * kTop + lane];
      w = a.topw[(size_t)cur * kTop + lane];
    }
    // go on behind c; when c is not listed it came from a rescan, and the list is used up
    const unsigned listed = __ballot_sync(full, lane < kTop && id == c);
    from = listed ? __ffs(listed) : kTop;
  }
}

}  // namespace
}  // namespace cm
