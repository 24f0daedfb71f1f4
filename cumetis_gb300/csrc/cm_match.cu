// cm_match.cu -- deterministic heavy-edge matching.
//
// Replaces (cuMetis.cu) initcuda_match (1411), the per-level bb_segsort of
// every adjacency row by weight (1723, used only to find each row's maximum),
// cuda_shem2 (1563-1595, racy plain stores), cuda_cleanv (1600) and findc1
// (1621).  Eligibility follows cuda_shem2: a pair (v,k) may match if
// vwgt[v]+vwgt[k] <= maxvwgt and one end is light (3*vwgt < maxvwgt).
//
// Rule: every vertex prefers its heaviest eligible neighbour, ties to the lower
// vertex id (CM_MATCH_HEM) or to the lower edge hash (CM_MATCH_HEM_HASH, then
// lower id).  Both orders are strict total orders on edges, so the greedy
// matching of the order is unique, and any schedule of proposals that ends in
// the stable state finds it.
//
// Proposals (the Suitor scheme of Manne and Halappanavar): best[u] is the best
// proposal u has received; a free vertex offers itself to its most preferred
// neighbour whose best[] it beats, and the vertex it displaces there becomes
// free and goes on with its own next candidate.  best[u] only improves, so a
// rejected candidate never has to be looked at again, and no vertex state is
// read beside best[]: there are no rounds of propose / commit / filter.  When
// nobody is free, best[u] = v and best[v] = u for every matched pair.
//
//   k_match_prep     zeroes best[], finds the largest vertex weight, lists the
//                    chunks of rows longer than kSerialDeg, and gives the
//                    vertices of shorter rows their kTop most preferred
//                    neighbours, from weights alone.
//   k_match_first    the same for the longer rows, kFirstKeepChunk neighbours.
//                    The lists are not written again, so the later kernels read
//                    them without ordering.
//   k_match_propose  one thread a vertex follows the chain of displacements
//                    that its vertex's offer starts: per step one list read and
//                    one atomic.  A short row whose list is used up is rescanned
//                    by the thread; a longer one is queued.
//   k_match_rounds   queued rows, one warp per row of up to kChunk entries, the
//                    warp following the chain; rows of several chunks are merged
//                    by the last chunk's warp, and a displaced one is queued for
//                    the next round (grid barrier; a round with few chunks runs
//                    on one block).
//   k_match_finish   match[v] = the partner, or v.
//
// Only an adjacency that is not symmetric can end with an offer that is not
// returned (best[u] = v, best[v] != u).  k_match_finish sees that and the
// matching is then computed again by handshakes (handshake_rounds), whose
// result is defined for such inputs too.
#include <climits>

#include <algorithm>

#include "cm_ctx.h"

namespace cm {
namespace {

// Threads per block of the round kernel and the blocks per SM it is compiled
// for (its grid is every resident block, up to the graph's need).
#ifndef CM_MATCH_THREADS
#define CM_MATCH_THREADS 1024
#endif
#ifndef CM_MATCH_MINBLOCKS
#define CM_MATCH_MINBLOCKS 1
#endif
constexpr int kMatchThreads = CM_MATCH_THREADS, kMatchMinBlocks = CM_MATCH_MINBLOCKS;
constexpr int64_t kWorkPerBlock = 32768;  // vertices + entries per block of the matching grid
// Rows of at most kSerialDeg entries are scanned by one lane, longer rows in
// kChunk-entry warp work items (tuning parameters, set through the build).
#ifndef CM_SERIAL_DEG
#define CM_SERIAL_DEG 16
#endif
#ifndef CM_MATCH_CHUNK
#define CM_MATCH_CHUNK 256
#endif
constexpr int kSerialDeg = CM_SERIAL_DEG;
constexpr int kChunk = CM_MATCH_CHUNK;
static_assert(kSerialDeg == 8 || kSerialDeg == 16, "CM_SERIAL_DEG: 8 or 16");
static_assert(kChunk == 128 || kChunk == 256 || kChunk == 512, "CM_MATCH_CHUNK: 128, 256 or 512");
constexpr int kTop = 4;          // listed candidates per vertex
// Tail mode (one block runs the remaining rounds) once a round has at most
// kTailChunks row chunks.
#ifndef CM_TAIL_CHUNKS
#define CM_TAIL_CHUNKS 64
#endif
constexpr int kTailChunks = CM_TAIL_CHUNKS;
constexpr int kNone = -1;        // list slot: no further candidate
constexpr int kUnknown = -3;     // list slot not computed (more candidates may exist)
// Candidates listed for rows of more than kSerialDeg entries (short rows: kTop).
#ifndef CM_FIRST_KEEP_CHUNK
#define CM_FIRST_KEEP_CHUNK 4
#endif
constexpr int kFirstKeepChunk = CM_FIRST_KEEP_CHUNK;
static_assert(kFirstKeepChunk >= 1 && kFirstKeepChunk <= kTop, "CM_FIRST_KEEP_CHUNK: 1 to 4");

struct Slot {      // rows to scan in one round
  int *big_base, *big_done;  // per row: first chunk, chunks done
  int4 *desc;      // per chunk: (vertex, first entry, end entry, row index or -1 if one chunk)
};

struct MatchArgs {
  int n, span;                   // span: vertices a warp takes at a time (multiple of 32, at most kSpan)
  const int *xadj, *adjncy, *adjwgt, *vwgt;
  long long maxvwgt;
  int mode;
  int *m2;                       // the matching (output)
  unsigned long long *best;      // best proposal received: (weight, proposer), 0 = none (best_key)
  int *top, *topw;               // kTop listed candidates per vertex: ids, weights
  Slot slot[2];
  unsigned long long *big;       // [3] = (rows << 32 | chunks) of the slots, by round
  int *tick;                     // [3] work tickets of the round kernel, by round
  int *vmax;                     // largest vertex weight (zeroed before the launch)
  int *odd;                      // [2]: an offer was not returned; blocks of k_match_finish done
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
__device__ __forceinline__ unsigned long long ld_best(const MatchArgs &a, int k) { return __ldcg(a.best + k); }

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

// Loads entries [b, e) (e - b <= kChunk) of v's row, slot u of a lane entry
// b + lane + 32 u, all loads issued before any is used, and marks with
// k[u] = -1 those that are no candidates: the vertex itself, pairs that do not
// fit (`all`: every pair fits), and neighbours that hold a proposal v cannot
// beat: by its weight alone (kWeak), or at all (kExact).
enum : int { kStatic = 0, kWeak = 1, kExact = 2 };
template <bool H, int FILTER>
__device__ __forceinline__ void load_entries(const MatchArgs &a, int v, int b, int e, bool all, int hb,
                                             int (&k)[kChunk / 32], int (&w)[kChunk / 32]) {
  const int lane = threadIdx.x & 31;
  constexpr int U = kChunk / 32;
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
      bw[u] = (u < nu && k[u] >= 0) ? __ldcg(reinterpret_cast<const unsigned *>(a.best + k[u]) + 1) : 0u;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (((unsigned)w[u] ^ 0x80000000u) < bw[u]) k[u] = -1;
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

// Inserts x into the descending list tw (the KK largest values seen, with
// repeats).
template <int KK>
__device__ __forceinline__ void wlist_insert(int (&tw)[KK], int x) {
#pragma unroll
  for (int i = 0; i < KK; ++i) {
    const int hi = max(tw[i], x);
    x = min(tw[i], x);
    tw[i] = hi;
  }
}

// The warp's best KK candidates over entries [b, e) (e - b <= kChunk) of v's
// row; every lane gets the list.  Hash order: most entries are lighter than
// the chunk's KK-th heaviest eligible entry and can never enter the list, so
// a weight threshold W is found first and only entries of weight >= W get an
// edge hash and a full comparison.  W is the KK-th largest weight of the
// union of the lanes' own KK heaviest (a sub-multiset of the chunk), so at
// least KK entries weigh >= W and the chunk's best KK are all among them.
// The qualifying entries (usually KK plus the ties at W) are packed one per
// lane through the warp's 32-entry buffer wbuf; more than 32 of them (many
// equal weights) take the per-lane lists instead.
template <bool H, int KK, int FILTER>
__device__ __forceinline__ TopK<H, KK> chunk_best(const MatchArgs &a, int v, int b, int e, bool all, int2 *wbuf) {
  constexpr int U = kChunk / 32;
  const int nu = (e - b + 31) >> 5;
  const int hb = hash_base(a, v);
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
    int tw[KK], rem = 0;
#pragma unroll
    for (int i = 0; i < KK; ++i) tw[i] = INT_MIN;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;
      if (k[u] >= 0) {
        wlist_insert(tw, w[u]);
        ++rem;
      }
    }
    rem = min(rem, KK);
    // threshold: pop the lanes' list heads in descending order until KK
    // entries are taken (or every list is empty: then all eligible entries
    // qualify, W being the lightest of them)
    int W = INT_MIN, taken = 0;
#pragma unroll
    for (int r = 0; r < KK; ++r) {
      const bool has = rem > 0;
      if (!__ballot_sync(full, has)) break;
      const int mine = has ? tw[0] : INT_MIN;
      const int mx = __reduce_max_sync(full, mine);
      const bool pop = has && mine == mx;
      taken += __popc(__ballot_sync(full, pop));
      W = mx;
      if (pop) {
#pragma unroll
        for (int i = 0; i + 1 < KK; ++i) tw[i] = tw[i + 1];
        --rem;
      }
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
    // exist is recomputed over every eligible entry, so that a short list
    // still means "no other candidate".
    if (taken >= KK && !out.c[KK - 1].valid()) {
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
      desc[rc + j] = make_int4(rx, rs + j * kChunk, min(rs + rd, rs + (j + 1) * kChunk), ri);
  }
}

// Queues x (row of deg > kSerialDeg entries starting at xs) for a scan: slot
// `par`, counter `ctr`; convergent.
__device__ __forceinline__ void append_scan(const MatchArgs &a, int par, int ctr, bool take, int x, int xs, int deg) {
  if (!__any_sync(0xffffffffu, take)) return;
  const Slot &S = a.slot[par];
  const int lane = threadIdx.x & 31;
  const int nch = take ? (deg + kChunk - 1) / kChunk : 0;
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

constexpr int kPrepThreads = 256;
// Resident blocks per SM the list kernel is compiled for (register cap).
#ifndef CM_FIRST_MINBLOCKS
#define CM_FIRST_MINBLOCKS 8
#endif
constexpr int kFirstMinBlocks = CM_FIRST_MINBLOCKS;

// Vertices a warp takes at a time in k_match_prep and k_match_propose: it first
// packs those it has work for (short rows; rows with entries) in shared memory,
// so that all lanes work although half of an R-MAT graph's vertices are
// isolated and the low ids have long rows.  Small graphs take fewer per warp.
constexpr int kSpan = 256;

// best[] = none, the largest vertex weight, the chunks of the rows longer than
// kSerialDeg (slot 0), and the lists of the shorter rows, one lane each (from
// the weights and the cap alone).  The counters are zeroed by the host.
template <bool H>
__global__ void __launch_bounds__(kPrepThreads) k_match_prep(MatchArgs a) {
  __shared__ int sh_v[kPrepThreads / 32][kSpan];
  int *list = sh_v[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int gwarp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  const int n = a.n;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.st->rounds = 1;
  int wmax = 0;
  for (long long b0 = (long long)gwarp * a.span; b0 < n; b0 += (long long)nwarps * a.span) {
    int cnt = 0;
    for (int i = 0; i < a.span; i += 32) {
      const int v = (int)(b0 + i + lane);
      int xs = 0, deg = 0;
      if (v < n) {
        wmax = max(wmax, a.vwgt[v]);
        a.best[v] = 0ull;
        xs = a.xadj[v];
        deg = a.xadj[v + 1] - xs;
      }
      append_scan(a, 0, 0, deg > kSerialDeg, v, xs, deg);
      const bool small = deg > 0 && deg <= kSerialDeg;
      const unsigned m = __ballot_sync(0xffffffffu, small);
      if (small) list[cnt + __popc(m & below)] = v;
      cnt += __popc(m);
    }
    __syncwarp();
    for (int i = lane; i < cnt; i += 32) {
      const int v = list[i];
      const int xs = a.xadj[v], deg = a.xadj[v + 1] - xs;
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
    __syncwarp();  // the list is free for the next span
  }
  wmax = __reduce_max_sync(0xffffffffu, wmax);
  if (lane == 0 && wmax > 0) atomicMax(a.vmax, wmax);
}

// The lists of the rows longer than kSerialDeg, one warp a chunk, the warp of
// a row's last chunk merging the chunks' lists.  Two forms: with every edge
// eligible the scan reads no vertex weights and fits 32 registers.  Both are
// launched (the choice is made on the device, from the largest vertex
// weight); the one that does not apply returns at once.
template <bool H, bool ALL>
__global__ void __launch_bounds__(kPrepThreads, ALL ? kFirstMinBlocks : kFirstMinBlocks / 2) k_match_first(MatchArgs a) {
  if (all_eligible(a) != ALL) return;
  const int lane = threadIdx.x & 31;
  const int gwarp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  __shared__ int2 sh_q[kPrepThreads / 32][32];
  const Slot &S = a.slot[0];
  const int nchunks = (int)(__ldcg(a.big) & 0xffffffffu);
  constexpr int KC = kFirstKeepChunk;
  int4 d = gwarp < nchunks ? __ldcg(S.desc + gwarp) : make_int4(0, 0, 0, 0);
  for (int q = gwarp; q < nchunks; q += nwarps) {
    const int4 dn = q + nwarps < nchunks ? __ldcg(S.desc + q + nwarps) : d;
    const int v = d.x;
    const TopK<H, KC> r = chunk_best<H, KC, kStatic>(a, v, d.y, d.z, ALL, sh_q[threadIdx.x >> 5]);
    if (d.w < 0) {
      if (lane == 0) store_top(a, v, r);
    } else {
      const int nch = (a.xadj[v + 1] - a.xadj[v] + kChunk - 1) / kChunk;
      if (part_done<H, KC>(a, S, q, d, nch, r)) {
        const int base = __ldcg(S.big_base + d.w);
        const TopK<H, KC> rr =
            merge_parts<H, KC>(a, nch * KC, [&](int t) { return (size_t)(base + t / KC) * kTop + t % KC; });
        if (lane == 0) store_top(a, v, rr);
      }
    }
    d = dn;
  }
}

// Best candidate of a short row (deg <= kSerialDeg) that takes v now, by one
// lane; *seen = the proposal it holds.  -1: none.
template <bool H>
__device__ __forceinline__ int rescan_short(const MatchArgs &a, int v, int xs, int deg, bool all, int hb, int *weight,
                                            unsigned long long *seen) {
  constexpr int kHalf = 8;
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

// One lane a vertex: offers the vertex to its candidates in order and goes on
// with whomever a taker gives up, until nobody is left without a proposal or
// the free vertex needs a scan of a long row, which is queued (slot 1).  A lane
// whose chain has ended takes the span's next vertex.
template <bool H>
__global__ void __launch_bounds__(kPrepThreads) k_match_propose(MatchArgs a) {
  __shared__ int sh_v[kPrepThreads / 32][kSpan];
  int *list = sh_v[threadIdx.x >> 5];
  const bool all = all_eligible(a);
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int gwarp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  const int n = a.n;
  for (long long b0 = (long long)gwarp * a.span; b0 < n; b0 += (long long)nwarps * a.span) {
    int cnt = 0, taken = 0;
    for (int i = 0; i < a.span; i += 32) {
      const int v = (int)(b0 + i + lane);
      const bool has = v < n && a.xadj[v + 1] > a.xadj[v];
      const unsigned m = __ballot_sync(0xffffffffu, has);
      if (has) list[cnt + __popc(m & below)] = v;
      cnt += __popc(m);
    }
    __syncwarp();
    int cur = -1, hb = 0;
    List L;
    for (;;) {
      const unsigned idle = __ballot_sync(0xffffffffu, cur < 0);
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
      int qv = -1, qx = 0, qdeg = 0;
      if (cur >= 0) {
        L.check<H>(a, cur, hb);
        int c = L.id[0], w = L.w[0];
        unsigned long long held = L.seen[0];
        if (c == kUnknown) {
          qx = a.xadj[cur];
          qdeg = a.xadj[cur + 1] - qx;
          if (qdeg > kSerialDeg) qv = cur;
          else c = rescan_short<H>(a, cur, qx, qdeg, all, hb, &w, &held);
        }
        if (c < 0) {  // queued, or no candidate is left
          cur = -1;
        } else {
          int out = -1;
          if (offer<H>(a, cur, c, w, held, hb, &out)) {
            cur = out;
            if (cur >= 0) {
              L.load(a, cur);
              L.after(c);
            }
          }  // refused: c holds a better proposal now, which the next check sees
        }
      }
      __syncwarp();
      append_scan(a, 1, 1, qv >= 0, qv, qx, qdeg);
    }
    __syncwarp();  // the list is free for the next span
  }
}

// A warp's chain, starting with v (free): its row is scanned, or `r` holds the
// candidates of a scan already made (rows of several chunks).  With hashed ties
// a scan first filters by weight alone -- the hash of every entry that ties
// with its neighbour's proposal costs more than the scan -- and only when all
// the candidates so found turn out to be refused is the row scanned again with
// the full test.  A free vertex whose row has several chunks is queued for the
// next round (slot par, counter ctr).  Convergent.
template <bool H>
__device__ __forceinline__ void warp_chain(const MatchArgs &a, int v, int xs, int xe, bool scanned,
                                           const TopK<H, kTop> &r, bool all, int par, int ctr, int2 *wbuf) {
  const int lane = threadIdx.x & 31;
  const int hb = hash_base(a, v);
  int cur = v;
  List L;
  auto take = [&](const TopK<H, kTop> &t) {  // the scan's candidates as a list
#pragma unroll
    for (int i = 0; i < kTop; ++i) {
      L.id[i] = t.c[i].id();
      L.w[i] = t.c[i].weight();
    }
    L.check<H>(a, cur, hb);
  };
  if (scanned) take(r);
  else L.id[0] = kUnknown;
  for (;;) {
    if (L.id[0] == kUnknown) {
      if (cur != v || scanned) {
        xs = a.xadj[cur];
        xe = a.xadj[cur + 1];
      }
      if (xe - xs > kChunk) {
        append_scan(a, par, ctr, lane == 0, cur, xs, xe - xs);
        return;
      }
      if constexpr (H) take(chunk_best<H, kTop, kWeak>(a, cur, xs, xe, all, wbuf));
      if (!H || L.id[0] == kUnknown) take(chunk_best<H, kTop, kExact>(a, cur, xs, xe, all, wbuf));
    }
    const int c = L.id[0];
    if (c == kNone) return;
    if (c == kUnknown) continue;  // others took all of them meanwhile
    int res = -2;  // -2: refused, else the vertex given up (-1: none)
    if (lane == 0) {
      int out = -1;
      if (offer<H>(a, cur, c, L.w[0], L.seen[0], hb, &out)) res = out;
    }
    res = __shfl_sync(0xffffffffu, res, 0);
    if (res == -2) {
      L.drop();
    } else {
      if (res < 0) return;
      cur = res;
      L.load(a, cur);
      L.after(c);
      scanned = true;  // xs, xe are another row's
    }
    L.check<H>(a, cur, hb);
  }
}

// Scans of the queued rows and the chains they start, in rounds; ONE_PASS: no
// row has several chunks, so nothing is queued again and no barrier is needed
// (an ordinary launch).
template <bool H, bool ONE_PASS>
__global__ void __launch_bounds__(kMatchThreads, kMatchMinBlocks) k_match_rounds(MatchArgs a) {
  __shared__ int2 sh_q[kMatchThreads / 32][32];  // per warp: packed candidates of a chunk scan
  const int lane = threadIdx.x & 31;
  const bool all = all_eligible(a);
  int2 *wbuf = sh_q[threadIdx.x >> 5];
  DevStatus *st = a.st;
  const bool first_thread = blockIdx.x == 0 && threadIdx.x == 0;
  auto trace = [&](int row, int col, unsigned long long v) {
    if (a.trace != nullptr && first_thread && row < a.trace_rows) a.trace[row * 8 + col] = v;
  };
  trace(0, 0, global_timer_ns());
  trace(0, 1, global_timer_ns());
  bool tail = false;
  int round = 1;  // slot and counter 1 hold what k_match_propose queued
  for (;; ++round) {
    const int par = round & 1, ctr = round % 3, next = (round + 1) % 3;
    const Slot &S = a.slot[par];
    const unsigned long long bc = __ldcg(a.big + ctr);
    const int nchunks = (int)(bc & 0xffffffffu);
    trace(round, 0, global_timer_ns());
    trace(round, 5, bc >> 32);
    trace(round, 6, (unsigned long long)nchunks);
    if (nchunks == 0) break;
    if (round > a.max_rounds) {
      if (first_thread) record_error(st, CM_ERR_LIMIT, ERR_SITE_ROUNDS);
      break;
    }
    // All blocks decide alike, from the counter read after a grid barrier.
    if (!ONE_PASS && !tail && round > 1 && nchunks <= kTailChunks) {
      tail = true;
      if (blockIdx.x != 0) return;
    }
    if (!ONE_PASS && first_thread) {  // the counters of the round after the next
      a.big[(round + 2) % 3] = 0;
      a.tick[(round + 2) % 3] = 0;
    }
    // Chunks are taken from a ticket: rows and chains differ in length.
    int q = 0;
    if (lane == 0) q = atomicAdd(a.tick + ctr, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    int4 d = q < nchunks ? __ldcg(S.desc + q) : make_int4(0, 0, 0, 0);
    while (q < nchunks) {
      int qn = 0;
      if (lane == 0) qn = atomicAdd(a.tick + ctr, 1);
      TopK<H, kTop> r;
      bool mine = true;
      if (d.w >= 0) {
        r = chunk_best<H, kTop, kExact>(a, d.x, d.y, d.z, all, wbuf);
        const int nch = (a.xadj[d.x + 1] - a.xadj[d.x] + kChunk - 1) / kChunk;
        mine = part_done<H, kTop>(a, S, q, d, nch, r);
        if (mine) {
          const int base = __ldcg(S.big_base + d.w);
          r = merge_parts<H, kTop>(a, nch * kTop, [&](int t) { return (size_t)base * kTop + t; });
        }
      }
      qn = __shfl_sync(0xffffffffu, qn, 0);
      const int4 dn = qn < nchunks ? __ldcg(S.desc + qn) : d;
      if (mine) warp_chain<H>(a, d.x, d.y, d.z, d.w >= 0, r, all, par ^ 1, next, wbuf);
      q = qn;
      d = dn;
    }
    trace(round, 3, global_timer_ns());
    if (ONE_PASS) break;
    if (!tail) {
      if (!grid_barrier(st, gridDim.x)) return;
    } else {
      __threadfence();
      __syncthreads();
      if (ld_relaxed(&st->error) != 0) return;
    }
  }
  if (first_thread) st->rounds = round;
  trace(0, 3, global_timer_ns());
  trace(0, 4, (unsigned long long)(round - 1));
}

// The matching of an adjacency that is not symmetric: mutual proposals in
// rounds until no pair forms.  Every unmatched vertex points at its most
// preferred unmatched neighbour (ptr), and vertices that point at each other
// are matched.  One warp a vertex, over the warps gw, gw + nw, ...; barrier()
// separates the phases and returns false to give up.  Reads and writes of
// other warps' vertices go to L2.
template <bool H, typename B>
__device__ void handshake_rounds(const MatchArgs &a, int *ptr, int *changed, int gw, int nw, B barrier) {
  const int lane = threadIdx.x & 31;
  const int n = a.n;
  for (long long v = (long long)gw * 32 + lane; v < n; v += (long long)nw * 32) a.m2[v] = -1;
  if (gw == 0 && lane == 0) changed[0] = changed[1] = changed[2] = 0;
  if (!barrier()) return;
  for (int round = 0;; ++round) {
    if (gw == 0 && lane == 0) changed[(round + 1) % 3] = 0;
    for (long long v = gw; v < n; v += nw) {
      if (__ldcg(a.m2 + v) >= 0) continue;
      const int hb = hash_base(a, (int)v);
      const long long vw = a.vwgt[v], cap = weight_cap(a, (int)v);
      Cand<H> c;
      for (int j = a.xadj[v] + lane; j < a.xadj[v + 1]; j += 32) {
        const int k = a.adjncy[j];
        if (k == (int)v || __ldcg(a.m2 + k) >= 0 || !pair_fits(cap, vw, a.vwgt[k])) continue;
        const Cand<H> x = Cand<H>::make((int)v, k, a.adjwgt[j], hb);
        if (x.better(c)) c = x;
      }
      const int p = c.warp_best().id();
      if (lane == 0) ptr[v] = p;
    }
    if (!barrier()) return;
    bool any = false;
    for (long long v = (long long)gw * 32 + lane; v < n; v += (long long)nw * 32) {
      if (__ldcg(a.m2 + v) >= 0) continue;
      const int p = __ldcg(ptr + v);
      if (p > (int)v && __ldcg(ptr + p) == (int)v) {  // the lower end commits both
        a.m2[v] = p;
        a.m2[p] = (int)v;
        any = true;
      }
    }
    if (any) changed[round % 3] = 1;
    if (!barrier()) return;
    if (__ldcg(changed + round % 3) == 0) break;
  }
  for (long long v = (long long)gw * 32 + lane; v < n; v += (long long)nw * 32)
    if (a.m2[v] < 0) a.m2[v] = (int)v;
}

// match[v] from best[]; a proposal that is not returned sets odd[0].  With
// `alone` the last block then computes the matching by handshakes itself.
template <bool H>
__global__ void __launch_bounds__(kPrepThreads) k_match_finish(MatchArgs a, int alone) {
  bool odd = false;
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < a.n;
       v += (long long)gridDim.x * blockDim.x) {
    const int h = best_holder(a.best[v]);
    const bool mutual = h >= 0 && best_holder(a.best[h]) == (int)v;
    a.m2[v] = mutual ? h : (int)v;
    odd |= h >= 0 && !mutual;
  }
  if (odd) atomicOr(a.odd, 1);
  if (!alone) return;
  __threadfence();
  __syncthreads();
  __shared__ int s_last;
  if (threadIdx.x == 0) s_last = atomicAdd(a.odd + 1, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!s_last || __ldcg(a.odd) == 0) return;
  handshake_rounds<H>(a, a.top, a.odd + 2, threadIdx.x >> 5, blockDim.x >> 5, [&] {
    __threadfence();
    __syncthreads();
    return true;
  });
}

// The same for large graphs, with every resident block.
template <bool H>
__global__ void __launch_bounds__(kMatchThreads, kMatchMinBlocks) k_match_handshake(MatchArgs a) {
  if (__ldcg(a.odd) == 0) return;
  handshake_rounds<H>(a, a.top, a.odd + 2, (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5),
                      (int)((gridDim.x * blockDim.x) >> 5), [&] { return grid_barrier(a.st, gridDim.x); });
}

// ---------------------------------------------------------------------------
// CM_MATCH_RACY: one unsynchronised proposal pass and its cleanup, as the
// reference's cuda_shem2 (cu:1563-1595) + cuda_cleanv (cu:1600) + findc1
// (cu:1621).  A light vertex (3 vwgt < cap) that nobody has claimed takes,
// among its neighbours that already point at it or are unmatched within the
// weight cap, the heaviest one (the reference walks its row sorted by weight,
// heaviest first, and stops at the first such neighbour), and writes both
// ends with plain stores; concurrent writers race.  The cleanup then turns
// every vertex whose partner does not point back into a singleton.  The
// result is a legal matching, not a maximal one, and depends on the schedule.
// One warp per vertex (the reference uses one thread per vertex).
// ---------------------------------------------------------------------------
constexpr int kRacyThreads = 256;

__global__ void k_racy_init(int n, int *__restrict__ m) {
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x)
    m[v] = -1;
}

__global__ void __launch_bounds__(kRacyThreads) k_racy_propose(MatchArgs a) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (kRacyThreads / 32);
  volatile int *m = a.m2;
  for (long long v = (long long)blockIdx.x * (kRacyThreads / 32) + (threadIdx.x >> 5); v < a.n; v += warps) {
    const long long cap = weight_cap(a, (int)v);
    const long long vw = a.vwgt[v];
    if (!(3 * vw < cap)) continue;
    if (m[v] != -1) continue;  // already claimed
    // heaviest candidate; equal weights by the edge hash (both ends of an
    // edge rank it alike, which the reference's unstable weight sort leaves
    // to chance)
    const int hb = hash_base(a, (int)v);
    int bw = INT_MIN, bk = -1;
    unsigned bh = 0xffffffffu;
    for (int j = a.xadj[v] + lane; j < a.xadj[v + 1]; j += 32) {
      const int k = a.adjncy[j];
      if (k == v) continue;
      const int mk = m[k];
      const bool ok = mk == (int)v || (mk == -1 && vw + a.vwgt[k] <= cap);
      if (!ok) continue;
      const int w = a.adjwgt[j];
      const unsigned h = edge_hash((unsigned)(min((int)v, k) - hb), (unsigned)(max((int)v, k) - hb));
      if (w > bw || (w == bw && h < bh)) {
        bw = w;
        bh = h;
        bk = k;
      }
    }
    const int top = __reduce_max_sync(0xffffffffu, bk >= 0 ? bw : INT_MIN);
    const unsigned hmin = __reduce_min_sync(0xffffffffu, (bk >= 0 && bw == top) ? bh : 0xffffffffu);
    const unsigned holders = __ballot_sync(0xffffffffu, bk >= 0 && bw == top && bh == hmin);
    if (holders == 0) continue;
    const int k = __shfl_sync(0xffffffffu, bk, __ffs(holders) - 1);
    if (lane == 0 && m[v] == -1) {
      m[v] = k;
      if (m[k] != (int)v) m[k] = (int)v;
    }
  }
}

// s[v] = 1 if v keeps its partner (unmatched, or the partner points back).
__global__ void k_racy_clean(int n, const int *__restrict__ m, int *__restrict__ s) {
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
    const int u = m[v];
    s[v] = (u == -1 || m[u] == (int)v) ? 1 : 0;
  }
}

__global__ void k_racy_apply(int n, int *__restrict__ m, const int *__restrict__ s) {
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x)
    if (s[v] == 0 || m[v] == -1) m[v] = (int)v;
}

int64_t max_chunks(int64_t n, int64_t m) { return m / kChunk + n + 64; }

}  // namespace

size_t match_ws_bytes(int64_t n, int64_t m) {
  const int64_t ch = max_chunks(n, m);
  size_t b = (size_t)n * (8 + 2 * 4 * kTop);                  // best, lists
  b += 2 * ((size_t)n * 4 * 2 + (size_t)ch * 16);             // two slots
  b += (size_t)ch * 4 * kPartInts * kTop;                     // chunk partial lists
  return b + 64 * 256;
}

// Graphs above this many vertices + entries get the handshake kernel with
// every block behind k_match_finish (a launch that returns at once costs a few
// us, under 5% there); below it the last block of k_match_finish does the work.
constexpr int64_t kAloneWork = 1 << 21;

int launch_match(cm_ctx *ctx, const cm_graph *g, int32_t maxvwgt, int32_t mode, int32_t *d_match, cudaStream_t s,
                 const int32_t *vgid, const int32_t *gbase, const int32_t *gcap, int64_t max_deg) {
  const int n = g->nvtxs;
  if (n == 0) return CM_OK;
  if (mode != CM_MATCH_HEM && mode != CM_MATCH_HEM_HASH && mode != CM_MATCH_RACY)
    return cm_fail(CM_ERR_INVALID, "cm_match: unknown mode %d", mode);
  if (mode == CM_MATCH_RACY) {
    MatchArgs a{};
    a.n = n;
    a.xadj = g->xadj; a.adjncy = g->adjncy; a.adjwgt = g->adjwgt; a.vwgt = g->vwgt;
    a.maxvwgt = maxvwgt;
    a.m2 = d_match;
    a.vgid = vgid;
    a.gbase = gbase;
    a.gcap = gcap;
    int *flags = (int *)ws_take(ctx, (size_t)n * 4);
    if (!flags) return cm_fail(CM_ERR_NOMEM, "cm_match: workspace too small");
    const unsigned vg = (unsigned)std::min<int64_t>((int64_t)ctx->num_sms * 8, n / 256 + 1);
    const unsigned wg = (unsigned)std::min<int64_t>((int64_t)ctx->num_sms * 16, n / (kRacyThreads / 32) + 1);
    stage_begin(ctx, s);
    k_racy_init<<<vg, 256, 0, s>>>(n, d_match);
    k_racy_propose<<<wg, kRacyThreads, 0, s>>>(a);
    k_racy_clean<<<vg, 256, 0, s>>>(n, d_match, flags);
    k_racy_apply<<<vg, 256, 0, s>>>(n, d_match, flags);
    stage_end(ctx, CM_STAGE_MATCH, s);
    ctx->launches += 4;
    cudaMemsetAsync(&ctx->d_status->rounds, 0, sizeof(int), s);
    return check_launch(ctx, "cm_match (racy)");
  }
  const int64_t ch = max_chunks(n, g->nedges);
  MatchArgs a;
  a.n = n;
  a.xadj = g->xadj; a.adjncy = g->adjncy; a.adjwgt = g->adjwgt; a.vwgt = g->vwgt;
  a.maxvwgt = maxvwgt;  // with graphs side by side: the smallest cap (it gates the all-eligible first round)
  a.mode = mode;
  a.m2 = d_match;
  a.vgid = vgid;
  a.gbase = gbase;
  a.gcap = gcap;
  bool ok = true;
  auto take = [&](size_t bytes) {
    void *p = ws_take(ctx, bytes);
    ok = ok && p != nullptr;
    return (int *)p;
  };
  a.best = (unsigned long long *)take((size_t)n * 8);
  a.top = take((size_t)n * 4 * kTop);
  a.topw = take((size_t)n * 4 * kTop);
  for (int p = 0; p < 2; ++p) {
    Slot &S = a.slot[p];
    S.big_base = take((size_t)n * 4);
    S.big_done = take((size_t)n * 4);
    S.desc = (int4 *)take((size_t)ch * 16);
  }
  a.part = take((size_t)ch * 4 * kPartInts * kTop);
  int *ctrs = take(256);  // counters of the slots, the largest vertex weight, flags
  if (!ok) return cm_fail(CM_ERR_NOMEM, "cm_match: workspace too small");
  a.big = (unsigned long long *)ctrs;
  a.tick = ctrs + 8;
  a.vmax = ctrs + 16;
  a.odd = ctrs + 24;
  cudaMemsetAsync(ctrs, 0, 256, s);
  a.max_rounds = (long long)n + g->nedges + 8;
  a.st = ctx->d_status;
  a.trace = ctx->d_trace;
  a.trace_rows = ctx->trace_rows;
  const bool hash = mode == CM_MATCH_HEM_HASH;
  // No row longer than kChunk: the queued rows take one pass and no barrier.
  const bool one_pass = max_deg <= kChunk;
  const bool rounds = max_deg > kSerialDeg || a.trace != nullptr;
  const bool alone = (int64_t)n + g->nedges <= kAloneWork;
  const void *fn = hash ? (const void *)k_match_rounds<true, false> : (const void *)k_match_rounds<false, false>;
  const void *hfn = hash ? (const void *)k_match_handshake<true> : (const void *)k_match_handshake<false>;
  int &per_sm = ctx->match_blocks_per_sm[hash];  // queried once per context and tie order
  if (per_sm == 0) {
    int h_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kMatchThreads, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&h_sm, hfn, kMatchThreads, 0);
    per_sm = std::min(per_sm, h_sm);
  }
  if (per_sm < 1) {
    per_sm = 0;
    return cm_fail(CM_ERR_CUDA, "cm_match: kernel cannot be resident");
  }
  // Small graphs take a few SMs, so that kernels of other contexts (other
  // streams) can run beside this one; the kernels are grid-size agnostic.
  const int64_t want = (n + g->nedges) / kWorkPerBlock + 1;
  const int grid = (int)std::min<int64_t>((int64_t)ctx->num_sms * per_sm, want);
  void *args[] = {(void *)&a};
  stage_begin(ctx, s);
  const unsigned pgrid = (unsigned)std::min<int64_t>((int64_t)ctx->num_sms * 8, n / kPrepThreads + 1);
  a.span = (int)std::max<int64_t>(32, std::min<int64_t>(kSpan, n / ((int64_t)pgrid * kPrepThreads) * 32));
  const unsigned fgrid = (unsigned)std::min<int64_t>((int64_t)ctx->num_sms * 8, std::max<int64_t>(want * 4, pgrid));
  if (hash) k_match_prep<true><<<pgrid, kPrepThreads, 0, s>>>(a);
  else k_match_prep<false><<<pgrid, kPrepThreads, 0, s>>>(a);
  if (max_deg > kSerialDeg) {
    if (hash) {
      k_match_first<true, true><<<fgrid, kPrepThreads, 0, s>>>(a);
      k_match_first<true, false><<<fgrid, kPrepThreads, 0, s>>>(a);
    } else {
      k_match_first<false, true><<<fgrid, kPrepThreads, 0, s>>>(a);
      k_match_first<false, false><<<fgrid, kPrepThreads, 0, s>>>(a);
    }
    ctx->launches += 2;
  }
  if (hash) k_match_propose<true><<<pgrid, kPrepThreads, 0, s>>>(a);
  else k_match_propose<false><<<pgrid, kPrepThreads, 0, s>>>(a);
  ctx->launches += 2;
  cudaError_t e = cudaSuccess;
  if (rounds && one_pass) {
    if (hash) k_match_rounds<true, true><<<grid, kMatchThreads, 0, s>>>(a);
    else k_match_rounds<false, true><<<grid, kMatchThreads, 0, s>>>(a);
    ctx->launches++;
  } else if (rounds) {
    e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kMatchThreads), args, 0, s);
    ctx->launches++;
  }
  const unsigned vgrid = (unsigned)std::min<int64_t>((int64_t)ctx->num_sms * 8, n / kPrepThreads + 1);
  if (hash) k_match_finish<true><<<vgrid, kPrepThreads, 0, s>>>(a, alone);
  else k_match_finish<false><<<vgrid, kPrepThreads, 0, s>>>(a, alone);
  ctx->launches++;
  if (e == cudaSuccess && !alone) {
    e = cudaLaunchCooperativeKernel(hfn, dim3(grid), dim3(kMatchThreads), args, 0, s);
    ctx->launches++;
  }
  stage_end(ctx, CM_STAGE_MATCH, s);
  return cuda_status(e != cudaSuccess ? e : cudaGetLastError(), "cm_match launch");
}

}  // namespace cm
