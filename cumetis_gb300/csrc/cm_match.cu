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
//   k_match_rounds   queued rows, one warp per row of up to kMatchChunk entries, the
//                    warp following the chain; rows of several chunks are merged
//                    by the last chunk's warp, and a displaced one is queued for
//                    the next round (grid barrier; a round with few chunks runs
//                    on one block), as is the free vertex of a long chain.
//   k_match_finish   match[v] = the partner, or v.
//
// Only an adjacency that is not symmetric can end with an offer that is not
// returned (best[u] = v, best[v] != u), or returned with another weight (the two
// entries of an edge differ).  k_match_finish sees that and the matching is then
// computed again by handshakes (handshake_rounds), whose result is defined for
// such inputs too.
#include <climits>

#include <algorithm>

// The header's row thresholds, which the tuner searches as this source's.
#ifndef CM_SERIAL_DEG
#define CM_SERIAL_DEG 16
#endif
#ifndef CM_MATCH_CHUNK
#define CM_MATCH_CHUNK 256
#endif
#include "cm_match.cuh"

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
// Tail mode (one block runs the remaining rounds) once a round has at most
// kTailChunks row chunks.
#ifndef CM_TAIL_CHUNKS
#define CM_TAIL_CHUNKS 64
#endif
constexpr int kTailChunks = CM_TAIL_CHUNKS;
// Candidates listed for rows of more than kSerialDeg entries (short rows: kTop).
#ifndef CM_FIRST_KEEP_CHUNK
#define CM_FIRST_KEEP_CHUNK 4
#endif
constexpr int kFirstKeepChunk = CM_FIRST_KEEP_CHUNK;
static_assert(kFirstKeepChunk >= 1 && kFirstKeepChunk <= kTop, "CM_FIRST_KEEP_CHUNK: 1 to 4");

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
      const int xs = a.xadj[v];
      short_list<H>(a, v, xs, a.xadj[v + 1] - xs);
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
      const int nch = (a.xadj[v + 1] - a.xadj[v] + kMatchChunk - 1) / kMatchChunk;
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

// The proposals (propose_span); free vertices that need a scan of a long row are
// queued (slot 1).  Bound by latency.  Hashed ties end chains early and leave the
// chip to many short ones: 48 registers for 5 resident blocks per SM and 4
// entries a rescan step (1400 x 1400 grid's matching 269 -> 241 us, R-MAT 22's
// 2026 -> 1991).  Ties by id make few long chains, which want their reads in
// flight together and no spills (a 700 x 700 triangulation: 3.51 ms with those
// settings, 2.95 ms with 8 entries and lists read ahead).
template <bool H>
__global__ void __launch_bounds__(kPrepThreads, H ? 5 : 0) k_match_propose(MatchArgs a) {
  __shared__ int sh_v[kPrepThreads / 32][kSpan];
  int *list = sh_v[threadIdx.x >> 5];
  const bool all = all_eligible(a);
  const int gwarp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  const int n = a.n;
  const long long step = (long long)nwarps * a.span;
  for (long long b0 = (long long)gwarp * a.span; b0 < n; b0 += step) {
    const ChainEnd end =
        propose_span<H, !H, H ? 4 : 8, false>(a, b0, a.span, all, list, nullptr, [&](int v, int xs, int deg) {
          append_scan(a, 1, 1, v >= 0, v, xs, deg);
        });
    if (end != kChainDone || (b0 + step < n && warp_sees_error(a.st))) return;
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
    // Chunks are taken from a ticket: rows and chains differ in length.  No more
    // once a kernel has failed.
    int q = 0;
    if (lane == 0) q = atomicAdd(a.tick + ctr, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    int4 d = q < nchunks ? __ldcg(S.desc + q) : make_int4(0, 0, 0, 0);
    unsigned steps = kChainSteps;  // of this warp in this round
    while (q < nchunks) {
      int qn = 0;
      if (lane == 0) {
        qn = atomicAdd(a.tick + ctr, 1);
        if (ld_relaxed(&st->error) != 0) qn = INT_MAX;
      }
      TopK<H, kTop> r;
      bool mine = true;
      if (d.w >= 0) {
        r = chunk_best<H, kTop, kExact>(a, d.x, d.y, d.z, all, wbuf);
        const int nch = (a.xadj[d.x + 1] - a.xadj[d.x] + kMatchChunk - 1) / kMatchChunk;
        mine = part_done<H, kTop>(a, S, q, d, nch, r);
        if (mine) {
          const int base = __ldcg(S.big_base + d.w);
          r = merge_parts<H, kTop>(a, nch * kTop, [&](int t) { return (size_t)base * kTop + t; });
        }
      }
      qn = __shfl_sync(0xffffffffu, qn, 0);
      const int4 dn = qn < nchunks ? __ldcg(S.desc + qn) : d;
      if (mine && warp_chain<H, ONE_PASS ? kEndless : kQueue>(a, d.x, d.y, d.z, d.w >= 0, r, all, par ^ 1, next,
                                                              &steps, wbuf) != kChainDone)
        break;
      q = qn;
      d = dn;
    }
    trace(round, 3, global_timer_ns());
    if (ONE_PASS) break;
    if (!tail) {
      if (!grid_barrier(st, gridDim.x)) return;
    } else {
      __threadfence();
      if (__syncthreads_or(ld_relaxed(&st->error) != 0)) return;  // one answer for the block
    }
  }
  if (first_thread) st->rounds = round;
  trace(0, 3, global_timer_ns());
  trace(0, 4, (unsigned long long)(round - 1));
}

// The matching of an adjacency that is not symmetric: mutual proposals until no
// pair forms.  Every unmatched vertex points at its most preferred unmatched
// neighbour, and vertices that point at each other are matched; whichever pairs
// are matched first, the outcome is the same.  Rounds over a list of the vertices
// that have to point anew (at first all):
//   point   the first unmatched of the vertex's listed candidates; with none left a
//           lane scans a row of up to kSerialDeg entries, longer rows are queued;
//   scan    the queued rows, by chunks, a new list for each;
//   commit  the pairs;
//   wake    neighbours that point at a vertex matched now go on the next list.
// A vertex is woken through the matched one's row, of up to kMatchChunk entries while
// lists are short and up to kSerialDeg (a lane each) while they are long.  It is missed
// where that row is longer or its own entry has no counterpart: a pass over all
// vertices finds those, in the round after such a row, in every kPassRounds-th (else
// chains that wait for a vertex run one after another: a 1000 x 1000 grid without 0.1%
// of its entries 162 ms, so 43) and when the list is empty.  The work is that of the rows looked at, not rounds times vertices: a
// path in order takes n / 2 rounds of a few vertices each.  Latency: three barriers a
// round, four with queued rows, each phase some dependent trips to L2.  At most
// 4 n + 8 rounds: of any four before the last one matches a pair.
// With GRID all blocks work together (a cooperative launch), and block 0 goes on alone,
// with block barriers, while lists are short (kSoloEntries; the others wait at a grid
// barrier, for kSoloRounds at most); else the calling block is the only one.
// wbuf: the warp's 32 int2 of shared memory.  What other warps write is read fresh.
constexpr int kSoloEntries = 1024, kSoloRounds = 4096, kPassRounds = 6;
constexpr int kSoloPass = 16384;  // vertices that one block passes over
template <bool H, bool GRID>
__device__ void handshake_rounds(const MatchArgs &a, int2 *wbuf) {
  constexpr unsigned full = 0xffffffffu;
  constexpr int kHalf = 8;
  const int lane = threadIdx.x & 31, n = a.n;
  const unsigned below = (1u << lane) - 1u;
  // the proposals' scratch is free: targets, the round of the last listing, the
  // lists; slot 1 for the queued rows
  int *ptr = reinterpret_cast<int *>(a.best), *stamp = ptr + n;
  int *lists[2] = {reinterpret_cast<int *>(a.slot[0].desc), reinterpret_cast<int *>(a.slot[0].desc) + n};
  int *count = a.odd + 2, *search = a.odd + 5;  // [3] each, by round: the list's length, a pass over all is due
  int *solo_end = a.odd + 8;  // the round in which block 0 has stopped to work alone
  const Slot &S = a.slot[1];
  const int block_warps = (int)(blockDim.x >> 5), warp = (int)(threadIdx.x >> 5);
  int gw = warp, nw = block_warps;
  if (GRID) {
    gw += (int)blockIdx.x * block_warps;
    nw *= (int)gridDim.x;
  }
  bool solo = !GRID;
  int alone = 0;  // rounds of block 0 alone, weighted by what a warp has in them: up to 30 us a unit
  auto barrier = [&]() -> bool {
    if (!solo) return grid_barrier(a.st, gridDim.x);
    __threadfence();
    return !__syncthreads_or(ld_relaxed(&a.st->error) != 0);  // one answer for the block
  };
  for (long long v = (long long)gw * 32 + lane, step = (long long)nw * 32; v < n; v += step) {
    a.m2[v] = -1;
    ptr[v] = kNone;
    stamp[v] = 0;
    lists[0][v] = (int)v;
  }
  if (gw == 0 && lane == 0) {
    count[0] = n;
    count[1] = count[2] = 0;
    search[0] = search[1] = search[2] = 0;
    a.big[0] = 0;
    a.tick[0] = 0;
  }
  if (!barrier()) return;
  bool searched = false;  // the last round only made a pass over all vertices
  for (int round = 0;; ++round) {
    const int k = ld_fresh(count + round % 3);
    const bool pass = k == 0 || ld_fresh(search + round % 3) != 0 || round % kPassRounds == kPassRounds - 1;
    if (GRID) {
      const bool small = k > 0 && k <= kSoloEntries && (!pass || n <= kSoloPass);
      if (!solo && small) {  // all have read the counters before block 0 goes on
        if (!barrier()) return;
        if (blockIdx.x != 0) {
          if (!barrier()) return;
          round = ld_fresh(solo_end) - 1;
          searched = false;
          continue;
        }
        solo = true;
        gw = warp;
        nw = block_warps;
        alone = 0;
      } else if (solo && (!small || alone > kSoloRounds)) {
        if (threadIdx.x == 0) *solo_end = round;
        solo = false;
        nw = block_warps * (int)gridDim.x;
        if (!barrier()) return;
        --round;  // this round, together
        continue;
      }
      alone += 1;
    }
    const long long step = (long long)nw * 32;
    const int *list = lists[round & 1];
    int *more = lists[~round & 1], *nmore = count + (round + 1) % 3;
    if (gw == 0 && lane == 0) {
      count[(round + 2) % 3] = 0;
      search[(round + 2) % 3] = 0;
    }
    if (k == 0 && searched) break;
    if ((long long)round > 4ll * n + 8) {
      if (gw == 0 && lane == 0) record_error(a.st, CM_ERR_LIMIT, ERR_SITE_ROUNDS);
      return;
    }
    auto append = [&](bool take, int v) {  // convergent
      const unsigned who = __ballot_sync(full, take);
      if (!who) return;
      int base = 0;
      if (lane == 0) base = atomicAdd(nmore, __popc(who));
      base = __shfl_sync(full, base, 0);
      if (take) more[base + __popc(who & below)] = v;
    };
    if (pass) {  // those whose target is matched, unless they point anew in this round
      for (long long b = (long long)gw * 32; b < n; b += step) {
        const long long v = b + lane;
        bool stale = false;
        if (v < n && ld_fresh(a.m2 + v) < 0 && ld_fresh(stamp + v) != round) {
          const int p = ld_fresh(ptr + v);
          stale = p >= 0 && ld_fresh(a.m2 + p) >= 0;
        }
        if (stale) stamp[v] = round + 1;
        append(stale, (int)v);
      }
    }
    searched = k == 0;
    if (searched) {
      if (!barrier()) return;
      continue;
    }
    // entries of the list a warp takes at a time: few where there are few
    const int per = (int)min(32ll, max(1ll, ((long long)k + nw - 1) / nw));
    const long long stride = (long long)nw * per;
    alone += per;  // (a warp's rows one after another)
    const int wake_deg = k <= n >> 6 ? kMatchChunk : kSerialDeg;  // longest row that wakes

    // ---- point
    for (long long b = (long long)gw * per; b < k; b += stride) {
      const int v = lane < per && b + lane < k ? ld_fresh(list + b + lane) : -1;
      int p = kNone, xs = 0, deg = 0;
      if (v >= 0) {
        xs = a.xadj[v];
        deg = a.xadj[v + 1] - xs;
      }
      if (deg > 0) {
        const int4 q = __ldcg(reinterpret_cast<const int4 *>(a.top) + v);
        const int c[kTop] = {q.x, q.y, q.z, q.w};
        p = kUnknown;
#pragma unroll
        for (int t = kTop - 1; t >= 0; --t)
          if (c[t] < 0 || ld_fresh(a.m2 + c[t]) < 0) p = c[t];
      }
      const bool queue = p == kUnknown && deg > kSerialDeg;
      if (p == kUnknown && !queue) {
        const int hb = hash_base(a, v);
        const long long vw = a.vwgt[v], cap = weight_cap(a, v);
        Cand<H> best;
        for (int j = 0; j < deg; j += kHalf) {  // 8 entries in flight
          int y[kHalf], w[kHalf], yw[kHalf], ym[kHalf];
#pragma unroll
          for (int t = 0; t < kHalf; ++t) {
            y[t] = j + t < deg ? a.adjncy[xs + j + t] : v;
            w[t] = j + t < deg ? a.adjwgt[xs + j + t] : 0;
          }
#pragma unroll
          for (int t = 0; t < kHalf; ++t) {
            yw[t] = a.vwgt[y[t]];
            ym[t] = y[t] != v ? ld_fresh(a.m2 + y[t]) : 0;
          }
#pragma unroll
          for (int t = 0; t < kHalf; ++t) {
            if (ym[t] >= 0 || !pair_fits(cap, vw, yw[t])) continue;
            const Cand<H> e = Cand<H>::make(v, y[t], w[t], hb);
            if (e.better(best)) best = e;
          }
        }
        p = best.id();
      }
      append_scan(a, 1, 0, queue, v, xs, deg);
      if (v >= 0 && !queue) ptr[v] = p;
    }
    if (!barrier()) return;

    // ---- scan
    const int nchunks = (int)(ld_fresh(a.big) & 0xffffffffu);
    alone += nchunks / 32;
    if (nchunks > 0) {
      for (;;) {
        int q = 0;
        if (lane == 0) q = atomicAdd(a.tick, 1);
        q = __shfl_sync(full, q, 0);
        if (q >= nchunks) break;
        const int4 d = __ldcg(S.desc + q);
        TopK<H, kTop> r = chunk_best<H, kTop, kOpen>(a, d.x, d.y, d.z, false, wbuf);
        bool mine = true;
        if (d.w >= 0) {
          const int nch = (a.xadj[d.x + 1] - a.xadj[d.x] + kMatchChunk - 1) / kMatchChunk;
          mine = part_done<H, kTop>(a, S, q, d, nch, r);
          if (mine) {
            const int base = ld_fresh(S.big_base + d.w);
            r = merge_parts<H, kTop>(a, nch * kTop, [&](int t) { return (size_t)base * kTop + t; });
          }
        }
        if (mine && lane == 0) {
          store_top(a, d.x, r);
          ptr[d.x] = r.c[0].id();
        }
      }
      if (!barrier()) return;
    }

    // ---- commit (by either end that is listed: the same words)
    if (gw == 0 && lane == 0) {
      a.big[0] = 0;
      a.tick[0] = 0;
    }
    for (long long i = (long long)gw * 32 + lane; i < k; i += step) {
      const int v = ld_fresh(list + i), p = ld_fresh(ptr + v);
      if (p >= 0 && ld_fresh(ptr + p) == v) {
        a.m2[v] = p;
        a.m2[p] = v;
      }
    }
    if (!barrier()) return;

    // ---- wake
    for (long long b = (long long)gw * per; b < k; b += stride) {
      const int v = lane < per && b + lane < k ? ld_fresh(list + b + lane) : -1;
      const int u = v >= 0 ? ld_fresh(a.m2 + v) : -1;
      // v's row, and u's where u is not listed
      int xx[2] = {u >= 0 ? v : -1, u >= 0 && ld_fresh(stamp + u) != round ? u : -1}, xxs[2], xdeg[2];
#pragma unroll
      for (int end = 0; end < 2; ++end) {
        xxs[end] = xx[end] >= 0 ? a.xadj[xx[end]] : 0;
        xdeg[end] = xx[end] >= 0 ? a.xadj[xx[end] + 1] - xxs[end] : 0;
      }
      // (the stamp: once on a list, though a row may name a vertex twice)
      auto listed = [&](int y) { return atomicExch(stamp + y, round + 1) == round + 1; };
#pragma unroll 1
      for (int end = 0; end < 2; ++end) {
        const int x = end ? xx[1] : xx[0], xs = end ? xxs[1] : xxs[0], deg = end ? xdeg[1] : xdeg[0];
        if (deg > wake_deg) search[(round + 1) % 3] = 1;
        for (int j = 0; deg <= kSerialDeg && j < deg; j += kHalf) {
          int y[kHalf];
          bool waits[kHalf];
#pragma unroll
          for (int t = 0; t < kHalf; ++t) y[t] = j + t < deg ? a.adjncy[xs + j + t] : x;
#pragma unroll
          for (int t = 0; t < kHalf; ++t) {
            const int yp = ld_fresh(ptr + y[t]), ym = ld_fresh(a.m2 + y[t]);
            waits[t] = yp == x && ym < 0;  // (x is matched)
          }
#pragma unroll
          for (int t = 0; t < kHalf; ++t)
            if (waits[t] && !listed(y[t])) more[atomicAdd(nmore, 1)] = y[t];
        }
        unsigned rows = __ballot_sync(full, deg > kSerialDeg && deg <= wake_deg);
        while (rows) {
          const int src = __ffs(rows) - 1;
          rows &= rows - 1;
          const int on = __shfl_sync(full, x, src), s0 = __shfl_sync(full, xs, src), e0 = s0 + __shfl_sync(full, deg, src);
          for (int j0 = s0; j0 < e0; j0 += 32) {
            const int y = j0 + lane < e0 ? a.adjncy[j0 + lane] : on;
            const int yp = ld_fresh(ptr + y), ym = ld_fresh(a.m2 + y);
            append(yp == on && ym < 0 && !listed(y), y);
          }
        }
      }
    }
    if (!barrier()) return;
  }
  for (long long v = (long long)gw * 32 + lane, step = (long long)nw * 32; v < n; v += step)
    if (ld_fresh(a.m2 + v) < 0) a.m2[v] = (int)v;
}

// match[v] from best[]; a proposal that is not returned alike sets odd[0].  With ALONE
// the last block then computes the matching by handshakes itself (a form of its own:
// the registers of that cost the large graphs' kernel occupancy, R-MAT 22 14 -> 31 us).
template <bool H, bool ALONE>
__global__ void __launch_bounds__(kPrepThreads, ALONE ? 0 : 8) k_match_finish(MatchArgs a) {
  bool odd = false;
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < a.n;
       v += (long long)gridDim.x * blockDim.x) {
    const unsigned long long b = a.best[v];
    const int h = best_holder(b);
    const bool mutual = h >= 0 && best_mutual(b, a.best[h], (int)v);
    a.m2[v] = mutual ? h : (int)v;
    odd |= h >= 0 && !mutual;
  }
  if (odd) atomicOr(a.odd, 1);
  if constexpr (ALONE) {
    __shared__ int s_last;
    __shared__ int2 sh_q[kPrepThreads / 32][32];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(a.odd + 1, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (ld_fresh(a.odd) != 0) handshake_rounds<H, false>(a, sh_q[threadIdx.x >> 5]);
  }
}

// The same for large graphs, with every resident block.
template <bool H>
__global__ void __launch_bounds__(kMatchThreads, kMatchMinBlocks) k_match_handshake(MatchArgs a) {
  if (__ldcg(a.odd) == 0) return;
  __shared__ int2 sh_q[kMatchThreads / 32][32];
  handshake_rounds<H, true>(a, sh_q[threadIdx.x >> 5]);
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

int64_t max_chunks(int64_t n, int64_t m) { return m / kMatchChunk + n + 64; }

}  // namespace

size_t match_ws_bytes(int64_t n, int64_t m) {
  const int64_t ch = max_chunks(n, m);
  size_t b = (size_t)n * (8 + 2 * 4 * kTop);                  // best, lists
  b += 2 * ((size_t)n * 4 * 2 + (size_t)ch * 16);             // two slots
  b += (size_t)ch * 4 * kPartInts * kTop;                     // chunk partial lists
  return b + 64 * 256;
}

// Graphs above this many vertices + entries get the handshake kernel behind
// k_match_finish (a launch that returns at once costs 3 us); below it, where that
// kernel would be one block, the last block of k_match_finish does the work (a grid of
// 900 vertices 50 instead of 55 us).
constexpr int64_t kAloneWork = kWorkPerBlock;

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
  a.maxvwgt = maxvwgt;  // with graphs side by side: the smallest cap (all_eligible)
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
  // No row longer than kMatchChunk: the queued rows take one pass and no barrier.
  const bool one_pass = max_deg <= kMatchChunk;
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
  if (alone) {
    if (hash) k_match_finish<true, true><<<vgrid, kPrepThreads, 0, s>>>(a);
    else k_match_finish<false, true><<<vgrid, kPrepThreads, 0, s>>>(a);
  } else {
    if (hash) k_match_finish<true, false><<<vgrid, kPrepThreads, 0, s>>>(a);
    else k_match_finish<false, false><<<vgrid, kPrepThreads, 0, s>>>(a);
  }
  ctx->launches++;
  if (e == cudaSuccess && !alone) {
    e = cudaLaunchCooperativeKernel(hfn, dim3(grid), dim3(kMatchThreads), args, 0, s);
    ctx->launches++;
  }
  stage_end(ctx, CM_STAGE_MATCH, s);
  return cuda_status(e != cudaSuccess ? e : cudaGetLastError(), "cm_match launch");
}

}  // namespace cm
