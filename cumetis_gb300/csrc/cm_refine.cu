// cm_refine.cu -- k-way refinement and projection on the device, and the
// whole partition driver (coarsen -> initial partition -> refine/project per
// level).
//
// Replaces the uncoarsening half of cuMetis_kway_partition (cuMetis.cu:
// 3544-3616): cuMetis_uncoarsen (3494-3514) with cuMetis_findgraphbndinfo
// (3389-3418), Find_real_bnd_info (3236-3262), find_kayparams (3267-3306),
// the bb_segsort of boundary vertices by target part (3406), findcsr
// (3322-3352), Exnode_part1/2 (3436-3488); cuMetis_kway_project / projectback
// (3067-3086); and cuMetis_PartGraph (3622-3664).
//
// One refinement pass, as in the reference (refine_pass = 1, cu:3319):
//   1. part weights pwgts[p] and the balance window of every part,
//      max = (int)(tpwgts * tvwgt * 1.03f), min = (int)(tpwgts * tvwgt / 1.03f)
//      with tpwgts = 1/k (Sum_maxmin_pwgts, cu:3424-3433);
//   2. a vertex is a boundary vertex when the weight of its edges to other
//      parts exceeds the weight to its own part; its target is the part with
//      the largest connection, the lowest such part id, unless no part beats
//      its own (find_kayparams' scan, cu:3290-3298);
//   3. boundary vertices grouped by target part -- here in vertex-id order
//      within a part (a stable counting sort), where the reference's
//      segmented sort leaves equal targets in an unspecified order;
//   4. per target part one block takes its group in order and moves a vertex
//      when both parts stay inside their windows: first the moves towards a
//      higher part id, then (second launch) towards a lower one.
//      Part weights are updated with atomics while the other parts' blocks
//      run, as by the reference's part threads, so concurrent groups see each
//      other's moves in whatever order the hardware interleaves them.
#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <vector>

#include "cm_ctx.h"

namespace cm {
namespace {

constexpr int kRefThreads = 256;          // 8 warps; one warp per vertex
constexpr int kRefWarps = kRefThreads / 32;
constexpr int kSmemParts = 1024;          // per-warp part accumulators in shared memory up to this k
constexpr int kSortBlock = 1024;          // boundary entries per counting-sort block

// Part weights (atomics, shared-memory histogram when k is small).  With a
// coarser level given (cmap, cwhere), the kernel first projects it:
// where[v] = cwhere[cmap[v]] (cuMetis_kway_project fused into the pass).
__global__ void k_part_weights(int n, int *__restrict__ where, const int *__restrict__ vwgt, int nparts,
                               int *__restrict__ pwgts, const int *__restrict__ cmap, const int *__restrict__ cwhere) {
  extern __shared__ int h[];
  const bool sh = nparts <= 8192;
  if (sh)
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
    int p;
    if (cmap) {
      p = cwhere[cmap[v]];
      where[v] = p;
    } else {
      p = where[v];
    }
    if (sh) atomicAdd(&h[p], vwgt[v]);
    else atomicAdd(&pwgts[p], vwgt[v]);
  }
  __syncthreads();
  if (sh)
    for (int i = threadIdx.x; i < nparts; i += blockDim.x)
      if (h[i]) atomicAdd(&pwgts[i], h[i]);
}

// Boundary test and target part of a vertex with at most N entries, by one lane.
template <int N>
__device__ __forceinline__ int lane_target(int xs, int deg, int me, const int *__restrict__ adjncy,
                                           const int *__restrict__ adjwgt, const int *__restrict__ where, bool *bnd) {
  int p[N], w[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    p[i] = i < deg ? adjncy[xs + i] : -1;
    w[i] = i < deg ? adjwgt[xs + i] : 0;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = p[i] >= 0 ? where[p[i]] : -1;
  int mw = 0, ow = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (p[i] == me) mw += w[i];
    else ow += w[i];
  }
  *bnd = ow > mw;
  if (!*bnd) return me;
  int bw = INT_MIN, bp = INT_MAX;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (p[i] < 0) continue;
    int c = 0;
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (p[j] == p[i]) c += w[j];
    if (c > bw || (c == bw && p[i] < bp)) {
      bw = c;
      bp = p[i];
    }
  }
  return bw > mw ? bp : me;
}

// Boundary test and target part of the vertices with at most kLaneDeg entries,
// one lane each (a warp each left 28 of 32 lanes idle on a 5-point mesh: 131 us for
// 1000 x 1000 vertices, now 16); the others are listed, those above kWarpDeg from
// the end of the list backwards.
constexpr int kLaneDeg = 16, kWarpDeg = 1024;
__global__ void __launch_bounds__(kRefThreads)
k_boundary_short(int n, const int *__restrict__ xadj, const int *__restrict__ adjncy, const int *__restrict__ adjwgt,
                 const int *__restrict__ where, int *__restrict__ flag, int *__restrict__ target,
                 int *__restrict__ longer, int *nlonger) {
  const int lane = threadIdx.x & 31;
  const long long gw = (blockIdx.x * (long long)kRefThreads + threadIdx.x) >> 5;
  const long long nw = (long long)gridDim.x * kRefWarps;
  for (long long b0 = gw * 32; b0 < n; b0 += nw * 32) {
    const long long v = b0 + lane;
    int xs = 0, deg = 0, t = 0;
    bool bnd = false;
    if (v < n) {
      xs = xadj[v];
      deg = xadj[v + 1] - xs;
    }
    const bool listed = deg > kLaneDeg;
    if (v < n && !listed) {
      t = where[v];
      if (deg > 0 && deg <= kLaneDeg / 2) t = lane_target<kLaneDeg / 2>(xs, deg, t, adjncy, adjwgt, where, &bnd);
      else if (deg > 0) t = lane_target<kLaneDeg>(xs, deg, t, adjncy, adjwgt, where, &bnd);
      flag[v] = bnd ? 1 : 0;
      target[v] = t;
    }
    const unsigned below = (1u << lane) - 1u;
    const unsigned mid = __ballot_sync(0xffffffffu, listed && deg <= kWarpDeg);
    const unsigned top = __ballot_sync(0xffffffffu, deg > kWarpDeg);
    if (mid | top) {
      int base = 0;
      if (lane == 0 && mid) base = atomicAdd(nlonger, __popc(mid));
      if (lane == 1 && top) base = atomicAdd(nlonger + 1, __popc(top));
      const int bm = __shfl_sync(0xffffffffu, base, 0), bt = __shfl_sync(0xffffffffu, base, 1);
      if (listed && deg <= kWarpDeg) longer[bm + __popc(mid & below)] = (int)v;
      if (deg > kWarpDeg) longer[n - 1 - bt - __popc(top & below)] = (int)v;
    }
  }
}

// Boundary test and target part of one vertex by NT threads (a warp, or the
// block); acc: one zeroed int per part, zero again at the end; red: NT / 32 + 1
// int2 of shared memory (unused by a warp).
template <int NT>
__device__ __forceinline__ void group_target(int v, const int *__restrict__ xadj, const int *__restrict__ adjncy,
                                             const int *__restrict__ adjwgt, const int *__restrict__ where, int *acc,
                                             int2 *red, int *__restrict__ flag, int *__restrict__ target) {
  const int tid = NT == 32 ? threadIdx.x & 31 : threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int xs = xadj[v], xe = xadj[v + 1], me = where[v];
  int mw = 0, ow = 0;
  for (int j = xs + tid; j < xe; j += NT) {
    const int w = adjwgt[j];
    if (where[adjncy[j]] == me) mw += w;
    else ow += w;
  }
  mw = __reduce_add_sync(0xffffffffu, mw);
  ow = __reduce_add_sync(0xffffffffu, ow);
  if (NT > 32) {
    if (lane == 0) red[wid] = make_int2(mw, ow);
    __syncthreads();
    const int2 x = lane < NT / 32 ? red[lane] : make_int2(0, 0);
    mw = __reduce_add_sync(0xffffffffu, x.x);
    ow = __reduce_add_sync(0xffffffffu, x.y);
    __syncthreads();
  }
  const bool bnd = ow > mw;
  int t = me;
  if (bnd) {
    for (int j = xs + tid; j < xe; j += NT) atomicAdd(&acc[where[adjncy[j]]], adjwgt[j]);
    row_sync<NT>();
    int bw = INT_MIN, bp = INT_MAX;
    for (int j = xs + tid; j < xe; j += NT) {
      const int p = where[adjncy[j]];
      const int w = acc[p];
      if (w > bw || (w == bw && p < bp)) {
        bw = w;
        bp = p;
      }
    }
    int wmax = __reduce_max_sync(0xffffffffu, bw);
    int pmin = __reduce_min_sync(0xffffffffu, bw == wmax ? bp : INT_MAX);
    if (NT > 32) {
      if (lane == 0) red[wid] = make_int2(wmax, pmin);
      __syncthreads();
      const int2 x = lane < NT / 32 ? red[lane] : make_int2(INT_MIN, INT_MAX);
      wmax = __reduce_max_sync(0xffffffffu, x.x);
      pmin = __reduce_min_sync(0xffffffffu, x.x == wmax ? x.y : INT_MAX);
    }
    t = wmax > acc[me] ? pmin : me;
    row_sync<NT>();
    for (int j = xs + tid; j < xe; j += NT) acc[where[adjncy[j]]] = 0;
    row_sync<NT>();
  }
  if (tid == 0) {
    flag[v] = bnd ? 1 : 0;
    target[v] = t;
  }
}

// The listed vertices: the longest rows one block each (R-MAT 17: 204 us when one
// warp made the hub's three passes, now 53), then
// the others one warp each (round robin: an R-MAT graph's long rows have
// neighbouring ids).  acc: one zeroed int per part for each warp (shared memory
// when k <= kSmemParts, else a global slice).
template <bool kShared>
__global__ void __launch_bounds__(kRefThreads)
k_boundary(int n, const int *__restrict__ longer, const int *__restrict__ nlonger, const int *__restrict__ xadj,
           const int *__restrict__ adjncy, const int *__restrict__ adjwgt, const int *__restrict__ where, int nparts,
           int *__restrict__ acc_global, int *__restrict__ flag, int *__restrict__ target) {
  extern __shared__ int acc_s[];
  __shared__ int2 red[kRefWarps + 1];
  const int warp = threadIdx.x >> 5;
  const int gw = blockIdx.x * kRefWarps + warp, nw = gridDim.x * kRefWarps;
  const int count = nlonger[0], top = nlonger[1];
  if ((int)blockIdx.x * kRefWarps >= count && (int)blockIdx.x >= top) return;
  int *acc_block = kShared ? acc_s : acc_global + (long long)blockIdx.x * kRefWarps * nparts;
  if (kShared) {
    for (int i = threadIdx.x; i < kRefWarps * nparts; i += kRefThreads) acc_s[i] = 0;
    __syncthreads();
  }
  for (int i = blockIdx.x; i < top; i += gridDim.x)
    group_target<kRefThreads>(longer[n - 1 - i], xadj, adjncy, adjwgt, where, acc_block, red, flag, target);
  for (int i = gw; i < count; i += nw)
    group_target<32>(longer[i], xadj, adjncy, adjwgt, where, acc_block + warp * nparts, red, flag, target);
}

// Boundary list in vertex order (decoupled look-back over 2048-vertex tiles), and
// the entries of every target part in every kSortBlock entries of the list (the
// first step of the stable counting sort by target: counts, prefix over blocks,
// in-order scatter).  *d_nb = the list's length.
constexpr int kScanThreads = 256, kScanItems = 8;
__global__ void __launch_bounds__(kScanThreads)
k_boundary_list(const int *__restrict__ flags, const int *__restrict__ target, int n, int nparts,
                int *__restrict__ bnd_v, int *__restrict__ bnd_t, int *__restrict__ bhist, int *__restrict__ d_nb,
                unsigned long long *lb, DevStatus *st) {
  __shared__ int s_tile;
  __shared__ unsigned long long s_warp[kScanThreads / 32];
  __shared__ unsigned long long s_excl;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tile = (int)atomicAdd(lb, 1ull);
  __syncthreads();
  const int tile = s_tile;
  const long long base = (long long)tile * kScanThreads * kScanItems + (long long)threadIdx.x * kScanItems;
  int v[kScanItems];
  unsigned long long sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = base + i < n ? flags[base + i] : 0;
    sum += (unsigned)v[i];
  }
  const unsigned long long inc = warp_inclusive_scan_u64(sum);
  if (lane == 31) s_warp[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const unsigned long long x = lane < kScanThreads / 32 ? s_warp[lane] : 0ull;
    const unsigned long long xi = warp_inclusive_scan_u64(x);
    const unsigned long long agg = __shfl_sync(0xffffffffu, xi, kScanThreads / 32 - 1);
    if (lane < kScanThreads / 32) s_warp[lane] = xi - x;
    const unsigned long long ex = lookback_exclusive(lb, tile, agg, st);
    if (lane == 0) s_excl = ex;
  }
  __syncthreads();
  long long run = (long long)(s_excl + s_warp[wid] + inc - sum);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i >= n) break;
    if (v[i]) {
      const int t = target[base + i];
      bnd_v[run] = (int)(base + i);
      bnd_t[run] = t;
      atomicAdd(&bhist[run / kSortBlock * nparts + t], 1);
      ++run;
    }
    if (base + i == n - 1) *d_nb = (int)run;
  }
}

// Prefix of every part's counts over the blocks (one warp a part), then by the
// last block to finish: pstart[t], the exclusive prefix of the parts' totals, a
// second count of the parts' weights (k_moves), and the parts' balance windows from
// the total vertex weight (Sum_maxmin_pwgts).
constexpr int kOffsetThreads = 256;
__global__ void __launch_bounds__(kOffsetThreads)
k_sort_offsets(const int *__restrict__ d_nb, int nparts, float tp, const int *__restrict__ pwgts,
               int *__restrict__ bhist, int *pcount, int *__restrict__ pstart, int *__restrict__ maxw,
               int *__restrict__ minw, int *__restrict__ left, unsigned *done) {
  __shared__ int scan[kOffsetThreads / 32 + 1];
  __shared__ bool s_last;
  __shared__ unsigned long long s_tot;
  const int lane = threadIdx.x & 31;
  const int nb = *d_nb;
  const int nblocks = (nb + kSortBlock - 1) / kSortBlock;
  const int warps = gridDim.x * (kOffsetThreads / 32);
  for (int t = blockIdx.x * (kOffsetThreads / 32) + (threadIdx.x >> 5); t < nparts; t += warps) {
    int run = 0;
    for (int b0 = 0; b0 < nblocks; b0 += 32) {
      const int b = b0 + lane;
      const int c = b < nblocks ? bhist[(size_t)b * nparts + t] : 0;
      const int inc = warp_inclusive_scan_i32(c);
      if (b < nblocks) bhist[(size_t)b * nparts + t] = run + inc - c;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) pcount[t] = run;
  }
  __threadfence();
  if (threadIdx.x == 0) s_tot = 0ull;
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  int carry = 0;
  long long wt = 0;
  for (int b = 0; b < nparts; b += kOffsetThreads) {
    const int t = b + threadIdx.x;
    const int c = t < nparts ? __ldcg(pcount + t) : 0;
    int tot;
    const int ex = block_exclusive_scan<kOffsetThreads>(c, scan, &tot);
    if (t < nparts) {
      pstart[t] = carry + ex;
      left[t] = pwgts[t];  // the moves' second count
      wt += pwgts[t];
    }
    carry += tot;
  }
  if (threadIdx.x == 0) pstart[nparts] = carry;
  atomicAdd(&s_tot, (unsigned long long)wt);
  __syncthreads();
  const int tvwgt = (int)(long long)s_tot;
  const float ub = 1.03f;
  for (int i = threadIdx.x; i < nparts; i += kOffsetThreads) {
    maxw[i] = (int)(__fmul_rn(__fmul_rn(tp, (float)tvwgt), ub));
    minw[i] = (int)(__fdiv_rn(__fmul_rn(tp, (float)tvwgt), ub));
  }
}

// One warp per block of kSortBlock entries, in order: an entry's place is its
// part's start + the block's offset for the part + its rank among the part's
// earlier entries in the block (running counts in shared memory up to
// kSmemParts parts, so that the steps do not wait for global reads of each
// other's counts).  The sorted record holds what the moves need -- vertex,
// weight, part -- so that the walks read memory in order.
__global__ void __launch_bounds__(32)
k_sort_scatter(const int *__restrict__ d_nb, const int *__restrict__ bnd_v, const int *__restrict__ bnd_t, int nparts,
               int *__restrict__ bhist, const int *__restrict__ pstart, const int *__restrict__ vwgt,
               const int *__restrict__ where, int4 *__restrict__ sorted) {
  extern __shared__ int s_cnt[];
  const int nb = *d_nb;
  const int lane = threadIdx.x & 31;
  const long long b = blockIdx.x;
  const long long lo = b * kSortBlock, hi = min((long long)nb, lo + kSortBlock);
  if (lo >= hi) return;
  int *cnt = bhist + b * nparts;
  if (nparts <= kSmemParts) {
    for (int t = lane; t < nparts; t += 32) s_cnt[t] = cnt[t] + pstart[t];
    __syncwarp();
  }
  constexpr int kAhead = 4;  // steps whose loads are in flight together
  for (long long i0 = lo; i0 < hi; i0 += 32 * kAhead) {
    int t[kAhead], v[kAhead], vw[kAhead], me[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const long long i = i0 + 32 * u + lane;
      t[u] = i < hi ? bnd_t[i] : -1;
      v[u] = i < hi ? bnd_v[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      vw[u] = t[u] >= 0 ? vwgt[v[u]] : 0;
      me[u] = t[u] >= 0 ? where[v[u]] : 0;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const unsigned m = __match_any_sync(0xffffffffu, t[u]);
      const int rank = __popc(m & ((1u << lane) - 1));
      int base = 0;
      if (t[u] >= 0) base = nparts <= kSmemParts ? s_cnt[t[u]] : pstart[t[u]] + cnt[t[u]];
      __syncwarp();
      if (t[u] >= 0) {
        sorted[base + rank] = make_int4(v[u], vw[u], me[u], 0);
        if (rank == 0) {
          if (nparts <= kSmemParts) s_cnt[t[u]] = base + __popc(m);
          else cnt[t[u]] += __popc(m);
        }
      }
      __syncwarp();
    }
  }
}

// The group of target part `to` (blockIdx.x) in order (Exnode_part1 when kUp:
// moves to a higher part id; Exnode_part2 otherwise): a vertex moves when part
// to stays within [tomin, tomax] with it and its own part within its window
// without it, given the moves before it.
//
// A walk vertex by vertex waits for several memory trips each (10.7 ms a phase
// for an R-MAT 17 bisection, 0.49 ms for a 1000 x 1000 grid in 64 parts; a whole
// pass went from 17.4 to 0.53 ms and from 0.86 to 0.26 ms; with the boundary test
// by row length it takes 0.28 and 0.13), although most
// stretches of a group are moved or refused as a whole.  So the block takes
// kMoveThreads records at a time and settles them together when it can:
//   - everyone moves: the records' weights are added up by part, in a table of the
//     block; if every part stays above its lower limit (and was not above its upper
//     one before) and the sum fits part to, each vertex alone was allowed in order,
//     for weights >= 0;
//   - everyone is refused: nobody fits as the weights are now, and refusals
//     change no weight.
// Else the first warp settles the records in order, 32 at a time, by stretches:
// the longest prefix that moves, then the longest that is refused.  Either way
// the outcome for two parts is that of the walk.  With more parts the blocks race
// as the reference's threads do, but no limit is crossed.  Weight is first taken
// from a second count of the part (left), where it is put back if that falls below
// the lower limit, and only then from its weight: pwgts never shows room that may
// go again, and left never exceeds it.  Only the part's own block adds to it, after a
// look at its weight, which the others can only lower.  A part that another block
// took from first leaves its records to the walk.  (Compare-and-swap on pwgts alone
// keeps the limits too, but 64 blocks that take from the same parts wait for one
// another: projection and pass of a 1000 x 1000 grid in 64 parts 170 us.)
constexpr int kMoveThreads = 512, kMoveSlots = 2 * kMoveThreads;

// Takes w out of part p while it keeps at least lo; whether it did.  left: null
// where no other block takes from the part, and the caller has looked already.
__device__ __forceinline__ bool take_weight(int *pwgts, int *left, int p, int w, int lo) {
  if (left && atomicSub(left + p, w) - w < lo) {
    atomicAdd(left + p, w);
    return false;
  }
  atomicSub(pwgts + p, w);
  return true;
}
// Adds w to part p: to its weight first.
__device__ __forceinline__ void give_weight(int *pwgts, int *left, int p, int w) {
  atomicAdd(pwgts + p, w);
  if (!left) return;
  __threadfence();
  atomicAdd(left + p, w);
}

template <bool kUp>
__global__ void __launch_bounds__(kMoveThreads)
k_moves(const int *__restrict__ pstart, const int4 *__restrict__ sorted, const int *__restrict__ maxw,
        const int *__restrict__ minw, int *pwgts, int *left, int *where, unsigned long long *moves) {
  __shared__ int4 s_rec[kMoveThreads];
  __shared__ int s_part[kMoveSlots], s_out[kMoveSlots];  // by slot: a source part, the weight that leaves it
  __shared__ int s_sum, s_pto;
  const int to = blockIdx.x;
  if (gridDim.x <= 2) left = nullptr;  // two parts: nobody else takes from the same part
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tomax = maxw[to], tomin = minw[to];
  const int i0 = pstart[to], i1 = pstart[to + 1];
  volatile int *pw = pwgts;
  unsigned long long nm = 0;
  const int4 none = make_int4(-1, 0, to, 0);
  int4 next = i0 + (int)threadIdx.x < i1 ? sorted[i0 + threadIdx.x] : none;
  for (int b = i0; b < i1; b += kMoveThreads) {
    int4 r = next;
    next = b + kMoveThreads + (int)threadIdx.x < i1 ? sorted[b + kMoveThreads + threadIdx.x] : none;
    const int me = r.z, vw = r.y;
    // me == to would add and remove the same weight: a no-op move, skipped
    // (the reference applies it, leaving a transient in pwgts[me]).
    const bool cand = kUp ? me < to : me > to;
    if (threadIdx.x == 0) s_pto = pw[to];  // one value for all: other blocks may change it
    if (!__syncthreads_or(cand)) continue;
    const int pto = s_pto, pme = cand ? pw[me] : 0;
    const int lo = cand ? minw[me] : 0, hi = cand ? maxw[me] : 0;
    const bool fits = cand && pto + vw >= tomin && pto + vw <= tomax && pme - vw >= lo && pme - vw <= hi;
    if (!__syncthreads_or(fits)) continue;  // everyone is refused
    const bool plain = !cand || (vw >= 0 && vw < (1 << 20) && fits && pme <= hi);
    if (__syncthreads_and(plain)) {
      for (int i = threadIdx.x; i < kMoveSlots; i += kMoveThreads) {
        s_part[i] = -1;
        s_out[i] = 0;
      }
      if (threadIdx.x == 0) s_sum = 0;
      __syncthreads();
      // The record's part's slot: at most kMoveThreads parts in twice as many slots.
      // The records of a warp whose source is one part come together (with two parts
      // all do).
      int slot = me & (kMoveSlots - 1);
      const int sum = __reduce_add_sync(0xffffffffu, cand ? vw : 0);  // below 2^29 for the whole block
      const unsigned some = __ballot_sync(0xffffffffu, cand);
      const int first = __ffs(some) - 1, part = __shfl_sync(0xffffffffu, me, first & 31);
      const bool alike = __all_sync(0xffffffffu, !cand || me == part);
      if (cand && (!alike || lane == first)) {
        for (;;) {
          const int p = atomicCAS(&s_part[slot], -1, me);
          if (p == -1 || p == me) break;
          slot = (slot + 1) & (kMoveSlots - 1);
        }
        atomicAdd(&s_out[slot], alike ? sum : vw);
      }
      if (lane == first) atomicAdd(&s_sum, sum);
      if (alike) slot = __shfl_sync(0xffffffffu, slot, first & 31);
      __syncthreads();
      bool room = (long long)pto + s_sum <= tomax;
      for (int i = threadIdx.x; i < kMoveSlots; i += kMoveThreads)
        if (s_part[i] >= 0) room = room && pw[s_part[i]] - s_out[i] >= minw[s_part[i]];
      if (__syncthreads_and(room)) {
        for (int i = threadIdx.x; i < kMoveSlots; i += kMoveThreads) {
          if (s_part[i] >= 0 && !take_weight(pwgts, left, s_part[i], s_out[i], minw[s_part[i]])) {
            atomicSub(&s_sum, s_out[i]);
            s_out[i] = -1;  // another block came first
          }
        }
        __syncthreads();
        const bool moved = cand && s_out[slot] >= 0;
        if (moved) {
          where[r.x] = to;
          ++nm;
          r.z = to;  // settled
        }
        if (threadIdx.x == 0) {
          give_weight(pwgts, left, to, s_sum);
          __threadfence();
        }
        if (__syncthreads_and(!cand || moved)) continue;
      }
    }
    s_rec[threadIdx.x] = r;
    __threadfence();
    __syncthreads();
    if (warp == 0) {
      for (int c = 0; c < kMoveThreads && b + c < i1; c += 32) {
        const int4 x = s_rec[c + lane];
        unsigned open = __ballot_sync(0xffffffffu, kUp ? x.z < to : x.z > to);
        while (open) {
          const bool mine = open >> lane & 1u;
          const int p = pw[to], q = mine ? pw[x.z] : 0;
          const int qlo = mine ? minw[x.z] : 0, qhi = mine ? maxw[x.z] : 0;
          // weights before each vertex if all of `open` move
          int before = 0, gone = 0;
          for (int j = 0; j < 32; ++j) {
            const int wj = __shfl_sync(0xffffffffu, x.y, j), mj = __shfl_sync(0xffffffffu, x.z, j);
            if ((open >> j & 1u) && j < lane) {
              before += wj;
              if (mj == x.z) gone += wj;
            }
          }
          const int pt = p + before + x.y, pm = q - gone - x.y;
          const bool ok = pt >= tomin && pt <= tomax && pm >= qlo && pm <= qhi;
          const unsigned bad = __ballot_sync(0xffffffffu, mine && !ok);
          const unsigned go = bad ? open & ((1u << (__ffs(bad) - 1)) - 1u) : open;
          if (go) {
            bool moved = go >> lane & 1u;
            if (moved) {
              // (false: another block came first)
              moved = take_weight(pwgts, left, x.z, x.y, x.y > 0 ? qlo : INT_MIN);
            }
            const int sum = __reduce_add_sync(0xffffffffu, moved ? x.y : 0);
            if (lane == 0 && sum) give_weight(pwgts, left, to, sum);
            if (moved) {
              where[x.x] = to;
              ++nm;
            }
            open &= ~go;
            __threadfence();
            __syncwarp();
          } else {
            // the first is refused, and with it everyone up to the next that fits as things are
            const bool fit = mine && p + x.y >= tomin && p + x.y <= tomax && q - x.y >= qlo && q - x.y <= qhi;
            const unsigned yes = __ballot_sync(0xffffffffu, fit) & ~(open & (0u - open));
            open = yes ? open & ~((1u << (__ffs(yes) - 1)) - 1u) : 0u;
          }
        }
      }
    }
    __syncthreads();
  }
  const int n32 = (int)__reduce_add_sync(0xffffffffu, (unsigned)nm);
  if (lane == 0 && n32) atomicAdd(moves, (unsigned long long)n32);
}

__global__ void k_project(int n, const int *__restrict__ cmap, const int *__restrict__ cwhere,
                          int *__restrict__ where) {
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x)
    where[v] = cwhere[cmap[v]];
}

// Sum of weights of cut entries (each undirected cut edge counted twice).
__global__ void k_cut(int n, const int *__restrict__ xadj, const int *__restrict__ adjncy,
                      const int *__restrict__ adjwgt, const int *__restrict__ where, unsigned long long *out) {
  const int lane = threadIdx.x & 31;
  const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  long long s = 0;
  for (long long v = gw; v < n; v += nw) {
    const int me = where[v];
    for (int j = xadj[v] + lane; j < xadj[v + 1]; j += 32)
      if (where[adjncy[j]] != me) s += adjwgt[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0 && s) atomicAdd(out, (unsigned long long)s);
}

struct RefineWs {
  int *pwgts, *left, *maxw, *minw, *flag, *target, *bnd_v, *bnd_t, *bhist, *pcount, *pstart, *acc;
  int4 *sorted;  // boundary records (vertex, weight, part, 0) by target part
  unsigned long long *counters;  // [0] = moves, [1] = cut
  // cleared at the start of a pass, as one block: part weights, the list's
  // length and the offsets kernel's block count, look-back words, counts
  char *clear;
  int *nb;
  unsigned *done;
  unsigned long long *lb;
  size_t acc_ints;
};

int grid_warps(cm_ctx *ctx) { return ctx->num_sms * 8 * kRefWarps; }

size_t pad256(size_t b) { return (b + 255) & ~(size_t)255; }
// Bytes of the cleared block for a graph of n vertices, counts included.
size_t clear_bytes(int64_t n, int nparts) {
  const int64_t nblocks = (n + kSortBlock - 1) / kSortBlock + 1;
  return pad256((size_t)nparts * 4) + 256 + pad256((size_t)(n / (kScanThreads * kScanItems) + 4) * 8) +
         pad256((size_t)nblocks * nparts * 4);
}

size_t refine_ws_bytes(cm_ctx *ctx, int64_t n, int nparts) {
  size_t b = 0;
  b += (size_t)(3 * nparts + 2 * (nparts + 1)) * 4 + 6 * 256;
  b += (size_t)(8 * n + 8) * 4 + 6 * 256;
  b += clear_bytes(n, nparts) + 256;
  if (nparts > kSmemParts) b += (size_t)grid_warps(ctx) * nparts * 4 + 256;
  return b + 4096;
}

int take_refine_ws(cm_ctx *ctx, int64_t n, int nparts, RefineWs &w) {
  w.maxw = (int *)ws_take(ctx, (size_t)nparts * 4);
  w.minw = (int *)ws_take(ctx, (size_t)nparts * 4);
  w.left = (int *)ws_take(ctx, (size_t)nparts * 4);
  w.pcount = (int *)ws_take(ctx, (size_t)(nparts + 1) * 4);
  w.pstart = (int *)ws_take(ctx, (size_t)(nparts + 1) * 4);
  w.flag = (int *)ws_take(ctx, (size_t)n * 4 + 4);
  w.target = (int *)ws_take(ctx, (size_t)n * 4 + 4);
  w.bnd_v = (int *)ws_take(ctx, (size_t)n * 4 + 4);
  w.bnd_t = (int *)ws_take(ctx, (size_t)n * 4 + 4);
  w.sorted = (int4 *)ws_take(ctx, (size_t)n * 16 + 16);
  w.clear = (char *)ws_take(ctx, clear_bytes(n, nparts));
  w.acc_ints = nparts > kSmemParts ? (size_t)grid_warps(ctx) * nparts : 0;
  w.acc = w.acc_ints ? (int *)ws_take(ctx, w.acc_ints * 4) : nullptr;
  w.counters = (unsigned long long *)ws_take(ctx, 64);
  if (!w.maxw || !w.minw || !w.left || !w.pcount || !w.pstart || !w.flag || !w.target || !w.bnd_v || !w.bnd_t || !w.sorted ||
      !w.clear || (w.acc_ints && !w.acc) || !w.counters)
    return cm_fail(CM_ERR_NOMEM, "refine: workspace too small");
  return CM_OK;
}

// One refinement pass over level graph g (device) with partition where.
int refine_pass(cm_ctx *ctx, const cm_graph &g, int nparts, int32_t *where, RefineWs &w, cudaStream_t s,
                const int32_t *proj_cmap = nullptr, const int32_t *proj_cwhere = nullptr) {
  const int n = g.nvtxs;
  if (n == 0) return CM_OK;
  const int sms = ctx->num_sms;
  // the cleared block, laid out for this graph's size
  char *c = w.clear;
  w.pwgts = (int *)c;
  c += pad256((size_t)nparts * 4);
  w.nb = (int *)c;
  w.done = (unsigned *)c + 1;
  c += 256;
  w.lb = (unsigned long long *)c;
  c += pad256((size_t)(n / (kScanThreads * kScanItems) + 4) * 8);
  w.bhist = (int *)c;
  cudaMemsetAsync(w.clear, 0, clear_bytes(n, nparts), s);
  const size_t hsh = nparts <= 8192 ? (size_t)nparts * 4 : 0;
  const int vblocks = std::min(sms * 4, n / 256 + 1);
  k_part_weights<<<vblocks, 256, hsh, s>>>(n, where, g.vwgt, nparts, w.pwgts, proj_cmap, proj_cwhere);
  const int bblocks = std::min(sms * 8, n / kRefThreads + 1);
  int *longer = w.bnd_v, *nlonger = w.nb + 2;  // listed until the boundary list is made
  k_boundary_short<<<bblocks, kRefThreads, 0, s>>>(n, g.xadj, g.adjncy, g.adjwgt, where, w.flag, w.target, longer,
                                                   nlonger);
  const int lblocks = (int)std::min<int64_t>(sms * 8, g.nedges / (kLaneDeg + 1) / kRefWarps + 1);
  if (nparts <= kSmemParts) {
    const size_t sm = (size_t)kRefWarps * nparts * 4;
    if (sm > 48 * 1024)
      cudaFuncSetAttribute(k_boundary<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_boundary<true><<<lblocks, kRefThreads, sm, s>>>(n, longer, nlonger, g.xadj, g.adjncy, g.adjwgt, where, nparts,
                                                     nullptr, w.flag, w.target);
  } else {
    cudaMemsetAsync(w.acc, 0, w.acc_ints * 4, s);
    k_boundary<false><<<lblocks, kRefThreads, 0, s>>>(n, longer, nlonger, g.xadj, g.adjncy, g.adjwgt, where, nparts,
                                                     w.acc, w.flag, w.target);
  }
  const int scan_tiles = (n + kScanThreads * kScanItems - 1) / (kScanThreads * kScanItems);
  k_boundary_list<<<scan_tiles, kScanThreads, 0, s>>>(w.flag, w.target, n, nparts, w.bnd_v, w.bnd_t, w.bhist, w.nb,
                                                      w.lb, ctx->d_status);
  const int sort_blocks = (n + kSortBlock - 1) / kSortBlock;
  // tpwgts = 1.0 / nparts rounded to float, as cuMetis_set_graph_admin stores it (cu:384)
  k_sort_offsets<<<std::min(sms, (nparts + 7) / 8), kOffsetThreads, 0, s>>>(
      w.nb, nparts, (float)(1.0 / nparts), w.pwgts, w.bhist, w.pcount, w.pstart, w.maxw, w.minw, w.left, w.done);
  k_sort_scatter<<<sort_blocks, 32, nparts <= kSmemParts ? nparts * 4 : 0, s>>>(
      w.nb, w.bnd_v, w.bnd_t, nparts, w.bhist, w.pstart, g.vwgt, where, w.sorted);
  k_moves<true><<<nparts, kMoveThreads, 0, s>>>(w.pstart, w.sorted, w.maxw, w.minw, w.pwgts, w.left, where,
                                                w.counters);
  k_moves<false><<<nparts, kMoveThreads, 0, s>>>(w.pstart, w.sorted, w.maxw, w.minw, w.pwgts, w.left, where,
                                                 w.counters);
  ctx->launches += 8;
  return check_launch(ctx, "refine");
}

int edge_cut_dev(cm_ctx *ctx, const cm_graph &g, const int32_t *where, unsigned long long *d_out, int64_t *cut,
                 cudaStream_t s) {
  cudaMemsetAsync(d_out, 0, 8, s);
  k_cut<<<ctx->num_sms * 8, 256, 0, s>>>(g.nvtxs, g.xadj, g.adjncy, g.adjwgt, where, d_out);
  ctx->launches++;
  unsigned long long h = 0;
  int rc = cuda_status(cudaMemcpyAsync(&h, d_out, 8, cudaMemcpyDeviceToHost, s), "cut readback");
  if (!rc) rc = stream_wait(ctx, s, "cut sync");
  if (!rc) *cut = (int64_t)(h / 2);
  return rc;
}

double ms_since(std::chrono::steady_clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

}  // namespace
}  // namespace cm

using namespace cm;

extern "C" int cm_refine_kway(cm_ctx *ctx, const cm_graph *g_dev, int32_t nparts, int32_t *d_where,
                              int64_t *moves, void *stream) {
  if (!ctx || !g_dev || !d_where || nparts < 1 || g_dev->nvtxs < 0)
    return cm_fail(CM_ERR_INVALID, "cm_refine_kway: bad arguments");
  int rc = set_device(ctx);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  ws_reset(ctx);
  if ((rc = ws_ensure(ctx, refine_ws_bytes(ctx, g_dev->nvtxs, nparts)))) return rc;
  RefineWs w;
  if ((rc = take_refine_ws(ctx, g_dev->nvtxs, nparts, w))) return rc;
  cudaMemsetAsync(w.counters, 0, 64, s);
  if ((rc = refine_pass(ctx, *g_dev, nparts, d_where, w, s))) return rc;
  if ((rc = take_device_error(ctx, s))) return rc;
  if (moves) {
    unsigned long long h = 0;
    if ((rc = cuda_status(cudaMemcpyAsync(&h, w.counters, 8, cudaMemcpyDeviceToHost, s), "moves readback")) ||
        (rc = stream_wait(ctx, s, "moves sync")))
      return rc;
    *moves = (int64_t)h;
  }
  return CM_OK;
}

extern "C" int cm_project(cm_ctx *ctx, int32_t n, const int32_t *d_cmap, const int32_t *d_cwhere, int32_t *d_where,
                          void *stream) {
  if (!ctx || n < 0 || (n > 0 && (!d_cmap || !d_cwhere || !d_where)))
    return cm_fail(CM_ERR_INVALID, "cm_project: bad arguments");
  int rc = set_device(ctx);
  if (rc) return rc;
  if (n == 0) return CM_OK;
  k_project<<<ctx->num_sms * 4, 256, 0, (cudaStream_t)stream>>>(n, d_cmap, d_cwhere, d_where);
  ctx->launches++;
  return check_launch(ctx, "project");
}

extern "C" void cm_part_default_params(cm_part_params *p) {
  if (!p) return;
  p->seed = 1;
  // Hash-ordered ties: on unit-weight meshes the lowest-id order makes long chains
  // of displaced proposals, hashed ties end them early; both give deterministic
  // heavy-edge matchings.
  p->match_mode = CM_MATCH_HEM_HASH;
  p->refine_passes = 1;
  p->coarsen_to = 0;
}

// Initial partition of the hierarchy's coarsest graph on the host, then per
// level, coarsest to finest, projection and refinement on the context's
// stream (cuMetis_kway_partition after cuMetis_coarsen, cu:3544-3616).  Takes
// the hierarchy (frees it); part receives the finest level's partition.
int part_hierarchy(cm_ctx *ctx, cm_hierarchy *h, int32_t nparts, const cm_part_params &P, int32_t *part,
                   int32_t *objval, cm_part_stats *stats) {
  cm_part_stats S = stats ? *stats : cm_part_stats{};
  int rc = set_device(ctx);
  if (rc) {
    cm_hierarchy_free(h);
    return rc;
  }
  cudaStream_t s = ctx->stream;
  const int32_t nvtxs = h->levels[0].g.nvtxs;
  auto t0 = std::chrono::steady_clock::now();
  const int L = cm_hierarchy_levels(h);
  S.levels = L;
  std::vector<cm_graph> lg(L);
  std::vector<const int32_t *> lcmap(L);
  for (int l = 0; l < L; ++l) cm_hierarchy_level(h, l, &lg[l], &lcmap[l], nullptr);
  S.coarsest_nvtxs = lg[L - 1].nvtxs;

  // Initial partition of the coarsest graph on the host.
  t0 = std::chrono::steady_clock::now();
  cm_graph coarsest{};
  if ((rc = cm_hierarchy_copy_level(h, L - 1, &coarsest, nullptr, nullptr))) {
    cm_hierarchy_free(h);
    return rc;
  }
  std::vector<int32_t> cwhere(std::max(coarsest.nvtxs, 1));
  int32_t initobj = 0;
  rc = cm_initial_partition(&coarsest, nparts, (uint32_t)P.seed, cwhere.data(), &initobj);
  cm_graph_free(&coarsest);
  if (rc) {
    cm_hierarchy_free(h);
    return rc;
  }
  S.init_ms = ms_since(t0);
  S.initial_cut = initobj;

  // Refinement and projection, coarsest to finest.
  t0 = std::chrono::steady_clock::now();
  int64_t total_n = 0;
  for (int l = 0; l < L; ++l) total_n += lg[l].nvtxs;
  int32_t *wbuf = nullptr;
  if ((rc = cuda_status(cudaMallocFromPoolAsync((void **)&wbuf, (size_t)std::max<int64_t>(total_n, 1) * 4, ctx->pool, s), "where alloc"))) {
    cm_hierarchy_free(h);
    return rc;
  }
  std::vector<int32_t *> wl(L);
  {
    int64_t off = 0;
    for (int l = 0; l < L; ++l) {
      wl[l] = wbuf + off;
      off += lg[l].nvtxs;
    }
  }
  auto finish = [&](int code) {
    cudaFreeAsync(wbuf, s);
    stream_wait(ctx, s, "free");
    cm_hierarchy_free(h);
    return code;
  };
  ws_reset(ctx);
  if ((rc = ws_ensure(ctx, refine_ws_bytes(ctx, nvtxs, nparts)))) return finish(rc);
  RefineWs w;
  if ((rc = take_refine_ws(ctx, nvtxs, nparts, w))) return finish(rc);
  cudaMemsetAsync(w.counters, 0, 64, s);
  cudaMemcpyAsync(wl[L - 1], cwhere.data(), (size_t)lg[L - 1].nvtxs * 4, cudaMemcpyHostToDevice, s);
  const int passes = std::max(1, P.refine_passes);
  for (int l = L - 1; l >= 0; --l) {
    // the first pass of a finer level projects the coarser partition itself
    for (int p = 0; p < passes; ++p) {
      const bool proj = l < L - 1 && p == 0;
      if ((rc = refine_pass(ctx, lg[l], nparts, wl[l], w, s, proj ? lcmap[l] : nullptr, proj ? wl[l + 1] : nullptr)))
        return finish(rc);
    }
  }
  if ((rc = take_device_error(ctx, s))) return finish(rc);
  int64_t cut = 0;
  if ((rc = edge_cut_dev(ctx, lg[0], wl[0], w.counters + 1, &cut, s))) return finish(rc);
  unsigned long long moves = 0;
  cudaMemcpyAsync(&moves, w.counters, 8, cudaMemcpyDeviceToHost, s);
  if ((rc = cuda_status(cudaMemcpyAsync(part, wl[0], (size_t)nvtxs * 4, cudaMemcpyDeviceToHost, s), "part readback")))
    return finish(rc);
  if ((rc = stream_wait(ctx, s, "part sync"))) return finish(rc);
  S.uncoarsen_ms = ms_since(t0);
  S.moves = (int64_t)moves;
  S.edge_cut = cut;
  if (objval) *objval = (int32_t)cut;
  if (stats) *stats = S;
  return finish(CM_OK);
}

extern "C" int cm_part_graph(cm_ctx *ctx, int32_t nvtxs, const int32_t *xadj, const int32_t *adjncy,
                             const int32_t *vwgt, const int32_t *adjwgt, int32_t nparts, const float *tpwgts,
                             const float *ubvec, int32_t *objval, int32_t *part, const cm_part_params *params,
                             cm_part_stats *stats) {
  (void)tpwgts;  // accepted and ignored, as by the reference (cu:370-394)
  (void)ubvec;
  if (!ctx || nvtxs < 0 || !part || nparts < 1 || (nvtxs > 0 && (!xadj || xadj[nvtxs] < 0 || (xadj[nvtxs] > 0 && !adjncy))))
    return cm_fail(CM_ERR_INVALID, "cm_part_graph: bad arguments");
  cm_part_params P;
  cm_part_default_params(&P);
  if (params) P = *params;
  const auto t_all = std::chrono::steady_clock::now();
  cm_part_stats S{};
  if (nvtxs == 0 || nparts == 1) {
    for (int i = 0; i < nvtxs; ++i) part[i] = 0;
    if (objval) *objval = 0;
    if (stats) *stats = S;
    return CM_OK;
  }
  int rc = set_device(ctx);
  if (rc) return rc;
  cudaStream_t s = ctx->stream;  // the context's own stream: concurrent contexts overlap
  const int64_t m = xadj[nvtxs];
  // Unit weights where the caller passes none (cuMetis_set_graph, cu:479-503).
  std::vector<int32_t> uv, ue;
  if (!vwgt) {
    uv.assign(nvtxs, 1);
    vwgt = uv.data();
  }
  if (!adjwgt) {
    ue.assign(std::max<int64_t>(m, 1), 1);
    adjwgt = ue.data();
  }
  cm_graph hg{nvtxs, (int32_t)m, const_cast<int32_t *>(xadj), const_cast<int32_t *>(adjncy), const_cast<int32_t *>(adjwgt),
              const_cast<int32_t *>(vwgt)};
  cm_coarsen_params cp;
  cm_coarsen_default_params(nvtxs, nparts, &cp);
  if (P.coarsen_to > 0) cp.coarsen_to = P.coarsen_to;
  cp.match_mode = P.match_mode;
  cm_hierarchy *h = nullptr;
  auto t0 = std::chrono::steady_clock::now();
  if ((rc = cm_coarsen(ctx, &hg, 0, &cp, &h, s))) return rc;
  S.coarsen_ms = ms_since(t0);
  rc = part_hierarchy(ctx, h, nparts, P, part, objval, &S);
  S.total_ms = ms_since(t_all);
  if (stats) *stats = S;
  return rc;
}

// Drop-in with the reference's parameter list (include/cuMetis.h:18-19): one
// context on the current device for the call.  Returns 1 on success like the
// reference, 0 on failure (message in cm_last_error()) where the reference
// would exit.
extern "C" int cuMetis_PartGraph(int *nvtxs, int *xadj, int *adjncy, int *vwgt, int *adjwgt, int *nparts,
                                 float *tpwgts, float *ubvec, int *objval, int *part) {
  if (!nvtxs || !nparts) {
    cm_fail(CM_ERR_INVALID, "cuMetis_PartGraph: null size arguments");
    return 0;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  cm_ctx *ctx = nullptr;
  if (cm_ctx_create(dev, &ctx) != CM_OK) return 0;
  const int rc = cm_part_graph(ctx, *nvtxs, xadj, adjncy, vwgt, adjwgt, *nparts, tpwgts, ubvec, objval, part,
                               nullptr, nullptr);
  cm_ctx_destroy(ctx);
  return rc == CM_OK ? 1 : 0;
}
