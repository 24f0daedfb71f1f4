// cm_rows.cuh -- coarse rows: one warp sorts and merges the short rows of a unit,
// a block or a warp a longer row, one warp copies 32 finished rows
// (cm_contract.cu describes the contraction).
#pragma once

#include "cm_ctx.h"
#include "cm_sort.cuh"

namespace cm {
namespace {

__host__ __device__ constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v >> 1); }

// Tiny units: rows of at most kTinyMax entries, D = kTinyDiag diagonals per
// unit, one warp per unit (fewer than D + kTinyMax entries, at most D/2
// non-empty rows).
#ifndef CM_TINY_MAX
#define CM_TINY_MAX 64
#endif
constexpr int kTinyMax = CM_TINY_MAX;
// Diagonals per unit (a multiple of 32).  A unit's entries stay below
// kTinyDiag + kTinyMax (its last row may run past the unit's diagonals by at
// most one row), which sets the capacity.
#ifndef CM_TINY_DIAG
#define CM_TINY_DIAG (2 * CM_TINY_MAX)
#endif
constexpr int kTinyDiag = CM_TINY_DIAG;
constexpr int kTinyCap = (kTinyDiag + kTinyMax + 31) / 32 * 32;
static_assert(kTinyDiag % 32 == 0 && kTinyDiag >= 2 * kTinyMax && kTinyCap <= 256, "CM_TINY_DIAG");
constexpr int kTinyItems = kTinyCap / 32;
constexpr int kTinyRowsPerLane = kTinyDiag / 32;
constexpr int kTinyMaxNz = kTinyDiag / 2;
static_assert(kTinyMax == 16 || kTinyMax == 32 || kTinyMax == 64, "CM_TINY_MAX: 16, 32 or 64");
// Expanded entry o (0 <= o < L) of a coarse row: the leader's entries first
// (as find_cnvtxsedge_original places them, cuMetis.cu:1014-1020).
__device__ __forceinline__ int expanded_src(int o, int xl, int dl, int xf) { return o < dl ? xl + o : xf + (o - dl); }

// ---------------------------------------------------------------------------
// Tiny units: one warp each
// ---------------------------------------------------------------------------
struct TinySmem {
  SortPair<unsigned> work[kTinyCap];        // (id, weight): gathered order, then bucket order, then sorted
  __align__(16) int start[kTinyCap + 4];    // entries per bucket, then the buckets' first places
  int4 rmeta[kTinyMaxNz];                   // per non-empty row: first entry in the unit, leader row start and length, follower row start
  uint2 rmap[kTinyMaxNz];                   // ... its id -> bucket map: lowest id, scale
  int rcount[kTinyMaxNz], rfirst[kTinyMaxNz], rdst[kTinyMaxNz];
  unsigned char rowid[kTinyCap];            // row of every gathered entry, then of every sorted one
  unsigned char nz_row[kTinyMaxNz];
};
static_assert(kTinyMaxNz <= 256 && kTinyDiag <= 256, "tiny unit row ids are 8-bit");

// One warp sorts and merges the rows of unit u (of units 0 .. last): the rows'
// metadata, every entry's row (a max-scan of the rows' first entries), the
// gather of (coarse id, weight) pairs without self loops, the sort of every
// row, and every run of equal ids written once, weights summed, to
// stage[eoff[c] ...) of its row; counted(c, the row's unique entries) for every
// row of the unit but those above kTinyMax (0 for empty rows).
//
// The sort: a row of L entries has L buckets, its share of one array of
// counters, and an id goes to the bucket at its place between the lowest and
// the highest of four of the row's ids (the ends of its two fine rows; ids
// beyond them go to the end buckets).  An atomic count per entry, one scan of
// all counters and one scatter leave the entries in bucket order; an entry
// then finds its place among the few of its bucket by comparing with them.
// The work does not depend on the width of the ids; the radix sort of (row, id)
// keys that this replaces took a pass per 4 bits, seven for 22-bit ids (R-MAT
// 22: 472 -> 298 us, a weighted 101^3 grid's levels: 549 -> 380 us).  Bound by
// issue and shared-memory latency at 32 resident warps per SM.
template <typename F>
__device__ __forceinline__ void tiny_unit(TinySmem &S, int u, int last, int nc, const int *adjncy, const int *adjwgt,
                                          const int *cmap, const int *first_row, const int4 *row_meta,
                                          const int *eoff, int2 *stage, DevStatus *st, F counted) {
  constexpr int RPL = kTinyRowsPerLane;
  const int lane = threadIdx.x & 31;
  const unsigned below = lanemask_lt();
  const int clo = first_row[u];
  const int chi = u < last ? first_row[u + 1] : nc;
  int R = chi - clo;
  if (R < 0 || R > kTinyDiag) {  // inconsistent unit map: report, touch nothing
    if (lane == 0) record_error(st, CM_ERR_INVALID, ERR_SITE_BOUNDS);
    R = 0;
  }
  // ---- rows: metadata, sorted-row index, entry layout (lane l: rows RPL*l ..)
  int len[RPL], jr[RPL], off[RPL], packed = 0;
  int4 md[RPL];
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int r = lane * RPL + i;
    md[i] = make_int4(0, 0, 0, 0);
    off[i] = 0;
    if (r < R) {
      md[i] = row_meta[clo + r];
      off[i] = eoff[clo + r];
    }
    const bool tiny = r < R && md[i].w <= kTinyMax;
    len[i] = tiny ? md[i].w : 0;
    if (tiny && len[i] == 0) counted(clo + r, 0);
    packed += (len[i] > 0 ? (1 << 16) : 0) + len[i];
  }
  const int incl = warp_inclusive_scan_i32(packed);
  const int tot = __shfl_sync(0xffffffffu, incl, 31);
  int ex = incl - packed;
  int ntot = tot & 0xffff, nnz = tot >> 16;
  if (ntot >= kTinyCap || nnz > kTinyMaxNz) {  // inconsistent row metadata: report, touch nothing
    if (lane == 0) record_error(st, CM_ERR_INVALID, ERR_SITE_BOUNDS);
    ntot = 0;
    nnz = 0;
#pragma unroll
    for (int i = 0; i < RPL; ++i) len[i] = 0;
  }
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    jr[i] = -1;
    if (len[i] > 0) {
      const int j = ex >> 16, e0 = ex & 0xffff;
      jr[i] = j;
      S.rmeta[j] = make_int4(e0, md[i].x, md[i].y, md[i].z);
      S.nz_row[j] = (unsigned char)(lane * RPL + i);
      S.rcount[j] = 0;
      S.rdst[j] = off[i];
      ex += (1 << 16) + len[i];
    }
  }
  for (int e = lane; e < kTinyCap; e += 32) {
    S.rowid[e] = 0;
    S.start[e] = 0;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < RPL; ++i)
    if (jr[i] > 0) S.rowid[S.rmeta[jr[i]].x] = (unsigned char)jr[i];
  __syncwarp();
  {  // every entry's row: inclusive max-scan of the first-entry marks
    unsigned v[kTinyItems], run = 0;
#pragma unroll
    for (int i = 0; i < kTinyItems; ++i) {
      v[i] = S.rowid[lane * kTinyItems + i];
      run = max(run, v[i]);
    }
    unsigned wmax = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, wmax, o);
      if (lane >= o) wmax = max(wmax, y);
    }
    unsigned cur = __shfl_up_sync(0xffffffffu, wmax, 1);
    if (lane == 0) cur = 0;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kTinyItems; ++i) {
      cur = max(cur, v[i]);
      S.rowid[lane * kTinyItems + i] = (unsigned char)cur;
    }
  }
  __syncwarp();
  // ---- gather (coarse id, weight); at[q] = the entry's row, -1 for none or a self loop
  // (slots past the unit's entries are skipped by the whole warp: an average
  // unit fills half of them)
  int x[kTinyItems], w[kTinyItems], at[kTinyItems];
  const int nq = (ntot + 31) >> 5;
  {
    int src[kTinyItems];
#pragma unroll
    for (int q = 0; q < kTinyItems; ++q) {
      const int e = q * 32 + lane;
      src[q] = -1;
      at[q] = -1;
      if (q < nq && e < ntot) {
        const int j = S.rowid[e];
        at[q] = j;
        const int4 r = S.rmeta[j];
        src[q] = expanded_src(e - r.x, r.y, r.z, r.w);
      }
    }
#pragma unroll
    for (int q = 0; q < kTinyItems; ++q) {
      if (q >= nq) break;
      x[q] = src[q] >= 0 ? __ldcs(adjncy + src[q]) : 0;
      w[q] = src[q] >= 0 ? __ldcs(adjwgt + src[q]) : 0;
    }
#pragma unroll
    for (int q = 0; q < kTinyItems; ++q) {
      if (q >= nq) break;
      if (src[q] >= 0) x[q] = cmap[x[q]];
    }
  }
#pragma unroll
  for (int q = 0; q < kTinyItems; ++q) {
    if (q >= nq) break;
    if (at[q] >= 0) S.work[q * 32 + lane].k = (unsigned)x[q];
  }
  __syncwarp();
  // ---- every row's id -> bucket map
  for (int j = lane; j < nnz; j += 32) {
    const int e0 = S.rmeta[j].x, dl = S.rmeta[j].z;
    const int L = (j + 1 < nnz ? S.rmeta[j + 1].x : ntot) - e0;
    const unsigned a0 = S.work[e0].k, a1 = S.work[e0 + max(dl, 1) - 1].k;
    const unsigned b0 = S.work[e0 + min(dl, L - 1)].k, b1 = S.work[e0 + L - 1].k;
    const unsigned lo = min(min(a0, a1), min(b0, b1)), hi = max(max(a0, a1), max(b0, b1));
    S.rmap[j] = make_uint2(lo, bucket_scale(L, hi - lo));
  }
  __syncwarp();
  // ---- count, scan, scatter in bucket order
#pragma unroll
  for (int q = 0; q < kTinyItems; ++q) {
    if (q >= nq) break;
    const int j = at[q];
    if (j < 0) continue;
    const int c = clo + (int)S.nz_row[j];
    at[q] = -1;
    if (x[q] == c) continue;
    const uint2 mp = S.rmap[j];
    const int e0 = S.rmeta[j].x, L = (j + 1 < nnz ? S.rmeta[j + 1].x : ntot) - e0;
    const int b = e0 + min(L - 1, bucket_of((unsigned)x[q], mp));
    at[q] = j << 24 | b << 16 | atomicAdd(&S.start[b], 1);
  }
  __syncwarp();
  int n;
  {
    int v[kTinyItems], sum = 0;
#pragma unroll
    for (int i = 0; i < kTinyItems; ++i) {
      v[i] = sum;
      sum += S.start[lane * kTinyItems + i];
    }
    const int inc = warp_inclusive_scan_i32(sum);
    n = __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll
    for (int i = 0; i < kTinyItems; ++i) S.start[lane * kTinyItems + i] = inc - sum + v[i];
    if (lane == 0) S.start[kTinyCap] = n;
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < kTinyItems; ++q) {
    if (q >= nq) break;
    if (at[q] == -1) continue;
    const int p = S.start[at[q] >> 16 & 255] + (at[q] & 0xffff);
    S.work[p] = make_pair_kv<unsigned>((unsigned)x[q], w[q]);
    S.rowid[p] = (unsigned char)((unsigned)at[q] >> 24);
  }
  __syncwarp();
  // ---- places within the buckets
  unsigned crowded = 0;
#pragma unroll
  for (int q = 0; q < kTinyItems; ++q) {
    if (q >= nq) break;
    if (at[q] == -1) continue;
    const int b = at[q] >> 16 & 255, s0 = S.start[b], s1 = S.start[b + 1];
    if (s1 - s0 > 1) {
      at[q] = bucket_place(S.work, s0, s1, s0 + (at[q] & 0xffff), (unsigned)x[q]);
      crowded |= 1u << q;
    }
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < kTinyItems; ++q) {
    if (q >= nq) break;
    if (crowded >> q & 1u) S.work[at[q]] = make_pair_kv<unsigned>((unsigned)x[q], w[q]);
  }
  __syncwarp();
  // ---- runs of equal ids: per row, its first run's index and its number of
  // runs; then every run to the row's stage
  unsigned hm[kTinyItems];
  int qbase = 0;
#pragma unroll
  for (int r = 0; r < kTinyItems; ++r) {
    hm[r] = 0u;
    if (r * 32 >= n) continue;
    const int i = r * 32 + lane;
    bool head = i < n, first = false;
    int j = 0;
    if (head) {
      j = S.rowid[i];
      first = i == 0 || S.rowid[i - 1] != j;
      head = first || S.work[i - 1].k != S.work[i].k;
      if (head) atomicAdd(&S.rcount[j], 1);
    }
    hm[r] = __ballot_sync(0xffffffffu, head);
    if (first) S.rfirst[j] = qbase + __popc(hm[r] & below);
    qbase += __popc(hm[r]);
  }
  __syncwarp();
  for (int j = lane; j < nnz; j += 32) counted(clo + (int)S.nz_row[j], S.rcount[j]);
  qbase = 0;
#pragma unroll
  for (int r = 0; r < kTinyItems; ++r) {
    if (r * 32 >= n) break;
    const int i = r * 32 + lane;
    if (hm[r] >> lane & 1u) {
      const unsigned key = S.work[i].k;
      const int j = S.rowid[i];
      unsigned sum = (unsigned)S.work[i].v;
      for (int j2 = i + 1; j2 < n && S.work[j2].k == key && S.rowid[j2] == j; ++j2) sum += (unsigned)S.work[j2].v;
      const int q = qbase + __popc(hm[r] & below);
      stage[S.rdst[j] + (q - S.rfirst[j])] = make_int2((int)key, (int)sum);
    }
    qbase += __popc(hm[r]);
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// One block or warp sorts a segment of one row (class rows and chunks)
// ---------------------------------------------------------------------------
template <int NT, int ITEMS>
struct RowSmem {
  SortPair<unsigned> work[NT * ITEMS];
  int start[rslots(NT * ITEMS + 1)];        // at rslot(b): entries of bucket b, then its first place
  int tab[NT], scan[NT / 32 + 1];
  unsigned lo, hi;                          // range of the row's places
  int load;                                 // sum over the entries of their bucket's size
};
// A row whose entries share their buckets with more than this many on average
// is sorted by comparator passes instead: a comparison within a bucket costs
// about 5 instructions, a comparator pass of a row of L entries about 10 in each
// of log2(L) (log2(L) + 1) / 2 steps, 360 to 1050 for L from 200 to 16384.
constexpr int kCrowded = 48;

// Ascending sort of work[0..n) by id: Batcher's bitonic network in its form
// with one comparator direction, in which places past n are never touched.
template <int NT>
__device__ __noinline__ void bitonic_sort(SortPair<unsigned> *work, int n) {
  for (int k = 2; (k >> 1) < n; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      const int flip = j == (k >> 1) ? k - 1 : j;
      for (int t = NT == 32 ? threadIdx.x & 31 : threadIdx.x; t < (n + j + 1) >> 1; t += NT) {
        const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1)), p = i ^ flip;
        if (p < n && work[i].k > work[p].k) {
          const SortPair<unsigned> x = work[i];
          work[i] = work[p];
          work[p] = x;
        }
      }
      row_sync<NT>();
    }
  }
}

// Writes the unique entries (coarse id, summed weight) of entries
// [cs, cs + cnt) of coarse row c's expanded row (metadata md), ascending by
// id, self loops dropped, to dst[0..U).  Returns U.  cnt <= NT * ITEMS.  All
// threads of the block call it, or with NT = 32 those of a warp; it ends with
// their barrier.
//
// Bucket sort: entry x's bucket is its place between the row's lowest and
// highest, where places are the expanded offsets (cplace: a fine vertex's
// coarse id and offset in one 8-byte gather).  Offsets grow with
// the ids' degrees, and an edge leads to a vertex about in proportion to its
// degree, so the buckets fill evenly also where most entries have low ids
// (R-MAT: the top ten id bits are all zero for 6% of the entries).  As many
// buckets as places: the entries of a bucket, one or two, find their order by
// comparing with one another.  One pass over the entries replaces the radix
// sort's pass per 4 id bits: the row kernels of an R-MAT 22 level take 2.09 ms
// of overlapped time against 2.92 ms (8193-12288 entries 367 -> 213 us, 257-384
// 195 -> 115 us).  Bound by issue (46% busy) and by the L1 / shared-memory pipe
// (72%): every gather of cplace takes a wavefront per entry.
template <int NT, int ITEMS>
__device__ __forceinline__ int row_sorted_unique(RowSmem<NT, ITEMS> &S, int c, const int4 &md, int cs,
                                                 int cnt, const int *__restrict__ adjncy,
                                                 const int *__restrict__ adjwgt, const int2 *__restrict__ cplace,
                                                 int2 *__restrict__ dst) {
  constexpr int kCap = NT * ITEMS;
  static_assert(kCap <= 1 << 14, "places are packed in 14 bits");
  const int tid = NT == 32 ? threadIdx.x & 31 : threadIdx.x, lane = tid & 31;
  int x[ITEMS], w[ITEMS], at[ITEMS];  // at: -1 none or a self loop, then place, then bucket | rank << 16
#pragma unroll
  for (int u = 0; u < ITEMS; ++u) {
    const int t = u * NT + tid;
    at[u] = -1;
    if (t < cnt) {
      const int src = expanded_src(cs + t, md.x, md.y, md.z);
      x[u] = __ldcs(adjncy + src);
      w[u] = __ldcs(adjwgt + src);
      at[u] = 0;
    }
  }
#pragma unroll
  for (int u = 0; u < ITEMS; ++u) S.start[rslot(u * NT + tid)] = 0;
  if (tid == 0) {
    S.lo = 0xffffffffu;
    S.hi = 0u;
    S.load = 0;
  }
  unsigned lo = 0xffffffffu, hi = 0u;
#pragma unroll
  for (int u = 0; u < ITEMS; ++u)
    if (at[u] == 0) {
      const int2 y = cplace[x[u]];
      x[u] = y.x;
      at[u] = y.y;
    }
#pragma unroll
  for (int u = 0; u < ITEMS; ++u) {
    if (at[u] >= 0 && x[u] == c) at[u] = -1;
    if (at[u] >= 0) {
      lo = min(lo, (unsigned)at[u]);
      hi = max(hi, (unsigned)at[u]);
    }
  }
  row_sync<NT>();
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0 && lo <= hi) {
    atomicMin(&S.lo, lo);
    atomicMax(&S.hi, hi);
  }
  row_sync<NT>();
  if (S.lo > S.hi) {  // only self loops
    row_sync<NT>();
    return 0;
  }
  const uint2 map = make_uint2(S.lo, bucket_scale(kCap, S.hi - S.lo));
#pragma unroll
  for (int u = 0; u < ITEMS; ++u)
    if (at[u] >= 0) {
      const int b = min(bucket_of((unsigned)at[u], map), kCap - 1);
      at[u] = b | atomicAdd(&S.start[rslot(b)], 1) << 16;
    }
  row_sync<NT>();
  int n;
  {
    int sum = 0;
#pragma unroll
    for (int u = 0; u < ITEMS; ++u) sum += S.start[rslot(tid * ITEMS + u)];
    int run = block_exclusive_scan<NT>(sum, S.scan, &n);
#pragma unroll
    for (int u = 0; u < ITEMS; ++u) {
      const int v = S.start[rslot(tid * ITEMS + u)];
      S.start[rslot(tid * ITEMS + u)] = run;
      run += v;
    }
    if (tid == 0) S.start[rslot(kCap)] = n;
  }
  row_sync<NT>();
  // at: -1 if alone in its bucket, else the bucket's first place | rank << 14 | (size - 1) << 22
  int load = 0;
#pragma unroll
  for (int u = 0; u < ITEMS; ++u)
    if (at[u] >= 0) {
      const int b = at[u] & 0xffff, r = at[u] >> 16, s0 = S.start[rslot(b)], size = S.start[rslot(b + 1)] - s0;
      S.work[s0 + r] = make_pair_kv<unsigned>((unsigned)x[u], w[u]);
      load += size <= 256 ? size : kCap;  // too many for the packed form: as a crowded row
      at[u] = size == 1 ? -1 : s0 | (r & 255) << 14 | (size - 1) << 22;
    }
  load = __reduce_add_sync(0xffffffffu, load);
  if (lane == 0) atomicAdd(&S.load, load);
  row_sync<NT>();
  if (S.load <= kCrowded * n) {
#pragma unroll
    for (int u = 0; u < ITEMS; ++u)
      if (at[u] >= 0) {
        const int s0 = at[u] & 0x3fff;
        at[u] = bucket_place(S.work, s0, s0 + (at[u] >> 22) + 1, s0 + (at[u] >> 14 & 255), (unsigned)x[u]);
      }
    row_sync<NT>();
#pragma unroll
    for (int u = 0; u < ITEMS; ++u)
      if (at[u] >= 0) S.work[at[u]] = make_pair_kv<unsigned>((unsigned)x[u], w[u]);
    row_sync<NT>();
  } else {
    bitonic_sort<NT>(S.work, n);
  }
  return block_unique_emit<unsigned, NT, ITEMS>(S.work, n, S.tab, S.scan, [&](unsigned key, int sum, int q) {
    dst[q] = make_int2((int)key, sum);
  });
}

// One warp moves 32 rows from the stage to their final place: lane l's row has
// cnt entries at stage[src ..], which go to cadj...[dst ..].  A warp scan lays
// the rows' entries out back to back, and the warp walks them 32 at a time
// (kCopyBatch steps in flight), each lane finding its entry's row by a five-step
// search over the prefixes held in the lanes.
constexpr int kCopyBatch = 4;  // stage loads in flight per thread before their stores
__device__ __forceinline__ void copy_32_rows(int src, int cnt, int dst, const int2 *stage, int *cadjncy,
                                             int *cadjwgt) {
  const int lane = threadIdx.x & 31;
  const int incl = warp_inclusive_scan_i32(cnt);
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const int excl = incl - cnt;
  for (int k0 = 0; k0 < total; k0 += 32 * kCopyBatch) {
    int2 e[kCopyBatch];
    int d[kCopyBatch];
#pragma unroll
    for (int q = 0; q < kCopyBatch; ++q) {
      const int k = k0 + 32 * q + lane;
      int r = 0;  // the last row whose first entry is at or before k
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int v = __shfl_sync(0xffffffffu, excl, r + step);
        if (v <= k) r += step;
      }
      const int off = k - __shfl_sync(0xffffffffu, excl, r);
      const int s0 = __shfl_sync(0xffffffffu, src, r), d0 = __shfl_sync(0xffffffffu, dst, r);
      d[q] = k < total ? d0 + off : -1;
      e[q] = k < total ? __ldcs(stage + s0 + off) : make_int2(0, 0);
    }
#pragma unroll
    for (int q = 0; q < kCopyBatch; ++q)
      if (d[q] >= 0) {
        cadjncy[d[q]] = e[q].x;
        cadjwgt[d[q]] = e[q].y;
      }
  }
}

}  // namespace
}  // namespace cm
