// cm_levels.cu -- whole coarsening levels of small graphs in one kernel.
//
// A level of a small graph is about twenty launches and memsets (cm_match.cu,
// cm_cmap.cu, cm_contract.cu) of a few microseconds of work each, and a host
// round trip for the stop rule: 110 to 130 us a level whatever its size, 24 to
// 65 us here.  Bound by latency: a chain of displaced proposals takes about 1 us
// a step (10 to 20 us a level), a warp 7 us for a unit of rows, a barrier 2 us.  Here
// the same steps are phases of one cooperative kernel, separated by six grid
// barriers a level, and the kernel goes on to the next level by the stop rule
// of cuMetis_coarsen (cuMetis.cu:1843-1845) itself:
//
//   lists      every vertex's most preferred neighbours
//   proposals  chains of displaced proposals to their end
//   partners   match[], and per block its coarse vertices and entries
//   vertices   cmap, vertex weights, expanded offsets, row metadata, the tiny
//              units' first rows and the list of longer rows
//   rows       every coarse row sorted and merged into the stage, its unique
//              entries counted for the block that owns the row
//   copy       coarse offsets, rows to their final place
//
// Blocks own ranges of vertices (partners, vertices) and of coarse rows (copy);
// the prefix over the ranges comes from one sum per block.  The coarse
// levels are carved out of one allocation at their exact sizes.
//
// What the kernel does not handle ends it before that level -- rows of more
// than kMaxRow expanded or kMatchChunk fine entries, an adjacency that is not
// symmetric, a very long chain, an allocation that turns out too small -- and the
// caller does the level with the separate kernels.
#include <algorithm>

#include "cm_ctx.h"
#include "cm_match.cuh"
#include "cm_rows.cuh"

namespace cm {
namespace {

constexpr int kLvThreads = 512, kLvWarps = kLvThreads / 32;
// Vertices + entries per block of the grid: one tiny unit (128 diagonals) per
// warp.  A level of a 69 x 69 mesh takes 81, 53 and 52 us with 4096, 2048 and
// 1024 (more blocks only make the barriers dearer), one of 51,000 vertices 77,
// 65 and 66.
#ifndef CM_LEVEL_WORK
#define CM_LEVEL_WORK 2048
#endif
constexpr int kLvWork = CM_LEVEL_WORK;
constexpr int kLvItems = 8, kMaxRow = 32 * kLvItems;  // longest expanded row: one warp sorts it
// Turns of a warp's chains in one level: about 0.3 s, while the other blocks wait at
// a barrier.  A level with a longer chain is left to the separate kernels, where
// nobody waits for it.
constexpr unsigned kFusedSteps = 1u << 18;
// Why a level is not handled: a row of more than kMatchChunk entries; an adjacency
// that is not symmetric, or a long chain.  The levels behind an odd one are most likely
// odd too and are not tried.
enum : int { kRowTooLong = 1, kOdd = 2 };
constexpr int kMaxFused = 64;                         // levels of one launch
constexpr int kCountBits = 21;                        // vertices and entries stay below 2^21 (packed scan)
static_assert(kTinyMax < kMaxRow, "row lengths");

// One produced level: sizes, its arrays' places in the allocation, and the
// longest expanded row of the contraction that made it.
struct FusedLevel {
  int n, m, longest, pad;
  long long xadj, vwgt, match, cmap, adjncy, adjwgt;
};

struct LevelArgs {
  MatchArgs match;           // scratch pointers and the cap; the graph's are set per level
  int n, m;
  const int *xadj, *adjncy, *adjwgt, *vwgt;  // the first level
  int *m0, *cmap0;
  int *arena;                // coarse levels
  long long arena_ints;
  int *eoff, *ucount, *first_row, *long_rows;
  int4 *row_meta;
  int2 *cplace, *stage;
  unsigned long long *sums;  // [2][gridDim.x]: the blocks' vertices, the blocks' coarse entries
  int *flags;                // [kMaxFused][4]: not handled (kRowTooLong, kOdd), longest expanded row, longer rows, -
  unsigned *bar;             // barrier arrivals
  FusedLevel *out;           // [kMaxFused]
  int *result;               // [0] levels produced, [1] 1 if the stop rule ended the coarsening, [6] kOdd: see there
  // First level not measured yet: take the sum of its weights and its longest row
  // into result[2..5] and, with derive_cap, the weight limit from them.
  int measure, derive_cap;
  int coarsen_to, max_levels;
  double shrink;
};

union WarpSmem {
  TinySmem tiny;
  RowSmem<32, kLvItems> row;
  struct {
    int list[32], queue[32];
    int2 wbuf[32];
  } prop;
};

// Barrier of blocks 0 .. nb-1 (all resident).  Arrivals only count up, so
// blocks may leave between barriers.  False (CM_ERR_LIMIT) on a timeout.
__device__ __forceinline__ bool level_barrier(unsigned *bar, unsigned &target, unsigned nb, DevStatus *st) {
  __shared__ int s_ok;
  target += nb;
  if (nb == 1) {
    __threadfence();
    __syncthreads();
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();
    atomicAdd(bar, 1u);
    const uint64_t t0 = global_timer_ns();
    while ((int)(ld_acquire(bar) - target) < 0) {
      if (ld_relaxed(&st->error) != 0) {
        ok = 0;
        break;
      }
      if (global_timer_ns() - t0 > kWaitLimitNs) {
        record_error(st, CM_ERR_LIMIT, ERR_SITE_BARRIER);
        ok = 0;
        break;
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Exclusive scan of one value per thread over the block; sh: kLvWarps + 1.
__device__ __forceinline__ unsigned long long block_scan_u64(unsigned long long v, unsigned long long *sh,
                                                             unsigned long long *total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long inc = warp_inclusive_scan_u64(v);
  if (lane == 31) sh[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long x = lane < kLvWarps ? sh[lane] : 0ull;
    const unsigned long long xi = warp_inclusive_scan_u64(x);
    if (lane < kLvWarps) sh[lane] = xi - x;
    if (lane == kLvWarps - 1) sh[kLvWarps] = xi;
  }
  __syncthreads();
  const unsigned long long r = sh[warp] + inc - v;
  *total = sh[kLvWarps];
  __syncthreads();
  return r;
}

// The sum of the blocks' values before this block; *total: of all nb (nb <=
// kLvThreads).
__device__ __forceinline__ unsigned long long blocks_before(const unsigned long long *sums, int nb,
                                                            unsigned long long *sh, unsigned long long *total) {
  const unsigned long long v = (int)threadIdx.x < nb ? __ldcg(sums + threadIdx.x) : 0ull;
  __shared__ unsigned long long s_mine;
  const unsigned long long ex = block_scan_u64(v, sh, total);
  if (threadIdx.x == blockIdx.x) s_mine = ex;
  __syncthreads();
  const unsigned long long r = s_mine;
  __syncthreads();
  return r;
}

// Packed scan value of a coarse vertex: 1, its expanded row length, and that
// length again if the row goes to the tiny units.
constexpr unsigned long long kCountMask = (1ull << kCountBits) - 1;
__device__ __forceinline__ unsigned long long pack_row(int L) {
  return 1ull | (unsigned long long)L << kCountBits |
         (L <= kTinyMax ? (unsigned long long)L << (2 * kCountBits) : 0ull);
}

template <bool H>
__global__ void __launch_bounds__(kLvThreads, 1) k_levels(LevelArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long sh[kLvWarps + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = lanemask_lt();
  WarpSmem &S = reinterpret_cast<WarpSmem *>(smem_raw)[warp];
  MatchArgs a = A.match;
  DevStatus *st = a.st;
  int n = A.n, m = A.m;
  const int *xadj = A.xadj, *vwgt = A.vwgt;
  int *match = A.m0, *cmap = A.cmap0;
  a.adjncy = A.adjncy;
  a.adjwgt = A.adjwgt;
  long long used = 0;  // of the allocation
  unsigned target = 0;
  auto carve = [&](long long ints) {
    const long long at = used;
    used += (ints + 63) & ~63ll;
    return at;
  };
  if (A.measure) {
    unsigned long long *stats = reinterpret_cast<unsigned long long *>(A.result + 2), sum = 0ull, longest = 0ull;
    for (int v = blockIdx.x * kLvThreads + threadIdx.x; v < n; v += gridDim.x * kLvThreads) {
      sum += (unsigned long long)(long long)vwgt[v];
      longest = max(longest, (unsigned long long)(unsigned)(xadj[v + 1] - xadj[v]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
    }
    if (lane == 0) {
      atomicAdd(stats, sum);
      atomicMax(stats + 1, longest);
    }
    if (!level_barrier(A.bar, target, gridDim.x, st)) return;
    if (__ldcg(stats + 1) > kMatchChunk) return;  // the separate kernels' graph
    if (A.derive_cap) a.maxvwgt = cm_weight_limit((int64_t)__ldcg(stats), A.coarsen_to);
  }
  for (int level = 0;; ++level) {
    const int nb = min((int)gridDim.x, 1 + (n + m) / kLvWork);
    if ((int)blockIdx.x >= nb) return;
    const int gw = blockIdx.x * kLvWarps + warp, nw = nb * kLvWarps;
    int *flags = A.flags + 4 * level;
    a.n = n;
    a.xadj = xadj;
    a.vwgt = vwgt;

    // ---- lists
    if (threadIdx.x == 0) A.sums[gridDim.x + blockIdx.x] = 0ull;
    bool unfit = false;
    for (int b0 = gw * 32; b0 < n; b0 += nw * 32) {
      const int v = b0 + lane;
      int xs = 0, deg = 0;
      if (v < n) {
        a.best[v] = 0ull;
        xs = xadj[v];
        deg = xadj[v + 1] - xs;
      }
      if (deg > 0 && deg <= kSerialDeg) short_list<H>(a, v, xs, deg);
      unfit |= deg > kMatchChunk;
      unsigned longer = __ballot_sync(0xffffffffu, deg > kSerialDeg && deg <= kMatchChunk);
      while (longer) {
        const int src = __ffs(longer) - 1;
        longer &= longer - 1;
        const int x = b0 + src, s0 = __shfl_sync(0xffffffffu, xs, src), d = __shfl_sync(0xffffffffu, deg, src);
        const TopK<H, kTop> r = chunk_best<H, kTop, kStatic>(a, x, s0, s0 + d, false, S.prop.wbuf);
        if (lane == 0) store_top(a, x, r);
      }
    }
    if (unfit) flags[0] = kRowTooLong;
    if (!level_barrier(A.bar, target, nb, st)) return;
    if (__ldcg(flags) != 0) return;
    unfit = false;

    // ---- proposals
    unsigned steps = kFusedSteps;
    for (int b0 = gw * 32; b0 < n; b0 += nw * 32) {
      int nq = 0;
      ChainEnd end = propose_span<H, true, 8, true>(a, b0, 32, false, S.prop.list, &steps, [&](int v, int, int) {
        const unsigned q = __ballot_sync(0xffffffffu, v >= 0);
        if (v >= 0) S.prop.queue[nq + __popc(q & below)] = v;
        nq += __popc(q);
      });
      __syncwarp();
      for (int i = 0; i < nq && end == kChainDone; ++i) {
        const int v = S.prop.queue[i];
        end = warp_chain<H, kGiveUp>(a, v, xadj[v], xadj[v + 1], false, TopK<H, kTop>(), false, 0, 0, &steps,
                                     S.prop.wbuf);
      }
      __syncwarp();
      if (end == kChainLong) unfit = true;  // the level is given up behind the partners
      if (end != kChainDone || (b0 + nw * 32 < n && warp_sees_error(st))) break;  // (a barrier sees errors)
    }
    if (!level_barrier(A.bar, target, nb, st)) return;

    // ---- partners
    const int r0 = (int)((long long)n * blockIdx.x / nb), r1 = (int)((long long)n * (blockIdx.x + 1) / nb);
    {
      unsigned long long sum = 0ull;
      int longest = 0;
      for (int v = r0 + (int)threadIdx.x; v < r1; v += kLvThreads) {
        const unsigned long long b = ld_best(a, v);
        const int h = best_holder(b);
        const bool mutual = h >= 0 && best_mutual(b, ld_best(a, h), v);
        unfit |= h >= 0 && !mutual;
        const int u = mutual ? h : v;
        match[v] = u;
        if (v <= u) {
          const int L = xadj[v + 1] - xadj[v] + (u != v ? xadj[u + 1] - xadj[u] : 0);
          sum += pack_row(L);
          longest = max(longest, L);
        }
      }
      unsigned long long total;
      block_scan_u64(sum, sh, &total);
      if (threadIdx.x == 0) A.sums[blockIdx.x] = total;
      longest = __reduce_max_sync(0xffffffffu, longest);
      if (lane == 0 && longest > 0) atomicMax(flags + 1, longest);
      if (unfit) flags[0] = kOdd;
    }
    if (!level_barrier(A.bar, target, nb, st)) return;
    const int longest = __ldcg(flags + 1);
    const int odd = __ldcg(flags);
    if (odd != 0 || longest > kMaxRow) {
      if (blockIdx.x == 0 && threadIdx.x == 0) A.result[6] = odd;
      return;
    }

    // ---- vertices
    unsigned long long total;
    unsigned long long carry = blocks_before(A.sums, nb, sh, &total);
    const int nc = (int)(total & kCountMask);
    const long long o_xadj = carve(nc + 1), o_vwgt = carve(nc), o_match = carve(nc), o_cmap = carve(nc);
    if (used > A.arena_ints) return;
    int *cxadj = A.arena + o_xadj, *cvwgt = A.arena + o_vwgt;
    for (int t0 = r0; t0 < r1; t0 += kLvThreads) {
      const int v = t0 + (int)threadIdx.x;
      int u = -1, xv = 0, xu = 0, dv = 0, L = 0;
      if (v < r1) {
        u = match[v];  // written by this thread
        if (v <= u) {
          xv = xadj[v];
          dv = xadj[v + 1] - xv;
          xu = u != v ? xadj[u] : 0;
          L = dv + (u != v ? xadj[u + 1] - xu : 0);
        }
      }
      const bool leads = v < r1 && v <= u;
      unsigned long long tile;
      const unsigned long long P = carry + block_scan_u64(leads ? pack_row(L) : 0ull, sh, &tile);
      carry += tile;
      if (!leads) continue;
      const int c = (int)(P & kCountMask), e = (int)(P >> kCountBits & kCountMask);
      cmap[v] = c;
      if (u != v) cmap[u] = c;
      if (longest > kTinyMax) {
        A.cplace[v] = make_int2(c, e);
        if (u != v) A.cplace[u] = make_int2(c, e);
      }
      cvwgt[c] = (int)((unsigned)vwgt[v] + (u != v ? (unsigned)vwgt[u] : 0u));
      A.eoff[c] = e;
      A.row_meta[c] = make_int4(xv, dv, xu, L);
      if (L > kTinyMax) A.long_rows[atomicAdd(flags + 2, 1)] = c;
      // a row costs 1 + (its entries if it is tiny) diagonals
      const int d0 = c + (int)(P >> (2 * kCountBits)), d1 = d0 + 1 + (L <= kTinyMax ? L : 0);
      for (int k = d0 / kTinyDiag + 1; k <= d1 / kTinyDiag; ++k) A.first_row[k] = c + 1;
      if (c == 0) A.first_row[0] = 0;
      if (c == nc - 1) flags[3] = d0 / kTinyDiag;  // the last unit
    }
    if (!level_barrier(A.bar, target, nb, st)) return;

    // ---- rows
    const int nlong = __ldcg(flags + 2), last = __ldcg(flags + 3);
    const int own = (nc + nb - 1) / nb;  // coarse rows per block in the copy
    unsigned long long *row_sums = A.sums + gridDim.x;
    auto counted = [&](int c, int cnt) {
      A.ucount[c] = cnt;
      if (cnt) atomicAdd(row_sums + c / own, (unsigned long long)cnt);
    };
    for (int i = gw; i < nlong; i += nw) {
      const int c = __ldcg(A.long_rows + i);
      const int4 md = A.row_meta[c];
      const int U = row_sorted_unique<32, kLvItems>(S.row, c, md, 0, md.w, a.adjncy, a.adjwgt, A.cplace,
                                                    A.stage + A.eoff[c]);
      if (lane == 0) counted(c, U);
    }
    __syncwarp();
    for (int u = gw; u <= last; u += nw)
      tiny_unit(S.tiny, u, last, nc, a.adjncy, a.adjwgt, cmap, A.first_row, A.row_meta, A.eoff, A.stage, st, counted);
    if (!level_barrier(A.bar, target, nb, st)) return;

    // ---- copy
    const int c0 = min(nc, own * (int)blockIdx.x), c1 = min(nc, c0 + own);
    carry = blocks_before(row_sums, nb, sh, &total);
    const int mc = (int)total;
    const long long o_adjncy = carve(mc), o_adjwgt = carve(mc);
    if (used > A.arena_ints) return;
    int *cadjncy = A.arena + o_adjncy, *cadjwgt = A.arena + o_adjwgt;
    for (int t0 = c0; t0 < c1; t0 += kLvThreads) {
      const int c = t0 + (int)threadIdx.x;
      const int cnt = c < c1 ? A.ucount[c] : 0, src = c < c1 ? A.eoff[c] : 0;
      unsigned long long tile;
      const int dst = (int)(carry + block_scan_u64((unsigned)cnt, sh, &tile));
      carry += tile;
      if (c < c1) cxadj[c + 1] = dst + cnt;
      copy_32_rows(src, cnt, dst, A.stage, cadjncy, cadjwgt);
    }
    const bool go_on = nc > A.coarsen_to && (double)nc < A.shrink * (double)n && mc > nc / 2 &&
                       level + 1 < A.max_levels;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      cxadj[0] = 0;
      FusedLevel &o = A.out[level];
      o.n = nc;
      o.m = mc;
      o.longest = longest;
      o.xadj = o_xadj;
      o.vwgt = o_vwgt;
      o.match = o_match;
      o.cmap = o_cmap;
      o.adjncy = o_adjncy;
      o.adjwgt = o_adjwgt;
      A.result[0] = level + 1;
      A.result[1] = go_on ? 0 : 1;
    }
    if (!go_on || level + 1 == kMaxFused) return;
    if (!level_barrier(A.bar, target, nb, st)) return;
    n = nc;
    m = mc;
    xadj = cxadj;
    vwgt = cvwgt;
    a.adjncy = cadjncy;
    a.adjwgt = cadjwgt;
    match = A.arena + o_match;
    cmap = A.arena + o_cmap;
  }
}

int64_t fused_units(int64_t n, int64_t m) { return (n + m) / kTinyDiag + 2; }

}  // namespace

size_t fused_ws_bytes(int64_t n, int64_t m) {
  size_t b = (size_t)n * (8 + 2 * 4 * kTop);                 // best, lists
  b += (size_t)(n + 1) * 4 * 3 + (size_t)n * (16 + 8) + (size_t)m * 8;  // eoff, ucount, long_rows, row_meta, cplace, stage
  b += (size_t)fused_units(n, m) * 4;
  b += 2 * kLvThreads * 8 + kMaxFused * (16 + sizeof(FusedLevel));
  return b + 32 * 256;
}

bool fused_fits(const cm_ctx *ctx, int64_t n, int64_t m, int64_t max_deg, int32_t mode) {
  return (mode == CM_MATCH_HEM || mode == CM_MATCH_HEM_HASH) && n > 0 && n + m <= kFusedWork && max_deg <= kMatchChunk &&
         !ctx->timing && !ctx->d_trace;
}

int launch_fused(cm_ctx *ctx, cm_hierarchy *h, const cm_coarsen_params *p, cudaStream_t s, int *produced, int *stopped,
                 int64_t *row_bound, bool measure, bool *odd) {
  static_assert(kFusedWork < 1 << kCountBits, "packed scan: counts of isolated vertices, too, stay below 2^kCountBits");
  *produced = 0;
  *stopped = 0;
  const cm_level F = h->levels.back();
  const int64_t n = F.g.nvtxs, m = F.g.nedges;
  const bool hash = p->match_mode == CM_MATCH_HEM_HASH;
  const void *fn = hash ? (const void *)k_levels<true> : (const void *)k_levels<false>;
  constexpr int smem = kLvWarps * (int)sizeof(WarpSmem);
  if (!ctx->levels_attrs_set) {
    int rc = CM_OK;
    for (const void *f : {(const void *)k_levels<true>, (const void *)k_levels<false>}) {
      if (!rc) rc = cuda_status(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "levels");
      int b = 0;
      if (!rc) rc = cuda_status(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, kLvThreads, smem), "levels");
      if (!rc && b < 1) rc = cm_fail(CM_ERR_CUDA, "levels: kernel cannot be resident");
    }
    if (rc) return rc;
    ctx->levels_attrs_set = true;
  }
  const int grid = (int)std::min<int64_t>(std::min(ctx->num_sms, kLvThreads), 1 + (n + m) / kLvWork);
  // The coarse levels' vertices come to at most 3 n (each level has at most
  // 3/4 of the last's under the default rule), usually n; their entries to 1.5 m
  // on meshes.  What does not fit is left to the separate kernels.
  auto slab = std::make_shared<cm_slab>();
  const long long arena_ints = 4 * 2 * n + 2 * (2 * m) + 64 * 6 * 16;
  int rc = cuda_status(cudaMallocFromPoolAsync(&slab->ptr, (size_t)arena_ints * 4, ctx->pool, s), "levels alloc");
  if (rc) return rc;
  slab->device = ctx->device;
  slab->stream = s;
  LevelArgs A{};
  bool ok = true;
  auto take = [&](size_t bytes) {
    void *q = ws_take(ctx, bytes);
    ok = ok && q != nullptr;
    return q;
  };
  A.match.best = (unsigned long long *)take((size_t)n * 8);
  A.match.top = (int *)take((size_t)n * 4 * kTop);
  A.match.topw = (int *)take((size_t)n * 4 * kTop);
  A.eoff = (int *)take((size_t)(n + 1) * 4);
  A.ucount = (int *)take((size_t)n * 4);
  A.long_rows = (int *)take((size_t)n * 4);
  A.first_row = (int *)take((size_t)fused_units(n, m) * 4);
  A.row_meta = (int4 *)take((size_t)n * 16);
  A.cplace = (int2 *)take((size_t)n * 8);
  A.stage = (int2 *)take((size_t)m * 8 + 8);
  A.sums = (unsigned long long *)take(2 * (size_t)grid * 8);
  // cleared together: flags, barrier, result; read back together: result, levels
  const size_t fb = kMaxFused * 16, head = fb + 64;
  char *q = (char *)take(head + kMaxFused * sizeof(FusedLevel));
  if (!ok) return cm_fail(CM_ERR_NOMEM, "levels: workspace too small");
  A.flags = (int *)q;
  A.bar = (unsigned *)(q + fb);
  A.result = (int *)(q + fb + 32);
  A.out = (FusedLevel *)(q + head);
  cudaMemsetAsync(q, 0, head, s);
  A.match.maxvwgt = h->maxvwgt;
  A.match.st = ctx->d_status;
  A.n = (int)n;
  A.m = (int)m;
  A.xadj = F.g.xadj;
  A.adjncy = F.g.adjncy;
  A.adjwgt = F.g.adjwgt;
  A.vwgt = F.g.vwgt;
  A.m0 = F.match;
  A.cmap0 = F.cmap;
  A.arena = (int *)slab->ptr;
  A.arena_ints = arena_ints;
  A.measure = measure;
  A.derive_cap = measure && p->maxvwgt <= 0;
  A.coarsen_to = p->coarsen_to;
  A.max_levels = p->max_levels - ((int)h->levels.size() - 1);
  A.shrink = p->shrink;
  void *args[] = {(void *)&A};
  if ((rc = cuda_status(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kLvThreads), args, smem, s), "levels launch")))
    return rc;
  ctx->launches++;
  struct Readback {
    int result[8];
    FusedLevel level[kMaxFused];
  };
  static_assert(sizeof(Readback) <= cm_ctx::kReadbackBytes, "readback");
  Readback *r = reinterpret_cast<Readback *>(ctx->h_levels);
  cudaMemcpyAsync(r, A.result, sizeof(Readback), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(ctx->h_status, ctx->d_status, sizeof(DevStatus), cudaMemcpyDeviceToHost, s);
  if ((rc = stream_wait(ctx, s, "levels sync"))) return rc;
  if (ctx->h_status->error) {
    rc = take_device_error(ctx, s);  // also resets the status block
    return rc ? rc : CM_ERR_CUDA;
  }
  *produced = r->result[0];
  *stopped = r->result[1];
  *odd = r->result[6] == kOdd;
  if (measure) {
    long long stats[2];
    memcpy(stats, r->result + 2, sizeof stats);
    if (p->maxvwgt <= 0) h->maxvwgt = cm_weight_limit(stats[0], p->coarsen_to);
    *row_bound = 2 * stats[1];
  }
  if (*produced > 0) h->slabs.push_back(slab);
  for (int i = 0; i < *produced; ++i) {
    const FusedLevel &o = r->level[i];
    cm_level L;
    L.g.nvtxs = o.n;
    L.g.nedges = o.m;
    L.g.xadj = A.arena + o.xadj;
    L.g.vwgt = A.arena + o.vwgt;
    L.g.adjncy = A.arena + o.adjncy;
    L.g.adjwgt = A.arena + o.adjwgt;
    L.match = A.arena + o.match;
    L.cmap = A.arena + o.cmap;
    h->levels.push_back(L);
    h->rounds.push_back(1);
    *row_bound = 2 * (int64_t)o.longest;
  }
  return CM_OK;
}

}  // namespace cm
