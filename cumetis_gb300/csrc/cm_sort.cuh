// cm_sort.cuh -- shared-memory sorting helpers of the contraction.
//
// bucket_scale, bucket_of, bucket_place: the steps of a bucket sort whose
// buckets hold an entry or two each.
//
// block_unique_emit: merges runs of equal keys of a sorted buffer into
// (key, sum of the values) pairs, in order.
#pragma once

#include <cuda_runtime.h>

#include "cm_device.cuh"

namespace cm {

// Padded shared-memory index for keys of type K: one spare word every 32
// (32-bit keys) or 16 (64-bit keys), so that lanes reading runs of E
// consecutive keys hit distinct banks.
template <typename K>
__host__ __device__ __forceinline__ int padk(int i) {
  return sizeof(K) == 4 ? i + (i >> 5) : i + (i >> 4);
}
template <typename K>
__host__ __device__ constexpr int padded_k(int n) {
  return sizeof(K) == 4 ? n + (n >> 5) + 1 : n + (n >> 4) + 1;
}

// A (key, value) pair.
template <typename K> struct SortPair;
template <> struct __align__(8) SortPair<unsigned> {
  unsigned k;
  int v;
};
template <typename K>
__device__ __forceinline__ SortPair<K> make_pair_kv(K k, int v) {
  SortPair<K> p;
  p.k = k;
  p.v = v;
  return p;
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Slot of word i in a padded buffer: one spare word after every 8, so that a
// thread reading its 8 (or 16) consecutive words does not share banks with its
// neighbours.
__host__ __device__ __forceinline__ int rslot(int i) { return i + (i >> 3); }
__host__ __device__ constexpr int rslots(int cap) { return cap + cap / 8 + 1; }

// Bucket sorts: an id goes to the bucket at its place between a row's lowest
// and highest id; few ids share a bucket, and find their places in it by
// comparing with one another.

// Scale of the map from ids in [lo, lo + range] to `buckets` buckets.
__device__ __forceinline__ unsigned bucket_scale(int buckets, unsigned range) {
  const float f = (float)buckets * 4294967296.0f / ((float)range + 1.0f);
  return f < 4294967040.0f ? (unsigned)f : 4294967040u;
}
// Bucket of id x under the map (lo, scale); not decreasing in x.  Ids above the
// range may exceed the last bucket: the caller clamps.
__device__ __forceinline__ int bucket_of(unsigned x, uint2 map) {
  return (int)min(__umulhi(max(x, map.x) - map.x, map.y), 0x7fffffffu);
}
// Place of the pair at p (id x) among the pairs of its bucket [s0, s1): by id,
// equal ids in their present order.
__device__ __forceinline__ int bucket_place(const SortPair<unsigned> *work, int s0, int s1, int p, unsigned x) {
  int place = s0;
  for (int j = s0; j < s1; ++j) {
    const unsigned y = work[j].k;
    place += (y < x || (y == x && j < p)) ? 1 : 0;
  }
  return place;
}

// Visits the runs of equal keys of the sorted pairs s[0..n): for each run,
// emit(key, sum of the run's values (wrapping like int atomicAdd), q) with q
// the run's index in key order.  Returns the number of runs.  n <= NT * 32;
// scratch: tab of NT ints, scan of NT / 32 + 1.
// All threads of the block call it, or with NT = 32 those of a warp; it ends
// with their barrier.
template <typename K, int NT, int ITEMS, typename F>
__device__ __forceinline__ int block_unique_emit(const SortPair<K> *s, int n, int *tab, int *scan, F emit) {
  constexpr int NW = NT / 32;
  const int tid = NT == 32 ? threadIdx.x & 31 : threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rounds = (n + NT - 1) / NT;  // <= ITEMS
  const unsigned below = lanemask_lt();
  unsigned hm[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    hm[r] = 0u;
    if (r < rounds) {
      const int i = r * NT + tid;
      const bool head = i < n && (i == 0 || s[i].k != s[i - 1].k);
      hm[r] = __ballot_sync(0xffffffffu, head);
      if (lane == 0) tab[r * NW + warp] = __popc(hm[r]);
    }
  }
  row_sync<NT>();
  const int ncell = rounds * NW;  // <= NT
  int total;
  const int ex = block_exclusive_scan<NT>(tid < ncell ? tab[tid] : 0, scan, &total);
  if (tid < ncell) tab[tid] = ex;
  row_sync<NT>();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    if (r < rounds && (hm[r] >> lane & 1u)) {
      const int i = r * NT + tid;
      const K key = s[i].k;
      unsigned sum = (unsigned)s[i].v;
      for (int j = i + 1; j < n && s[j].k == key; ++j) sum += (unsigned)s[j].v;
      emit(key, (int)sum, tab[r * NW + warp] + __popc(hm[r] & below));
    }
  }
  row_sync<NT>();
  return total;
}

}  // namespace cm
