// Merge and sort, shared by libb2p (b2p_merge, b2p_sort) and the
// header-only C++ layer (hipsycl::algorithms::merge / sort and the stdpar
// std::merge / std::sort overloads with any comparator).
//
// Replaces the reference's merge (algorithms/merge/merge.hpp:222-313:
// merge-path partitioning, hierarchical hybrid merge) and sort
// (algorithms/sort/bitonic_sort.hpp:69-110: an in-place bitonic network of
// log2(n)^2 / 2 global passes) with:
//   merge  one pass over the output in tiles: a partition kernel finds
//          where every tile starts on the merge path (one warp per tile,
//          a 32-way search along the tile's first diagonal), then each
//          block stages its tile's two input ranges in shared memory and
//          every thread merges its ITEMS outputs after its own merge-path
//          search in shared memory; outputs leave in coalesced rows.
//          Reads each input once, writes each output once.  Standard keys
//          have a kernel of their own (merge_keys_kernel).
//   sort   a merge sort: blocks sort tiles in shared memory (a stable
//          odd-even sort of each thread's ITEMS keys in registers, then
//          log2(threads) rounds of merge-path merges of runs in shared
//          memory), then log2(n / tile) global passes of the merge above on
//          pairs of runs, ping-ponging between the keys and a scratch array.
// Both are stable: on equal keys the element of the first range (the
// earlier run) comes first, as std::merge requires.  comp(x, y) is a strict
// weak order ("x before y").
#pragma once

#include "common.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <limits>

namespace b2p {

constexpr int kMergeThreads = 256;
// Keys per thread: 64 bytes of keys (the block sort's two shared tiles stay
// within 32 KiB), at most 16.
template <class T>
__host__ __device__ constexpr int merge_items() {
  return sizeof(T) <= 4 ? 16 : (sizeof(T) <= 8 ? 8 : (sizeof(T) <= 16 ? 4 : (sizeof(T) <= 32 ? 2 : 1)));
}
template <class T>
__host__ __device__ constexpr int merge_tile() {
  return kMergeThreads * merge_items<T>();
}

// Number of elements of `a` among the first `diag` outputs of the stable
// merge of a[0..na) and b[0..nb) (a(i), b(i) read element i): the first i
// in [max(0, diag - nb), min(diag, na)] whose b[diag - 1 - i] is strictly
// before a[i].
template <class T, class Comp, class IdxA, class IdxB>
__device__ __forceinline__ long long merge_path(IdxA a, long long na, IdxB b, long long nb, long long diag,
                                                const Comp &comp) {
  long long lo = diag > nb ? diag - nb : 0;
  long long hi = diag < na ? diag : na;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    // a[mid] goes before b[diag - 1 - mid] unless b's key is strictly smaller
    if (!comp(b(diag - 1 - mid), a(mid))) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// merge_path() by one warp: each round the 32 lanes test 32 evenly spaced
// points of the remaining range at once and keep the gap where the answer
// lies (a range of `span` shrinks to about span / 33 per round: 6 rounds of
// global-memory latency for 2^28 keys instead of 28).  Every lane returns
// the same value.
template <class T, class Comp, class IdxA, class IdxB>
__device__ __forceinline__ long long merge_path_warp(IdxA a, long long na, IdxB b, long long nb, long long diag,
                                                     const Comp &comp) {
  const int lane = threadIdx.x & 31;
  long long lo = diag > nb ? diag - nb : 0;
  long long hi = diag < na ? diag : na;
  while (lo < hi) {
    const long long span = hi - lo;
    if (span <= 32) {
      const bool p = lane < span && comp(b(diag - 1 - (lo + lane)), a(lo + lane));
      const unsigned m = __ballot_sync(0xffffffffu, p);
      return m ? lo + (__ffs(m) - 1) : hi;
    }
    // probes lo + span * (k + 1) / 33, k = 0..31: strictly increasing, < hi
    const long long pk = lo + span * (lane + 1) / 33;
    const bool p = comp(b(diag - 1 - pk), a(pk));
    const unsigned m = __ballot_sync(0xffffffffu, p);
    const int j = m ? __ffs(m) - 1 : 32;
    const long long new_lo = j == 0 ? lo : lo + span * j / 33 + 1;
    const long long new_hi = j == 32 ? hi : lo + span * (j + 1) / 33;
    lo = new_lo;
    hi = new_hi;
  }
  return lo;
}

// merge_path() by groups of G lanes, each group with its own diagonal and
// range [lo, hi] (which must hold the answer): a range of `span` shrinks to
// about span / (G + 1) per round.  All 32 lanes call it; every lane of a group
// returns the group's value.
template <int G, class Int, class Comp, class IdxA, class IdxB>
__device__ __forceinline__ Int merge_path_groups(IdxA a, IdxB b, Int lo, Int hi, Int diag, const Comp &comp) {
  const int lane = threadIdx.x & 31, gl = lane % G;
  constexpr unsigned kMask = G == 32 ? 0xffffffffu : (1u << G) - 1u;
  while (__any_sync(0xffffffffu, lo < hi)) {
    const Int span = hi - lo;
    const bool few = span <= G;
    const Int pk = few ? lo + gl : lo + span * (gl + 1) / (G + 1);
    const bool p = pk < hi && comp(b(diag - 1 - pk), a(pk));
    const unsigned m = (__ballot_sync(0xffffffffu, p) >> (lane - gl)) & kMask;
    const int j = m ? __ffs(m) - 1 : G;
    const Int at = lo;
    if (few) {
      lo = hi = m ? at + j : hi;
    } else {
      if (j > 0) lo = at + span * j / (G + 1) + 1;
      if (j < G) hi = at + span * (j + 1) / (G + 1);
    }
  }
  return lo;
}

// Shared-memory slot of tile element i: one pad slot after every 32, so
// the threads of a warp, whose runs start ITEMS (a power of two) apart,
// read and write 32 different banks.
__device__ __forceinline__ int spad(int i) { return i + (i >> 5); }
__host__ __device__ constexpr int spad_size(int n) { return n + n / 32; }
// Shared slots of a padded tile of n keys plus the spare slot one past it
// (read, never used, by merge_serial when a side ends at the tile's end).
__host__ __device__ constexpr int spad_alloc(int n) { return spad_size(n) + 1; }

// Serial stable merge of ITEMS outputs starting at a[ia], b[ib] of the two
// ranges s[pad(a0 + i)] and s[pad(b0 + i)] of one padded shared array
// into out[]; the current key of each range stays in a register, and each
// output costs one shared load, without branches (the warp's threads take
// different sides).  Outputs past the end of both ranges are left
// unspecified.  The second range follows the first (b0 >= a0 + na), and
// reads stay in slots a0 .. b0 + nb: one past the end of a side is the
// first slot of the next range or, past the tile, the array's spare last
// slot (kept by spad_alloc); once both sides are exhausted the a-side index,
// which keeps counting, is held at b0 + nb.  Keys read past a side's end
// are never compared or used.
template <class T, int ITEMS, class Comp>
__device__ __forceinline__ void merge_serial(const T *s, int a0, int ia, int na, int b0, int ib, int nb,
                                             T (&out)[ITEMS], const Comp &comp) {
  const int end = b0 + nb;
  T va = s[spad(a0 + ia)];
  T vb = s[spad(b0 + ib)];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const bool take_b = ib < nb && (ia >= na || comp(vb, va));
    out[k] = take_b ? vb : va;
    ia += take_b ? 0 : 1;
    ib += take_b ? 1 : 0;  // ib <= nb: b is taken only while ib < nb
    // the next key of the side just taken (one past its end when exhausted)
    const T v = s[spad(take_b ? b0 + ib : min(a0 + ia, end))];
    vb = take_b ? v : vb;
    va = take_b ? va : v;
  }
}

// Store the ITEMS keys of v to dst[0..count): 16-byte vector stores when the
// whole run is there and dst is 16-byte aligned.
template <class T, int ITEMS>
__device__ __forceinline__ void store_run(T *dst, const T (&v)[ITEMS], int count) {
  constexpr int kBytes = (int)sizeof(T) * ITEMS;
  if constexpr (kBytes % 16 == 0) {
    if (count == ITEMS && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
      uint4 w[kBytes / 16];
      memcpy(w, v, kBytes);
#pragma unroll
      for (int j = 0; j < kBytes / 16; ++j) reinterpret_cast<uint4 *>(dst)[j] = w[j];
      return;
    }
  }
#pragma unroll
  for (int k = 0; k < ITEMS; ++k)
    if (k < count) dst[k] = v[k];
}

// Where each tile starts on its merge path, for the pairwise merge of runs
// of length `run` (PAIRS; a == b == src, na = n, nb = 0) or the one merge
// of a[0..na) and b[0..nb): one warp per tile, splits[t] = the number of
// keys of the tile's first range (A) before the tile's first output.  All
// searches run at once, so the merge kernel starts loading at once.
template <class T>
struct PairView {
  const T *A, *B;
  long long nA, nB, base;
};

template <class T, bool PAIRS>
__device__ __forceinline__ PairView<T> pair_of(const T *a, long long na, const T *b, long long nb, long long run,
                                               long long d0) {
  PairView<T> v{a, b, na, nb, 0};
  if constexpr (PAIRS) {
    v.base = d0 / (2 * run) * (2 * run);
    v.A = a + v.base;
    v.nA = min(run, na - v.base);
    v.B = a + v.base + v.nA;
    v.nB = min(run, na - v.base - v.nA);
  }
  return v;
}

// Keys of the first range among a tile's cnt outputs, from the tile's start
// (i0 and j0 of nA and nB keys) and the first range's index i1 where the tile
// ends.  i1 - i0 for ordered ranges; ranges that are not (NaNs among the keys)
// can give tile starts that cross, and the result then keeps the tile inside
// both ranges.
__host__ __device__ __forceinline__ int merge_tile_count(long long i0, long long i1, long long nA, long long j0,
                                                         long long nB, int cnt) {
  const long long low = cnt - (nB - j0), high = nA - i0;
  long long n = i1 - i0;
  n = n > low ? n : low;
  n = n > 0 ? n : 0;
  n = n < high ? n : high;
  return (int)(n < cnt ? n : cnt);
}

template <class T, class Comp, bool PAIRS>
__global__ void __launch_bounds__(256) merge_partition_kernel(const T *a, long long na, const T *b, long long nb,
                                                              long long run, long long ntiles, long long *splits,
                                                              Comp comp) {
  constexpr int kMergeTile = merge_tile<T>();
  const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= ntiles) return;  // whole warps leave together
  const PairView<T> v = pair_of<T, PAIRS>(a, na, b, nb, run, t * kMergeTile);
  const T *A = v.A, *B = v.B;
  auto ga = [&](long long i) { return A[i]; };
  auto gb = [&](long long i) { return B[i]; };
  const long long sp = merge_path_warp<T>(ga, v.nA, gb, v.nB, t * kMergeTile - v.base, comp);
  if ((threadIdx.x & 31) == 0) splits[t] = sp;
}

// Merge tile `blockIdx.x` of the pairwise merge of runs of length `run`
// (PAIRS) or of the one merge of a and b, from the tile starts in `splits`
// (merge_partition_kernel).  The tile ends where the next tile starts, or,
// for the last tile of its pair, at the end of both ranges.
template <class T, class Comp, bool PAIRS>
__global__ void __launch_bounds__(kMergeThreads) merge_kernel(const T *a, long long na, const T *b, long long nb,
                                                              T *out, long long run, const long long *splits,
                                                              Comp comp) {
  constexpr int kMergeItems = merge_items<T>(), kMergeTile = merge_tile<T>();
  __shared__ T s_in[spad_alloc(kMergeTile)];
  const long long total = PAIRS ? na : na + nb;
  const long long d0 = (long long)blockIdx.x * kMergeTile;
  if (d0 >= total) return;
  const PairView<T> v = pair_of<T, PAIRS>(a, na, b, nb, run, d0);
  const T *A = v.A, *B = v.B;
  const long long tile_end = min(d0 + kMergeTile, total);
  const long long l1 = tile_end - v.base;
  const long long i0 = splits[blockIdx.x];
  const long long i1 = l1 == v.nA + v.nB ? v.nA : splits[blockIdx.x + 1];
  const long long j0 = (d0 - v.base) - i0;
  const int cnt = (int)(tile_end - d0);
  const int na_t = merge_tile_count(i0, i1, v.nA, j0, v.nB, cnt), nb_t = cnt - na_t;
  if (cnt == kMergeTile) {
    // a full tile: every thread's ITEMS loads in flight at once
    const T *pa = A + i0, *pb = B + (j0 - na_t);
    T r[kMergeItems];
#pragma unroll
    for (int q = 0; q < kMergeItems; ++q) {
      const int k = threadIdx.x + q * kMergeThreads;
      r[q] = (k < na_t ? pa : pb)[k];
    }
#pragma unroll
    for (int q = 0; q < kMergeItems; ++q) s_in[spad(threadIdx.x + q * kMergeThreads)] = r[q];
  } else {
    for (int k = threadIdx.x; k < cnt; k += kMergeThreads)
      s_in[spad(k)] = k < na_t ? A[i0 + k] : B[j0 + (k - na_t)];
  }
  __syncthreads();
  const int dt = min((int)threadIdx.x * kMergeItems, cnt);
  auto sa = [&](long long i) { return s_in[spad((int)i)]; };
  auto sb = [&](long long i) { return s_in[spad(na_t + (int)i)]; };
  const int it = (int)merge_path<T>(sa, na_t, sb, nb_t, dt, comp);
  T v_[kMergeItems];
  merge_serial(s_in, 0, it, na_t, na_t, dt - it, nb_t, v_, comp);
  // each thread's outputs are contiguous: straight from registers
  store_run(out + d0 + dt, v_, min(kMergeItems, cnt - dt));
}

// Sort tile `blockIdx.x` of keys[0..n) in place (stable).
template <class T, class Comp>
__global__ void __launch_bounds__(kMergeThreads) block_sort_kernel(T *keys, long long n, Comp comp) {
  constexpr int kMergeItems = merge_items<T>(), kMergeTile = merge_tile<T>();
  __shared__ T s_a[spad_alloc(kMergeTile)];
  __shared__ T s_b[spad_alloc(kMergeTile)];
  const long long t0 = (long long)blockIdx.x * kMergeTile;
  const int cnt = (int)min((long long)kMergeTile, n - t0);
  if (cnt == kMergeTile) {
    T r[kMergeItems];
#pragma unroll
    for (int q = 0; q < kMergeItems; ++q) r[q] = keys[t0 + threadIdx.x + q * kMergeThreads];
#pragma unroll
    for (int q = 0; q < kMergeItems; ++q) s_a[spad(threadIdx.x + q * kMergeThreads)] = r[q];
  } else {
    for (int k = threadIdx.x; k < cnt; k += kMergeThreads) s_a[spad(k)] = keys[t0 + k];
  }
  __syncthreads();
  // each thread: its ITEMS keys, sorted by odd-even transposition (stable:
  // neighbours swap only when the right one is strictly before the left)
  const int b0 = threadIdx.x * kMergeItems;
  const int mine = max(0, min(kMergeItems, cnt - b0));
  T v[kMergeItems];
#pragma unroll
  for (int k = 0; k < kMergeItems; ++k)
    if (k < mine) v[k] = s_a[spad(b0 + k)];
#pragma unroll
  for (int r = 0; r < kMergeItems; ++r) {
#pragma unroll
    for (int k = r & 1; k + 1 < kMergeItems; k += 2) {
      if (k + 1 < mine && comp(v[k + 1], v[k])) {
        const T x = v[k];
        v[k] = v[k + 1];
        v[k + 1] = x;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kMergeItems; ++k)
    if (k < mine) s_a[spad(b0 + k)] = v[k];
  __syncthreads();
  // rounds: runs of ITEMS, 2 ITEMS, ... merged pairwise in shared memory
  T *src = s_a, *dst = s_b;
  for (int run = kMergeItems; run < cnt; run *= 2) {
    const int d = b0;  // this thread's outputs [d, d + ITEMS)
    const bool last = 2 * run >= cnt;  // the same for the whole block
    if (d < cnt) {
      const int pb = d / (2 * run) * (2 * run);
      const int la = min(run, cnt - pb), lb = max(0, min(run, cnt - pb - la));
      auto sa = [&](long long i) { return src[spad(pb + (int)i)]; };
      auto sb = [&](long long i) { return src[spad(pb + la + (int)i)]; };
      const int dl = d - pb;
      const int ia = (int)merge_path<T>(sa, la, sb, lb, dl, comp);
      T w[kMergeItems];
      merge_serial(src, pb, ia, la, pb + la, dl - ia, lb, w, comp);
      if (last) {  // the sorted tile leaves from registers
        store_run(keys + t0 + d, w, min(kMergeItems, cnt - d));
      } else {
#pragma unroll
        for (int k = 0; k < kMergeItems; ++k)
          if (d + k < cnt) dst[spad(d + k)] = w[k];
      }
    }
    if (last) return;
    __syncthreads();
    T *x = src;
    src = dst;
    dst = x;
  }
  // no merge round (cnt <= ITEMS): the first thread's sorted keys
  for (int k = threadIdx.x; k < cnt; k += kMergeThreads) keys[t0 + k] = src[spad(k)];
}

// ------------------------------------------------- merge of standard keys
//
// The same merge for int, float and 64-bit keys under < or >, where a key is
// its own order.  The keys of a thread's ITEMS outputs are read as an ascending
// run of a followed by a descending run of b (begun one key late, at a key that
// is no earlier than any of them), which the log2(ITEMS + 1) rounds of a
// bitonic merge sort in registers (a min and a max per two keys and round),
// instead of a serial merge whose every output takes about 16 instructions and
// waits for a shared load.  ITEMS is odd: the threads' searches start, and
// their outputs lie, in different banks.  Keys that compare equal have the same bits, so
// their order cannot be seen; a thread that meets an exception, a -0.0 (equal
// to +0.0) or a NaN (unordered), merges serially, and so does one whose
// outputs run past the end.
//
// 133 M floats: 229 us, 4.65 TB/s (the serial merge's kernel took 283 us); 2^28
// int32: 455 us (559).  Bound by latency between its barriers at 25 warps per
// SM, with the shared-memory pipe 63 % and the ALU pipe 49 % busy; the random
// banks of the windows and searches are two thirds of the wavefronts.
template <class T>
struct MergeNet {
  static constexpr int kItems = sizeof(T) == 4 ? 31 : 15, kThreads = 160, kBlocksPerSm = 5;
  static constexpr int kTile = kItems * kThreads;  // no smaller than merge_tile<T>(): no more tile starts
  // a staged tile: both sides from and to 16-byte boundaries, a key after b
  static constexpr int kSlots = kTile + 5 * 16 / (int)sizeof(T);
};

template <class T, bool DESC>
struct KeyOrder {
  __device__ __forceinline__ bool operator()(const T &x, const T &y) const { return DESC ? y < x : x < y; }
  __device__ __forceinline__ static T first(T x, T y) {
    if constexpr (std::is_same<T, float>::value) return DESC ? fmaxf(x, y) : fminf(x, y);
    else return DESC ? (x < y ? y : x) : (y < x ? y : x);
  }
  __device__ __forceinline__ static T second(T x, T y) {
    if constexpr (std::is_same<T, float>::value) return DESC ? fminf(x, y) : fmaxf(x, y);
    else return DESC ? (x < y ? x : y) : (y < x ? x : y);
  }
  // a key that none goes after
  __device__ __forceinline__ static T last_key() {
    using L = std::numeric_limits<T>;
    if constexpr (std::is_floating_point<T>::value) return DESC ? -L::infinity() : L::infinity();
    else return DESC ? L::min() : L::max();
  }
  // a key whose order against an equal or any other key is not in its bits
  __device__ __forceinline__ static bool special(T x) {
    if constexpr (std::is_same<T, float>::value) {
      const unsigned u = __float_as_uint(x);
      return u == 0x80000000u || (u << 1) > 0xff000000u;
    } else if constexpr (std::is_same<T, double>::value) {
      const unsigned long long u = (unsigned long long)__double_as_longlong(x);
      return u == 0x8000000000000000ull || (u << 1) > 0xffe0000000000000ull;
    } else {
      return false;
    }
  }
};

// splits[t] = keys of a before output t * kTile.  A warp takes TILES tiles: the
// merge path at both ends of their outputs (16 lanes each), then each tile's
// start between them (32 / TILES lanes each).  TILES = 1: one 32-lane search
// per tile, the fewest rounds of latency (2.8 us for 167 tiles of two 64-bit
// sides, against 6.7 us for eight tiles a warp), but 345 scattered sectors a
// tile: 85 us for 133 M floats, where 32 tiles a warp take 27 us.
template <class T, bool DESC, int TILES>
__global__ void __launch_bounds__(128) merge_keys_partition_kernel(const T *a, long long na, const T *b, long long nb,
                                                                   long long ntiles, long long *splits) {
  constexpr long long kTile = MergeNet<T>::kTile;
  const KeyOrder<T, DESC> comp;
  const int lane = threadIdx.x & 31;
  const long long t0 = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * TILES;
  grid_wait();
  grid_trigger();
  if (t0 >= ntiles) return;  // whole warps leave together
  auto ga = [&](long long i) { return a[i]; };
  auto gb = [&](long long i) { return b[i]; };
  const long long d0 = t0 * kTile;
  if constexpr (TILES == 1) {
    const long long i = merge_path_warp<T>(ga, na, gb, nb, d0, comp);
    if (lane == 0) splits[t0] = i;
  } else {
    constexpr int G = 32 / TILES;
    const long long d1 = min(d0 + TILES * kTile, na + nb);
    long long d = lane < 16 ? d0 : d1;
    const long long e = merge_path_groups<16, long long>(ga, gb, d > nb ? d - nb : 0, min(d, na), d, comp);
    const long long i0 = __shfl_sync(0xffffffffu, e, 0), i1 = __shfl_sync(0xffffffffu, e, 16);
    const long long t = t0 + lane / G;
    d = min(t * kTile, d1);
    // outputs [d0, d) take at least d - (keys of b up to d1), and no more than
    // d - (keys of b up to d0), keys of a
    const long long i =
        merge_path_groups<G, long long>(ga, gb, max(i0, d - (d1 - i1)), min(i1, d - (d0 - i0)), d, comp);
    if (lane % G == 0 && t < ntiles) splits[t] = i;
  }
}

// One side of a tile, keys [0, count) from src, into the 16-byte chunks of
// `slots` from chunk c0 on, by cp.async: chunks as they lie in memory, so the
// first key is at slot (src's offset from a 16-byte boundary).  Only keys of
// the side's array [begin, end) are read.
template <class T>
__device__ __forceinline__ void merge_stage_chunk(T *slots, int c, const T *src, int chunk, const T *begin,
                                                  const T *end) {
  const char *p = reinterpret_cast<const char *>(reinterpret_cast<uintptr_t>(src) & ~uintptr_t(15)) + 16ll * chunk;
  const unsigned d = (unsigned)__cvta_generic_to_shared(reinterpret_cast<uint4 *>(slots) + c);
  if (p >= reinterpret_cast<const char *>(begin) && p + 16 <= reinterpret_cast<const char *>(end)) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(p) : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 16; i += (int)sizeof(T)) {
      const char *e = p + i;
      if (e >= reinterpret_cast<const char *>(begin) && e < reinterpret_cast<const char *>(end))
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + i), "l"(e), "n"((int)sizeof(T)) : "memory");
    }
  }
}

// Keys of a among the ITEMS outputs between a thread's split and the next one's:
// their difference when both sides are in order.  Keys that are not, NaNs among
// others, can give splits that cross or lie more than ITEMS apart; the bounds then
// keep the thread's keys inside the tile, for each split by itself leaves no
// more keys of a side than there are.
template <int ITEMS>
__host__ __device__ __forceinline__ int merge_window(int lo, int next) {
  return (int)min((unsigned)max(next, lo) - (unsigned)lo, (unsigned)ITEMS);
}

// Persistent blocks: a block's next tile is on its way into the other buffer
// while it merges the one it holds.
template <class T, bool DESC>
__global__ void __launch_bounds__(MergeNet<T>::kThreads, MergeNet<T>::kBlocksPerSm)
    merge_keys_kernel(const T *a, long long na, const T *b, long long nb, T *out, long long ntiles,
                      const long long *splits) {
  constexpr int ITEMS = MergeNet<T>::kItems, N = ITEMS + 1, NT = MergeNet<T>::kThreads, TILE = MergeNet<T>::kTile,
                SLOTS = MergeNet<T>::kSlots, IPV = 16 / (int)sizeof(T);
  static_assert(TILE % IPV == 0 && SLOTS % IPV == 0, "tiles and buffers start on 16-byte boundaries");
  using K = KeyOrder<T, DESC>;
  __shared__ __align__(16) T buf[2 * SLOTS];
  __shared__ int s_lo[NT + 1];
  const K comp;
  const int t = threadIdx.x;
  const long long total = na + nb;
  const bool vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;

  // the tile's keys of a: [i0, i1)
  auto range = [&](long long tile, long long &i0, long long &i1) {
    if (tile >= ntiles) return;
    i0 = __ldcg(splits + tile);
    i1 = tile + 1 < ntiles ? __ldcg(splits + tile + 1) : na;
  };
  // start staging a tile; where its sides are: na_t keys of a from slot a0, the
  // others of its cnt keys from slot b0
  auto stage = [&](T *slots, long long tile, long long i0, long long i1, int &na_t, int &cnt, int &a0, int &b0) {
    const long long d0 = tile * TILE;
    cnt = (int)min((long long)TILE, total - d0);
    na_t = merge_tile_count(i0, i1, na, d0 - i0, nb, cnt);
    const T *pa = a + i0, *pb = b + (d0 - i0);
    a0 = (int)(reinterpret_cast<uintptr_t>(pa) & 15) / (int)sizeof(T);
    const int shift_b = (int)(reinterpret_cast<uintptr_t>(pb) & 15) / (int)sizeof(T);
    const int ca = (a0 + na_t + IPV - 1) / IPV, cb = (shift_b + (cnt - na_t) + IPV - 1) / IPV;
    b0 = ca * IPV + shift_b;
    for (int c = t; c < ca + cb; c += NT)
      merge_stage_chunk(slots, c, c < ca ? pa : pb, c < ca ? c : c - ca, c < ca ? a : b, c < ca ? a + na : b + nb);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  long long tile = blockIdx.x, i0 = 0, i1 = 0;
  int na_n = 0, cnt_n = 0, a0_n = 0, b0_n = 0;
  grid_wait();
  grid_trigger();
  range(tile, i0, i1);
  stage(buf, tile, i0, i1, na_n, cnt_n, a0_n, b0_n);
  range(tile + gridDim.x, i0, i1);
  T *s = buf, *other = buf + SLOTS;
  for (; tile < ntiles; tile += gridDim.x) {
    const int na_t = na_n, cnt = cnt_n, nb_t = cnt_n - na_n;
    const T *sa = s + a0_n;
    T *sb = s + b0_n;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the tile is staged, and the other buffer's outputs are stored
    if (tile + gridDim.x < ntiles) {
      stage(other, tile + gridDim.x, i0, i1, na_n, cnt_n, a0_n, b0_n);
      range(tile + 2 * (long long)gridDim.x, i0, i1);
    }
    const int d = min(t * ITEMS, cnt);
    // keys of a before output d: the first in [lo, hi] that a key of b precedes
    int lo = max(0, d - nb_t);
    {
      const int hi = min(d, na_t);  // hi - lo <= TILE / 2
      constexpr int kTop = sizeof(T) == 4 ? 2048 : 1024;
      static_assert(2 * kTop - 1 >= TILE / 2, "the steps reach every place");
      const T *pa = sa + lo, *pb = sb + (d - 1 - lo);
#pragma unroll
      for (int step = kTop; step > 0; step /= 2) {
        if (lo + step <= hi && !comp(pb[1 - step], pa[step - 1])) {
          lo += step;
          pa += step;
          pb -= step;
        }
      }
    }
    s_lo[t] = lo;
    if (t == 0) {
      s_lo[NT] = na_t;
      sb[nb_t] = K::last_key();
    }
    __syncthreads();
    const int ca = merge_window<ITEMS>(lo, s_lo[t + 1]);
    T v[N];
    bool serial = d + ITEMS > cnt;
    if (!serial) {
      const T *pa = sa + lo, *pb = sb + (d - lo + ITEMS);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        v[i] = *(i < ca ? pa + i : pb - i);
        serial |= K::special(v[i]);
      }
#pragma unroll
      for (int h = N / 2; h > 0; h >>= 1) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
          if (i & h) continue;
          const T x = v[i], y = v[i + h];
          v[i] = K::first(x, y);
          v[i + h] = K::second(x, y);
        }
      }
    }
    if (serial) {
      int ia = lo, ib = d - lo;
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        const T x = sa[min(ia, na_t)], y = sb[min(ib, nb_t)];
        const bool take_b = ib < nb_t && (ia >= na_t || comp(y, x));
        v[k] = take_b ? y : x;
        ia += !take_b;
        ib += take_b;
      }
    }
    __syncthreads();  // every key is read
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) s[t * ITEMS + k] = v[k];
    __syncthreads();
    T *o = out + tile * TILE;
    if (cnt == TILE && vec) {
#pragma unroll
      for (int q = t; q < TILE / IPV; q += NT)
        st_stream_v4(reinterpret_cast<uint4 *>(o) + q, reinterpret_cast<const uint4 *>(s)[q]);
    } else {
      for (int k = t; k < cnt; k += NT) o[k] = s[k];
    }
    T *const x = s;
    s = other;
    other = x;
  }
}

// ------------------------------------------------------------------ host

// Scratch of a merge of `total` keys: the tile starts.
template <class T>
inline size_t merge_scratch_bytes(size_t total) {
  return ((total + merge_tile<T>() - 1) / merge_tile<T>() + 1) * sizeof(long long) + 256;
}

// Stable merge of a[0..na) and b[0..nb) into out (asynchronous on st);
// scratch: merge_scratch_bytes<T>(na + nb) bytes of device memory.
template <class T, class Comp>
int launch_merge(const T *a, size_t na, const T *b, size_t nb, T *out, const Comp &comp, void *scratch,
                 size_t scratch_bytes, cudaStream_t st) {
  const long long total = (long long)(na + nb);
  if (total == 0) return B2P_OK;
  const long long tiles = (total + merge_tile<T>() - 1) / merge_tile<T>();
  if (tiles > 0x7fffffffLL / 32) return B2P_ERR_INVALID_ARG;
  if (!scratch || scratch_bytes < merge_scratch_bytes<T>((size_t)total) - 256) return B2P_ERR_SCRATCH;
  long long *splits = reinterpret_cast<long long *>(scratch);
  merge_partition_kernel<T, Comp, false><<<(unsigned)((tiles * 32 + 255) / 256), 256, 0, st>>>(
      a, (long long)na, b, (long long)nb, total, tiles, splits, comp);
  merge_kernel<T, Comp, false><<<(unsigned)tiles, kMergeThreads, 0, st>>>(a, (long long)na, b, (long long)nb, out,
                                                                          total, splits, comp);
  return cudaGetLastError() == cudaSuccess ? B2P_OK : B2P_ERR_CUDA;
}

// Whether a merge of standard keys takes the kernels below or launch_merge().
// The network's tiles are larger, so the GPU fills later: up to 2^18 keys that
// does not matter (one tile per SM or fewer) and the two kernels overlap their
// starts, from 7 x 2^18 on the cheaper merge outweighs it, between them
// launch_merge() is the faster one (600,000 + 500,000 int32 7.7 us against 9.1,
// int64 9.6 against 9.9; 1,000,000 + 900,000 int32 10.5 against 9.2).  8-byte
// keys that come nearly all from one side are a copy, bound by L2 while it
// holds them: 3,000,000 + 3,000 int64 13.7 against 15.2, 14,500,000 + 3,900 54.7
// against 56.1, 25,000,000 + 3,000 94.8 against 93.9.
constexpr long long kMergeEarlyKeys = 1ll << 18, kMergeNetKeys = 7ll << 18, kMergeLopsidedKeys = 1ll << 24;

template <class T>
inline bool merge_by_network(size_t na, size_t nb) {
  const long long total = (long long)(na + nb), small = (long long)std::min(na, nb);
  if (total <= kMergeEarlyKeys) return true;
  if (sizeof(T) == 8 && small < total / 64 && total < kMergeLopsidedKeys) return false;
  return total >= kMergeNetKeys;
}

// The same for standard keys, ascending or descending.
template <class T, bool DESC>
int launch_merge_keys(const T *a, size_t na, const T *b, size_t nb, T *out, void *scratch, size_t scratch_bytes,
                      int sm_count, cudaStream_t st) {
  const long long total = (long long)(na + nb);
  if (total == 0) return B2P_OK;
  const long long tiles = (total + MergeNet<T>::kTile - 1) / MergeNet<T>::kTile;
  if (tiles > 0x7fffffffLL / 32) return B2P_ERR_INVALID_ARG;
  if (!scratch || scratch_bytes < merge_scratch_bytes<T>((size_t)total) - 256) return B2P_ERR_SCRATCH;
  long long *splits = reinterpret_cast<long long *>(scratch);
  // Tiles per partition warp: one search per warp while the tiles are few
  // (latency), more as their scattered reads add up.  10.5 M + 10.5 M int32 (4,234
  // tiles) 58.0 us with 1, 57.6 with 8, 64.0 with 32; 25 M + 25 M (10,081 tiles)
  // 133, 109, 114; 133 M (26,882 tiles) 308, 259, 255.
  const int per_warp = tiles <= 4096 ? 1 : tiles <= 16384 ? 8 : 32;
  const auto partition = per_warp == 1   ? merge_keys_partition_kernel<T, DESC, 1>
                         : per_warp == 8 ? merge_keys_partition_kernel<T, DESC, 8>
                                         : merge_keys_partition_kernel<T, DESC, 32>;
  const long long grid = std::min<long long>(tiles, (long long)sm_count * MergeNet<T>::kBlocksPerSm);
  // Started while the kernel before ends only when the SMs have room for both:
  // an early partition of the next merge keeps merge blocks of this one waiting
  // (2,000,000 + 1,500,000 int32 12.0 us in order, 19.1 early).
  const bool early = total <= kMergeEarlyKeys;
  if (launch_dependent(early, partition, (unsigned)((tiles + 4 * per_warp - 1) / (4 * per_warp)), 128, 0, st, a,
                       (long long)na, b, (long long)nb, tiles, splits) != cudaSuccess ||
      launch_dependent(early, merge_keys_kernel<T, DESC>, (unsigned)grid, MergeNet<T>::kThreads, 0, st, a, (long long)na,
                       b, (long long)nb, out, tiles, (const long long *)splits) != cudaSuccess)
    return B2P_ERR_CUDA;
  return B2P_OK;
}

// Scratch a sort of n keys of T needs: a second array of n keys, then the
// tile starts of the merge passes.
template <class T>
inline size_t sort_keys_bytes(size_t n) {
  return (n * sizeof(T) + 255) / 256 * 256;
}
template <class T>
inline size_t sort_scratch_bytes(size_t n) {
  return sort_keys_bytes<T>(n) + merge_scratch_bytes<T>(n);
}

// Stable merge sort of keys[0..n) in place; scratch: sort_scratch_bytes<T>(n)
// bytes of device memory (none when n fits one tile).
template <class T, class Comp>
int launch_sort(T *keys, size_t n, const Comp &comp, void *scratch, size_t scratch_bytes, cudaStream_t st) {
  if (n <= 1) return B2P_OK;
  constexpr long long kMergeTile = merge_tile<T>();
  const long long tiles = ((long long)n + kMergeTile - 1) / kMergeTile;
  if (tiles > 0x7fffffffLL / 32) return B2P_ERR_INVALID_ARG;
  if (tiles > 1 && (!scratch || scratch_bytes < sort_scratch_bytes<T>(n) - 256)) return B2P_ERR_SCRATCH;
  block_sort_kernel<T, Comp><<<(unsigned)tiles, kMergeThreads, 0, st>>>(keys, (long long)n, comp);
  if (tiles == 1) return cudaGetLastError() == cudaSuccess ? B2P_OK : B2P_ERR_CUDA;
  T *src = keys, *dst = reinterpret_cast<T *>(scratch);
  long long *splits = reinterpret_cast<long long *>(reinterpret_cast<char *>(scratch) + sort_keys_bytes<T>(n));
  for (long long run = kMergeTile; run < (long long)n; run *= 2) {
    merge_partition_kernel<T, Comp, true><<<(unsigned)((tiles * 32 + 255) / 256), 256, 0, st>>>(
        src, (long long)n, src, 0, run, tiles, splits, comp);
    merge_kernel<T, Comp, true><<<(unsigned)tiles, kMergeThreads, 0, st>>>(src, (long long)n, src, 0, dst, run,
                                                                          splits, comp);
    T *x = src;
    src = dst;
    dst = x;
  }
  if (src != keys && cudaMemcpyAsync(keys, src, n * sizeof(T), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
    return B2P_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? B2P_OK : B2P_ERR_CUDA;
}

}  // namespace b2p
