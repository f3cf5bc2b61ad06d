// LSD radix sort of 4- and 8-byte keys: b2p_sort's path for the standard key
// types (int32/int64/uint32/uint64/float/double with < or >), where the
// reference runs its bitonic network (algorithms/sort/bitonic_sort.hpp:
// 69-110, log2(n)^2 / 2 global passes).
//
// Keys are mapped to unsigned "order keys" whose unsigned order is the key
// order (signed: sign bit flipped; floats: all bits flipped when negative,
// else the sign bit set; -0.0 takes the order key of +0.0, so the two zeros
// are equal as under <; descending: the complement).  The sort moves the
// original bits and is stable, so its result is the stable sort by the key
// order: the same as a stable merge sort with < or >.
//
// Each digit pass (4 for 32-bit keys, 8 for 64-bit) is a reduce-then-scan
// over persistent blocks, ping-ponging between the keys and a second array:
//   * upsweep: block b counts the digits of its contiguous chunk of tiles
//     (shared-memory counters by digit and lane), counts[d][b];
//   * spine: per digit, an exclusive scan of its counts over the chunks and
//     its total; a digit's first slot in chunk b is then the keys of smaller
//     digits plus the keys of that digit in chunks before b;
//   * downsweep: block b walks its chunk's tiles in order, ranks each tile's
//     keys in key order, reorders the tile by digit in shared memory and
//     writes the keys to their slots (running slot of the digit + position in
//     the tile's run of that digit); the running slots advance by the tile's
//     counts.
// Nothing waits on another block, and the sort is stable: chunks, tiles and
// keys inside a tile are taken in index order.
#pragma once

#include "common.cuh"

#include <algorithm>
#include <limits>

namespace b2p {

constexpr int kRadixBits = 8, kRadixBins = 1 << kRadixBits;
// upsweep blocks
constexpr int kRadixThreads = 256, kRadixItems = 16;
constexpr int kRadixStep = kRadixThreads * kRadixItems;  // 4096 keys
// downsweep blocks
constexpr int kDownThreads = 128;
constexpr int kRadixItemBytes = 256;                             // keys of one thread
constexpr int kRadixTileBytes = kDownThreads * kRadixItemBytes;  // 32 KiB
constexpr int kDownBlocksPerSm = 3;                              // 2 x 32 KiB of shared memory each
template <class T>
constexpr long long radix_tile() {
  return kRadixTileBytes / (long long)sizeof(T);
}
constexpr int kRadixSpineThreads = 1024;
// 32-bit slots: inputs below 2^31 keys
constexpr size_t kRadixMaxKeys = (size_t)1 << 31;

// Scratch of a radix sort of n keys of T with `blocks` persistent blocks:
// the per-chunk digit counts (then their prefixes), the digit totals and the
// second key array.
struct RadixLayout {
  size_t counts, totals, keys, total;
  long long ntiles;
  int blocks;
  long long chunk;  // tiles per block
};

template <class T>
inline RadixLayout radix_layout(size_t n, int sm_count) {
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  RadixLayout l;
  l.ntiles = ((long long)n + radix_tile<T>() - 1) / radix_tile<T>();
  const long long want = (long long)std::max(sm_count, 1) * kDownBlocksPerSm;
  l.chunk = (l.ntiles + want - 1) / want;
  l.blocks = (int)((l.ntiles + l.chunk - 1) / l.chunk);
  l.counts = kHeaderBytes;
  l.totals = l.counts + up((size_t)kRadixBins * l.blocks * 4);
  l.keys = l.totals + up((size_t)kRadixBins * 4);
  l.total = l.keys + up(n * sizeof(T));
  return l;
}

// Scratch bytes for any device of up to 256 SMs (the block count follows the
// SM count).
template <class T>
inline size_t radix_scratch_bytes(size_t n) {
  return radix_layout<T>(n, 256).total + 256;
}

// Digit `pass` of a key under the key order.  A key's order digit is its own
// digit, xored with a constant of the pass (the sign bit, the complement of a
// descending sort) and, for floats, with the sign of the key.
template <class T>
struct RadixDigit {
  static constexpr bool kFloat = std::is_floating_point<T>::value;
  static constexpr int kLast = (int)sizeof(T) - 1;
  unsigned place, flip, top;
  bool high;
  __device__ __forceinline__ RadixDigit(int pass, bool desc)
      : place(8u * (pass & 3)),
        flip((desc ? 0xffu : 0u) ^ (std::is_integral<T>::value && std::is_signed<T>::value && pass == kLast ? 0x80u : 0u)),
        top(kFloat && pass == kLast ? 0x80u : 0u),
        high(pass >= 4) {}
  // (digit << SHIFT) ^ c
  template <int SHIFT>
  __device__ __forceinline__ unsigned at(const T &x, unsigned c) const {
    constexpr unsigned M = 0xffu << SHIFT;
    unsigned w, sign = 0;
    if constexpr (sizeof(T) == 4) {
      memcpy(&w, &x, 4);
      if constexpr (kFloat) {
        if (w == 0x80000000u) w = 0;  // -0.0 == +0.0
        sign = (unsigned)((int)w >> 31);
      }
    } else {
      uint2 v;
      memcpy(&v, &x, 8);
      if constexpr (kFloat) {
        if (v.y == 0x80000000u && v.x == 0) v.y = 0;
        sign = (unsigned)((int)v.y >> 31);
      }
      w = high ? v.y : v.x;
    }
    unsigned r = __funnelshift_r(w, w, (place - SHIFT) & 31u) & M;
    if constexpr (kFloat) r ^= (sign & M) | (top << SHIFT);
    return r ^ (c ^ (flip << SHIFT));
  }
};

// Upsweep: digit counts of block b's chunk of tiles, counts[d * blocks + b].
// Counter (digit, lane) is word digit * 32 + lane, one for the lanes of that
// number in all warps: a warp's 32 atomics lie in 32 different banks.  Bound
// by the read: 2^28 int32 keys take 185 us (5.8 TB/s); one counter per digit
// and warp, with its bank conflicts and scalar loads, took 209 us.
template <class T>
__global__ void __launch_bounds__(kRadixThreads) radix_upsweep_kernel(const T *keys, unsigned n, bool desc, int pass,
                                                                    long long chunk, unsigned *counts) {
  __shared__ __align__(16) unsigned sh[kRadixBins * 32];
  constexpr unsigned IPV = 16 / sizeof(T), V = kRadixItems / IPV;
  const unsigned t = threadIdx.x, lane = t & 31u;
  for (unsigned i = t; i < kRadixBins * 8; i += kRadixThreads)
    reinterpret_cast<uint4 *>(sh)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  grid_wait();
  grid_trigger();
  const RadixDigit<T> dg(pass, desc);
  auto count = [&](const T &k) {
    atomicAdd(reinterpret_cast<unsigned *>(reinterpret_cast<char *>(sh) + dg.template at<7>(k, lane << 2)), 1u);
  };
  const unsigned b0 = (unsigned)(blockIdx.x * chunk * radix_tile<T>());
  const unsigned b1 = (unsigned)min((long long)n, b0 + chunk * radix_tile<T>());
  unsigned i = b0;
  if ((reinterpret_cast<uintptr_t>(keys) & 15) == 0) {
    // every thread's V 16-byte loads in flight together
    for (; i + kRadixStep <= b1; i += kRadixStep) {
      uint4 v[V];
#pragma unroll
      for (unsigned r = 0; r < V; ++r) v[r] = ld_stream_l2_v4(keys + i + (r * kRadixThreads + t) * IPV);
#pragma unroll
      for (unsigned r = 0; r < V; ++r) {
        T k[IPV];
        memcpy(k, &v[r], 16);
#pragma unroll
        for (unsigned e = 0; e < IPV; ++e) count(k[e]);
      }
    }
  }
  // what is left, or keys that are not 16-byte aligned: 4-byte keys with eight
  // loads in flight (a last tile's counts: 300,000 int32 56 -> 47 us a sort;
  // 3.6 M unaligned int64 got slower that way, 242 -> 254 us)
  constexpr unsigned kLate = sizeof(T) == 4 ? 8 : 1;
  for (i += t; i < b1; i += kLate * kRadixThreads) {
    T k[kLate];
#pragma unroll
    for (unsigned r = 0; r < kLate; ++r)
      if (i + r * kRadixThreads < b1) k[r] = __ldcg(keys + i + r * kRadixThreads);
#pragma unroll
    for (unsigned r = 0; r < kLate; ++r)
      if (i + r * kRadixThreads < b1) count(k[r]);
  }
  __syncthreads();
  for (unsigned d = t; d < kRadixBins; d += kRadixThreads) {
    unsigned c = 0;
#pragma unroll
    for (unsigned r = 0; r < 32; ++r) c += sh[d * 32 + ((r + d) & 31u)];
    counts[(size_t)d * gridDim.x + blockIdx.x] = c;
  }
}

// Spine, one block per digit d: exclusive scan of the digit's chunk counts
// counts[d][0 .. blocks) in place (blocks <= kRadixSpineThreads), and the
// digit's total into totals[d].
__global__ void __launch_bounds__(kRadixSpineThreads) radix_spine_kernel(unsigned *counts, int blocks,
                                                                       unsigned *totals) {
  __shared__ unsigned s_warp[kRadixSpineThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  unsigned *row = counts + (size_t)blockIdx.x * blocks;
  grid_wait();
  grid_trigger();
  const unsigned c = t < blocks ? __ldcg(row + t) : 0u;
  unsigned incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  unsigned before = 0;
  for (int w = 0; w < warp; ++w) before += s_warp[w];
  if (t < blocks) row[t] = before + incl - c;
  if (t == kRadixSpineThreads - 1) totals[blockIdx.x] = before + incl;
}

// ------------------------------------------------------------- downsweep
//
// Ranking.  Every thread owns kRadixItemBytes / sizeof(T) consecutive keys of
// the tile and its own 8-bit counter of every digit.  Counter (digit, thread)
// is byte `warp` of word digit * 32 + lane, so a warp's 32 counters of any 32
// digits lie in 32 different banks: one shared atomicAdd per key, one
// wavefront per warp whatever the digits are, returns the key's rank among
// the thread's keys of its digit.  A word holds the four threads (one of each
// warp) that own neighbouring key blocks: thread (warp, lane) owns block
// 4 * lane + warp.
//
// The prefix of the counters along the key order is a product with a
// triangular matrix of ones, taken by integer mma.sync straight from the
// counter words: row = digit, k = the bytes of the 32 words, column = word,
// giving for every word the keys of the digit up to and with it.  The bytes
// of the word from the thread's own on are taken off again with one dp4a.
//
// Bound by shared-memory wavefronts: 14.4 per 32 keys (4.2 of them the
// scatter into the sorted tile, whose banks are random), the data pipe 73 %
// busy at 2^26 keys.  2^28 random int32 keys: 670 us a pass; ranking by eight
// ballots per key, 118 instructions per 32 keys, took 1,525 us.  64 keys a
// thread halve the counters' clearing and prefix work per key against 32.
// Three blocks of 128 threads is what 2 x 32 KiB each leaves room for; the
// keys stay in registers (168 per thread) from the count to the scatter.

// D += A * B, 16 digits x 8 words, k = 32 counter bytes.
__device__ __forceinline__ void radix_mma(int (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                          unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Byte offset of 16-byte chunk c of thread row r in the staged tile: rows of
// 256 bytes, chunks swizzled so that neighbouring rows' equal chunks lie in
// different banks.
__device__ __forceinline__ unsigned radix_stage(unsigned r, unsigned c) {
  return r * kRadixItemBytes + ((c ^ (r & 15u)) << 4);
}

// Bring tile `t0 .. t0 + count` of `in` into `buf`, block kb in row
// (kb & 3) * 32 + kb / 4; keys past the end are `pad` (digit 255 in every
// pass, so that they stay behind the tile's real keys).  Full tiles of
// 16-byte aligned input come by cp.async, other tiles key by key.  ALONE: the
// block has nothing to do until the tile is there, so a partial aligned tile
// comes by cp.async too, up to the vector in which the input ends.  (Key by
// key, one after the other, the last tile kept every pass waiting: 400,000
// int32, 49 tiles, 72 us a sort and 49 with it.)
template <class T, bool ALONE>
__device__ __forceinline__ void radix_load_tile(char *buf, const T *in, unsigned t0, unsigned count, bool vec, T pad) {
  constexpr unsigned K = kRadixItemBytes / sizeof(T), TILE = K * kDownThreads, IPV = 16 / sizeof(T);
  const unsigned t = threadIdx.x;
  if (vec && (ALONE || count == TILE)) {
    const char *g = reinterpret_cast<const char *>(in + t0) + t * 16;
    const unsigned c = t & 15u, row0 = ((t >> 4) & 3u) * 32u + (t >> 6), nvec = count / IPV;
#pragma unroll
    for (unsigned q = 0; q < 16; ++q) {
      char *const to = buf + radix_stage(row0 + 2 * q, c);
      const unsigned v = q * kDownThreads + t;
      if (!ALONE || v < nvec) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(to);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(g + (size_t)q * kDownThreads * 16)
                     : "memory");
      } else {
#pragma unroll
        for (unsigned e = 0; e < IPV; ++e)
          reinterpret_cast<T *>(to)[e] = v * IPV + e < count ? __ldcg(in + t0 + v * IPV + e) : pad;
      }
    }
  } else {
    for (unsigned e = t; e < TILE; e += kDownThreads) {
      const unsigned kb = e / K, b = (e % K) * (unsigned)sizeof(T);
      const T x = e < count ? __ldcg(in + t0 + e) : pad;
      *reinterpret_cast<T *>(buf + radix_stage((kb & 3u) * 32u + (kb >> 2), b >> 4) + (b & 15u)) = x;
    }
  }
}

template <class T>
constexpr size_t radix_pass_smem() {
  return 2 * (size_t)kRadixTileBytes;
}

// Downsweep: block b moves its chunk's keys from `in` to their slots in
// `out` by digit `pass`, tile by tile; prefix[d * blocks + b] counts digit d
// in the chunks before b, totals[d] in the whole input (the spine's results).
//
// Two 32 KiB buffers change places from tile to tile: x holds the staged
// keys, then (the keys being in registers) the prefixes, then the tile sorted
// by digit; y holds the counters, then the next tile on its way in.
template <class T>
__global__ void __launch_bounds__(kDownThreads, kDownBlocksPerSm)
    radix_downsweep_kernel(const T *in, T *out, unsigned n, bool desc, int pass, long long chunk,
                           const unsigned *prefix, const unsigned *totals, T pad) {
  constexpr unsigned S = sizeof(T), K = kRadixItemBytes / S, TILE = K * kDownThreads;
  static_assert(K <= 64, "a word's four counters stay below 256 and signed");
  extern __shared__ __align__(128) unsigned char radix_smem[];
  __shared__ __align__(16) unsigned s_tot[kRadixBins], s_start[kRadixBins], s_base[kRadixBins];
  char *x = reinterpret_cast<char *>(radix_smem), *y = x + kRadixTileBytes;

  const unsigned t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const RadixDigit<T> dg(pass, desc);
  auto counter = [&](const T &k) { return dg.template at<7>(k, lane << 2); };

  // exclusive scan of 256 values of shared memory, two per thread
  auto start_of = [&](uint2 &mine) {
    mine = *reinterpret_cast<const uint2 *>(s_tot + 2 * t);
    unsigned before = 0;
    for (unsigned k = 0; k < 2 * warp; ++k) before += s_tot[32 * k + lane];
    before = __reduce_add_sync(0xffffffffu, before);
    unsigned incl = mine.x + mine.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (unsigned)o) incl += v;
    }
    return before + incl - mine.x - mine.y;
  };

  const unsigned ntiles = (n + TILE - 1) / TILE;
  const unsigned tile_begin = (unsigned)(blockIdx.x * chunk);
  const unsigned tile_end = min(ntiles, tile_begin + (unsigned)chunk);
  const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;

  // constants of the rank arithmetic: which byte of an old counter word is
  // this thread's (as byte_perm selectors), minus S for the bytes of a word
  // from this thread's on, and the triangular matrix's three kinds of words
  unsigned sel[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) sel[j] = (0x3210u & ~(0xfu << (4 * j))) | ((4u + warp) << (4 * j));
  const int taken = (int)((((256u - S) & 0xffu) * 0x01010101u) << (8 * warp));
  const unsigned one = 1u << (8 * warp);
  const unsigned g = lane >> 2, q = lane & 3u;
  const unsigned ones = S * 0x01010101u;
  const unsigned b_lt = q < (g >> 1) ? ones : 0u, b_le = q <= (g >> 1) ? ones : 0u,
                 b_mid = (g & 1u) ? b_le : b_lt;

#pragma unroll
  for (int i = 0; i < kRadixTileBytes / (kDownThreads * 16); ++i)
    *reinterpret_cast<uint4 *>(y + (i * kDownThreads + t) * 16) = make_uint4(0, 0, 0, 0);
  grid_wait();
  grid_trigger();
  if (tile_begin < tile_end)
    radix_load_tile<T, true>(x, in, tile_begin * TILE, min(TILE, n - tile_begin * TILE), vec, pad);

  // next output slot of this thread's digits 2t and 2t + 1 in this chunk
  uint2 mine;
  unsigned run0 = __ldcg(prefix + (size_t)(2 * t) * gridDim.x + blockIdx.x),
           run1 = __ldcg(prefix + (size_t)(2 * t + 1) * gridDim.x + blockIdx.x);
  *reinterpret_cast<uint2 *>(s_tot + 2 * t) = __ldcg(reinterpret_cast<const uint2 *>(totals) + t);
  __syncthreads();
  {
    const unsigned start = start_of(mine);
    run0 += start;
    run1 += start + mine.x;
  }

  for (unsigned tile = tile_begin; tile < tile_end; ++tile) {
    const unsigned count = min(TILE, n - tile * TILE);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // keys staged in x, counters in y zero

    // count: the keys' ranks among the thread's own keys of their digits
    T key[K];
    unsigned rk[K / 4];
#pragma unroll
    for (unsigned c = 0; c < 16; ++c) {
      const uint4 v = *reinterpret_cast<const uint4 *>(x + radix_stage(t, c));
      memcpy(key + c * (K / 16), &v, 16);
    }
#pragma unroll
    for (unsigned j = 0; j < K; ++j) {
      const unsigned old = atomicAdd(reinterpret_cast<unsigned *>(y + counter(key[j])), one);
      rk[j / 4] = __byte_perm(j % 4 ? rk[j / 4] : 0u, old, sel[j % 4]);
    }
    __syncthreads();

    // prefixes of the counter words, warp w: digits 64 w .. 64 w + 63.  Lane
    // (g, q) holds words 8 q .. 8 q + 7 of rows g and g + 8 (odd rows load
    // and store their halves the other way round: no bank conflicts).
    unsigned pk[4][8];  // words 8 q + i: row g in the low half, row g + 8 in the high half
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      unsigned a[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const char *row = y + (64 * warp + 16 * m + 8 * h + g) * 128 + q * 32;
        const uint4 u = *reinterpret_cast<const uint4 *>(row + 16 * (g & 1u));
        const uint4 v = *reinterpret_cast<const uint4 *>(row + 16 * (~g & 1u));
        const bool odd = g & 1u;
        a[h][0] = odd ? v.x : u.x, a[h][1] = odd ? v.y : u.y, a[h][2] = odd ? v.z : u.z, a[h][3] = odd ? v.w : u.w;
        a[h][4] = odd ? u.x : v.x, a[h][5] = odd ? u.y : v.y, a[h][6] = odd ? u.z : v.z, a[h][7] = odd ? u.w : v.w;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int d[4] = {0, 0, 0, 0};
#pragma unroll
        for (int s = 0; s < 4; ++s)
          radix_mma(d, a[0][2 * s], a[1][2 * s], a[0][2 * s + 1], a[1][2 * s + 1],
                    2 * s <= 2 * j ? b_le : b_lt,
                    2 * s + 1 <= 2 * j ? b_le : (2 * s + 1 == 2 * j + 1 ? b_mid : b_lt));
        pk[m][2 * j] = __byte_perm(d[0], d[2], 0x5410);
        pk[m][2 * j + 1] = __byte_perm(d[1], d[3], 0x5410);
      }
      if (q == 3) {  // the last word's prefix is the digit's count
        s_tot[64 * warp + 16 * m + g] = (pk[m][7] & 0xffffu) / S;
        s_tot[64 * warp + 16 * m + 8 + g] = (pk[m][7] >> 16) / S;
      }
    }
    __syncthreads();
    {
      const unsigned start = start_of(mine);
      *reinterpret_cast<uint2 *>(s_start + 2 * t) = make_uint2(start * S, (start + mine.x) * S);
      *reinterpret_cast<uint2 *>(s_base + 2 * t) = make_uint2(run0 - start, run1 - (start + mine.x));
      run0 += mine.x;
      run1 += mine.y;
    }
    __syncwarp();  // a warp's rows are its own threads' digits
#pragma unroll
    for (int m = 0; m < 4; ++m) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const unsigned r = 64 * warp + 16 * m + 8 * h + g, st = s_start[r];
        unsigned w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = (h ? pk[m][i] >> 16 : pk[m][i] & 0xffffu) + st;
        const bool odd = g & 1u;
        char *row = x + r * 128 + q * 32;
        *reinterpret_cast<uint4 *>(row + 16 * (g & 1u)) =
            make_uint4(odd ? w[4] : w[0], odd ? w[5] : w[1], odd ? w[6] : w[2], odd ? w[7] : w[3]);
        *reinterpret_cast<uint4 *>(row + 16 * (~g & 1u)) =
            make_uint4(odd ? w[0] : w[4], odd ? w[1] : w[5], odd ? w[2] : w[6], odd ? w[3] : w[7]);
      }
    }
    __syncthreads();

    // each key's place in the sorted tile, in bytes (two 16-bit places per
    // register); 4- or 8-byte slots swizzled by the place's bits from 10 on,
    // so that a warp whose keys all have one digit writes different banks
    constexpr unsigned kSwzShift = S == 4 ? 8 : 7, kSwzMask = S == 4 ? 0x7c : 0x78;
    unsigned pos[K / 2];
#pragma unroll
    for (unsigned j = 0; j < K; ++j) {
      const unsigned o = counter(key[j]);
      int p = __dp4a(*reinterpret_cast<const int *>(y + o), taken, *reinterpret_cast<const int *>(x + o));
      p = __dp4a((int)rk[j / 4], (int)(S << (8 * (j % 4))), p);
      const unsigned z = (unsigned)p ^ (((unsigned)p >> kSwzShift) & kSwzMask);
      pos[j / 2] = j % 2 ? pos[j / 2] | (z << 16) : z;
    }
    __syncthreads();  // counters and prefixes are used up

    if (tile + 1 < tile_end)
      radix_load_tile<T, false>(y, in, (tile + 1) * TILE, min(TILE, n - (tile + 1) * TILE), vec, pad);
#pragma unroll
    for (unsigned j = 0; j < K; ++j) {
      const unsigned z = j % 2 ? pos[j / 2] >> 16 : pos[j / 2] & 0xffffu;
      *reinterpret_cast<T *>(x + z) = key[j];
    }
    __syncthreads();

    // each key to its slot
    auto put = [&](unsigned r) {
      const unsigned i = r * kDownThreads + t;
      const unsigned z = (i * S) ^ (((r * kDownThreads * S) >> kSwzShift) & kSwzMask);
      const T k = *reinterpret_cast<const T *>(x + z);
      const unsigned o = dg.template at<2>(k, 0);
      const unsigned slot = *reinterpret_cast<const unsigned *>(reinterpret_cast<const char *>(s_base) + o) + i;
      if (slot < n) out[slot] = k;
    };
    if (count == TILE) {
#pragma unroll 16
      for (unsigned r = 0; r < K; ++r) put(r);
    } else {
#pragma unroll 4
      for (unsigned r = 0; r * kDownThreads + t < count; ++r) put(r);
    }
    __syncthreads();

    // the sorted tile's buffer takes the next tile's counters
#pragma unroll
    for (int i = 0; i < kRadixTileBytes / (kDownThreads * 16); ++i)
      *reinterpret_cast<uint4 *>(x + (i * kDownThreads + t) * 16) = make_uint4(0, 0, 0, 0);
    char *const z = x;
    x = y;
    y = z;
  }
}

// Radix sort of keys[0..n) in place (stable, by the key order; descending:
// the reversed order, still stable).  1 < n < kRadixMaxKeys; scratch:
// radix_scratch_bytes<T>(n) bytes of device memory, 256-byte aligned.
// The pad key's digit is 255 in every pass.
template <class T>
inline T radix_pad(bool desc) {
  if constexpr (std::is_floating_point<T>::value) {
    const unsigned long long u = desc ? ~0ull : ~0ull >> 1;
    const unsigned v = desc ? ~0u : ~0u >> 1;
    T x;
    if constexpr (sizeof(T) == 4) memcpy(&x, &v, 4);
    else memcpy(&x, &u, 8);
    return x;
  } else {
    return desc ? std::numeric_limits<T>::min() : std::numeric_limits<T>::max();
  }
}

template <class T>
int launch_radix_sort(T *keys, size_t n, bool desc, void *scratch, size_t scratch_bytes, int sm_count,
                      cudaStream_t st) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "4- or 8-byte keys");
  constexpr int P = (int)sizeof(T) * 8 / kRadixBits;
  if (n <= 1) return B2P_OK;
  if (n >= kRadixMaxKeys || sm_count > 256) return B2P_ERR_UNSUPPORTED;
  const RadixLayout l = radix_layout<T>(n, sm_count);
  if (!scratch || scratch_bytes < l.total || (reinterpret_cast<uintptr_t>(scratch) & 255)) return B2P_ERR_SCRATCH;
  char *s = reinterpret_cast<char *>(scratch);
  unsigned *counts = reinterpret_cast<unsigned *>(s + l.counts);
  unsigned *totals = reinterpret_cast<unsigned *>(s + l.totals);
  T *buf = reinterpret_cast<T *>(s + l.keys);
  if (l.blocks > kRadixSpineThreads) return B2P_ERR_UNSUPPORTED;
  constexpr size_t smem = radix_pass_smem<T>();
  if (cudaFuncSetAttribute((const void *)radix_downsweep_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess)
    return B2P_ERR_CUDA;
  // One tile per block: 3 P launches of 3 to 10 us each, whose spine starts
  // while the upsweep ends (1,000,003 doubles 116 -> 113 us, 400,000 103 -> 97).
  // Up to 32 tiles the other two do so as well (131,072 int32 46 -> 43 us).  With
  // more, blocks that wait take places on few SMs, where they then work several
  // to an SM while others have none: 196,608 int64 87 us against 110 with all
  // early, 1,000,003 int32 52 against 66.  Launches of several tiles per block
  // start in order (2^28 int32: 3.81 ms against 4.18).
  const bool spine_early = l.chunk == 1, early = spine_early && l.blocks <= 32;
  const T *src = keys;
  T *dst = buf;
  for (int p = 0; p < P; ++p) {
    if (launch_dependent(early, radix_upsweep_kernel<T>, l.blocks, kRadixThreads, 0, st, src, (unsigned)n, desc, p, l.chunk,
                         counts) != cudaSuccess ||
        launch_dependent(spine_early, radix_spine_kernel, kRadixBins, kRadixSpineThreads, 0, st, counts, l.blocks, totals) !=
            cudaSuccess ||
        launch_dependent(early, radix_downsweep_kernel<T>, l.blocks, kDownThreads, smem, st, src, dst, (unsigned)n, desc, p,
                         l.chunk, counts, totals, radix_pad<T>(desc)) != cudaSuccess)
      return B2P_ERR_CUDA;
    src = dst;
    dst = (dst == buf) ? keys : buf;
  }
  // an even number of passes ends in `keys`
  return cudaGetLastError() == cudaSuccess ? B2P_OK : B2P_ERR_CUDA;
}

}  // namespace b2p
