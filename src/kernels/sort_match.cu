// Utility kernels for key lists: radix sort of 64-bit keys, 8 bits per pass (with an optional
// payload of 32-bit indices), sums of the values of equal keys (sorted by 8 or up to 10 bits per
// pass) and ordered match (merge-join) of two sorted key lists with an assignment operator applied
// to the values of the keys present in both.
//
// They are the device form of helpers the reference ships as headers that nothing includes
// and that do not compile as written: ParallelSort (include/ps/internal/parallel_sort.h:23-55,
// recursive std::thread split + inplace_merge), ParallelOrderedMatch
// (include/ps/internal/parallel_kv_match.h:29-120, recursive merge-join applying
// `dst op= src` per matched key with value width k) and the AssignOp enum
// (include/ps/internal/assign_op.h:12-21).  Users need them to turn unsorted, possibly
// repeated keys into the sorted unique lists Push/Pull require, and servers to match request
// keys against stored keys.
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cmath>
#include <type_traits>
#include <utility>

#include "ps/device/chain.cuh"
#include "ps/device/psdev.h"

namespace psdev {
extern std::atomic<uint64_t> g_launches;

namespace sortk {
// Least-significant-digit radix sort of 64-bit items.  The items are cut into a few hundred
// contiguous chunks, one per CTA that fits on the GPU at a time, and a pass is three launches:
//   digit_count  counts the digits of every chunk;
//   digit_scan   turns the counts of each digit into how many items of the chunks before have it
//                (left to the scatter when there are few chunks, see kSelfScan);
//   scatter      takes its chunk tile by tile: ranks each item among the items of the same digit in
//                input order (the sort is stable), puts the tile in sorted order in shared
//                memory and stores runs of equal digits to consecutive addresses.
// No CTA ever waits for another one.  An item is a key, or a key of up to 32 bits above a value of
// 32 bits (which then needs no array of its own: one store of 8 bytes per item where two of 4 went
// to different places).
//
// Digits have 8 bits, or up to 10 where that saves a pass (kWidePairs, kWideKeys).  Runs of equal
// digits are then a quarter as long, for keys all over the key space shorter than what DRAM takes
// at a time.  Calls of sort_unique_sum pass by pass (which those above 4.7 million items and others
// that piece_sum.cuh is not for still go), us, ids with many repeats / all different:
//   30 bits         10^6     2^22       2^23       2^24       2^25         4 10^7
//   four passes    90 / 92  194 / 204  341 / 373  647 / 694  1265 / 1328  1487 / 1569
//   three          81 / 87  168 / 182  312 / 377  615 / 715  1185 / 1360  1394 / 1594
//   form before    98 / 93  212 / 203  348 / 355  662 / 671  1277 / 1305  1498 / 1550
//   40 bits, five passes and four: 113 / 113 and 102 / 106 (10^6), 251 / 262 and 260 / 306 (2^22)
// Pairs have wide digits up to 2^25: ids that repeat, which a batch has and which the sums are for,
// gain 5 to 14 %, those all different lose 1 to 4 from 2^23 on.  (Larger sorts would be the same
// trade.  The form before had keys and values in two arrays, four passes, and counted the distinct
// keys before it summed: for ids all different from 2^23 on the faster way, by 3 to 7 %.)
//
// Up to some million items everything stays in L2.  The single-sweep form (one launch per pass,
// tiles finding their offsets by looking back over the words that earlier tiles publish) spent a
// third of its time in the look-back and another third in a second wave of tiles: 54 us per pass
// on 2^22 pairs against 41 us for three launches.  What bounds the scatter is the shared-memory
// pipe (busy for 0.9 of the clocks of an SM at work): the accesses of a digit's random place, for
// mask, counter, position and exchange.
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;                  // keys per thread and tile of the one-CTA sort
constexpr int kTile = kThreads * kItems;
constexpr int kRadixBits = 8;
constexpr int kDigits = 1 << kRadixBits;
constexpr int kWideBits = 10;
constexpr int kMaxChunks = 2 * 148;        // two CTAs per SM
constexpr int kMinChunk = 2048;
constexpr long long kWidePairs = 1 << 25, kWideKeys = 2 << 20;
// Up to so many items pairs that keep to digits of 8 bits travel in one word from the first pass
// on.  More have arrays of keys and values until the last one.  us, ids of 24 bits all over the key
// space / with many repeats / half of them one id:
//               2^20            2^22               2^24
//   together    71 / 74 / 75   162 / 164 / 174   535 / 539 / 579
//   apart       74 / 75 / 77   153 / 152 / 161   522 / 498 / 528
//   form before 73 / 75 / 73   161 / 168 / 174   545 / 519 / 538
constexpr long long kPairsTogether = 3 << 19;
// Up to so many chunks the scatter adds up the counts itself: sorts of that size are bound by the
// number of launches (64-bit keys without payload, 2^14 / 2^16, us: 119 / 110 with three launches
// per pass, 64 / 74 with two; the single-sweep form 97 / 101).  With digits of 8 bits there are no
// more up to 128 Ki items, in chunks of up to 4096: 80 Ki keys of 64 bits 80.8 us in 40 chunks of
// 2048, 67.4 in 32 of 2560; 24 bits 32.8 and 26.6.  Wider digits have four times the counts: 64 Ki
// pairs of 40 bits 75.8 us when 32 chunks were added up, 65.6 with a scan; and pairs whose wide
// digits would save one pass of six or more keep to 8 bits there (64 bits, 64 Ki: 102.6 and 95.3).
constexpr int kSelfScan = 32, kSelfScanWide = 16, kMaxSelfChunk = 4096;

// Head of the scratch memory.
struct SortHead {
  int too_wide;                            // 1: a key has bits beyond key_bits
  int groups;                              // of segments (piece_sum.cuh); 0: rounds
  int shift;                               // of the group in a key, 0: items have whole keys
  unsigned int pieces, several;
  int split, separate;                     // parts begin at b.splits; keys and sums in two arrays
  unsigned int done;                       // CTAs of the merge
  int crowded;                             // 1: a part has too many distinct keys
};

// The chunks of n items.  A tile of the scatter has `rows` rows of 32 items per warp; the tiles of
// a chunk are equally long, so that no SM ends on a nearly empty one.
struct Chunks {
  int count;
  int size;  // items per chunk (the last one: what is left)
  int rows;
};
inline Chunks chunks_of(long long n, int bits, int threads, int max_rows) {
  long long per = (n + kMaxChunks - 1) / kMaxChunks;
  if (per < kMinChunk) per = kMinChunk;
  if (bits == kRadixBits && n > (long long)kSelfScan * per && n <= kSelfScan * kMaxSelfChunk)
    per = (n + kSelfScan - 1) / kSelfScan;
  const long long tile = (long long)threads * max_rows, tiles = (per + tile - 1) / tile;
  Chunks c;
  c.rows = (int)((per + tiles * threads - 1) / (tiles * threads));
  c.size = (int)(tiles * c.rows * threads);
  c.count = (int)((n + c.size - 1) / c.size);
  return c;
}

template <typename K>
__device__ __forceinline__ unsigned int digit_of(K k, int shift) {
  return (unsigned int)((k >> shift) & (kDigits - 1));
}
__device__ __forceinline__ unsigned int lanemask_lt() {
  unsigned int m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Exclusive prefix sum of one value per thread over a CTA of WARPS warps; `part`: WARPS words of
// shared memory, free again after the next __syncthreads.
template <int WARPS = kWarps>
__device__ __forceinline__ unsigned int cta_exclusive(unsigned int v, unsigned int* part,
                                                      unsigned int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) part[warp] = incl;
  __syncthreads();
  unsigned int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    const unsigned int t = part[w];
    if (w < warp) before += t;
    all += t;
  }
  if (total) *total = all;
  return before + incl - v;
}

// The kernels of a sort are chained (chain.cuh): 2^22 pairs of 30-bit keys take 249 us launched
// one after the other and 227 chained, 153 035 of 24 bits 92 and 74.  What the kernel before has
// written is read through L2 (__ldcg): a read-only path may not be used for it.

using Item = unsigned long long;
__device__ __forceinline__ unsigned int item_digit(Item k, int shift, unsigned int mask) {
  return (unsigned int)(k >> shift) & mask;
}

// What a sort reports to the host, one word in mapped memory: whether a key was too wide, whether
// the keys are too close together for buckets, and the number of distinct keys.
constexpr unsigned long long kReported = 1ull << 63, kReportWide = 1ull << 62,
                             kReportCrowded = 1ull << 61;
__device__ __forceinline__ void host_report(unsigned long long* host, unsigned int total,
                                            bool too_wide) {
  *reinterpret_cast<volatile unsigned long long*>(host) =
      kReported | (too_wide ? kReportWide : 0) | total;
  __threadfence_system();
}

// Counters of two digits in a word.
__device__ __forceinline__ unsigned int half_of(unsigned int word, unsigned int d) {
  return (d & 1) ? word >> 16 : word & 0xffffu;
}

// In how many rows of 32 a lane has an item: `left` from its first one to the end of them all.
__device__ __forceinline__ int valid_rows(int left, int rows) {
  const int have = (left + 31) >> 5;
  return have < rows ? have : rows;
}

// Ranks of a warp's items, in rows of 32: of each among those with the same digit, in index order;
// two of 16 bits in a word of `rank`.  `cnt`, of zeros, ends up with the number of each digit's
// items; `lanes`: zeros, and again afterwards.  A lane has items in its first `valid` rows.
//
// The lanes that hold the same digit find each other through a mask in shared memory (32 keys of an
// SM in 9 ns; 15 with ballots, 32 with match.any), and the first of them advances the counter.
// FREE: items of a digit may be in any order, the counter gives out the ranks.  (Lanes of one
// instruction get theirs in the hardware's order, on which nothing but rounding depends: the order
// in which the values of a key are added up.  It has been the same from run to run, with nothing
// that guarantees it; masks, which would, take the scatter of 2^22 pairs from 37 to 42 us.)
// (32 atomics on one address take an SM some 70 clocks, which popular ids among others do not
// need.)
template <bool FREE, int ROWS, typename Digit>
__device__ __forceinline__ void rank_rows(const Digit& digit, int rows, int valid,
                                          unsigned int* lanes, unsigned short* cnt,
                                          unsigned int (&rank)[ROWS / 2]) {
  const unsigned int mine = 1u << (threadIdx.x & 31), below = lanemask_lt();
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    if (j % 2 == 0 && j >= rows) break;
    const bool in = j < valid;
    const unsigned int d = digit(j);
    unsigned int r = 0;
    if constexpr (FREE) {
      if (in)
        r = half_of(atomicAdd(reinterpret_cast<unsigned int*>(cnt) + d / 2, 1u << (d & 1) * 16), d);
    } else {
      if (in) atomicOr(&lanes[d], mine);
      __syncwarp();
      const unsigned int same = lanes[d];
      const unsigned int first = cnt[d], before = __popc(same & below);
      __syncwarp();
      if (in && before == 0) {
        lanes[d] = 0;
        cnt[d] = (unsigned short)(first + __popc(same));
      }
      r = first + before;
      __syncwarp();
    }
    if (j & 1) rank[j / 2] |= r << 16;
    else rank[j / 2] = r;
  }
}

}  // namespace sortk
}  // namespace psdev
#include "kernels/piece_sum.cuh"
namespace psdev {
namespace sortk {

// counts[c * 2^BITS + d] = items of chunk c whose digit is d.  SAMPLE: one CTA more looks at a
// sample of the keys, and wide keys are noted chunk by chunk.
template <typename K, int BITS, bool SAMPLE>
__global__ void __launch_bounds__(kThreads, 2)
    digit_count_kernel(const K* __restrict__ keys, long long n, int shift, unsigned int mask,
                       Chunks ch, int key_bits, unsigned int* counts, SortHead* head,
                       const __grid_constant__ Buckets b, unsigned long long* host) {
  grid_launch_next();
  if constexpr (SAMPLE) {
    if (blockIdx.x == ch.count) {
      grid_wait();
      __shared__ __align__(16) unsigned int slots[kSampleSlots];
      __shared__ unsigned int found[kMaxBuckets];
      sample_buckets<kThreads>(keys, (unsigned int)n, __popc(mask), b, {slots, found}, head, host);
      return;
    }
  }
  constexpr int kDigits = 1 << BITS, kSets = BITS > 8 ? 2 : 4;
  constexpr int kItems = 14;  // (2^22 items: 28 per thread; 8.4 us, 8.9 with 8 loads in flight)
  __shared__ unsigned int s[kSets][kDigits];  // groups of warps share a set of counters
  unsigned int* mine = s[threadIdx.x / (kThreads / kSets)];
  for (int i = threadIdx.x; i < kSets * kDigits; i += kThreads) s[0][i] = 0;
  grid_wait();
  __syncthreads();
  const long long lo = (long long)blockIdx.x * ch.size;
  const long long hi = lo + ch.size < n ? lo + ch.size : n;
  bool wide = false;
  for (long long base = lo + threadIdx.x; base < hi; base += kThreads * kItems) {
    K k[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j)
      k[j] = base + j * kThreads < hi ? __ldcg(keys + base + j * kThreads) : (K)0;
#pragma unroll
    for (int j = 0; j < kItems; ++j)
      if (base + j * kThreads < hi) {
        if constexpr (sizeof(K) == 8)
          if (key_bits < 64) wide |= (k[j] >> (key_bits & 63)) != 0;
        atomicAdd(&mine[item_digit(k[j], shift, mask)], 1u);
      }
  }
  if constexpr (SAMPLE) {
    wide = __syncthreads_or(wide);
    if (threadIdx.x == 0) b.wide[blockIdx.x] = wide;
  } else {
    if (wide) head->too_wide = 1;
    __syncthreads();
  }
  for (int d = threadIdx.x; d < kDigits; d += kThreads) {
    unsigned int c = 0;
#pragma unroll
    for (int w = 0; w < kSets; ++w) c += s[w][d];
    counts[(size_t)blockIdx.x * kDigits + d] = c;
  }
}

// 32 digits per CTA: exclusive prefix over the chunks in place, and the digits' totals.  A warp
// takes a run of chunks, a lane a digit.
__global__ void __launch_bounds__(1024)
    digit_scan_kernel(unsigned int* counts, int digits, int chunks, unsigned int* totals) {
  grid_launch_next();
  grid_wait();
  constexpr int kRun = (kMaxChunks + 31) / 32;
  __shared__ unsigned int s_part[32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = (chunks + 31) / 32, first = warp * run;
  unsigned int* col = counts + blockIdx.x * 32 + lane;
  unsigned int c[kRun], sum = 0;
#pragma unroll
  for (int i = 0; i < kRun; ++i)
    c[i] = i < run && first + i < chunks ? __ldcg(col + (size_t)(first + i) * digits) : 0;
#pragma unroll
  for (int i = 0; i < kRun; ++i) sum += c[i];
  s_part[warp][lane] = sum;
  __syncthreads();
  unsigned int before = 0;
  for (int w = 0; w < warp; ++w) before += s_part[w][lane];
#pragma unroll
  for (int i = 0; i < kRun; ++i)
    if (i < run && first + i < chunks) {
      col[(size_t)(first + i) * digits] = before;
      before += c[i];
    }
  if (warp == 31) totals[blockIdx.x * 32 + lane] = before;
}

// What travels beside the keys of a pass: nothing, the key's index or a value of 32 bits in an
// array of its own, or a value that a first pass puts below its key.  With values in an array, keys
// of up to 32 bits can have 32 too: the first pass narrows them (kNarrow), the last one puts pairs
// together (kShortToPairs).  (First passes of sums without masks, FREE, would save 1 to 2 % from
// 2^23 items on and leave the order of a key's values to the hardware.)
enum {
  kNoPayload = 0, kMakeIndex = 1, kPayload = 2, kToPairs = 3,
  kNarrow = 4, kShort = 5, kShortToPairs = 6
};
template <int PAY>
struct Form {
  static constexpr bool kShortIn = PAY == kShort || PAY == kShortToPairs;
  static constexpr bool kShortKey = kShortIn || PAY == kNarrow;
  static constexpr bool kArray = PAY == kMakeIndex || PAY == kPayload || kShortKey;
  using In = std::conditional_t<kShortIn, unsigned int, Item>;    // as a pass reads them
  using Key = std::conditional_t<kShortKey, unsigned int, Item>;  // and ranks them
};

// Rank of each of a thread's keys (index base + 32 j, below hi) among the keys of its warp that
// have the same digit, in index order; cnt[d] ends up as the number of such keys.
template <typename K>
__device__ __forceinline__ void rank_tile(const K* k, long long base, long long hi, int shift,
                                          unsigned int* cnt, unsigned int* lanes,
                                          unsigned int* rank) {
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    // the lanes that hold the same digit find each other through a mask in shared memory; the
    // first of them advances the warp's counter for all of them
    const bool valid = base + j * 32 < hi;
    const unsigned int d = digit_of(k[j], shift);
    if (valid) atomicOr(&lanes[d], 1u << (threadIdx.x & 31));
    __syncwarp();
    const unsigned int same = valid ? lanes[d] : 1u << (threadIdx.x & 31);
    const unsigned int before = __popc(same & lanemask_lt());
    unsigned int r = 0;
    __syncwarp();
    if (valid && before == 0) {
      lanes[d] = 0;
      r = cnt[d];
      cnt[d] = r + __popc(same);
    }
    rank[j] = __shfl_sync(0xffffffffu, r, __ffs(same) - 1) + before;
    __syncwarp();
  }
}

// Shared memory of a scatter: the tile's items and payloads in sorted order (before that, the lane
// masks), the warps' digit counters and a table of output places.
template <int BITS, int WARPS, int ROWS, int PAY>
struct ScatterCfg {
  static constexpr int kDigits = 1 << BITS, kThreads = WARPS * 32, kTile = kThreads * ROWS;
  static constexpr int kKeys = kTile * (int)sizeof(typename Form<PAY>::Key);
  static constexpr int kExchange = kKeys + (Form<PAY>::kArray ? kTile * 4 : 0);
  static constexpr int kMasks = WARPS * kDigits * 4;
  static constexpr int kShared = kExchange > kMasks ? kExchange : kMasks;
  static constexpr int kSmemBytes = kShared + WARPS * kDigits * 2 + kDigits * 4;
};
// Two CTAs per SM, of 16 warps with 14 rows each (2^22 pairs, 10 bits: 132 us; 8 warps with 28
// rows 133, 16 with 16 rows 137, one CTA of 32 warps with 14 rows 156); with small chunks 8 warps
// with 16 rows, whose counters are fewer (2^17 pairs: 36 and 39 us).
template <int BITS, int WARPS, int ROWS, int PAY>
__global__ void __launch_bounds__(WARPS * 32, 2)
    scatter_kernel(const typename Form<PAY>::In* __restrict__ keys_in, void* __restrict__ out,
                   const unsigned int* __restrict__ pay_in, unsigned int* __restrict__ pay_out,
                   long long n, int shift, unsigned int mask, Chunks ch,
                   const unsigned int* __restrict__ prefix,
                   const unsigned int* __restrict__ totals) {
  grid_launch_next();
  constexpr bool kArray = Form<PAY>::kArray;
  using K = typename Form<PAY>::Key;
  using C = ScatterCfg<BITS, WARPS, ROWS, PAY>;
  constexpr int kDigits = C::kDigits, kThreads = C::kThreads, kPairs = kDigits / 2;
  constexpr int kPer = kPairs > kThreads ? kPairs / kThreads : 1;  // pairs of digits per thread
  static_assert(kPairs % kThreads == 0 || kThreads % kPairs == 0, "every pair has a thread");
  static_assert(ROWS % 2 == 0 && C::kTile < 65536, "ranks and positions have 16 bits");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  K* skeys = reinterpret_cast<K*>(smem_raw);
  unsigned int* spay = reinterpret_cast<unsigned int*>(smem_raw + C::kKeys);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // lanes[d]: lanes of this warp whose present item has digit d; zero in between.  The memory of
  // the exchange, which begins when all warps have their ranks.
  unsigned int* lanes = reinterpret_cast<unsigned int*>(smem_raw) + warp * kDigits;
  // cnt[d]: first the number of items with digit d seen so far by this warp, afterwards the sorted
  // position in the tile of its first one.  count2: the counters of digits 2 i and 2 i + 1 at once.
  unsigned short* cnt =
      reinterpret_cast<unsigned short*>(smem_raw + C::kShared) + warp * kDigits;
  unsigned int* count2 = reinterpret_cast<unsigned int*>(smem_raw + C::kShared);
  // output index of sorted position q: goff[d] + q
  unsigned int* goff = reinterpret_cast<unsigned int*>(smem_raw + C::kShared + WARPS * kDigits * 2);
  __shared__ unsigned int s_part[2][WARPS];
  const bool digits = threadIdx.x * kPer < kPairs;
  grid_wait();
  // output index of the chunk's next item with each of this thread's digits
  unsigned int next[2 * kPer], total[2 * kPer], mine = 0;
#pragma unroll
  for (int i = 0; i < 2 * kPer; ++i) next[i] = total[i] = 0;
  if (digits) {
    const int d0 = threadIdx.x * 2 * kPer;
    if (totals) {
#pragma unroll
      for (int i = 0; i < 2 * kPer; ++i) {
        next[i] = __ldcg(prefix + (size_t)blockIdx.x * kDigits + d0 + i);
        total[i] = __ldcg(totals + d0 + i);
      }
    } else {
      // (eight chunks' counts in flight, the last ones too: one by one 29 chunks cost more than 32)
      for (int c0 = 0; c0 < ch.count; c0 += 8) {
        uint2 v[8][kPer];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int i = 0; i < kPer; ++i)
            v[j][i] = c0 + j < ch.count
                          ? __ldcg(reinterpret_cast<const uint2*>(
                                       prefix + (size_t)(c0 + j) * kDigits + d0) + i)
                          : make_uint2(0, 0);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int i = 0; i < kPer; ++i) {
            if (c0 + j < blockIdx.x) {
              next[2 * i] += v[j][i].x;
              next[2 * i + 1] += v[j][i].y;
            }
            total[2 * i] += v[j][i].x;
            total[2 * i + 1] += v[j][i].y;
          }
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * kPer; ++i) mine += total[i];
  }
  unsigned int smaller = cta_exclusive<WARPS>(mine, s_part[0], nullptr);
#pragma unroll
  for (int i = 0; i < 2 * kPer; ++i) {
    next[i] += smaller;
    smaller += total[i];
  }
  const long long lo = (long long)blockIdx.x * ch.size;
  const long long hi = lo + ch.size < n ? lo + ch.size : n;
  const int rows = ch.rows, tile = kThreads * rows;
  // A tile is loaded before the one before it is stored: its items and payloads take the registers
  // of those that have gone to shared memory.
  K k[ROWS];
  unsigned int pay[kArray ? ROWS : 1];
  auto load = [&](long long base) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (j >= rows) break;
      const long long i = base + j * 32;
      k[j] = i < hi ? (K)__ldcg(keys_in + i) : (K)~0ull;
      if constexpr (PAY == kToPairs) k[j] = k[j] << 32 | (i < hi ? __ldcg(pay_in + i) : 0u);
      if constexpr (PAY == kMakeIndex) pay[j] = (unsigned int)i;
      else if constexpr (kArray) pay[j] = i < hi ? __ldcg(pay_in + i) : 0u;
    }
  };
  load(lo + (long long)warp * (32 * rows) + lane);
  for (long long tile_base = lo; tile_base < hi; tile_base += tile) {
    const long long base = tile_base + (long long)warp * (32 * rows) + lane;
    const int tile_n = (int)(hi - tile_base < tile ? hi - tile_base : tile);
    for (int i = lane; i < kDigits; i += 32) lanes[i] = 0;
    for (int i = lane; i < kPairs; i += 32) reinterpret_cast<unsigned int*>(cnt)[i] = 0;
    __syncwarp();
    unsigned int rank[ROWS / 2];  // two of 16 bits each
    const int valid = valid_rows((int)(hi - base), rows);
    rank_rows<false, ROWS>(
        [&](int j) { return item_digit(k[j], shift, mask); }, rows, valid, lanes, cnt, rank);
    __syncthreads();
    // where the runs of this thread's digits start in the tile, and each warp's part of them
    unsigned int run[kPer], items = 0;
    if (digits) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        run[i] = 0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) run[i] += count2[w * kPairs + threadIdx.x * kPer + i];
        items += (run[i] & 0xffffu) + (run[i] >> 16);
      }
    }
    unsigned int start = cta_exclusive<WARPS>(items, s_part[1], nullptr);
    if (digits) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const unsigned int r0 = run[i] & 0xffffu, r1 = run[i] >> 16;
        const int d = (threadIdx.x * kPer + i) * 2;
        unsigned int at = start | (start + r0) << 16;
        goff[d] = next[2 * i] - start;
        goff[d + 1] = next[2 * i + 1] - (start + r0);
        next[2 * i] += r0;
        next[2 * i + 1] += r1;
        start += r0 + r1;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          unsigned int* p = &count2[w * kPairs + threadIdx.x * kPer + i];
          const unsigned int c = *p;
          *p = at;
          at += c;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (j >= rows) break;
      if (base + j * 32 < hi) {
        const unsigned int q = cnt[item_digit(k[j], shift, mask)] +
                               ((j & 1) ? rank[j / 2] >> 16 : rank[j / 2] & 0xffffu);
        skeys[q] = k[j];
        if constexpr (kArray) spay[q] = pay[j];
      }
    }
    load(base + tile);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (j >= rows) break;
      const int q = threadIdx.x + j * kThreads;
      if (q < tile_n) {
        const K key = skeys[q];
        const unsigned int p = goff[item_digit(key, shift, mask)] + (unsigned int)q;
        if constexpr (PAY == kShortToPairs) {
          static_cast<Item*>(out)[p] = (Item)key << 32 | spay[q];
        } else {
          static_cast<K*>(out)[p] = key;
          if constexpr (kArray) pay_out[p] = spay[q];
        }
      }
    }
    __syncthreads();
  }
}

// All passes of a sort of at most one tile in one launch of one CTA (the three launches per pass of
// the general form take longer than the work: 2^12 keys of 24 bits, with the sums of equal
// keys, 111 us in nine launches).  `unique`: receives the number of distinct keys, or NULL;
// `host`: the report for the host (see host_report), or NULL.  Keys of 32 bits come out as pairs.
template <typename K, int PAY>
constexpr int small_smem() {
  return kTile * ((int)sizeof(K) + (PAY ? 4 : 0)) + 2 * kWarps * kDigits * 4;
}
template <typename K, int PAY>
__global__ void __launch_bounds__(kThreads)
    small_sort_kernel(const Item* keys_in, Item* keys_out, const unsigned int* pay_in,
                      unsigned int* pay_out, int n, int passes, int key_bits, SortHead* head,
                      unsigned int* unique, unsigned long long* host) {
  grid_launch_next();
  grid_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  K* skeys = reinterpret_cast<K*>(smem_raw);
  unsigned int* spay = reinterpret_cast<unsigned int*>(smem_raw + kTile * sizeof(K));
  unsigned int (*cnt)[kDigits] = reinterpret_cast<unsigned int (*)[kDigits]>(
      smem_raw + kTile * sizeof(K) + (PAY ? kTile * 4 : 0));
  unsigned int (*lanes)[kDigits] = cnt + kWarps;
  __shared__ unsigned int s_part[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int base = warp * (32 * kItems) + lane;
  bool wide = false;
  for (int i = threadIdx.x; i < n; i += kThreads) {
    const Item k = keys_in[i];
    if (key_bits < 64) wide |= (k >> (key_bits & 63)) != 0;
    skeys[i] = (K)k;
    if constexpr (PAY != kNoPayload) spay[i] = PAY == kPayload ? pay_in[i] : (unsigned int)i;
  }
  if (wide) head->too_wide = 1;
  const bool any_wide = __syncthreads_or(wide);
  for (int i = threadIdx.x; i < kWarps * kDigits; i += kThreads) lanes[0][i] = 0;
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = pass * kRadixBits;
    for (int i = threadIdx.x; i < kWarps * kDigits; i += kThreads) cnt[0][i] = 0;
    __syncthreads();
    K k[kItems];
    unsigned int pay[kItems], rank[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      k[j] = base + j * 32 < n ? skeys[base + j * 32] : (K)~0ull;
      pay[j] = PAY != kNoPayload && base + j * 32 < n ? spay[base + j * 32] : 0;
    }
    rank_tile(k, base, n, shift, cnt[warp], lanes[warp], rank);
    __syncthreads();
    unsigned int run = 0;
    if (threadIdx.x < kDigits) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) run += cnt[w][threadIdx.x];
    }
    unsigned int at = cta_exclusive(run, s_part, nullptr);
    if (threadIdx.x < kDigits) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const unsigned int c = cnt[w][threadIdx.x];
        cnt[w][threadIdx.x] = at;
        at += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      if (base + j * 32 < n) {
        const unsigned int q = cnt[warp][digit_of(k[j], shift)] + rank[j];
        skeys[q] = k[j];
        if constexpr (PAY != kNoPayload) spay[q] = pay[j];
      }
    }
    __syncthreads();
  }
  unsigned int heads = 0;
  for (int i = threadIdx.x; i < n; i += kThreads) {
    if constexpr (sizeof(K) == 4) {
      keys_out[i] = (Item)skeys[i] << 32 | spay[i];
    } else {
      keys_out[i] = skeys[i];
      if constexpr (PAY != kNoPayload) pay_out[i] = spay[i];
    }
    heads += i == 0 || skeys[i] != skeys[i - 1];
  }
  if (unique) {
    unsigned int total;
    cta_exclusive(heads, s_part, &total);
    if (threadIdx.x == 0) {
      *unique = total;
      if (host) host_report(host, total, any_wide);
    }
  }
}

static size_t round256(size_t b) { return (b + 255) & ~size_t(255); }

// Working memory of a sort: the head and one set of counts and totals (passes follow each other
// on one stream).
struct SortWork {
  SortHead* head;
  unsigned int* counts;
  unsigned int* totals;
  // (no form has more chunks than items / kMinChunk, nor more than kMaxChunks)
  static size_t count_bytes(long long n, int bits) {
    long long chunks = n / kMinChunk + 1;
    if (chunks > kMaxChunks) chunks = kMaxChunks;
    return round256(((size_t)chunks << bits) * 4);
  }
  static size_t bytes(long long n, int bits) {
    return round256(sizeof(SortHead)) + count_bytes(n, bits) + round256((size_t)4 << bits);
  }
  SortWork(char* p, long long n, int bits) {
    head = reinterpret_cast<SortHead*>(p);
    p += round256(sizeof(SortHead));
    counts = reinterpret_cast<unsigned int*>(p);
    p += count_bytes(n, bits);
    totals = reinterpret_cast<unsigned int*>(p);
  }
};

// Dynamic shared memory beyond the default limit, once per kernel and device.
template <auto Kernel>
static int allow_smem(int bytes) {
  static std::atomic<bool> set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (!set[dev & 63].load(std::memory_order_acquire)) {
    const cudaError_t e =
        cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    set[dev & 63].store(true, std::memory_order_release);
  }
  return 0;
}

template <typename K, int PAY>
static int small_sort(const Item* in, Item* out, const unsigned int* pin, unsigned int* pout, int n,
                      int passes, int key_bits, SortHead* head, unsigned int* unique,
                      unsigned long long* host, cudaStream_t s) {
  if (int rc = allow_smem<small_sort_kernel<K, PAY>>(small_smem<K, PAY>())) return rc;
  const int rc = launch_chained(small_sort_kernel<K, PAY>, 1, kThreads, small_smem<K, PAY>(), s, 1,
                                in, out, pin, pout, n, passes, key_bits, head, unique, host);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}

struct Pass {
  const void* in;
  void* out;
  const unsigned int* pin;
  unsigned int* pout;
  long long n;
  int shift, width;    // of the digit in an item
  int count_shift;     // and in the items as they are read
  int check_bits;      // of the keys, 64: not checked
};
template <int BITS, int WARPS, int ROWS, int PAY>
static int sort_pass(const Pass& p, const SortWork& w, cudaStream_t s) {
  using C = ScatterCfg<BITS, WARPS, ROWS, PAY>;
  using In = typename Form<PAY>::In;
  const In* in = static_cast<const In*>(p.in);
  if (int rc = allow_smem<scatter_kernel<BITS, WARPS, ROWS, PAY>>(C::kSmemBytes)) return rc;
  const Chunks ch = chunks_of(p.n, BITS, C::kThreads, ROWS);
  const unsigned int mask = (1u << p.width) - 1;
  int rc = launch_chained(digit_count_kernel<In, BITS, false>, ch.count, kThreads, 0, s, 1, in, p.n,
                          p.count_shift, mask, ch, p.check_bits, w.counts, w.head, Buckets{},
                          nullptr);
  const bool scan = ch.count > (BITS == kRadixBits ? kSelfScan : kSelfScanWide);
  if (!rc && scan)
    rc = launch_chained(digit_scan_kernel, C::kDigits / 32, 1024, 0, s, 1, w.counts, C::kDigits,
                        ch.count, w.totals);
  if (!rc)
    rc = launch_chained(scatter_kernel<BITS, WARPS, ROWS, PAY>, ch.count, C::kThreads,
                        C::kSmemBytes, s, 1, in, p.out, p.pin, p.pout, p.n, p.shift, mask, ch,
                        w.counts, scan ? w.totals : nullptr);
  g_launches.fetch_add(scan ? 3 : 2, std::memory_order_relaxed);
  return rc;
}
// The form of a pass by its digits and the length of its chunks (ScatterCfg).
template <int PAY>
static int any_pass(int bits, const Pass& p, const SortWork& w, cudaStream_t s) {
  if (bits == kRadixBits) return sort_pass<kRadixBits, 16, 8, PAY>(p, w, s);
  if constexpr (PAY == kMakeIndex || Form<PAY>::kShortKey) {
    return PSDEV_ERR_ARG;
  } else {
    if (p.n <= kMaxChunks * 4096ll) return sort_pass<kWideBits, 8, 16, PAY>(p, w, s);
    return sort_pass<kWideBits, 16, PAY == kPayload ? 10 : 14, PAY>(p, w, s);
  }
}

// ---- sums of the values of equal keys --------------------------------------------------------
// On sorted (key, value) pairs, in three kernels, the outputs allocated before the last:
//   unique_local  every CTA adds up the values of equal keys in a round of pairs and stores its
//                 distinct keys and their sums at the round's place in a scratch array.  A key
//                 belongs to the round that it begins in; what a round finds of a key that began
//                 before is its lead;
//   unique_scan   one CTA: prefix of the rounds' counts, and the report to the host;
//   unique_gather moves every round's keys and sums to their places and adds the leads of the
//                 rounds behind it to its last sum.
// Of 2^22 pairs with 0.85 million keys they take 15, 5 and 12 us, cold; the form before, which
// counted the distinct keys, waited for the outputs and then went over the pairs once more, 9, 5
// and 22.
// Nothing is added up with atomics: sums do not depend on the order of the CTAs.
constexpr int kUniqueThreads = 256;
constexpr int kUniquePer = 8;
constexpr int kRound = kUniqueThreads * kUniquePer;
constexpr unsigned kGatherCtas = 6 * 148;
template <bool PAIRS, int THREADS>
constexpr int unique_smem() {  // (a thread's pairs start in different banks)
  return THREADS * (kUniquePer + 1) * (8 + (PAIRS ? 0 : 4));
}
static inline long long rounds_of(long long n) { return (n + kRound - 1) / kRound; }

struct Unique {
  const Item* items;          // sorted: keys, or pairs
  const float* vals;          // values of keys; NULL: pairs
  long long n;
  Item* keys;                 // distinct keys (with their sums: pairs) of every round
  float* sums;
  unsigned int* counts;       // of every round, later their prefix
  float* leads;
  unsigned long long* out_keys;  // one round only: the outputs, or NULL
  float* out_sums;
};

template <bool PAIRS, int THREADS>
__global__ void __launch_bounds__(THREADS, 1536 / THREADS)
    unique_local_kernel(const __grid_constant__ Unique u) {
  constexpr int kPer = kUniquePer, kWarps = THREADS / 32, kRound = THREADS * kPer;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Item* s_item = reinterpret_cast<Item*>(smem_raw);
  float* s_val = reinterpret_cast<float*>(smem_raw + THREADS * (kPer + 1) * 8);
  __shared__ unsigned int s_part[kWarps];
  __shared__ float s_tail[kWarps];
  __shared__ bool s_flag[kWarps];
  grid_launch_next();
  grid_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long base = (long long)blockIdx.x * kRound;
  const int count = (int)(u.n - base < kRound ? u.n - base : kRound);
  const Item* items = u.items + base;
  auto key_of = [](Item i) { return PAIRS ? i >> 32 : i; };
  const bool follows = base > 0;  // (is the first pair's key that of the pair before the round?)
  const Item last = follows ? key_of(__ldcg(items - 1)) : 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int q = threadIdx.x + j * THREADS;
    if (q < count) {
      s_item[q + q / kPer] = __ldcg(items + q);
      if constexpr (!PAIRS) s_val[q + q / kPer] = __ldcg(u.vals + base + q);
    }
  }
  __syncthreads();
  const int q0 = threadIdx.x * kPer, p0 = q0 + threadIdx.x;
  Item key[kPer];
  float val[kPer];
  Item prev = last;
  if (q0 > 0 && q0 < count) prev = key_of(s_item[p0 - 2]);
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const bool valid = q0 + j < count;
    const Item i = valid ? s_item[p0 + j] : 0;
    key[j] = key_of(i);
    val[j] = 0.f;
    if constexpr (PAIRS) val[j] = valid ? __uint_as_float((unsigned int)i) : 0.f;
    else if (valid) val[j] = s_val[p0 + j];
  }
  bool head[kPer];
  unsigned int heads = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const bool valid = q0 + j < count;
    head[j] = valid && ((q0 + j == 0 && !follows) || key[j] != prev);
    heads += head[j];
    if (valid) prev = key[j];
  }
  unsigned int total;
  // (all threads have read their pairs: the memory is free for the round's keys and sums)
  const unsigned int first_slot = cta_exclusive<kWarps>(heads, s_part, &total);
  // Slot i holds the i-th key that begins here, slot 0 (with its own place) the lead.  A thread's
  // sum of what belongs to the slot that is open before its first pair, then its own slots; the
  // last one stays open.
  Item* slot_key = s_item;
  float* slot_sum = PAIRS ? nullptr : s_val;
  auto put_sum = [&](unsigned int slot, float v) {
    if constexpr (PAIRS)
      reinterpret_cast<unsigned int*>(slot_key + slot)[0] = __float_as_uint(v);
    else
      slot_sum[slot] = v;
  };
  unsigned int slot = first_slot;
  float lead = 0.f, sum = 0.f;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (head[j]) {
      if (slot == first_slot) lead = sum;
      else put_sum(slot, sum);
      ++slot;
      sum = 0.f;
      if constexpr (PAIRS)
        reinterpret_cast<unsigned int*>(slot_key + slot)[1] = (unsigned int)key[j];
      else
        slot_key[slot] = key[j];
    }
    sum += val[j];
  }
  // segmented inclusive scan of (has heads, open sum) over the threads
  const bool any = heads > 0;
  bool f = any;
  float v = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float pv = __shfl_up_sync(0xffffffffu, v, o);
    const bool pf = __shfl_up_sync(0xffffffffu, f, o);
    if (lane >= o) {
      if (!f) v += pv;
      f |= pf;
    }
  }
  if (lane == 31) {
    s_tail[warp] = v;
    s_flag[warp] = f;
  }
  float carry = __shfl_up_sync(0xffffffffu, v, 1);
  bool carried = __shfl_up_sync(0xffffffffu, f, 1);
  if (lane == 0) {
    carry = 0.f;
    carried = false;
  }
  __syncthreads();
  if (!carried)
    for (int w = warp - 1; w >= 0; --w) {
      carry += s_tail[w];
      if (s_flag[w]) break;
    }
  if (any) put_sum(first_slot, carry + lead);
  if (threadIdx.x == THREADS - 1) put_sum(total, any ? sum : carry + sum);
  __syncthreads();
  auto sum_at = [&](unsigned int i) {
    if constexpr (PAIRS) return __uint_as_float((unsigned int)slot_key[i]);
    else return slot_sum[i];
  };
  if (threadIdx.x == 0 && u.counts) {
    u.counts[blockIdx.x] = total;
    u.leads[blockIdx.x] = follows ? sum_at(0) : 0.f;
  }
  for (unsigned int i = threadIdx.x; i < total; i += THREADS) {
    if (u.out_keys) {
      u.out_keys[i] = key_of(slot_key[i + 1]);
      u.out_sums[i] = sum_at(i + 1);
    } else {
      u.keys[base + i] = slot_key[i + 1];
      if constexpr (!PAIRS) u.sums[base + i] = slot_sum[i + 1];
    }
  }
}

// A kernel that writes a word of mapped memory which the host polls is cheaper than a copy and a
// wait for the stream (with the call from Python native: 4096 ids 58 us before, 41 now; 2^22 216
// and 204).
__global__ void __launch_bounds__(kThreads)
    unique_scan_kernel(unsigned int* counts, int rounds, const SortHead* head,
                       unsigned long long* host) {
  __shared__ unsigned int s_part[2][kWarps];
  grid_launch_next();
  grid_wait();
  constexpr int kEach = 4;
  unsigned int before = 0;
  int turn = 0;
  for (int r0 = 0; r0 < rounds; r0 += kThreads * kEach, turn ^= 1) {
    const int i0 = r0 + threadIdx.x * kEach;
    unsigned int c[kEach], mine = 0, all;
#pragma unroll
    for (int j = 0; j < kEach; ++j) c[j] = i0 + j < rounds ? __ldcg(counts + i0 + j) : 0;
#pragma unroll
    for (int j = 0; j < kEach; ++j) mine += c[j];
    unsigned int at = before + cta_exclusive(mine, s_part[turn], &all);
#pragma unroll
    for (int j = 0; j < kEach; ++j) {
      if (i0 + j < rounds) counts[i0 + j] = at;
      at += c[j];
    }
    before += all;
  }
  if (threadIdx.x == 0) {
    counts[rounds] = before;
    host_report(host, before, __ldcg(&head->too_wide) != 0);
  }
}

// The keys and sums of segments: CTA i takes the groups i, i + grid, ..., or with more CTAs than
// groups one of several shares of a group.
__device__ __forceinline__ void gather_segments(const Unique& u, const Segments& seg, int groups,
                                                int shift, bool separate) {
  const unsigned int low = shift > 0 && shift < 32 ? (1u << shift) - 1 : ~0u;
  const unsigned int shares = gridDim.x / groups ? gridDim.x / groups : 1;
  for (unsigned int g = blockIdx.x; g < groups * shares; g += gridDim.x) {
    const unsigned int group = g / shares, share = g % shares;
    const Item high = shift ? (Item)group << shift : 0;
    const unsigned int *prefix = seg.counts + group * kGroup, *place = seg.place + group * kGroup;
    unsigned int begin[kGroup + 1], from[kGroup];
#pragma unroll
    for (int p = 0; p <= kGroup; ++p) begin[p] = __ldcg(prefix + p);
#pragma unroll
    for (int p = 0; p < kGroup; ++p) from[p] = __ldcg(place + p);
#pragma unroll 4
    for (unsigned int i = begin[0] + share * kUniqueThreads + threadIdx.x; i < begin[kGroup];
         i += shares * kUniqueThreads) {
      unsigned int first = begin[0], at = from[0];
#pragma unroll
      for (int p = 1; p < kGroup; ++p)
        if (i >= begin[p]) {
          first = begin[p];
          at = from[p];
        }
      const unsigned int q = (at & ~kMerged) + (i - first);
      const Item k = __ldcg((at & kMerged ? u.keys : u.items) + q);
      if (separate) {
        u.out_keys[i] = k;
        u.out_sums[i] = __ldcg((at & kMerged ? u.sums : u.vals) + q);
        continue;
      }
      u.out_keys[i] = high | ((unsigned int)(k >> 32) & low);
      u.out_sums[i] = __uint_as_float((unsigned int)k);
    }
  }
}

// The keys and sums of a round.
template <bool PAIRS>
__device__ __forceinline__ void gather_round(const Unique& u, int round, int rounds) {
  const unsigned int at = __ldcg(u.counts + round);
  const unsigned int count = __ldcg(u.counts + round + 1) - at;
  const long long base = (long long)round * kRound;
  if (count == 0) return;
  // What the rounds behind have found of the last key.  A warp looks at 32 of them, which is enough
  // for most keys, and then at 512 at a time: 32 at a time took 90 us of 2^24 pairs with one key,
  // where one CTA goes through all 8192 rounds.
  float more = 0.f;
  if (threadIdx.x < 32) {
    auto open_behind = [&](int r0, auto groups) {  // whether the key goes on behind these rounds
      constexpr int kGroups = decltype(groups)::value;
      float lead[kGroups], v = 0.f;
      bool ends[kGroups], open = true;
#pragma unroll
      for (int j = 0; j < kGroups; ++j) {
        const int r = r0 + j * 32 + (int)threadIdx.x;
        const bool in = r < rounds;
        lead[j] = in ? __ldcg(u.leads + r) : 0.f;
        ends[j] = !in || __ldcg(u.counts + r + 1) != __ldcg(u.counts + r);
      }
#pragma unroll
      for (int j = 0; j < kGroups; ++j) {
        const unsigned int stop = __ballot_sync(0xffffffffu, ends[j]);
        const int n = stop ? __ffs(stop) : 32;  // (the round of the next key's begin has a lead)
        if (open && (int)threadIdx.x < n) v += lead[j];
        if (stop) open = false;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      more += v;
      return open;
    };
    int r0 = round + 1;
    if (open_behind(r0, std::integral_constant<int, 1>{}))
      for (r0 += 32; open_behind(r0, std::integral_constant<int, 16>{}); r0 += 512) {}
  }
  for (unsigned int i = threadIdx.x; i < count; i += kUniqueThreads) {
    const Item k = __ldcg(u.keys + base + i);
    if constexpr (PAIRS) {
      u.out_keys[at + i] = k >> 32;
      if (i + 1 < count) u.out_sums[at + i] = __uint_as_float((unsigned int)k);
    } else {
      u.out_keys[at + i] = k;
      if (i + 1 < count) u.out_sums[at + i] = __ldcg(u.sums + base + i);
    }
  }
  if (threadIdx.x == 0) {
    const long long i = base + count - 1;
    const float v = PAIRS ? __uint_as_float((unsigned int)__ldcg(u.keys + i)) : __ldcg(u.sums + i);
    u.out_sums[at + count - 1] = v + more;
  }
}

template <bool PAIRS>
__global__ void __launch_bounds__(kUniqueThreads, 6)
    unique_gather_kernel(const __grid_constant__ Unique u, int rounds, const SortHead* head,
                         Segments seg) {
  grid_launch_next();
  grid_wait();
  if (const int groups = __ldcg(&head->groups)) {
    gather_segments(u, seg, groups, __ldcg(&head->shift), __ldcg(&head->separate) != 0);
    return;
  }
  for (int round = blockIdx.x; round < rounds; round += gridDim.x)
    gather_round<PAIRS>(u, round, rounds);
}

// ---- ordered match -------------------------------------------------------------------------
template <typename V>
__device__ __forceinline__ V apply_op(int op, V dst, V src) {
  switch (op) {
    case 0: return src;        // ASSIGN
    case 1: return dst + src;  // PLUS
    case 2: return dst - src;  // MINUS
    case 3: return dst * src;  // TIMES
    case 4: return dst / src;  // DIVIDE
    default: return dst;
  }
}
__device__ __forceinline__ int apply_bitop(int op, int dst, int src) {
  switch (op) {
    case 5: return dst & src;  // AND
    case 6: return dst | src;  // OR
    case 7: return dst ^ src;  // XOR
    default: return apply_op<int>(op, dst, src);
  }
}

// For every src key: binary search among the dst keys; on a hit, dst_val[j*k..] op= src_val[i*k..]
template <typename V, bool INT>
__global__ void ordered_match_kernel(const unsigned long long* src_keys, const V* src_vals,
                                     long long n_src, const unsigned long long* dst_keys,
                                     V* dst_vals, long long n_dst, int k, int op,
                                     unsigned long long* matched) {
  unsigned long long local = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_src;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long key = src_keys[i];
    long long lo = 0, hi = n_dst;
    while (lo < hi) {
      const long long m = (lo + hi) >> 1;
      if (dst_keys[m] < key) lo = m + 1; else hi = m;
    }
    if (lo < n_dst && dst_keys[lo] == key) {
      ++local;
      for (int j = 0; j < k; ++j) {
        V* d = dst_vals + lo * k + j;
        const V s = src_vals[i * k + j];
        if constexpr (INT) *d = (V)apply_bitop(op, (int)*d, (int)s);
        else *d = apply_op<V>(op, *d, s);
      }
    }
  }
  if (local) atomicAdd(matched, local);
}

}  // namespace sortk
}  // namespace psdev

using namespace psdev;
using namespace psdev::sortk;

extern "C" {

// Bytes of scratch psdev_sort_keys needs for n keys (with or without a payload).
size_t psdev_sort_scratch_bytes(int64_t n, int with_payload) {
  size_t b = SortWork::bytes(n > 0 ? n : 1, kRadixBits);
  b += round256((size_t)n * 8);                        // second key buffer
  if (with_payload) b += round256((size_t)n * 4);      // second payload buffer
  return b + 256;
}

// Sorts `n` 64-bit keys ascending by their low `key_bits` bits (64 for full keys; fewer bits
// = fewer passes).  `keys` is sorted in place.  If `perm` is not NULL it receives, for every
// output position, the index the key had in the input (a stable sort permutation).
// `scratch` is device memory of psdev_sort_scratch_bytes(n, perm != NULL) bytes; n < 2^30.
int psdev_sort_keys(uint64_t* keys, uint32_t* perm, int64_t n, int key_bits, void* scratch,
                    size_t scratch_bytes, void* stream) {
  if (n < 0 || key_bits < 1 || key_bits > 64 || !keys) return PSDEV_ERR_ARG;
  if (n == 0) return 0;
  if (n >= (int64_t)1 << 30) return PSDEV_ERR_UNSUPPORTED;
  if (!scratch || scratch_bytes < psdev_sort_scratch_bytes(n, perm != nullptr))
    return PSDEV_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int passes = (key_bits + kRadixBits - 1) / kRadixBits;
  char* p = static_cast<char*>(scratch);
  p = reinterpret_cast<char*>(((uintptr_t)p + 255) & ~uintptr_t(255));
  const SortWork w(p, n, kRadixBits);
  p += SortWork::bytes(n, kRadixBits);
  Item* in = reinterpret_cast<Item*>(keys);
  if (n <= kTile) {
    const int rc = perm ? small_sort<Item, kMakeIndex>(in, in, nullptr, perm, (int)n, passes, 64,
                                                       w.head, nullptr, nullptr, s)
                        : small_sort<Item, kNoPayload>(in, in, nullptr, nullptr, (int)n, passes,
                                                       64, w.head, nullptr, nullptr, s);
    return rc ? rc : (int)cudaGetLastError();
  }
  Item* out = reinterpret_cast<Item*>(p);
  p += round256((size_t)n * 8);
  unsigned int* pin = perm;
  unsigned int* pout = perm ? reinterpret_cast<unsigned int*>(p) : nullptr;
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = pass * kRadixBits;
    const Pass q{in, out, pass ? pin : nullptr, pout, n, shift, kRadixBits, shift, 64};
    // the first pass makes the payload: the index of every key in the input
    const int rc = !perm       ? any_pass<kNoPayload>(kRadixBits, q, w, s)
                   : pass == 0 ? any_pass<kMakeIndex>(kRadixBits, q, w, s)
                               : any_pass<kPayload>(kRadixBits, q, w, s);
    if (rc) return rc;
    std::swap(in, out);
    std::swap(pin, pout);
  }
  if (passes & 1) {
    // an odd number of passes leaves the result in the scratch buffers
    cudaMemcpyAsync(keys, in, (size_t)n * 8, cudaMemcpyDeviceToDevice, s);
    if (perm) cudaMemcpyAsync(perm, pin, (size_t)n * 4, cudaMemcpyDeviceToDevice, s);
  }
  return (int)cudaGetLastError();
}

// Waits for `stream` and reports whether the sorts on it ran (the kernels have no wait of their
// own that could run out).
int psdev_sort_status(const void* scratch, void* stream) {
  if (!scratch) return PSDEV_ERR_ARG;
  return (int)cudaStreamSynchronize((cudaStream_t)stream);
}

}  // extern "C"

// ---- unsorted, repeated (key, value) pairs -> sorted distinct keys and sums ---------------------
namespace {
// How (key, value) pairs are sorted: pairs in one word up to 32 bits, and digits of 10 bits where
// they save a pass.  Where they do not, many keys have an array of their own until the last pass,
// so that counting reads 4 bytes per item (kPairsTogether).
struct UniquePlan {
  bool pairs, apart;
  int bits, passes, width;
  UniquePlan(int64_t n, int key_bits) {
    pairs = key_bits <= 32;
    const int narrow = (key_bits + kRadixBits - 1) / kRadixBits;
    const int wide = (key_bits + kWideBits - 1) / kWideBits;
    // (a pass of 10 bits has three launches where one of 8 bits has two)
    const bool self = n > kSelfScanWide * kMinChunk && n <= kSelfScan * kMaxSelfChunk;
    const bool take = n > kTile && n <= (pairs ? kWidePairs : kWideKeys) && wide < narrow &&
                      !(self && 3 * wide > 2 * narrow + 2);
    bits = take ? kWideBits : kRadixBits;
    passes = take ? wide : narrow;
    width = (key_bits + passes - 1) / passes;
    apart = pairs && !take && passes > 1 && n > kPairsTogether;
  }
};

// Which calls sort piece by piece (piece_sum.cuh), and how: fewer than 16 bits are one or two
// passes of the general way.
struct BucketPlan {
  bool take = false;
  int pieces = 0;                    // of the input, 0: scattered into buckets
  int top = 0;                       // bits of a bucket
  Buckets b{};
  static bool sized(int64_t n) { return n > kTile && n <= kMaxBucketItems; }
  static void digits(int bits, int* passes, int* width) {
    *passes = (bits + kWideBits - 1) / kWideBits;
    *width = (bits + *passes - 1) / *passes;
  }
  BucketPlan(int64_t n, int key_bits) {
    const bool few = n <= kFewItems && key_bits <= 64 - kIndexBits;
    if (!sized(n) || key_bits < 16 || (!few && key_bits > 32 + kWideBits)) return;
    take = true;
    b.sample = n > kFewItems / 2 ? kMaxSample : kMaxSample / 2;
    int spread;                      // bits that the sample's keys are told apart by
    if (few) {
      // pieces and parts of 512 items and more
      pieces = (int)((n + 511) / 512);
      if (pieces > kFewPieces) pieces = kFewPieces;
      for (spread = 3; 512ll << spread < n && 1 << spread < kFewPieces;) ++spread;
      b.parts = 1 << spread;
      b.part_shift = b.shift = key_bits - spread;
      digits(key_bits, &b.passes, &b.width);
      digits(b.shift, &b.merge_passes, &b.merge_width);
      b.chunks = pieces;
    } else {
      // 2048 to 4608 items per bucket, and no more than 32 bits of a key below
      for (top = kRadixBits; top < kWideBits && 4096ll << top < n;) ++top;
      if (top < key_bits - 32) top = key_bits - 32;
      spread = top;
      b.shift = key_bits - top;
      b.count = 1 << top;
      b.parts = kGroup;
      b.part_shift = b.shift - 3;
      b.key_shift = key_bits > 32 ? b.shift : 0;
      digits(b.shift, &b.passes, &b.width);
      b.merge_passes = b.passes;
      b.merge_width = b.width;
    }
    // A range with kPiece distinct keys has x in the sample on average, and one with many more has
    // more than this.  (2^22 ids all different have 2 in each of 1024 buckets, the limit is 16, and
    // the average is not to be above 2.5.)
    const double x = (double)kPiece * b.sample / n;
    b.limit = (unsigned int)(x + 6 * sqrt(x) + 4);
    b.mean = (float)x;
    b.key_mask = ~0ull >> (64 - key_bits);
  }
};

// Working memory of the buckets, beside that of the scatter.
struct BucketWork {
  unsigned int *wide, *distinct, *bounds;
  Item* splits;
  Piece* pieces;
  Several* several;
  static size_t bytes() {
    return kOf.wide + kOf.pieces + kOf.several + kOf.splits + kOf.distinct + kOf.bounds;
  }
  explicit BucketWork(char* p) {
    wide = reinterpret_cast<unsigned int*>(p);
    p += kOf.wide;
    pieces = reinterpret_cast<Piece*>(p);
    p += kOf.pieces;
    several = reinterpret_cast<Several*>(p);
    p += kOf.several;
    splits = reinterpret_cast<Item*>(p);
    p += kOf.splits;
    distinct = reinterpret_cast<unsigned int*>(p);
    p += kOf.distinct;
    bounds = reinterpret_cast<unsigned int*>(p);
  }

 private:
  struct Of {
    size_t wide, pieces, several, splits, distinct, bounds;
  };
  static_assert(kMaxPieces * kGroup <= kFewPieces * kFewParts, "bounds of either kind");
  static_assert(kMaxChunks <= 512 && kMaxPieces <= 3072, "of every piece");
  static constexpr Of kOf{4 * 512, 16 * 3072, 16 * kMaxBuckets, 8 * kFewParts, 4 * 3072,
                          4 * kFewPieces * kFewParts};
};

// Layout of the scratch memory: counts and leads of the rounds of distinct keys, two buffers of
// items and, for keys of more than 32 bits, of values, then the working memory of the sort.  (The
// second half of a call reads all but the last part, and of key_bits it needs `pairs` alone.)
struct UniqueScratch {
  SortHead* head;
  Segments seg;
  unsigned int* counts;
  float* leads;
  Item* keys[2];
  unsigned int* vals[2];
  char* work;
  size_t bytes;
  UniqueScratch(void* scratch, int64_t n, bool pairs) {
    const uintptr_t base = ((uintptr_t)scratch + 255) & ~uintptr_t(255);
    uintptr_t p = base;
    head = reinterpret_cast<SortHead*>(p);
    p += round256(sizeof(SortHead));
    seg = {};
    if (BucketPlan::sized(n)) {
      seg.counts = reinterpret_cast<unsigned int*>(p);
      p += round256((kMaxSegments + 1) * 4);
      seg.place = reinterpret_cast<unsigned int*>(p);
      p += round256(kMaxSegments * 4);
    }
    counts = reinterpret_cast<unsigned int*>(p);
    p += round256((size_t)(rounds_of(n) + 1) * 4);
    leads = reinterpret_cast<float*>(p);
    p += round256((size_t)rounds_of(n) * 4);
    for (int i = 0; i < 2; ++i) {
      keys[i] = reinterpret_cast<Item*>(p);
      p += round256((size_t)n * 8);
      vals[i] = reinterpret_cast<unsigned int*>(p);
      if (!pairs) p += round256((size_t)n * 4);
    }
    work = reinterpret_cast<char*>(p);
    bytes = p - base + 256;  // (without `work`, whose size depends on the digits)
  }
  Unique unique(int64_t n, bool pairs, unsigned long long* out_keys, float* out_sums) const {
    Unique u{};
    u.items = keys[0];
    u.vals = pairs ? nullptr : reinterpret_cast<const float*>(vals[0]);
    u.n = n;
    u.keys = keys[1];
    u.sums = pairs ? nullptr : reinterpret_cast<float*>(vals[1]);
    u.counts = counts;
    u.leads = leads;
    u.out_keys = out_keys;
    u.out_sums = out_sums;
    return u;
  }
};

// A word of mapped host memory for the time of one call.  64 of them in one page, allocated at the
// first use and kept; a call that finds all taken gets memory of its own.
struct ReportSlot {
  // (behind nothing else the sample has been looked at 8 to 31 us after the launch, the more the
  // larger the call before)
  static constexpr int kSampleMicros = 50;
  unsigned long long* word = nullptr;
  int index = -1;
  static std::atomic<unsigned long long>& used() {
    static std::atomic<unsigned long long> bits{0};
    return bits;
  }
  static unsigned long long* page() {
    static unsigned long long* p = [] {
      void* m = nullptr;
      if (cudaHostAlloc(&m, 64 * 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess)
        m = nullptr;
      return static_cast<unsigned long long*>(m);
    }();
    return p;
  }
  ReportSlot() {
    if (unsigned long long* p = page()) {
      unsigned long long have = used().load(std::memory_order_relaxed);
      while (~have) {
        const int i = __builtin_ctzll(~have);
        if (used().compare_exchange_weak(have, have | 1ull << i, std::memory_order_acquire)) {
          index = i;
          word = p + 8 * i;
          break;
        }
      }
    }
    if (!word) {
      void* m = nullptr;
      if (cudaHostAlloc(&m, 16, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess)
        word = static_cast<unsigned long long*>(m);
    }
    if (word) word[0] = word[1] = 0;
  }
  ReportSlot(const ReportSlot&) = delete;
  ~ReportSlot() {
    if (index >= 0) used().fetch_and(~(1ull << index), std::memory_order_release);
    else if (word) cudaFreeHost(word);
  }
  // What the sample has shown, once it has (the second word of the slot).  Behind other work on the
  // stream it is not waited for: the rest is launched then too, and whatever the keys are like, its
  // kernels find that out by themselves.
  bool spread() const {
    const volatile unsigned long long* w = word;
    const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(kSampleMicros);
    do {
      for (int i = 0; i < 16; ++i) {
        if (const unsigned long long got = w[1]) return !(got & kReportCrowded);
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
      }
    } while (std::chrono::steady_clock::now() < until);
    return true;
  }
  // Polls while a sort takes microseconds; a long one is waited for without using the core.
  int wait(cudaStream_t s, unsigned long long* got) const {
    const volatile unsigned long long* w = word;
    cudaError_t e = cudaErrorNotReady;
    for (int round = 0; round < 200 && e == cudaErrorNotReady; ++round) {
      for (int i = 0; i < 256; ++i) {
        if ((*got = *w)) return 0;
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
      }
      e = cudaStreamQuery(s);
    }
    if (e == cudaErrorNotReady) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return (int)e;
    return (*got = *w) ? 0 : (int)cudaErrorUnknown;
  }
};

template <bool PAIRS, int THREADS>
int unique_local(unsigned rounds, const Unique& u, cudaStream_t s) {
  constexpr int smem = unique_smem<PAIRS, THREADS>();
  if (int rc = allow_smem<unique_local_kernel<PAIRS, THREADS>>(smem)) return rc;
  return launch_chained(unique_local_kernel<PAIRS, THREADS>, rounds, THREADS, smem, s, 1, u);
}

// Sums piece by piece: of the buckets, or (RAW) of the input.
template <bool RAW, bool LONG>
int piece_sums(const Item* keys, const unsigned int* vals, int64_t n, const UniqueScratch& u,
                const Buckets& b, const ReportSlot& slot, cudaStream_t s) {
  constexpr int smem = piece_smem<LONG>();
  if (int rc = allow_smem<piece_sum_kernel<RAW, LONG>>(smem)) return rc;
  const bool help = RAW && n > kHelpItems;
  auto* merge = help ? piece_merge_kernel<LONG, true> : piece_merge_kernel<LONG, false>;
  if (int rc = help ? allow_smem<piece_merge_kernel<LONG, true>>(smem)
                    : allow_smem<piece_merge_kernel<LONG, false>>(smem))
    return rc;
  const Items mine{u.keys[0], LONG ? reinterpret_cast<float*>(u.vals[0]) : nullptr};
  const Items merged{u.keys[1], LONG ? reinterpret_cast<float*>(u.vals[1]) : nullptr};
  const unsigned grid = RAW ? b.chunks + 1 : b.count + (unsigned)(n / kSmallPiece);
  int rc = launch_chained(piece_sum_kernel<RAW, LONG>, grid, kPieceThreads, smem, s, 1,
                          RAW ? keys : u.keys[1], vals, (long long)n, mine, b, u.head,
                          slot.word);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (!rc && RAW && !b.splits && !slot.spread()) return 0;
  // (a bucket in several pieces has more than kPiece items)
  const int64_t units = RAW ? b.parts + (help ? kHelpers : 0) : n / kPiece * b.parts;
  if (!rc)
    rc = launch_chained(merge,
                        units < 1 ? 1 : units < kMergeCtas ? (unsigned)units : kMergeCtas,
                        kPieceThreads, smem, s, 1, mine, merged, b, u.head, slot.word);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}
// Scatters into buckets.  The host hears what the sample has shown while the count and the scan are
// running, before it launches the rest.
template <int BITS, bool CUT>
int bucket_sums(const Item* keys, const unsigned int* vals, int64_t n, int key_bits,
                const BucketPlan& plan, const UniqueScratch& u, const SortWork& w, Buckets b,
                const ReportSlot& slot, cudaStream_t s) {
  using C = BucketCfg<BITS, CUT>;
  constexpr auto* kScatter = bucket_scatter_kernel<BITS, CUT>;
  if (int rc = allow_smem<kScatter>(C::kSmemBytes)) return rc;
  const Chunks ch = chunks_of(n, kWideBits, C::kThreads, C::kRows);
  const unsigned int mask = (1u << plan.top) - 1;
  b.chunks = ch.count;
  int rc = launch_chained(digit_count_kernel<Item, BITS, true>, ch.count + 1, kThreads, 0, s, 1,
                          keys, (long long)n, b.shift, mask, ch, key_bits, w.counts, w.head, b,
                          slot.word);
  if (!rc)
    rc = launch_chained(digit_scan_kernel, C::kDigits / 32, 1024, 0, s, 1, w.counts, C::kDigits,
                        ch.count, w.totals);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  if (rc || !slot.spread()) return rc;
  rc = launch_chained(kScatter, ch.count, C::kThreads, C::kSmemBytes, s, 1, keys, vals, u.keys[1],
                      (unsigned int)n, mask, ch, w.counts, w.totals, b, w.head);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc ? rc : piece_sums<false, false>(keys, vals, n, u, b, slot, s);
}
template <int BITS>
int bucket_sums(const Item* keys, const unsigned int* vals, int64_t n, int key_bits,
                const BucketPlan& plan, const UniqueScratch& u, const SortWork& w, const Buckets& b,
                const ReportSlot& slot, cudaStream_t s) {
  return key_bits <= 32
             ? bucket_sums<BITS, false>(keys, vals, n, key_bits, plan, u, w, b, slot, s)
             : bucket_sums<BITS, true>(keys, vals, n, key_bits, plan, u, w, b, slot, s);
}
int unique_by_pieces(const Item* keys, const float* vals, int64_t n, int key_bits,
                     const BucketPlan& plan, const UniqueScratch& u, const SortWork& w,
                     const ReportSlot& slot, cudaStream_t s) {
  const BucketWork own(u.work + SortWork::bytes(n, kWideBits));
  Buckets b = plan.b;
  b.wide = own.wide;
  b.pieces = own.pieces;
  b.several = own.several;
  b.distinct = own.distinct;
  b.bounds = own.bounds;
  b.splits = plan.pieces && n <= kSplitItems ? own.splits : nullptr;
  b.seg = u.seg;
  const unsigned int* v = reinterpret_cast<const unsigned int*>(vals);
  if (plan.pieces)
    return key_bits <= 32 ? piece_sums<true, false>(keys, v, n, u, b, slot, s)
                          : piece_sums<true, true>(keys, v, n, u, b, slot, s);
  if (plan.top == 8) return bucket_sums<8>(keys, v, n, key_bits, plan, u, w, b, slot, s);
  if (plan.top == 9) return bucket_sums<9>(keys, v, n, key_bits, plan, u, w, b, slot, s);
  return bucket_sums<10>(keys, v, n, key_bits, plan, u, w, b, slot, s);
}

int unique_sort(const Item* keys, const float* vals, int64_t n, int key_bits,
                const UniqueScratch& u, const SortWork& w, unsigned long long* host,
                cudaStream_t s) {
  const unsigned int* v = reinterpret_cast<const unsigned int*>(vals);
  const UniquePlan plan(n, key_bits);
  if (n <= kTile)
    return plan.pairs ? small_sort<unsigned int, kPayload>(keys, u.keys[0], v, nullptr, (int)n,
                                                           plan.passes, key_bits, w.head, u.counts,
                                                           host, s)
                      : small_sort<Item, kPayload>(keys, u.keys[0], v, u.vals[0], (int)n,
                                                   plan.passes, key_bits, w.head, u.counts, host,
                                                   s);
  for (int pass = 0; pass < plan.passes; ++pass) {
    // buffers alternate so that the last pass writes buffer 0
    const int to = (plan.passes - 1 - pass) & 1, low = pass * plan.width;
    const int width = key_bits - low < plan.width ? key_bits - low : plan.width;
    const int shift = low + (plan.pairs ? 32 : 0);
    Pass p{pass ? u.keys[to ^ 1] : keys, u.keys[to], pass ? u.vals[to ^ 1] : v, u.vals[to], n,
           shift, width, pass ? shift : low, pass ? 64 : key_bits};
    if (plan.apart) {  // (a buffer of pairs holds the keys, then the values)
      const bool last = pass + 1 == plan.passes;
      p.shift = p.count_shift = low;
      if (pass) p.pin = reinterpret_cast<const unsigned int*>(u.keys[to ^ 1]) + n;
      p.pout = last ? nullptr : reinterpret_cast<unsigned int*>(u.keys[to]) + n;
      const int rc = pass == 0 ? any_pass<kNarrow>(plan.bits, p, w, s)
                     : last    ? any_pass<kShortToPairs>(plan.bits, p, w, s)
                               : any_pass<kShort>(plan.bits, p, w, s);
      if (rc) return rc;
      continue;
    }
    const int rc = !plan.pairs ? any_pass<kPayload>(plan.bits, p, w, s)
                   : pass == 0 ? any_pass<kToPairs>(plan.bits, p, w, s)
                               : any_pass<kNoPayload>(plan.bits, p, w, s);
    if (rc) return rc;
  }
  const unsigned rounds = (unsigned)rounds_of(n);
  const Unique q = u.unique(n, plan.pairs, nullptr, nullptr);
  int rc = plan.pairs ? unique_local<true, kUniqueThreads>(rounds, q, s)
                      : unique_local<false, kUniqueThreads>(rounds, q, s);
  if (!rc)
    rc = launch_chained(unique_scan_kernel, 1, kThreads, 0, s, 1, u.counts, (int)rounds, u.head,
                        host);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  return rc;
}

int unique_write(const UniqueScratch& u, int64_t n, bool pairs, unsigned long long* out_keys,
                 float* out_sums, cudaStream_t s) {
  Unique q = u.unique(n, pairs, out_keys, out_sums);
  int rc;
  if (n <= kTile) {
    q.counts = nullptr;
    rc = pairs ? unique_local<true, kThreads>(1, q, s) : unique_local<false, kThreads>(1, q, s);
  } else {
    auto* gather = pairs ? unique_gather_kernel<true> : unique_gather_kernel<false>;
    const unsigned rounds = (unsigned)rounds_of(n);
    const unsigned grid = rounds < 256 ? 256 : rounds < kGatherCtas ? rounds : kGatherCtas;
    rc = launch_chained(gather, grid, kUniqueThreads, 0, s, 1, q, (int)rounds, u.head, u.seg);
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}
}  // namespace

extern "C" {

size_t psdev_unique_sum_scratch_bytes(int64_t n, int key_bits) {
  if (n < 1 || key_bits < 1 || key_bits > 64) return 0;
  const UniquePlan plan(n, key_bits);
  const bool buckets = BucketPlan(n, key_bits).take;
  return UniqueScratch(nullptr, n, plan.pairs).bytes +
         SortWork::bytes(n, buckets ? kWideBits : plan.bits) + (buckets ? BucketWork::bytes() : 0);
}

// Sorts n (key, value) pairs by key into `scratch` (psdev_unique_sum_scratch_bytes) and counts the
// distinct keys; keys and vals are not changed.  Waits for `stream`: the outputs of
// psdev_unique_sum_write, which follows on the same stream, are sized by the count.
// PSDEV_ERR_ARG when a key is not below 2^key_bits.
int psdev_unique_sum_sort(const uint64_t* keys, const float* vals, int64_t n, int key_bits,
                          void* scratch, size_t scratch_bytes, int64_t* n_unique, void* stream) {
  if (!keys || !vals || !n_unique || n < 1 || key_bits < 1 || key_bits > 64) return PSDEV_ERR_ARG;
  if (n >= (int64_t)1 << 30) return PSDEV_ERR_UNSUPPORTED;
  if (!scratch || scratch_bytes < psdev_unique_sum_scratch_bytes(n, key_bits)) return PSDEV_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const UniquePlan plan(n, key_bits);
  const UniqueScratch u(scratch, n, plan.pairs);
  const unsigned long long* k = reinterpret_cast<const unsigned long long*>(keys);
  ReportSlot slot;
  if (!slot.word) return (int)cudaErrorMemoryAllocation;
  const BucketPlan buckets(n, key_bits);
  int rc = 0;
  unsigned long long got = 0;
  if (buckets.take) {
    SortWork w(u.work, n, kWideBits);
    w.head = u.head;
    rc = unique_by_pieces(k, vals, n, key_bits, buckets, u, w, slot, s);
    if (!rc) rc = slot.wait(s, &got);
  }
  if (!rc && (!buckets.take || (got & kReportCrowded))) {
    SortWork w(u.work, n, plan.bits);
    w.head = u.head;
    // (behind the buckets' kernels, whose report has come: the word is free again)
    cudaMemsetAsync(u.head, 0, sizeof(SortHead), s);
    *slot.word = got = 0;
    rc = unique_sort(k, vals, n, key_bits, u, w, slot.word, s);
    if (!rc) rc = slot.wait(s, &got);
  }
  if (rc) {
    cudaStreamSynchronize(s);  // (a kernel before the one that failed may still report)
    return rc;
  }
  if (got & kReportWide) return PSDEV_ERR_ARG;
  *n_unique = (int64_t)(got & 0xffffffffu);
  return 0;
}

// Second half: the distinct keys, ascending, and the sums of their values.  `n` and `key_bits` are
// those of the first half, `n_unique` what it counted.
int psdev_unique_sum_write(const void* scratch, int64_t n, int key_bits, int64_t n_unique,
                           uint64_t* out_keys, float* out_sums, void* stream) {
  if (!scratch || !out_keys || !out_sums || n < 1 || n_unique < 1 || key_bits < 1 || key_bits > 64)
    return PSDEV_ERR_ARG;
  if (n >= (int64_t)1 << 30) return PSDEV_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  const bool pairs = key_bits <= 32;
  const UniqueScratch u(const_cast<void*>(scratch), n, pairs);
  return unique_write(u, n, pairs, reinterpret_cast<unsigned long long*>(out_keys), out_sums, s);
}

// dst_vals[j] op= src_vals[i] for every key present in both sorted unique lists; values have
// `k` elements per key.  op: 0 assign, 1 plus, 2 minus, 3 times, 4 divide, and for int32
// values also 5 and, 6 or, 7 xor.  dtype: 0 = float32, 1 = int32.  `*matched` (device, 8
// bytes, must be zeroed by the caller) receives the number of matched keys.
int psdev_ordered_match(const uint64_t* src_keys, const void* src_vals, int64_t n_src,
                        const uint64_t* dst_keys, void* dst_vals, int64_t n_dst, int k, int op,
                        int dtype, uint64_t* matched, void* stream) {
  if (k < 1 || op < 0 || op > 7 || (dtype == 0 && op > 4) || !matched) return PSDEV_ERR_ARG;
  if (n_src == 0 || n_dst == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const unsigned long long* sk = reinterpret_cast<const unsigned long long*>(src_keys);
  const unsigned long long* dk = reinterpret_cast<const unsigned long long*>(dst_keys);
  unsigned long long* m = reinterpret_cast<unsigned long long*>(matched);
  if (dtype == 0)
    ordered_match_kernel<float, false><<<592, 256, 0, s>>>(sk, static_cast<const float*>(src_vals),
                                                           n_src, dk, static_cast<float*>(dst_vals),
                                                           n_dst, k, op, m);
  else if (dtype == 1)
    ordered_match_kernel<int, true><<<592, 256, 0, s>>>(sk, static_cast<const int*>(src_vals),
                                                        n_src, dk, static_cast<int*>(dst_vals),
                                                        n_dst, k, op, m);
  else
    return PSDEV_ERR_UNSUPPORTED;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return (int)cudaGetLastError();
}

}  // extern "C"
