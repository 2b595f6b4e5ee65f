// Utility kernels for key lists: radix sort of 64-bit keys, 8 bits per pass (with an
// optional payload of 32-bit indices) and ordered match (merge-join) of two sorted key lists
// with an assignment operator applied to the values of the keys present in both.
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
#include <utility>

#include "ps/device/chain.cuh"
#include "ps/device/psdev.h"

namespace psdev {
extern std::atomic<uint64_t> g_launches;

namespace sortk {
// Least-significant-digit radix sort with 8-bit digits.  The keys are cut into a few hundred
// contiguous chunks, one per CTA that fits on the GPU at a time, and a pass is three launches:
//   digit_count  counts the digits of every chunk;
//   digit_scan   turns the counts of each digit into how many keys of the chunks before have it
//                (left to the scatter when there are few chunks);
//   scatter      takes its chunk tile by tile: ranks each key among the keys of the same digit in
//                input order (the sort is stable), puts the tile in sorted order in shared
//                memory and stores runs of equal digits to consecutive addresses.
// ceil(key_bits / 8) passes: a caller that knows its keys are below 2^30 pays four passes,
// not eight.  No CTA ever waits for another one.
//
// Up to some ten million keys everything stays in L2 and a pass is bound by latencies.  The
// single-sweep form (one launch per pass, tiles finding their offsets by looking back over the
// words that earlier tiles publish) spent a third of its time in the look-back and another third
// in a second wave of tiles: 54 us per pass on 2^22 keys of 30 bits with a payload, against 41 us
// for these three launches (5.5 + 2.2 + 33).  What bounds the scatter now is the shared-memory
// pipe: 40 wavefronts per 32 keys, half of them bank conflicts of random digits.
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;                  // keys per thread and tile
constexpr int kTile = kThreads * kItems;
constexpr int kRadixBits = 8;
constexpr int kDigits = 1 << kRadixBits;
constexpr int kMaxChunks = 2 * 148;        // two CTAs per SM
// Up to so many chunks the scatter adds up the counts itself: sorts of that size are bound by the
// number of launches (64-bit keys without payload, 2^14 / 2^16, us: 119 / 110 with three launches
// per pass, 64 / 74 with two; the single-sweep form 97 / 101).
constexpr int kSelfScan = 32;

// Head of the scratch memory.
struct SortHead {
  int too_wide;                            // 1: a key has bits beyond key_bits
};

// The chunks of n keys: `tiles` tiles each, the last ones possibly fewer.
struct Chunks {
  int count;
  int tiles;
};
__host__ __device__ inline Chunks chunks_of(long long n) {
  const long long ntiles = (n + kTile - 1) / kTile;
  const long long per = (ntiles + kMaxChunks - 1) / kMaxChunks;
  return Chunks{(int)((ntiles + per - 1) / per), (int)per};
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

// Exclusive prefix sum of one value per thread over a CTA of kThreads; `part`: kWarps words of
// shared memory, free again after the next __syncthreads.
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
  for (int w = 0; w < kWarps; ++w) {
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

// counts[d * chunks + c] = keys of chunk c whose digit is d
template <typename K>
__global__ void __launch_bounds__(kThreads, 2)
    digit_count_kernel(const K* __restrict__ keys, long long n, int shift, Chunks ch,
                       int key_bits, unsigned int* counts, SortHead* head) {
  grid_launch_next();
  constexpr int kSets = 4;
  __shared__ unsigned int s[kSets][kDigits];  // four warps share a set of counters
  unsigned int* mine = s[threadIdx.x / (kThreads / kSets)];
  for (int i = threadIdx.x; i < kSets * kDigits; i += kThreads) s[0][i] = 0;
  grid_wait();
  __syncthreads();
  const long long lo = (long long)blockIdx.x * ch.tiles * kTile;
  const long long hi = lo + (long long)ch.tiles * kTile < n ? lo + (long long)ch.tiles * kTile : n;
  bool wide = false;
  for (long long base = lo + threadIdx.x; base < hi; base += kTile) {
    K k[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j)
      k[j] = base + j * kThreads < hi ? __ldcg(keys + base + j * kThreads) : (K)0;
#pragma unroll
    for (int j = 0; j < kItems; ++j)
      if (base + j * kThreads < hi) {
        if (sizeof(K) == 8 && key_bits < 64) wide |= (k[j] >> (key_bits & 63)) != 0;
        atomicAdd(&mine[digit_of(k[j], shift)], 1u);
      }
  }
  if (wide) head->too_wide = 1;
  __syncthreads();
  if (threadIdx.x < kDigits) {
    unsigned int c = 0;
#pragma unroll
    for (int w = 0; w < kSets; ++w) c += s[w][threadIdx.x];
    counts[(size_t)threadIdx.x * ch.count + blockIdx.x] = c;
  }
}

// What a sort reports to the host, one word in mapped memory: whether a key was too wide and the
// number of distinct keys.
constexpr unsigned long long kReported = 1ull << 63, kReportWide = 1ull << 62;
__device__ __forceinline__ void host_report(unsigned long long* host, unsigned int total,
                                            bool too_wide) {
  *reinterpret_cast<volatile unsigned long long*>(host) =
      kReported | (too_wide ? kReportWide : 0) | total;
  __threadfence_system();
}

// One CTA per digit: exclusive prefix over the chunks in place, and the digit's total.
__global__ void __launch_bounds__(kThreads)
    digit_scan_kernel(unsigned int* counts, int chunks, unsigned int* totals) {
  grid_launch_next();
  grid_wait();
  __shared__ unsigned int s_part[kWarps];
  static_assert(kMaxChunks <= kThreads && kDigits <= kThreads, "one thread per chunk, digit");
  unsigned int* row = counts + (size_t)blockIdx.x * chunks;
  const unsigned int c = threadIdx.x < chunks ? row[threadIdx.x] : 0;
  unsigned int total;
  const unsigned int before = cta_exclusive(c, s_part, &total);
  if (threadIdx.x < chunks) row[threadIdx.x] = before;
  if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

// What travels beside the keys of a pass.
enum { kNoPayload = 0, kMakeIndex = 1, kPayload = 2 };

template <typename KO>
constexpr int scatter_smem(int payload) {
  return kTile * ((int)sizeof(KO) + (payload ? 4 : 0)) +
         2 * kWarps * kDigits * 4 + 2 * kDigits * 4;
}

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

// KI, KO: type of the keys as read and as written (a sort of short keys narrows them in its first
// pass).  Shared memory: the tile's keys and payloads in sorted order, per-warp digit counters
// and lane masks, and two 256-entry tables.
template <typename KI, typename KO, int PAY>
__global__ void __launch_bounds__(kThreads, 2)
    scatter_kernel(const KI* __restrict__ keys_in, KO* __restrict__ keys_out,
                   const unsigned int* __restrict__ pay_in, unsigned int* __restrict__ pay_out,
                   long long n, int shift, Chunks ch, const unsigned int* __restrict__ prefix,
                   const unsigned int* __restrict__ totals) {
  grid_launch_next();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KO* skeys = reinterpret_cast<KO*>(smem_raw);
  unsigned int* spay = reinterpret_cast<unsigned int*>(smem_raw + kTile * sizeof(KO));
  // cnt[w][d]: first the number of keys with digit d seen so far by warp w, afterwards the
  // sorted position in the tile of that warp's first key with digit d
  unsigned int (*cnt)[kDigits] = reinterpret_cast<unsigned int (*)[kDigits]>(
      smem_raw + kTile * sizeof(KO) + (PAY ? kTile * 4 : 0));
  // lanes[w][d]: lanes of warp w whose present key has digit d; zero in between
  unsigned int (*lanes)[kDigits] = cnt + kWarps;
  unsigned int* goff = &lanes[kWarps][0];  // output index of sorted position q: goff[d] + q
  __shared__ unsigned int s_part[2][kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool digit = threadIdx.x < kDigits;
  for (int i = threadIdx.x; i < kWarps * kDigits; i += kThreads) lanes[0][i] = 0;
  grid_wait();
  // output index of the chunk's next key with digit threadIdx.x
  unsigned int before = 0, total = 0;
  if (digit) {
    const unsigned int* row = prefix + (size_t)threadIdx.x * ch.count;
    if (totals) {
      before = __ldcg(row + blockIdx.x);
      total = __ldcg(totals + threadIdx.x);
    } else {
      for (int c = 0; c < ch.count; ++c) {
        const unsigned int v = __ldcg(row + c);
        if (c < blockIdx.x) before += v;
        total += v;
      }
    }
  }
  unsigned int next = cta_exclusive(total, s_part[0], nullptr) + before;
  const long long lo = (long long)blockIdx.x * ch.tiles * kTile;
  const long long hi = lo + (long long)ch.tiles * kTile < n ? lo + (long long)ch.tiles * kTile : n;
  // A tile is loaded before the one before it is stored: its keys and payloads take the registers
  // of those that have gone to shared memory.
  KO k[kItems];
  unsigned int pay[kItems];
  auto load = [&](long long base) {
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const long long i = base + j * 32;
      k[j] = i < hi ? (KO)__ldcg(keys_in + i) : (KO)~0ull;
      if constexpr (PAY == kPayload) pay[j] = i < hi ? __ldcg(pay_in + i) : 0u;
      else pay[j] = (unsigned int)i;
    }
  };
  load(lo + (long long)warp * (32 * kItems) + lane);
  for (long long tile_base = lo; tile_base < hi; tile_base += kTile) {
    const long long base = tile_base + (long long)warp * (32 * kItems) + lane;
    const int tile_n = (int)(hi - tile_base < kTile ? hi - tile_base : kTile);
    unsigned int rank[kItems];
    for (int i = threadIdx.x; i < kWarps * kDigits; i += kThreads) cnt[0][i] = 0;
    __syncthreads();
    rank_tile(k, base, hi, shift, cnt[warp], lanes[warp], rank);
    __syncthreads();
    // digit threadIdx.x: where its run starts in the tile, and each warp's part of it
    unsigned int run = 0;
    if (digit) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) run += cnt[w][threadIdx.x];
    }
    const unsigned int start = cta_exclusive(run, s_part[1], nullptr);
    if (digit) {
      unsigned int at = start;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const unsigned int c = cnt[w][threadIdx.x];
        cnt[w][threadIdx.x] = at;
        at += c;
      }
      goff[threadIdx.x] = next - start;
      next += run;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      if (base + j * 32 < hi) {
        const unsigned int q = cnt[warp][digit_of(k[j], shift)] + rank[j];
        skeys[q] = k[j];
        if constexpr (PAY != kNoPayload) spay[q] = pay[j];
      }
    }
    load(base + kTile);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const int q = threadIdx.x + j * kThreads;
      if (q < tile_n) {
        const KO key = skeys[q];
        const unsigned int p = goff[digit_of(key, shift)] + (unsigned int)q;
        keys_out[p] = key;
        if constexpr (PAY != kNoPayload) pay_out[p] = spay[q];
      }
    }
  }
}

// All passes of a sort of at most one tile in one launch of one CTA (the three launches per pass of
// the general form take longer than the work: 2^12 keys of 24 bits, with the sums of equal
// keys, 111 us in nine launches).  `unique`: receives the number of distinct keys, or NULL;
// `host`: the report for the host (see host_report), or NULL.
template <typename KI, typename K, int PAY>
__global__ void __launch_bounds__(kThreads)
    small_sort_kernel(const KI* keys_in, K* keys_out, const unsigned int* pay_in,
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
    const KI k = keys_in[i];
    if (sizeof(KI) == 8 && key_bits < 64) wide |= (k >> (key_bits & 63)) != 0;
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
    keys_out[i] = skeys[i];
    if constexpr (PAY != kNoPayload) pay_out[i] = spay[i];
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
  static size_t bytes(long long n) {
    return round256(sizeof(SortHead)) + round256((size_t)kDigits * chunks_of(n).count * 4) +
           round256(kDigits * 4);
  }
  SortWork(char* p, long long n) {
    head = reinterpret_cast<SortHead*>(p);
    p += round256(sizeof(SortHead));
    counts = reinterpret_cast<unsigned int*>(p);
    p += round256((size_t)kDigits * chunks_of(n).count * 4);
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

template <typename KI, typename K, int PAY>
static int small_sort(const KI* in, K* out, const unsigned int* pin, unsigned int* pout, int n,
                      int passes, int key_bits, SortHead* head, unsigned int* unique,
                      unsigned long long* host, cudaStream_t s) {
  if (int rc = allow_smem<small_sort_kernel<KI, K, PAY>>(scatter_smem<K>(PAY))) return rc;
  const int rc = launch_chained(small_sort_kernel<KI, K, PAY>, 1, kThreads, scatter_smem<K>(PAY), s,
                                1, in, out, pin, pout, n, passes, key_bits, head, unique, host);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}

template <typename KI, typename KO, int PAY>
static int sort_pass(const KI* in, KO* out, const unsigned int* pin, unsigned int* pout,
                     long long n, int pass, int key_bits, const SortWork& w, cudaStream_t s) {
  if (int rc = allow_smem<scatter_kernel<KI, KO, PAY>>(scatter_smem<KO>(PAY))) return rc;
  const Chunks ch = chunks_of(n);
  const int shift = pass * kRadixBits;
  int rc = launch_chained(digit_count_kernel<KI>, ch.count, kThreads, 0, s, 1, in, n, shift, ch,
                          pass ? 64 : key_bits, w.counts, w.head);
  const bool scan = ch.count > kSelfScan;
  if (!rc && scan)
    rc = launch_chained(digit_scan_kernel, kDigits, kThreads, 0, s, 1, w.counts, ch.count,
                        w.totals);
  if (!rc)
    rc = launch_chained(scatter_kernel<KI, KO, PAY>, ch.count, kThreads, scatter_smem<KO>(PAY), s,
                        1, in, out, pin, pout, n, shift, ch, w.counts,
                        scan ? w.totals : nullptr);
  g_launches.fetch_add(scan ? 3 : 2, std::memory_order_relaxed);
  return rc;
}

// ---- sums of the values of equal keys --------------------------------------------------------
// On sorted (key, value) pairs, in two kernels with the allocation of the outputs between them:
// unique_count counts the first occurrences in each chunk, unique_sum writes every distinct key
// and the sum of its values.  Their chunks are smaller than those of the sort (a CTA has little
// to do per pair): up to 2048, as many counts as unique_sum adds up at its start.
constexpr int kMaxUniqueChunks = 2048;
__host__ __device__ inline Chunks unique_chunks_of(long long n) {
  const long long ntiles = (n + kTile - 1) / kTile;
  const long long per = (ntiles + kMaxUniqueChunks - 1) / kMaxUniqueChunks;
  return Chunks{(int)((ntiles + per - 1) / per), (int)per};
}

template <typename K>
__global__ void __launch_bounds__(kThreads, 2)
    unique_count_kernel(const K* __restrict__ keys, long long n, Chunks ch, unsigned int* counts) {
  grid_launch_next();
  grid_wait();
  __shared__ unsigned int s_part[kWarps];
  const int lane = threadIdx.x & 31;
  const long long lo = (long long)blockIdx.x * ch.tiles * kTile;
  const long long hi = lo + (long long)ch.tiles * kTile < n ? lo + (long long)ch.tiles * kTile : n;
  unsigned int heads = 0;
  for (long long base = lo + threadIdx.x; base - lane < hi; base += kTile) {
    K k[kItems], before[kItems];  // before: of lane 0, the last key of the warp's neighbour
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const long long i = base + j * kThreads;
      k[j] = i < hi ? __ldcg(keys + i) : (K)0;
      before[j] = lane == 0 && i > 0 && i < hi ? __ldcg(keys + i - 1) : (K)0;
    }
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const long long i = base + j * kThreads;
      const K up = __shfl_up_sync(0xffffffffu, k[j], 1);
      heads += i < hi && (i == 0 || k[j] != (lane ? up : before[j]));
    }
  }
  unsigned int total;
  cta_exclusive(heads, s_part, &total);
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// Adds up the chunks' counts for the host.  A kernel that writes a word of mapped memory which the
// host polls is cheaper than a copy and a wait for the stream (with the call from Python native:
// 4096 ids 58 us before, 41 now; 2^22 216 and 204).
__global__ void __launch_bounds__(kThreads)
    unique_total_kernel(const unsigned int* counts, int chunks, const SortHead* head,
                        unsigned long long* host) {
  __shared__ unsigned int s_part[kWarps];
  grid_launch_next();
  grid_wait();
  unsigned int c = 0, total;
  for (int i = threadIdx.x; i < chunks; i += kThreads) c += __ldcg(counts + i);
  cta_exclusive(c, s_part, &total);
  if (threadIdx.x == 0) host_report(host, total, __ldcg(&head->too_wide) != 0);
}

// Each thread walks kPer consecutive pairs of a round and adds up what belongs to one key; a
// segmented scan over the threads carries open sums on, so that a key that fills whole chunks
// costs no atomics inside one.  Keys that begin and end inside a round are stored; what is open at
// either end of a round is added to its (cleared) output, two global atomics per round.
constexpr int kUniquePer = 8;
template <typename K>
__global__ void __launch_bounds__(kThreads, 2)
    unique_sum_kernel(const K* __restrict__ keys, const float* __restrict__ vals, long long n,
                      Chunks ch, const unsigned int* __restrict__ counts,
                      unsigned long long* out_keys, float* out_sums) {
  grid_launch_next();
  grid_wait();
  constexpr int kPer = kUniquePer;
  constexpr int kRound = kThreads * kPer;
  constexpr int kPadded = kRound + kRound / kPer;  // (a thread's pairs start in different banks)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  K* skey = reinterpret_cast<K*>(smem_raw);
  K* ukey = skey + kPadded;                        // distinct keys of the round, from 1
  float* sval = reinterpret_cast<float*>(ukey + kRound + 1);
  float* usum = sval + kPadded;                    // 0: the key that was open before the round
  __shared__ unsigned int s_part[kWarps];
  __shared__ float s_tail[kWarps];
  __shared__ bool s_flag[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // index of the chunk's first new key: what the chunks before found
  unsigned int next;
  {
    unsigned int c = 0;
    for (int i = threadIdx.x; i < blockIdx.x; i += kThreads) c += __ldcg(counts + i);
    cta_exclusive(c, s_part, &next);
  }
  const long long lo = (long long)blockIdx.x * ch.tiles * kTile;
  const long long hi = lo + (long long)ch.tiles * kTile < n ? lo + (long long)ch.tiles * kTile : n;
  for (long long base = lo; base < hi; base += kRound) {
    const int count = (int)(hi - base < kRound ? hi - base : kRound);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int q = threadIdx.x + j * kThreads;
      if (q < count) {
        skey[q + q / kPer] = __ldcg(keys + base + q);
        sval[q + q / kPer] = __ldcg(vals + base + q);
      }
    }
    __syncthreads();
    const int q0 = threadIdx.x * kPer, p0 = q0 + threadIdx.x;
    K prev{};
    if (q0 < count) {
      if (q0 > 0) prev = skey[p0 - 2];
      else if (base > 0) prev = __ldcg(keys + base - 1);
    }
    bool head[kPer];
    unsigned int heads = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const bool valid = q0 + j < count;
      const K key = valid ? skey[p0 + j] : prev;
      head[j] = valid && (base + q0 + j == 0 || key != prev);
      heads += head[j];
      prev = key;
    }
    unsigned int total;
    unsigned int slot = cta_exclusive(heads, s_part, &total);  // slot of the key open before q0
    // sum of what belongs to that key, then the thread's own keys; the last one stays open
    const unsigned int first_slot = slot;
    float lead = 0.f, sum = 0.f;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (head[j]) {
        if (slot == first_slot) lead = sum;
        else usum[slot] = sum;
        ++slot;
        sum = 0.f;
        ukey[slot] = skey[p0 + j];
      }
      if (q0 + j < count) sum += sval[p0 + j];
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
    if (any) usum[first_slot] = carry + lead;
    if (threadIdx.x == kThreads - 1) usum[total] = any ? sum : carry + sum;
    __syncthreads();
    for (unsigned int u = threadIdx.x; u <= total; u += kThreads) {
      if (u > 0) out_keys[next + u - 1] = (unsigned long long)ukey[u];
      if (u > 0 && u < total) out_sums[next + u - 1] = usum[u];
      else if (next + u > 0) atomicAdd(&out_sums[next + u - 1], usum[u]);
    }
    next += total;
  }
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
  size_t b = SortWork::bytes(n > 0 ? n : 1);
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
  const SortWork w(p, n);
  p += SortWork::bytes(n);
  using K = unsigned long long;
  K* in = reinterpret_cast<K*>(keys);
  if (n <= kTile) {
    const int rc = perm ? small_sort<K, K, kMakeIndex>(in, in, nullptr, perm, (int)n, passes, 64,
                                                       w.head, nullptr, nullptr, s)
                        : small_sort<K, K, kNoPayload>(in, in, nullptr, nullptr, (int)n, passes,
                                                       64, w.head, nullptr, nullptr, s);
    return rc ? rc : (int)cudaGetLastError();
  }
  K* out = reinterpret_cast<K*>(p);
  p += round256((size_t)n * 8);
  unsigned int* pin = perm;
  unsigned int* pout = perm ? reinterpret_cast<unsigned int*>(p) : nullptr;
  for (int pass = 0; pass < passes; ++pass) {
    // the first pass makes the payload: the index of every key in the input
    const int rc =
        !perm ? sort_pass<K, K, kNoPayload>(in, out, nullptr, nullptr, n, pass, 64, w, s)
        : pass == 0 ? sort_pass<K, K, kMakeIndex>(in, out, nullptr, pout, n, pass, 64, w, s)
                    : sort_pass<K, K, kPayload>(in, out, pin, pout, n, pass, 64, w, s);
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
// Layout of the scratch memory: working memory of the sort, counts of the chunks' distinct keys,
// then two buffers of keys (4 bytes each up to 32 bits) and of values.
struct UniqueScratch {
  char* work;
  SortHead* head;
  unsigned int* counts;
  char* keys[2];
  unsigned int* vals[2];
  size_t bytes;
  UniqueScratch(void* scratch, int64_t n, int key_bits) {
    const size_t ksz = key_bits <= 32 ? 4 : 8;
    const uintptr_t base = ((uintptr_t)scratch + 255) & ~uintptr_t(255);
    uintptr_t p = base;
    work = reinterpret_cast<char*>(p);
    p += SortWork::bytes(n);
    head = reinterpret_cast<SortHead*>(p);
    counts = reinterpret_cast<unsigned int*>(p + sizeof(SortHead));
    p += round256(sizeof(SortHead) + kMaxUniqueChunks * 4);
    for (int i = 0; i < 2; ++i) {
      keys[i] = reinterpret_cast<char*>(p);
      p += round256((size_t)n * ksz);
      vals[i] = reinterpret_cast<unsigned int*>(p);
      p += round256((size_t)n * 4);
    }
    bytes = p - base + 256;
  }
};

// A word of mapped host memory for the time of one call.  64 of them in one page, allocated at the
// first use and kept; a call that finds all taken gets memory of its own.
struct ReportSlot {
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
      if (cudaHostAlloc(&m, 8, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess)
        word = static_cast<unsigned long long*>(m);
    }
    if (word) *word = 0;
  }
  ReportSlot(const ReportSlot&) = delete;
  ~ReportSlot() {
    if (index >= 0) used().fetch_and(~(1ull << index), std::memory_order_release);
    else if (word) cudaFreeHost(word);
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

template <typename K>
int unique_sort(const unsigned long long* keys, const float* vals, int64_t n, int key_bits,
                const UniqueScratch& u, const SortWork& w, unsigned long long* host,
                cudaStream_t s) {
  const unsigned int* v = reinterpret_cast<const unsigned int*>(vals);
  const int passes = (key_bits + kRadixBits - 1) / kRadixBits;
  if (n <= kTile)
    return small_sort<unsigned long long, K, kPayload>(keys, reinterpret_cast<K*>(u.keys[0]), v,
                                                       u.vals[0], (int)n, passes, key_bits,
                                                       w.head, u.counts, host, s);
  for (int pass = 0; pass < passes; ++pass) {
    // buffers alternate so that the last pass writes buffer 0
    const int to = (passes - 1 - pass) & 1;
    K* out = reinterpret_cast<K*>(u.keys[to]);
    const int rc =
        pass == 0 ? sort_pass<unsigned long long, K, kPayload>(keys, out, v, u.vals[to], n, 0,
                                                               key_bits, w, s)
                  : sort_pass<K, K, kPayload>(reinterpret_cast<const K*>(u.keys[to ^ 1]), out,
                                              u.vals[to ^ 1], u.vals[to], n, pass, key_bits, w, s);
    if (rc) return rc;
  }
  const Chunks ch = unique_chunks_of(n);
  int rc = launch_chained(unique_count_kernel<K>, ch.count, kThreads, 0, s, 1,
                          reinterpret_cast<const K*>(u.keys[0]), n, ch, u.counts);
  if (!rc)
    rc = launch_chained(unique_total_kernel, 1, kThreads, 0, s, 1, u.counts, ch.count, u.head,
                        host);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  return rc;
}

template <typename K>
int unique_write(const UniqueScratch& u, int64_t n, unsigned long long* out_keys, float* out_sums,
                 cudaStream_t s) {
  // the pairs of a round (padded) and its outputs
  constexpr int smem = (kThreads * (kUniquePer + 1) + kThreads * kUniquePer + 1) *
                       (int)(sizeof(K) + 4);
  if (int rc = allow_smem<unique_sum_kernel<K>>(smem)) return rc;
  const Chunks ch = unique_chunks_of(n);
  const int rc = launch_chained(unique_sum_kernel<K>, ch.count, kThreads, smem, s, 1,
                                reinterpret_cast<const K*>(u.keys[0]),
                                reinterpret_cast<const float*>(u.vals[0]), n, ch, u.counts,
                                out_keys, out_sums);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}
}  // namespace

extern "C" {

size_t psdev_unique_sum_scratch_bytes(int64_t n, int key_bits) {
  if (n < 1 || key_bits < 1 || key_bits > 64) return 0;
  return UniqueScratch(nullptr, n, key_bits).bytes;
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
  const UniqueScratch u(scratch, n, key_bits);
  SortWork w(u.work, n);
  w.head = u.head;
  cudaMemsetAsync(u.head, 0, sizeof(SortHead), s);
  const unsigned long long* k = reinterpret_cast<const unsigned long long*>(keys);
  ReportSlot slot;
  if (!slot.word) return (int)cudaErrorMemoryAllocation;
  auto* sort = key_bits <= 32 ? unique_sort<unsigned int> : unique_sort<unsigned long long>;
  int rc = sort(k, vals, n, key_bits, u, w, slot.word, s);
  if (rc) {
    cudaStreamSynchronize(s);  // (a kernel before the one that failed may still report)
    return rc;
  }
  unsigned long long got = 0;
  rc = slot.wait(s, &got);
  if (rc) return rc;
  if (got & kReportWide) return PSDEV_ERR_ARG;
  *n_unique = (int64_t)(got & 0xffffffffu);
  return 0;
}

// Second half: the distinct keys, ascending, and the sums of their values.
int psdev_unique_sum_write(const void* scratch, int64_t n, int key_bits, int64_t n_unique,
                           uint64_t* out_keys, float* out_sums, void* stream) {
  if (!scratch || !out_keys || !out_sums || n < 1 || n_unique < 1) return PSDEV_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const UniqueScratch u(const_cast<void*>(scratch), n, key_bits);
  cudaMemsetAsync(out_sums, 0, (size_t)n_unique * 4, s);
  unsigned long long* ok = reinterpret_cast<unsigned long long*>(out_keys);
  return key_bits <= 32 ? unique_write<unsigned int>(u, n, ok, out_sums, s)
                        : unique_write<unsigned long long>(u, n, ok, out_sums, s);
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
