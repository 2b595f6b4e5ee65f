// Sums of equal keys for ids that are spread over their key space: sorted in shared memory, piece
// by piece, with at most one scatter of all items before.
//
// A pass over all items costs a count, a scan and a scatter whose every item goes to a random
// place; 30 bits take three of them (sort_match.cu).  Here many items are scattered once, by their
// highest up to 10 bits, into buckets that a CTA can sort, and few items not at all:
//   digit_count, digit_scan, scatter   as there (more than kFewItems);
//   piece_sum     a CTA per bucket, or per piece of a bucket with more than kPiece items, or per
//                 piece of the input: sorts the items by their remaining bits, adds up the values
//                 of equal keys and stores the distinct ones at the piece's place;
//   piece_merge   does the same once more with the distinct keys of the pieces of a bucket (or of
//                 the input), by parts of its key range.  The last CTA to end makes the prefix of
//                 the counts and reports to the host;
//   unique_gather moves keys and sums to their places in the outputs.
// Every sum has a fixed tree: results do not depend on the order of the CTAs.  In buckets, which of
// a key's values comes where in it depends on the order in which the lanes of an instruction that
// count on one address get their turn (rank_rows), which has always been the same and is not
// guaranteed.
//
// Popular ids make large buckets, in pieces of which little is left to merge.  Keys that crowd
// together would not fit: a CTA of the first kernel looks at a sample of them.  Parts of the input
// then begin at keys of the sample instead of multiples of a power of two; buckets are given up for
// the general way, of which the host hears before that kernel has ended.  So they are where the
// merge finds a part with too many distinct keys.
//
// Whole calls, us, before (pass by pass) and now; ids with many repeats, ids all different:
//                24 bits                   30 bits                   40 bits
//   2^14       47 ->  36,  40 ->  32      43 ->  31,  44 ->  38      53 ->  32,  54 ->  35
//   2^16       45 ->  32,  46 ->  32      50 ->  32,  51 ->  34      63 ->  32,  64 ->  36
//   2^18       55 ->  37,  59 ->  38      59 ->  40,  64 ->  41      80 ->  47,  86 ->  49
//   2^19       61 ->  43,  63 ->  50      65 ->  46,  71 ->  55      84 ->  56,  91 ->  63
//   700000     64 ->  60,  65 ->  58      68 ->  52,  73 ->  63      89 ->  64,  96 ->  73
//   2^20       71 ->  68,  70 ->  60      80 ->  77,  86 ->  66     102 ->  90, 107 ->  73
//   2^21       97 ->  89,  96 ->  82     103 -> 103, 111 ->  87     147 -> 112, 161 ->  98
//   2^22      153 -> 132, 152 -> 130     169 -> 134, 181 -> 139     250 -> 159, 262 -> 160
// Half of all items one id: 0.50 to 0.75 of the time before up to 786 432 items, 0.61 to 0.97
// beyond.  Keys that crowd together in seven narrow ranges: 0.75 to 1.16 up to 2^19, where a sample
// makes the parts, 1.05 to 1.22 up to 655 360; then the general way comes after the pieces, which
// were for nothing, 1.27 to 1.33, and beyond 786 432 items after a count, 1.06 to 1.15.
// What bounds it: up to 2^18 items the chain of some ten trips to L2 and three sorts of 2400 clocks
// per pass; at 2^22 piece_sum (48 us; 0.52 of the issue slots, two thirds of the shared-memory
// pipe, 24 warps per SM), bucket_scatter (26 to 32), and the latency of piece_merge (25).
//
// An item is a key of up to 32 bits above its value, or (LONG) one of up to 51 above the index that
// its value has in the CTA.
#pragma once

namespace psdev {
namespace sortk {

constexpr int kPieceWarps = 8, kPieceRows = 20;
constexpr int kPieceThreads = kPieceWarps * 32;
constexpr int kPiece = kPieceThreads * kPieceRows;   // items that a CTA sorts
constexpr int kPieceCounters = 1 << kWideBits;       // of a digit inside a piece
constexpr int kIndexBits = 13;                       // of an item of a piece
static_assert(kPiece <= 1 << kIndexBits, "every item has an index");
constexpr int kGroup = 8;                            // segments are counted in groups
constexpr int kMaxBuckets = 1 << kWideBits;
constexpr int kMaxSegments = kMaxBuckets * kGroup;
constexpr long long kMaxBucketItems = 9ll << 19;     // (in 1024 buckets 4608 on average)
// Up to so many items are not scattered: pieces of the input and parts of the key range, at most,
// so that all units of a merge run at a time (444 pieces and 512 parts: 2^18 items 52 us, with 256
// of both 40).  786 432 ids of 30 bits, many repeats / all different: 54 / 66 us, in buckets 75
// / 58; 2^20 (where no CTAs helped yet) 66 / 78 and 75 / 65.
constexpr long long kFewItems = 3 << 18;
// Up to so many of them the parts of crowded keys are those of a sample; beyond, one of 256 parts
// by a sample of 5120 would often have more keys than a CTA sorts, and the host goes the general
// way as soon as it hears of the crowd.  Seven narrow ranges, 24 / 30 / 40 bits, before sums went
// piece by piece, the general way and by the sample: 560 000 items 62 / 69 / 91, 79 / 88 / 114, 79
// / 81 / 97; 655 360 64 / 71 / 94, 80 / 91 / 119, 81 / 87 / 102; 720 896 64 / 73 / 96, 82 / 94 /
// 123, 107 / 108 / 132.  (The host has nothing to wait for then: others gain a microsecond.)
constexpr long long kSplitItems = 5 << 17;
constexpr int kFewPieces = 256, kFewParts = 256;
// With more items than this CTAs that are left over help to merge the parts of the input.  700 000
// ids of 24 bits with 25 popular ones in one part 73 -> 60 us, others with repeats from 530 000 on
// 0.91 to 1.01, all different 0.94 to 1.00, half of them one id 0.89 to 1.00.  Fewer items seldom
// make a part of more than a round, and looking for it costs up to a microsecond (2^16 ids 31.0 and
// 32.1, 2^19 45.8 and 46.6).
constexpr long long kHelpItems = 1 << 19;
// A bucket with more items than a CTA sorts is cut in smaller pieces, which do not keep the others
// waiting, or in whole ones where those would be too many to merge.
constexpr int kSmallPiece = kPiece / 2, kManyItems = 1 << 20;
constexpr int kMaxPieces = kMaxBuckets + (int)(kMaxBucketItems / kSmallPiece);
constexpr int kMaxOfBucket = (int)(kMaxBucketItems / kPiece) + 1;
constexpr int kMergeCtas = 2 * 148;
constexpr int kMaxSample = 2048, kSampleSlots = 4 * kMaxSample;

// A piece: items [start, start + count) of the scattered array, all of one bucket, or of the input.
struct Piece {
  unsigned int start, count, bucket, pieces;         // (how many the bucket has)
};
// A bucket in several pieces.
struct Several {
  unsigned int bucket, first, pieces, start;
};
// Where distinct keys and their sums are: counts[s] (later prefix[s]) of them at place[s], in the
// order of the keys.
struct Segments {
  unsigned int* counts;
  unsigned int* place;
};

struct Buckets {
  int shift;             // of the bucket in a key; no buckets: of the parts
  int count;             // buckets, 0: the input is cut in pieces
  int key_shift;         // 0: items have whole keys, else the bucket's bits are not among them
  int parts, part_shift; // of a bucket (or the input) in several pieces
  int passes, width;     // digits of a piece's sort
  int merge_passes, merge_width;
  Item key_mask;         // of a key's bits: wider ones, which are refused, are cut
  int sample;            // keys
  unsigned int limit;    // distinct ones among them in one bucket or part, at most
  float mean;            // others in the bucket of such a key on average, at most
  int chunks;               // of the scatter, or pieces of the input
  unsigned int* wide;       // whether a chunk of the scatter has a key of too many bits
  Piece* pieces;
  Several* several;
  unsigned int* distinct;   // of every piece
  unsigned int* bounds;     // of every piece of several: where each part of the key range begins
  Item* splits;             // parts of crowded keys: their first keys; NULL: left to the host
  Segments seg;
};

// Shared memory for a sample.
struct SampleShared {
  unsigned int* slots;      // kSampleSlots, 16-byte aligned
  unsigned int* found;      // kMaxBuckets
};

// CTA of THREADS threads: whether a sample of the keys, left in `k`, is spread over 2^bits ranges
// of the key space.
template <int THREADS, int ROWS>
__device__ __forceinline__ bool sample_spread(const Item* keys, unsigned int n, int bits,
                                              const Buckets& b, const SampleShared& sh,
                                              Item (&k)[ROWS]) {
  __shared__ unsigned int most, distinct, squares;
  constexpr int kEach = kMaxSample / THREADS;
  static_assert(kEach <= ROWS, "rows of the sample");
  const unsigned int step = n / b.sample;  // (b.sample <= n)
  const unsigned int mask = (1u << bits) - 1;
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const unsigned int i = threadIdx.x + j * THREADS;
    k[j] = i < b.sample ? __ldcg(keys + (size_t)i * step) : 0;
  }
  for (int i = threadIdx.x; i < kSampleSlots / 4; i += THREADS)
    reinterpret_cast<uint4*>(sh.slots)[i] = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < kMaxBuckets; i += THREADS) sh.found[i] = 0;
  if (threadIdx.x == 0) most = distinct = squares = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    if (threadIdx.x + j * THREADS >= b.sample) break;
    unsigned int h = (unsigned int)((k[j] * 0x9e3779b97f4a7c15ull) >> 32);
    h += h == 0;
    // (at most a quarter of the slots are taken: a free one comes)
    for (unsigned int at = h % kSampleSlots;; at = (at + 1) % kSampleSlots) {
      unsigned int there = *(volatile unsigned int*)&sh.slots[at];
      if (there == 0) there = atomicCAS(&sh.slots[at], 0u, h);
      if (there == h) break;
      if (there == 0) {
        atomicAdd(&sh.found[(unsigned int)(k[j] >> b.shift) & mask], 1u);
        break;
      }
    }
  }
  __syncthreads();
  unsigned int top = 0, all = 0, square = 0;
  for (int i = threadIdx.x; i <= mask; i += THREADS) {
    const unsigned int f = sh.found[i];
    top = f > top ? f : top;
    all += f;
    square += f * f;
  }
  top = __reduce_max_sync(0xffffffffu, top);
  all = __reduce_add_sync(0xffffffffu, all);
  square = __reduce_add_sync(0xffffffffu, square);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&most, top);
    atomicAdd(&distinct, all);
    atomicAdd(&squares, square);
  }
  __syncthreads();
  return most <= b.limit && (float)(squares - distinct) <= b.mean * distinct;
}

// What the sample has shown, for a host that decides by it: the second word of the report says so
// early, the first one is the call's.
__device__ __forceinline__ void sample_report(bool spread, unsigned long long* host) {
  volatile unsigned long long* out = host;
  if (!spread) out[0] = kReported | kReportCrowded;
  out[1] = kReported | (spread ? 0 : kReportCrowded);
}

// One CTA more of the count of the buckets: head of the scratch memory, and what the host is told.
template <int THREADS>
__device__ __forceinline__ void sample_buckets(const Item* keys, unsigned int n, int bits,
                                               const Buckets& b, const SampleShared& sh,
                                               SortHead* head, unsigned long long* host) {
  Item k[kMaxSample / THREADS];
  const bool spread = sample_spread<THREADS>(keys, n, bits, b, sh, k);
  if (threadIdx.x) return;
  sample_report(spread, host);
  SortHead h{};
  h.shift = b.key_shift;
  h.groups = spread ? b.count * b.parts / kGroup : 0;
  *head = h;
}

// CTA of WARPS warps, of which a thread has N digits' totals and the start of the first: the pieces
// of the buckets, and which buckets have several.
template <int WARPS, int N>
__device__ __forceinline__ void list_pieces(const Buckets& b, SortHead* head, bool digits,
                                            unsigned int start, const unsigned int (&total)[N],
                                            unsigned int* part) {
  const int d0 = threadIdx.x * N;
  auto pieces_of = [&](int i) {
    if (!digits || d0 + i >= b.count) return 0u;
    const unsigned int size = total[i] <= kManyItems ? kSmallPiece : kPiece;
    return total[i] <= (unsigned int)kPiece ? 1u : (total[i] + size - 1) / size;
  };
  unsigned int mine = 0, all;
#pragma unroll
  for (int i = 0; i < N; ++i) mine += pieces_of(i) + ((pieces_of(i) > 1) << 16);
  const unsigned int before = cta_exclusive<WARPS>(mine, part, &all);
  unsigned int at = before & 0xffffu, severals = before >> 16;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const unsigned int bucket = d0 + i, pieces = pieces_of(i);
    if (pieces > 1) b.several[severals++] = {bucket, at, pieces, start};
    const unsigned int size = pieces > 1 ? (total[i] + pieces - 1) / pieces : total[i];
    for (unsigned int p = 0; p < pieces; ++p) {
      const unsigned int from = p * size, left = total[i] - from;
      b.pieces[at++] = {start + from, left < size ? left : size, bucket, pieces};
    }
    start += total[i];
  }
  if (threadIdx.x == 0) {
    head->pieces = all & 0xffffu;
    head->several = all >> 16;
  }
}

// Zeros, by the lanes of a warp; `words`: a power of two, of 16-byte aligned memory from 4 on.
__device__ __forceinline__ void clear_words(unsigned int* at, int words) {
  const int lane = threadIdx.x & 31;
  if (words >= 128)
#pragma unroll 4
    for (int i = lane; i < words / 4; i += 32)
      reinterpret_cast<uint4*>(at)[i] = make_uint4(0, 0, 0, 0);
  else
    for (int i = lane; i < words; i += 32) at[i] = 0;
}

// ---- the scatter into buckets ---------------------------------------------------------------
template <int BITS, bool CUT>
struct BucketCfg {
  static constexpr int kWarps = 16, kRows = 14;  // two CTAs per SM, tiles of 7168 items
  static constexpr int kDigits = 1 << BITS, kThreads = kWarps * 32, kTile = kThreads * kRows;
  static constexpr int kItemBytes = kTile * 8, kDigitBytes = CUT ? kTile * 2 : 0;
  static constexpr int kCountBytes = kWarps * kDigits * 2;
  static constexpr int kSmemBytes = kItemBytes + kDigitBytes + kCountBytes + kDigits * 4;
};

// As scatter_kernel (sort_match.cu), but an item's place among those of its bucket is free, so that
// there are no masks, and keys and values meet only when they go to shared memory: ranking begins
// when the keys have come, of which it reads the lower half.  (2^22 pairs into 1024 buckets: 26 us,
// 37 as a form of scatter_kernel without masks, 42 with them.  Four CTAs per SM of 8 warps: 5 %
// more. It waits for loads and stores: 0.34 of the issue slots, 0.4 of the shared-memory pipe.)
// CUT: keys of more than 32 bits, whose digit is kept beside the lower 32.  `out`: pairs of (lower
// half of the) key and value.
template <int BITS, bool CUT>
__global__ void __launch_bounds__(BucketCfg<BITS, CUT>::kThreads, 2)
    bucket_scatter_kernel(const Item* __restrict__ keys, const unsigned int* __restrict__ vals,
                          Item* __restrict__ out, unsigned int n, unsigned int mask, Chunks ch,
                          const unsigned int* __restrict__ prefix,
                          const unsigned int* __restrict__ totals,
                          const __grid_constant__ Buckets b, SortHead* head) {
  using C = BucketCfg<BITS, CUT>;
  constexpr int WARPS = C::kWarps, ROWS = C::kRows;
  constexpr int kDigits = C::kDigits, kT = C::kThreads, kPairs = kDigits / 2;
  constexpr int kPer = kPairs > kT ? kPairs / kT : 1;  // pairs of digits per thread
  static_assert(kPairs % kT == 0 || kT % kPairs == 0, "every pair has a thread");
  static_assert(ROWS % 2 == 0 && C::kTile < 65536, "ranks and positions have 16 bits");
  grid_launch_next();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned int s_part[2][WARPS];
  Item* items = reinterpret_cast<Item*>(smem_raw);
  unsigned short* digits_of = reinterpret_cast<unsigned short*>(smem_raw + C::kItemBytes);
  unsigned char* counters = smem_raw + C::kItemBytes + C::kDigitBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // cnt[d]: first the number of items with digit d seen so far by this warp, afterwards the sorted
  // position in the tile of its first one.  count2: the counters of digits 2 i and 2 i + 1 at once.
  unsigned short* cnt = reinterpret_cast<unsigned short*>(counters) + warp * kDigits;
  unsigned int* count2 = reinterpret_cast<unsigned int*>(counters);
  // output index of sorted position q: goff[d] + q
  unsigned int* goff = reinterpret_cast<unsigned int*>(counters + C::kCountBytes);
  grid_wait();
  if (__ldcg(&head->groups) == 0) return;
  const unsigned int lo = blockIdx.x * (unsigned int)ch.size;
  const unsigned int hi = lo + ch.size < n ? lo + ch.size : n;
  const int rows = ch.rows, tile = kT * rows;
  unsigned int key[ROWS], val[ROWS], dig[CUT ? ROWS / 2 : 1];
  auto load = [&](unsigned int at) {
    const int valid = valid_rows((int)hi - (int)at, rows);
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      const unsigned int i = at + j * 32;
      if constexpr (CUT) {
        const Item k = j < valid ? __ldcg(keys + i) : 0;
        key[j] = (unsigned int)k;
        const unsigned int d = item_digit(k, b.shift, mask);
        if (j & 1) dig[j / 2] |= d << 16;
        else dig[j / 2] = d;
      } else {
        key[j] = j < valid ? __ldcg(reinterpret_cast<const unsigned int*>(keys + i)) : 0;
        key[j] &= (unsigned int)b.key_mask;
      }
    }
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      val[j] = j < valid ? __ldcg(vals + at + j * 32) : 0u;
    }
  };
  auto digit = [&](int j) {
    if constexpr (CUT) return half_of(dig[j / 2], j);
    else return key[j] >> b.shift & mask;
  };
  load(lo + warp * (32 * rows) + lane);
  const bool mine = (int)threadIdx.x * kPer < kPairs;
  const int d0 = threadIdx.x * 2 * kPer;
  // output index of the chunk's next item with each of this thread's digits
  unsigned int next[2 * kPer], total[2 * kPer], sum = 0;
#pragma unroll
  for (int i = 0; i < 2 * kPer; ++i) {
    next[i] = mine ? __ldcg(prefix + (size_t)blockIdx.x * kDigits + d0 + i) : 0;
    total[i] = mine ? __ldcg(totals + d0 + i) : 0;
  }
#pragma unroll
  for (int i = 0; i < 2 * kPer; ++i) sum += total[i];
  unsigned int smaller = cta_exclusive<WARPS>(sum, s_part[0], nullptr);
  if (blockIdx.x == 0) list_pieces<WARPS, 2 * kPer>(b, head, mine, smaller, total, s_part[1]);
#pragma unroll
  for (int i = 0; i < 2 * kPer; ++i) {
    next[i] += smaller;
    smaller += total[i];
  }
  for (unsigned int tile_base = lo; tile_base < hi; tile_base += tile) {
    const unsigned int base = tile_base + warp * (32 * rows) + lane;
    const int tile_n = (int)(hi - tile_base < (unsigned int)tile ? hi - tile_base : tile);
    const int valid = valid_rows((int)hi - (int)base, rows);
    clear_words(reinterpret_cast<unsigned int*>(cnt), kPairs);
    __syncwarp();
    unsigned int rank[ROWS / 2];  // two of 16 bits each
    rank_rows<true, ROWS>(digit, rows, valid, nullptr, cnt, rank);
    __syncthreads();
    // where the runs of this thread's digits start in the tile, and each warp's part of them
    unsigned int run[kPer], have = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      run[i] = 0;
      if (mine) {
#pragma unroll 4
        for (int w = 0; w < WARPS; ++w) run[i] += count2[w * kPairs + threadIdx.x * kPer + i];
      }
      have += (run[i] & 0xffffu) + (run[i] >> 16);
    }
    unsigned int start = cta_exclusive<WARPS>(have, s_part[1], nullptr);
    if (mine) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const unsigned int r0 = run[i] & 0xffffu, r1 = run[i] >> 16;
        unsigned int at = start | (start + r0) << 16;
        goff[d0 + 2 * i] = next[2 * i] - start;
        goff[d0 + 2 * i + 1] = next[2 * i + 1] - (start + r0);
        next[2 * i] += r0;
        next[2 * i + 1] += r1;
        start += r0 + r1;
#pragma unroll 1
        for (int w0 = 0; w0 < WARPS; w0 += 4) {
          unsigned int* of = count2 + w0 * kPairs + threadIdx.x * kPer + i;
          unsigned int c[4];
#pragma unroll
          for (int w = 0; w < 4; ++w) c[w] = of[w * kPairs];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            of[w * kPairs] = at;
            at += c[w];
          }
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      if (j < valid) {
        const unsigned int d = digit(j), q = cnt[d] + half_of(rank[j / 2], j);
        items[q] = (Item)key[j] << 32 | val[j];
        if constexpr (CUT) digits_of[q] = (unsigned short)d;
      }
    }
    load(base + tile);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      const int q = threadIdx.x + j * kT;
      if (q < tile_n) {
        const Item i = items[q];
        const unsigned int d =
            CUT ? (unsigned int)digits_of[q] : (unsigned int)(i >> 32) >> b.shift & mask;
        out[goff[d] + (unsigned int)q] = i;
      }
    }
    __syncthreads();
  }
}

// ---- the sums of a piece --------------------------------------------------------------------
constexpr int kPieceItems = kPiece * 8 > kPieceWarps * kPieceCounters * 4
                                ? kPiece * 8 : kPieceWarps * kPieceCounters * 4;
constexpr int kPieceCount = kPieceWarps * kPieceCounters * 2;
template <bool LONG>
constexpr int piece_smem() {
  return kPieceItems + kPieceCount + (LONG ? kPiece * 4 : 0);
}
static_assert(kSampleSlots * 4 + kMaxBuckets * 4 <= kPieceItems + kPieceCount, "a sample fits");
struct PieceShared {
  Item* items;            // kPiece; before that the warps' lane masks
  unsigned short* cnt;    // kPieceWarps counters of every digit
  float* vals;            // LONG: kPiece
  unsigned int* part;     // 2 x kPieceWarps words
  __device__ PieceShared(unsigned char* smem, unsigned int* part)
      : items(reinterpret_cast<Item*>(smem)),
        cnt(reinterpret_cast<unsigned short*>(smem + kPieceItems)),
        vals(reinterpret_cast<float*>(smem + kPieceItems + kPieceCount)), part(part) {}
};

// Sorts up to 512 items, two per thread: every warp its own in registers (bitonic), then runs are
// merged two by two, each item finding its place in the other run by bisection.  `mem`: 1024 items,
// which begins with the sorted ones.  A pass of the radix sort takes some 2400 clocks however few
// the items are, this sort about as long in all (2^16 items in two rows, 30 bits: 33.5 -> 31 us;
// four rows are faster by radix, 2^17 items 33.5 and 36 us).  The loops are not unrolled: a kernel
// of a few CTAs runs through its code once, and waits for the code.
// Pairs are sorted with their numbers in place of the values: in the order of the values' bits all
// positive ones of a key would be added up before the negative ones, at three times the error.
template <bool LONG>
__device__ __forceinline__ void sort_few(Item k0, Item k1, int valid, Item* mem) {
  constexpr int kRun = 64, kAll = kRun * kPieceWarps;
  const int lane = threadIdx.x & 31;
  Item *from = mem + kAll, *to = mem;
  int at0 = 2 * threadIdx.x, at1 = at0 + 1;
  unsigned int* const low = reinterpret_cast<unsigned int*>(from + (at0 & -kRun));
  unsigned int low0 = 0, low1 = 0;
  if constexpr (!LONG) {
    low[2 * lane] = (unsigned int)k0;
    low[2 * lane + 1] = (unsigned int)k1;
    k0 = (k0 >> 32 << 32) | at0;
    k1 = (k1 >> 32 << 32) | at1;
    __syncwarp();
  }
  if (valid < 1) k0 = ~0ull;  // (behind all others)
  if (valid < 2) k1 = ~0ull;
#pragma unroll 1
  for (int size = 2; size <= kRun; size *= 2) {
    const bool up = ((2 * lane) & size) == 0;  // elements 2 lane and 2 lane + 1
#pragma unroll 1
    for (int away = size / 4; away > 0; away /= 2) {
      const Item o0 = __shfl_xor_sync(0xffffffffu, k0, away);
      const Item o1 = __shfl_xor_sync(0xffffffffu, k1, away);
      const bool least = ((lane & away) == 0) == up;
      if ((o0 < k0) == least) k0 = o0;
      if ((o1 < k1) == least) k1 = o1;
    }
    if ((k1 < k0) == up) {
      const Item t = k0;
      k0 = k1;
      k1 = t;
    }
  }
  if constexpr (!LONG) {
    low0 = low[k0 % kRun];
    low1 = low[k1 % kRun];
    __syncwarp();
  }
  from[at0] = k0;
  from[at1] = k1;
#pragma unroll 1
  for (int run = kRun; run < kAll; run *= 2) {
    __syncthreads();
    const int mine = at0 / run;  // (both of a thread's items are in one run)
    const bool second = mine & 1;  // equal items of the first run go before those of the second
    const Item* other = from + (mine ^ 1) * run;
    int less0 = 0, less1 = 0;
#pragma unroll 1
    for (int step = run / 2; step > 0; step /= 2) {
      const Item o0 = other[less0 + step - 1], o1 = other[less1 + step - 1];
      if (o0 < k0 || (second && o0 == k0)) less0 += step;
      if (o1 < k1 || (second && o1 == k1)) less1 += step;
    }
    const Item o0 = other[less0], o1 = other[less1];
    at0 += less0 + (o0 < k0 || (second && o0 == k0)) - (second ? run : 0);
    at1 += less1 + (o1 < k1 || (second && o1 == k1)) - (second ? run : 0);
    to[at0] = k0;
    to[at1] = k1;
    Item* const t = from;
    from = to;
    to = t;
  }
  if constexpr (!LONG) {  // (places that only this thread writes, and nobody reads before)
    from[at0] = (k0 >> 32 << 32) | low0;
    from[at1] = (k1 >> 32 << 32) | low1;
  }
  __syncthreads();
}

// Turns the warps' counts of every digit, two digits in a word, into where the warps' parts of the
// digits start.
__device__ __forceinline__ void place_counts(unsigned int* count2, int pairs, unsigned int* part) {
  // Where the warps' parts of this thread's digits start in the piece: of two pairs of digits
  // side by side, or of one.  (Two words at a time: one by one, two apart, they took twice the
  // clocks.)
  constexpr int kWarps = kPieceWarps, kT = kPieceThreads;
  static_assert(kPieceCounters / 2 == 2 * kT, "two pairs per thread at most");
  const bool two = pairs > kT, mine = two || (int)threadIdx.x < pairs;
  unsigned int* const at0 = count2 + (two ? 2 * threadIdx.x : threadIdx.x);
  auto counts_of = [&](int w) {
    if (two) return *reinterpret_cast<const uint2*>(at0 + w * pairs);
    return make_uint2(mine ? at0[w * pairs] : 0u, 0u);
  };
  uint2 run = make_uint2(0, 0);
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const uint2 c = counts_of(w);
    run.x += c.x;
    run.y += c.y;
  }
  const unsigned int items0 = (run.x & 0xffffu) + (run.x >> 16);
  const unsigned int items1 = (run.y & 0xffffu) + (run.y >> 16);
  const unsigned int start = cta_exclusive<kWarps>(items0 + items1, part, nullptr);
  if (mine) {
    uint2 at;
    at.x = start | (start + (run.x & 0xffffu)) << 16;
    at.y = (start + items0) | (start + items0 + (run.y & 0xffffu)) << 16;
#pragma unroll
    for (int w0 = 0; w0 < kWarps; w0 += 4) {
      uint2 c[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) c[w] = counts_of(w0 + w);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        if (two) *reinterpret_cast<uint2*>(at0 + (w0 + w) * pairs) = at;
        else at0[(w0 + w) * pairs] = at.x;
        at.x += c[w].x;
        at.y += c[w].y;
      }
    }
  }
}

// Sorts the items of a CTA, which it has in registers in rows of 32 per warp, by `passes` digits of
// `width` bits from the lowest of the key on; leaves them in order in sh.items.  FREE: with equal
// keys in any order, which a first pass then ranks without masks.  (2^22 ids of 30 bits all
// different in buckets 138 us, 145 with masks; the fewer items of a piece of the input or of a
// merge gain nothing by it: 2^18 ids with repeats 41.3 and 39.7 us, 2^19 all different 54.3 and
// 54.8.)
template <bool LONG, bool FREE = false>
__device__ __forceinline__ void sort_piece(Item (&k)[kPieceRows], int count, int passes, int width,
                                           const PieceShared& sh) {
  constexpr int kRows = kPieceRows, kT = kPieceThreads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = (count + kT - 1) / kT;
  const int base = warp * (32 * rows) + lane;
  const int valid = valid_rows(count - base, rows);
  if (rows <= 2) {
    sort_few<LONG>(k[0], k[1], valid, sh.items);
    return;
  }
  const int digits = 1 << width, pairs = digits / 2;
  const unsigned int mask = digits - 1;
  unsigned int* lanes = reinterpret_cast<unsigned int*>(sh.items) + warp * digits;
  unsigned short* cnt = sh.cnt + warp * digits;
  unsigned int* mine2 = reinterpret_cast<unsigned int*>(cnt);
  unsigned int* count2 = reinterpret_cast<unsigned int*>(sh.cnt);
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = pass * width;
    if (pass || !FREE) clear_words(lanes, digits);
    clear_words(mine2, pairs);
    __syncwarp();
    unsigned int rank[kRows / 2];
    auto digit = [&](int j) {
      return LONG ? item_digit(k[j], shift + kIndexBits, mask)
                  : (unsigned int)(k[j] >> 32) >> shift & mask;
    };
    if (FREE && pass == 0) rank_rows<true, kRows>(digit, rows, valid, lanes, cnt, rank);
    else rank_rows<false, kRows>(digit, rows, valid, lanes, cnt, rank);
    __syncthreads();
    place_counts(count2, pairs, sh.part + (pass & 1) * kPieceWarps);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      if (j < valid)
        sh.items[cnt[digit(j)] + half_of(rank[j / 2], j)] = k[j];
    }
    __syncthreads();
    if (pass + 1 < passes) {
#pragma unroll
      for (int j = 0; j < kRows; ++j) {
        if (j % 2 == 0 && j >= rows) break;
        if (j < valid) k[j] = sh.items[base + j * 32];
      }
      __syncthreads();
    }
  }
}

// Pieces of a large bucket: most of their items are those of one popular id, or of a few.  Such a
// key is looked for among the first ones of the warps; the values of its items are added up as they
// are, and one item with the sum joins the others, which alone are left to sort.  Once more while
// that takes away a quarter.  Returns how many items there are now, in `k` as before.
__device__ __forceinline__ int add_up_popular(Item (&k)[kPieceRows], int count,
                                              const PieceShared& sh) {
  __shared__ unsigned int s_key[kPieceWarps], s_kept[kPieceWarps];
  __shared__ float s_sum[kPieceWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int round = 0; round < 4; ++round) {
    const int rows = (count + kPieceThreads - 1) / kPieceThreads;
    if (rows <= 2) break;
    const int valid = valid_rows(count - warp * (32 * rows) - lane, rows);
    // (a warp without items shows some key that may not be there, and is outvoted)
    if (lane == 0) s_key[warp] = (unsigned int)(k[0] >> 32);
    __syncthreads();
    const unsigned int seen = s_key[lane % kPieceWarps];
    const unsigned int times = __popc(__match_any_sync(0xffffffffu, seen));
    const unsigned int most = __reduce_max_sync(0xffffffffu, times << 8 | (31u - lane));
    const unsigned int key = __shfl_sync(0xffffffffu, seen, 31 - (most & 0xff));
    unsigned int kept = 0;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < kPieceRows; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      const bool is = j < valid && (unsigned int)(k[j] >> 32) == key;
      if (is) sum += __uint_as_float((unsigned int)k[j]);
      kept += __popc(__ballot_sync(0xffffffffu, j < valid && !is));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) {
      s_kept[warp] = kept;
      s_sum[warp] = sum;
    }
    __syncthreads();
    unsigned int at = 0, all = 0;
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < kPieceWarps; ++w) {
      if (w < warp) at += s_kept[w];
      all += s_kept[w];
      total += s_sum[w];
    }
    if (4 * all > 3 * (unsigned int)count) break;  // (the same for all threads)
#pragma unroll
    for (int j = 0; j < kPieceRows; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      const bool keep = j < valid && (unsigned int)(k[j] >> 32) != key;
      const unsigned int m = __ballot_sync(0xffffffffu, keep);
      if (keep) sh.items[at + __popc(m & lanemask_lt())] = k[j];
      at += __popc(m);
    }
    if (threadIdx.x == 0) sh.items[all] = (Item)key << 32 | __float_as_uint(total);
    __syncthreads();
    count = (int)all + 1;
    const int left = (count + kPieceThreads - 1) / kPieceThreads;
    const int base = warp * (32 * left) + lane, have = valid_rows(count - base, left);
#pragma unroll
    for (int j = 0; j < kPieceRows; ++j) {
      if (j % 2 == 0 && j >= left) break;
      if (j < have) k[j] = sh.items[base + j * 32];
    }
    __syncthreads();
  }
  return count;
}

// What the threads before have of the key that is open where this thread begins; `any`: whether a
// key begins in this thread's items, `sum`: of its open one (of all of them, where none begins).
__device__ __forceinline__ float carry_into(bool any, float sum) {
  __shared__ float s_tail[kPieceWarps];
  __shared__ bool s_flag[kPieceWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // segmented inclusive scan of (has heads, open sum) over the threads
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
  return carry;
}

// The sums of the values of equal keys in `count` sorted items.  The distinct keys end up at the
// front of sh.items, above their sums or (LONG) alone, with the sums in sh.vals.  Returns how many.
template <bool LONG>
__device__ __forceinline__ unsigned int sum_piece(int count, const PieceShared& sh) {
  constexpr int kWarps = kPieceWarps, kMost = kPieceRows + 1;
  using Key = std::conditional_t<LONG, Item, unsigned int>;
  auto key_of = [](Item i) { return (Key)(i >> (LONG ? kIndexBits : 32)); };
  auto put_sum = [&](unsigned int slot, float v) {
    if constexpr (LONG) sh.vals[slot] = v;
    else reinterpret_cast<unsigned int*>(sh.items + slot)[0] = __float_as_uint(v);
  };
  auto put_key = [&](unsigned int slot, Key k) {
    if constexpr (LONG) sh.items[slot] = k;
    else reinterpret_cast<unsigned int*>(sh.items + slot)[1] = k;
  };
  // every thread takes a run of items, an odd number: threads then start in different banks
  const int each = ((count + kPieceThreads - 1) / kPieceThreads) | 1;
  const int q0 = threadIdx.x * each, have = count - q0;
  Key key[kMost], prev = 0;
  float val[kMost];
  if (q0 > 0 && have > 0) prev = key_of(sh.items[q0 - 1]);
  unsigned int head_bits = 0;
#pragma unroll
  for (int j = 0; j < kMost; ++j) {
    if (j >= each) break;
    val[j] = 0.f;
    if (j < have) {
      const Item i = sh.items[q0 + j];
      key[j] = key_of(i);
      val[j] = LONG ? sh.vals[(unsigned int)i & ((1u << kIndexBits) - 1)]
                    : __uint_as_float((unsigned int)i);
      head_bits |= (unsigned int)(q0 + j == 0 || key[j] != prev) << j;
      prev = key[j];
    }
  }
  const unsigned int heads = __popc(head_bits);
  unsigned int total;
  // (all threads have read their items: the memory is free for keys and sums)
  const unsigned int first_slot = cta_exclusive<kWarps>(heads, sh.part, &total);
  // `lead`: what belongs to the key that is open before this thread's first item
  unsigned int slot = first_slot;
  float lead = 0.f, sum = 0.f;
#pragma unroll
  for (int j = 0; j < kMost; ++j) {
    if (j >= each) break;
    if (head_bits >> j & 1) {
      if (slot == first_slot) lead = sum;
      else put_sum(slot - 1, sum);
      put_key(slot++, key[j]);
      sum = 0.f;
    }
    sum += val[j];
  }
  const bool any = heads > 0;
  const float carry = carry_into(any, sum);
  if (any && first_slot > 0) put_sum(first_slot - 1, carry + lead);
  if (threadIdx.x == kPieceThreads - 1 && total > 0) put_sum(total - 1, any ? sum : carry + sum);
  __syncthreads();
  return total;
}

constexpr unsigned int kWidePiece = 1u << 31;  // beside a piece's distinct keys: some are too wide

// The arrays of a kernel: items, and (LONG) their values in another one.
struct Items {
  Item* keys;
  float* vals;
};

// The sampling CTA of piece_sum: the parts of the input are ranges of the highest bits or, where
// the sample's keys crowd together, of the sorted sample.
template <bool LONG>
__device__ __forceinline__ void sample_parts(const Item* keys, unsigned int n, const Buckets& b,
                                             const PieceShared& sh, SortHead* head,
                                             unsigned long long* host) {
  Item k[kPieceRows];
  int bits = 0;
  while (b.parts >> bits > 1) ++bits;
  const SampleShared mine{reinterpret_cast<unsigned int*>(sh.items),
                          reinterpret_cast<unsigned int*>(sh.items) + kSampleSlots};
  const bool spread = sample_spread<kPieceThreads>(keys, n, bits, b, mine, k);
  const bool split = !spread && b.splits;
  if (split) {
    constexpr int kLow = LONG ? kIndexBits : 32;
    // a larger one: as many keys in every part as make it unlikely that one has five times its
    // share
    constexpr int kRows = kPieceRows;
    const int rows = n < kPieceThreads * kRows ? n / kPieceThreads : kRows;
    const unsigned int count = kPieceThreads * rows, step = n / count;
#pragma unroll
    for (int j = 0; j < kPieceRows; ++j)
      if (j < rows) {
        const size_t i = (size_t)(threadIdx.x + j * kPieceThreads) * step;
        k[j] = (__ldcg(keys + i) & b.key_mask) << kLow;
      }
    if constexpr (LONG) {  // (what the index 0 reads)
      if (threadIdx.x == 0) sh.vals[0] = 0.f;
    }
    __syncthreads();
    // (every lane has an item in every row)
    sort_piece<LONG>(k, count, b.passes, b.width, sh);
    const unsigned int total = sum_piece<LONG>(count, sh);
    for (int q = threadIdx.x; q < b.parts; q += kPieceThreads) {
      const Item i = sh.items[(unsigned int)q * total / b.parts];
      b.splits[q] = LONG ? i : i >> 32;
    }
  }
  if (threadIdx.x == 0) {
    if (!b.splits) sample_report(spread, host);
    SortHead h{};
    h.groups = spread || split ? (n > kHelpItems ? 2 : 1) * b.parts / kGroup : 0;
    h.several = 1;
    h.split = split;
    h.separate = LONG;
    *head = h;
  }
}

// RAW: piece i is the i-th part of the input, and one CTA more looks at a sample of the keys.
template <bool RAW, bool LONG>
__global__ void __launch_bounds__(kPieceThreads, LONG ? 2 : 3)
    piece_sum_kernel(const Item* __restrict__ in, const unsigned int* __restrict__ vals,
                     long long n, Items out, const __grid_constant__ Buckets b, SortHead* head,
                     unsigned long long* host) {
  static_assert(RAW || !LONG, "buckets have pairs");
  constexpr int kLow = LONG ? kIndexBits : 32;
  grid_launch_next();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned int s_part[2 * kPieceWarps];
  const PieceShared sh(smem_raw, s_part);
  grid_wait();
  Piece p;
  if constexpr (RAW) {
    if (blockIdx.x == b.chunks) {
      sample_parts<LONG>(in, (unsigned int)n, b, sh, head, host);
      return;
    }
    const unsigned int size = (unsigned int)((n + b.chunks - 1) / b.chunks);
    const unsigned int from = blockIdx.x * size < n ? blockIdx.x * size : (unsigned int)n;
    p = {from, n - from < size ? (unsigned int)(n - from) : size, 0, (unsigned int)b.chunks};
    if (threadIdx.x == 0) b.pieces[blockIdx.x] = p;
  } else {
    if (__ldcg(&head->groups) == 0 || blockIdx.x >= __ldcg(&head->pieces)) return;
    const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(b.pieces + blockIdx.x));
    p = {raw.x, raw.y, raw.z, raw.w};
  }
  int count = (int)p.count;
  const int rows = (count + kPieceThreads - 1) / kPieceThreads;
  const int base = (threadIdx.x >> 5) * (32 * rows) + (threadIdx.x & 31);
  const int valid = valid_rows(count - base, rows);
  Item k[kPieceRows];
  bool wide = false;
#pragma unroll
  for (int j = 0; j < kPieceRows; ++j) {
    if (j % 2 == 0 && j >= rows) break;
    k[j] = j < valid ? __ldcg(in + p.start + base + j * 32) : 0;
  }
  if constexpr (RAW) {
#pragma unroll
    for (int j = 0; j < kPieceRows; ++j) {
      if (j % 2 == 0 && j >= rows) break;
      const int i = base + j * 32;
      const unsigned int v = j < valid ? __ldcg(vals + p.start + i) : 0u;
      wide |= (k[j] & ~b.key_mask) != 0;
      k[j] &= b.key_mask;
      if constexpr (LONG) {
        if (j < valid) sh.vals[i] = __uint_as_float(v);
        k[j] = k[j] << kLow | (unsigned int)i;
      } else {
        k[j] = k[j] << kLow | v;
      }
    }
    wide = __syncthreads_or(wide);
  }
  if (!RAW && p.pieces > 1) count = add_up_popular(k, count, sh);
  sort_piece<LONG, !RAW>(k, count, b.passes, b.width, sh);
  const unsigned int total = sum_piece<LONG>(count, sh);
  const int parts = b.parts;
  unsigned int* bounds = b.bounds + (size_t)blockIdx.x * parts;
  for (unsigned int i = threadIdx.x; i < total; i += kPieceThreads) {
    out.keys[p.start + i] = sh.items[i];
    if constexpr (LONG) out.vals[p.start + i] = sh.vals[i];
  }
  if (RAW || p.pieces > 1) {
    // where the parts begin: the first keys that are not below theirs
    const Item mask = (Item)(parts - 1) << b.part_shift;  // (the bits above are a bucket's)
    for (int q = threadIdx.x; q < parts; q += kPieceThreads) {
      unsigned int lo = 0, hi = total;
      while (lo < hi) {
        const unsigned int m = (lo + hi) / 2;
        const Item key = LONG ? sh.items[m] : sh.items[m] >> 32;
        if ((key & mask) < (Item)q << b.part_shift) lo = m + 1;
        else hi = m;
      }
      bounds[q] = lo;
    }
    if (threadIdx.x == 0) b.distinct[blockIdx.x] = total | (wide ? kWidePiece : 0);
  } else if (threadIdx.x < parts) {
    b.seg.counts[p.bucket * parts + threadIdx.x] = threadIdx.x ? 0 : total;
    b.seg.place[p.bucket * parts + threadIdx.x] = p.start;
  }
}

constexpr unsigned int kMerged = 1u << 31;  // a place in the merge's output
constexpr int kMaxGroup = 8;                // parts of the input that one CTA helps
static_assert(kFewPieces <= kPieceThreads && kMaxOfBucket <= 4 * kPieceThreads, "of a thread");
constexpr int kHelpers = kMergeCtas - kFewParts;
static_assert(kHelpers * kMaxGroup >= kFewParts && 2 * kFewParts <= kMaxSegments,
              "every part has a group, and segments");

// The input's parts of `group`, group + kHelpers, ...: the one with the most items, if those are
// more than a CTA sorts, else b.parts.  (One piece per thread.)
__device__ __forceinline__ unsigned int heaviest(const Buckets& b, unsigned int group,
                                                 unsigned int (&sums)[kMaxGroup][kPieceWarps]) {
  const unsigned int parts = b.parts, p = threadIdx.x;
  int j = 0;
  for (unsigned int q = group; q < parts; q += kHelpers, ++j) {
    unsigned int have = 0;
    if (p < (unsigned int)b.chunks) {
      const unsigned int* bound = b.bounds + (size_t)p * parts + q;
      have = (q + 1 < parts ? __ldcg(bound + 1) : __ldcg(b.distinct + p) & ~kWidePiece) -
             __ldcg(bound);
    }
    have = __reduce_add_sync(0xffffffffu, have);
    if ((p & 31) == 0) sums[j][p >> 5] = have;
  }
  __syncthreads();
  unsigned int most = kPiece, which = parts;
  j = 0;
  for (unsigned int q = group; q < parts; q += kHelpers, ++j) {
    unsigned int all = 0;
#pragma unroll
    for (int w = 0; w < kPieceWarps; ++w) all += sums[j][w];
    if (all > most) {
      most = all;
      which = q;
    }
  }
  return which;
}

// Unit u: part u / m of the u % m-th of the m buckets in several pieces.  A bucket is merged in as
// few parts as have room for the distinct keys of its pieces, with a third to spare: a unit then
// takes several parts, and those that follow have nothing to do.  The input is merged part by part.
//
// Popular ids, which every piece has, may make more than kPiece items of few keys, and a round more
// would be the longest of the kernel.  HELP: the CTAs that the parts of the input leave over help;
// each has a group of parts and takes the upper half of the heaviest, if that is more than one
// round.  A part then has two segments, the second one for its helper.
template <bool LONG, bool HELP>
__global__ void __launch_bounds__(kPieceThreads, 2)
    piece_merge_kernel(Items in, Items out, const __grid_constant__ Buckets b, SortHead* head,
                       unsigned long long* host) {
  constexpr int kLow = LONG ? kIndexBits : 32;
  grid_launch_next();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned int s_part[2 * kPieceWarps], s_scan[2][kPieceWarps], s_before[kPieceWarps];
  __shared__ unsigned int s_sums[HELP ? kMaxGroup : 1][kPieceWarps];
  __shared__ Item s_middle;
  __shared__ bool s_last;
  bool wide = false;
  const PieceShared sh(smem_raw, s_part);
  // of every piece: where its items go, and what to add to that for where they are (the memory of
  // the counters)
  unsigned int* to_at = reinterpret_cast<unsigned int*>(sh.cnt);
  unsigned int* from_at = to_at + kMaxOfBucket;
  static_assert(2 * kMaxOfBucket * 4 <= kPieceCount && kFewPieces <= kMaxOfBucket &&
                    kManyItems / kSmallPiece < kMaxOfBucket, "to_at and from_at");
  grid_wait();
  const int groups = __ldcg(&head->groups);
  const unsigned int buckets = __ldcg(&head->several), parts = b.parts;
  const bool split = __ldcg(&head->split) != 0;
  if (groups == 0) return;
  for (unsigned int u = blockIdx.x; u < buckets * parts + (HELP ? kHelpers : 0); u += gridDim.x) {
    Several s{0, 0, (unsigned int)b.chunks, 0};
    if (b.count) {
      const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(b.several + u % buckets));
      s = {raw.x, raw.y, raw.z, raw.w};
    }
    unsigned int part = u / buckets;
    bool halved = false;
    if constexpr (HELP) {
      halved = part >= parts;  // (a helper)
      if (halved) {
        if (split) continue;
        part = heaviest(b, u - parts, s_sums);
        if (part == parts) {  // (the same for all threads)
          __syncthreads();
          continue;
        }
      }
    }
    const bool helping = halved;
    const unsigned int segment = HELP ? 2 * part + helping : s.bucket * parts + part;
    Item low = 0, high = 0;
    if (split) {
      low = __ldcg(b.splits + part);
      if (part + 1 < parts) high = __ldcg(b.splits + part + 1);
    }
    // Each thread's pieces follow one another: what they have in all, of this part and of the parts
    // before.  (Up to four pieces of a bucket, one of the input; the first one's numbers are kept.)
    const unsigned int run = (s.pieces + kPieceThreads - 1) / kPieceThreads;
    const unsigned int p0 = threadIdx.x * run, p1 = p0 + run < s.pieces ? p0 + run : s.pieces;
    unsigned int span = 1;
    if (b.count) {
      unsigned int all = 0, total;
      for (unsigned int i = p0; i < p1; ++i) all += __ldcg(b.distinct + s.first + i);
      cta_exclusive<kPieceWarps>(all, s_scan[0], &total);
      for (span = parts; span > 1 && total * span / parts > kPiece * 3 / 4;) span /= 2;
      if (part % span) {  // (the same for all threads, like the other way out)
        if (threadIdx.x == 0) b.seg.counts[segment] = 0;
        __syncthreads();
        continue;
      }
    }
    struct Share {
      unsigned int from, to, start;
    };
    auto share_of = [&](unsigned int i) {
      const unsigned int p = s.first + i;
      Share h;
      unsigned int all = __ldcg(b.distinct + p);
      wide |= all >= kWidePiece;
      all &= ~kWidePiece;
      h.start = __ldcg(&b.pieces[p].start);
      const unsigned int* bound = b.bounds + (size_t)p * parts + part;
      h.from = split ? 0 : __ldcg(bound);
      h.to = part + span < parts && !split ? __ldcg(bound + span) : all;
      return h;
    };
    Share first{0, 0, 0};
    if (p0 < p1) first = share_of(p0);
    if (split) {
      // the first keys that are not below `low` and `high`
      const Item* keys = in.keys + first.start;
      unsigned int f0 = 0, f1 = part ? first.to : 0, t0 = 0, t1 = first.to;
      if (part + 1 == parts) t0 = t1;
      while (f0 < f1 || t0 < t1) {
        const unsigned int f = (f0 + f1) / 2, t = (t0 + t1) / 2;
        const Item kf = f0 < f1 ? __ldcg(keys + f) : 0, kt = t0 < t1 ? __ldcg(keys + t) : 0;
        if (f0 < f1) {
          if ((LONG ? kf : kf >> 32) < low) f0 = f + 1;
          else f1 = f;
        }
        if (t0 < t1) {
          if ((LONG ? kt : kt >> 32) < high) t0 = t + 1;
          else t1 = t;
        }
      }
      first.from = f0;
      first.to = t0;
    }
    unsigned int have = first.to - first.from, smaller = first.from;
    for (unsigned int i = p0 + 1; i < p1; ++i) {
      const Share h = share_of(i);
      have += h.to - h.from;
      smaller += h.from;
    }
    unsigned int count, before = 0;
    smaller = __reduce_add_sync(0xffffffffu, smaller);
    if ((threadIdx.x & 31) == 0) s_before[threadIdx.x >> 5] = smaller;
    unsigned int at = cta_exclusive<kPieceWarps>(have, s_scan[1], &count);
#pragma unroll
    for (int w = 0; w < kPieceWarps; ++w) before += s_before[w];
    if constexpr (HELP) {
      if (!helping && !split && count > kPiece)
        halved = heaviest(b, part % kHelpers, s_sums) == part;
      if (halved) {
        // the upper half begins at the key in the middle of what the first piece has
        if (threadIdx.x == 0) {
          const unsigned int size = first.to - first.from;
          Item k = ((Item)part << b.part_shift) + ((Item)1 << (b.part_shift - 1));
          if (size) {
            k = __ldcg(in.keys + first.start + first.from + size / 2);
            if constexpr (!LONG) k >>= 32;
          }
          s_middle = k;
        }
        __syncthreads();
        const Item* keys = in.keys + first.start;
        unsigned int lo = first.from, hi = first.to;
        while (lo < hi) {
          const unsigned int m = (lo + hi) / 2;
          const Item k = __ldcg(keys + m);
          if ((LONG ? k : k >> 32) < s_middle) lo = m + 1;
          else hi = m;
        }
        if (helping) first.from = lo;
        else first.to = lo;
        smaller = __reduce_add_sync(0xffffffffu, first.from);
        if ((threadIdx.x & 31) == 0) s_before[threadIdx.x >> 5] = smaller;
        at = cta_exclusive<kPieceWarps>(first.to - first.from, s_scan[0], &count);
        before = 0;
#pragma unroll
        for (int w = 0; w < kPieceWarps; ++w) before += s_before[w];
      }
    }
    // As many items as there is room for, in one round; where there are more, distinct keys make
    // room for the next ones.  (Given up where they leave less than a quarter, unless the next
    // round is the last: 560 000 ids of 24 bits in seven ranges have parts of 5000 items and some
    // more, 110 us when these were given up, now 79.)
    unsigned int taken = 0, total = 0;
    for (;;) {
      if (p0 < p1) {
        to_at[p0] = at;
        from_at[p0] = first.start + first.from - at;
        unsigned int to = at + (first.to - first.from);
        for (unsigned int i = p0 + 1; i < p1; ++i) {
          const Share h = share_of(i);
          to_at[i] = to;
          from_at[i] = h.start + h.from - to;
          to += h.to - h.from;
        }
      }
      __syncthreads();
      const unsigned int kept = total;
      const unsigned int room = kPiece - kept, left = count - taken;
      const unsigned int items = kept + (left < room ? left : room);
      const int rows = ((int)items + kPieceThreads - 1) / kPieceThreads;
      const int base = (threadIdx.x >> 5) * (32 * rows) + (threadIdx.x & 31);
      const int valid = valid_rows((int)items - base, rows);
      Item k[kPieceRows];
#pragma unroll
      for (int j = 0; j < kPieceRows; ++j) {
        if (j % 2 == 0 && j >= rows) break;
        const unsigned int q = base + j * 32;
        if (q < kept) {
          k[j] = sh.items[q];
        } else {
          const unsigned int i = q - kept + taken;
          unsigned int lo = 0, hi = s.pieces;  // the last piece that begins at i or before has it
          while (hi - lo > 1) {
            const unsigned int m = (lo + hi) / 2;
            if (to_at[m] <= i) lo = m;
            else hi = m;
          }
          const unsigned int from = from_at[lo] + i;
          k[j] = j < valid ? __ldcg(in.keys + from) : 0;
          if constexpr (LONG) {
            if (j < valid) sh.vals[q] = __ldcg(in.vals + from);
          }
        }
        if constexpr (LONG) k[j] = k[j] << kLow | q;
      }
      __syncthreads();
      if (split) sort_piece<LONG>(k, (int)items, b.passes, b.width, sh);
      else sort_piece<LONG>(k, (int)items, b.merge_passes, b.merge_width, sh);
      total = sum_piece<LONG>((int)items, sh);
      taken += items - kept;
      if (taken == count || (int)total > max(kPiece * 3 / 4, kPiece - (int)(count - taken))) break;
    }
    if (taken < count) {  // (the same for all threads)
      if (threadIdx.x == 0) {
        head->crowded = 1;
        b.seg.counts[segment] = 0;
      }
      __syncthreads();
      continue;
    }
    for (unsigned int i = threadIdx.x; i < total; i += kPieceThreads) {
      out.keys[s.start + before + i] = sh.items[i];
      if constexpr (LONG) out.vals[s.start + before + i] = sh.vals[i];
    }
    if (threadIdx.x == 0) {
      b.seg.counts[segment] = total;
      b.seg.place[segment] = (s.start + before) | kMerged;
      if (HELP && !halved) b.seg.counts[segment + 1] = 0;
    }
    __syncthreads();
  }
  // the last CTA: prefix of the counts.  (What this CTA's threads have written comes before its
  // thread 0 counts it done, and what all others have before whatever the last one's threads read.)
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int done;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                 : "=r"(done) : "l"(&head->done) : "memory");
    s_last = done + 1 == gridDim.x;
  }
  __syncthreads();
  if (!s_last) return;
  if (b.count)
    for (int i = threadIdx.x; i < b.chunks; i += kPieceThreads) wide |= __ldcg(b.wide + i) != 0;
  // (all loads of a thread are in flight at once)
  constexpr int kEach = kMaxSegments / kPieceThreads;
  const int segments = groups * kGroup, each = (segments + kPieceThreads * 4 - 1) /
                                               (kPieceThreads * 4) * 4;
  uint4* at4 = reinterpret_cast<uint4*>(b.seg.counts + threadIdx.x * each);
  uint4 c[kEach / 4];
  unsigned int sum = 0, total;
#pragma unroll
  for (int j = 0; j < kEach / 4; ++j)
    c[j] = j * 4 < each && (int)threadIdx.x * each + j * 4 < segments ? __ldcg(at4 + j)
                                                                      : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int j = 0; j < kEach / 4; ++j) sum += c[j].x + c[j].y + c[j].z + c[j].w;
  unsigned int at = cta_exclusive<kPieceWarps>(sum, s_scan[0], &total);
#pragma unroll
  for (int j = 0; j < kEach / 4; ++j) {
    if (j * 4 < each && (int)threadIdx.x * each + j * 4 < segments) {
      uint4 p;
      p.x = at;
      p.y = p.x + c[j].x;
      p.z = p.y + c[j].y;
      p.w = p.z + c[j].z;
      at = p.w + c[j].w;
      at4[j] = p;
    }
  }
  wide = __syncthreads_or(wide);
  if (threadIdx.x == 0) {
    b.seg.counts[segments] = total;
    const bool crowded = *(volatile int*)&head->crowded != 0;
    // (without a fence behind it, which the end of the kernel is)
    *(volatile unsigned long long*)host = kReported | (wide ? kReportWide : 0) |
                                          (crowded ? kReportCrowded : 0) | total;
  }
}

}  // namespace sortk
}  // namespace psdev
