// Part of pull_gemm.cu: the GEMM of large products, C[M,N] = X[M,K] * W[N,K]^T.
//
// A pair of CTAs (tcgen05 cta_group::2) owns a 256 x 512 output tile.  Large products run under the
// power limit, where every byte moved costs clock: this tile takes 48 bytes per tensor-pipe clock
// and SM from L2, the 256 x 256 tile of the other pair kernel 64.  Tiles of 256 columns (NT = 256)
// remain for products of about one round, which wide tiles would fill unevenly.
//
// Accumulators are two halves of 256 columns and fill the tensor memory.  With NT = 256 a tile uses
// one and the next tile the other.  With NT = 512 it uses both, and a tile could not start while
// its predecessor is being drained -- except half by half: the first and the last kWideSkew
// k-blocks are multiplied for one half and then for the other, so half 0 is complete kWideSkew *
// 516 clocks before half 1 and drained in that time, and half 1 is drained while the next tile
// begins with half 0.
//
// Results leave through shared memory (128-byte swizzle) and TMA stores of 64 x 32 values: rows of
// any length leave in whole sectors.
//
// What a small number of tiles costs is latency.  The kernel is launched with programmatic stream
// serialization, so that its prologue runs beside the end of the kernel before it; no barrier is
// looked at where the answer may take a time slice (a try_wait for a k-block that does not come
// held back the last commit by 10 000 clocks); and shared memory is given up once it has been
// read.
//
// Measured, us, launches back to back, this kernel / pull_gemm_pair_kernel before it / cuBLAS:
//   16384 x 3072 x 1024 86 / 96 / 89          2048 x 4096 x 1024 15.1 / 21.2 / 14.3
//   16384 x 3000 x 1000 96 / 125 / 100        2048 x 2048 x 1024 10.3 / 16.0 / 8.4
//   8192 x 4096 x 4096 203 / 232 (one-CTA 256-row tile) / 210
//
// Every wait is bounded; on expiry the kernel records an error, lets its copies land and leaves.
#pragma once

namespace psdev {
namespace gemm {

constexpr int kWideThreads = 352;  // warp 0 TMA loads, 1 MMA, 2..9 epilogue, 10 watches loads
constexpr int kWideSkew = 2;
// NT: columns of a tile, 256 or 512.
template <int NT>
struct WideCfg {
  static constexpr int kHalf = 128 * BK * 2;         // 128 rows of one operand, 64 columns of K
  static constexpr int kStageBytes = (1 + NT / 256) * kHalf;  // X, W of half 0, W of half 1
  static constexpr int kStages = NT == 512 ? 4 : 6;
  static constexpr int kOutBytes = 32 * 64 * 2;      // one store: 32 rows of 64 values
  static constexpr int kSmemBytes = kStages * kStageBytes + 8 * kOutBytes + 1024;
};

struct WideArgs {
  long long M, N;
  int num_kb, tiles_m, tiles_n, group;
  int* status;
  unsigned long long timeout_ns;
};

template <int NT>
__global__ void __launch_bounds__(kWideThreads, 1)
    wide_gemm_kernel(const __grid_constant__ WideArgs a, const __grid_constant__ CUtensorMap tmap_x,
                     const __grid_constant__ CUtensorMap tmap_w,
                     const __grid_constant__ CUtensorMap tmap_w64,
                     const __grid_constant__ CUtensorMap tmap_c) {
  using namespace sm100;
  using C = WideCfg<NT>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[C::kStages], empty_bar[C::kStages];
  __shared__ __align__(8) uint64_t tmem_full[2], tmem_empty[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ uint32_t s_ready;  // k-blocks in place
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* out = smem + C::kStages * C::kStageBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();  // 0 = leader
  const long long pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const long long num_tiles = (long long)a.tiles_m * a.tiles_n;
  const int num_kb = a.num_kb;
  // The tiles of a last round that is at most half full are cut along N into 2 or 4 items, each
  // for a pair of its own.
  const long long rest = num_tiles % num_pairs;
  int split = 1;
  if (rest != 0) split = NT == 512 && rest * 4 <= num_pairs ? 4 : rest * 2 <= num_pairs ? 2 : 1;
  const long long num_whole = split > 1 ? num_tiles - rest : num_tiles;
  const long long num_items = num_whole + (split > 1 ? rest * split : 0);
  // item -> first row and column, halves (0: nothing of it lies inside C) and columns per half
  auto item_of = [&](long long i, int* row, int* col, int* halves, int* width) {
    const long long j = i - num_whole;
    int tn, tm;
    tile_order(i < num_whole ? i : num_whole + j / split, a.tiles_m, a.tiles_n, a.group, &tn, &tm);
    *row = tm * 256;
    *col = tn * NT;
    int cols = NT;
    if (i >= num_whole) {
      cols = NT / split;
      *col += (int)(j % split) * cols;
    }
    *width = cols < 256 ? cols : 256;
    *halves = *col >= a.N ? 0 : (NT == 512 && cols > 256 && *col + 256 < a.N) ? 2 : 1;
  };

  if (threadIdx.x == 0) {
    grid_launch_next();
    s_abort = 0;
    s_ready = 0;
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full_bar[s], 1);   // the leader's arrive.expect_tx; bytes come from both CTAs
      mbar_init(&empty_bar[s], 1);  // the leader's commit, delivered to both CTAs
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&tmem_full[h], 1);
      mbar_init(&tmem_empty[h], 16);  // eight epilogue warps of each CTA
    }
    fence_barrier_init();
    prefetch_tmap(&tmap_x);
    prefetch_tmap(&tmap_w);
    prefetch_tmap(&tmap_c);
  }
  if (warp == 1) {
    tmem_alloc_pair(&s_tmem, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();  // both CTAs' barriers exist before anything can signal them
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  volatile int* abort_flag = &s_abort;

  if (warp == 0) {
    grid_wait();  // (all other accesses to global memory follow from these loads)
    uint32_t c = 0;  // k-blocks loaded
    bool ok = true;
    for (long long it = pair; it < num_items && ok; it += num_pairs) {
      int row, col, halves, width;
      item_of(it, &row, &col, &halves, &width);
      if (halves == 0) continue;
      const int wrow = col + (int)cta * (width / 2);
      const CUtensorMap* tw = width == 128 ? &tmap_w64 : &tmap_w;  // box: 64 or 128 rows
      const uint32_t bytes =
          (uint32_t)(2 * C::kHalf + (width == 128 ? C::kHalf : halves * 2 * C::kHalf));
      for (int kb = 0; kb < num_kb; ++kb, ++c) {
        const int s = (int)(c % C::kStages);
        ok = mbar_wait_bounded(&empty_bar[s], ((c / C::kStages) & 1) ^ 1, abort_flag, a.timeout_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (elect_one()) {
          unsigned char* sa = smem + s * C::kStageBytes;
          if (cta == 0) mbar_arrive_expect_tx(&full_bar[s], bytes);
          tma_load_2d_pair(sa, &tmap_x, kb * BK, row + (int)cta * 128, &full_bar[s]);
          tma_load_2d_pair(sa + C::kHalf, tw, kb * BK, wrow, &full_bar[s]);
          if (halves == 2)
            tma_load_2d_pair(sa + 2 * C::kHalf, tw, kb * BK, wrow + 256, &full_bar[s]);
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) {
      atomicMin(a.status, (int)PSDEV_ERR_TIMEOUT_PIPE);
      // copies in flight land before shared memory is released (the other CTA waits for this one
      // at the end)
      for (uint32_t j = c > C::kStages ? c - C::kStages : 0; cta == 0 && j < c; ++j) {
        const unsigned long long t0 = gtimer_ns();
        while (!mbar_try_wait(&full_bar[j % C::kStages], (j / C::kStages) & 1) &&
               gtimer_ns() - t0 < 2000000ull) {}
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (cta == 0) {
      // The whole warp walks the k-blocks and one elected thread issues (descriptors in uniform
      // registers).  It touches no mbarrier between two commits (see wait_ready).
      const uint64_t desc_a = make_desc_k128(smem), desc_b = make_desc_k128(smem + C::kHalf);
      uint32_t idesc = 0;
      uint32_t c = 0, seen = 0;  // k-blocks multiplied by earlier items; known to be in place
      uint32_t used[2] = {0, 0};
      bool ok = true;
      auto drained = [&](int h) {
        const bool o = mbar_wait_bounded(&tmem_empty[h], (used[h] & 1) ^ 1, abort_flag,
                                         a.timeout_ns);
        ok = __all_sync(0xffffffffu, o);
        tc_fence_after();
        ++used[h];
        return ok;
      };
      auto arrived = [&](uint32_t k) {
        if (k >= seen) ok = wait_ready(&s_ready, k, &seen, abort_flag, a.timeout_ns);
        return ok;
      };
      auto mma = [&](uint32_t k, int h, int acc, bool first) {
        if (elect_one()) {
          const uint64_t off = (uint64_t)((k % C::kStages) * (C::kStageBytes >> 4));
          const uint64_t da = desc_a + off, db = desc_b + off + (uint64_t)(h * (C::kHalf >> 4));
#pragma unroll
          for (int i = 0; i < BK / UMMA_K; ++i)
            umma_f16_pair(tmem + (uint32_t)(acc * 256), da + (uint64_t)(2 * i),
                          db + (uint64_t)(2 * i), idesc, first && i == 0 ? 0u : 1u);
        }
        __syncwarp();
      };
      auto commit = [&](uint64_t* bar) {
        if (elect_one()) umma_commit_pair(bar);
        __syncwarp();
      };
      int acc0 = NT == 512 ? 0 : 1;
      for (long long it = pair; it < num_items && ok; it += num_pairs) {
        int row, col, halves, width;
        item_of(it, &row, &col, &halves, &width);
        if (halves == 0) continue;
        idesc = make_idesc_bf16(256, width);
        if (NT == 256) acc0 ^= 1;
        if (!drained(acc0)) break;
        const int skew = halves == 1 ? 0 : num_kb / 2 < kWideSkew ? num_kb / 2 : kWideSkew;
        for (int kb = 0; kb < skew && ok; ++kb)
          if (arrived(c + kb)) mma(c + kb, 0, acc0, kb == 0);
        if (!ok || (halves == 2 && !drained(1))) break;
        for (int kb = 0; kb < num_kb && ok; ++kb) {
          const uint32_t k = c + kb;
          if (kb == num_kb - skew) {
            for (int j = kb; j < num_kb && ok; ++j)
              if (arrived(c + j)) mma(c + j, 0, acc0, j == 0);
            if (!ok) break;
            commit(&tmem_full[acc0]);
          }
          if (kb >= skew && kb < num_kb - skew) {
            if (!arrived(k)) break;
            mma(k, 0, acc0, kb == 0);
          }
          if (halves == 2) mma(k, 1, 1, kb == 0);
          commit(&empty_bar[k % C::kStages]);
        }
        if (!ok) break;
        if (skew == 0) commit(&tmem_full[acc0]);
        if (halves == 2) commit(&tmem_full[1]);
        c += (uint32_t)num_kb;
      }
      if (!ok && lane == 0) atomicMin(a.status, (int)PSDEV_ERR_TIMEOUT_PIPE);
    }
    __syncwarp();
  } else if (warp == 10) {
    if (cta == 0 && lane == 0) {
      uint32_t c = 0;
      bool ok = true;
      for (long long it = pair; it < num_items && ok; it += num_pairs) {
        int row, col, halves, width;
        item_of(it, &row, &col, &halves, &width);
        if (halves == 0) continue;
        for (int kb = 0; kb < num_kb && ok; ++kb, ++c) {
          ok = mbar_wait_bounded(&full_bar[c % C::kStages], (c / C::kStages) & 1, abort_flag,
                                 a.timeout_ns);
          if (ok) st_ready(&s_ready, c + 1);
        }
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3;            // tensor-memory lane quarter this warp may read
    const int side = (warp - 2) >> 2;  // first or second part of the columns of a half
    unsigned char* slab = out + (warp - 2) * C::kOutBytes;
    uint32_t used[2] = {0, 0};
    bool ok = true;
    int acc0 = NT == 512 ? 0 : 1;
    for (long long it = pair; it < num_items && ok; it += num_pairs) {
      int row, col, halves, width;
      item_of(it, &row, &col, &halves, &width);
      if (halves == 0) continue;
      if (NT == 256) acc0 ^= 1;
      row += (int)cta * 128 + q * 32;
      for (int h = 0; h < halves; ++h) {
        const int acc = NT == 512 ? h : acc0;
        ok = mbar_wait_bounded(&tmem_full[acc], used[acc] & 1, abort_flag, a.timeout_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        ++used[acc];
        tc_fence_after();
        const int cols = width / 2;  // 64 or 128
        for (int c0 = 0; c0 < cols; c0 += 64) {
          const int in_half = side * cols + c0;
          uint32_t r[2][32];
          const uint32_t taddr =
              tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 256 + in_half);
          tmem_ld_32x32(taddr, r[0]);
          tmem_ld_32x32(taddr + 32, r[1]);
          tmem_ld_wait();
          if (c0 + 64 == cols) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(&tmem_empty[acc]);
          }
          const int gcol = col + h * 256 + in_half;
          if (lane == 0) bulk_wait_read<0>();  // the previous store has left the slab
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t* v = &r[j >> 2][8 * (j & 3)];
            uint4 u;
            u.x = f2_to_bf16x2(__uint_as_float(v[0]), __uint_as_float(v[1]));
            u.y = f2_to_bf16x2(__uint_as_float(v[2]), __uint_as_float(v[3]));
            u.z = f2_to_bf16x2(__uint_as_float(v[4]), __uint_as_float(v[5]));
            u.w = f2_to_bf16x2(__uint_as_float(v[6]), __uint_as_float(v[7]));
            *reinterpret_cast<uint4*>(slab + lane * 128 + ((j ^ (lane & 7)) << 4)) = u;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && gcol < a.N && row < a.M) {
            tma_store_2d(&tmap_c, gcol, row, slab);
            bulk_commit();
          }
        }
      }
    }
    if (lane == 0) {
      bulk_wait_read<0>();  // shared memory outlives its stores
      if (!ok) atomicMin(a.status, (int)PSDEV_ERR_TIMEOUT_PIPE);
    }
    __syncwarp();
  }
  // neither CTA frees its tensor memory while a pair MMA might still use it
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

}  // namespace gemm
}  // namespace psdev
