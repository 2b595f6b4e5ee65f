// C[M,N] = X[M,K] * W[N,K]^T for products that are too small to fill the GPU with the large
// tiles of the persistent kernels (pull_gemm.cu).
//
// One 128 x BN output tile per cluster of S CTAs; CTA s of the cluster multiplies the s-th part
// of K.  With S > 1 the partial sums (fp32) are exchanged through distributed shared memory: every
// CTA stores into each of the others the BN / S columns that are theirs, out of its tensor memory,
// meets them once, and adds up its own columns in the order of the parts.  When every CTA read its
// columns from the others between two barriers, and the sums lay row by row (a warp's accesses 32
// pieces of 16 bytes), the exchange took 3 us among four CTAs and 6 among eight; now 1.5.  us,
// 75 x 928 x 3504 with S = 4 / 8: 8.7 / 9.8 before, 7.2 / 5.9 now (S = 1 13.6); 64 x 256 x 4096
// 9.2 / 9.9 and 7.3 / 5.7; 92 x 592 x 1360 6.9 / 11.4 and 5.1 / 5.5.
// There is no loop over tiles, no counter in global memory, and the first loads are issued before
// the CTA has met at its first barrier, because what bounds these products is a chain of
// latencies: launch, operands from L2 or HBM, a few MMAs, accumulator, store.
//   warp 0      TMA producer; sets up the barriers and starts loading at once;
//   warp 1      allocates tensor memory, issues tcgen05.mma;
//   warps 2..5  epilogue, each its quarter of the accumulator rows.
// Launched with programmatic stream serialization: the prologue runs beside the end of the kernel
// before it.
//
// Two forms.  With more CTAs than SMs up to 100 KB of shared memory per CTA, so that two share an
// SM and one loads while the other stores (121 KB and one with 128 columns and S = 4 or 8, whose
// exchange takes 48 and 56).  Otherwise (DEEP) one CTA has the SM, and a stage holds
// two k-blocks: per stage the ring costs some 300 clocks (commit, barrier, producer) whatever it
// carries, and 128 columns of K make up for them.  The issuer of the deep form touches no mbarrier
// (see wait_ready).  1024 x 1024 x 4096 with BN = 64 / 128 20.9 / 24.5 us shallow, 16.5 / 18.2
// deep; what is left is the loads, 70 bytes per clock and SM.
//
// Measured, us (this kernel / the persistent 128 x 256 kernel): 64x256x256 2.8 / 6.5,
// 1024x1024x256 4.1 / 8.4, 1024x1024x1024 6.0 / 11.9, 64x256x4096 5.7 / 23.4 (S = 8).
#pragma once
#include "ps/device/sm100_ptx.cuh"

namespace psdev {
namespace gemm {

constexpr int kSplitThreads = 192;
constexpr int kMaxSplit = 8;

struct SplitArgs {
  long long M, N;
  int num_kb, tiles_m;
  __nv_bfloat16* c;
  int* status;
  unsigned long long timeout_ns;
};

template <int BN, int S, bool DEEP>
struct SplitCfg {
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBlockBytes = kABytes + BN * BK * 2;  // one k-block
  static constexpr int kSub = DEEP ? 2 : 1;                  // k-blocks of a stage
  static constexpr int kStageBytes = kSub * kBlockBytes;
  // What the other parts send has memory of its own: they may be ahead of this CTA's operands.
  // (Four columns of all rows, then the next four: a warp's stores and loads are contiguous.)
  static constexpr int kPartBytes = BM * (BN / S) * 4;
  static constexpr int kExchange = (S - 1) * kPartBytes;
  static constexpr int kStages = S == 1 ? (BN == 64 ? 4 : 3)
                                 : BN == 128 ? 2 : (S == 8 ? 2 : 3) + (DEEP ? 1 : 0);
  static constexpr int kTiles = kStages * kStageBytes;
  static constexpr int kSmemBytes = kTiles + kExchange + 1024 /*align*/;
};

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, const uint32_t* r) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, uint32_t cta) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(cta));
  return a;
}
__device__ __forceinline__ void store_bf16x8(__nv_bfloat16* p, const float* f) {
  uint4 u;
  u.x = f2_to_bf16x2(f[0], f[1]);
  u.y = f2_to_bf16x2(f[2], f[3]);
  u.z = f2_to_bf16x2(f[4], f[5]);
  u.w = f2_to_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

template <int BN, int S, bool DEEP>
__global__ void __launch_bounds__(kSplitThreads)
    split_gemm_kernel(const __grid_constant__ SplitArgs a,
                      const __grid_constant__ CUtensorMap tmap_x,
                      const __grid_constant__ CUtensorMap tmap_w) {
  using namespace sm100;
  using C = SplitCfg<BN, S, DEEP>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[C::kStages], empty_bar[C::kStages], done_bar;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ uint32_t s_ready;  // k-blocks in place (DEEP)
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = S > 1 ? (int)cluster_ctarank() : 0;
  const int tile = (int)blockIdx.x / S;
  const int tm = tile % a.tiles_m, tn = tile / a.tiles_m;
  const int kb0 = (int)((long long)a.num_kb * part / S);
  const int nkb = (int)((long long)a.num_kb * (part + 1) / S) - kb0;

  const int nst = (nkb + C::kSub - 1) / C::kSub;  // stages to fill

  auto load = [&](int i, int s) {
    const int n = nkb - i * C::kSub < C::kSub ? nkb - i * C::kSub : C::kSub;
    uint64_t* bar = &full_bar[s];
    mbar_arrive_expect_tx(bar, n * C::kBlockBytes);
    for (int j = 0; j < n; ++j) {
      unsigned char* sa = smem + s * C::kStageBytes + j * C::kBlockBytes;
      const int x = (kb0 + i * C::kSub + j) * BK;
      tma_load_2d(sa, &tmap_x, x, tm * BM, bar);
      tma_load_2d(sa + C::kABytes, &tmap_w, x, tn * BN, bar);
    }
  };
  const int ahead = nst < C::kStages ? nst : C::kStages;
  if (threadIdx.x == 0) {
    s_abort = 0;
    s_ready = 0;
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&done_bar, 1);
    fence_barrier_init();
    grid_launch_next();
    grid_wait();  // (all other accesses to global memory follow from these loads)
    for (int i = 0; i < ahead; ++i) load(i, i);
  }
  if (warp == 1) {
    tmem_alloc(&s_tmem, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if constexpr (S > 1) cluster_arrive();
  const uint32_t tmem = s_tmem;
  volatile int* abort_flag = &s_abort;

  if (warp == 0) {
    int s = 0;
    uint32_t phase = 0;
    for (int i = ahead; i < nst; ++i) {
      const bool ok = mbar_wait_bounded(&empty_bar[s], phase, abort_flag, a.timeout_ns);
      if (!__all_sync(0xffffffffu, ok)) {
        // copies in flight land before shared memory is released
        if (lane == 0) {
          atomicMin(a.status, (int)PSDEV_ERR_TIMEOUT_PIPE);
          for (int j = i - C::kStages; j < i; ++j) {
            const unsigned long long t0 = gtimer_ns();
            while (!mbar_try_wait(&full_bar[j % C::kStages], (uint32_t)(j / C::kStages) & 1) &&
                   gtimer_ns() - t0 < 2000000ull) {}
          }
        }
        break;
      }
      if (elect_one()) load(i, s);
      __syncwarp();
      if (++s == C::kStages) { s = 0; phase ^= 1; }
    }
    __syncwarp();
  } else if (warp == 1) {
    // The whole warp walks the stages and one elected thread issues, so that descriptors stay in
    // uniform registers.  The shallow form looks at the next stage's barrier between the MMAs and
    // their commit: an mbarrier access behind a commit waits for it.  And no fence follows the
    // wait: operands arrive through the async proxy, whose barrier has been observed.
    constexpr uint32_t idesc = make_idesc_bf16(BM, BN);
    const uint64_t desc_a = make_desc_k128(smem), desc_b = make_desc_k128(smem + C::kABytes);
    bool ok = true, ready = false;
    uint32_t phase = 0, seen = 0;
    // (stages unrolled: their descriptors are constants away from two that stay in registers)
    for (int i0 = 0; i0 < nst && ok; i0 += C::kStages, phase ^= 1) {
#pragma unroll
      for (int s = 0; s < C::kStages; ++s) {
        const int i = i0 + s;
        if (i >= nst) break;
        if constexpr (DEEP) {
          if ((uint32_t)i >= seen)
            ok = wait_ready(&s_ready, (uint32_t)i, &seen, abort_flag, a.timeout_ns);
          if (!ok) break;
        } else if (!ready) {
          ok = mbar_wait_bounded(&full_bar[s], phase, abort_flag, a.timeout_ns);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < C::kSub; ++j) {
            if (j > 0 && i * C::kSub + j >= nkb) break;
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k) {
              const int off = (s * C::kStageBytes + j * C::kBlockBytes) >> 4;
              umma_f16(tmem, desc_a + (uint64_t)(off + 2 * k), desc_b + (uint64_t)(off + 2 * k),
                       idesc, (i | j | k) != 0 ? 1u : 0u);
            }
          }
        }
        __syncwarp();
        constexpr int kLast = C::kStages - 1;
        if constexpr (!DEEP)
          ready = __all_sync(0xffffffffu, i + 1 < nst &&
                             mbar_test_wait(&full_bar[s == kLast ? 0 : s + 1],
                                            s == kLast ? phase ^ 1 : phase));
        if (elect_one()) {
          if (i + C::kStages < nst) umma_commit(&empty_bar[s]);
          if (i == nst - 1) umma_commit(&done_bar);
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) atomicMin(a.status, (int)PSDEV_ERR_TIMEOUT_PIPE);
    __syncwarp();
  } else {
    const int q = warp & 3;  // tensor-memory lane quarter this warp may read
    if (DEEP && warp == 2) {  // nothing to store yet: count the k-blocks in place
      if (lane == 0) {
        for (int i = 0; i < nst; ++i) {
          if (!mbar_wait_bounded(&full_bar[i % C::kStages], (uint32_t)(i / C::kStages) & 1,
                                 abort_flag, a.timeout_ns))
            break;
          st_ready(&s_ready, (uint32_t)i + 1);
        }
      }
      __syncwarp();
    }
    const bool ok = mbar_wait_bounded(&done_bar, 0, abort_flag, a.timeout_ns);
    __syncwarp();
    tc_fence_after();
    const int in_tile = q * 32 + lane;
    const long long row = (long long)tm * BM + in_tile;
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
    const bool all_ok = __all_sync(0xffffffffu, ok);
    if constexpr (S == 1) {
      if (all_ok) {
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32(taddr + (uint32_t)c0, r);
          tmem_ld_wait();
          if (row < a.M) {
            const long long col = (long long)tn * BN + c0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col + j * 8 + 8 <= a.N) {
                float f[8];
#pragma unroll
                for (int x = 0; x < 8; ++x) f[x] = __uint_as_float(r[8 * j + x]);
                store_bf16x8(a.c + row * a.N + col + j * 8, f);
              }
          }
        }
      }
      tc_fence_before();
    } else {
      constexpr int kCols = BN / S, kOnce = kCols < 32 ? kCols : 32;
      const uint32_t inbox = smem_u32(smem) + C::kTiles;
      cluster_wait();  // the other parts have begun: their memory can be written
      uint32_t own[kCols];
      if (all_ok) {
#pragma unroll 1
        for (int d = 1; d < S; ++d) {
          const int to = (part + d) % S;
          const uint32_t dst = cluster_addr(
              inbox + (uint32_t)((part < to ? part : part - 1) * C::kPartBytes + in_tile * 16),
              (uint32_t)to);
#pragma unroll
          for (int c0 = 0; c0 < kCols; c0 += kOnce) {
            uint32_t r[kOnce];
#pragma unroll
            for (int j = 0; j < kOnce; j += 8)
              tmem_ld_32x8(taddr + (uint32_t)(to * kCols + c0 + j), r + j);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < kOnce; j += 4) st_cluster_v4(dst + (c0 + j) * BM * 4, r + j);
          }
        }
#pragma unroll
        for (int j = 0; j < kCols; j += 8)
          tmem_ld_32x8(taddr + (uint32_t)(part * kCols + j), own + j);
        tmem_ld_wait();
      }
      tc_fence_before();
      __syncwarp();
      cluster_sync_all();  // every part's columns are in place, and nobody writes here any more
      // (a part that gave up has sent nothing and recorded its error: the results are void)
      if (all_ok && row < a.M) {
#pragma unroll
        for (int c0 = 0; c0 < kCols; c0 += 8) {
          float f[8] = {};
#pragma unroll
          for (int s = 0; s < S; ++s) {
            float4 lo, hi;
            if (s == part) {
              lo = make_float4(__uint_as_float(own[c0]), __uint_as_float(own[c0 + 1]),
                               __uint_as_float(own[c0 + 2]), __uint_as_float(own[c0 + 3]));
              hi = make_float4(__uint_as_float(own[c0 + 4]), __uint_as_float(own[c0 + 5]),
                               __uint_as_float(own[c0 + 6]), __uint_as_float(own[c0 + 7]));
            } else {
              const float4* from = reinterpret_cast<const float4*>(
                  smem + C::kTiles + (s < part ? s : s - 1) * C::kPartBytes + in_tile * 16 +
                  c0 * BM * 4);
              lo = from[0];
              hi = from[BM];
            }
            f[0] += lo.x; f[1] += lo.y; f[2] += lo.z; f[3] += lo.w;
            f[4] += hi.x; f[5] += hi.y; f[6] += hi.z; f[7] += hi.w;
          }
          const long long col = (long long)tn * BN + part * kCols + c0;
          if (col + 8 <= a.N) store_bf16x8(a.c + row * a.N + col, f);
        }
      }
    }
  }
  if constexpr (S > 1) {
    if (warp < 2) {
      cluster_wait();
      cluster_sync_all();
    }
  } else {
    __syncthreads();
  }
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, BN);
}

}  // namespace gemm
}  // namespace psdev
