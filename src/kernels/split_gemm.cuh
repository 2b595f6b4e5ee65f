// C[M,N] = X[M,K] * W[N,K]^T for products that are too small to fill the GPU with the large
// tiles of the persistent kernels (pull_gemm.cu).
//
// One 128 x BN output tile per cluster of S CTAs; CTA s of the cluster multiplies the s-th part
// of K.  With S > 1 the partial sums (fp32) are exchanged through distributed shared memory:
// every CTA adds up BN / S columns of all parts, in the order of the parts, and stores them.
// There is no loop over tiles, no counter in global memory, and the first loads are issued before
// the CTA has met at its first barrier, because what bounds these products is a chain of
// latencies: launch, operands from L2 or HBM, a few MMAs, accumulator, store.
//   warp 0      TMA producer; sets up the barriers and starts loading at once;
//   warp 1      allocates tensor memory, issues tcgen05.mma;
//   warps 2..5  epilogue, each its quarter of the accumulator rows.
// Launched with programmatic stream serialization: the prologue runs beside the end of the kernel
// before it.
//
// Two forms.  With more CTAs than SMs about 100 KB of shared memory per CTA, so that two share an
// SM and one loads while the other stores.  Otherwise (DEEP) one CTA has the SM, and a stage holds
// two k-blocks: per stage the ring costs some 300 clocks (commit, barrier, producer) whatever it
// carries, and 128 columns of K make up for them.  The issuer of the deep form touches no mbarrier
// (see wait_ready).  1024 x 1024 x 4096 with BN = 64 / 128 20.9 / 24.5 us shallow, 16.5 / 18.2
// deep; what is left is the loads, 70 bytes per clock and SM.
//
// Measured, us (this kernel / the persistent 128 x 256 kernel): 64x256x256 2.8 / 6.5,
// 1024x1024x256 4.1 / 8.4, 1024x1024x1024 6.0 / 11.9, 64x256x4096 8.6 / 23.4 (S = 4).
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

template <int BN, bool DEEP>
struct SplitCfg {
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBlockBytes = kABytes + BN * BK * 2;  // one k-block
  static constexpr int kSub = DEEP ? 2 : 1;                  // k-blocks of a stage
  static constexpr int kStageBytes = kSub * kBlockBytes;
  static constexpr int kStages = BN == 64 ? 4 : 3;
  static constexpr int kPitch = BN + 4;  // floats per row of the exchanged partial sums
  static constexpr int kExchange = BM * kPitch * 4;
  static constexpr int kTiles = kStages * kStageBytes;
  static constexpr int kSmemBytes = (kTiles > kExchange ? kTiles : kExchange) + 1024 /*align*/;
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
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
  using C = SplitCfg<BN, DEEP>;
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
    if (__all_sync(0xffffffffu, ok)) {
#pragma unroll
      for (int c0 = 0; c0 < BN; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + (uint32_t)c0, r);
        tmem_ld_wait();
        if constexpr (S > 1) {
          // (all MMAs have read their operands: the stages' memory is free)
          float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(smem) +
                                                  in_tile * C::kPitch + c0);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            dst[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                 __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
        } else if (row < a.M) {
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
  }
  if constexpr (S > 1) {
    cluster_sync_all();  // every part's sums are in place
    if (warp >= 2) {
      constexpr int kCols = BN / S;
      const int in_tile = (warp & 3) * 32 + lane;
      const long long row = (long long)tm * BM + in_tile;
      const uint32_t mine =
          smem_u32(smem) + (uint32_t)(in_tile * C::kPitch + part * kCols) * 4;
#pragma unroll
      for (int c0 = 0; c0 < kCols; c0 += 8) {
        float4 lo[S], hi[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const uint32_t from = cluster_addr(mine + c0 * 4, s);
          lo[s] = ld_cluster_v4(from);
          hi[s] = ld_cluster_v4(from + 16);
        }
        float f[8] = {};
#pragma unroll
        for (int s = 0; s < S; ++s) {
          f[0] += lo[s].x; f[1] += lo[s].y; f[2] += lo[s].z; f[3] += lo[s].w;
          f[4] += hi[s].x; f[5] += hi[s].y; f[6] += hi[s].z; f[7] += hi[s].w;
        }
        const long long col = (long long)tn * BN + part * kCols + c0;
        if (row < a.M && col + 8 <= a.N) store_bf16x8(a.c + row * a.N + col, f);
      }
    }
    cluster_sync_all();  // nobody leaves while its sums are being read
  } else {
    __syncthreads();
  }
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, BN);
}

}  // namespace gemm
}  // namespace psdev
