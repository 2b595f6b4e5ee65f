// Communication filters: transforms applied to a value buffer before it is pushed and after
// it is pulled.  The reference advertises "user-defined filters for communication
// compression" (README.md:24-25) but ships no filter code; these are the two this package
// provides on the device:
//   * cast / scale  fp32 <-> bf16 with a scale factor (the dense push kernel also applies the
//     same cast and scale while it loads, so this standalone form is for custom pipelines);
//   * int8 block-scale  groups of 256 values share one fp32 scale = max|x| / 127; values are
//     rounded to int8.  4x smaller than fp32 on the wire plus 1.6 % for the scales.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>

#include "ps/device/chain.cuh"
#include "ps/device/psdev.h"

namespace psdev {
extern std::atomic<uint64_t> g_launches;
namespace filt {
constexpr int kGroup = 256;

// bf16 as its bits: a copy of one type keeps them.
using Bf16 = unsigned short;
template <typename To, typename From>
__device__ __forceinline__ To cast_to(From v) {
  if constexpr (sizeof(To) == sizeof(From)) return v;
  else if constexpr (sizeof(To) == 2) return __bfloat16_as_ushort(__float2bfloat16_rn(v));
  else return __bfloat162float(__ushort_as_bfloat16(v));
}

// Eight values per thread and trip (two 16-byte loads, one 16-byte store, or the reverse) when
// both arrays are 16-byte aligned; scalar accesses for the tail and for unaligned arrays.
__global__ void cast_scale_f32_to_bf16(const float* in, __nv_bfloat16* out, long long n, float s) {
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  long long vec = 0;
  if ((((uintptr_t)in | (uintptr_t)out) & 15) == 0) {
    vec = n / 8;
    for (long long v = tid; v < vec; v += nthreads) {
      const float4 a = reinterpret_cast<const float4*>(in)[2 * v];
      const float4 b = reinterpret_cast<const float4*>(in)[2 * v + 1];
      __nv_bfloat162 p0 = __floats2bfloat162_rn(a.x * s, a.y * s);
      __nv_bfloat162 p1 = __floats2bfloat162_rn(a.z * s, a.w * s);
      __nv_bfloat162 p2 = __floats2bfloat162_rn(b.x * s, b.y * s);
      __nv_bfloat162 p3 = __floats2bfloat162_rn(b.z * s, b.w * s);
      uint4 u;
      u.x = *reinterpret_cast<unsigned int*>(&p0);
      u.y = *reinterpret_cast<unsigned int*>(&p1);
      u.z = *reinterpret_cast<unsigned int*>(&p2);
      u.w = *reinterpret_cast<unsigned int*>(&p3);
      reinterpret_cast<uint4*>(out)[v] = u;
    }
  }
  for (long long i = vec * 8 + tid; i < n; i += nthreads) out[i] = __float2bfloat16_rn(in[i] * s);
}
__global__ void cast_scale_bf16_to_f32(const __nv_bfloat16* in, float* out, long long n, float s) {
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  long long vec = 0;
  if ((((uintptr_t)in | (uintptr_t)out) & 15) == 0) {
    vec = n / 8;
    for (long long v = tid; v < vec; v += nthreads) {
      const uint4 u = reinterpret_cast<const uint4*>(in)[v];
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
      const float2 c = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.z));
      const float2 d = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.w));
      reinterpret_cast<float4*>(out)[2 * v] = make_float4(a.x * s, a.y * s, b.x * s, b.y * s);
      reinterpret_cast<float4*>(out)[2 * v + 1] = make_float4(c.x * s, c.y * s, d.x * s, d.y * s);
    }
  }
  for (long long i = vec * 8 + tid; i < n; i += nthreads) out[i] = __bfloat162float(in[i]) * s;
}

// A copy, with a cast where the types differ: what a gradient hook does with a gradient that it may
// not leave where it is, once per parameter.  Short arrays, hundreds of them, are bound by the
// launch, which is why this is a kernel of its own, chained and no larger than the array: a host
// thread takes 1.9 us for it, 2.3 for cast_scale_f32_to_bf16 and 4.05 for cudaMemcpyAsync.  Long
// ones are bound by HBM.  Eight values per thread and trip where both arrays allow it.
constexpr int kCopyThreads = 256;
template <typename From, typename To>
__global__ void __launch_bounds__(kCopyThreads)
    copy_cast(const From* in, To* out, long long n) {
  grid_launch_next();
  grid_wait();
  const long long tid = blockIdx.x * (long long)kCopyThreads + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * kCopyThreads;
  long long vec = 0;
  if ((((uintptr_t)in | (uintptr_t)out) & 15) == 0) {
    vec = n / 8;
    for (long long v = tid; v < vec; v += nthreads) {
      constexpr int kIn = 8 * sizeof(From) / 16, kOut = 8 * sizeof(To) / 16;
      union { uint4 words[kIn]; From values[8]; } from;
      union { uint4 words[kOut]; To values[8]; } to;
#pragma unroll
      for (int j = 0; j < kIn; ++j) from.words[j] = reinterpret_cast<const uint4*>(in)[v * kIn + j];
#pragma unroll
      for (int j = 0; j < 8; ++j) to.values[j] = cast_to<To>(from.values[j]);
#pragma unroll
      for (int j = 0; j < kOut; ++j) reinterpret_cast<uint4*>(out)[v * kOut + j] = to.words[j];
    }
  }
  for (long long i = vec * 8 + tid; i < n; i += nthreads) out[i] = cast_to<To>(in[i]);
}

// One warp per group of 256 values, kPackGroups groups per warp.  Bound by HBM (5 bytes per
// value).  With VEC a lane holds eight neighbours, so a group is one 32-byte load and one 8-byte
// store per lane and both groups are in flight together; the CTAs are small and as many as there
// are groups, since the hardware replaces a drained CTA faster than a loop over a fixed grid
// comes round.  The input is read once and marked to leave L2 first: the codes stay there for
// the push that follows.  25.6 M values: 32.9 us before, 20.5 now.  Arrays without that alignment
// (32 bytes in, 8 out) keep four-byte loads with neighbouring lanes on neighbouring values
// (26.7 us).
constexpr int kPackThreads = 128;
constexpr int kPackGroups = 2;
template <bool VEC>
__global__ void __launch_bounds__(kPackThreads)
    int8_pack(const float* in, signed char* q, float* scales, long long n) {
  grid_launch_next();
  grid_wait();
  const long long ngroups = (n + kGroup - 1) / kGroup;
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)gridDim.x * (kPackThreads / 32) * kPackGroups;
  for (long long g0 = ((blockIdx.x * (long long)kPackThreads + threadIdx.x) >> 5) * kPackGroups;
       g0 < ngroups; g0 += stride) {
    float v[kPackGroups][8];
    auto at = [&](int u, int j) {
      return (g0 + u) * kGroup + (VEC ? lane * 8 + j : j * 32 + lane);
    };
#pragma unroll
    for (int u = 0; u < kPackGroups; ++u) {
      if (VEC && (g0 + u + 1) * kGroup <= n) {
        asm volatile("ld.global.L2::evict_first.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(v[u][0]), "=f"(v[u][1]), "=f"(v[u][2]), "=f"(v[u][3]), "=f"(v[u][4]),
                       "=f"(v[u][5]), "=f"(v[u][6]), "=f"(v[u][7])
                     : "l"(in + at(u, 0)));
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[u][j] = at(u, j) < n ? in[at(u, j)] : 0.f;
      }
    }
#pragma unroll
    for (int u = 0; u < kPackGroups; ++u) {
      if (g0 + u >= ngroups) break;
      float m = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(v[u][j]));
      // floats that are not negative (and not NaN: fmaxf drops it) order as their bits do
      m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
      const float scale = m > 0.f ? m / 127.f : 1.f;
      const float inv = 1.f / scale;
      if (lane == 0) scales[g0 + u] = scale;
      int c[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        c[j] = __float2int_rn(fminf(fmaxf(v[u][j] * inv, -127.f), 127.f));
      if (VEC && (g0 + u + 1) * kGroup <= n) {
        uint2 w;
        w.x = (c[0] & 0xff) | (c[1] & 0xff) << 8 | (c[2] & 0xff) << 16 | (unsigned)c[3] << 24;
        w.y = (c[4] & 0xff) | (c[5] & 0xff) << 8 | (c[6] & 0xff) << 16 | (unsigned)c[7] << 24;
        *reinterpret_cast<uint2*>(q + at(u, 0)) = w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (at(u, j) < n) q[at(u, j)] = (signed char)c[j];
      }
    }
  }
}
__global__ void int8_unpack(const signed char* q, const float* scales, float* out, long long n,
                            int accumulate) {
  // sixteen values per thread and trip (one 16-byte load, four 16-byte stores) when aligned; a
  // vector of 16 never straddles a group of 256
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  long long vec = 0;
  if ((((uintptr_t)q | (uintptr_t)out) & 15) == 0) {
    vec = n / 16;
    for (long long v = tid; v < vec; v += nthreads) {
      const uint4 u = reinterpret_cast<const uint4*>(q)[v];
      const float sc = scales[(v * 16) / kGroup];
      const unsigned int w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float4 o = make_float4((float)(signed char)(w[j] & 0xff) * sc,
                               (float)(signed char)((w[j] >> 8) & 0xff) * sc,
                               (float)(signed char)((w[j] >> 16) & 0xff) * sc,
                               (float)(signed char)((w[j] >> 24) & 0xff) * sc);
        float4* dst = reinterpret_cast<float4*>(out) + 4 * v + j;
        if (accumulate) {
          const float4 p = *dst;
          o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w;
        }
        *dst = o;
      }
    }
  }
  for (long long i = vec * 16 + tid; i < n; i += nthreads) {
    const float v = (float)q[i] * scales[i / kGroup];
    out[i] = accumulate ? out[i] + v : v;
  }
}
}  // namespace filt
}  // namespace psdev

using namespace psdev;

extern "C" {
// dir 0: fp32 -> bf16, dir 1: bf16 -> fp32; out[i] = cast(in[i] * scale)
int psdev_filter_cast(const void* in, void* out, int64_t n, float scale, int dir, void* stream) {
  if (n < 0 || (dir != 0 && dir != 1)) return PSDEV_ERR_ARG;
  if (n == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (dir == 0)
    filt::cast_scale_f32_to_bf16<<<592, 256, 0, s>>>((const float*)in, (__nv_bfloat16*)out, n,
                                                     scale);
  else
    filt::cast_scale_bf16_to_f32<<<592, 256, 0, s>>>((const __nv_bfloat16*)in, (float*)out, n,
                                                     scale);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return (int)cudaGetLastError();
}
// out[i] = in[i], each of PSDEV_F32 or PSDEV_BF16.
int psdev_copy_cast(const void* in, int from, void* out, int to, int64_t n, void* stream) {
  const bool f32_in = from == PSDEV_F32, f32_out = to == PSDEV_F32;
  if (n < 0 || (!f32_in && from != PSDEV_BF16) || (!f32_out && to != PSDEV_BF16))
    return PSDEV_ERR_ARG;
  if (n == 0) return 0;
  const long long ctas = (n + 8 * filt::kCopyThreads - 1) / (8 * filt::kCopyThreads);
  const unsigned grid = (unsigned)(ctas < (1ll << 30) ? ctas : 1ll << 30);
  auto launch = [&](auto* kernel, auto* typed_in, auto* typed_out) {
    return launch_chained(kernel, grid, filt::kCopyThreads, 0, (cudaStream_t)stream, 1, typed_in,
                          typed_out, (long long)n);
  };
  using filt::Bf16;
  const float* in32 = (const float*)in;
  const Bf16* in16 = (const Bf16*)in;
  const int rc = f32_in ? f32_out ? launch(filt::copy_cast<float, float>, in32, (float*)out)
                                  : launch(filt::copy_cast<float, Bf16>, in32, (Bf16*)out)
                        : f32_out ? launch(filt::copy_cast<Bf16, float>, in16, (float*)out)
                                  : launch(filt::copy_cast<Bf16, Bf16>, in16, (Bf16*)out);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}
// fp32 -> int8 values + one fp32 scale per 256 values (scales has ceil(n/256) entries)
int psdev_filter_int8_pack(const float* in, int8_t* q, float* scales, int64_t n, void* stream) {
  if (n < 0) return PSDEV_ERR_ARG;
  if (n == 0) return 0;
  constexpr long long kPerCta = filt::kPackThreads / 32 * filt::kPackGroups * filt::kGroup;
  const long long ctas = (n + kPerCta - 1) / kPerCta;
  const unsigned int grid = (unsigned int)(ctas < (1ll << 30) ? ctas : 1ll << 30);
  const bool vec = ((uintptr_t)in & 31) == 0 && ((uintptr_t)q & 7) == 0;
  auto* kern = vec ? filt::int8_pack<true> : filt::int8_pack<false>;
  const int rc = launch_chained(kern, grid, filt::kPackThreads, 0, (cudaStream_t)stream, 1, in,
                                (signed char*)q, scales, n);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return rc;
}
// out[i] = (accumulate ? out[i] : 0) + q[i] * scales[i / 256]
int psdev_filter_int8_unpack(const int8_t* q, const float* scales, float* out, int64_t n,
                             int accumulate, void* stream) {
  if (n < 0) return PSDEV_ERR_ARG;
  if (n == 0) return 0;
  filt::int8_unpack<<<592, 256, 0, (cudaStream_t)stream>>>((const signed char*)q, scales, out, n,
                                                           accumulate);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return (int)cudaGetLastError();
}
}  // extern "C"
