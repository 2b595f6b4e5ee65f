// Dense push / pull of a job with one rank: the server update without any exchange.
//
// With one rank the worker's gradients, the server's fp32 master weights and state, and the
// pulled weights all live on this GPU, block ownership is the identity, and nobody has to be
// met.  What remains is a pass over memory, bound by HBM, so this kernel is laid out for that
// alone:
//   * eight values per thread: one 32-byte access per fp32 array (256-bit loads and stores of
//     sm_100), 16 bytes for bf16, 8 for int8;
//   * one tile of 128 x 8 values per CTA and as many CTAs as tiles, not a persistent grid: the
//     hardware keeps ~16 small CTAs per SM and replaces each as it drains.  Measured on
//     64 Mi values: SGD fp32 (16 bytes per value) 162 us against 187 us for the best persistent
//     grid, Adam with bf16 gradients and weights (28 bytes per value) 300 against 323 us; a
//     device copy of the same bytes takes 164 and 287 us;
//   * gradients are read where the caller has them and new weights are stored where the caller
//     wants them (besides the tensor's own weight buffer), so a request on arrays outside the
//     arena costs no copy before or after the kernel;
//   * several pieces of one tensor, each with its own gradient array, go out in one launch; the
//     list travels in the kernel's parameters.
#pragma once
#include <type_traits>

#include "ps/device/chain.cuh"
#include "ps/device/done.cuh"
#include "ps/device/push_pull.cuh"

namespace psdev {

constexpr int kLocalThreads = 128;
constexpr int kLocalVec = 8;
constexpr int kLocalTile = kLocalThreads * kLocalVec;
constexpr int kLocalMaxSegs = PSDEV_MAX_LOCAL_SEGS;

struct LocalArgs {
  const char* grad;    // gradient of element 0 of the table (arena)
  const char* src;     // the caller's gradients, element `begin` first, or NULL
  char* weight;        // weight buffer of the table (arena)
  char* dst;           // the caller's output, element `begin` first, or NULL
  const float* gscale; // int8 gradients: one scale per 256 values
  float* master;
  float* s1;
  float* s2;
  long long begin, end;
  long long n_valid;   // elements from here on do not exist in src / dst
  psdev_opt_t opt;
  const SchedEntry* sched;  // device-side slice schedule (nseg + 1 entries), or NULL
  int nseg;
  bool wide;           // every fp32 array is aligned to 32 bytes
  bool src_vec, dst_vec;  // the caller's arrays are aligned to eight values
  // checks build only
  void* base;
  int channel;
  unsigned long long grad_off, weight_off, heap_bytes;
  long long n_total, local_len;
};

// Pieces of a table with gradients in arrays of their own.
struct LocalSeg {
  long long begin, end;  // element range, multiples of 8
  const char* src;       // gradient of element `begin`; NULL: the table's gradient buffer
  int dtype;             // of src: PSDEV_F32 or PSDEV_BF16
  int tile_begin;        // number of its first tile
  long long n_valid;     // elements from here on are padding: no gradient
};
struct LocalSegs {
  int n, tiles;
  LocalSeg seg[kLocalMaxSegs];
};
struct NoSegs {};
struct Told {            // one piece, and the host waits for a word
  DoneArgs done;
};

__device__ __forceinline__ void load8(const float* p, float* f, bool wide) {
  if (wide) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]),
                   "=f"(f[6]), "=f"(f[7])
                 : "l"(p)
                 : "memory");
  } else {
    load_f32<8>(p, f);
  }
}
__device__ __forceinline__ void store8(float* p, const float* f, bool wide) {
  if (wide) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(f[0]),
                 "f"(f[1]), "f"(f[2]), "f"(f[3]), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7])
                 : "memory");
  } else {
    store_f32<8>(p, f);
  }
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f, bool) {
  VecOf<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(p), f);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float* f, bool) {
  store_out<__nv_bfloat16, 8>(p, f);
}
__device__ __forceinline__ void load8(const signed char* p, float* f, bool) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    f[b] = (float)(signed char)((u.x >> (8 * b)) & 0xff);
    f[4 + b] = (float)(signed char)((u.y >> (8 * b)) & 0xff);
  }
}
__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f32(signed char v) { return (float)v; }
__device__ __forceinline__ void from_f32(float* p, float v) { *p = v; }
__device__ __forceinline__ void from_f32(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// Eight gradients starting at p, of which `count` exist; `vec`: p is aligned to all eight.
template <typename T>
__device__ __forceinline__ void load_part(const T* p, long long count, bool vec, float* f) {
  if (vec && count >= kLocalVec) {
    load8(p, f, true);
  } else {
#pragma unroll
    for (int q = 0; q < kLocalVec; ++q) f[q] = q < count ? to_f32(p[q]) : 0.f;
  }
}

// Elements [lo, hi) one by one, from and to the table's own buffers: the part of a vector that
// belongs to a slice which starts or ends inside it (the rest is another CTA's).
template <typename GT, typename OT, class Opt, bool REDUCE, bool BCAST>
__device__ __forceinline__ void update_part(const LocalArgs& a, long long lo, long long hi) {
#pragma unroll 1
  for (long long e = lo; e < hi; ++e) {
    float w = a.master[e];
    if constexpr (REDUCE) {
      float g = to_f32(reinterpret_cast<const GT*>(a.grad)[e]);
      float m = Opt::kStates >= 1 ? a.s1[e] : 0.f;
      float v = Opt::kStates >= 2 ? a.s2[e] : 0.f;
      if constexpr (sizeof(GT) == 1) g *= a.gscale[e / kInt8Group];
      Opt::apply(w, g * a.opt.scale, m, v, a.opt);
      a.master[e] = w;
      if (Opt::kStates >= 1) a.s1[e] = m;
      if (Opt::kStates >= 2) a.s2[e] = v;
    }
    if constexpr (BCAST) from_f32(reinterpret_cast<OT*>(a.weight) + e, w);
  }
}

// (two states per value: 56 registers, so that nine CTAs fit an SM)
template <typename GT, typename OT, class Opt, bool REDUCE, bool BCAST, typename Segs>
__global__ void __launch_bounds__(kLocalThreads, Opt::kStates >= 2 ? 9 : 0)
    local_update_kernel(const __grid_constant__ LocalArgs a, const __grid_constant__ Segs segs) {
  constexpr bool kSegs = std::is_same<Segs, LocalSegs>::value;
  constexpr bool kTold = std::is_same<Segs, Told>::value;
  grid_launch_next();
  if constexpr (kTold) expect_done(segs.done);
  grid_wait();
  long long ntiles;
  if constexpr (kSegs) ntiles = segs.tiles;
  else if (a.sched) ntiles = a.sched[a.nseg].tile_begin;
  else ntiles = a.end > a.begin ? (a.end - 1) / kLocalTile - a.begin / kLocalTile + 1 : 0;
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    long long begin = a.begin, end = a.end, tl = t, n_valid = a.n_valid;
    const char* src = a.src;
    int dtype = 0;
    if constexpr (kSegs) {
      int lo = 0, hi = segs.n - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (segs.seg[mid].tile_begin <= t) lo = mid; else hi = mid - 1;
      }
      begin = segs.seg[lo].begin; end = segs.seg[lo].end;
      src = segs.seg[lo].src; dtype = segs.seg[lo].dtype; n_valid = segs.seg[lo].n_valid;
      tl = t - segs.seg[lo].tile_begin;
    } else if (a.sched) {
      int lo = 0, hi = a.nseg - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.sched[mid].tile_begin <= t) lo = mid; else hi = mid - 1;
      }
      begin = a.sched[lo].begin; end = a.sched[lo].end;
      tl = t - a.sched[lo].tile_begin;
    }
    const long long i = (begin / kLocalTile + tl) * kLocalTile + threadIdx.x * kLocalVec;
    if (i + kLocalVec <= begin || i >= end) continue;
#ifdef PSDEV_CHECKS
    if (i + kLocalVec > a.n_total || i + kLocalVec > a.local_len ||
        (a.heap_bytes &&
         (a.grad_off + (unsigned long long)(i + kLocalVec) * sizeof(GT) > a.heap_bytes ||
          a.weight_off + (unsigned long long)(i + kLocalVec) * sizeof(OT) > a.heap_bytes))) {
      atomicMin(&ctrl_of(a.base)->status[a.channel], (int)PSDEV_ERR_BOUNDS);
      continue;
    }
#endif
    if constexpr (!kSegs) {
      if (i < begin || i + kLocalVec > end) {  // (slices of the device's list: any boundaries)
        update_part<GT, OT, Opt, REDUCE, BCAST>(a, i < begin ? begin : i,
                                                i + kLocalVec < end ? i + kLocalVec : end);
        continue;
      }
    }
    float w[kLocalVec];
    if constexpr (REDUCE) {
      float g[kLocalVec], m[kLocalVec], v[kLocalVec];
      if (src == nullptr) {
        load8(reinterpret_cast<const GT*>(a.grad) + i, g, a.wide);
      } else if constexpr (kSegs) {
        if (dtype == PSDEV_F32) {
          const float* p = reinterpret_cast<const float*>(src) + (i - begin);
          load_part(p, n_valid - i, ((uintptr_t)src & 31) == 0, g);
        } else {
          const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(src) + (i - begin);
          load_part(p, n_valid - i, ((uintptr_t)src & 15) == 0, g);
        }
        if constexpr (sizeof(GT) == 2) {
          // the gradient travels in bf16 whatever it was computed in
#pragma unroll
          for (int q = 0; q < kLocalVec; ++q)
            g[q] = __bfloat162float(__float2bfloat16_rn(g[q]));
        }
      } else {
        load_part(reinterpret_cast<const GT*>(src) + (i - begin), n_valid - i, a.src_vec, g);
      }
      load8(a.master + i, w, a.wide);
      if constexpr (Opt::kStates >= 1) load8(a.s1 + i, m, a.wide);
      if constexpr (Opt::kStates >= 2) load8(a.s2 + i, v, a.wide);
      if constexpr (sizeof(GT) == 1) {
        const float sc = a.gscale[i / kInt8Group];  // a vector never straddles a group
#pragma unroll
        for (int q = 0; q < kLocalVec; ++q) g[q] *= sc;
      }
#pragma unroll
      for (int q = 0; q < kLocalVec; ++q) {
        float mm = Opt::kStates >= 1 ? m[q] : 0.f;
        float vv = Opt::kStates >= 2 ? v[q] : 0.f;
        Opt::apply(w[q], g[q] * a.opt.scale, mm, vv, a.opt);
        if (Opt::kStates >= 1) m[q] = mm;
        if (Opt::kStates >= 2) v[q] = vv;
      }
      store8(a.master + i, w, a.wide);
      if constexpr (Opt::kStates >= 1) store8(a.s1 + i, m, a.wide);
      if constexpr (Opt::kStates >= 2) store8(a.s2 + i, v, a.wide);
    } else {
      load8(a.master + i, w, a.wide);
    }
    if constexpr (BCAST) {
      store8(reinterpret_cast<OT*>(a.weight) + i, w, a.wide);
      if constexpr (!kSegs) {
        if (a.dst) {
          OT* p = reinterpret_cast<OT*>(a.dst) + (i - begin);
          if (a.dst_vec && i + kLocalVec <= n_valid) {
            store8(p, w, true);
          } else {
#pragma unroll
            for (int q = 0; q < kLocalVec; ++q)
              if (i + q < n_valid) from_f32(p + q, w[q]);
          }
        }
      }
    }
  }
  if constexpr (kTold) signal_done(segs.done);
}

}  // namespace psdev
