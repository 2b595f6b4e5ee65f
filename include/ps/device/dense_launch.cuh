// Launch helpers of the fused dense kernel: pick the kernel variant for the world size and the
// path (peer accesses or NVSwitch multicast), size the grid, run the device-side slice schedule
// when the launch carries several slices.  Shared by the library's own instantiations
// (src/kernels/dense_inst.inl) and by user-defined server handles (user_handle.cuh).
#pragma once
#include <cuda_runtime.h>

#include "ps/device/chain.cuh"
#include "ps/device/local_update.cuh"
#include "ps/device/push_pull_ll.cuh"

extern "C" void psdev_count_launch(void);

namespace psdev {
void launch_p3_schedule(const long long* segs, int nseg, long long blk, int world, int rank,
                        long long tiles_per_blk, SchedEntry* out, cudaStream_t s);

template <typename GT, typename OT, class Opt, bool RED, bool BC, int WMAX>
inline int launch_w(DenseArgs a, int num_ctas, cudaStream_t s) {
  constexpr int tile = DenseTile<GT, OT, RED, WMAX>::kElems;
  a.tiles_per_blk = (a.blk + tile - 1) / tile;
  const long long ntiles = a.n_owned * a.tiles_per_blk;
  int ctas = num_ctas > 0 ? num_ctas : 2 * 148;
  if (a.nseg > 0) {
    // device-side schedule: slices ordered by priority, tiles numbered across slices
    launch_p3_schedule(a.segs_in, a.nseg, a.blk, a.world, a.rank, a.tiles_per_blk,
                       const_cast<SchedEntry*>(a.sched), s);
  } else if (ntiles < ctas) {
    ctas = ntiles > 0 ? (int)ntiles : 1;
  }
  dense_kernel<GT, OT, Opt, RED, BC, WMAX><<<ctas, kDenseThreads, 0, s>>>(a);
  psdev_count_launch();
  return (int)cudaGetLastError();
}

template <typename GT, typename OT, class Opt, bool RED, bool BC>
inline int launch_mc(DenseArgs a, int num_ctas, cudaStream_t s) {
  constexpr int tile = DenseTile<GT, OT, RED, 1>::kElems;
  a.tiles_per_blk = (a.blk + tile - 1) / tile;
  const long long ntiles = a.n_owned * a.tiles_per_blk;
  int ctas = num_ctas > 0 ? num_ctas : 2 * 148;
  if (a.nseg > 0) {
    launch_p3_schedule(a.segs_in, a.nseg, a.blk, a.world, a.rank, a.tiles_per_blk,
                       const_cast<SchedEntry*>(a.sched), s);
  } else if (ntiles < ctas) {
    ctas = ntiles > 0 ? (int)ntiles : 1;
  }
  dense_kernel<GT, OT, Opt, RED, BC, 1, true><<<ctas, kDenseThreads, 0, s>>>(a);
  psdev_count_launch();
  return (int)cudaGetLastError();
}

// One rank.  As many CTAs as tiles unless the caller limits them (local_update.cuh says why).
template <typename GT, typename OT, class Opt, bool RED, bool BC>
inline int launch_local(const DenseArgs& d, int num_ctas, cudaStream_t s) {
  LocalArgs a{};
  char* base = static_cast<char*>(d.base[0]);
  a.grad = base + d.grad_off;
  a.weight = base + d.weight_off;
  a.src = static_cast<const char*>(d.src);
  a.dst = static_cast<char*>(d.dst);
  a.gscale = reinterpret_cast<const float*>(base + d.gscale_off);
  a.master = d.master;
  a.s1 = d.s1;
  a.s2 = d.s2;
  a.begin = d.begin;
  a.end = d.end;
  a.n_valid = d.n_valid;
  a.opt = d.opt;
  uintptr_t bits = (uintptr_t)d.master;
  if (Opt::kStates >= 1) bits |= (uintptr_t)d.s1;
  if (Opt::kStates >= 2) bits |= (uintptr_t)d.s2;
  if (sizeof(GT) == 4) bits |= (uintptr_t)a.grad;
  if (sizeof(OT) == 4) bits |= (uintptr_t)a.weight;
  a.wide = (bits & 31) == 0;
  a.src_vec = ((uintptr_t)d.src & (sizeof(GT) * kLocalVec - 1)) == 0;
  a.dst_vec = ((uintptr_t)d.dst & (sizeof(OT) * kLocalVec - 1)) == 0;
  a.base = base;
  a.channel = d.channel;
  a.grad_off = d.grad_off;
  a.weight_off = d.weight_off;
  a.heap_bytes = d.heap_bytes;
  a.n_total = d.n_total;
  a.local_len = d.local_len;
  if (d.nlsegs > 0) {
    if constexpr (RED && sizeof(GT) > 1) {
      LocalSegs list{};
      for (int at = 0; at < d.nlsegs; at += list.n) {
        list.n = list.tiles = 0;
        for (; at + list.n < d.nlsegs && list.n < kLocalMaxSegs; ++list.n) {
          const psdev_seg_t& in = d.lsegs[at + list.n];
          LocalSeg& out = list.seg[list.n];
          out.begin = in.begin;
          out.end = in.end;
          out.src = static_cast<const char*>(in.src);
          out.dtype = in.dtype;
          out.n_valid = in.n_valid;
          out.tile_begin = list.tiles;
          list.tiles += (int)((in.end - 1) / kLocalTile - in.begin / kLocalTile + 1);
        }
        const int ctas = num_ctas > 0 && num_ctas < list.tiles ? num_ctas : list.tiles;
        const int rc = launch_chained(local_update_kernel<GT, OT, Opt, RED, BC, LocalSegs>,
                                      (unsigned)ctas, kLocalThreads, 0, s, 1, a, list);
        psdev_count_launch();
        if (rc) return rc;
      }
      return 0;
    }
    return PSDEV_ERR_UNSUPPORTED;
  }
  long long ntiles;
  if (d.nseg > 0) {
    // the number of tiles is known on the device only; every slice may start inside a tile
    launch_p3_schedule(d.segs_in, d.nseg, kLocalTile, 1, 0, 1, const_cast<SchedEntry*>(d.sched), s);
    a.sched = d.sched;
    a.nseg = d.nseg;
    ntiles = d.end / kLocalTile + d.nseg + 1;
  } else {
    ntiles = d.end > d.begin ? (d.end - 1) / kLocalTile - d.begin / kLocalTile + 1 : 1;
  }
  const long long ctas = num_ctas > 0 && num_ctas < ntiles ? num_ctas : ntiles;
  const unsigned grid = (unsigned)(ctas < (1ll << 30) ? ctas : 1ll << 30);
  // (int8 gradients come through a table of their own, not as requests)
  if constexpr (sizeof(GT) > 1) {
    const Told told{arm_done(d.done, ctas)};
    if (told.done.word) {
      const int rc = launch_chained(local_update_kernel<GT, OT, Opt, RED, BC, Told>, grid,
                                    kLocalThreads, 0, s, 1, a, told);
      psdev_count_launch();
      return rc;
    }
  }
  const int rc = launch_chained(local_update_kernel<GT, OT, Opt, RED, BC, NoSegs>, grid,
                                kLocalThreads, 0, s, 1, a, NoSegs{});
  psdev_count_launch();
  return rc;
}

template <typename GT, typename OT, class Opt, bool RED, bool BC>
inline int launch(const DenseArgs& a, int ctas, cudaStream_t s) {
  if (a.mc_base && a.world > 1) return launch_mc<GT, OT, Opt, RED, BC>(a, ctas, s);
  if (a.world == 1) return launch_local<GT, OT, Opt, RED, BC>(a, ctas, s);
  if (a.world == 2) return launch_w<GT, OT, Opt, RED, BC, 2>(a, ctas, s);
  if (a.world <= 4) return launch_w<GT, OT, Opt, RED, BC, 4>(a, ctas, s);
  return launch_w<GT, OT, Opt, RED, BC, 8>(a, ctas, s);
}


template <typename GT, typename OT, class Opt>
inline int launch_ll(const LLArgs& a, cudaStream_t s) {
  const long long m = a.end - a.begin;
  long long ctas = (m + kLLThreads - 1) / kLLThreads;
  if (ctas > 148) ctas = 148;  // every CTA of every rank must get to run: stay within one wave
  if (ctas < 1) ctas = 1;
  dense_ll_kernel<GT, OT, Opt><<<(int)ctas, kLLThreads, 0, s>>>(a);
  psdev_count_launch();
  return (int)cudaGetLastError();
}

}  // namespace psdev
