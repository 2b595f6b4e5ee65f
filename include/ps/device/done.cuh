// The end of a request of one rank, told to the host by the kernel itself.
//
// The host hears of an event behind a kernel 8.7 to 9.2 us after it begins to launch that kernel,
// of a word that the kernel writes to mapped memory as its last act after 7.2 us (1 CTA) to 8.3
// (600).  The CTAs count themselves done; the last one writes the word.  The order is that of this
// GPU (GPU scope): what a request writes is memory of this GPU, and whatever reads it once the host
// has seen the word - a kernel, a copy engine, a peer - reads it through the GPU's L2, where it is
// by then.  (A fence of system scope takes the 1.3 us back: 8.1 to 9.5 us.)  Requests with arrays
// on the host wait for an event, and so does everything that the host orders by events or streams.
#pragma once
#include "ps/device/psdev.h"

namespace psdev {

// Up to so many CTAs count themselves one by one on one address.  (fp32 values pushed and pulled,
// SGD, an event / the word: 500 000 in 489 CTAs 13.5 / 12.5 us, 4 10^6 in 3907 19.7 / 18.9, 1.6
// 10^7 in 15625 61.0 / 59.0, 3.2 10^7 in 31250 108.6 / 106.4, but 2^26 in 65536 216 / 251.)
constexpr long long kDoneCtas = 16384;

struct DoneArgs {
  unsigned int* word;     // NULL: the host waits for an event
  unsigned int* ticket;
  unsigned int value, last;
};

// For a launch of `ctas` CTAs; `done` may be NULL.
inline DoneArgs arm_done(psdev_done_t* done, long long ctas) {
  DoneArgs a{};
  if (!done || ctas < 1 || ctas > kDoneCtas) return a;
  a.word = done->word;
  a.ticket = done->ticket;
  a.value = done->value;
  if (ctas > 1) done->tickets += (unsigned int)ctas;
  a.last = done->tickets;
  done->armed = 1;
  return a;
}

// At the beginning of a kernel: brings its arguments near, so that the end does not wait for them.
// (Kernels that tell nobody are compiled without either: such a read at the end, of a pointer that
// is NULL, takes 0.5 us of a launch, keyed calls one behind the other 4.1 and 4.6 us.  Held in
// registers from here on, the arguments cost occupancy: 3.2 10^7 values 77.6 and 80.5 us.)
__device__ __forceinline__ void expect_done(const DoneArgs& a) {
  asm volatile("" ::"l"(a.word), "r"(a.last));
}

// At its end, by all threads of every CTA.
__device__ __forceinline__ void signal_done(const DoneArgs& a) {
  __syncthreads();
  if (threadIdx.x) return;
  if (gridDim.x > 1) {
    unsigned int before;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                 : "=r"(before) : "l"(a.ticket) : "memory");
    if (before + 1 != a.last) return;
  }
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(a.word), "r"(a.value) : "memory");
}

}  // namespace psdev
