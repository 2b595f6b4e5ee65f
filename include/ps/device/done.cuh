// The end of a small dense request of one rank, told to the host by the kernel itself.
//
// The CTAs count themselves done; the last one writes a word in mapped memory.  What a request has
// written may be read by anybody whom the host tells that it is done - a kernel of another stream,
// a copy, a peer, the host itself - with no event in between, so the word is released at system
// scope: the other CTAs' writes come before their counts at GPU scope, and those before the last
// one's fence.  The fence takes 1.2 us of what the word saves against an event: a launch is known
// to be done after 9.1 us with one CTA and 9.7 to 9.9 with more (7.8 and 8.5 to 8.8 behind a fence
// of GPU scope, which would order nothing for a reader that the host starts), by an event after
// 9.1 to 9.5.  In whole requests the word gains more (kDoneCtas).
#pragma once
#include "ps/device/psdev.h"

namespace psdev {

// Up to so many CTAs a request has a word.  Waited for from Python, us, fp32 SGD / bf16 momentum,
// pushed and pulled, by an event and by the word: 1024 values (1 CTA) 12.3 / 12.5 and 11.4 / 11.7,
// 100 000 (98) 12.4 / 12.5 and 12.0 / 12.1, 200 000 (196) 12.7 / 12.8 and 12.5 / 12.6, 500 000
// (489) 13.3 / 13.4 and 13.2 / 13.3, 2 10^6 (1954) 16.1 / 16.5 and 16.2 / 17.1; pushed alone 2
// 10^6 13.8 / 15.1 and 14.1 / 15.9.  (Keyed requests gained nothing: 50 001 rows 14.8 and 14.9,
// with lengths 30.4 and 31.2.)
constexpr long long kDoneCtas = 128;

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
// is NULL, takes 0.5 us of a launch.)
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
  asm volatile("fence.acq_rel.sys;" ::: "memory");
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(a.word), "r"(a.value) : "memory");
}

}  // namespace psdev
