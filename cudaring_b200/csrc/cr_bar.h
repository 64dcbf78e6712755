// Word of the grid barrier in the multi-step kernels: the arrivals of one
// launch in the low 32 bits and, above them, two 16-bit counts of the arrivals
// that asked for the loop to end, one for the launch's even and one for its odd
// barriers.  The poll that sees barrier k complete brings its stop decision
// too, and every CTA gets the same one: when a CTA polls barrier k, the others
// can be at barrier k + 1 at most, whose stops go to the other count.  (With
// one count, a fast CTA's stop at k + 1 could end a slow one's loop at k, and
// k + 1 then waited for an arrival that never came.)  Every launch starts on a
// word of zeros and a stop ends it, so no count carries: a launch makes at most
// 2 x 64 barriers of fewer than 2^16 CTAs.
#pragma once

#ifdef __CUDACC__
#define CR_BAR_HD __host__ __device__ __forceinline__
#else
#define CR_BAR_HD inline
#endif

namespace cr {

CR_BAR_HD int bar_stop_shift(int k) { return 32 + 16 * (k & 1); }
// What a CTA adds to the word when it arrives at barrier k (from 0).
CR_BAR_HD unsigned long long bar_arrival(int k, bool stop) {
  return 1ull | (stop ? 1ull << bar_stop_shift(k) : 0ull);
}
CR_BAR_HD bool bar_complete(unsigned long long word, int k, unsigned ctas) {
  return (unsigned)word >= (unsigned)(k + 1) * ctas;
}
// Of a word that shows barrier k complete: whether some CTA asked to stop there.
CR_BAR_HD bool bar_stopped(unsigned long long word, int k) { return (word >> bar_stop_shift(k) & 0xffffull) != 0; }

}  // namespace cr
