// fft_line.h -- what the FFT passes are called with (fft_line.cuh, fft.cu).
#pragma once

#include "qob_internal.h"

namespace qob {

// What a final pass is called with.
struct FftOut {
  void* y;
  int64_t yes, ycs;
  c128 alpha, beta;
  const GatherPlan* add;  // a diagonal term of the same sum (kDiag), on the vectors at add_x
  const void* add_x;
  int64_t add_xes, add_xcs;
};

inline int log2_of(int64_t n) {
  int l = 0;
  while ((int64_t(1) << l) < n) ++l;
  return l;
}

// Few long lines are spread over many blocks each.
inline bool four_step(const FftAxis& ax, int64_t lines, int sms) {
  return ax.n1 > 0 && lines < sms && lines * ax.n2 <= INT32_MAX;
}

// One axis of an FFT plan, or two transforms of one axis with a diagonal operator between
// (fft_f64.cu, fft_f32.cu, fft_df.cu).
template <typename R>
void fft_axis(const FftAxis& ax, int64_t len, const void* x, int64_t xes, int64_t xcs, const FftOut& o, int64_t ncols,
              void* scratch, int sms, cudaStream_t s);
template <typename R>
void fft_turn(const FftAxis& ax, const FftAxis& bx, const GatherPlan& d, const void* mid, int64_t len, const void* x,
              int64_t xes, int64_t xcs, const FftOut& o, int64_t ncols, void* scratch, void* scratch2, int sms,
              cudaStream_t s);

}  // namespace qob
