// k_multi_launch.cuh -- the launch of k_gather_m: its shape for a call.
#pragma once

#include "k_gather.cuh"

namespace qob {
namespace gather {

template <typename R, int VM, bool WIDE, int BMODE>
void launch_m(const GatherView& v, int ls, int kper, const void* x, int64_t xes, int64_t xcs, void* y, int64_t yes,
              int64_t ycs, int64_t ncols, typename Cx<R>::T a, typename Cx<R>::T b, cudaStream_t s) {
  using CT = typename Cx<R>::T;
  using ET = typename Ell<R, true>::T;
  using X = typename Multi<R>::X;
  GatherView w = v;
  w.lane_split = ls;
  const size_t ell_bytes = (size_t)v.ell_slots * sizeof(ET);
  w.ell_smem = ell_bytes <= kStageSlotsMax ? 1 : 0;
  const size_t smem = (size_t)v.ngroups * (sizeof(int4) + 16) + (w.ell_smem ? ell_bytes : 0);
  constexpr int NI = flip_block(std::is_same<R, float>::value ? QOB_C64 : QOB_C128, std::is_same<R, DF>::value);
  auto kern = k_gather_m<R, VM, NI, WIDE, BMODE>;
  const int64_t jpb = (int64_t)NI * (kFlipThreads / ls);  // output indices per block
  const unsigned gx = (unsigned)((v.m + jpb - 1) / jpb);
  w.jmul = gx <= 4096 ? chunk_multiplier(gx) : 1;  // block order as launch_j
  const int64_t per_y = (int64_t)kper * ls;
  for (int64_t c0 = 0; c0 < ncols; c0 += (int64_t)65535 * per_y) {  // grid.y limit
    const int64_t nc = std::min<int64_t>(ncols - c0, (int64_t)65535 * per_y);
    launch_kernel(v.pdl != 0, kern, dim3(gx, (unsigned)((nc + per_y - 1) / per_y)), kFlipThreads, smem, s, w,
                  (const void*)((const X*)x + c0 * xcs), xes, xcs, (CT*)y + c0 * ycs, yes, ycs, (int)nc, kper, a, b);
    QOB_LAUNCHED();
  }
}

template <typename R, int VM>
void launch_multi(const GatherView& v, const void* x, int64_t xes, int64_t xcs, void* y, int64_t yes, int64_t ycs,
                  int64_t ncols, c128 alpha, c128 beta, cudaStream_t s) {
  using S = decltype(Cx<R>::T::x);
  typename Cx<R>::T a, b;
  a.x = (S)alpha.re;
  a.y = (S)alpha.im;
  b.x = (S)beta.re;
  b.y = (S)beta.im;
  const int64_t xsz = sizeof(typename In<R>::T), ysz = sizeof(typename Cx<R>::T);
  // 32-byte loads and stores: contiguous vectors that start on 32 bytes
  const bool wide = xes == 1 && yes == 1 && (((uintptr_t)x | (uintptr_t)y) & 31) == 0 &&
                    (ncols == 1 || (xcs * xsz % 32 == 0 && ycs * ysz % 32 == 0));
  // Vectors per warp.  Vectors across lanes keep more of a warp's lanes on the same
  // groups; contiguous vectors stay at 8 (16 in ComplexF64), where 32 / ls lanes
  // still read whole 128-byte lines, and give up a tenth of the lanes at most.  14
  // spins on 64 kets, ls = 1 / 8 / 16 / 32: ComplexF64 58.4 / - / 51.2 / 49.2 us,
  // ComplexF32 13.3 / 12.7 / 13.6 / 17.0; 7 kets, ComplexF64, 1 / 8: 9.3 / 10.8.
  int ls = 1;
  if (xes == 1 && yes == 1) {
    ls = std::is_same<R, double>::value ? 32 : 8;
    while (ls > 1 && (ncols + ls - 1) / ls * ls * 10 > ncols * 11) ls >>= 1;
  } else {
    while (ls < 32 && ls < ncols) ls *= 2;
  }
  // Vector sets per block: the group look-up then serves several, while the grid
  // keeps about seven blocks per SM (16 spins on 51 kets, ComplexF32, 1 / 2 / 3
  // sets: 39 / 36.5 / 35.2 us; 16 spins on 40, double-float, 1 / 2 / 4: 76 / 70.6 /
  // 67.6).  The FP64 form is bound by its pipe and loses balance (49.2 / 52.6).
  int kper = 1;
  if (!std::is_same<R, double>::value) {
    constexpr int NI = flip_block(std::is_same<R, float>::value ? QOB_C64 : QOB_C128, std::is_same<R, DF>::value);
    const int64_t blocks = (v.m * ls / (NI * kFlipThreads) + 1) * ((ncols + ls - 1) / ls);
    kper = (int)std::max<int64_t>(1, std::min<int64_t>(std::is_same<R, float>::value ? 3 : 4, blocks / (7 * current_sms()) + 1));
  }
#define QOB_M_CALL(W, B) launch_m<R, VM, W, B>(v, ls, kper, x, xes, xcs, y, yes, ycs, ncols, a, b, s)
  if (is_zero(beta))
    wide ? QOB_M_CALL(true, 0) : QOB_M_CALL(false, 0);
  else if (beta.im == 0.0)
    wide ? QOB_M_CALL(true, 3) : QOB_M_CALL(false, 3);
  else
    wide ? QOB_M_CALL(true, 2) : QOB_M_CALL(false, 2);
#undef QOB_M_CALL
}

}  // namespace gather
}  // namespace qob
