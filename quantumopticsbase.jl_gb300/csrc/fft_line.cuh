// fft_line.cuh -- the kernels of the FFT passes; each form is compiled in a file of its
// own (fft_f64.cu, fft_f32.cu, fft_df.cu).
#pragma once

#include <cmath>
#include <type_traits>

#include "fft_line.h"
#include "k_gather.cuh"  // double-float helpers

namespace qob {
namespace {

using gather::DF;

// Element types per precision: G in memory (vectors, alpha, beta), S for the
// arithmetic (shared-memory lines, twiddles, phases).  The double-float form
// (ComplexF64 data) computes on (re hi, re lo, im hi, im lo) quadruples.
template <typename R>
struct FT;
template <>
struct FT<double> {
  using G = double2;
  using S = double2;
  static __device__ __forceinline__ S in(G g) { return g; }
};
template <>
struct FT<float> {
  using G = float2;
  using S = float2;
  static __device__ __forceinline__ S in(G g) { return g; }
};
template <>
struct FT<DF> {
  using G = double2;
  using S = float4;
  static __device__ __forceinline__ S in(G g) {
    const float2 a = gather::ff_split(g.x), b = gather::ff_split(g.y);
    return make_float4(a.x, a.y, b.x, b.y);
  }
};

// Constants of the butterflies.  FP64: in vector registers, and every sum and
// product an fma with them, which this pipe issues at 1.89 lanes a clock for 1.60
// of an addition, a multiplication or a constant operand (the same numbers).
template <typename R>
struct Cs {
  R one, s, r, nz;  // 1, the transform's sign, sqrt(1/2), -0
  __device__ __forceinline__ explicit Cs(int sign)
      : one(gather::in_register((R)1)),
        s(gather::in_register((R)sign)),
        r(gather::in_register((R)0.70710678118654752440)),
        nz(gather::in_register(-(R)0)) {}
};
template <>
struct Cs<DF> {
  float s;
  float2 r;
  __device__ __forceinline__ explicit Cs(int sign) : s((float)sign), r(make_float2(0.70710677f, 1.21016175e-8f)) {}
};

// u * c + v, one rounding
__device__ __forceinline__ double axpy(double u, double c, double v) { return __fma_rn(u, c, v); }
__device__ __forceinline__ float axpy(float u, float c, float v) { return __fmaf_rn(u, c, v); }
__device__ __forceinline__ double2 cm(double2 a, double2 b, double nz) {
  return make_double2(__fma_rn(a.x, b.x, -__fma_rn(a.y, b.y, nz)), __fma_rn(a.x, b.y, __fma_rn(a.y, b.x, nz)));
}
__device__ __forceinline__ double2 cm(double2 a, double2 b, const Cs<double>& c) { return cm(a, b, c.nz); }
__device__ __forceinline__ float2 cm(float2 a, float2 b, const Cs<float>&) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float4 cm(float4 a, float4 b, const Cs<DF>&) {
  const float2 ar = make_float2(a.x, a.y), ai = make_float2(a.z, a.w);
  const float2 br = make_float2(b.x, b.y), bi = make_float2(b.z, b.w);
  const float2 re = gather::ff_add(gather::ff_mul(ar, br), gather::ff_neg(gather::ff_mul(ai, bi)));
  const float2 im = gather::ff_add(gather::ff_mul(ar, bi), gather::ff_mul(ai, br));
  return make_float4(re.x, re.y, im.x, im.y);
}
// u + v, u - v
template <typename R, typename CT>
__device__ __forceinline__ CT cadd(CT u, CT v, const Cs<R>& c) {
  return CT{axpy(v.x, c.one, u.x), axpy(v.y, c.one, u.y)};
}
template <typename R, typename CT>
__device__ __forceinline__ CT csub(CT u, CT v, const Cs<R>& c) {
  return CT{axpy(v.x, -c.one, u.x), axpy(v.y, -c.one, u.y)};
}
__device__ __forceinline__ float4 cadd(float4 a, float4 b, const Cs<DF>&) {
  const float2 re = gather::ff_add(make_float2(a.x, a.y), make_float2(b.x, b.y));
  const float2 im = gather::ff_add(make_float2(a.z, a.w), make_float2(b.z, b.w));
  return make_float4(re.x, re.y, im.x, im.y);
}
__device__ __forceinline__ float4 csub(float4 a, float4 b, const Cs<DF>& c) {
  return cadd(a, make_float4(-b.x, -b.y, -b.z, -b.w), c);
}
// u + i s v, u - i s v (s the transform's sign)
template <typename R, typename CT>
__device__ __forceinline__ CT cadd_i(CT u, CT v, const Cs<R>& c) {
  return CT{axpy(v.y, -c.s, u.x), axpy(v.x, c.s, u.y)};
}
template <typename R, typename CT>
__device__ __forceinline__ CT csub_i(CT u, CT v, const Cs<R>& c) {
  return CT{axpy(v.y, c.s, u.x), axpy(v.x, -c.s, u.y)};
}
__device__ __forceinline__ float4 cadd_i(float4 u, float4 v, const Cs<DF>& c) {
  return cadd(u, make_float4(-c.s * v.z, -c.s * v.w, c.s * v.x, c.s * v.y), c);
}
__device__ __forceinline__ float4 csub_i(float4 u, float4 v, const Cs<DF>& c) {
  return cadd(u, make_float4(c.s * v.z, c.s * v.w, -c.s * v.x, -c.s * v.y), c);
}
// v = sqrt(1/2) o: e + v, e - v (one rounding each outside the double-float form)
template <typename R, typename CT>
__device__ __forceinline__ void half_turns(CT e, CT o, const Cs<R>& c, CT& plus, CT& minus) {
  plus = CT{axpy(o.x, c.r, e.x), axpy(o.y, c.r, e.y)};
  minus = CT{axpy(o.x, -c.r, e.x), axpy(o.y, -c.r, e.y)};
}
__device__ __forceinline__ void half_turns(float4 e, float4 o, const Cs<DF>& c, float4& plus, float4& minus) {
  const float2 re = gather::ff_mul(make_float2(o.x, o.y), c.r), im = gather::ff_mul(make_float2(o.z, o.w), c.r);
  const float4 v = make_float4(re.x, re.y, im.x, im.y);
  plus = cadd(e, v, c);
  minus = csub(e, v, c);
}

template <typename R, typename CT>
__device__ __forceinline__ void dft2(CT& a, CT& b, const Cs<R>& c) {
  const CT d = csub(a, b, c);
  a = cadd(a, b, c);
  b = d;
}
// length-4 transform in place, natural order
template <typename R, typename CT>
__device__ __forceinline__ void dft4(CT& a0, CT& a1, CT& a2, CT& a3, const Cs<R>& c) {
  dft2(a0, a2, c);
  dft2(a1, a3, c);
  const CT y1 = cadd_i(a2, a3, c), y3 = csub_i(a2, a3, c);
  const CT y0 = cadd(a0, a1, c), y2 = csub(a0, a1, c);
  a0 = y0;
  a1 = y1;
  a2 = y2;
  a3 = y3;
}
// length-E transform in place, natural order: 4, 16, 52 operations
template <typename R, typename CT>
__device__ __forceinline__ void dft(CT (&u)[2], const Cs<R>& c) {
  dft2(u[0], u[1], c);
}
template <typename R, typename CT>
__device__ __forceinline__ void dft(CT (&u)[4], const Cs<R>& c) {
  dft4(u[0], u[1], u[2], u[3], c);
}
template <typename R, typename CT>
__device__ __forceinline__ void dft(CT (&u)[8], const Cs<R>& c) {
  dft4(u[0], u[2], u[4], u[6], c);  // e0 .. e3
  dft4(u[1], u[3], u[5], u[7], c);  // o0 .. o3
  const CT e0 = u[0], e1 = u[2], e2 = u[4], e3 = u[6], o0 = u[1], o2 = u[5];
  const CT o1 = cadd_i(u[3], u[3], c);  // (1 + i s) o1
  const CT o3 = csub_i(u[7], u[7], c);  // (1 - i s) o3, the twiddle with its sign turned
  u[0] = cadd(e0, o0, c);
  u[4] = csub(e0, o0, c);
  half_turns(e1, o1, c, u[1], u[5]);
  u[2] = cadd_i(e2, o2, c);
  u[6] = csub_i(e2, o2, c);
  half_turns(e3, o3, c, u[7], u[3]);
}

// Element k of line `line`: the line is (vector c, position p among the len/n
// lines of one vector); p = lo + stride * hi with lo < stride.
__device__ __forceinline__ int64_t line_base(int64_t line, int64_t lines_per_vec, int64_t stride, int64_t n,
                                             int64_t es, int64_t cs) {
  int64_t c, p, lo, hi;
  udivmod(line, lines_per_vec, c, p);
  udivmod(p, stride, hi, lo);
  return c * cs + (lo + hi * stride * n) * es;
}

// What the last pass does with alpha v, v its results times the phases: y = it; y += it (a
// later term of a sum); y = it + beta y; y = it + beta y with a diagonal term of the
// same sum added to v, beta y read where beta is not zero.
enum StoreMode { kPut = 0, kAdd = 1, kAxpby = 2, kDiag = 3 };

// i^q v, exact
__device__ __forceinline__ double turned_sign(double a, bool minus) {
  return __hiloint2double(__double2hiint(a) ^ (minus ? (int)0x80000000 : 0), __double2loint(a));
}
__device__ __forceinline__ float turned_sign(float a, bool minus) { return minus ? -a : a; }
template <typename G>
__device__ __forceinline__ G quarter_turns(G v, int q) {
  const bool odd = q & 1;
  const auto x = odd ? v.y : v.x, y = odd ? v.x : v.y;
  return G{turned_sign(x, q == 1 || q == 2), turned_sign(y, q >= 2)};
}

__device__ __forceinline__ double2 joined(double2 v) { return v; }
__device__ __forceinline__ float2 joined(float2 v) { return v; }
__device__ __forceinline__ double2 joined(float4 v) {
  return make_double2(gather::ff_join(v.x, v.y), gather::ff_join(v.z, v.w));
}

// the arithmetic of the last pass' scalars
template <typename R>
using Out = typename std::conditional<std::is_same<R, DF>::value, double, R>::type;
template <typename R>
__device__ __forceinline__ const Cs<R>& out_consts(const Cs<R>& c) {
  return c;
}
__device__ __forceinline__ Cs<double> out_consts(const Cs<DF>&) { return Cs<double>(1); }

// E results of a thread to y + at(m) * so; quarter: alpha = i^quarter (-1: any other)
template <typename R, int MODE, int E, typename AT>
__device__ __forceinline__ void store(typename FT<R>::G* y, int64_t so, AT at, typename FT<R>::G (&o)[E], int quarter,
                                      typename FT<R>::G alpha, typename FT<R>::G beta, const Cs<Out<R>>& c) {
  alpha.x = gather::in_register(alpha.x);
  alpha.y = gather::in_register(alpha.y);
  beta.x = gather::in_register(beta.x);
  beta.y = gather::in_register(beta.y);
  if (quarter >= 0) {
#pragma unroll
    for (int m = 0; m < E; ++m) o[m] = quarter_turns(o[m], quarter);
  } else {
#pragma unroll
    for (int m = 0; m < E; ++m) o[m] = cm(o[m], alpha, c);
  }
  if constexpr (MODE == kAdd) {
#pragma unroll
    for (int m = 0; m < E; ++m) o[m] = cadd(o[m], y[at(m) * so], c);
  }
  if (MODE == kAxpby || (MODE == kDiag && (beta.x != 0 || beta.y != 0))) {
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const typename FT<R>::G v = y[at(m) * so];
      o[m].x = axpy(v.x, beta.x, axpy(v.y, -beta.y, o[m].x));
      o[m].y = axpy(v.y, beta.x, axpy(v.x, beta.y, o[m].y));
    }
  }
#pragma unroll
  for (int m = 0; m < E; ++m) y[at(m) * so] = o[m];
}

// One pass over lines of n = 2^log2n elements, C = 2^log2c lines a block, E
// elements a thread.
//   kWhole  the whole transform of an axis.
//   kTurn  two of them with a diagonal operator between: the first one's results are where
//     the second one's inputs are wanted, in the same thread.
//   kFirst, kSecond  four-step form (Bailey 1990) of a transform of length
//     N = n1 n2, element j = j2 + n2 j1: for each (line, j2) the length-n1 transform
//     over j1, times w_N^(j2 k1), to scratch[line][j2 + n2 k1]; then for each (line, k1)
//     the length-n2 transform over j2, element k = k1 + n1 k2.
//   kTurnMid  kSecond, the diagonal operator, and kFirst of a transform with n1 and
//     n2 exchanged, whose (line, j2) elements are those of (line, k1).
enum PassKind { kWhole, kFirst, kSecond, kTurn, kTurnMid };

template <typename G>
struct PassArgs {
  int n, log2n, log2c, ls;  // ls: elements between two lines in shared memory
  bool line_fast;           // neighbouring threads take neighbouring lines, not elements
  int sign;
  int64_t lines;
  int log2o, log2nn;  // four-step: sub-lines of a line, its length N
  int64_t stride, lines_per_vec, xes, xcs, yes, ycs, tws;
  const void* x;
  void* y;
  const void *tw, *pre, *post;
  G alpha, beta;
  int quarter;
  // turns: the second transform's sign and twiddles, the phases between the two, the
  // diagonal operator's values (real or complex)
  int sign2;
  const void *tw2, *mid, *turn_diag;
  bool turn_real, add_real;
  // kDiag: the diagonal term's values and its input
  const void *add_diag, *add_x;
  int64_t add_xes, add_xcs;
};

// (hi, lo) pairs with |lo| <= ulp(hi) / 2 again, which sums leave larger
__device__ __forceinline__ double2 tidy(double2 v) { return v; }
__device__ __forceinline__ float2 tidy(float2 v) { return v; }
__device__ __forceinline__ float4 tidy(float4 v) {
  const float2 re = gather::ff_add(make_float2(v.x, 0.f), make_float2(v.y, 0.f));
  const float2 im = gather::ff_add(make_float2(v.z, 0.f), make_float2(v.w, 0.f));
  return make_float4(re.x, re.y, im.x, im.y);
}
// v times a diagonal's value
__device__ __forceinline__ double2 times(double2 v, double d, const Cs<double>& c) {
  return make_double2(__fma_rn(v.x, d, c.nz), __fma_rn(v.y, d, c.nz));
}
__device__ __forceinline__ float2 times(float2 v, float d, const Cs<float>&) { return make_float2(v.x * d, v.y * d); }
__device__ __forceinline__ float4 times(float4 v, float2 d, const Cs<DF>&) {
  const float2 re = gather::ff_mul(make_float2(v.x, v.y), d), im = gather::ff_mul(make_float2(v.z, v.w), d);
  return make_float4(re.x, re.y, im.x, im.y);
}
template <typename R, typename CT>
__device__ __forceinline__ CT times(CT v, CT d, const Cs<R>& c) {
  return cm(v, d, c);
}

// Eight ComplexF64 elements and a spare one: stores eight elements apart, as a first
// stage's are, and loads of neighbours each touch every bank once.
__device__ __forceinline__ int padded(int i) { return i + (i >> 3); }

// w + d g for a diagonal's value d
__device__ __forceinline__ double2 add_times(double2 w, double2 g, double d, const Cs<double>&) {
  return make_double2(__fma_rn(g.x, d, w.x), __fma_rn(g.y, d, w.y));
}
__device__ __forceinline__ float2 add_times(float2 w, float2 g, float d, const Cs<float>&) {
  return make_float2(__fmaf_rn(g.x, d, w.x), __fmaf_rn(g.y, d, w.y));
}
template <typename R, typename G>
__device__ __forceinline__ G add_times(G w, G g, G d, const Cs<R>& c) {
  return cadd(w, cm(g, d, c), c);
}
template <typename D>
__device__ __forceinline__ double2 add_times(double2 w, double2 g, D d, const Cs<DF>& c) {
  const double2 t = joined(times(FT<DF>::in(g), d, c));
  return make_double2(w.x + t.x, w.y + t.y);
}

// The stages of one line's transform: element m of thread t is t + m tl before and
// after.  sm: the line's shared memory, which no thread reads any more.
template <typename R, int E>
__device__ __forceinline__ void line_stages(typename FT<R>::S (&u)[E], typename FT<R>::S* sm, int t, int log2n,
                                            const typename FT<R>::S* tw, int64_t tws, const Cs<R>& c) {
  constexpr int LE = E == 8 ? 3 : E == 4 ? 2 : 1;
  const int log2t = log2n - LE, tl = 1 << log2t;
  // the first stage, of radix E or of what log2 n leaves over
  const int rest = log2n % LE;
  int lns = LE;  // log2 of the length transformed so far
  if (rest == 0) {
    dft(u, c);
  } else if (rest == 1) {
#pragma unroll
    for (int i = 0; i < E / 2; ++i) dft2(u[i], u[i + E / 2], c);
    lns = 1;
  } else if constexpr (E == 8) {
#pragma unroll
    for (int i = 0; i < 2; ++i) dft4(u[i], u[i + 2], u[i + 4], u[i + 6], c);
    lns = 2;
  }
  if (lns < log2n) {
#pragma unroll
    for (int m = 0; m < E; ++m) {
      int i = E * t + m;
      if (rest == 1) i = 2 * (t + (m % (E / 2)) * tl) + m / (E / 2);
      if (E == 8 && rest == 2) i = 4 * (t + (m & 1) * tl) + (m >> 1);
      sm[padded(i)] = u[m];
    }
    while (true) {
      __syncthreads();
#pragma unroll
      for (int m = 0; m < E; ++m) u[m] = sm[padded(t + m * tl)];
      const int k = t & ((1 << lns) - 1);
      const int64_t step = ((int64_t)k << (log2t - lns)) * tws;
#pragma unroll
      for (int q = 1; q < E; ++q) u[q] = cm(u[q], __ldg(tw + q * step), c);
      dft(u, c);
      if (lns + LE == log2n) break;
      __syncthreads();
      const int i0 = ((t >> lns) << (lns + LE)) + k;
#pragma unroll
      for (int q = 0; q < E; ++q) sm[padded(i0 + (q << lns))] = u[q];
      lns += LE;
    }
  }
}


template <typename R>
constexpr int kFftThreads = std::is_same<R, float>::value ? 1024 : 512;

template <typename R, int E, int KIND, int MODE>
__global__ void __launch_bounds__(kFftThreads<R>) k_fft_line(const __grid_constant__ PassArgs<typename FT<R>::G> a) {
  using CT = typename FT<R>::S;
  using G = typename FT<R>::G;
  extern __shared__ __align__(16) unsigned char smem[];
  const int log2t = a.log2n - (E == 8 ? 3 : E == 4 ? 2 : 1), tl = 1 << log2t;
  const int tid = threadIdx.x;
  const int l = a.line_fast ? tid & ((1 << a.log2c) - 1) : tid >> log2t;
  const int t = a.line_fast ? tid >> a.log2c : tid & (tl - 1);
  CT* sm = reinterpret_cast<CT*>(smem) + l * a.ls;
  const int64_t sub = ((int64_t)blockIdx.x << a.log2c) + l;
  const bool on = sub < a.lines;
  constexpr bool kSteps = KIND == kFirst || KIND == kSecond || KIND == kTurnMid;
  const int64_t line = kSteps ? sub >> a.log2o : sub;
  const int o = kSteps ? (int)(sub & ((1 << a.log2o) - 1)) : 0;
  const int64_t nn = kSteps ? int64_t(1) << a.log2nn : a.n;
  // element m of this thread in the transform
  auto at = [&](int m) { return kSteps ? o + ((int64_t)(t + m * tl) << a.log2o) : (int64_t)(t + m * tl); };
  using DT = typename gather::Val<R, true>::T;
  const CT* tw = static_cast<const CT*>(a.tw);
  const Cs<R> c(a.sign);
  CT u[E];
  if (on) {
    if (KIND == kSecond || KIND == kTurnMid) {
      const CT* in = static_cast<const CT*>(a.x) + sub * a.n + t;
#pragma unroll
      for (int m = 0; m < E; ++m) u[m] = in[m * tl];
    } else {
      const CT* pre = static_cast<const CT*>(a.pre);
      const G* x = static_cast<const G*>(a.x) + line_base(line, a.lines_per_vec, a.stride, nn, a.xes, a.xcs);
      const int64_t se = a.stride * a.xes;
      G g[E];
#pragma unroll
      for (int m = 0; m < E; ++m) g[m] = x[at(m) * se];
#pragma unroll
      for (int m = 0; m < E; ++m)
        u[m] = cm(FT<R>::in(g[m]), __ldg(pre + at(m)), c);
    }
  }
  line_stages<R, E>(u, sm, t, a.log2n, tw, a.tws, c);
  if constexpr (KIND == kTurn || KIND == kTurnMid) {
    const Cs<R> c2(a.sign2);
    if (on) {
      const CT* mid = static_cast<const CT*>(a.mid);
      const int64_t base = line_base(line, a.lines_per_vec, a.stride, nn, 1, 0);
#pragma unroll
      for (int m = 0; m < E; ++m) u[m] = cm(tidy(u[m]), __ldg(mid + at(m)), c);
      if (a.turn_real) {
#pragma unroll
        for (int m = 0; m < E; ++m)
          u[m] = times(u[m], __ldg(static_cast<const DT*>(a.turn_diag) + base + at(m) * a.stride), c);
      } else {
#pragma unroll
        for (int m = 0; m < E; ++m)
          u[m] = times(u[m], __ldg(static_cast<const CT*>(a.turn_diag) + base + at(m) * a.stride), c);
      }
    }
    __syncthreads();
    line_stages<R, E>(u, sm, t, a.log2n, static_cast<const CT*>(a.tw2), a.tws, c2);
  }
  if (!on) return;
  if constexpr (KIND == kFirst || KIND == kTurnMid) {
    CT* out = static_cast<CT*>(a.y) + line * nn;
    const CT* w = KIND == kFirst ? tw : static_cast<const CT*>(a.tw2);
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int k = t + m * tl;
      out[o + ((int64_t)k << a.log2o)] = cm(u[m], __ldg(w + (((int64_t)o * k) & (nn - 1))), c);
    }
  } else {
    const CT* post = static_cast<const CT*>(a.post);
    G* y = static_cast<G*>(a.y) + line_base(line, a.lines_per_vec, a.stride, nn, a.yes, a.ycs);
    G w[E];
#pragma unroll
    for (int m = 0; m < E; ++m) w[m] = joined(cm(u[m], __ldg(post + at(m)), c));
    if constexpr (MODE == kDiag) {
      const G* x = static_cast<const G*>(a.add_x) + line_base(line, a.lines_per_vec, a.stride, nn, a.add_xes, a.add_xcs);
      const int64_t sx = a.stride * a.add_xes, base = line_base(line, a.lines_per_vec, a.stride, nn, 1, 0);
      G g[E];
#pragma unroll
      for (int m = 0; m < E; ++m) g[m] = x[at(m) * sx];
      if (a.add_real) {
#pragma unroll
        for (int m = 0; m < E; ++m)
          w[m] = add_times(w[m], g[m], __ldg(static_cast<const DT*>(a.add_diag) + base + at(m) * a.stride), c);
      } else {
#pragma unroll
        for (int m = 0; m < E; ++m)
          w[m] = add_times(w[m], g[m], __ldg(static_cast<const CT*>(a.add_diag) + base + at(m) * a.stride), c);
      }
    }
    store<R, MODE, E>(y, a.stride * a.yes, at, w, a.quarter, a.alpha, a.beta, out_consts(c));
  }
}

// e += s re(w), o += d im(w)
__device__ __forceinline__ void fma_parts(double2& e, double2& o, double2 s, double2 d, double2 w) {
  e.x = __fma_rn(s.x, w.x, e.x);
  e.y = __fma_rn(s.y, w.x, e.y);
  o.x = __fma_rn(d.x, w.y, o.x);
  o.y = __fma_rn(d.y, w.y, o.y);
}
__device__ __forceinline__ void fma_parts(float2& e, float2& o, float2 s, float2 d, float2 w) {
  e.x = __fmaf_rn(s.x, w.x, e.x);
  e.y = __fmaf_rn(s.y, w.x, e.y);
  o.x = __fmaf_rn(d.x, w.y, o.x);
  o.y = __fmaf_rn(d.y, w.y, o.y);
}
__device__ __forceinline__ void fma_parts(float4& e, float4& o, float4 s, float4 d, float4 w) {
  const float2 co = make_float2(w.x, w.y), si = make_float2(w.z, w.w);
  const float2 ex = gather::ff_mul(make_float2(s.x, s.y), co), ey = gather::ff_mul(make_float2(s.z, s.w), co);
  const float2 ox = gather::ff_mul(make_float2(d.x, d.y), si), oy = gather::ff_mul(make_float2(d.z, d.w), si);
  const Cs<DF> c(1);
  e = cadd(e, make_float4(ex.x, ex.y, ey.x, ey.y), c);
  o = cadd(o, make_float4(ox.x, ox.y, oy.x, oy.y), c);
}
template <typename CT>
__device__ __forceinline__ CT shfl_xor(CT v, int m) {
  return CT{__shfl_xor_sync(~0u, v.x, m), __shfl_xor_sync(~0u, v.y, m)};
}
__device__ __forceinline__ float4 shfl_xor(float4 v, int m) {
  return make_float4(__shfl_xor_sync(~0u, v.x, m), __shfl_xor_sync(~0u, v.y, m), __shfl_xor_sync(~0u, v.z, m),
                     __shfl_xor_sync(~0u, v.w, m));
}

// Direct DFT of one line of any length n: with s_j = a_j + a_(n-j), d_j = a_j - a_(n-j)
// the outputs k and n - k are E + i O and E - i O, E = a_0 + sum_j s_j cos(jk) (and
// a_(n/2) (-1)^k), O = sum_j d_j sin(jk), j < n / 2: a quarter of the products of the plain sum.
// `parts` neighbouring threads share an output pair, grid.y blocks a line.
template <typename R, int MODE>
__global__ void __launch_bounds__(128) k_dft_line(const __grid_constant__ PassArgs<typename FT<R>::G> a, int parts) {
  using CT = typename FT<R>::S;
  using G = typename FT<R>::G;
  extern __shared__ __align__(16) unsigned char smem[];
  CT* in = reinterpret_cast<CT*>(smem);  // a_0, s_j at j, a_(n/2), d_j at n - j
  const int n = a.n, h = (n - 1) / 2;
  const Cs<R> c(1);
  const CT *tw = static_cast<const CT*>(a.tw), *pre = static_cast<const CT*>(a.pre);
  const CT* post = static_cast<const CT*>(a.post);
  const G* x = static_cast<const G*>(a.x) + line_base(blockIdx.x, a.lines_per_vec, a.stride, n, a.xes, a.xcs);
  const int64_t se = a.stride * a.xes;
  for (int j = threadIdx.x; 2 * j <= n; j += blockDim.x) {
    const CT v = cm(FT<R>::in(x[j * se]), __ldg(pre + j), c);
    if (j == 0 || 2 * j == n) {
      in[j] = v;
    } else {
      const CT w = cm(FT<R>::in(x[(n - j) * se]), __ldg(pre + n - j), c);
      in[j] = cadd(v, w, c);
      in[n - j] = csub(v, w, c);
    }
  }
  __syncthreads();
  const int id = blockIdx.y * blockDim.x + threadIdx.x;
  const int k = id / parts, part = id - k * parts;
  const bool on = 2 * k <= n;
  CT e{}, d{};
  if (on) {
    if (part == 0) {
      e = in[0];
      if ((n & 1) == 0) e = (k & 1) ? csub(e, in[n / 2], c) : cadd(e, in[n / 2], c);
    }
    const int step = (int)((int64_t)k * parts % n);
    int idx = (int)((int64_t)k * (part + 1) % n);
#pragma unroll 4
    for (int j = part + 1; j <= h; j += parts) {
      const CT w = __ldg(tw + idx);
      fma_parts(e, d, in[j], in[n - j], w);
      idx += step;
      if (idx >= n) idx -= n;
    }
  }
  for (int p = 1; p < parts; p *= 2) {  // parts divides 32: the groups lie within a warp
    e = cadd(e, shfl_xor(e, p), c);
    d = cadd(d, shfl_xor(d, p), c);
  }
  if (!on || part != 0) return;
  G* y = static_cast<G*>(a.y) + line_base(blockIdx.x, a.lines_per_vec, a.stride, n, a.yes, a.ycs);
  const int64_t so = a.stride * a.yes;
  G w[1] = {joined(cm(cadd_i(e, d, c), __ldg(post + k), c))};
  store<R, MODE, 1>(y, so, [&](int) { return (int64_t)k; }, w, a.quarter, a.alpha, a.beta, out_consts(c));
  if (k > 0 && 2 * k < n) {
    w[0] = joined(cm(csub_i(e, d, c), __ldg(post + n - k), c));
    store<R, MODE, 1>(y, so, [&](int) { return (int64_t)(n - k); }, w, a.quarter, a.alpha, a.beta, out_consts(c));
  }
}

template <typename R, int E, int KIND, int MODE>
void launch_line(PassArgs<typename FT<R>::G>& p, int64_t lines, int cols, cudaStream_t s) {
  using CT = typename FT<R>::S;
  const int tl = p.n / E;
  // lines of a block: a warp at least, and `cols` neighbouring lines where those are
  // neighbours in memory (64 bytes: two sectors)
  int C = 1;
  while (C < lines && (C * tl < 32 || (C < cols && 2 * C * tl <= kFftThreads<R> / 2))) C *= 2;
  p.log2c = log2_of(C);
  // two elements past a multiple of 128 bytes: neighbouring lines start in other banks
  const int unit = 128 / (int)sizeof(CT);
  p.ls = (p.n + p.n / 8 + unit - 1) / unit * unit + 2;
  p.line_fast = cols > 1;
  p.lines = lines;
  const size_t smem = (size_t)C * p.ls * sizeof(CT);
  auto k = k_fft_line<R, E, KIND, MODE>;
  if (smem > 48 * 1024) QOB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<(unsigned)((lines + C - 1) / C), C * tl, smem, s>>>(p);
  QOB_LAUNCHED();
}

// Elements a thread.  Eight need the fewest operations a point (with the phases 19 for
// 64 points; four 26, two 32), but the pipe gives one warp a quarter of an SM's rate
// at most: while a quarter has no second warp to run, a thread's own operations are the time.
template <typename R, int KIND, int MODE>
void launch_line(PassArgs<typename FT<R>::G>& p, int64_t lines, int cols, int sms, cudaStream_t s) {
  int best = 8;
  double least = 0;
  for (int e = 8; e >= 2; e /= 2) {
    if (p.n / e > kFftThreads<R> / 2 && e < 8) break;
    const int le = log2_of(e), stages = (p.log2n + le - 1) / le;
    const double ops = 8.0 * e + stages * (e == 8 ? 52 : e == 4 ? 16 : 4) + (stages - 1) * 4.0 * (e - 1);  // one transform
    const double warps = (double)lines * p.n / (32.0 * e) / (4.0 * sms);
    const double t = std::max(warps, 1.0) * ops;
    if (e == 8 || t < 0.9 * least) {
      best = e;
      least = t;
    }
  }
  if (best == 8)
    launch_line<R, 8, KIND, MODE>(p, lines, cols, s);
  else if (best == 4)
    launch_line<R, 4, KIND, MODE>(p, lines, cols, s);
  else
    launch_line<R, 2, KIND, MODE>(p, lines, cols, s);
}

template <typename R>
PassArgs<typename FT<R>::G> pass_args(const FftAxis& ax, int64_t len, const void* x, int64_t xes, int64_t xcs,
                                      const FftOut& o) {
  PassArgs<typename FT<R>::G> p{};
  using E = decltype(p.alpha.x);
  p.alpha.x = (E)o.alpha.re;
  p.alpha.y = (E)o.alpha.im;
  p.beta.x = (E)o.beta.re;
  p.beta.y = (E)o.beta.im;
  p.quarter = -1;
  if (o.alpha.im == 0.0 && std::abs(o.alpha.re) == 1.0) p.quarter = o.alpha.re > 0 ? 0 : 2;
  if (o.alpha.re == 0.0 && std::abs(o.alpha.im) == 1.0) p.quarter = o.alpha.im > 0 ? 1 : 3;
  p.n = (int)ax.n;
  p.tws = 1;
  p.sign = ax.sign;
  p.stride = ax.stride;
  p.lines_per_vec = len / ax.n;
  p.x = x;
  p.xes = xes;
  p.xcs = xcs;
  p.y = o.y;
  p.yes = o.yes;
  p.ycs = o.ycs;
  p.tw = ax.tw.p;
  p.pre = ax.pre.p;
  p.post = ax.post.p;
  if (o.add) {
    p.add_diag = o.add->diag.p;
    p.add_real = o.add->real_vals;
    p.add_x = o.add_x;
    p.add_xes = o.add_xes;
    p.add_xcs = o.add_xcs;
  }
  return p;
}

template <typename G>
void split_first(PassArgs<G>& p, int64_t n1, int64_t n2) {  // over j1 and the n2 sub-lines
  p.n = (int)n1;
  p.log2n = log2_of(n1);
  p.log2o = log2_of(n2);
  p.log2nn = p.log2n + p.log2o;
  p.tws = n2;
}

// One axis; scratch: room for the vectors, or null (no four-step form).
template <typename R, int MODE>
void launch_axis(const FftAxis& ax, int64_t len, const void* x, int64_t xes, int64_t xcs, const FftOut& o,
                 int64_t ncols, void* scratch, int sms, cudaStream_t s) {
  using G = typename FT<R>::G;  // vectors, alpha, beta
  using CT = typename FT<R>::S;  // twiddles, phases, shared memory, scratch
  PassArgs<G> p = pass_args<R>(ax, len, x, xes, xcs, o);
  const int64_t lines = p.lines_per_vec * ncols;
  const int near = 64 / (int)sizeof(G);  // elements of 64 bytes
  if (scratch && four_step(ax, lines, sms)) {
    PassArgs<G> q = p;
    split_first(p, ax.n1, ax.n2);
    split_first(q, ax.n2, ax.n1);
    p.y = scratch;
    q.x = scratch;
    launch_line<R, kFirst, kPut>(p, lines * ax.n2, near, sms, s);
    launch_line<R, kSecond, MODE>(q, lines * ax.n1, near, sms, s);
    return;
  }
  // whole vectors per launch, at most 2^31 - 1 lines (blocks)
  const int64_t vec_per_launch = std::max<int64_t>(1, (int64_t)INT32_MAX / p.lines_per_vec);
  for (int64_t c0 = 0; c0 < ncols; c0 += vec_per_launch) {
    const int64_t nl = std::min<int64_t>(ncols - c0, vec_per_launch) * p.lines_per_vec;
    p.x = (const G*)x + c0 * xcs;
    p.y = (G*)o.y + c0 * o.ycs;
    if (o.add) p.add_x = (const G*)o.add_x + c0 * o.add_xcs;
    if (ax.pow2) {
      p.log2n = log2_of(ax.n);
      launch_line<R, kWhole, MODE>(p, nl, ax.stride > 1 ? near : 1, sms, s);
    } else if constexpr (MODE != kDiag) {
      const size_t smem = (size_t)ax.n * sizeof(CT);
      auto k = k_dft_line<R, MODE>;
      if (smem > 48 * 1024) QOB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      const int64_t pairs = ax.n / 2 + 1;
      int parts = 1;  // threads that share an output pair: as many as fill the SMs
      while (parts < 16 && parts * 2 <= ax.n && nl * ((pairs * parts + 127) / 128) < 2 * sms) parts *= 2;
      k<<<dim3((unsigned)nl, (unsigned)((pairs * parts + 127) / 128)), 128, smem, s>>>(p, parts);
      QOB_LAUNCHED();
    }
  }
}

// Two transforms of one axis with the diagonal d between; two rooms of scratch for
// the four-step form, or null.
template <typename R, int MODE>
void launch_turn(const FftAxis& ax, const FftAxis& bx, const GatherPlan& d, const void* mid, int64_t len, const void* x,
                 int64_t xes, int64_t xcs, const FftOut& o, int64_t ncols, void* scratch, void* scratch2, int sms,
                 cudaStream_t s) {
  using G = typename FT<R>::G;
  PassArgs<G> p = pass_args<R>(ax, len, x, xes, xcs, o);
  p.post = bx.post.p;
  p.sign2 = bx.sign;
  p.tw2 = bx.tw.p;
  p.mid = mid;
  p.turn_diag = d.diag.p;
  p.turn_real = d.real_vals;
  const int64_t lines = p.lines_per_vec * ncols;
  const int near = 64 / (int)sizeof(G);
  if (scratch && four_step(ax, lines, sms)) {
    PassArgs<G> m = p, q = p;
    split_first(p, ax.n1, ax.n2);
    split_first(m, ax.n2, ax.n1);
    split_first(q, ax.n1, ax.n2);
    q.tw = bx.tw.p;
    q.sign = bx.sign;
    p.y = scratch;
    m.x = scratch;
    m.y = scratch2;
    q.x = scratch2;
    launch_line<R, kFirst, kPut>(p, lines * ax.n2, near, sms, s);
    launch_line<R, kTurnMid, kPut>(m, lines * ax.n1, near, sms, s);
    launch_line<R, kSecond, MODE>(q, lines * ax.n2, near, sms, s);
    return;
  }
  p.log2n = log2_of(ax.n);
  const int64_t vec_per_launch = std::max<int64_t>(1, (int64_t)INT32_MAX / p.lines_per_vec);
  for (int64_t c0 = 0; c0 < ncols; c0 += vec_per_launch) {
    const int64_t nl = std::min<int64_t>(ncols - c0, vec_per_launch) * p.lines_per_vec;
    p.x = (const G*)x + c0 * xcs;
    p.y = (G*)o.y + c0 * o.ycs;
    if (o.add) p.add_x = (const G*)o.add_x + c0 * o.add_xcs;
    launch_line<R, kTurn, MODE>(p, nl, ax.stride > 1 ? near : 1, sms, s);
  }
}

// f with the store mode that beta and the added diagonal ask for
template <typename F>
void with_mode(const FftOut& o, F f) {
  if (o.add)
    f(std::integral_constant<int, kDiag>());
  else if (o.beta.re == 0.0 && o.beta.im == 0.0)
    f(std::integral_constant<int, kPut>());
  else if (o.beta.re == 1.0 && o.beta.im == 0.0)
    f(std::integral_constant<int, kAdd>());
  else
    f(std::integral_constant<int, kAxpby>());
}

}  // namespace

template <typename R>
void fft_axis(const FftAxis& ax, int64_t len, const void* x, int64_t xes, int64_t xcs, const FftOut& o, int64_t ncols,
              void* scratch, int sms, cudaStream_t s) {
  with_mode(o, [&](auto m) {
    launch_axis<R, decltype(m)::value>(ax, len, x, xes, xcs, o, ncols, scratch, sms, s);
  });
}

template <typename R>
void fft_turn(const FftAxis& ax, const FftAxis& bx, const GatherPlan& d, const void* mid, int64_t len, const void* x,
              int64_t xes, int64_t xcs, const FftOut& o, int64_t ncols, void* scratch, void* scratch2, int sms,
              cudaStream_t s) {
  with_mode(o, [&](auto m) {
    launch_turn<R, decltype(m)::value>(ax, bx, d, mid, len, x, xes, xcs, o, ncols, scratch, scratch2, sms, s);
  });
}

}  // namespace qob
