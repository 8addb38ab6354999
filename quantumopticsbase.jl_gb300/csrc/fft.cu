// fft.cu -- FFTOperator (src/particle.jl:196-535): the transform between a
// position grid and its momentum grid, applied to kets, bras and operators.
//
// The reference multiplies by a phase array (mul_before), runs FFTW's in-place
// fft!/bfft! over the transformed dimensions, and multiplies by a second phase
// array that includes 1/sqrt(N) (mul_after); bras and the rows of an operator
// multiplied from the right go through conj -> opposite-sign transform -> conj,
// which is the same-sign transform of the row with the two phase arrays
// swapped (the DFT matrix is symmetric).  Both phase arrays are Kronecker
// products of per-axis vectors, so a multi-dimensional transform is one pass per
// axis, each pass multiplying by its axis's phases.
//
// Powers of two from 8 on: a thread owns eight elements of a line in registers and
// does radix-8 Stockham stages on them (Van Loan, Computational Frameworks for the
// FFT, 1992; one stage of radix 2 or 4 first where log2 n is no multiple of 3), with
// one exchange through shared memory between two stages; the first stage reads and the
// last one writes global memory.  Other lengths: a direct DFT on the even and odd
// parts of the line.  The last pass applies alpha and beta.
//
// What bounds it is the FP64 pipe, two lanes a clock and SM: 6.5 operations
// a point and radix-8 stage, 3.5 for its twiddles, 4 for each phase array.
// Measured against radix-2 stages through shared memory and the plain sum (a particle
// Hamiltonian, two transforms and two diagonals, us): 4096 points, 64 kets, ComplexF64 103 -> 84,
// ComplexF32 58 -> 36; 256 x 256 points, 8 kets 210 -> 188, double-float 122 -> 98; 800 points,
// 32 kets 2375 -> 117, one ket 2364 -> 42.
#include <cmath>
#include <type_traits>
#include <vector>

#include "k_gather.cuh"  // double-float helpers
#include "qob_internal.h"

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
  __device__ __forceinline__ explicit Cs(int sign) : one(1), s((R)sign), r((R)0.70710678118654752440), nz(-(R)0) {
    if constexpr (std::is_same<R, double>::value) asm volatile("" : "+d"(one), "+d"(s), "+d"(r), "+d"(nz));
  }
};
template <>
struct Cs<DF> {
  float s;
  float2 r;
  __device__ __forceinline__ explicit Cs(int sign) : s((float)sign), r(make_float2(0.70710677f, 1.21016175e-8f)) {}
};

// u * c + v for a factor that makes the product exact (1, -1, the sign)
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

// How the last pass writes: y = v; alpha v; alpha v + y (a later term of a sum); alpha v + beta y.
enum StoreMode { kPut = 0, kScale = 1, kAdd = 2, kAxpby = 3 };

template <typename R, int MODE>
__device__ __forceinline__ void store(typename FT<R>::G* y, typename FT<R>::S v, typename FT<R>::S post,
                                      typename FT<R>::G alpha, typename FT<R>::G beta, const Cs<R>& c) {
  using G = typename FT<R>::G;
  using A = typename std::conditional<std::is_same<R, DF>::value, double, R>::type;
  const Cs<A> ca(1);
  G o;
  if constexpr (std::is_same<R, DF>::value) {
    const float4 w = cm(v, post, c);  // double-float, then joined; alpha / beta in FP64
    o = make_double2(gather::ff_join(w.x, w.y), gather::ff_join(w.z, w.w));
  } else {
    o = cm(v, post, c);
  }
  if constexpr (MODE != kPut) o = cm(o, alpha, ca);
  if constexpr (MODE == kAdd) o = cadd(o, *y, ca);
  if constexpr (MODE == kAxpby) o = cadd(o, cm(*y, beta, ca), ca);
  *y = o;
}

// One pass over lines of n = 2^log2n elements, C = 2^log2c lines a block, E
// elements a thread.
//   kWhole  the whole transform of an axis.
//   kFirst, kSecond  four-step form (Bailey 1990) of a transform of length
//     N = n1 n2, element j = j2 + n2 j1: for each (line, j2) the length-n1 transform
//     over j1, times w_N^(j2 k1), to scratch[line][j2 + n2 k1]; then for each (line, k1)
//     the length-n2 transform over j2, element k = k1 + n1 k2.
enum PassKind { kWhole, kFirst, kSecond };

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
};

// Eight ComplexF64 elements and a spare one: stores eight elements apart, as a first
// stage's are, and loads of neighbours each touch every bank once.
__device__ __forceinline__ int padded(int i) { return i + (i >> 3); }

template <typename R>
constexpr int kFftThreads = std::is_same<R, float>::value ? 1024 : 512;

template <typename R, int E, int KIND, int MODE>
__global__ void __launch_bounds__(kFftThreads<R>) k_fft_line(const __grid_constant__ PassArgs<typename FT<R>::G> a) {
  using CT = typename FT<R>::S;
  using G = typename FT<R>::G;
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int LE = E == 8 ? 3 : E == 4 ? 2 : 1;
  const int log2t = a.log2n - LE, tl = 1 << log2t;
  const int tid = threadIdx.x;
  const int l = a.line_fast ? tid & ((1 << a.log2c) - 1) : tid >> log2t;
  const int t = a.line_fast ? tid >> a.log2c : tid & (tl - 1);
  CT* sm = reinterpret_cast<CT*>(smem) + l * a.ls;
  const int64_t sub = ((int64_t)blockIdx.x << a.log2c) + l;
  const bool on = sub < a.lines;
  const int64_t line = KIND == kWhole ? sub : sub >> a.log2o;
  const int o = KIND == kWhole ? 0 : (int)(sub & ((1 << a.log2o) - 1));
  const int64_t nn = KIND == kWhole ? a.n : int64_t(1) << a.log2nn;
  const CT* tw = static_cast<const CT*>(a.tw);
  const Cs<R> c(a.sign);
  CT u[E];
  if (on) {
    if (KIND == kSecond) {
      const CT* in = static_cast<const CT*>(a.x) + sub * a.n + t;
#pragma unroll
      for (int m = 0; m < E; ++m) u[m] = in[m * tl];
    } else {
      const CT* pre = static_cast<const CT*>(a.pre);
      const G* x = static_cast<const G*>(a.x) + line_base(line, a.lines_per_vec, a.stride, nn, a.xes, a.xcs);
      const int64_t se = a.stride * a.xes;
      G g[E];
#pragma unroll
      for (int m = 0; m < E; ++m) g[m] = x[(KIND == kFirst ? o + ((t + m * tl) << a.log2o) : t + m * tl) * se];
#pragma unroll
      for (int m = 0; m < E; ++m)
        u[m] = cm(FT<R>::in(g[m]), __ldg(pre + (KIND == kFirst ? o + ((t + m * tl) << a.log2o) : t + m * tl)), c);
    }
  }
  // the first stage, of radix E or of what log2 n leaves over
  const int rest = a.log2n % LE;
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
  if (lns < a.log2n) {
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
      const int64_t step = ((int64_t)k << (log2t - lns)) * a.tws;
#pragma unroll
      for (int q = 1; q < E; ++q) u[q] = cm(u[q], __ldg(tw + q * step), c);
      dft(u, c);
      if (lns + LE == a.log2n) break;
      __syncthreads();
      const int i0 = ((t >> lns) << (lns + LE)) + k;
#pragma unroll
      for (int q = 0; q < E; ++q) sm[padded(i0 + (q << lns))] = u[q];
      lns += LE;
    }
  }
  if (!on) return;
  if (KIND == kFirst) {
    CT* out = static_cast<CT*>(a.y) + line * nn;
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int k = t + m * tl;
      out[o + ((int64_t)k << a.log2o)] = cm(u[m], __ldg(tw + (((int64_t)o * k) & (nn - 1))), c);
    }
  } else {
    const CT* post = static_cast<const CT*>(a.post);
    G* y = static_cast<G*>(a.y) + line_base(line, a.lines_per_vec, a.stride, nn, a.yes, a.ycs);
    const int64_t so = a.stride * a.yes;
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int64_t k = KIND == kSecond ? o + ((int64_t)(t + m * tl) << a.log2o) : t + m * tl;
      store<R, MODE>(y + k * so, u[m], __ldg(post + k), a.alpha, a.beta, c);
    }
  }
}

// e += s re(w), d += d im(w)
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
  store<R, MODE>(y + k * so, cadd_i(e, d, c), __ldg(post + k), a.alpha, a.beta, c);
  if (k > 0 && 2 * k < n)
    store<R, MODE>(y + (n - k) * so, csub_i(e, d, c), __ldg(post + n - k), a.alpha, a.beta, c);
}

int log2_of(int64_t n) {
  int l = 0;
  while ((int64_t(1) << l) < n) ++l;
  return l;
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
    const double ops = 8.0 * e + stages * (e == 8 ? 52 : e == 4 ? 16 : 4) + (stages - 1) * 4.0 * (e - 1);
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

template <typename R, int MODE>
void launch_typed(const FftAxis& ax, int64_t len, const void* x, int64_t xes, int64_t xcs, void* y, int64_t yes,
                  int64_t ycs, int64_t ncols, c128 alpha, c128 beta, bool final, void* scratch, cudaStream_t s) {
  using G = typename FT<R>::G;  // vectors, alpha, beta
  using CT = typename FT<R>::S;  // twiddles, phases, shared memory, scratch
  PassArgs<G> p{};
  using E = decltype(p.alpha.x);
  p.alpha.x = (E)alpha.re;
  p.alpha.y = (E)alpha.im;
  p.beta.x = (E)beta.re;
  p.beta.y = (E)beta.im;
  p.sign = ax.sign;
  p.stride = ax.stride;
  p.lines_per_vec = len / ax.n;
  p.xes = xes;
  p.xcs = xcs;
  p.yes = yes;
  p.ycs = ycs;
  p.tw = ax.tw.p;
  p.pre = ax.pre.p;
  p.post = ax.post.p;
  int dev = 0, sms = 0;
  QOB_CUDA(cudaGetDevice(&dev));
  QOB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t lines = p.lines_per_vec * ncols;
  const int near = 64 / (int)sizeof(G);  // elements of 64 bytes
  if (final && ax.n1 > 0 && scratch && lines < sms && lines * ax.n2 <= INT32_MAX) {
    // few long lines: spread each over many blocks (two launches)
    PassArgs<G> q = p;
    p.n = (int)ax.n1;
    p.log2n = log2_of(ax.n1);
    q.n = (int)ax.n2;
    q.log2n = log2_of(ax.n2);
    p.log2nn = q.log2nn = log2_of(ax.n);
    p.log2o = q.log2n;
    q.log2o = p.log2n;
    p.tws = ax.n2;
    q.tws = ax.n1;
    p.x = x;
    p.y = scratch;
    q.x = scratch;
    q.y = y;
    launch_line<R, kFirst, kPut>(p, lines * ax.n2, near, sms, s);
    launch_line<R, kSecond, MODE>(q, lines * ax.n1, near, sms, s);
    return;
  }
  p.n = (int)ax.n;
  p.tws = 1;
  // whole vectors per launch, at most 2^31 - 1 lines (blocks)
  const int64_t vec_per_launch = std::max<int64_t>(1, (int64_t)INT32_MAX / p.lines_per_vec);
  for (int64_t c0 = 0; c0 < ncols; c0 += vec_per_launch) {
    const int64_t nl = std::min<int64_t>(ncols - c0, vec_per_launch) * p.lines_per_vec;
    p.x = (const G*)x + c0 * xcs;
    p.y = (G*)y + c0 * ycs;
    if (ax.pow2) {
      p.log2n = log2_of(ax.n);
      launch_line<R, kWhole, MODE>(p, nl, ax.stride > 1 ? near : 1, sms, s);
    } else {
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

template <typename R>
void launch_form(const FftAxis& ax, int64_t len, const void* x, int64_t xes, int64_t xcs, void* y, int64_t yes,
                 int64_t ycs, int64_t ncols, c128 alpha, c128 beta, bool final, void* scratch, cudaStream_t s) {
  const bool a1 = alpha.re == 1.0 && alpha.im == 0.0, b0 = beta.re == 0.0 && beta.im == 0.0;
  const bool b1 = beta.re == 1.0 && beta.im == 0.0;
  if (!final || (a1 && b0))
    launch_typed<R, kPut>(ax, len, x, xes, xcs, y, yes, ycs, ncols, alpha, beta, final, scratch, s);
  else if (b0)
    launch_typed<R, kScale>(ax, len, x, xes, xcs, y, yes, ycs, ncols, alpha, beta, final, scratch, s);
  else if (b1)
    launch_typed<R, kAdd>(ax, len, x, xes, xcs, y, yes, ycs, ncols, alpha, beta, final, scratch, s);
  else
    launch_typed<R, kAxpby>(ax, len, x, xes, xcs, y, yes, ycs, ncols, alpha, beta, final, scratch, s);
}

void upload_prec(DeviceBuf& d, const std::vector<c128>& v, int precision, bool ff) {
  if (ff) {  // (re hi, re lo, im hi, im lo)
    std::vector<float> q(4 * v.size());
    for (size_t i = 0; i < v.size(); ++i) {
      const float rh = (float)v[i].re, ih = (float)v[i].im;
      q[4 * i] = rh;
      q[4 * i + 1] = (float)(v[i].re - (double)rh);
      q[4 * i + 2] = ih;
      q[4 * i + 3] = (float)(v[i].im - (double)ih);
    }
    d.upload(q.data(), q.size() * sizeof(float));
  } else if (precision == QOB_C128) {
    d.upload(v.data(), v.size() * sizeof(c128));
  } else {
    std::vector<c64> f(v.size());
    for (size_t i = 0; i < v.size(); ++i) f[i] = {(float)v[i].re, (float)v[i].im};
    d.upload(f.data(), f.size() * sizeof(c64));
  }
}

}  // namespace

void launch_fft_pass(int precision, const FftAxis& ax, int64_t len, const void* x, int64_t xes, int64_t xcs,
                     void* y, int64_t yes, int64_t ycs, int64_t ncols, c128 alpha, c128 beta, bool final,
                     void* scratch, cudaStream_t s, bool ff) {
  if (ff)
    launch_form<DF>(ax, len, x, xes, xcs, y, yes, ycs, ncols, alpha, beta, final, scratch, s);
  else if (precision == QOB_C128)
    launch_form<double>(ax, len, x, xes, xcs, y, yes, ycs, ncols, alpha, beta, final, scratch, s);
  else
    launch_form<float>(ax, len, x, xes, xcs, y, yes, ycs, ncols, alpha, beta, final, scratch, s);
}

// LEFT (kets, operator columns): pre = before, post = after.  RIGHT (bras,
// operator rows): pre = after, post = before, same sign.
std::unique_ptr<Plan> compile_fft(const NodeP& op, int side, int precision_code) {
  const bool ff = precision_code == QOB_C128X;
  const int precision = ff ? QOB_C128 : precision_code;
  auto P = std::make_unique<Plan>();
  P->kind = Plan::Kind::Fft;
  P->side = side;
  P->precision = precision;
  P->ff = ff;
  P->m = side == QOB_RIGHT ? op->n : op->m;
  P->n = side == QOB_RIGHT ? op->m : op->n;
  P->root = op.get();
  const std::vector<int64_t>& shape = op->shape_l;
  int64_t off = 0;
  for (size_t a = 0; a < op->fft_sites.size(); ++a) {
    const int site = op->fft_sites[a];
    FftAxis ax;
    ax.n = shape[site];
    ax.stride = 1;
    for (int q = 0; q < site; ++q) ax.stride *= shape[q];
    ax.pow2 = (ax.n & (ax.n - 1)) == 0 && ax.n >= 8;
    const size_t esz = precision == QOB_C128 ? 16 : 8;
    const size_t smem = ((ax.n & (ax.n - 1)) == 0 && ax.n >= 2 ? 2 : 1) * (size_t)ax.n * esz;
    if (smem > 200 * 1024) fail(QOB_ERR_UNSUPPORTED, "FFT axis too long for one block's shared memory");
    ax.sign = op->fft_sign[a] < 0 ? -1 : 1;
    std::vector<c128> tw((size_t)ax.n);
    for (int64_t m = 0; m < ax.n; ++m) {
      const double th = 6.283185307179586476925286766559 * (double)m / (double)ax.n;
      tw[(size_t)m] = {std::cos(th), ax.sign * std::sin(th)};
    }
    std::vector<c128> before(op->fft_before.begin() + off, op->fft_before.begin() + off + ax.n);
    std::vector<c128> after(op->fft_after.begin() + off, op->fft_after.begin() + off + ax.n);
    off += ax.n;
    upload_prec(ax.tw, tw, precision, ff);
    if (ax.pow2 && ax.n >= 512) {
      ax.n1 = int64_t(1) << (log2_of(ax.n) / 2);
      ax.n2 = ax.n / ax.n1;
    }
    upload_prec(ax.pre, side == QOB_RIGHT ? after : before, precision, ff);
    upload_prec(ax.post, side == QOB_RIGHT ? before : after, precision, ff);
    P->fft.push_back(std::move(ax));
  }
  return P;
}

}  // namespace qob

namespace {
qob_op* wrap_node(qob::NodeP n) {
  auto* h = new qob_op;
  h->node = std::move(n);
  return h;
}
}  // namespace

extern "C" int qob_op_fft(qob_ctx* ctx, int nsub, const int64_t* shape, int naxes, const int64_t* axes,
                          const int* sign, const double* before, const double* after, qob_op** out) {
  if (!ctx) return QOB_ERR_ARG;
  try {
    using namespace qob;
    if (!out || nsub < 1 || nsub > kMaxSites || !shape || naxes < 1 || naxes > nsub || !axes || !sign || !before ||
        !after)
      fail(QOB_ERR_ARG, "qob_op_fft: bad arguments");
    auto nd = std::make_shared<OpNode>();
    nd->kind = Kind::Fft;
    nd->shape_l.assign(shape, shape + nsub);
    nd->shape_r = nd->shape_l;
    int64_t len = 1;
    for (int i = 0; i < nsub; ++i) {
      if (shape[i] < 1) fail(QOB_ERR_ARG, "qob_op_fft: bad subsystem length");
      len *= shape[i];
    }
    if (len > INT32_MAX) fail(QOB_ERR_UNSUPPORTED, "dimension exceeds 2^31-1");
    nd->m = nd->n = len;
    int64_t total = 0;
    for (int a = 0; a < naxes; ++a) {
      if (axes[a] < 1 || axes[a] > nsub || (a > 0 && axes[a] <= axes[a - 1]))
        fail(QOB_ERR_ARG, "qob_op_fft: axes must be increasing 1-based subsystem indices");
      nd->fft_sites.push_back((int)axes[a] - 1);
      nd->fft_sign.push_back(sign[a] < 0 ? -1 : 1);
      total += shape[axes[a] - 1];
    }
    for (int64_t k = 0; k < total; ++k) {
      nd->fft_before.push_back({before[2 * k], before[2 * k + 1]});
      nd->fft_after.push_back({after[2 * k], after[2 * k + 1]});
    }
    *out = wrap_node(nd);
    return QOB_OK;
  } catch (const qob::Error& e) {
    ctx->c.err = e.msg;
    return e.code;
  }
}
