// k_multi.cuh -- the fused LazySum gather for plans in the flip form: every
// merged group acts on at most two runs of power-of-two subsystems of a square
// basis, has one stored entry per row whose input index is the output index with
// a fixed set of bits flipped, and the same value in all its stored entries (Pauli
// strings, bonds and ladder products of spin chains and qubit registers, the
// Liouvillians of both).
//
// A thread owns NI consecutive, aligned output indices J0 .. J0 + NI - 1 and
// walks the vectors of its block's share.  A group that leaves the bits below NI
// alone is active for all NI indices or for none, and reads NI consecutive
// inputs at J0 ^ flip in 32-byte loads.  Which of these groups are active
// depends on J0 only: a bit mask, made once and used for every vector.  The few
// groups that touch the bits below NI read one block too, permuted by the low
// part of the flip.  Per active group and vector that leaves one 8- or 16-byte
// record read, the loads (the next group's issued before this one's are used) and
// the multiply-adds.
//
// The walk over the mask keeps the tests of activity real branches: as
// predicated instructions (what a test around each group's multiply-adds becomes)
// the skipped multiply-adds still occupy GB300's FP64 pipe, two lanes a clock.
//
// FP32 and double-float arithmetic runs on (re, im) pairs with the packed FP32
// instructions (fma.rn.f32x2 and its relatives round each half as the scalar
// ones do), half the issue slots of the scalar form.
//
// Measured (one-index kernel before -> this one; the call's device time): 14 spins
// on 64 kets, ComplexF64, 71.0 -> 49.2 us, FP64-pipe bound (21 pipe instructions
// per element, 39 us at the rates below); 16 spins on 51 kets, ComplexF32, 56.5 ->
// 35.2 us, waiting on gathered loads (half the issue slots, 0.25 of the L2's rate);
// one ket of 2^20 entries, double-float, 46.3 -> 40.0 us; the Liouvillian of 10
// spins 139 -> 85 us and 1000 operator rows times 10 spins 56.8 -> 40.7 us (both
// ComplexF64, FP64-pipe bound).
//
// Included by k_gather.cuh (after the accumulators).
#pragma once

namespace qob {
namespace gather {

// Row records: x = shift of the first run | shift of the second << 8 | log2 of
// the second run's local stride << 16, y = mask of the first run | mask of the
// second << 16, z = first slot, w = rows with a stored value (bit mask); flips: x
// = flip, y = slot of a stored entry.
template <bool TWO>
__device__ __forceinline__ uint32_t multi_row(const int4& f, uint32_t J) {
  const uint32_t m = (uint32_t)f.y;
  const uint32_t r = (J >> ((uint32_t)f.x & 0xffu)) & (m & 0xffffu);
  if (!TWO) return r;
  return r + (((J >> (((uint32_t)f.x >> 8) & 0xffu)) & (m >> 16)) << ((uint32_t)f.x >> 16));
}
template <bool TWO>
__device__ __forceinline__ uint32_t multi_active(const int4& f, uint32_t J) {
  return ((uint32_t)f.w >> multi_row<TWO>(f, J)) & 1u;
}

// ---- packed FP32 pairs ----
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 upk(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 swp(f2 v) {
  const float2 a = upk(v);
  return pk(a.y, a.x);
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
constexpr f2 kMinus1 = 0xbf800000bf800000ull;  // (-1, -1)
// a - b, one rounding
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, kMinus1, a); }

// Per precision: the input element X, the value V as an entry keeps it, the
// operand W made from it once per entry, the accumulator.
template <typename R>
struct Multi;

template <>
struct Multi<double> {
  using X = double2;
  using Acc = AccD;
  struct Rec {
    uint32_t flip, pad;
    double v;
  };
  using W = double;
  static __device__ __forceinline__ Rec record(uint32_t flip, double v) { return {flip, 0, v}; }
  template <bool IM>
  static __device__ __forceinline__ W operand(double v) {
    return v;
  }
  template <bool IM>
  static __device__ __forceinline__ W operand(const Rec& r) {
    return r.v;
  }
  template <bool IM>
  static __device__ __forceinline__ void mac(Acc& a, const W& w, X x) {
    if constexpr (IM)
      a.mac_i(w, x);
    else
      a.mac(w, x);
  }
  static __device__ __forceinline__ void set(Acc& a, double d, X x, double nzero) {
    a.re = fma(d, x.x, nzero);
    a.im = fma(d, x.y, nzero);
  }
  static __device__ __forceinline__ void set(Acc& a, double2 d, X x, double nzero) {
    a.re = fma(-d.y, x.y, fma(d.x, x.x, nzero));
    a.im = fma(d.y, x.x, fma(d.x, x.y, nzero));
  }
  static __device__ __forceinline__ double2 total(const Acc& a) { return a.total(); }
};

// FP32 with Kahan compensation (AccF on pairs; c is kept negated)
template <>
struct Multi<float> {
  using X = f2;
  struct Acc {
    f2 a, nc;
    __device__ void zero() { a = nc = 0ull; }
  };
  struct Rec {
    uint32_t flip;
    float v;
  };
  using W = f2;
  static __device__ __forceinline__ Rec record(uint32_t flip, float v) { return {flip, v}; }
  template <bool IM>
  static __device__ __forceinline__ W operand(float v) {
    return pk(IM ? -v : v, v);
  }
  template <bool IM>
  static __device__ __forceinline__ W operand(const Rec& r) {
    return operand<IM>(r.v);
  }
  template <bool IM>
  static __device__ __forceinline__ void mac(Acc& a, const W& w, X x) {
    if constexpr (IM) x = swp(x);
    const f2 y = fma2(w, x, a.nc);
    const f2 s = add2(a.a, y);
    a.nc = sub2(y, sub2(s, a.a));
    a.a = s;
  }
  static __device__ __forceinline__ void set(Acc& a, float d, X x, double) {
    a.a = mul2(pk(d, d), x);
    a.nc = 0ull;
  }
  static __device__ __forceinline__ void set(Acc& a, float2 d, X x, double) {
    AccF t;
    t.set(d, upk(x));
    a.a = pk(t.re, t.im);
    a.nc = 0ull;
  }
  static __device__ __forceinline__ float2 total(const Acc& a) { return upk(add2(a.a, a.nc)); }
};

// double-float (AccFF on pairs)
template <>
struct Multi<DF> {
  struct X {
    f2 h, l;  // (re hi, im hi), (re lo, im lo)
  };
  struct Acc {
    f2 h, l;
    __device__ void zero() { h = l = 0ull; }
  };
  struct Rec {
    uint32_t flip;
    float vh, vl;
    uint32_t pad;
  };
  struct W {
    f2 h, nh, l;
  };
  static __device__ __forceinline__ Rec record(uint32_t flip, float2 v) { return {flip, v.x, v.y, 0}; }
  template <bool IM>
  static __device__ __forceinline__ W operand(float2 v) {
    return {pk(IM ? -v.x : v.x, v.x), pk(IM ? v.x : -v.x, -v.x), pk(IM ? -v.y : v.y, v.y)};
  }
  template <bool IM>
  static __device__ __forceinline__ W operand(const Rec& r) {
    return operand<IM>(make_float2(r.vh, r.vl));
  }
  static __device__ __forceinline__ void madd(Acc& a, const W& w, const X& x) {
    const f2 np = mul2(w.nh, x.h);  // -p
    f2 pe = fma2(w.h, x.h, np);
    pe = fma2(w.h, x.l, pe);
    pe = fma2(w.l, x.h, pe);
    const f2 s = sub2(a.h, np);
    const f2 nb = sub2(a.h, s);  // -bb
    const f2 err = add2(sub2(a.h, add2(s, nb)), sub2(nb, np));
    a.l = add2(a.l, add2(err, pe));
    a.h = s;
  }
  template <bool IM>
  static __device__ __forceinline__ void mac(Acc& a, const W& w, X x) {
    if constexpr (IM) {
      x.h = swp(x.h);
      x.l = swp(x.l);
    }
    madd(a, w, x);
  }
  static __device__ __forceinline__ void set(Acc& a, float2 d, const X& x, double) {
    const f2 h = pk(d.x, d.x);
    a.h = mul2(h, x.h);
    f2 pe = fma2(h, x.h, mul2(pk(-d.x, -d.x), x.h));
    pe = fma2(h, x.l, pe);
    a.l = fma2(pk(d.y, d.y), x.h, pe);
  }
  static __device__ __forceinline__ void set(Acc& a, float4 d, const X& x, double) {
    a.zero();
    madd(a, operand<false>(make_float2(d.x, d.y)), x);
    mac<true>(a, operand<true>(make_float2(d.z, d.w)), x);
  }
  static __device__ __forceinline__ float4 total(const Acc& a) {
    const float2 h = upk(a.h), l = upk(a.l);
    return make_float4(h.x, l.x, h.y, l.y);
  }
};

// One element, and 32 bytes of consecutive ones at a 32-byte aligned address.
__device__ __forceinline__ double2 ld_one(const double2* p) { return __ldg(p); }
__device__ __forceinline__ f2 ld_one(const f2* p) { return __ldg(p); }
__device__ __forceinline__ Multi<DF>::X ld_one(const Multi<DF>::X* p) {
  const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2*>(p));
  return {q.x, q.y};
}
__device__ __forceinline__ void ld_32(const double2* p, double2* o) {
    asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
        : "=d"(o[0].x), "=d"(o[0].y), "=d"(o[1].x), "=d"(o[1].y)
        : "l"(p));
}
__device__ __forceinline__ void ld_32(const f2* p, f2* o) {
  asm("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(o[0]), "=l"(o[1]), "=l"(o[2]), "=l"(o[3]) : "l"(p));
}
__device__ __forceinline__ void ld_32(const Multi<DF>::X* p, Multi<DF>::X* o) {
    asm("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];"
        : "=l"(o[0].h), "=l"(o[0].l), "=l"(o[1].h), "=l"(o[1].l)
        : "l"(p));
}
// NI elements es apart; WIDE: contiguous and 32-byte aligned
template <typename X, int NI, bool WIDE>
__device__ __forceinline__ void ld_block(const X* p, int64_t es, X (&o)[NI]) {
  if constexpr (WIDE) {
#pragma unroll
    for (int h = 0; h < NI; h += 32 / (int)sizeof(X)) ld_32(p + h, o + h);
  } else {
#pragma unroll
    for (int e = 0; e < NI; ++e) o[e] = ld_one(p + e * es);
  }
}
// results: 32-byte loads and stores
__device__ __forceinline__ void ldy_32(const double2* p, double2* o) {
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(o[0].x), "=d"(o[0].y), "=d"(o[1].x), "=d"(o[1].y)
                 : "l"(p));
}
__device__ __forceinline__ void ldy_32(const float2* p, float2* o) {
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(o[0].x), "=f"(o[0].y), "=f"(o[1].x), "=f"(o[1].y), "=f"(o[2].x), "=f"(o[2].y), "=f"(o[3].x),
                 "=f"(o[3].y)
               : "l"(p));
}
__device__ __forceinline__ void sty_32(double2* p, const double2* o) {
  asm volatile("st.global.v4.f64 [%4], {%0,%1,%2,%3};" ::"d"(o[0].x), "d"(o[0].y), "d"(o[1].x), "d"(o[1].y), "l"(p)
               : "memory");
}
__device__ __forceinline__ void sty_32(float2* p, const float2* o) {
  asm volatile("st.global.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"f"(o[0].x), "f"(o[0].y), "f"(o[1].x),
               "f"(o[1].y), "f"(o[2].x), "f"(o[2].y), "f"(o[3].x), "f"(o[3].y), "l"(p)
               : "memory");
}
// the merged diagonal's values at two consecutive indices (an even first one)
__device__ __forceinline__ void ld_diag(const double* p, double* d) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p));
  d[0] = a.x;
  d[1] = a.y;
}
__device__ __forceinline__ void ld_diag(const float* p, float* d) {
  const float2 a = __ldg(reinterpret_cast<const float2*>(p));
  d[0] = a.x;
  d[1] = a.y;
}
__device__ __forceinline__ void ld_diag(const float2* p, float2* d) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p));
  d[0] = make_float2(a.x, a.y);
  d[1] = make_float2(a.z, a.w);
}
template <typename DT>
__device__ __forceinline__ void ld_diag(const DT* p, DT* d) {
  d[0] = __ldg(p);
  d[1] = __ldg(p + 1);
}

// y block = alpha * acc + beta * y block
template <typename R, int NI, bool WIDE, int BMODE>
__device__ __forceinline__ void combine_block(typename Cx<R>::T* yp, int64_t yes,
                                              const typename Multi<R>::Acc (&acc)[NI], typename Cx<R>::T alpha,
                                              typename Cx<R>::T beta, double nzero) {
  typename Cx<R>::T o[NI];
  if constexpr (BMODE != 0) {
    if constexpr (WIDE) {
#pragma unroll
      for (int h = 0; h < NI; h += 32 / (int)sizeof(o[0])) ldy_32(yp + h, o + h);
    } else {
#pragma unroll
      for (int e = 0; e < NI; ++e) o[e] = yp[e * yes];
    }
  }
#pragma unroll
  for (int e = 0; e < NI; ++e) combine_nz<BMODE>(&o[e], Multi<R>::total(acc[e]), alpha, beta, nzero);
  if constexpr (WIDE) {
#pragma unroll
    for (int h = 0; h < NI; h += 32 / (int)sizeof(o[0])) sty_32(yp + h, o + h);
  } else {
#pragma unroll
    for (int e = 0; e < NI; ++e) yp[e * yes] = o[e];
  }
}

// acc[e] += v_e * u[e ^ LOW] for the indices e of a thread where the group, whose
// record is f, has a stored entry.
template <typename R, int NI, bool IM, int LOW>
__device__ __forceinline__ void low_group(typename Multi<R>::Acc (&acc)[NI], const typename Multi<R>::X (&u)[NI],
                                          const int4& f, const typename Ell<R, true>::T* ell, uint32_t J0,
                                          const GatherView& g) {
  using M = Multi<R>;
#pragma unroll
  for (int e = 0; e < NI; ++e) {
    if (kDebugBounds && out_of_range((int64_t)f.z + multi_row<true>(f, J0 + e), g.ell_slots, g.status)) continue;
    const auto v = Ell<R, true>::v(ell[f.z + multi_row<true>(f, J0 + e)]);
    int turn = nz(v) ? 1 : 0;
    if constexpr (std::is_same<R, double>::value) {
      // a loop of at most one turn: a branch that stays one
      asm volatile("" : "+r"(turn));
#pragma unroll 1
      while (turn) {
        M::template mac<IM>(acc[e], M::template operand<IM>(v), u[e ^ LOW]);
        turn = 0;
        asm volatile("" : "+r"(turn));
      }
    } else {
      if (turn) M::template mac<IM>(acc[e], M::template operand<IM>(v), u[e ^ LOW]);
    }
  }
}

constexpr int kFlipThreads = 128;
// resident blocks per SM asked of the compiler: the FP32 forms wait on loads, and
// at most 64 registers a thread (16 warps more) beats the few spills they cost
// (16 spins on 51 kets, ComplexF32, 41.4 -> 35.2 us; 20 spins, double-float, 42.6
// -> 39.9); the FP64 form is bound by its pipe
template <typename R>
struct MultiOcc {
  static constexpr int value = std::is_same<R, double>::value ? 1 : 8;
};

// One launch block: blockDim.x / ls index blocks of NI indices x the vector sets
// (ls vectors each, one per lane group) kper * blockIdx.y ... of kper.
template <typename R, int VM, int NI, bool WIDE, int BMODE>
__global__ void __launch_bounds__(kFlipThreads, MultiOcc<R>::value) k_gather_m(GatherView g, const void* __restrict__ xv, int64_t xes, int64_t xcs,
                                                  typename Cx<R>::T* __restrict__ y, int64_t yes, int64_t ycs,
                                                  int ncols, int kper, typename Cx<R>::T alpha,
                                                  typename Cx<R>::T beta) {
  using M = Multi<R>;
  using X = typename M::X;
  using Rec = typename M::Rec;
  static_assert(NI * sizeof(X) % 32 == 0, "a thread's block of inputs is read in 32-byte pieces");
  using ET = typename Ell<R, true>::T;
  using DT = typename Val<R, VM == kReal>::T;  // merged diagonal
  constexpr bool PH = VM == kPhased;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_enter();
  // the groups' row records, their flips with the current values, the slots when staged
  int4* rec = reinterpret_cast<int4*>(smem_raw);
  Rec* fl = reinterpret_cast<Rec*>(rec + g.ngroups);
  const ET* ell = static_cast<const ET*>(g.ell);
  for (int i = threadIdx.x; i < g.ngroups; i += blockDim.x) {
    int4 f = g.mrec[2 * i];
    const int rows = f.w;  // at most 32
    f.w = 0;
    for (int r = 0; r < rows; ++r) {
      if (kDebugBounds && out_of_range((int64_t)f.z + r, g.ell_slots, g.status)) continue;
      f.w |= (nz(Ell<R, true>::v(ell[f.z + r])) ? 1 : 0) << r;
    }
    rec[i] = f;
    const int4 q = g.mrec[2 * i + 1];
    fl[i] = M::record((uint32_t)q.x, Ell<R, true>::v(ell[kDebugBounds && out_of_range(q.y, g.ell_slots, g.status) ? 0 : q.y]));
  }
  if (g.ell_smem) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(smem_raw + (size_t)g.ngroups * (sizeof(int4) + 16));
    const uint32_t* src = reinterpret_cast<const uint32_t*>(g.ell);
    const int words = g.ell_slots * (int)(sizeof(ET) / 4);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    ell = reinterpret_cast<const ET*>(dst);
  }
  __syncthreads();

  const int ls = g.lane_split;
  const int lsh = __ffs(ls) - 1, jsh = 5 - lsh;
  const int lane = threadIdx.x & 31;
  const uint32_t blk = g.jmul == 1u ? blockIdx.x : (blockIdx.x * g.jmul) % gridDim.x;
  const uint32_t J0 =
      NI * (blk * (blockDim.x >> lsh) + ((threadIdx.x >> 5) << jsh) + (lane & ((1u << jsh) - 1)));
  if (J0 >= g.m) return;
  // groups by position: [0, nlow_re) low real, [nlow_re, nlow) low imaginary,
  // [nlow, nre) real, [nre, ngroups) imaginary
  const int nlow = g.nlow, nre = PH ? g.nre : g.ngroups, nlow_re = PH ? g.nlow_re : g.nlow;
  uint32_t act_re = 0, act_im = 0;
  auto activity = [&](auto two) {
    constexpr bool TWO = decltype(two)::value;
#pragma unroll 4
    for (int k = nlow; k < nre; ++k) act_re |= multi_active<TWO>(rec[k], J0) << (k - nlow);
    if constexpr (PH) {
#pragma unroll 4
      for (int k = nre; k < g.ngroups; ++k) act_im |= multi_active<TWO>(rec[k], J0) << (k - nre);
    }
  };
  if (g.two_runs)
    activity(std::true_type{});
  else
    activity(std::false_type{});
  if (kDebugBounds) {  // groups whose block of inputs starts or ends outside the vector, or is not aligned, do not run
    auto inside = [&](uint32_t act, const Rec* r0) {
      for (uint32_t a = act; a; a &= a - 1) {
        const int b = __ffs((int)a) - 1;
        const uint32_t p = J0 ^ r0[b].flip;
        if (out_of_range((p & (NI - 1)) ? -1 : (int64_t)p + NI - 1, g.n, g.status)) act &= ~(1u << b);
      }
      return act;
    };
    act_re = inside(act_re, fl + nlow);
    if constexpr (PH) act_im = inside(act_im, fl + nre);
  }
  DT d[NI];
  if (g.has_diag) {
#pragma unroll
    for (int h = 0; h < NI; h += 2) ld_diag(static_cast<const DT*>(g.diag) + J0 + h, d + h);
  }
  typename Cx<R>::T al = alpha, be = beta;
  double nzero = -0.0;
  if constexpr (!std::is_same<R, float>::value) {
    al.x = in_register(alpha.x);
    al.y = in_register(alpha.y);
    be.x = in_register(beta.x);
    be.y = in_register(beta.y);
    nzero = in_register(-0.0);
  }
  const X* x = static_cast<const X*>(xv);
  const int c_end = min(ncols, (int)(blockIdx.y + 1) * kper * ls);
  for (int c = (int)blockIdx.y * kper * ls + (lane >> jsh); c < c_end; c += ls) {
    const X* xb = x + (int64_t)c * xcs;
    typename M::Acc acc[NI];
    if (g.has_diag) {
      X u[NI];
      ld_block<X, NI, WIDE>(xb + (int64_t)J0 * xes, xes, u);
#pragma unroll
      for (int e = 0; e < NI; ++e) M::set(acc[e], d[e], u[e], nzero);
    } else {
#pragma unroll
      for (int e = 0; e < NI; ++e) acc[e].zero();
    }
    auto low = [&](auto imag, int k0, int k1) {
      constexpr bool IM = decltype(imag)::value;
#pragma unroll 1
      for (int k = k0; k < k1; ++k) {
        const int4 f = rec[k];
        const uint32_t flip = fl[k].flip;
        if (kDebugBounds && out_of_range((int64_t)(J0 ^ (flip & ~(uint32_t)(NI - 1))) + NI - 1, g.n, g.status)) continue;
        X u[NI];
        ld_block<X, NI, WIDE>(xb + (int64_t)(J0 ^ (flip & ~(uint32_t)(NI - 1))) * xes, xes, u);
        switch (flip & (NI - 1)) {
          case 0: low_group<R, NI, IM, 0>(acc, u, f, ell, J0, g); break;
          case 1: low_group<R, NI, IM, 1>(acc, u, f, ell, J0, g); break;
          case 2: if constexpr (NI > 2) low_group<R, NI, IM, 2>(acc, u, f, ell, J0, g); break;
          default: if constexpr (NI > 2) low_group<R, NI, IM, 3>(acc, u, f, ell, J0, g);
        }
      }
    };
    low(std::false_type{}, 0, nlow_re);
    if constexpr (PH) low(std::true_type{}, nlow_re, nlow);
    // the active groups of a mask one by one, the next one's inputs in flight
    auto high = [&](auto imag, uint32_t act, const Rec* r0) {
      constexpr bool IM = decltype(imag)::value;
      struct Part {
        typename M::W w;
        X u[NI];
      };
      auto fetch = [&](Part& p) {
        const Rec r = r0[__ffs((int)act) - 1];
        act &= act - 1;
        p.w = M::template operand<IM>(r);
        ld_block<X, NI, WIDE>(xb + (int64_t)(J0 ^ r.flip) * xes, xes, p.u);
      };
      auto use = [&](const Part& p) {
#pragma unroll
        for (int e = 0; e < NI; ++e) M::template mac<IM>(acc[e], p.w, p.u[e]);
      };
      if (!act) return;
      Part a, b;
      fetch(a);
      while (true) {
        const bool more_b = act != 0;
        if (more_b) fetch(b);
        use(a);
        if (!more_b) break;
        const bool more_a = act != 0;
        if (more_a) fetch(a);
        use(b);
        if (!more_a) break;
      }
    };
    high(std::false_type{}, act_re, fl + nlow);
    if constexpr (PH) high(std::true_type{}, act_im, fl + nre);
    combine_block<R, NI, WIDE, BMODE>(y + (int64_t)J0 * yes + (int64_t)c * ycs, yes, acc, al, be, nzero);
  }
}

}  // namespace gather
}  // namespace qob
