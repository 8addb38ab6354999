// k_slice.cu -- dense operators and the mode products of dense LazyTensor factors
// (mul! on a DenseOperator, src/operators_dense.jl:394-396, and
// _tp_matmul_first!/_mid!/_last!, src/operators_lazytensor.jl:281-428) as exact
// integer products on the 5th-generation tensor cores (tcgen05.mma kind::f16,
// bf16 operands, FP32 accumulators in tensor memory).
//
// GB300's FP64 pipe gives 1.2 TFLOP/s, its FP32 pipes 78, its tensor cores 1900 in
// bf16.  A bf16 number holds every integer up to 256, so each operand is cut into
// S signed 8-bit digits of a fixed-point number (Ozaki, Ogita, Oishi & Rump 2012,
// "Error-free transformations of matrix multiplication"): row i of the matrix
// relative to 2^ea(i), the power of two above its largest component, vector c
// relative to 2^ex(c), both per chunk of at most 256 contracted indices, 8 S - 2 bits
// below it and truncated there.  The pairs (i, j) of digits with i + j = d < S are summed in
// one FP32 accumulator, a diagonal, as integers; the S diagonals are added as 64-bit
// integers and rounded once.  S = 8 in ComplexF64 (62 bits), 7 in double-float (54), 4 in
// ComplexF32 (30).
//
// What the digits leave out is small against a row's and a vector's largest
// components, and the products of those may be absent from a sum: a product is made of
// digits only where a bound says that little is lost.  Per row or vector and chunk the split
// kernel keeps the sum of the magnitudes, of the digits squared, and how many
// components reach 2^-1 .. 2^-6 of the power of two.  The first two bound the error
// (digit_error: the truncation of either side, the diagonals from S on; nothing rounds in an
// accumulator below 2^24), the counts bound sum |a| |x| from below (overlap).  The error's bound has to be
// at most 8 units (2^-53) of that in ComplexF64, 32 (2^-24) in ComplexF32, 64 (2^-48) in
// double-float, for every row, vector and chunk, Re and Im apart: what a chain of
// multiply-adds over 4, 16 and 32 terms is bounded by, where the shortest sums here have 32
// pairs.  The error itself is far below: over Gaussian, uniform, constant, lognormal, graded,
// cancelling and sparse entries that pass, 64 or 256 of them (digits and chains emulated on the
// CPU), 0.3 to 0.9 units in relative l2 in ComplexF32 where the chain has 1.8 to 7, and up to
// 1 against 16 units of sum |a| |x|.  Gaussian entries (matrices of 32 to 4096 rows) reach 0.9
// of the limits and 650 of the 1024 that keep a diagonal exact.
//
// A tile of vectors that fails (graded ones, sparse ones, components that are not finite or
// far from 1) is left to the FMA kernels: the split kernel flags it, the GEMM does not store
// it and the FMA kernels, launched behind it, compute the flagged tiles alone (FmaGate).  A
// matrix that fails with vectors of ones has no planes.
//
// Layout.  The complex product is one real GEMM as in k_tc32.cu: rows 2i, 2i + 1 of
// a 128-row tile hold Re and Im of matrix row i, rows j and BN/2 + j of a BN-row
// tile Re and Im of vector j.  One k step (16 contracted indices) of a tile is S
// digit planes.  The MMA reads a plane of (rows x 16) bf16 as 8-row groups of two
// 128-byte core matrices, without a swizzle.  The vectors' planes are stored that
// way; the matrix's, read for every column tile or streamed once from memory,
// as bytes in the same order (half the traffic: the matrix's own size again), and
// four warps widen them to bf16 in shared memory.  Since digit planes 0 .. S - 1 - i
// of the vectors follow one another, digit i of the matrix times all of them is one
// MMA of N = (S - i) BN columns (two above 256) into the accumulators of the
// diagonals i .. S - 1.
//
// Block: warp 0 issues the copies, warp 1 owns the tensor memory and
// issues the MMAs, warp 2 does its waiting (an mbarrier wait by the thread that
// issued MMAs lasts until they are done; the two meet at a named barrier instead),
// 6 or 8 warps widen digits and 16 or 8 add up the diagonals and write, beside the
// next unit's MMAs where the tensor memory holds two sets of accumulators.  Units (column tile, row tile, chunk) in equal runs
// over one block per SM; a run's part of a row tile either covers it (written to y)
// or goes to a partial product that k_slice_reduce adds in chunk order.  Waits are
// bounded as in k_tc32.cu.
// Measured (a call among others, Gaussian entries, FMA kernels -> this; one GB300): two mode products
// with 199 x 199 and 201 x 201 factors on 15 kets, ComplexF64 4791 -> 343 us,
// double-float 1412 -> 322, ComplexF32 475 -> 175; a 4096 x 4096 operator on 16 kets
// 1743 -> 118, 672 -> 111, 161 -> 70.  Error against 128-bit products: ComplexF64
// 1e-16 (FMA 4e-16), double-float 1e-15 (4e-14), ComplexF32 6e-8 (2e-7).  Bound by
// the tensor pipe's rate on short MMAs (80 to 110 cycles each up to N = 160) with
// their commits and, on many columns, by adding up the diagonals (about 9000 cycles
// per unit beside 13 k steps of 1800).  bf16 planes of the matrix in memory instead of
// bytes: 370 us and 122 us in ComplexF64.
#include <cuda_runtime.h>

#include <algorithm>

#include "k_gather.cuh"  // double-float helpers
#include "launch.cuh"
#include "qob_internal.h"
#include "tcgen05.cuh"

namespace qob {

namespace {

constexpr int kSlChunk = 16;      // k steps of 16 in a chunk, at most
constexpr int kSlRows = 128;      // real matrix rows of a tile

// The chunks of nkb k steps are of equal length but for one step: chunk c is the k
// steps from chunk_start(c) to chunk_start(c + 1).
__host__ __device__ inline int chunk_start(int c, int nkb, int nch) { return (int)((int64_t)c * nkb / nch); }

// K-major operand without swizzle: core matrices of 8 rows x 16 bytes, the two of
// a k step 128 bytes apart, 8-row groups 256 bytes apart; descriptor version 1
__device__ __forceinline__ uint64_t plane_desc(const void* p) {
  const uint64_t a = (saddr(p) & 0x3FFFFu) >> 4;
  return a | (uint64_t(128 >> 4) << 16) | (uint64_t(256 >> 4) << 32) | (uint64_t(1) << 46);
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[4]) {  // completion: tcgen05.wait::ld
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[2]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
}
// two signed bytes (sel picks them into the low bytes of the halves) as bf16: the
// low seven bits on 128.0 less 128.0, or 256.0 where the sign bit is set (0x4300
// + 0x80 is 256.0), both exact
__device__ __forceinline__ uint32_t widen2(uint32_t bytes, uint32_t sel) {
  const uint32_t h = __byte_perm(bytes, 0x43434343u, sel);
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(h & 0xff7fff7fu), "r"(h & 0xff80ff80u));
  return r;
}

// Digits per form, element types, and the fixed-point number of a component:
// |v| < 2^e times 2^kBits, truncated towards zero.
template <int FORM>  // QOB_C128, QOB_C64, QOB_C128X
struct Sl;
template <>
struct Sl<QOB_C128> {
  static constexpr int S = 8;
  using V = double2;  // vectors
  using M = double2;  // the stored matrix
};
template <>
struct Sl<QOB_C128X> {
  static constexpr int S = 7;
  using V = double2;
  using M = float4;
};
template <>
struct Sl<QOB_C64> {
  static constexpr int S = 4;
  using V = float2;
  using M = float2;
};
template <int S>
constexpr int kBits = 8 * S - 2;

// bits of a component's magnitude, its biased exponent, and whether it is finite
__device__ __forceinline__ uint32_t mag_hi(double v) { return (uint32_t)__double2hiint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t mag_hi(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ bool is_nonzero(double v) { return (mag_hi(v) | (uint32_t)__double2loint(v)) != 0u; }
__device__ __forceinline__ bool is_nonzero(float v) { return mag_hi(v) != 0u; }
// unbiased exponent e with |v| < 2^e from the high word's bits (subnormals count as the smallest normal)
template <typename T>
__device__ __forceinline__ int exp_above(uint32_t hi) {
  return sizeof(T) == 8 ? (int)(hi >> 20) - 1022 : (int)(hi >> 23) - 126;
}
// |eA|, |eX| beyond which a product or its scale could leave the type's range
template <typename T>
constexpr int kExpMax = sizeof(T) == 8 ? 400 : 50;

template <int S>
__device__ __forceinline__ long long fixed_point(double v, int e) {
  const uint32_t hi = mag_hi(v);
  const int ev = (int)(hi >> 20);
  const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (ev ? 0x100000u : 0u)) << 32) |
                               (uint32_t)__double2loint(v);  // 53 bits, |v| = m 2^(max(ev, 1) - 1075)
  const int sh = kBits<S> - 53 - (e - ((ev ? ev : 1) - 1022));  // m 2^sh
  long long f = sh >= 0 ? (long long)(m << sh) : sh > -64 ? (long long)(m >> -sh) : 0;
  return __double2hiint(v) < 0 ? -f : f;
}
template <int S>
__device__ __forceinline__ int fixed_point(float v, int e) {
  const uint32_t hi = mag_hi(v);
  const int ev = (int)(hi >> 23);
  const uint32_t m = (hi & 0x7fffffu) | (ev ? 0x800000u : 0u);
  const int sh = kBits<S> - 24 - (e - ((ev ? ev : 1) - 126));
  const int f = sh >= 0 ? (int)(m << sh) : sh > -32 ? (int)(m >> -sh) : 0;
  return __float_as_int(v) < 0 ? -f : f;
}
// All signed digits of f at once: f + sum 128 256^s has the bytes d_s + 128.
__device__ __forceinline__ uint2 digit_bytes(long long f) {
  const unsigned long long g = (unsigned long long)f + 0x8080808080808080ull;
  return make_uint2((uint32_t)g, (uint32_t)(g >> 32));
}
__device__ __forceinline__ uint2 digit_bytes(int f) { return make_uint2((uint32_t)f + 0x80808080u, 0x80808080u); }
__device__ __forceinline__ unsigned long long magnitude(long long f) { return f < 0 ? -f : f; }
__device__ __forceinline__ uint32_t magnitude(int f) { return f < 0 ? -f : f; }
// binary digits above the first of a magnitude's kBits
template <int S>
__device__ __forceinline__ int lead(unsigned long long mag) {
  return __clzll((long long)mag) - (64 - kBits<S>);
}
template <int S>
__device__ __forceinline__ int lead(uint32_t mag) {
  return __clz((int)mag) - (32 - kBits<S>);
}
// digits b of p and q, as two bytes (of d + 128)
__device__ __forceinline__ uint32_t digit_pair(uint2 p, uint2 q, int b) {
  return __byte_perm(b < 4 ? p.x : p.y, b < 4 ? q.x : q.y, (b & 3) | (((b & 3) + 4) << 4));
}
// digit b as the bits of a float: 2^23 + d + 128, less 2^23 + 128, exact
__device__ __forceinline__ uint32_t digit_float(uint2 p, int b) {
  return __float_as_uint(__uint_as_float(__byte_perm(b < 4 ? p.x : p.y, 0x4b000000u, 0x7440 | (b & 3))) - 8388736.f);
}

__device__ __forceinline__ double2 as_value(double2 v) { return v; }
__device__ __forceinline__ float2 as_value(float2 v) { return v; }
__device__ __forceinline__ double2 as_value(float4 v) {  // (re hi, re lo, im hi, im lo)
  return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
}

// What a row of the matrix or a vector tells about a chunk, the worst over the rows
// (Re and Im each one) of a tile or of the whole matrix.  In units of 2^e, the power of two above the
// row's largest component, |v| its components' magnitudes:
struct SliceSide {
  float n1;     // sum of |v|, at most
  float t;      // sqrt(sum of all digits squared) / 128, at most
  int c[6];     // components with |v| >= 1/2, 1/4, .. 1/64, at least
};
constexpr int kLevels = 6;

// Bound on the error of the digit products allowed, in 2^-kBits of sum |a| |x|: 8 units of 2^-53 in
// ComplexF64, 32 of 2^-24 in ComplexF32, 64 of 2^-48 in double-float.
template <int FORM>
constexpr float kSlLimit = FORM == QOB_C64 ? 2048.f : 4096.f;

// A lower bound of sum |a| |x| over n indices, term (i, j): at least n less the components
// of either side below their thresholds, 2^-(i + 1) and 2^-(j + 1), lie above both, and
// the thresholds' differences add up to the largest that a component reaches.
__host__ __device__ inline float overlap(const SliceSide& a, const SliceSide& x, int n, int i, int j) {
  const float wi = 1.f / (float)(i + 1 < kLevels ? 4 << i : 2 << i), wj = 1.f / (float)(j + 1 < kLevels ? 4 << j : 2 << j);
  const int both = a.c[i] + x.c[j] - n;
  return both > 0 ? wi * wj * (float)both : 0.f;
}
// An upper bound of the digit products' error on n indices, in 2^-kBits of the row's times the vector's
// power of two: each side's truncation, below 1, times the other's components, and the
// diagonals from S on (|sum of d_i d_(S-i)| <= |a's digits| |x's digits|, the ones after it
// 256 times smaller each).  Infinite where a diagonal's sum could leave 2^24, the
// integers that an FP32 accumulator holds.
__host__ __device__ inline float digit_error(const SliceSide& a, const SliceSide& x) {
  const float t = a.t * x.t;
  return t > 1024.f ? 3e38f : a.n1 + x.n1 + 1.01f * t;
}

// Digit planes of one tile's chunk: ROWS / 2 vectors (columns of x, or rows of the
// matrix with INTER) x up to 256 contracted indices.  blockIdx.x: tile, blockIdx.y:
// chunk.  exps[(tile nch + chunk) ROWS / 2 + vector]: the power of two above its
// largest component.  flags[tile nch + chunk]: 1 where the tile is left to the FMA
// form, by its exponents or, with the matrix's chunks in `other`, by the bounds above;
// own[tile nch + chunk]: the tile's side of them.  kfast: threads read along the contracted index.
constexpr int split_threads(int rows) { return rows == 32 ? 512 : 1024; }
template <int FORM, int ROWS, bool INTER, typename IN>
__global__ void __launch_bounds__(split_threads(ROWS)) k_slice_split(const IN* __restrict__ x, int64_t n, int64_t es, TcColMap map,
                                                     int64_t nvec, int nkb, int kfast, int sub,
                                                     unsigned char* __restrict__ out, int* __restrict__ exps,
                                                     int* __restrict__ flags, int* __restrict__ any,
                                                     const SliceSide* __restrict__ other, SliceSide* __restrict__ own) {
  constexpr int S = Sl<FORM>::S, H = ROWS / 2, kSlSplit = split_threads(ROWS);
  using C2 = decltype(as_value(IN{}));
  using T = decltype(C2{}.x);
  extern __shared__ __align__(16) unsigned char sl_smem[];
  __shared__ int ex[H], some[H];  // some: bit 0: nonzero real parts, bit 1: imaginary ones
  __shared__ int bad;
  __shared__ int64_t off[H];
  // per real row: components by their level, three counts of 10 bits a word, sum |v| in 2^-14, digits squared
  __shared__ uint32_t cnt_hi[ROWS], cnt_lo[ROWS], sum1[ROWS], sum2[ROWS];
  __shared__ SliceSide side;
  __shared__ int worst1, worst2;
  pdl_enter();
  const int nch = gridDim.y, kb0 = chunk_start(blockIdx.y, nkb, nch), nks = chunk_start(blockIdx.y + 1, nkb, nch) - kb0;
  const int64_t k0 = (int64_t)kb0 * 16;
  const int pitch = sub * 16 + 1;  // sub k steps are staged at a time
  C2* t = reinterpret_cast<C2*>(sl_smem);  // [vector][k]
  const int64_t v0 = (int64_t)blockIdx.x * H;
  if (threadIdx.x == 0) bad = worst1 = worst2 = 0;
  if (any && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) *any = 0;  // set by the GEMM
  if (threadIdx.x < kLevels) side.c[threadIdx.x] = kSlChunk * 16;
  if (threadIdx.x < ROWS) cnt_hi[threadIdx.x] = cnt_lo[threadIdx.x] = sum1[threadIdx.x] = sum2[threadIdx.x] = 0u;
  if (threadIdx.x < H) off[threadIdx.x] = v0 + threadIdx.x < nvec ? tc_col_offset(map, v0 + threadIdx.x) : -1;
  auto stage = [&](int b0) {  // k steps b0 .. of the chunk
    const int nk = min(sub, nks - b0) * 16;
    __syncthreads();
    // four elements of a thread in flight
    for (int i0 = threadIdx.x; i0 < H * nk; i0 += 4 * kSlSplit) {
      C2 val[4];
      int at[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * kSlSplit;
        val[u].x = val[u].y = 0;
        at[u] = -1;
        if (i >= H * nk) continue;
        const int q = i / (kfast ? nk : H), r = i - q * (kfast ? nk : H);
        const int v = kfast ? q : r, k = kfast ? r : q;
        const int64_t kg = k0 + b0 * 16 + k;
        at[u] = v * pitch + k;
        if (off[v] >= 0 && kg < n) val[u] = as_value(x[off[v] + kg * es]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (at[u] >= 0) t[at[u]] = val[u];
    }
    __syncthreads();
    return nk;
  };
  // largest component of each vector, a few threads per vector
  constexpr int PER = kSlSplit / H;
  static_assert(PER * H == kSlSplit && PER <= 32, "threads of a vector in one warp");
  {
    const int v = threadIdx.x / PER, part = threadIdx.x % PER;
    uint32_t mx = 0u, nonzero = 0u;
    for (int b0 = 0; b0 < nks; b0 += sub) {
      const int nk = stage(b0);
      for (int k = part; k < nk; k += PER) {
        const C2 c = t[v * pitch + k];
        mx = max(mx, max(mag_hi(c.x), mag_hi(c.y)));
        nonzero |= (is_nonzero(c.x) ? 1u : 0u) | (is_nonzero(c.y) ? 2u : 0u);
      }
    }
#pragma unroll
    for (int w = PER / 2; w > 0; w >>= 1) {
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, w));
      nonzero |= __shfl_xor_sync(0xffffffffu, nonzero, w);
    }
    if (part == 0) {
      const int e = nonzero ? exp_above<T>(mx) : 0;
      ex[v] = e;
      some[v] = (int)nonzero;
      if (nonzero && (e > kExpMax<T> || e < -kExpMax<T>)) atomicExch(&bad, 1);
    }
  }
  __syncthreads();
  const int64_t tile = (int64_t)blockIdx.x * nch + blockIdx.y;
  if (threadIdx.x < H) exps[tile * H + threadIdx.x] = ex[threadIdx.x];
  for (int b0 = 0; b0 < nks; b0 += sub) {
    const int nk = sub < nks ? stage(b0) : nks * 16;  // staged already when it is all of the chunk
    // 8 contracted indices of one real row per task: a store of 16 (INTER: 8) bytes per plane
    constexpr int kRow = INTER ? 16 : 32;  // bytes of a row in a plane
    unsigned char* o = out + ((int64_t)blockIdx.x * nkb + kb0 + b0) * (int64_t)(S * ROWS * kRow);
    for (int i = threadIdx.x; i < ROWS * nk / 8; i += kSlSplit) {
      const int r = i % ROWS, kc = i / ROWS;  // real row, run of 8 indices
      const int v = INTER ? r >> 1 : r % H;
      const bool im = INTER ? (r & 1) : r >= H;
      uint32_t w[S][INTER ? 2 : 4];
      unsigned long long levels = 0ull;
      uint32_t n1 = 0u;
      int n2 = 0;
#pragma unroll
      for (int p = 0; p < 4; p += 2) {
        uint2 g[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const C2 c = t[v * pitch + kc * 8 + 2 * p + e];
          const auto f = fixed_point<S>(im ? c.y : c.x, ex[v]);
          const auto mag = magnitude(f);
          g[e] = digit_bytes(f);
          levels += 1ull << (10 * min(lead<S>(mag), kLevels));
          n1 += (uint32_t)(mag >> (kBits<S> - 14));
          const int lo = (int)(g[e].x ^ 0x80808080u), hi = (int)((g[e].y ^ 0x80808080u) & (S == 8 ? ~0u : 0xffffffu));
          n2 = __dp4a(lo, lo, n2);
          if (S > 4) n2 = __dp4a(hi, hi, n2);
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const int d = S - 1 - s;
          if constexpr (INTER) {
            w[s][p >> 1] =
                __byte_perm(digit_pair(g[0], g[1], d), digit_pair(g[2], g[3], d), 0x5410) ^ 0x80808080u;
          } else {  // bf16: the upper half of a float
            w[s][p] = __byte_perm(digit_float(g[0], d), digit_float(g[1], d), 0x7632);
            w[s][p + 1] = __byte_perm(digit_float(g[2], d), digit_float(g[3], d), 0x7632);
          }
        }
      }
      unsigned char* q = o + (int64_t)(kc >> 1) * (S * ROWS * kRow) + (r >> 3) * (8 * kRow) + (kc & 1) * (4 * kRow) +
                         (r & 7) * (kRow / 2);
#pragma unroll
      for (int s = 0; s < S; ++s) {
        if constexpr (INTER)
          *reinterpret_cast<uint2*>(q + s * (ROWS * kRow)) = make_uint2(w[s][0], w[s][1]);
        else
          *reinterpret_cast<uint4*>(q + s * (ROWS * kRow)) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
      }
      atomicAdd(&cnt_hi[r], (uint32_t)levels & 0x3fffffffu);
      atomicAdd(&cnt_lo[r], (uint32_t)(levels >> 30) & 0x3fffffffu);
      atomicAdd(&sum1[r], n1);
      atomicAdd(&sum2[r], (uint32_t)n2);
    }
  }
  __syncthreads();
  // the worst of the rows that are not zero
  const int valid = (int)min((int64_t)nks * 16, n - k0);
  if (threadIdx.x < ROWS) {
    const int r = threadIdx.x, v = INTER ? r >> 1 : r % H;
    const bool im = INTER ? (r & 1) : r >= H;
    const bool on = (some[v] >> (im ? 1 : 0)) & 1;
    int c = 0;
#pragma unroll
    for (int i = 0; i < kLevels; ++i) {
      c += (int)(((i < 3 ? cnt_hi[r] : cnt_lo[r]) >> (10 * (i % 3))) & 0x3ffu);
      const int least = __reduce_min_sync(0xffffffffu, on ? c : kSlChunk * 16);
      if ((r & 31) == 0) atomicMin(&side.c[i], least);
    }
    const int most1 = __reduce_max_sync(0xffffffffu, on ? (int)sum1[r] + valid : 0);  // each of its terms rounded up
    const int most2 = __reduce_max_sync(0xffffffffu, on ? (int)sum2[r] : 0);
    if ((r & 31) == 0) {
      atomicMax(&worst1, most1);
      atomicMax(&worst2, most2);
    }
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  SliceSide mine;
  mine.n1 = (float)worst1 * (1.f / 16384.f);
  mine.t = sqrtf((float)worst2) * (1.f / 128.f);
#pragma unroll
  for (int i = 0; i < kLevels; ++i) mine.c[i] = side.c[i];
  bool left = bad != 0;
  if (other) {
    const SliceSide a = other[blockIdx.y];
    float least = 0.f;
    for (int q = threadIdx.x; q < kLevels * kLevels; q += 32) least += overlap(a, mine, valid, q / kLevels, q % kLevels);
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) least += __shfl_xor_sync(0xffffffffu, least, w);
    left |= digit_error(a, mine) > kSlLimit<FORM> * least;
  }
  if (threadIdx.x == 0) {
    flags[tile] = left ? 1 : 0;
    if (own) own[tile] = mine;
  }
}

template <int FORM, int BN>
struct SlCfg {
  static constexpr int S = Sl<FORM>::S;
  static constexpr int kCols = S * BN;                       // columns of one set of accumulators
  static constexpr int kSets = 2 * kCols <= 512 ? 2 : 1;     // sets in the tensor memory
  // k steps of a widened buffer (one rendezvous and its commits, ~300 cycles, beside
  // 80 or more per MMA) and of a stage
  static constexpr int kG = S == 4 ? 2 : 1, kKs = 2;
  static constexpr int kA = S * kSlRows * 16, kB = S * BN * 32;  // one k step: bytes of the M side, planes of the N side
  static constexpr int kWideStep = S * kSlRows * 32;             // one k step of the M side, widened
  static constexpr int kWide = kG * kWideStep;
  static constexpr int kWides = BN == 32 ? 2 : 3;
  static constexpr int kStageA = kKs * kA, kStageB = kKs * kB;
  static constexpr int kWidenWarps = BN == 32 ? 8 : 6, kAddWarps = BN == 32 ? 8 : 16;
  static constexpr int kWiden = 32 * kWidenWarps, kWork = 32 * kAddWarps;
  static constexpr int kThreads = 96 + kWiden + kWork;
  static constexpr int kBars = 512;
  // the M side's ring is released as soon as it is widened, the N side's by the MMAs
  static constexpr int kRingB = BN == 32 ? 3 : 2;
  static constexpr int kRingA = (226 * 1024 - kBars - kWides * kWide - kRingB * kStageB) / kStageA < 8
                                    ? (226 * 1024 - kBars - kWides * kWide - kRingB * kStageB) / kStageA
                                    : 8;
  static constexpr size_t smem =
      128 + (size_t)kWides * kWide + (size_t)kRingA * kStageA + (size_t)kRingB * kStageB + kBars;
  static_assert(kRingA >= 2, "two stages at least");
  static_assert(8 * (2 * kRingA + 2 * kRingB + 2 * kWides + 2 * kSets + 1) + 8 <= kBars, "barrier area");
  static_assert(smem <= 227 * 1024, "shared memory of a block");
};

// H 2^(8 (S - 4)) + L: the sum of the diagonals in units of the last one's
struct Sum2 {
  long long h, l;
};
template <int S>
__device__ __forceinline__ Sum2 add_diagonals(const uint32_t (&d)[S]) {
  auto in = [&](int i) { return (long long)__float2int_rn(__uint_as_float(d[i])); };
  Sum2 r;
  r.h = in(0) * (1 << 24) + in(1) * (1 << 16) + in(2) * (1 << 8) + in(3);
  r.l = 0;
  if constexpr (S == 8) r.l = in(4) * (1 << 24) + in(5) * (1 << 16) + in(6) * (1 << 8) + in(7);
  if constexpr (S == 7) r.l = in(4) * (1 << 16) + in(5) * (1 << 8) + in(6);
  return r;
}
// the sum in units of 2^(e - 36 - 8 (S - 4)), rounded to nearest, without the FP64 pipe
template <int S>
__device__ __forceinline__ double sum_to_double(Sum2 v, int e) {
  constexpr int LB = 8 * (S - 4);               // bits of the low part's unit below the high one's
  long long g = v.h + (v.l >> LB);              // floor
  unsigned long long f = (unsigned long long)v.l << (64 - LB);  // fraction, in units of 2^-64
  const bool neg = g < 0;
  if (neg) {  // -(g + f): complement
    f = 0ull - f;
    g = ~g + (f == 0ull ? 1 : 0);
  }
  if (g == 0) {  // only a fraction
    g = (long long)(f >> 32);
    f <<= 32;
    e -= 32;
    if (g == 0) {
      g = (long long)(f >> 32);
      f = 0ull;
      e -= 32;
      if (g == 0) return 0.0;
    }
  }
  const int s = __clzll(g);  // 1 .. 63
  unsigned long long m = ((unsigned long long)g << s) | (f >> (64 - s));
  m = (m >> 11) + ((m >> 10) & 1ull);
  // value = m 2^(11 - s + e - 36): m has 53 bits
  const long long bits = ((long long)(1022 + 63 - s + e - 36) << 52) + (long long)m;
  return __longlong_as_double(bits | (neg ? (long long)0x8000000000000000ull : 0ll));
}

template <int FORM>
struct SlAcc {
  using T = double;
};
template <>
struct SlAcc<QOB_C64> {
  using T = float;
};

// part: partial products, [row tile][segment][column][complex row of the tile]
template <int FORM, int BN>
__global__ void __launch_bounds__(SlCfg<FORM, BN>::kThreads, 1)
    k_slice_gemm(const unsigned char* __restrict__ A, const int* __restrict__ ea, const unsigned char* __restrict__ B,
                 const int* __restrict__ ex, const int* __restrict__ flags, int* __restrict__ any, int* __restrict__ left, int64_t m, int mt, int64_t ncols, int nkb,
                 int nch, int per, int64_t units, int smax, int swap, typename Sl<FORM>::V* y, int64_t yes, TcColMap ym,
                 typename Sl<FORM>::V alpha, typename Sl<FORM>::V beta, typename Sl<FORM>::V* part, unsigned* status) {
  using C = SlCfg<FORM, BN>;
  using T = typename SlAcc<FORM>::T;
  constexpr int S = C::S, NA = C::kRingA, NM = C::kRingB, NW = C::kWides, NB = C::kSets, KS = C::kKs, G = C::kG, H = BN / 2;
  extern __shared__ __align__(16) unsigned char sl_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)sl_raw + 127) & ~(uintptr_t)127);
  unsigned char* ring_a = base + (size_t)NW * C::kWide;
  unsigned char* ring_b = ring_a + (size_t)NA * C::kStageA;
  uint64_t* afull = reinterpret_cast<uint64_t*>(ring_b + (size_t)NM * C::kStageB);
  uint64_t* aempty = afull + NA;  // a stage widened (count kWiden)
  uint64_t* bfull = aempty + NA;
  uint64_t* bempty = bfull + NM;
  uint64_t* wfull = bempty + NM;  // a k step of the matrix widened (count kWiden)
  uint64_t* wempty = wfull + NW;  // and read by its MMAs
  uint64_t* accf = wempty + NW;   // a unit's accumulators written
  uint64_t* acce = accf + NB;     // and read (count kWork)
  uint64_t* fin = acce + NB;      // every MMA issued has completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(fin + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t u0 = (int64_t)blockIdx.x * per;
  int nu = (int)(units - u0 < (int64_t)per ? units - u0 : (int64_t)per);
  const int ch_start = (int)(u0 % nch);
  auto steps = [&](int ch) { return chunk_start(ch + 1, nkb, nch) - chunk_start(ch, nkb, nch); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < NA; ++s) {
      bar_init(&afull[s], 1);
      bar_init(&aempty[s], C::kWiden);
    }
    for (int s = 0; s < NM; ++s) {
      bar_init(&bfull[s], 1);
      bar_init(&bempty[s], 1);
    }
    for (int s = 0; s < NW; ++s) {
      bar_init(&wfull[s], C::kWiden);
      bar_init(&wempty[s], 1);
    }
    for (int s = 0; s < NB; ++s) {
      bar_init(&accf[s], 1);
      bar_init(&acce[s], C::kWork);
    }
    bar_init(fin, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  {  // the tiles left to the FMA kernels; a run of nothing else is not done
    bool live = false;
    for (int64_t rt = u0 / nch + threadIdx.x; rt <= (u0 + nu - 1) / nch; rt += blockDim.x) {
      const int64_t vt = swap ? rt % mt : rt / mt;
      int f = 0;
      for (int j = 0; j < nch; ++j) f |= flags[vt * nch + j];
      left[vt] = f;  // by each of its blocks
      if (f) *any = 1;
      live |= f == 0;
    }
    if (!__syncthreads_or(live)) nu = 0;
  }

  // warps 1 and 2 meet; true when either asks to stop
  auto meet = [&](bool ask) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\tbar.red.or.pred p, 1, 64, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)ask)
        : "memory");
    return r != 0u;
  };
  // the roles below walk the same units and k steps: st counts stages, w widened k steps
  if (warp == 0) {
    if (lane == 0) {
      int64_t rt = u0 / nch;
      int ch = ch_start, st = 0;
      bool stop = false;
      for (int u = 0; u < nu && !stop; ++u) {
        const int64_t mti = rt % mt, ct = rt / mt;
        const int ks = steps(ch);
        for (int k = 0; k < ks; k += KS, ++st) {
          const int sa = st % NA, sb = st % NM;
          if ((st >= NA && !bar_wait(&aempty[sa], ((st / NA) - 1) & 1)) ||
              (st >= NM && !bar_wait(&bempty[sb], ((st / NM) - 1) & 1)) || *(volatile int*)abort_flag) {
            atomicExch(abort_flag, 1);
            stop = true;
            break;
          }
          const int64_t kb = chunk_start(ch, nkb, nch) + k;
          const uint32_t q = (uint32_t)min(KS, ks - k);
          bar_expect(&afull[sa], q * C::kA);
          bulk_copy(ring_a + (size_t)sa * C::kStageA, A + (mti * nkb + kb) * C::kA, q * C::kA, &afull[sa]);
          bar_expect(&bfull[sb], q * C::kB);
          bulk_copy(ring_b + (size_t)sb * C::kStageB, B + (ct * nkb + kb) * C::kB, q * C::kB, &bfull[sb]);
        }
        if (++ch == nch) {
          ch = 0;
          ++rt;
        }
      }
      // every copy issued has landed before the block's shared memory goes away
      for (int j = max(0, st - NA); j < st; ++j) bar_wait(&afull[j % NA], (j / NA) & 1);
      for (int j = max(0, st - NM); j < st; ++j) bar_wait(&bfull[j % NM], (j / NM) & 1);
    }
  } else if (warp == 1) {
    // kind::f16: FP32 accumulators, bf16 operands, both K-major, M = 128
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kSlRows >> 4) << 24);
    int ch = ch_start, st = 0, w = 0;
    bool stop = false;
    for (int u = 0; u < nu && !stop; ++u) {
      const int b = u % NB;
      const int ks = steps(ch);
      for (int k0 = 0; k0 < ks; k0 += G, ++w) {
        const int s = st % NM, c = w % NW, kn = min(G, ks - k0);
        const bool last = (k0 + G) % KS == 0 || k0 + G >= ks;  // of its stage
        if (meet(false)) {
          stop = true;
          break;
        }
        if (lane == 0) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t ad0 = plane_desc(base + (size_t)c * C::kWide);
          const uint64_t bd0 = plane_desc(ring_b + (size_t)s * C::kStageB + (k0 % KS) * C::kB);
          for (int k = 0; k < kn; ++k) {
            const uint64_t bd = bd0 + (uint64_t)(k * (C::kB / 16)), ak = ad0 + (uint64_t)(k * (C::kWideStep / 16));
#pragma unroll
            for (int i = 0; i < S; ++i) {
              const uint64_t ad = ak + (uint64_t)(i * (kSlRows * 32 / 16));
              const uint32_t acc = (i > 0 || k0 + k > 0) ? 1u : 0u;
#pragma unroll
              for (int n0 = 0; n0 < (S - i) * BN; n0 += 256) {
                const int nn = (S - i) * BN - n0 < 256 ? (S - i) * BN - n0 : 256;
                mma_bf16(tmem + (uint32_t)(b * C::kCols + i * BN + n0), ad, bd + (uint64_t)(n0 * 32 / 16),
                         kIdesc | ((uint32_t)(nn >> 3) << 17), acc);
              }
            }
          }
          mma_commit(&wempty[c]);
          if (last) mma_commit(&bempty[s]);
          if (k0 + G >= ks) mma_commit(&accf[b]);
        }
        __syncwarp();
        if (last) ++st;
      }
      if (++ch == nch) ch = 0;
    }
    if (lane == 0) mma_commit(fin);
  } else if (warp == 2) {
    int ch = ch_start, st = 0, w = 0;
    bool stop = false;
    for (int u = 0; u < nu && !stop; ++u) {
      const int b = u % NB;
      const int ks = steps(ch);
      for (int k0 = 0; k0 < ks && !stop; k0 += G, ++w) {
        const int s = st % NM, c = w % NW;
        const bool ok = (k0 > 0 || u < NB || bar_wait(&acce[b], ((u / NB) - 1) & 1)) &&
                        (k0 % KS != 0 || bar_wait(&bfull[s], (st / NM) & 1)) && bar_wait(&wfull[c], (w / NW) & 1) &&
                        !*(volatile int*)abort_flag;
        stop = meet(!__all_sync(0xffffffffu, ok));
        if ((k0 + G) % KS == 0 || k0 + G >= ks) ++st;
      }
      if (++ch == nch) ch = 0;
    }
    if (stop) atomicExch(abort_flag, 1);
  } else if (warp < 3 + C::kWidenWarps) {
    const int t = threadIdx.x - 96;
    int ch = ch_start, st = 0, w = 0;
    bool ok = true;
    for (int u = 0; u < nu && ok; ++u) {
      const int ks = steps(ch);
      for (int k0 = 0; k0 < ks; k0 += G, ++w) {
        const int s = st % NA, c = w % NW, kn = min(G, ks - k0);
        if ((k0 % KS == 0 && !bar_wait(&afull[s], (st / NA) & 1)) ||
            (w >= NW && !bar_wait(&wempty[c], ((w / NW) - 1) & 1)) || *(volatile int*)abort_flag) {
          atomicExch(abort_flag, 1);
          ok = false;
          break;
        }
        const uint2* src = reinterpret_cast<const uint2*>(ring_a + (size_t)s * C::kStageA + (k0 % KS) * C::kA);
        uint4* dst = reinterpret_cast<uint4*>(base + (size_t)c * C::kWide);
#pragma unroll 4
        for (int i = t; i < kn * S * kSlRows * 2; i += C::kWiden) {  // 8 digits each
          const uint2 d = src[i];
          dst[i] = make_uint4(widen2(d.x, 0x4140), widen2(d.x, 0x4342), widen2(d.y, 0x4140), widen2(d.y, 0x4342));
        }
        // the MMAs read through the asynchronous proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        bar_arrive(&wfull[c]);
        if ((k0 + G) % KS == 0 || k0 + G >= ks) {
          bar_arrive(&aempty[s]);
          ++st;
        }
      }
      if (++ch == nch) ch = 0;
    }
  } else {
    // a warp reads the tensor-memory lanes 32 (warp % 4) ..; set h of four warps takes
    // the vectors [h KQ, (h + 1) KQ): their real columns and, BN/2 on, their imaginary ones
    const int q4 = warp & 3, half = (warp - 3 - C::kWidenWarps) >> 2;
    constexpr int KQ = BN / 2 / (C::kAddWarps / 4);
    constexpr int CG = S == 4 ? 4 : 2;  // columns at a time
    const uint32_t lane_addr = tmem + ((uint32_t)(q4 * 32) << 16);
    const int r = q4 * 32 + lane, il = r >> 1;
    const bool even = (lane & 1) == 0;
    T acc[KQ];
#pragma unroll
    for (int c = 0; c < KQ; ++c) acc[c] = 0;
    int64_t rt = u0 / nch;
    int ch = ch_start, ch_first = ch_start;
    bool ok = true, fresh = true;  // fresh: the segment's first chunk
    const bool scaled = alpha.x != (T)1 || alpha.y != (T)0, beta_re = beta.x != (T)0, beta_im = beta.y != (T)0;
    for (int u = 0; u < nu; ++u) {
      const int b = u % NB;
      if (!__all_sync(0xffffffffu, bar_wait(&accf[b], (u / NB) & 1) && !*(volatile int*)abort_flag)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int64_t mti = rt % mt, ct = rt / mt;
      const int er = ea[(mti * nch + ch) * (kSlRows / 2) + il];
      // lane c holds the exponent of this warp's vector c
      const int ec = lane < KQ ? ex[(ct * nch + ch) * H + half * KQ + lane] : 0;
#pragma unroll 1
      for (int c0 = 0; c0 < KQ; c0 += CG) {
        uint32_t p[S][CG], q[S][CG];
#pragma unroll
        for (int d = 0; d < S; ++d) {
          const uint32_t col = lane_addr + (uint32_t)(b * C::kCols + d * BN + half * KQ + c0);
          tmem_ld(col, p[d]);
          tmem_ld(col + H, q[d]);
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        T got[CG];
#pragma unroll
        for (int c = 0; c < CG; ++c) {
          uint32_t dp[S], dq[S];
#pragma unroll
          for (int d = 0; d < S; ++d) {
            dp[d] = p[d][c];
            dq[d] = q[d][c];
          }
          Sum2 a = add_diagonals<S>(dp), o = add_diagonals<S>(dq);
          // even lane: Re y = Re a Re x - Im a Im x; odd lane: Im y = Im a Re x + Re a Im x
          o.h = __shfl_xor_sync(0xffffffffu, o.h, 1);
          a.h += even ? -o.h : o.h;
          if constexpr (S > 4) {
            o.l = __shfl_xor_sync(0xffffffffu, o.l, 1);
            a.l += even ? -o.l : o.l;
            got[c] = sum_to_double<S>(a, er + __shfl_sync(0xffffffffu, ec, c0 + c));
          } else {
            const int e = __shfl_sync(0xffffffffu, ec, c0 + c);
            got[c] = __ll2float_rn(a.h) * __int_as_float((er - 18 + 127) << 23) * __int_as_float((e - 18 + 127) << 23);
          }
        }
#pragma unroll
        for (int j = 0; j < KQ; j += CG)  // acc[] stays in registers: its index is known
          if (j == c0) {
#pragma unroll
            for (int c = 0; c < CG; ++c) acc[j + c] = fresh ? got[c] : acc[j + c] + got[c];
          }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      bar_arrive(&acce[b]);
      const bool closes = ch == nch - 1;
      if (closes || u == nu - 1) {
        const bool whole = closes && ch_first == 0;
        bool skip = false;  // a tile of vectors left to the FMA form
        for (int j = 0; j < nch; ++j) skip |= flags[(swap ? mti : ct) * nch + j] != 0;
        const int64_t i = mti * (kSlRows / 2) + il;
        const int64_t seg = (int64_t)blockIdx.x - (rt * nch) / per;  // segment in the row tile
        // y offsets: of this lane's M-side row, and in lane c of the warp's N-side row c
        const int64_t cl = ct * H + half * KQ + lane;
        const int64_t moff = i >= m ? 0 : swap ? tc_col_offset(ym, i) : i * yes;
        const int64_t noff = lane >= KQ || cl >= ncols ? 0 : swap ? cl * yes : tc_col_offset(ym, cl);
        const bool reads = whole && (beta_re || beta_im);
        T own[KQ];  // y's component of this lane, all loaded before the first is used
#pragma unroll
        for (int c = 0; c < KQ; ++c) {
          own[c] = 0;
          const int64_t o = moff + __shfl_sync(0xffffffffu, noff, c);
          if (reads && !skip && i < m && ct * H + half * KQ + c < ncols)
            own[c] = reinterpret_cast<const T*>(y + o)[lane & 1];
        }
#pragma unroll
        for (int c = 0; c < KQ; ++c) {
          const T v = acc[c];
          const bool mine = !skip && i < m && ct * H + half * KQ + c < ncols;
          const int64_t o = moff + __shfl_sync(0xffffffffu, noff, c);
          if (!whole) {
            if (mine)
              reinterpret_cast<T*>(part + (((rt * smax + seg) * H + half * KQ + c) * (kSlRows / 2) + il))[lane & 1] = v;
            continue;
          }
          // each lane its own component of alpha v + beta y
          T r = v;
          if (scaled) {
            const T w = __shfl_xor_sync(0xffffffffu, v, 1);
            r = even ? alpha.x * v - alpha.y * w : alpha.x * v + alpha.y * w;
          }
          if (beta_im) {
            const T other = __shfl_xor_sync(0xffffffffu, own[c], 1);
            r += even ? beta.x * own[c] - beta.y * other : beta.x * own[c] + beta.y * other;
          } else if (beta_re) {
            r += beta.x * own[c];
          }
          if (mine) reinterpret_cast<T*>(y + o)[lane & 1] = r;
        }
        ch_first = 0;
      }
      fresh = closes;
      if (++ch == nch) {
        ch = 0;
        ++rt;
      }
    }
    if (!ok) {
      atomicExch(abort_flag, 1);
      if (lane == 0 && status) atomicOr(status, kTcErrTimeout);
    }
  }
  if (warp == 1 && lane == 0) bar_wait(fin, 0);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

template <typename V, typename T>
__device__ __forceinline__ void axpby_out(V* yp, T re, T im, V alpha, V beta) {
  V o;
  o.x = alpha.x * re - alpha.y * im;
  o.y = alpha.x * im + alpha.y * re;
  if (beta.x != (T)0 || beta.y != (T)0) {
    const V v = *yp;
    o.x += beta.x * v.x - beta.y * v.y;
    o.y += beta.x * v.y + beta.y * v.x;
  }
  *yp = o;
}

// y of the row tiles split over several blocks: their partial products in chunk order
template <int FORM, int BN>
__global__ void k_slice_reduce(const typename Sl<FORM>::V* __restrict__ part, const int* __restrict__ left, int mt,
                               int nch, int per, int smax, int swap, int64_t m, int64_t ncols,
                               typename Sl<FORM>::V* y, int64_t yes, TcColMap ym, typename Sl<FORM>::V alpha, typename Sl<FORM>::V beta) {
  using T = typename SlAcc<FORM>::T;
  constexpr int H = BN / 2;
  pdl_wait();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int il = (int)(i % (kSlRows / 2));
  const int64_t mti = i / (kSlRows / 2);
  for (int64_t cg = blockIdx.y; cg < ncols; cg += gridDim.y) {
    const int64_t ct = cg / H, rt = ct * mt + mti;
    const int64_t b0 = rt * nch / per, b1 = (rt * nch + nch - 1) / per;
    if (b0 == b1) continue;  // one block wrote it
    if (left[swap ? mti : ct]) continue;
    T re = 0, im = 0;
    for (int64_t j = 0; j <= b1 - b0; ++j) {
      const typename Sl<FORM>::V p = part[((rt * smax + j) * H + cg % H) * (kSlRows / 2) + il];
      re += p.x;
      im += p.y;
    }
    axpby_out(y + (swap ? cg * yes + tc_col_offset(ym, i) : i * yes + tc_col_offset(ym, cg)), re, im, alpha, beta);
  }
}

template <int FORM, int ROWS, bool INTER, typename IN>
void run_split(const IN* x, int64_t n, int64_t es, const TcColMap& map, int64_t nvec, int64_t tiles, int nkb,
               unsigned char* out, int* exps, int* flags, int* any, const SliceSide* other, SliceSide* own,
               cudaStream_t s, bool pdl) {
  const int nch = (nkb + kSlChunk - 1) / kSlChunk;
  auto kern = k_slice_split<FORM, ROWS, INTER, IN>;
  // k steps staged at a time: the chunk where it fits beside the tile's tables, otherwise half
  // of it, read once for the largest components and again for the digits
  auto bytes = [](int k) { return (size_t)(ROWS / 2) * (k * 16 + 1) * sizeof(typename Sl<FORM>::V); };
  int sub = std::min(nkb, kSlChunk);
  if (bytes(sub) > 220 * 1024) sub = kSlChunk / 2;
  const size_t smem = bytes(sub);
  QOB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_kernel(pdl, kern, dim3((unsigned)tiles, (unsigned)nch), (unsigned)split_threads(ROWS), smem, s, x, n, es, map, nvec, nkb,
                es == 1 ? 1 : 0, sub, out, exps, flags, any, other, own);
  QOB_LAUNCHED();
}

// swap: the vectors are the M side (their bytes widened), the matrix the N side.
template <int FORM, int BN>
FmaGate run_slices(const SliceDense& d, bool swap, const void* xv, int64_t xes, const TcColMap& xm, int64_t ncols, void* yv,
                   int64_t yes, const TcColMap& ym, c128 al, c128 be, Workspace* ws, cudaStream_t s,
                   unsigned* status, int num_sms, bool pdl) {
  using C = SlCfg<FORM, BN>;
  using V = typename Sl<FORM>::V;
  using T = typename SlAcc<FORM>::T;
  constexpr int H = BN / 2, HM = kSlRows / 2;
  const V* x = static_cast<const V*>(xv);
  V* y = static_cast<V*>(yv);
  V alpha, beta;
  alpha.x = (T)al.re;
  alpha.y = (T)al.im;
  beta.x = (T)be.re;
  beta.y = (T)be.im;
  const int nkb = d.nkb, nch = (nkb + kSlChunk - 1) / kSlChunk;
  const int64_t mrows = swap ? ncols : d.m, nrows = swap ? d.m : ncols;
  const int64_t mt = (mrows + HM - 1) / HM, nt = (nrows + H - 1) / H, vt = swap ? mt : nt;
  const int64_t rtiles = nt * mt, units = rtiles * nch, wave = num_sms;
  // equal runs over one wave; whole row tiles when those fill it
  int64_t per = (units + wave - 1) / wave;
  if (rtiles >= wave) per = (rtiles + wave - 1) / wave * nch;
  const int64_t blocks = (units + per - 1) / per;
  const int smax = (int)((nch - 1) / per + 2);
  const int64_t tile = swap ? HM : H;  // vectors of a tile
  const SlicePlanes& pl = swap ? d.nside : d.mside;
  const SliceSide* sides = static_cast<const SliceSide*>(pl.sides);
  const size_t bbytes = (size_t)vt * nkb * (swap ? C::kA : C::kB), ebytes = ((size_t)vt * (nch * (tile + 1) + 1) + 1) * sizeof(int);
  unsigned char* w = static_cast<unsigned char*>(ws->try_get(0, bbytes + ebytes, s));
  if (!w) return FmaGate();
  int* exps = reinterpret_cast<int*>(w + bbytes);
  int* flags = exps + vt * nch * tile;
  int *left = flags + vt * nch, *any = left + vt;
  V* part = nullptr;
  if (per % nch != 0) {
    part = static_cast<V*>(ws->try_get(1, (size_t)rtiles * smax * H * HM * sizeof(V), s));
    if (!part) return FmaGate();
  }
  if (swap)
    run_split<FORM, kSlRows, true, V>(x, d.n, xes, xm, ncols, vt, nkb, w, exps, flags, any, sides, nullptr, s, pdl);
  else
    run_split<FORM, BN, false, V>(x, d.n, xes, xm, ncols, vt, nkb, w, exps, flags, any, sides, nullptr, s, pdl);
  const unsigned char* mp = swap ? w : pl.planes;
  const unsigned char* np = swap ? pl.planes : w;
  const int* me = swap ? exps : pl.exps;
  const int* ne = swap ? pl.exps : exps;
  auto kern = k_slice_gemm<FORM, BN>;
  QOB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem));
  // the launches behind the split kernel overlap with the one before (pdl_enter, pdl_wait): the
  // GEMM's blocks set themselves up beside the split's (4096 x 4096 on 16 kets, ComplexF32, 89 -> 83 us)
  launch_kernel(true, kern, dim3((unsigned)blocks), (unsigned)C::kThreads, C::smem, s, mp, me, np, ne, (const int*)flags,
                any, left, mrows, (int)mt, nrows, nkb, nch, (int)per, units, smax, swap ? 1 : 0, y, yes, ym, alpha, beta, part,
                status);
  QOB_LAUNCHED();
  if (part) {
    launch_kernel(true, k_slice_reduce<FORM, BN>,
                  dim3((unsigned)((mrows + 127) / 128), (unsigned)std::min<int64_t>(nrows, 65535)), 128u, 0, s,
                  (const V*)part, (const int*)left, (int)mt, nch, (int)per, smax, swap ? 1 : 0, mrows, nrows, y, yes,
                  ym, alpha, beta);
    QOB_LAUNCHED();
  }
  FmaGate g;
  g.any = any;
  g.tiles = left;
  while (((int64_t)1 << g.log2_tile) < tile) ++g.log2_tile;
  return g;
}

constexpr int kSwapBN = 64;

// The matrix's planes as the M side (rows widened) or, swap, as the N side.
template <int FORM>
void build_slices(SliceDense& d, bool swap, const void* a, cudaStream_t s) {
  constexpr int S = Sl<FORM>::S;
  SlicePlanes& pl = swap ? d.nside : d.mside;
  const int nch = (d.nkb + kSlChunk - 1) / kSlChunk;
  const int64_t half = swap ? kSwapBN / 2 : kSlRows / 2, tiles = (d.m + half - 1) / half;
  // one allocation: planes, exponents, the chunks' sides, then what the host looks at, flags and
  // sides of each tile's chunks
  const size_t nt = (size_t)(tiles * nch), pbytes = (size_t)tiles * d.nkb * S * (swap ? kSwapBN * 32 : kSlRows * 16);
  pl.buf.alloc(pbytes + nt * half * sizeof(int) + (nt + nch) * sizeof(SliceSide) + nt * sizeof(int));
  unsigned char* planes = static_cast<unsigned char*>(pl.buf.p);
  int* exps = reinterpret_cast<int*>(planes + pbytes);
  auto* sides = reinterpret_cast<SliceSide*>(exps + nt * half);
  auto* tile_sides = sides + nch;
  int* flags = reinterpret_cast<int*>(tile_sides + nt);
  TcColMap map;  // "vectors" = matrix rows, one element apart; contracted index = column, m apart
  map.st = 1;
  const auto* m = static_cast<const typename Sl<FORM>::M*>(a);
  if (swap)
    run_split<FORM, kSwapBN, false, typename Sl<FORM>::M>(m, d.n, d.m, map, d.m, tiles, d.nkb,
                                                          planes, exps, flags, nullptr, nullptr, tile_sides, s, false);
  else
    run_split<FORM, kSlRows, true, typename Sl<FORM>::M>(m, d.n, d.m, map, d.m, tiles, d.nkb,
                                                         planes, exps, flags, nullptr, nullptr, tile_sides, s, false);
  std::vector<SliceSide> q(nt + (nt * sizeof(int) + sizeof(SliceSide) - 1) / sizeof(SliceSide)), worst((size_t)nch);
  QOB_CUDA(cudaMemcpyAsync(q.data(), tile_sides, nt * (sizeof(SliceSide) + sizeof(int)), cudaMemcpyDeviceToHost, s));
  QOB_CUDA(cudaStreamSynchronize(s));
  const int* f = reinterpret_cast<const int*>(q.data() + nt);
  int state = 1;
  for (size_t i = 0; i < nt; ++i)
    if (f[i]) state = -1;
  for (int ch = 0; ch < nch; ++ch) {
    SliceSide& w = worst[(size_t)ch] = q[(size_t)ch];
    for (int64_t t = 1; t < tiles; ++t) {
      const SliceSide& o = q[(size_t)(t * nch + ch)];
      w.n1 = std::max(w.n1, o.n1);
      w.t = std::max(w.t, o.t);
      for (int i = 0; i < kLevels; ++i) w.c[i] = std::min(w.c[i], o.c[i]);
    }
    // a matrix that fails even with vectors of ones is left to the FMA kernels at once
    const int n = (int)std::min<int64_t>(d.n, (int64_t)chunk_start(ch + 1, d.nkb, nch) * 16) -
                  chunk_start(ch, d.nkb, nch) * 16;
    const SliceSide ones{0.5f * (float)n, 0.f, {n, n, n, n, n, n}};
    float least = 0.f;
    for (int k = 0; k < kLevels * kLevels; ++k) least += overlap(w, ones, n, k / kLevels, k % kLevels);
    if (digit_error(w, ones) > kSlLimit<FORM> * least) state = -1;
  }
  if (state > 0) {
    QOB_CUDA(cudaMemcpyAsync(sides, worst.data(), worst.size() * sizeof(SliceSide), cudaMemcpyHostToDevice, s));
    QOB_CUDA(cudaStreamSynchronize(s));  // for calls on any stream
    pl.planes = planes;
    pl.exps = exps;
    pl.sides = sides;
  } else {
    pl.buf = DeviceBuf();
  }
  pl.state = state;
}

}  // namespace

// Which side the vectors take: the M side, whose rows lie across lanes, when they
// (and not the matrix's rows) are next to each other in y.
bool slice_swap(int64_t yes, const TcColMap& ym, int64_t ncols) {
  const bool vectors_next = ym.s1 > 1 ? ym.sa == 1 : ym.s3 > 1 ? ym.sb == 1 : ym.st == 1;
  return yes != 1 && vectors_next && ncols >= kSlRows / 2;
}

bool slice_ready(SliceDense& d, int form, const void* a, int64_t m, int64_t n, bool swap, cudaStream_t s) {
  SlicePlanes& pl = swap ? d.nside : d.mside;
  if (pl.state != 0) return pl.state > 0;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  QOB_CUDA(cudaStreamIsCapturing(s, &cs));
  if (cs != cudaStreamCaptureStatusNone) return false;  // not built inside a capture
  d.m = m;
  d.n = n;
  d.nkb = (int)((n + 15) / 16);
  try {
    if (form == QOB_C128)
      build_slices<QOB_C128>(d, swap, a, s);
    else if (form == QOB_C128X)
      build_slices<QOB_C128X>(d, swap, a, s);
    else
      build_slices<QOB_C64>(d, swap, a, s);
  } catch (const Error& e) {
    if (e.code != QOB_ERR_OOM) throw;
    pl.buf = DeviceBuf();  // no room for the planes: the FMA kernels
    pl.state = -1;
  }
  return pl.state > 0;
}

FmaGate launch_slices(const SliceDense& d, int form, c128 alpha, const void* x, int64_t xes, const TcColMap& xm,
                      c128 beta, void* y, int64_t yes, const TcColMap& ym, int64_t ncols, cudaStream_t s, Workspace* ws,
                      unsigned* status, int num_sms, bool pdl) {
  const bool swap = slice_swap(yes, ym, ncols);
#define QOB_SL(F, BN) \
  run_slices<F, BN>(d, swap, x, xes, xm, ncols, y, yes, ym, alpha, beta, ws, s, status, num_sms, pdl)
  if (form == QOB_C128) return ncols <= 16 ? QOB_SL(QOB_C128, 32) : QOB_SL(QOB_C128, kSwapBN);
  if (form == QOB_C128X) return ncols <= 16 ? QOB_SL(QOB_C128X, 32) : QOB_SL(QOB_C128X, kSwapBN);
  return ncols <= 16 ? QOB_SL(QOB_C64, 32) : QOB_SL(QOB_C64, kSwapBN);
#undef QOB_SL
}

}  // namespace qob
