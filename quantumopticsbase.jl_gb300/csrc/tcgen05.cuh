// tcgen05.cuh -- what the tensor-core kernels (k_tc32.cu, k_slice.cu) share: mbarriers with
// bounded waits, bulk copies, MMA commits, and the offsets of a product's columns.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "qob_internal.h"

namespace qob {
namespace {

constexpr int kBarPolls = 1 << 21;  // polls of a barrier before a wait gives up
constexpr unsigned kTcErrTimeout = 1u;

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* b, unsigned n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}
__device__ __forceinline__ bool bar_test(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
  for (int i = 0; i < kBarPolls; ++i) {
    if (bar_test(b, parity)) return true;
    if (i > 64) __nanosleep(32);
  }
  return false;
}
// bytes (a multiple of 16) from global src to shared dst, both 16-byte aligned, counted on b
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   saddr(dst)),
               "l"(src), "r"(bytes), "r"(saddr(b))
               : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(b))
               : "memory");
}

// element offset of column c of a column map (no division for a plain stride;
// 32-bit divisions: column counts and the map's extents stay below 2^31)
__host__ __device__ __forceinline__ int64_t tc_col_offset(const TcColMap& m, int64_t c) {
  if (m.s1 == 1 && m.s3 == 1) return c * m.st;
  const uint32_t cc = (uint32_t)c, s1 = (uint32_t)m.s1, s3 = (uint32_t)m.s3;
  const uint32_t a = cc % s1, q = cc / s1;
  return (int64_t)a * m.sa + (int64_t)(q % s3) * m.sb + (int64_t)(q / s3) * m.st;
}

}  // namespace
}  // namespace qob
