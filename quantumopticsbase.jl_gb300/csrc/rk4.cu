// rk4.cu -- fixed-step RK4 of one state in one launch.
//
// A step of dpsi/dt = -i H psi is four applications of H, each needing all of the
// one before.  As four launches per step (batch.cu's fused stages, replayed from a
// CUDA graph) a small state is bound by the launches: a stage of a 12-spin chain
// took 8.2 us for 0.4 us of arithmetic.  Here one cooperative launch runs all
// steps: every thread keeps its output index, and the blocks meet at a grid
// barrier after each stage (a counter in L2, about a microsecond).  The inputs,
// written by other SMs in the stage before, are read from L2.  The arithmetic and its
// order are those of the batched stages.
//
// H does not change, so a thread looks its row up once: the row's stored entries
// (input index, value) go to a list of its own in shared memory, psi and the stages'
// sum stay in registers, and a stage is the list's inputs, up to eight in flight,
// one store and the barrier (k_rk4_list).  States with more entries than resident
// threads, and rows too wide for the list, walk the compiled tables at each stage
// (k_rk4_grid).
//
// What bounds it: the barrier, one round trip to L2 and the chain of a row's dependent
// multiply-adds per stage, 3.1 us where the launches took 8.2.  Blocks of 128: 64 need
// twice the arrivals at the counter, 256 leave SMs without a block (100 steps,
// ComplexF64, us for 64 / 128 / 256: 10 spins 1178 / 1077 / 1293, 12 1271 / 1282 /
// 1533, 14 1370 / 1327 / 1722, 16 3445 / 2820 / 2750).  Against four launches per step
// (ComplexF64 / ComplexF32 / double-float): 8 spins 2670 -> 776 / 2264 -> 579 / 2675 -> 972,
// 12 3285 -> 1224 / 2880 -> 926 / 3493 -> 1451, 16 4518 -> 2701 / 3667 -> 1422 / 4516 -> 2385,
// 17 7608 -> 5071 (ComplexF64).
//
// Waits are bounded: a block that gives up marks the counter, every block leaves at
// its next barrier, the context's status word says so and the call fails.
#include <algorithm>

#include "batch.h"
#include "k_gather.cuh"
#include "rk4_stage.cuh"

namespace qob {

namespace {

constexpr int kRk4Threads = 128;
constexpr unsigned kBarGone = 0x80000000u;  // the counter of a launch that gave up
constexpr int kBarPolls = 1 << 20;
constexpr int kRk4StepsPerLaunch = 1024;  // keeps the counter (4 per step and block) below 2^31

struct Rk4Args {
  GatherView v;
  void *psi, *acc, *b0, *b1;  // stage outputs go to b0, b1, b0, psi
  double dt;
  int nsteps;
  unsigned* bar;
};

// -i v: a swap and a sign, where products with (0, -1) would be four FP64 operations
__device__ __forceinline__ double2 minus_i(double2 v) {
  return make_double2(v.y, __hiloint2double(__double2hiint(v.x) ^ (int)0x80000000, __double2loint(v.x)));
}
__device__ __forceinline__ float2 minus_i(float2 v) { return make_float2(v.y, -v.x); }
__device__ __forceinline__ double2 minus_i(float4 v) {
  return minus_i(make_double2(gather::ff_join(v.x, v.y), gather::ff_join(v.z, v.w)));
}

// All blocks of the grid; false when one gave up.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, unsigned* status) {
  __shared__ int gone;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    unsigned v = 0;
    for (int polls = 0; v < target && polls < kBarPolls; ++polls)
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
    if (v < target) {
      atomicOr(bar, kBarGone);
      if (status) atomicOr(status, gather::kErrWaitTimeout);
      v = kBarGone;
    }
    gone = (v & kBarGone) != 0u;
  }
  __syncthreads();
  return gone == 0;
}

template <typename R, bool REALV, bool W1>
__global__ void __launch_bounds__(kRk4Threads) k_rk4_grid(Rk4Args a) {
  using CT = typename gather::Cx<R>::T;
  using AT = typename gather::AccOf<R>::T;
  using ET = typename gather::Ell<R, REALV>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SiteTable st;  // not read: square
  st.nsites = 0;
  const ET* ell = gather::stage<ET>(smem_raw, a.v);
  const GGroup* sg = reinterpret_cast<const GGroup*>(smem_raw);
  const int64_t j0 = blockIdx.x * (int64_t)kRk4Threads + threadIdx.x, total = (int64_t)gridDim.x * kRk4Threads;
  unsigned target = 0;
  for (int step = 0; step < a.nsteps; ++step) {
    for (int stage = 1; stage <= 4; ++stage) {
      const CT* x = (const CT*)(stage == 1 ? a.psi : stage == 3 ? a.b1 : a.b0);
      void* out = stage == 2 ? a.b1 : a.b0;
      for (int64_t j = j0; j < a.v.m; j += total) {
        AT acc[1];
        gather::accumulate<R, REALV ? gather::kReal : gather::kComplex, true, W1, 1, true>(a.v, st, sg, ell, (uint32_t)j,
                                                                                         x, 1, 0, 1, acc);
        const CT kv = minus_i(acc[0].total());
        using S = typename std::conditional<std::is_same<R, float>::value, float, double>::type;
        rk4_stage_element<CT, S>(a.psi, a.acc, out, a.dt, j, kv, stage);
      }
      if (step + 1 == a.nsteps && stage == 4) return;
      target += gridDim.x;
      if (!grid_barrier(a.bar, target, a.v.status)) return;
    }
  }
}

// Stored entries of a row that a list holds: 96 KB of shared memory a block in
// ComplexF64 with real values; longer rows leave too few blocks resident.
constexpr int kRk4ListMax = 64;

// Seven blocks an SM hold 2^17 elements (double-float without the limit: 12 spins 1329, but 17
// 5728 for 4276, its rows then without room).
template <typename R, bool REALV>
__global__ void __launch_bounds__(kRk4Threads, 7) k_rk4_list(Rk4Args a, int cap) {
  using CT = typename gather::Cx<R>::T;
  using AT = typename gather::AccOf<R>::T;
  using ET = typename gather::Ell<R, REALV>::T;
  using VT = typename gather::Val<R, REALV>::T;
  using S = typename std::conditional<std::is_same<R, float>::value, float, double>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const GatherView& g = a.v;
  const ET* ell = gather::stage<ET>(smem_raw, g);
  const GGroup* sg = reinterpret_cast<const GGroup*>(smem_raw);
  // the lists behind the tables: values, then indices, entry e of thread t at [e][t]
  const size_t tables = (size_t)g.ngroups * (sizeof(GGroup) + (g.fast ? sizeof(int4) : 0)) +
                        (g.ell_smem ? (size_t)g.ell_slots * sizeof(ET) : 0);
  VT* vals = reinterpret_cast<VT*>(smem_raw + ((tables + 15) & ~(size_t)15)) + threadIdx.x;
  int* idx = reinterpret_cast<int*>(smem_raw + ((tables + 15) & ~(size_t)15) + (size_t)cap * kRk4Threads * sizeof(VT)) +
             threadIdx.x;
  const int64_t j = blockIdx.x * (int64_t)kRk4Threads + threadIdx.x;
  const bool on = j < g.m;
  int ne = 0;
  VT d{};
  CT p{}, sum{}, own{};
  if (on) {
    if (g.has_diag) d = static_cast<const VT*>(g.diag)[j];
    for (int gi = 0; gi < g.ngroups; ++gi) {
      const GGroup& G = sg[gi];
      uint32_t r, sub;
      gather::local_row(G, (uint32_t)j, r, sub);
      for (int k = 0; k < G.width; ++k) {
        if (gather::kDebugBounds &&
            gather::out_of_range((int64_t)G.ell_off + (int64_t)r * G.width + k, g.ell_slots, g.status))
          continue;
        const ET e = ell[G.ell_off + (int64_t)r * G.width + k];
        const VT v = gather::Ell<R, REALV>::v(e);
        if (gather::kDebugBounds && gather::nz(v) &&
            gather::out_of_range((int64_t)((uint32_t)j - sub) + e.col, g.n, g.status))
          continue;
        if (gather::nz(v) && ne < cap) {
          vals[ne * kRk4Threads] = v;
          idx[ne * kRk4Threads] = (int)((uint32_t)j - sub) + e.col;
          ++ne;
        }
      }
    }
    own = p = static_cast<const CT*>(a.psi)[j];
  }
  const int ne_warp = __reduce_max_sync(~0u, ne);
  const S dt = (S)a.dt;
  unsigned target = 0;
  for (int step = 0; step < a.nsteps; ++step) {
#pragma unroll
    for (int stage = 1; stage <= 4; ++stage) {
      const CT* x = (const CT*)(stage == 1 ? a.psi : stage == 3 ? a.b1 : a.b0);
      if (on) {
        AT acc;
        if (g.has_diag)
          acc.set(d, own);
        else
          acc.zero();
        for (int e = 0; e < ne_warp; e += 8) {
          CT u[8];
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (e + k < ne) u[k] = __ldcg(x + idx[(e + k) * kRk4Threads]);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if constexpr (std::is_same<R, double>::value) {
              if (e + k < ne) acc.mac(vals[(e + k) * kRk4Threads], u[k]);
            } else {
              // a loop of at most one turn stays a branch: the twenty (double-float) or
              // eight instructions of an entry that no thread of the warp has are
              // skipped; two FP64 ones are the faster under a predicate
              int turn = e + k < ne_warp;
              while (turn != 0) {
                if (e + k < ne) acc.mac(vals[(e + k) * kRk4Threads], u[k]);
                turn = 0;
                asm volatile("" : "+r"(turn));
              }
            }
          }
        }
        const CT kv = minus_i(acc.total());
        // the stage combination (rk4_stage.cuh), psi and the sum in registers
        if (stage == 4) {
          const S c = dt / (S)6;
          p.x += c * (sum.x + kv.x);
          p.y += c * (sum.y + kv.y);
          own = p;
          static_cast<CT*>(a.psi)[j] = p;
        } else {
          const S c = stage == 3 ? dt : dt * (S)0.5;
          if (stage == 1) {
            sum = kv;
          } else {
            sum.x += (S)2 * kv.x;
            sum.y += (S)2 * kv.y;
          }
          own.x = p.x + c * kv.x;
          own.y = p.y + c * kv.y;
          static_cast<CT*>(stage == 2 ? a.b1 : a.b0)[j] = own;
        }
      }
      if (step + 1 == a.nsteps && stage == 4) return;
      target += gridDim.x;
      if (!grid_barrier(a.bar, target, g.status)) return;
    }
  }
}

template <typename R, bool REALV>
const void* grid_kernel(bool w1) {
  return w1 ? (const void*)k_rk4_grid<R, REALV, true> : (const void*)k_rk4_grid<R, REALV, false>;
}

template <typename R, bool REALV>
const void* list_kernel() {
  return (const void*)k_rk4_list<R, REALV>;
}

}  // namespace

bool rk4_one_launch(Context& ctx, const Plan& P, void* psi, void* work, int64_t n, double dt, int nsteps,
                    cudaStream_t s) {
  if (!plan_fusable(P) || n > kRk4GridMax || nsteps < 1) return false;
  const GatherPlan& g = *P.gather;
  const size_t esz = P.precision == QOB_C128 ? 16 : 8, sz = (size_t)n * esz;
  Rk4Args a;
  a.v = g.view();
  size_t smem = (size_t)a.v.ngroups * (sizeof(GGroup) + (a.v.fast ? sizeof(int4) : 0));
  const size_t eb = (size_t)a.v.ell_slots * (P.precision == QOB_C128 ? (g.real_vals ? sizeof(EllD) : sizeof(EllZ))
                                                                   : (g.real_vals ? sizeof(EllF) : sizeof(EllC)));
  a.v.ell_smem = a.v.ell_slots > 0 && eb <= gather::kStageSlotsMax ? 1 : 0;
  if (a.v.ell_smem) smem += eb;
  char* w = static_cast<char*>(work);
  a.psi = psi;
  a.acc = w;
  a.b0 = w + sz;
  a.b1 = w + 2 * sz;
  a.dt = dt;
  if (!ctx.grid_bar.p) ctx.grid_bar.alloc(16);
  a.bar = static_cast<unsigned*>(ctx.grid_bar.p);
  // the list kernel when every row fits a list and every index a resident thread
  const size_t vsz = g.ff ? (g.real_vals ? 8 : 16) : (size_t)(g.real_vals ? 1 : 2) * esz / 2;
  const size_t lists = (size_t)g.row_max * kRk4Threads * (vsz + sizeof(int));
  size_t lsmem = ((smem + 15) & ~(size_t)15) + lists;
  int cap = (int)g.row_max;
  const void* kern = nullptr;
  int64_t fit = 0;
  auto resident = [&](const void* k, size_t sm) {
    int occ = 0;
    if (sm > 48 * 1024) QOB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    QOB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kRk4Threads, sm));
    return (int64_t)occ * ctx.num_sms;
  };
  bool list = g.all_ell && g.row_max <= kRk4ListMax && lsmem <= 160 * 1024;
  if (list) {
    kern = g.ff ? (g.real_vals ? list_kernel<gather::DFX, true>() : list_kernel<gather::DFX, false>())
           : P.precision == QOB_C128 ? (g.real_vals ? list_kernel<double, true>() : list_kernel<double, false>())
                                     : (g.real_vals ? list_kernel<float, true>() : list_kernel<float, false>());
    fit = resident(kern, lsmem);
    list = (n + kRk4Threads - 1) / kRk4Threads <= fit;
  }
  if (!list) {
    // walking the tables, 2^16 elements took 3831 us for 4518 with the launches (12 spins
    // 1796 for 3285), 2^17 more than the launches
    if (n > kRk4GridMax / 2) return false;
    kern = g.ff ? (g.real_vals ? grid_kernel<gather::DFX, true>(g.all_w1) : grid_kernel<gather::DFX, false>(g.all_w1))
           : P.precision == QOB_C128
               ? (g.real_vals ? grid_kernel<double, true>(g.all_w1) : grid_kernel<double, false>(g.all_w1))
               : (g.real_vals ? grid_kernel<float, true>(g.all_w1) : grid_kernel<float, false>(g.all_w1));
    fit = resident(kern, smem);
  }
  if (fit < 1) return false;
  const unsigned grid = (unsigned)std::min<int64_t>((n + kRk4Threads - 1) / kRk4Threads, fit);
  for (int done = 0; done < nsteps; done += a.nsteps) {
    a.nsteps = std::min(nsteps - done, kRk4StepsPerLaunch);
    QOB_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned), s));
    void* args[] = {&a, &cap};
    QOB_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kRk4Threads), args, list ? lsmem : smem, s));
    QOB_LAUNCHED();
    unsigned bar = 0;
    QOB_CUDA(cudaMemcpyAsync(&bar, a.bar, sizeof(bar), cudaMemcpyDeviceToHost, s));
    QOB_CUDA(cudaStreamSynchronize(s));
    if (bar & kBarGone) fail(QOB_ERR_CUDA, "RK4: a wait between blocks ran out");
  }
  return true;
}

}  // namespace qob
