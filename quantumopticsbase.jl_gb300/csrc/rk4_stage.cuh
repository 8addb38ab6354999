// rk4_stage.cuh -- the RK4 stage combination of one element, as the batched
// stages (batch.cu) and the one-launch evolution (rk4.cu) apply it.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace qob {

// k of an RK4 stage into the stage combination (the arithmetic of
// k_rk4_stage, element by element): 1: acc = k, tmp = psi + dt/2 k; 2, 3:
// acc += 2 k, tmp = psi + (dt/2 | dt) k; 4: psi += dt/6 (acc + k)
template <typename CT, typename S>
__device__ __forceinline__ void rk4_stage_element(void* psi_, void* acc_, void* tmp_, double dt_, int64_t j, CT kv,
                                                  int stage) {
  CT* psi = (CT*)psi_;
  CT* acc = (CT*)acc_;
  CT* tmp = (CT*)tmp_;
  const S dt = (S)dt_;
  if (stage == 1) {
    const CT p = psi[j];
    const S c = dt * (S)0.5;
    acc[j] = kv;
    CT o;
    o.x = p.x + c * kv.x;
    o.y = p.y + c * kv.y;
    tmp[j] = o;
  } else if (stage == 2 || stage == 3) {
    const CT p = psi[j];
    const S c = stage == 2 ? dt * (S)0.5 : dt;
    CT a = acc[j];
    a.x += (S)2 * kv.x;
    a.y += (S)2 * kv.y;
    acc[j] = a;
    CT o;
    o.x = p.x + c * kv.x;
    o.y = p.y + c * kv.y;
    tmp[j] = o;
  } else {
    const CT a = acc[j];
    CT p = psi[j];
    const S c = dt / (S)6;
    p.x += c * (a.x + kv.x);
    p.y += c * (a.y + kv.y);
    psi[j] = p;
  }
}

}  // namespace qob
