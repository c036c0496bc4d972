// optim.cuh -- the Adam update shared by the trained models of libgpg.
#pragma once

#include <cstdint>

namespace gpg {

struct AdamArgs {
  float *p, *m, *v;     // parameters, moments
  const float *g;       // gradient
  float lr, b1, b2;     // step, betas
  float eps, c1, c2;    // epsilon, bias corrections 1 - b1^t, 1 - b2^t
};

// parameter i of one Adam step: updates its moments and value, returns the value
__device__ __forceinline__ float adam_update(const AdamArgs &a, int64_t i) {
  const float gi = a.g[i];
  const float mi = a.b1 * a.m[i] + (1.f - a.b1) * gi;
  const float vi = a.b2 * a.v[i] + (1.f - a.b2) * gi * gi;
  a.m[i] = mi;
  a.v[i] = vi;
  const float x = a.p[i] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
  a.p[i] = x;
  return x;
}

static __global__ void adam_kernel(const AdamArgs a, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    adam_update(a, i);
}

}  // namespace gpg
