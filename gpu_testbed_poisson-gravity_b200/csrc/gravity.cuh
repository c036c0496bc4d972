// gravity.cuh -- finite-difference acceleration and momentum/energy update of
// one patch (CPU_GravitySolver.cpp:34-79): with Gra_Const = dt/(2dh) (3-point)
// or dt/(12dh) (5-point, GRA_GHOST_SIZE == 2),
//   a     = Gra_Const * dphi
//   Eint  = E - 0.5/rho * |p|^2
//   p    -= rho * a
//   E     = Eint + 0.5/rho * |p|^2
// The density component is read, never written.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace gpg {

// One cell: phi(i, j, k) returns the potential at patch-cell offset (i, j, k),
// which ranges over [-2, 10) (x fastest); q = rho, px, py, pz, E, updated.
template <typename T, typename Phi>
__device__ __forceinline__ void gravity_cell(int i, int j, int k, T gra_const, int p5, Phi phi, T (&q)[5]) {
  const T c8 = T(8);
  T ax, ay, az;
  if (p5) {
    ax = mul(gra_const, sub(add(add(-phi(i + 2, j, k), phi(i - 2, j, k)), mul(c8, phi(i + 1, j, k))),
                            mul(c8, phi(i - 1, j, k))));
    ay = mul(gra_const, sub(add(add(-phi(i, j + 2, k), phi(i, j - 2, k)), mul(c8, phi(i, j + 1, k))),
                            mul(c8, phi(i, j - 1, k))));
    az = mul(gra_const, sub(add(add(-phi(i, j, k + 2), phi(i, j, k - 2)), mul(c8, phi(i, j, k + 1))),
                            mul(c8, phi(i, j, k - 1))));
  } else {
    ax = mul(gra_const, sub(phi(i + 1, j, k), phi(i - 1, j, k)));
    ay = mul(gra_const, sub(phi(i, j + 1, k), phi(i, j - 1, k)));
    az = mul(gra_const, sub(phi(i, j, k + 1), phi(i, j, k - 1)));
  }
  const T temp = divide(T(0.5), q[0]);
  const T eint = sub(q[4], mul(temp, add(add(mul(q[1], q[1]), mul(q[2], q[2])), mul(q[3], q[3]))));
  q[1] = sub(q[1], mul(q[0], ax));
  q[2] = sub(q[2], mul(q[0], ay));
  q[3] = sub(q[3], mul(q[0], az));
  q[4] = add(eint, mul(temp, add(add(mul(q[1], q[1]), mul(q[2], q[2])), mul(q[3], q[3]))));
}

// Runs of 16 bytes (4 FP32 or 2 FP64 cells along x) of the patch's fluid, one
// per thread and step: 128 FP32 runs instead of 512 cells, so that a team of 96
// threads waits for two rounds of loads and not six.  flu points at one patch
// [5][8][8][8]; a pointer off the 16-byte alignment takes the values one by one.
// CELLS = 1: single cells.
template <typename T, int CELLS = 16 / sizeof(T)>
struct FluidRun {
  static constexpr int W = CELLS, RUNS = 512 / W;
  alignas(16) T q[5][W];  // component, cell; a row is one wide access
  __device__ __forceinline__ void load(const T *flu, int run, bool aligned) {
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const T *src = flu + c * 512 + run * W;
      if (W > 1 && aligned) {
        *reinterpret_cast<uint4 *>(q[c]) = *reinterpret_cast<const uint4 *>(src);
      } else {
#pragma unroll
        for (int e = 0; e < W; ++e) q[c][e] = src[e];
      }
    }
  }
  __device__ __forceinline__ void store(T *flu, int run, bool aligned) const {
#pragma unroll
    for (int c = 1; c < 5; ++c) {  // the density is read only
      T *dst = flu + c * 512 + run * W;
      if (W > 1 && aligned) {
        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(q[c]);
      } else {
#pragma unroll
        for (int e = 0; e < W; ++e) dst[e] = q[c][e];
      }
    }
  }
  template <typename Phi>
  __device__ __forceinline__ void update(int run, T gra_const, int p5, Phi phi) {
    const int c0 = run * W;
#pragma unroll
    for (int e = 0; e < W; ++e) {
      T cell[5] = {q[0][e], q[1][e], q[2][e], q[3][e], q[4][e]};
      gravity_cell((c0 & 7) + e, (c0 >> 3) & 7, c0 >> 6, gra_const, p5, phi, cell);
#pragma unroll
      for (int c = 1; c < 5; ++c) q[c][e] = cell[c];
    }
  }
};

__device__ __forceinline__ bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename T, int NT, typename Phi>
__device__ __forceinline__ void gravity_patch(T *__restrict__ flu, int tid, T gra_const, int p5,
                                              Phi phi) {
  for (int cell = tid; cell < 512; cell += NT) {
    FluidRun<T, 1> f;
    f.load(flu, cell, false);
    f.update(cell, gra_const, p5, phi);
    f.store(flu, cell, false);
  }
}

// What every solver kernel leaves of a patch: the GRA_NXT^3 window of the solved
// cube (CPU_PoissonSolver_SOR.cpp:305-311) and, with gra_acc, the updated fluid.
// cube(x, y, z) reads the solver's cube.  PRELOAD: the first fluid loads are under
// way while the window is written, at the price of their registers (20 in FP32,
// 20 to 40 in FP64) over the window's address arithmetic; the callers say where
// that pays.  CELLS: see FluidRun.
template <typename T, int G, int NT, bool PRELOAD = true, int CELLS = 16 / sizeof(T), typename Cube>
__device__ __forceinline__ void patch_output(const SolveArgs<T> &a, int64_t P, int tid, Cube cube) {
  T *flu = a.flu + P * 5 * 512;
  const bool al = aligned16(flu);
  FluidRun<T, CELLS> f;
  if (PRELOAD && a.gra_acc && tid < FluidRun<T, CELLS>::RUNS) f.load(flu, tid, al);
  // (edge GN a compile-time constant per GRA_GHOST_SIZE: the index split is
  // then multiply-shift, not division)
  auto window = [&](auto gg) {
    constexpr int GG = decltype(gg)::value, GN = 8 + 2 * GG, shift = G - GG, GN3 = GN * GN * GN;
    T *dst = a.pot_out + P * GN3;
    for (int t = tid; t < GN3; t += NT) {
      const int i = t % GN, j = (t / GN) % GN, k = t / (GN * GN);
      dst[t] = cube(i + shift, j + shift, k + shift);
    }
  };
  if (a.gra_ghost == 0)
    window(std::integral_constant<int, 0>{});
  else if (a.gra_ghost == 1)
    window(std::integral_constant<int, 1>{});
  else
    window(std::integral_constant<int, 2>{});
  // fused gravity update (CPU_GravitySolver.cpp:34-79)
  if (a.gra_acc) {
    auto phi = [&](int i, int j, int k) { return cube(i + G, j + G, k + G); };
    for (int run = tid; run < FluidRun<T, CELLS>::RUNS; run += NT) {
      if (!PRELOAD || run >= NT) f.load(flu, run, al);
      f.update(run, a.gra_const, a.p5, phi);
      f.store(flu, run, al);
    }
  }
}

// Lines of a patch's density and fluid into L2: needed only once the cube is
// interpolated, and at the end.
template <typename T, int G, int NT>
__device__ __forceinline__ void prefetch_patch(const SolveArgs<T> &a, int64_t P, int tid) {
  auto lines = [tid](const void *p, int bytes) {
    for (int o = tid * 128; o < bytes; o += NT * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char *>(p) + o));
  };
  using g = Geo<G>;
  lines(a.rho + P * g::RHO3, g::RHO3 * int(sizeof(T)));
  if (a.gra_acc) lines(a.flu + P * 5 * 512, 5 * 512 * int(sizeof(T)));
}

// Gravity alone (Poisson off): the potential comes from pot_out
// [P][GRA_NXT]^3.  One CTA of 256 threads per patch; the GRA window is staged
// in shared memory first.  Bound by memory (FP32, 4096 patches: 92 MB, within
// L2), so it needs all its threads: two single cells each and eight CTAs per SM,
// 12.7 us (FP64 35.3); runs of 16 bytes leave half of them without one in FP32
// and take 40 registers: 16.8 us (FP64 41.8).
template <typename T, int GG>
__global__ void __launch_bounds__(256) gravity_kernel(T *__restrict__ flu, const T *__restrict__ pot,
                                                      int64_t npatch, T gra_const, int p5) {
  constexpr int GN = 8 + 2 * GG, GN3 = GN * GN * GN;
  __shared__ T s_pot[GN3];
  const int64_t P = blockIdx.x;
  if (P >= npatch) return;
  const T *src = pot + P * GN3;
  for (int t = threadIdx.x; t < GN3; t += 256) s_pot[t] = src[t];
  __syncthreads();
  gravity_patch<T, 256>(flu + P * 5 * 512, threadIdx.x, gra_const, p5, [&](int i, int j, int k) {
    return s_pot[((k + GG) * GN + (j + GG)) * GN + (i + GG)];
  });
}

}  // namespace gpg
