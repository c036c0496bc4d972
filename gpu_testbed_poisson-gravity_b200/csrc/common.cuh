// common.cuh -- shared device helpers for the per-patch Poisson-gravity kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gpg {

// ---------------------------------------------------------------------------
// IEEE-exact arithmetic.  The reference CPU solvers evaluate every expression
// as separate float/double operations in source order (gcc, baseline x86-64,
// no FMA).  These wrappers are never contracted into FMA by nvcc, so a kernel
// that keeps the reference's operand order produces bit-identical values.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float absval(float a) { return fabsf(a); }
__device__ __forceinline__ double absval(double a) { return fabs(a); }
// a / b with IEEE round-to-nearest (the reference's `(real)0.5/rho`).
__device__ __forceinline__ float divide(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double divide(double a, double b) { return __ddiv_rn(a, b); }

// ---------------------------------------------------------------------------
// Patch geometry (Header/Macro.h:53-61), compile-time in the ghost size G.
//   N     fine cube edge the solver works in: 8 + 2G (interior + 1 ghost layer)
//   M     interior edge = RHO_NXT = N - 2
//   PN    POT_NXT = 4 + 2*((G+3)/2)
//   U     POT_USELESS = G % 2 (layers of the interpolated array outside the cube)
// ---------------------------------------------------------------------------
template <int G>
struct Geo {
  static constexpr int N = 8 + 2 * G;
  static constexpr int M = N - 2;
  static constexpr int HALF = M / 2;
  static constexpr int POT_INT = (G + 3) / 2;
  static constexpr int PN = 4 + 2 * POT_INT;
  static constexpr int U = G % 2;
  static constexpr int RHO3 = M * M * M;
  static constexpr int PN3 = PN * PN * PN;
  // number of interior x-pairs per patch (one SOR lane each)
  static constexpr int NPAIR = HALF * M;
};

// Colour of fine-cube cell (x, y, z): the SOR pass that updates it.  Pass 0 of
// the reference (CPU_PoissonSolver_SOR.cpp:220-270) updates interior cells
// whose rho index (x-1, y-1, z-1) has an even sum.
__host__ __device__ constexpr int colour(int x, int y, int z) { return (x + y + z + 1) & 1; }

// Team barrier: a warp barrier for one-warp teams, a named barrier (id = team
// index + 1, count = team threads) otherwise, so teams of one CTA that stop
// at different iterations never wait for each other.
template <int TEAM>
__device__ __forceinline__ void team_sync(int team) {
  if constexpr (TEAM == 32) {
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(TEAM) : "memory");
  }
}

__device__ __forceinline__ double warp_sum(double v) {
  // xor butterfly: every lane ends with the same bits (a+b == b+a exactly)
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

// On a lambda that reads or writes a lane's register arrays.  Left to the
// compiler's heuristics, which weigh the whole translation unit, one became a call
// and the arrays went to local memory (multigrid FP32 ghost 2 and 4: 512 and 672
// bytes of stack; 4096 patches 198 us instead of 87 and 465 instead of 185).
#define GPG_INLINE __attribute__((always_inline))

// Programmatic dependent launch: a kernel launched with launch_after() may become
// resident while the kernel before it in the stream still runs.  pdl_wait() holds
// it until that kernel has finished and its results are visible, before the first
// access to global memory.  Without pdl_trigger() the next kernel's CTAs come in
// once all of this one's have ended, which still saves 2 us of a launch.
// pdl_trigger() lets them in when every CTA of this kernel has called it or ended.
// The SOR kernels don't: the waiting CTAs then crowd onto the SMs that are free
// first, and a launch smaller than the device runs unevenly spread (FP64, back to
// back, triggered before the output / not at all: ghost 1, 1001 patches 51.2 / 41.5
// us, 2, 500 66.2 / 53.6, 4, 148 76.6 / 69.2, 5, 148 84.8 / 69.8; FP32 ghost 1,
// 256 11.8 / 11.3, and 1 % in the mean of 85 launches).
// The others do: multigrid before its output (FP64 ghost 2, 148 patches 77.7 us, 79.8
// without; ghost 1, 500 69.5 / 63.2), the learned start's kernel after its last
// patch (no difference), and the network's training kernels as early as nothing
// else is to be won, weight gradients and reductions right after their wait, since
// a step of few patches is a chain of ten short kernels (gradient of 1 patch 65 us,
// 85 without; 32 110 / 120; 500 343 / 350).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

// Kernel arguments shared by the Poisson kernels (values already rounded to
// `real` exactly where the reference rounds them).
template <typename T>
struct SolveArgs {
  const T *rho;
  const T *pot_in;
  T *pot_out;
  T *flu;
  const T *guess;
  int32_t *iters;
  double *resid;
  int64_t npatch;
  T sor_const;      // Poi_Coeff*dh*dh        (CPU_PoissonSolver_SOR.cpp:51)
  T omega_6;        // Omega/6                (CPU_PoissonSolver_SOR.cpp:52)
  T neg_zero;       // -0.0, unknown to the compiler: fma(a, b, neg_zero) is a * b rounded on its own
  T gra_const;      // dt/(2dh) or dt/(12dh)  (CPU_GravitySolver.cpp:23)
  T dh;
  T poi_coeff;
  T mg_tol;
  double sor_tol;   // relative L1 tolerance (GPG_STOP_TOLERANCE)
  int min_iter, max_iter;
  int mg_max_iter, mg_npre, mg_npost;
  int int_scheme;   // 4 CQUAD, 5 QUAD
  int init_mode;    // GPG_INIT_*
  int stop_mode;    // GPG_STOP_*
  int gra_ghost;    // 0..2
  int gra_acc;      // fused gravity update
  int p5;           // 5-point gradient
};

}  // namespace gpg
