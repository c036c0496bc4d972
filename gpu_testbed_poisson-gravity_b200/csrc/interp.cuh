// interp.cuh -- coarse -> fine potential interpolation of one patch.
//
// Every interior coarse cell (i, j, k) in [1, POT_NXT-1)^3 produces its 8 fine
// children; children outside the solver cube (the POT_USELESS layers for odd
// ghost sizes) are dropped.  CQUAD is the conservative quadratic form of
// CPU_PoissonSolver_SOR.cpp:110-174 (13 slopes weighted 1/8, 1/64, 1/512);
// QUAD the 27-point tensor product of CPU_PoissonSolver_SOR.cpp:177-203.
// Operand order follows those loops so the values are bit-identical.
#pragma once

#include "common.cuh"
#include "packed.cuh"

namespace gpg {

// CQUAD of two coarse cells along x, (i, j, k) and (i+1, j, k) with i odd, in
// packed FP32: the same operations in the same order as below, each instruction
// for both cells, and 18 64-bit loads instead of 54.  Per pair about 190
// instructions instead of 340 (the interpolation was a third of an FP32 solve:
// 37 of 107 us at ghost 3, 4096 patches; with it 105, and 144 instead of 153 at
// ghost 4, 191 instead of 202 at ghost 5).  c0 points at cell (i-1, j, k), 8-byte
// aligned.
// child[c] holds child c of both cells.
template <int PN, bool LDG>
__device__ __forceinline__ void cquad_pair(const float *__restrict__ c0, float neg_zero, f32x2 (&child)[8]) {
  const f32x2 nz = pack2(neg_zero, neg_zero), m1 = pack2(-1.f, -1.f);
  const f32x2 c8 = pack2(0.125f, 0.125f), c64 = pack2(0.015625f, 0.015625f), c512 = pack2(0.001953125f, 0.001953125f);
  // a row's values at x - 1 and x + 1; at x (shared by both loads)
  struct Row {
    f32x2 m, p;
    __device__ __forceinline__ f32x2 mid() const { return pack2(hi2(m), lo2(p)); }
  };
  auto row = [&](int dk, int dj) {
    const float *q = c0 + (dk * PN + dj) * PN;
    Row r;
    if constexpr (LDG) {
      const float2 a = __ldg(reinterpret_cast<const float2 *>(q)), b = __ldg(reinterpret_cast<const float2 *>(q + 2));
      r.m = pack2(a.x, a.y), r.p = pack2(b.x, b.y);
    } else {
      const float2 a = *reinterpret_cast<const float2 *>(q), b = *reinterpret_cast<const float2 *>(q + 2);
      r.m = pack2(a.x, a.y), r.p = pack2(b.x, b.y);
    }
    return r;
  };
  auto sub2 = [&](f32x2 a, f32x2 b) { return fma2(b, m1, a); };           // one rounding, as a - b
  auto slope = [&](f32x2 c, f32x2 a, f32x2 b) { return fma2(c, sub2(a, b), nz); };
  f32x2 s[13], centre;
  {
    const Row r = row(0, 0);
    s[0] = slope(c8, r.p, r.m);
    centre = r.mid();
  }
  {
    const Row u = row(0, 1), d = row(0, -1);
    s[1] = slope(c8, u.mid(), d.mid());
    s[5] = slope(c64, d.p, d.m);
    s[6] = slope(c64, u.p, u.m);
  }
  f32x2 below, above;
  {
    const Row r = row(-1, 0), u = row(-1, 1), d = row(-1, -1);
    below = r.mid();
    s[3] = slope(c64, r.p, r.m);
    s[4] = slope(c64, u.mid(), d.mid());
    s[9] = slope(c512, d.p, d.m);
    s[10] = slope(c512, u.p, u.m);
  }
  {
    const Row r = row(1, 0), u = row(1, 1), d = row(1, -1);
    above = r.mid();
    s[7] = slope(c64, r.p, r.m);
    s[8] = slope(c64, u.mid(), d.mid());
    s[11] = slope(c512, d.p, d.m);
    s[12] = slope(c512, u.p, u.m);
  }
  s[2] = slope(c8, above, below);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int sx = (c & 1) ? 1 : -1, sy = (c & 2) ? 1 : -1, sz = (c & 4) ? 1 : -1;
    const int sg[13] = {sx,      sy,      sz,           -sx * sz,      -sy * sz,
                        -sx * sy, sx * sy, sx * sz,      sy * sz,       sx * sy * sz,
                        -sx * sy * sz, -sx * sy * sz, sx * sy * sz};
    f32x2 v = sg[0] > 0 ? s[0] : fma2(s[0], m1, nz);
#pragma unroll
    for (int t = 1; t < 13; ++t) v = sg[t] > 0 ? add2(v, s[t]) : sub2(v, s[t]);
    child[c] = add2(v, centre);
  }
}

// `coarse` is one patch's [POT_NXT]^3 potential: in global memory, read
// through L1 (LDG; each value feeds up to 27 coarse cells), or a copy staged
// in shared memory (!LDG).
// neg_zero: see SolveArgs.
template <typename T, int G, int NT, bool LDG = true, typename Store>
__device__ __forceinline__ void interpolate(const T *__restrict__ coarse, int tid, int int_scheme, T neg_zero,
                                            Store store) {
  using g = Geo<G>;
  constexpr int PN = g::PN, NC = PN - 2, N = g::N, U = g::U;
  if constexpr (sizeof(T) == 4) {
    if (int_scheme == 4 && (reinterpret_cast<uintptr_t>(coarse) & 7) == 0) {
      for (int w = tid; w < NC * NC * (NC / 2); w += NT) {
        const int i = 1 + 2 * (w % (NC / 2)), j = 1 + (w / (NC / 2)) % NC, k = 1 + w / (NC * (NC / 2));
        f32x2 child[8];
        cquad_pair<PN, LDG>(coarse + (k * PN + j) * PN + i - 1, neg_zero, child);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int x = 2 * (i - 1) + (c & 1) - U, y = 2 * (j - 1) + ((c >> 1) & 1) - U,
                    z = 2 * (k - 1) + ((c >> 2) & 1) - U;
          if (U == 0 || ((unsigned)y < (unsigned)N && (unsigned)z < (unsigned)N)) {
            if (U == 0 || x >= 0) store(x, y, z, lo2(child[c]));
            if (U == 0 || x + 2 < N) store(x + 2, y, z, hi2(child[c]));
          }
        }
      }
      return;
    }
  }
  for (int w = tid; w < NC * NC * NC; w += NT) {
    const int i = 1 + w % NC, j = 1 + (w / NC) % NC, k = 1 + w / (NC * NC);
    const T *c0 = coarse + (k * PN + j) * PN + i;
    auto C = [c0](int dk, int dj, int di) -> T {
      const T *q = c0 + (dk * PN + dj) * PN + di;
      if constexpr (LDG) return __ldg(q);
      else return *q;
    };
    T child[8];
    if (int_scheme == 4) {
      const T c8 = T(0.125), c64 = T(0.015625), c512 = T(0.001953125);
      T s[13];
      s[0] = mul(c8, sub(C(0, 0, 1), C(0, 0, -1)));
      s[1] = mul(c8, sub(C(0, 1, 0), C(0, -1, 0)));
      s[2] = mul(c8, sub(C(1, 0, 0), C(-1, 0, 0)));
      s[3] = mul(c64, sub(C(-1, 0, 1), C(-1, 0, -1)));
      s[4] = mul(c64, sub(C(-1, 1, 0), C(-1, -1, 0)));
      s[5] = mul(c64, sub(C(0, -1, 1), C(0, -1, -1)));
      s[6] = mul(c64, sub(C(0, 1, 1), C(0, 1, -1)));
      s[7] = mul(c64, sub(C(1, 0, 1), C(1, 0, -1)));
      s[8] = mul(c64, sub(C(1, 1, 0), C(1, -1, 0)));
      s[9] = mul(c512, sub(C(-1, -1, 1), C(-1, -1, -1)));
      s[10] = mul(c512, sub(C(-1, 1, 1), C(-1, 1, -1)));
      s[11] = mul(c512, sub(C(1, -1, 1), C(1, -1, -1)));
      s[12] = mul(c512, sub(C(1, 1, 1), C(1, 1, -1)));
      const T centre = C(0, 0, 0);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        // half-signs of child c along x, y, z; each slope's sign is their product
        const int sx = (c & 1) ? 1 : -1, sy = (c & 2) ? 1 : -1, sz = (c & 4) ? 1 : -1;
        const int sg[13] = {sx,      sy,      sz,           -sx * sz,      -sy * sz,
                            -sx * sy, sx * sy, sx * sz,      sy * sz,       sx * sy * sz,
                            -sx * sy * sz, -sx * sy * sz, sx * sy * sz};
        T v = sg[0] > 0 ? s[0] : -s[0];
#pragma unroll
        for (int t = 1; t < 13; ++t) v = sg[t] > 0 ? add(v, s[t]) : sub(v, s[t]);
        child[c] = add(v, centre);
      }
    } else {
      const T wm[3] = {T(0.15625), T(0.9375), T(-0.09375)};  // Mm = {5, 30, -3}/32
      const T wp[3] = {T(-0.09375), T(0.9375), T(0.15625)};  // Mp = {-3, 30, 5}/32
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const T *wx = (c & 1) ? wp : wm, *wy = (c & 2) ? wp : wm, *wz = (c & 4) ? wp : wm;
        T v = T(0);
#pragma unroll
        for (int dk = -1; dk <= 1; ++dk)
#pragma unroll
          for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
            for (int di = -1; di <= 1; ++di)
              v = add(v, mul(mul(mul(C(dk, dj, di), wz[dk + 1]), wy[dj + 1]), wx[di + 1]));
        child[c] = v;
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int x = 2 * (i - 1) + (c & 1) - U, y = 2 * (j - 1) + ((c >> 1) & 1) - U,
                z = 2 * (k - 1) + ((c >> 2) & 1) - U;
      if (U == 0 || ((unsigned)x < (unsigned)N && (unsigned)y < (unsigned)N && (unsigned)z < (unsigned)N))
        store(x, y, z, child[c]);
    }
  }
}

}  // namespace gpg
