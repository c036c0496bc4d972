// mg_kernel.cuh -- per-patch multigrid V-cycle, one patch per CTA, all levels
// on chip (no device-side malloc).
//
// Semantics follow CPU_PoissonSolver_MG.cpp:46-377:
//   levels  N0 = 8+2G, N(l+1) = (N(l)+1)/2 while that is >= 3; dh(l) = dh (N0-1)/(N(l)-1)
//           (10-5-3, 12-6-3, 14-7-4, 16-8-4, 18-9-5-3), bottom smoothing 1 (3^3) or 7 (4^3)
//   cycle   per level down: NPre red-black Gauss-Seidel sweeps, defect, 27-point
//           restriction to the next RHS, zero correction; bottom smoothing; per level
//           up: trilinear prolongation added, NPost sweeps
//   error   dh^2 sum|defect| / sum|sol| on level 0 (sums in double), stop when
//           <= MG_Tolerated_Error or after Max_Iter cycles
// Operand order of every stencil follows the reference loops (bit-identical values).
//
// B200 layout.  Level 0, where the work is, uses the SOR's two-row, split-column
// lane layout (sor_kernel.cuh): each lane keeps its columns of the solution and
// of the right-hand side in registers, the shared cube is colour-split with
// conflict-free pitches, a smoothing update reads 2 shared values and stores 1
// (FP32: two heights per packed register pair).  The reference's red and black
// passes are the SOR's two colours.  While the solution is in registers the
// shared cube holds the defect for the restriction; the prolongation adds to the
// registers and publishes the cube again.  The coarse levels are dense arrays in
// shared memory, the 4^3 bottom level eight lanes of one warp (its 14 passes need
// no block barrier).
// Before, every level was a dense array, a thread per same-colour cell: 80 % of
// the shared pipe (half of it 2-way conflicts of the colour stride), 57 % of the
// issue slots, most of them index arithmetic.
// us per launch with gravity, 4096 FP32 patches / 1000 FP64 ones, before -> now:
// ghost 1 72 -> 53 / 212 -> 83, 2 122 -> 76 / 362 -> 188, 3 238 -> 129 / 705 -> 390,
// 4 337 -> 185 / 1098 -> 559, 5 522 -> 253 / 1266 -> 866.
#pragma once

#include <type_traits>

#include <cfloat>

#include "common.cuh"
#include "gravity.cuh"
#include "interp.cuh"
#include "sor_kernel.cuh"

namespace gpg {

template <int G>
struct MgLevels {
  static constexpr int n0 = 8 + 2 * G;
  static constexpr int next(int n) { return (n + 1) / 2; }
  static constexpr int count() {
    int n = n0, c = 1;
    while (next(n) >= 3 && c < 10) { n = next(n); ++c; }
    return c;
  }
  static constexpr int L = count();  // number of levels, bottom = L-1
  static constexpr int size(int lv) {
    int n = n0;
    for (int i = 0; i < lv; ++i) n = next(n);
    return n;
  }
  static constexpr int cells(int lv) { return size(lv) * size(lv) * size(lv); }
  // first cell of a coarse level (1..) in the coarse arrays
  static constexpr int offset(int lv) {
    int o = 0;
    for (int i = 1; i < lv; ++i) o += cells(i);
    return o;
  }
  static constexpr int coarse = offset(L);
  static constexpr int nbottom = size(L - 1) == 3 ? 1 : 7;
  static_assert(size(L - 1) == 3 || size(L - 1) == 4, "bottom grid must be 3^3 or 4^3");
  static_assert(L >= 3, "a level between the finest and the bottom");
};

template <typename T, int G, bool WIDE = false>
struct MgCfg {
  static constexpr int Z = 2;  // lanes per column
  using C = SorCfg<T, G, Z, 2>;
  using LV = MgLevels<G>;
  // threads of the CTA: the level-0 layout's, or (WIDE) at least twice as many, the
  // others helping with all but the level-0 sweeps
  static constexpr int TEAM = !WIDE ? C::TEAM : (2 * C::TEAM < 128 ? 128 : 2 * C::TEAM);
  static constexpr size_t round(size_t b) { return (b + 15) / 16 * 16; }
  static constexpr size_t cube = 0;                                         // level 0: solution, or its defect
  static constexpr size_t sol = cube + round(sizeof(T) * C::CUBE);          // levels 1..
  static constexpr size_t rhs = sol + round(sizeof(T) * LV::coarse);
  static constexpr size_t def = rhs + round(sizeof(T) * LV::coarse);        // of one coarse level at a time
  static constexpr size_t table = def + round(sizeof(T) * LV::cells(1));    // prolongation to level 0, per index
  static constexpr size_t red = table + round((2 * sizeof(T) + sizeof(int)) * (LV::n0 - 1));
  static constexpr size_t bytes = red + 2 * sizeof(double) * (TEAM / 32);
  // Resident CTAs the register allocation allows: what shared memory holds, at no
  // fewer registers per thread than REGS (a lane keeps its columns and their
  // right-hand sides across the coarse levels; spilling them costs more than the
  // CTAs gain: FP64 ghost 3 390 us at 255 registers, 530 at 168; FP32 ghost 3 129
  // at 128, 138 at 80, ghost 5 263 at 128, 253 at 96).
  static constexpr int REGS = sizeof(T) == 8 ? 255 : (G == 5 ? 96 : 128);
  static constexpr int by_smem = int((228 * 1024) / (bytes + 1024)), by_regs = 65536 / (TEAM * REGS);
  static constexpr int blocks = by_smem < by_regs ? (by_smem < 1 ? 1 : by_smem) : (by_regs < 1 ? 1 : by_regs);
};

// A thread's share of a dense coarse level: x-pairs (2s+1, 2s+2) of rows (j, k),
// one cell of each colour, whose values and right-hand sides stay in registers
// while the level is smoothed.  The pair mate is a register neighbour, the other
// five neighbours come from shared memory.
template <typename T, int NT, int n>
struct MgPairs {
  static constexpr int m = n - 2, w = (m + 1) / 2, items = m * m * w, K = (items + NT - 1) / NT;
  int id[K];       // left cell of the pair; 0: none
  bool right[K];   // the pair has a right cell (not where m is odd and the pair the row's last)
  bool first[K];   // the left cell belongs to pass 0 ((i+j+k) odd)
  T v[K][2], b[K][2];  // [left, right]: solution, right-hand side

  __device__ __forceinline__ MgPairs(int tid) {
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const int t = tid + q * NT, row = t / w, s = t - row * w, j = 1 + row % m, k = 1 + row / m, i = 1 + 2 * s;
      const bool mine = t < items;
      id[q] = mine ? (k * n + j) * n + i : 0;
      right[q] = mine && i + 1 < n - 1;
      first[q] = ((i + j + k) & 1) != 0;
    }
  }
  __device__ __forceinline__ void load_rhs(const T *rhs) {
#pragma unroll
    for (int q = 0; q < K; ++q) {
      b[q][0] = rhs[id[q]];
      b[q][1] = right[q] ? rhs[id[q] + 1] : T(0);
    }
  }
  __device__ __forceinline__ void load_sol(const T *sol) {
#pragma unroll
    for (int q = 0; q < K; ++q) {
      v[q][0] = sol[id[q]];
      v[q][1] = sol[id[q] + 1];  // the boundary's zero where the pair has no right cell
    }
  }
  // sum of the six neighbours of the pair's cell c, in the reference's order
  __device__ __forceinline__ T sum(const T *sol, int q, bool c) const {
    const T *p = sol + id[q] + c;
    const T xo = p[c ? 1 : -1];
    return add(add(add(add(add(p[n * n], p[-n * n]), p[n]), p[-n]), c ? xo : v[q][1]), c ? v[q][0] : xo);
  }
  // Red-black Gauss-Seidel (CPU_PoissonSolver_MG.cpp:392-441); every pass ends with a barrier
  __device__ __forceinline__ void smooth(T *sol, T dh, int sweeps) {
    const T dh2 = mul(dh, dh), one_six = divide(T(1), T(6));
#pragma unroll 1
    for (int pass = 0; pass < 2 * sweeps; ++pass) {
#pragma unroll
      for (int q = 0; q < K; ++q) {
        // the pair's cell of this pass; one path for both sides, so that a warp does not diverge
        const bool c = first[q] == bool(pass & 1);
        if (!id[q] || (c && !right[q])) continue;
        const T x = mul(one_six, sub(sum(sol, q, c), mul(dh2, c ? b[q][1] : b[q][0])));
        v[q][0] = c ? v[q][0] : x;
        v[q][1] = c ? x : v[q][1];
        sol[id[q] + c] = x;
      }
      team_sync<NT>(0);
    }
  }
  // def = -(lap(sol) - rhs) (CPU_PoissonSolver_MG.cpp:474-494)
  __device__ __forceinline__ void defect(const T *sol, T *def, T dh) const {
    const T m_dh2 = divide(T(-1), mul(dh, dh));
#pragma unroll
    for (int q = 0; q < K; ++q) {
      if (!id[q]) continue;
      def[id[q]] = add(mul(m_dh2, sub(sum(sol, q, false), mul(T(6), v[q][0]))), b[q][0]);
      if (right[q]) def[id[q] + 1] = add(mul(m_dh2, sub(sum(sol, q, true), mul(T(6), v[q][1]))), b[q][1]);
    }
  }
};

// 27-point restriction (CPU_PoissonSolver_MG.cpp:533-616) to the interior of the
// dense level c.  `fine(bz, by, bx)` returns a reader of the fine defect around
// base cell (bx, by, bz): reader(tz, ty, tx), each 0..2 and known at compile time.
// Only interior fine cells are read (every level ratio is at least 2).
template <typename T, int NT, int nf, int nc, typename Fine>
__device__ __forceinline__ void mg_restrict(Fine &&fine, T *c, int tid) {
  const T ratio = divide(T(nf - 1), T(nc - 1)), half = T(0.5);
  constexpr int mc = nc - 2;
  for (int t = tid; t < mc * mc * mc; t += NT) {
    const int i = 1 + t % mc, j = 1 + (t / mc) % mc, k = 1 + t / (mc * mc);
    T w[3][3];  // [z/y/x][left/centre/right]
    int base[3];
    const int ijk[3] = {k, j, i};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const T pos = mul(T(ijk[d]), ratio);
      const int cc = (int)add(pos, half);
      base[d] = cc - 1;
      w[d][0] = mul(half, sub(add(T(cc), half), pos));
      w[d][2] = sub(half, w[d][0]);
      w[d][1] = half;
    }
    auto at = fine(base[0], base[1], base[2]);
    T v = T(0);
#pragma unroll
    for (int tz = 0; tz < 3; ++tz)
#pragma unroll
      for (int ty = 0; ty < 3; ++ty)
#pragma unroll
        for (int tx = 0; tx < 3; ++tx) {
          const T term = mul(mul(mul(w[0][tz], w[1][ty]), w[2][tx]), at(tz, ty, tx));
          v = (tz | ty | tx) ? add(v, term) : term;
        }
    c[(k * nc + j) * nc + i] = v;
  }
}

// weights and base cell of the trilinear prolongation at fine index f
template <typename T>
__device__ __forceinline__ void mg_weights(int f, T ratio, T &w0, T &w1, int &base) {
  const T pos = mul(T(f), ratio);
  base = (int)pos;
  w0 = sub(T(base + 1), pos);
  w1 = sub(T(1), w0);
}

// the eight corner terms of one fine cell in the reference's order 000,001,010,
// 100,011,110,101,111 (z,y,x); zy[z][y] = wz * wy, c[z][y][x] the corners
template <typename T>
__device__ __forceinline__ T mg_corners(const T (&zy)[2][2], const T (&wx)[2], const T (&c)[2][2][2]) {
  constexpr int ord[8][3] = {{0, 0, 0}, {0, 0, 1}, {0, 1, 0}, {1, 0, 0},
                             {0, 1, 1}, {1, 1, 0}, {1, 0, 1}, {1, 1, 1}};
  T v = T(0);
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const int oz = ord[o][0], oy = ord[o][1], ox = ord[o][2];
    const T term = mul(mul(zy[oz][oy], wx[ox]), c[oz][oy][ox]);
    v = o ? add(v, term) : term;
  }
  return v;
}
template <typename T, int nc>
__device__ __forceinline__ void mg_load4(const T *p, T (&c)[2][2]) {
  c[0][0] = p[0], c[0][1] = p[1], c[1][0] = p[nc], c[1][1] = p[nc + 1];
}

// Trilinear prolongation added to the interior of a dense level
// (CPU_PoissonSolver_MG.cpp:635-684)
template <typename T, int NT, int nc, int nf>
__device__ __forceinline__ void mg_prolongate(const T *c, T *f, int tid) {
  const T ratio = divide(T(nc - 1), T(nf - 1));
  constexpr int mf = nf - 2;
  for (int t = tid; t < mf * mf * mf; t += NT) {
    const int i = 1 + t % mf, j = 1 + (t / mf) % mf, k = 1 + t / (mf * mf);
    T wz[2], wy[2], wx[2];
    int bz, by, bx;
    mg_weights(k, ratio, wz[0], wz[1], bz);
    mg_weights(j, ratio, wy[0], wy[1], by);
    mg_weights(i, ratio, wx[0], wx[1], bx);
    const T zy[2][2] = {{mul(wz[0], wy[0]), mul(wz[0], wy[1])}, {mul(wz[1], wy[0]), mul(wz[1], wy[1])}};
    const int id = (k * nf + j) * nf + i;
    T q[2][2][2];
    mg_load4<T, nc>(c + (bz * nc + by) * nc + bx, q[0]);
    mg_load4<T, nc>(c + ((bz + 1) * nc + by) * nc + bx, q[1]);
    f[id] = add(f[id], mg_corners(zy, wx, q));
  }
}

// Bottom level by one warp, from a zero solution: 3^3 has one cell and one
// sweep, 4^3 eight cells (lane = their index bits x, y, z) and seven sweeps.
template <typename T, int nb, int sweeps>
__device__ __forceinline__ void mg_bottom(T *sol, const T *rhs, T dh, int lane) {
  const T dh2 = mul(dh, dh), one_six = divide(T(1), T(6)), zero = T(0);
  const int i = nb == 3 ? 0 : lane & 1, j = nb == 3 ? 0 : (lane >> 1) & 1, k = nb == 3 ? 0 : (lane >> 2) & 1;
  const int id = ((k + 1) * nb + j + 1) * nb + i + 1;
  const T b = mul(dh2, rhs[id]);
  T s = zero;
#pragma unroll 1
  for (int n = 0; n < 2 * sweeps; ++n) {
    // the other cell along each axis; the far side is the zero boundary, whose
    // addition changes nothing but the sign of a zero, in the first sum
    const T zo = nb == 3 ? zero : __shfl_xor_sync(0xffffffffu, s, 4), yo = nb == 3 ? zero : __shfl_xor_sync(0xffffffffu, s, 2),
            xo = nb == 3 ? zero : __shfl_xor_sync(0xffffffffu, s, 1);
    const T sum = add(add(add(zo, zero), yo), xo);
    if (((i + j + k + 3) & 1) != (n & 1)) s = mul(one_six, sub(sum, b));  // pass 0: i + j + k odd
  }
  if (lane < (nb == 3 ? 1 : 8)) sol[id] = s;
}

// the bottom level, and a level above it whose pairs fit one warp (ghost 5's 5^3;
// the first coarse level goes to all threads, whose restriction and prolongation
// are then shorter)
template <int G>
constexpr bool mg_one_warp(int lv) {
  const int n = MgLevels<G>::size(lv), m = n - 2;
  return lv == MgLevels<G>::L - 1 || (lv >= 2 && m * m * ((m + 1) / 2) <= 32);
}

// Level lv >= 1: its RHS is set and its solution zero; leaves the correction.
// The levels that one warp can hold are left to one warp, whose passes then need
// no block barrier; the others wait at its end.
template <typename T, int G, int NT, int lv>
__device__ __forceinline__ void mg_coarse(const SolveArgs<T> &a, T *sol, T *rhs, T *def, int tid) {
  using LV = MgLevels<G>;
  constexpr int n = LV::size(lv);
  T *s = sol + LV::offset(lv), *r = rhs + LV::offset(lv);
  const T dh = divide(mul(a.dh, T(LV::n0 - 1)), T(n - 1));
  if constexpr (NT > 32 && mg_one_warp<G>(lv)) {
    if (tid < 32) mg_coarse<T, G, 32, lv>(a, sol, rhs, def, tid);
    team_sync<NT>(0);
  } else if constexpr (lv == LV::L - 1) {
    mg_bottom<T, n, LV::nbottom>(s, r, dh, tid);
    __syncwarp();
  } else {
    constexpr int nn = LV::size(lv + 1);
    T *rn = rhs + LV::offset(lv + 1), *sn = sol + LV::offset(lv + 1);
    MgPairs<T, NT, n> pairs(tid);
    pairs.load_rhs(r);
    pairs.load_sol(s);
    pairs.smooth(s, dh, a.mg_npre);
    pairs.defect(s, def, dh);
    team_sync<NT>(0);
    mg_restrict<T, NT, n, nn>(
        [def](int bz, int by, int bx) GPG_INLINE {
          const T *f = def + (bz * n + by) * n + bx;
          return [f](int tz, int ty, int tx) GPG_INLINE { return f[(tz * n + ty) * n + tx]; };
        },
        rn, tid);
    if constexpr (lv + 1 < LV::L - 1)
      for (int t = tid; t < LV::cells(lv + 1); t += NT) sn[t] = T(0);
    team_sync<NT>(0);
    mg_coarse<T, G, NT, lv + 1>(a, sol, rhs, def, tid);
    mg_prolongate<T, NT, nn, n>(sn, s, tid);
    team_sync<NT>(0);
    pairs.load_sol(s);
    pairs.smooth(s, dh, a.mg_npost);
  }
}

template <typename T, int NT>
__device__ __forceinline__ void block_sum2(double &a, double &b, double *s_red, int tid) {
  constexpr int NWARP = NT / 32;
  a = warp_sum(a);
  b = warp_sum(b);
  if constexpr (NWARP > 1) {
    if ((tid & 31) == 0) {
      s_red[tid >> 5] = a;
      s_red[NWARP + (tid >> 5)] = b;
    }
    team_sync<NT>(0);
    a = s_red[0];
    b = s_red[NWARP];
#pragma unroll
    for (int w = 1; w < NWARP; ++w) {
      a += s_red[w];
      b += s_red[NWARP + w];
    }
    team_sync<NT>(0);
  }
}

// One pass of colour p over the lane's columns: the neighbour reads of the SOR's
// two-row pass (sor_pass2), with the update given.
// `update(r, z, sum)` returns the cell's new value from the sum of its
// neighbours (row r, local height z).
template <typename T, int G, int Z, int p, int SIDE, typename Update>
__device__ __forceinline__ void pass2_cells(T (&v)[2][2][SorCfg<T, G, Z, 2>::MH + 2], T *s_cube, const SorLane &ln,
                                            Update &&update) {
  using C = SorCfg<T, G, Z, 2>;
  constexpr int N = Geo<G>::N, MH = C::MH, P = C::P, PP = C::PP;
  const int own0 = ln.own, own1 = ln.own + P;
  const T *nb = s_cube + (1 - p) * N * PP + ln.zoff;
  T *mine = s_cube + p * N * PP + ln.zoff;
  if constexpr (Z == 2) sor_reload_split<T, MH, PP, P, 2, p>(v, nb, ln);
  // row y1's colour-c cell is on the left iff ((zz + c) even) == left_even and
  // row y0's is then on the right; left_even is true at compile time unless an
  // odd MH makes it depend on the column half
  constexpr bool RT = (Z == 2) && (MH & 1);
  const bool le = SIDE >= 0 ? SIDE == 1 : (RT ? ln.left_even : true);
  // sum of the six neighbours of row r's colour-p cell at height z; yreg is
  // the y neighbour held in registers (y0+1 for row 0, y1-1 for row 1), ysm
  // the one read from shared memory
  auto nbsum = [&](int z, int r, T yreg, T ysm, bool left, T xo) GPG_INLINE -> T {
    const T mate = v[r][1 - p][z];
    const T yp = r == 0 ? yreg : ysm, ym = r == 0 ? ysm : yreg;
    const T xp = left ? mate : xo, xm = left ? xo : mate;
    return add(add(add(add(add(v[r][1 - p][z + 1], v[r][1 - p][z - 1]), yp), ym), xp), xm);
  };
#pragma unroll
  for (int z = 1; z <= MH; ++z) {
    const bool left1 = (((z + p) & 1) == 0) == le, left0 = !left1;
    const T xo0 = nb[z * PP + own0 + (left0 ? -1 : 1)];
    const T ym0 = nb[z * PP + own0 - P];
    const T xo1 = nb[z * PP + own1 + (left1 ? -1 : 1)];
    const T yp1 = nb[z * PP + own1 + P];
    const T sum0 = nbsum(z, 0, v[1][1 - p][z], ym0, left0, xo0), sum1 = nbsum(z, 1, v[0][1 - p][z], yp1, left1, xo1);
    v[0][p][z] = update(0, z, sum0);
    v[1][p][z] = update(1, z, sum1);
  }
#pragma unroll
  for (int z = 1; z <= MH; ++z) {
    mine[z * PP + own0] = v[0][p][z];
    mine[z * PP + own1] = v[1][p][z];
  }
}

template <typename T, int G, bool WIDE = false>
__global__ void __launch_bounds__(MgCfg<T, G, WIDE>::TEAM, (MgCfg<T, G, WIDE>::blocks))
    mg_kernel(const SolveArgs<T> a) {
  using LV = MgLevels<G>;
  using g = Geo<G>;
  using K = MgCfg<T, G, WIDE>;
  using C = typename K::C;
  constexpr int N = g::N, M = g::M, Z = K::Z, NT = K::TEAM, P = C::P, PP = C::PP, MH = C::MH;
  constexpr int n1 = LV::size(1);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *s_cube = reinterpret_cast<T *>(smem_raw + K::cube), *s_sol = reinterpret_cast<T *>(smem_raw + K::sol),
    *s_rhs = reinterpret_cast<T *>(smem_raw + K::rhs), *s_def = reinterpret_cast<T *>(smem_raw + K::def),
    *s_w0 = reinterpret_cast<T *>(smem_raw + K::table), *s_w1 = s_w0 + N - 1;
  int *s_base = reinterpret_cast<int *>(s_w1 + N - 1);
  double *s_red = reinterpret_cast<double *>(smem_raw + K::red);
  const int tid = threadIdx.x;
  const int64_t P_ = blockIdx.x;
  pdl_wait();
  prefetch_patch<T, G, NT>(a, P_, tid);

  // level-0 solution = interpolated cube; coarse boundaries 0; prolongation weights
  interpolate<T, G, NT>(a.pot_in + P_ * g::PN3, tid, a.int_scheme, a.neg_zero,
                        [s_cube](int x, int y, int z, T v) GPG_INLINE { s_cube[C::addr(x, y, z)] = v; });
  for (int t = tid; t < LV::coarse; t += NT) s_sol[t] = T(0);
  for (int f = tid + 1; f <= M; f += NT) mg_weights(f, divide(T(n1 - 1), T(N - 1)), s_w0[f], s_w1[f], s_base[f]);
  team_sync<NT>(0);

  int y, h, zbase;
  SorLane ln;
  const bool active = sor_lane<T, G, Z, 2>(tid, y, h, zbase, ln);
  // whether its colour-c cell of row r at local height zz is the left one of the
  // pair (y is odd; the column half matters only where it is an odd number of heights)
  const int odd_base = (MH & 1) ? zbase & 1 : 0;
  auto is_left = [&](int r, int c, int zz) GPG_INLINE { return ((1 + r + odd_base + zz + c) & 1) == 0; };
  // the lane's columns and Poi_Coeff * rho, [row][colour][height]
  T v[2][2][MH + 2], rhs[2][2][MH];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int zz = 0; zz < MH + 2; ++zz) v[r][c][zz] = s_cube[(c * N + zbase + zz) * PP + ln.own + r * P];
#pragma unroll
      for (int zz = 1; zz <= MH; ++zz) {
        const int z = zbase + zz, x = is_left(r, c, zz) ? 2 * h + 1 : 2 * h + 2;
        rhs[r][c][zz - 1] = mul(a.poi_coeff, __ldg(a.rho + P_ * g::RHO3 + ((z - 1) * M + (y + r - 1)) * M + (x - 1)));
      }
    }
  const T dh = a.dh, dh2 = mul(dh, dh), m_dh2 = divide(T(-1), dh2), one_six = divide(T(1), T(6));

  // red-black sweeps of level 0
  auto smooth = [&](int sweeps) GPG_INLINE {
    if (sweeps <= 0) return;
    auto by_side = [&](auto f) GPG_INLINE {  // the side of the lane's cells, where that is warp-uniform
      if constexpr (C::HALF_UNIFORM) {
        if (ln.left_even) f(std::integral_constant<int, 1>{});
        else f(std::integral_constant<int, 0>{});
      } else {
        f(std::integral_constant<int, -1>{});
      }
    };
    if constexpr (sizeof(T) == 4) {
      PackState<MH> st;
      st.load(v, rhs);  // nc = -rhs
      const f32x2 nz = pack2(a.neg_zero, a.neg_zero), d2 = pack2(dh2, dh2), s6 = pack2(one_six, one_six);
#pragma unroll 1
      for (int q = 0; q < sweeps; ++q) {
        auto pass = [&](auto pc) GPG_INLINE {
          constexpr int p = decltype(pc)::value;
          if (active)
            by_side([&](auto side) GPG_INLINE {
              pass2_packed_cells<G, Z, false, p, decltype(side)::value>(
                  st, s_cube, ln,
                  [&](int r, int k, f32x2 sum) GPG_INLINE {
                    return fma2(s6, add2(sum, fma2(d2, st.nc[r][p][k], nz)), nz);
                  },
                  [&](int r, float sum) GPG_INLINE { return mul(one_six, add(sum, mul(dh2, st.ncs[r][p]))); });
            });
          team_sync<NT>(0);
        };
        pass(std::integral_constant<int, 0>{});
        pass(std::integral_constant<int, 1>{});
      }
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int zz = 1; zz <= MH; ++zz) v[r][c][zz] = st.at(r, c, zz);
    } else {
#pragma unroll 1
      for (int q = 0; q < sweeps; ++q) {
        auto pass = [&](auto pc) GPG_INLINE {
          constexpr int p = decltype(pc)::value;
          if (active)
            by_side([&](auto side) GPG_INLINE {
              pass2_cells<T, G, Z, p, decltype(side)::value>(v, s_cube, ln, [&](int r, int z, T sum) GPG_INLINE {
                return mul(one_six, sub(sum, mul(dh2, rhs[r][p][z - 1])));
              });
            });
          team_sync<NT>(0);
        };
        pass(std::integral_constant<int, 0>{});
        pass(std::integral_constant<int, 1>{});
      }
    }
  };
  // f(r, zz, defect) for the lane's colour-c cells (the other colour's cube planes hold the solution)
  auto defects = [&](auto cc, auto f) GPG_INLINE {
    constexpr int c = decltype(cc)::value;
    const T *nb0 = s_cube + (1 - c) * N * PP + ln.zoff, *nb = nb0 + ln.own;
    sor_reload_split<T, MH, PP, P, 2, c>(v, nb0, ln);
#pragma unroll
    for (int zz = 1; zz <= MH; ++zz)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const bool left = is_left(r, c, zz);
        const T xo = nb[zz * PP + r * P + (left ? -1 : 1)], ysm = nb[zz * PP + (r ? 2 * P : -P)];
        const T yreg = v[1 - r][1 - c][zz], mate = v[r][1 - c][zz];
        const T sum = add(add(add(add(add(v[r][1 - c][zz + 1], v[r][1 - c][zz - 1]), r ? ysm : yreg), r ? yreg : ysm),
                              left ? mate : xo), left ? xo : mate);
        f(r, zz, add(mul(m_dh2, sub(sum, mul(T(6), v[r][c][zz]))), rhs[r][c][zz - 1]));
      }
  };
  constexpr std::integral_constant<int, 0> c0{};
  constexpr std::integral_constant<int, 1> c1{};
  auto place = [&](int r, int c, int zz) GPG_INLINE -> T & {
    return s_cube[(c * N + zbase + zz) * PP + ln.own + r * P];
  };

  int iter = 0;
  double err = (double)FLT_MAX;
  const double tol = (double)a.mg_tol;
  while (iter < a.mg_max_iter && err > tol) {
    smooth(a.mg_npre);
    {
      // the defect takes the solution's place in the cube, read by the restriction
      // alone: colour 1 (from colour 0's planes) waits in registers until colour 0's
      // planes are free for colour 0's own
      T d[2][MH];
      if (active) defects(c1, [&](int r, int zz, T x) GPG_INLINE { d[r][zz - 1] = x; });
      team_sync<NT>(0);
      if (active) defects(c0, [&](int r, int zz, T x) GPG_INLINE { place(r, 0, zz) = x; });
      team_sync<NT>(0);
      if (active) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int zz = 1; zz <= MH; ++zz) place(r, 1, zz) = d[r][zz - 1];
      }
      team_sync<NT>(0);
    }
    mg_restrict<T, NT, N, n1>(
        [s_cube](int bz, int by, int bx) GPG_INLINE {
          // cells with an even step count share a colour; the middle x sits in the next slot iff bx is even
          const int s = (bx + by + bz + 1) & 1, step = !(bx & 1);
          const T *even = s_cube + (s * N + bz) * PP + by * P + ((bx + 1) >> 1);
          const T *odd = even + (s ? -N * PP : N * PP);
          return [even, odd, step](int tz, int ty, int tx) GPG_INLINE {
            const T *q = ((tz + ty + tx) & 1) ? odd : even;
            return q[tz * PP + ty * P + (tx == 0 ? 0 : tx == 2 ? 1 : step)];
          };
        },
        s_rhs, tid);
    for (int t = tid; t < LV::cells(1); t += NT) s_sol[t] = T(0);
    team_sync<NT>(0);
    mg_coarse<T, G, NT, 1>(a, s_sol, s_rhs, s_def, tid);
    // prolongation added to the lane's cells, which then return to the cube
    if (active) {
      T wx[2][2], wy[2][2];
      int bx[2], by[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int x = 2 * h + 1 + q;
        wx[q][0] = s_w0[x], wx[q][1] = s_w1[x], bx[q] = s_base[x];
        wy[q][0] = s_w0[y + q], wy[q][1] = s_w1[y + q], by[q] = s_base[y + q];
      }
      // up the column, the corners of the two coarse planes around a height stay in
      // registers; the base plane steps by at most one (every level ratio is at least 2)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const T *col[2] = {s_sol + by[r] * n1 + bx[0], s_sol + by[r] * n1 + bx[1]};
        int plane = s_base[zbase + 1];
        T q[2][2][2][2];  // [left, right][z][y][x]
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          mg_load4<T, n1>(col[e] + plane * n1 * n1, q[e][0]);
          mg_load4<T, n1>(col[e] + (plane + 1) * n1 * n1, q[e][1]);
        }
#pragma unroll
        for (int zz = 1; zz <= MH; ++zz) {
          const int z = zbase + zz;
          if (s_base[z] != plane) {
            plane = s_base[z];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
              for (int o = 0; o < 4; ++o) q[e][0][o >> 1][o & 1] = q[e][1][o >> 1][o & 1];
              mg_load4<T, n1>(col[e] + (plane + 1) * n1 * n1, q[e][1]);
            }
          }
          const T wz0 = s_w0[z], wz1 = s_w1[z];
          const T zy[2][2] = {{mul(wz0, wy[r][0]), mul(wz0, wy[r][1])}, {mul(wz1, wy[r][0]), mul(wz1, wy[r][1])}};
          const T dl = mg_corners(zy, wx[0], q[0]), dr = mg_corners(zy, wx[1], q[1]);
          const bool left0 = is_left(r, 0, zz);
          v[r][0][zz] = add(v[r][0][zz], left0 ? dl : dr);
          v[r][1][zz] = add(v[r][1][zz], left0 ? dr : dl);
          place(r, 0, zz) = v[r][0][zz];
          place(r, 1, zz) = v[r][1][zz];
        }
      }
    }
    team_sync<NT>(0);
    smooth(a.mg_npost);
    double sd = 0, ss = 0;
    if (active) {
      defects(c0, [&](int r, int zz, T x) GPG_INLINE {
        sd += (double)absval(x);
        ss += (double)absval(v[r][0][zz]);
      });
      defects(c1, [&](int r, int zz, T x) GPG_INLINE {
        sd += (double)absval(x);
        ss += (double)absval(v[r][1][zz]);
      });
    }
    block_sum2<T, NT>(sd, ss, s_red, tid);
    err = ((double)mul(dh, dh) * sd) / ss;
    ++iter;
  }
  if (tid == 0) {
    if (a.iters) a.iters[P_] = iter;
    if (a.resid) a.resid[P_] = err;
  }
  pdl_trigger();
  patch_output<T, G, NT>(a, P_, tid, [s_cube](int x, int y, int z) GPG_INLINE { return s_cube[C::addr(x, y, z)]; });
}

}  // namespace gpg
