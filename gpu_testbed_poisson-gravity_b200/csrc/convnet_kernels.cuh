// convnet_kernels.cuh -- tensor-core 3^3 convolutions of the learned
// initial-guess network (ghost-size-1 patches on their 10^3 solver cube): the
// per-layer forward, backward-data and weight-gradient kernels of training.
//
// Activation layout in global memory, bfloat16: [patch][12 planes][C/8 chunks]
// [136 rows][8 channels].  Plane z+1 holds cube plane z, planes 0 and 11 stay
// zero; row (y+1)*11 + (x+1) holds cell (x, y) of the plane, the other rows
// (one halo column per line, the lines before and after) stay zero.  So the
// neighbour (dx, dy) of a cell is the row dy*11 + dx further, and the 128-row
// MMA operand of a tap is the plane read from a shifted start row: no im2col
// gather, one shared-memory descriptor per (plane, tap, 16 channels).  A plane
// is one contiguous bulk copy.  (Gathering 27 x 64 bytes per row through L2, as
// these kernels did before, took 0.74 ms per 32 -> 32 layer of 1024 patches.)
//
// Work is split into units of `zc` planes of a patch, streamed plane by plane
// through shared memory by one persistent CTA per SM:
//   * loading lanes: bulk copies, one mbarrier per slot;
//   * issuing lanes: tcgen05.mma (M = 128 rows, K = 16, BF16 -> FP32 in TMEM);
//   * groups of four warps: epilogues of the finished planes (bias / ReLU, ReLU
//     mask, loss).
// An MMA of M 128 takes 43-48 cycles for any N up to 64 and 56 for N = 96 (the
// operand read of A bounds it).  So from 16 input channels on, a plane's window
// (dy, dx) is multiplied by the weights of all three dz at once, N = 3 x 32, into
// the accumulators of the planes z+1, z, z-1, which lie side by side in TMEM:
// 18 MMAs of 56 cycles per plane instead of 54 of 43.  An output plane still
// sums its taps in order (dz = -1 with plane z-1, then 0, then +1; inside it dy,
// dx, channels), as the one-kernel forward pass (convnet_infer.cuh) does.
// 32 -> 32 channels, 1024 patches: 0.74 ms with im2col gathers, 0.118 with one
// MMA per tap, 0.057 with the three dz together (of which about 0.008 is the
// kernel's start and end; the MMAs' own time is 0.043).
//
// A wait that gives up (about a second) sets *err; every role then stops, the
// copies and MMAs in flight are waited for (bounded) and TMEM is released.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "tc_common.cuh"

namespace gpg {
namespace net {

constexpr int kCells = 1000;  // 10^3 cube per patch
constexpr int kEdge = 10;
constexpr int kPlaneRows = 136;
constexpr int kPlaneLine = 11;                               // rows per line of a plane
constexpr int kFirstRow = 12, kLastRow = 120;                // rows of cells (0, 0) and (9, 9)
constexpr int kPlanes = 12;                                  // per patch, zero planes included
constexpr uint32_t kPlaneChunkBytes = kPlaneRows * 16;       // 2176
// values of a patch's activation with c channels
__host__ __device__ constexpr int64_t plane_elems(int c) { return int64_t(kPlanes) * (c / 8) * kPlaneRows * 8; }
// first value of (plane z + 1, chunk, row 0)
__host__ __device__ __forceinline__ int64_t plane_at(int64_t patch, int z, int chunk, int chunks) {
  return ((patch * kPlanes + z + 1) * chunks + chunk) * (kPlaneRows * 8);
}

enum { EPI_RELU = 0, EPI_MASK = 1, EPI_LOSS = 2, EPI_GUESS = 3 };

struct ConvArgs {
  const __nv_bfloat16 *x;   // input planes
  const __nv_bfloat16 *w;   // packed weights [KCH][NOUT][8]
  const float *bias;        // [NOUT] (not EPI_MASK)
  __nv_bfloat16 *y;         // output planes; EPI_MASK: the activation that masks, replaced in place;
                            // EPI_LOSS: planes of 16 channels whose channel 0 receives d loss / d y4
  const float *scale;       // [P] (EPI_LOSS, EPI_GUESS)
  const float *target;      // [P][8]^3 (EPI_LOSS)
  float *guess;             // [P][8]^3 (EPI_GUESS)
  double *loss_part;        // [gridDim.x] (EPI_LOSS)
  float *bias_part;         // [gridDim.x][32] column sums of what was stored (EPI_MASK, EPI_LOSS)
  double inv;               // 1 / interior cells of the batch
  int64_t npatch;
  int zc;                   // planes per unit
  int *err;
};

template <int CIN>
struct KChunks {
  static constexpr int CPT = CIN / 8;                     // 8-k chunks per tap
  static constexpr int REAL = 27 * CPT;
  static constexpr int KCH = (REAL + 1) / 2 * 2;          // even: whole K=16 MMAs
};

constexpr int kEpiWarps = 8;  // two groups of four
constexpr uint32_t kOverread = 256;  // a tile's last rows reach 15 rows past the plane

// Waits of an issuing warp.  After one has given up, the rest return at once and
// the warp runs through its (bounded) work without waiting: its control flow
// depends on nothing but the sizes, which keeps operands in uniform registers.
struct IssueWait {
  int *err;
  bool ok = true;
  __device__ __forceinline__ void operator()(uint64_t *bar, uint32_t parity) {
    if (ok) ok = tc::mbar_wait_warp(bar, parity, err);
  }
};

// Epilogue of one plane: thread t of a group of 128 owns row kFirstRow + t.
// fetch() loads what the epilogue needs besides the accumulator, for the plane
// after the current one, so that the loads' latency passes during a plane's work;
// turn() makes the fetched plane the current one.
template <int NOUT, int EPI>
struct PlaneEpilogue {
  static constexpr bool INTERIOR = EPI == EPI_LOSS || EPI == EPI_GUESS;  // planes 1..8 only
  static constexpr int NZ = INTERIOR ? 8 : 10, ZB = INTERIOR ? 1 : 0;
  static constexpr int NC = EPI == EPI_MASK ? 32 : 1;  // column sums kept
  const ConvArgs &a;
  int r, cx, cy;
  bool cell, inner;
  float bias[INTERIOR ? 1 : NOUT];
  float col[NC];
  double loss;
  struct Plane {
    uint4 mask[EPI == EPI_MASK ? 4 : 1];
    float want, scale;
    __nv_bfloat16 *out;
    int64_t in;
  } now, next;

  __device__ __forceinline__ PlaneEpilogue(const ConvArgs &args, int t) : a(args), loss(0.0) {
    r = kFirstRow + t;
    cy = r / kPlaneLine - 1;
    cx = r - (cy + 1) * kPlaneLine - 1;
    cell = cx >= 0 && r <= kLastRow;
    inner = cell && cx >= 1 && cx <= 8 && cy >= 1 && cy <= 8;
#pragma unroll
    for (int n = 0; n < (INTERIOR ? 1 : NOUT); ++n) bias[n] = EPI == EPI_MASK ? 0.f : a.bias[n];
#pragma unroll
    for (int n = 0; n < NC; ++n) col[n] = 0.f;
  }
  __device__ __forceinline__ void turn() { now = next; }
  __device__ __forceinline__ void fetch(int64_t p, int z) {
    Plane &f = next;
    if constexpr (EPI != EPI_GUESS) f.out = a.y + plane_at(p, z, 0, EPI == EPI_LOSS ? 2 : NOUT / 8) + r * 8;
    if constexpr (EPI == EPI_MASK) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        f.mask[c] = cell ? *reinterpret_cast<const uint4 *>(f.out + c * (kPlaneRows * 8)) : make_uint4(0, 0, 0, 0);
    }
    if constexpr (INTERIOR) {
      f.in = p * 512 + ((z - 1) * 8 + (cy - 1)) * 8 + (cx - 1);
      f.scale = a.scale[p];
      if constexpr (EPI == EPI_LOSS) f.want = inner ? a.target[f.in] : 0.f;
    }
  }
  __device__ __forceinline__ void after(const float (&acc)[NOUT]) {
    if constexpr (INTERIOR) {
      if (!inner) return;
      const float y4 = acc[0] + bias[0];
      if constexpr (EPI == EPI_GUESS) {
        a.guess[now.in] = y4 * now.scale;
      } else {
        const float tgt = now.want / now.scale;
        const double d = double(y4) - double(tgt);
        loss += d * d;
        const __nv_bfloat16 g = __float2bfloat16_rn(float(2.0 * d * a.inv));
        *now.out = g;
        col[0] += __bfloat162float(g);
      }
    } else if (cell) {
#pragma unroll
      for (int c = 0; c < NOUT / 8; ++c) {
        __align__(16) __nv_bfloat16 o[8];
        if constexpr (EPI == EPI_MASK) {
          const __nv_bfloat16 *mv = reinterpret_cast<const __nv_bfloat16 *>(&now.mask[c]);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            o[i] = __float2bfloat16_rn(__bfloat162float(mv[i]) > 0.f ? acc[c * 8 + i] : 0.f);
            col[c * 8 + i] += __bfloat162float(o[i]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __float2bfloat16_rn(fmaxf(acc[c * 8 + i] + bias[c * 8 + i], 0.f));
        }
        *reinterpret_cast<uint4 *>(now.out + c * (kPlaneRows * 8)) = *reinterpret_cast<const uint4 *>(o);
      }
    }
  }
  // the CTA's column sums and loss, over its kEpiWarps warps in order (all call it)
  __device__ __forceinline__ void finish(float *s_red, int warp, int lane) {
    if constexpr (EPI == EPI_MASK || EPI == EPI_LOSS) {
#pragma unroll
      for (int n = 0; n < NC; ++n) {
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) col[n] += __shfl_xor_sync(0xffffffffu, col[n], m);
        if (lane == n) s_red[warp * 32 + n] = col[n];
      }
      double *s_loss = reinterpret_cast<double *>(s_red + kEpiWarps * 32);
      if constexpr (EPI == EPI_LOSS) {
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, m);
        if (lane == 0) s_loss[warp] = loss;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
      const int tid = warp * 32 + lane;
      if (tid < NC) {
        float t = 0.f;
        for (int w = 0; w < kEpiWarps; ++w) t += s_red[w * 32 + tid];
        a.bias_part[blockIdx.x * 32 + tid] = t;
      }
      if (EPI == EPI_LOSS && tid == 0) {
        double t = 0.0;
        for (int w = 0; w < kEpiWarps; ++w) t += s_loss[w];
        a.loss_part[blockIdx.x] = t * a.inv;
      }
    }
  }
};

// wait for an accumulator (one lane polls), read it, clear it (ZERO), hand it
// back (ARRIVE; otherwise a later arrival of the caller does)
template <int NOUT, bool ZERO, bool ARRIVE = true>
__device__ __forceinline__ bool take_accumulator(uint64_t *full, uint32_t parity, uint64_t *empty, uint32_t taddr,
                                                 volatile int *s_abort, int *err, int lane, float (&acc)[NOUT]) {
  int got = 1;
  if (lane == 0) got = !*s_abort && tc::mbar_wait(full, parity, err);
  if (!__shfl_sync(0xffffffffu, got, 0)) return false;
  tc::fence_after_sync();
#pragma unroll
  for (int h = 0; h < NOUT / 16; ++h)
    tc::tmem_ld16(taddr + uint32_t(h * 16), *reinterpret_cast<float(*)[16]>(acc + h * 16));
  tc::tmem_wait_ld();
  if (ZERO) {
#pragma unroll
    for (int h = 0; h < NOUT / 16; ++h) tc::tmem_zero16(taddr + uint32_t(h * 16));
    tc::tmem_wait_st();
  }
  tc::fence_before_sync();
  if (ARRIVE) {
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(empty);
  }
  return true;
}

// ---------------------------------------------------------------------------
// First layer (8 input channels): an MMA's two K chunks are two taps, so a
// unit's planes sit side by side in one slot and every tap pair of a plane is an
// MMA of N = 32.
// ---------------------------------------------------------------------------
struct Conv1Cfg {
  static constexpr int SLOTS = 3, ACCS = 4;
  static constexpr uint32_t slot_bytes = kPlanes * kPlaneChunkBytes;
  static constexpr uint32_t w_bytes = KChunks<8>::KCH * 32 * 16;
  static constexpr uint32_t w_off = SLOTS * slot_bytes + kOverread;
  static constexpr uint32_t bar_off = w_off + w_bytes;
  static constexpr int BARS = 2 * SLOTS + 2 * ACCS + 2;  // full, empty per slot and accumulator; weights, end
  static constexpr uint32_t bytes = bar_off + BARS * 8 + 16;
  static constexpr int LOAD_WARP = kEpiWarps, ISSUE_WARP = kEpiWarps + 1;
  static constexpr int THREADS = (ISSUE_WARP + 1) * 32;
  static_assert(bytes <= 227 * 1024 && bar_off % 8 == 0 && w_off % 16 == 0, "shared memory");
};

__global__ void __launch_bounds__(Conv1Cfg::THREADS) conv1_kernel(const ConvArgs a) {
  using C = Conv1Cfg;
  constexpr int SLOTS = C::SLOTS, ACCS = C::ACCS, NOUT = 32;
  constexpr uint32_t IDESC = tc::idesc_bf16(128, NOUT, false, false), TMEM_COLS = ACCS * 32;
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + C::bar_off), *empty = full + SLOTS, *acc_full = empty + SLOTS,
           *acc_empty = acc_full + ACCS, *wbar = acc_empty + ACCS, *stop = wbar + 1;
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(stop + 1);
  volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  if (tid == 0) {
    for (int i = 0; i < SLOTS; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < ACCS; ++i) {
      tc::mbar_init(&acc_full[i], 1);
      tc::mbar_init(&acc_empty[i], 4);
    }
    tc::mbar_init(wbar, 1);
    tc::mbar_init(stop, 1);
    *s_abort = 0;
    tc::mbar_fence_init();
  }
  if (warp == C::ISSUE_WARP) {
    tc::tmem_alloc(s_tmem, TMEM_COLS);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *s_tmem;
  pdl_wait();
  const int zc = a.zc, upp = kEdge / zc;
  const int64_t nunit = a.npatch * upp;

  if (warp == C::LOAD_WARP) {
    if (lane == 0) {
      tc::mbar_arrive_expect_tx(wbar, C::w_bytes);
      tc::bulk_load(smem + C::w_off, a.w, C::w_bytes, wbar);
      uint32_t q = 0;  // slots filled
      for (int64_t u = blockIdx.x; u < nunit && !*s_abort; u += gridDim.x, ++q) {
        const int64_t p = u / upp;
        const int z0 = int(u - p * upp) * zc;
        const uint32_t s = q % SLOTS, bytes = (zc + 2) * kPlaneChunkBytes;
        if (q >= SLOTS && !tc::mbar_wait(&empty[s], (q / SLOTS - 1) & 1u, a.err)) {
          *s_abort = 1;
          break;
        }
        tc::mbar_arrive_expect_tx(&full[s], bytes);
        tc::bulk_load(smem + s * C::slot_bytes, a.x + plane_at(p, z0 - 1, 0, 1), bytes, &full[s]);
      }
      // the last copies land before the CTA leaves
      tc::mbar_wait(wbar, 0, nullptr);
      for (uint32_t k = q > SLOTS ? q - SLOTS : 0; k < q; ++k) tc::mbar_wait(&full[k % SLOTS], (k / SLOTS) & 1u, nullptr);
    }
  } else if (warp >= C::ISSUE_WARP) {
    const uint32_t ring = tc::smem_u32(smem), wbase = tc::smem_u32(smem + C::w_off);
    const uint64_t b0 = tc::smem_desc(wbase, NOUT * 16, 128);
    uint32_t q = 0, tile = 0;  // units and planes so far
    IssueWait wait{a.err};
    wait(wbar, 0);
    for (int64_t u = blockIdx.x; u < nunit; u += gridDim.x, ++q) {
      wait(&full[q % SLOTS], (q / SLOTS) & 1u);
      const uint32_t base = ring + (q % SLOTS) * C::slot_bytes;
      for (int t = 0; t < zc; ++t, ++tile) {
        const uint32_t buf = tile % ACCS;
        if (tile >= ACCS) wait(&acc_empty[buf], (tile / ACCS - 1) & 1u);
        tc::fence_after_sync();
        // pair (2j, 2j+1) of taps; 27 is a tap of zero weights
        auto row_of = [&](int tap) {
          return (t + tap / 9) * kPlaneRows + kFirstRow + ((tap / 3) % 3 - 1) * kPlaneLine + tap % 3 - 1;
        };
#pragma unroll
        for (int j = 0; j < 14; ++j) {
          const int r0 = row_of(2 * j), lbo = j < 13 ? (row_of(2 * j + 1) - r0) * 16 : 16;
          tc::mma_bf16_warp(tmem + buf * 32, tc::smem_desc(base + r0 * 16, lbo, 128), b0 + uint64_t(j * (2 * NOUT)),
                            IDESC, j > 0);
        }
        tc::mma_commit_warp(&acc_full[buf]);
      }
      tc::mma_commit_warp(&empty[q % SLOTS]);
    }
    if (!wait.ok) *s_abort = 1;
    tc::mma_commit_warp(stop);
    tc::mbar_wait(stop, 0, nullptr);  // the MMAs have ended
  } else {
    const int group = warp >> 2, quarter = warp & 3;  // planes group, group + 2, ...; TMEM lanes
    PlaneEpilogue<NOUT, EPI_RELU> epi(a, tid & 127);
    uint32_t tile = 0;
    bool ok = true;
    for (int64_t u = blockIdx.x; u < nunit && ok; u += gridDim.x) {
      const int64_t p = u / upp;
      const int z0 = int(u - p * upp) * zc;
      for (int t = 0; t < zc && ok; ++t, ++tile) {
        if (tile % (kEpiWarps / 4) != uint32_t(group)) continue;
        const uint32_t buf = tile % ACCS;
        epi.fetch(p, z0 + t);  // addresses alone
        epi.turn();
        float acc[NOUT];
        ok = take_accumulator<NOUT, false>(&acc_full[buf], (tile / ACCS) & 1u, &acc_empty[buf],
                                    tmem + (uint32_t(quarter * 32) << 16) + buf * 32, s_abort, a.err, lane, acc);
        if (ok) epi.after(acc);
      }
    }
    if (!ok) *s_abort = 1;
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == C::ISSUE_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// 16 or 32 input channels, three dz per MMA, weights packed
// [(dy, dx)][chunk][dz, n][8].  Window plane w of a unit adds to the planes w+1, w,
// w-1 of the unit.  A stream's planes take its eight accumulators in turn, plane
// n at TMEM column (7 - n % 8) * NOUT of its half, so a window's accumulators are
// adjacent columns in the order of dz = -1, 0, +1 -- except where the ring wraps
// (2 of 8 planes), which takes two runs of MMAs.  Every MMA accumulates: an
// accumulator is handed back cleared.
//
// Two streams per CTA, each with a loading lane, an issuing warp, an epilogue
// group and a ring of slots, share the weights.  A barrier wait or a commit of
// an issuing warp takes 100-300 cycles while MMAs saturate shared memory, and its
// queue of MMAs runs dry meanwhile; the other stream's MMAs fill that gap.  One
// wait (its lanes watch the slot and the accumulators together) and one commit
// per window keep it short.
// ---------------------------------------------------------------------------
template <int CIN, int NOUT>
struct ConvCfg {
  static constexpr int CPT = CIN / 8, STREAMS = 2, SLOTS = 4, ACCS = 8;
  // windows whose completion a barrier each records: more than the epilogue can
  // lag behind (eight planes of at most three windows)
  static constexpr int DONE = 32;
  static constexpr uint32_t slot_bytes = CPT * kPlaneChunkBytes;
  static constexpr uint32_t w_bytes = 27 * CPT * NOUT * 16;
  static constexpr uint32_t w_off = STREAMS * SLOTS * slot_bytes + kOverread;
  static constexpr uint32_t bar_off = w_off + w_bytes;
  static constexpr int PER = SLOTS + ACCS + DONE + 1, BARS = STREAMS * PER + 1;
  static constexpr uint32_t red_off = bar_off + BARS * 8 + 8;
  static constexpr uint32_t bytes = red_off + kEpiWarps * (32 * 4 + 8);
  static constexpr int LOAD_WARP = kEpiWarps, ISSUE_WARP = LOAD_WARP + STREAMS;
  static constexpr int THREADS = (ISSUE_WARP + STREAMS) * 32;
  static constexpr uint32_t TMEM_COLS = STREAMS * ACCS * NOUT;
  static_assert(bytes <= 227 * 1024 && bar_off % 8 == 0 && w_off % 16 == 0 && red_off % 8 == 0, "shared memory");
  static_assert(kEpiWarps == 4 * STREAMS && TMEM_COLS <= 512, "an epilogue group and accumulators per stream");
};

template <int CIN, int NOUT, int EPI>
__global__ void __launch_bounds__(ConvCfg<CIN, NOUT>::THREADS) conv_kernel(const ConvArgs a) {
  using C = ConvCfg<CIN, NOUT>;
  using E = PlaneEpilogue<NOUT, EPI>;
  constexpr int CPT = C::CPT, SLOTS = C::SLOTS, ACCS = C::ACCS, DONE = C::DONE, STREAMS = C::STREAMS;
  static_assert(NOUT == 16 || NOUT == 32, "N");
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::bar_off), *wbar = bars + C::BARS - 1;
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(wbar + 1);
  volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // a stream's barriers: slots full; accumulators cleared; windows done; end
  const int stream = warp < C::LOAD_WARP ? warp >> 2 : warp < C::ISSUE_WARP ? warp - C::LOAD_WARP : warp - C::ISSUE_WARP;
  uint64_t *full = bars + stream * C::PER, *acc_empty = full + SLOTS, *done = acc_empty + ACCS, *stop = done + DONE;

  if (tid == 0) {
    for (int i = 0; i < C::BARS; ++i) {
      const int k = i % C::PER;  // an accumulator is handed back by four warps
      tc::mbar_init(&bars[i], i < C::BARS - 1 && k >= SLOTS && k < SLOTS + ACCS ? 4 : 1);
    }
    *s_abort = 0;
    tc::mbar_fence_init();
  }
  if (warp == C::ISSUE_WARP) {
    tc::tmem_alloc(s_tmem, C::TMEM_COLS);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *s_tmem + stream * (ACCS * NOUT);
  if (warp < C::LOAD_WARP) {
    for (int h = 0; h < ACCS * NOUT / 16; ++h) tc::tmem_zero16(tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(h * 16));
    tc::tmem_wait_st();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  pdl_wait();
  const int zc = a.zc, upp = E::NZ / zc;
  const int64_t nunit = a.npatch * upp, first = blockIdx.x + int64_t(stream) * gridDim.x,
                step = int64_t(STREAMS) * gridDim.x;
  unsigned char *ring = smem + stream * SLOTS * C::slot_bytes;
  // a unit's patch, first plane, first and last window
  auto unit = [&](int64_t u, int64_t &p, int &z0, int &w0, int &w1) {
    p = u / upp;
    z0 = E::ZB + int(u - p * upp) * zc;
    w0 = z0 > 0 ? z0 - 1 : 0;
    w1 = z0 + zc < kEdge ? z0 + zc : kEdge - 1;
  };
  int64_t p;
  int z0, w0, w1;

  if (warp >= C::LOAD_WARP && warp < C::ISSUE_WARP) {
    if (lane == 0) {
      if (stream == 0) {
        tc::mbar_arrive_expect_tx(wbar, C::w_bytes);
        tc::bulk_load(smem + C::w_off, a.w, C::w_bytes, wbar);
      }
      uint32_t q = 0;  // windows loaded
      bool ok = true;
      for (int64_t u = first; u < nunit && ok && !*s_abort; u += step) {
        unit(u, p, z0, w0, w1);
        const __nv_bfloat16 *src = a.x + plane_at(p, w0, 0, CPT);
        for (int w = w0; w <= w1; ++w, ++q, src += C::slot_bytes / 2) {
          const uint32_t s = q % SLOTS, b = q - SLOTS;  // the window that had the slot before
          if (q >= SLOTS && !tc::mbar_wait(&done[b % DONE], (b / DONE) & 1u, a.err)) {
            ok = false;
            break;
          }
          tc::mbar_arrive_expect_tx(&full[s], C::slot_bytes);
          tc::bulk_load(ring + s * C::slot_bytes, src, C::slot_bytes, &full[s]);
        }
      }
      if (!ok) *s_abort = 1;
      // the last copies land before the CTA leaves
      if (stream == 0) tc::mbar_wait(wbar, 0, nullptr);
      for (uint32_t k = q > SLOTS ? q - SLOTS : 0; k < q; ++k) tc::mbar_wait(&full[k % SLOTS], (k / SLOTS) & 1u, nullptr);
    }
  } else if (warp >= C::ISSUE_WARP) {
    const uint32_t ring0 = tc::smem_u32(ring);
    const uint64_t b0 = tc::smem_desc(tc::smem_u32(smem + C::w_off), 3 * NOUT * 16, 128);
    uint32_t q = 0, n0 = 0, opened = 0;  // windows; planes of the units before; planes given an accumulator
    IssueWait wait{a.err};
    wait(wbar, 0);
    for (int64_t u = first; u < nunit; u += step, n0 += zc) {
      unit(u, p, z0, w0, w1);
      for (int w = w0; w <= w1; ++w, ++q) {
        const int hi = w + 1 < z0 + zc ? w + 1 : z0 + zc - 1, lo = w - 1 > z0 ? w - 1 : z0;
        // lanes 1 and 2 watch the accumulators this window opens, the others the slot
        const uint32_t opens = n0 + uint32_t(hi - z0) + 1 - opened, n = opened + lane - 1;
        const bool acc = lane >= 1 && uint32_t(lane) <= opens && n >= ACCS;
        wait(acc ? &acc_empty[n % ACCS] : &full[q % SLOTS], (acc ? n / ACCS - 1 : q / SLOTS) & 1u);
        opened += opens;
        tc::fence_after_sync();
        const uint64_t a0 = tc::smem_desc(ring0 + (q % SLOTS) * C::slot_bytes, kPlaneChunkBytes, 128);
        for (int top = hi; top >= lo;) {  // adjacent accumulators, highest plane first
          const int i = int((n0 + uint32_t(top - z0)) % ACCS), cnt = top - lo < i ? top - lo + 1 : i + 1;
          const uint32_t d = tmem + uint32_t((ACCS - 1 - i) * NOUT);
          const uint32_t idesc = tc::idesc_bf16(128, 0, false, false) | uint32_t(cnt * (NOUT / 8)) << 17;
          const uint64_t b = b0 + uint64_t((w - top + 1) * NOUT);  // dz = w - z, from -1
#pragma unroll
          for (int k = 0; k < 9 * (CPT / 2); ++k) {
            const int yx = k / (CPT / 2), h = k % (CPT / 2);
            const int off = kFirstRow + (yx / 3 - 1) * kPlaneLine + yx % 3 - 1 + 2 * h * kPlaneRows;
            tc::mma_bf16_warp(d, a0 + uint64_t(off), b + uint64_t(k * (2 * 3 * NOUT)), idesc, 1u);
          }
          top -= cnt;
        }
        tc::mma_commit_warp(&done[q % DONE]);
      }
    }
    if (!wait.ok) *s_abort = 1;
    tc::mma_commit_warp(stop);
    tc::mbar_wait(stop, 0, nullptr);  // the MMAs have ended
  } else {
    E epi(a, tid & 127);
    const uint32_t mine = tmem + (uint32_t((warp & 3) * 32) << 16);
    uint32_t n = 0, q0 = 0;  // planes; windows of the units before
    bool ok = true;
    if (first < nunit) {
      unit(first, p, z0, w0, w1);
      epi.fetch(p, z0);
    }
    for (int64_t u = first; u < nunit && ok; u += step) {
      unit(u, p, z0, w0, w1);
      for (int z = z0; z < z0 + zc && ok; ++z, ++n) {
        const uint32_t i = n % ACCS, q = q0 + uint32_t((z + 1 < w1 ? z + 1 : w1) - w0);  // its last window
        epi.turn();
        if (z + 1 < z0 + zc) {
          epi.fetch(p, z + 1);
        } else if (u + step < nunit) {
          int64_t pn;
          int zn, wn0, wn1;
          unit(u + step, pn, zn, wn0, wn1);
          epi.fetch(pn, zn);
        }
        float acc[NOUT];
        ok = take_accumulator<NOUT, true>(&done[q % DONE], (q / DONE) & 1u, &acc_empty[i], mine + (ACCS - 1 - i) * NOUT,
                                          s_abort, a.err, lane, acc);
        if (ok) epi.after(acc);
      }
      q0 += uint32_t(w1 - w0 + 1);
    }
    if (!ok) *s_abort = 1;
    pdl_trigger();
    epi.finish(reinterpret_cast<float *>(smem + C::red_off), warp, lane);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == C::ISSUE_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(*s_tmem, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// Weight gradient dW[tap][c][n] = sum over cells of X[cell + tap][c] G[cell][n]
// as MN-major MMAs whose K runs over the rows of a plane (7 steps of 16):
//   A (M = 128): copies of the gradient plane, copy j shifted by s_j rows --
//     3 copies of 32 channels with s = dx' in {-1, 0, 1}, or 9 copies of 8 with
//     s = 11 dy' + dx' for the last layer, whose gradient is channel 0 alone;
//   B (N = 96): the three input planes z-1, z, z+1 with their channels, which
//     are chunks one distance apart (N = 32 with 8 input channels: the fourth
//     plane's columns are not used), read dy rows shifted.
// D[(s, n)][(dz, c)] for each dy then holds the taps (dz, dy, dx = -s): 3 MMAs of
// N 96 (or one) per K step instead of 27 small products, the accumulators (up
// to 288 TMEM columns) staying for the CTA's whole life.  The shifted copies
// are made by the bulk copies themselves (the destination moves by 16 bytes per
// row; what neighbouring copies both write is zero in both).
// Each CTA leaves its sums in partial[cta][27 * CIN][NG]; a second kernel adds
// them in a fixed order.  1024 patches, 32 -> 32: 0.755 ms with im2col tiles
// gathered through L2, 0.061 so (MMAs 0.042; 0.39 MB per patch through L2).
// ---------------------------------------------------------------------------
struct WgradArgs {
  const __nv_bfloat16 *x;  // layer input planes
  const __nv_bfloat16 *g;  // gradient planes (wrt the pre-activation)
  float *partial;
  int64_t npatch;
  int zc;
  int *err;
};

// CIN input channels; GC channels of the gradient's planes, of which one (LAST)
// or all are used
template <int CIN, bool LAST>
struct WgradCfg {
  static constexpr int CPT = CIN / 8;
  static constexpr int GCHUNKS = LAST ? 2 : 4;             // chunks of a gradient plane in memory
  static constexpr int COPIES = LAST ? 9 : 3;
  static constexpr int NY = LAST ? 1 : 3;                  // row shifts of B
  static constexpr int N = CIN == 8 ? 32 : 96;
  static constexpr int NG = LAST ? 1 : 32;                 // output channels kept
  static constexpr int R0 = LAST ? 12 : 11;                // first K row
  static constexpr int ZMAX = 5;                           // planes per unit at most
  static constexpr uint32_t a_stride = LAST ? 2560 : kPlaneChunkBytes;  // between the 8-channel chunks of A
  static constexpr uint32_t copy_bytes = LAST ? a_stride : 4 * kPlaneChunkBytes;
  static constexpr uint32_t g_bytes = COPIES * copy_bytes;
  static constexpr int GSLOTS = 4, XSLOTS = 2;
  static constexpr uint32_t x_plane = CPT * kPlaneChunkBytes;
  static constexpr uint32_t x_bytes = (ZMAX + 2) * x_plane;
  static constexpr uint32_t x_off = GSLOTS * g_bytes;
  // A reads 16 chunks from a slot's start; with few input channels that can
  // pass the X slots' end, as can B's unused fourth plane
  static constexpr uint32_t tail = 16 * a_stride;
  static constexpr uint32_t bar_off = x_off + XSLOTS * x_bytes + (CIN == 8 ? tail : 0);
  static constexpr int BARS = 2 * GSLOTS + 2 * XSLOTS + 1;
  static constexpr int THREADS = (5 + NY) * 32;            // results, loads, an issuing warp per dy
  static constexpr uint32_t bytes = bar_off + BARS * 8 + 16;
  static constexpr uint32_t TMEM_COLS = NY * N <= 128 ? 128 : 512;
  static_assert(bytes <= 227 * 1024 && bar_off % 8 == 0 && x_off % 16 == 0, "shared memory");
  static_assert((GSLOTS - 1) * g_bytes + tail <= bar_off, "A's unused rows stay inside the kernel's memory");
};

template <int CIN, bool LAST>
__global__ void __launch_bounds__(WgradCfg<CIN, LAST>::THREADS) wgrad_kernel(const WgradArgs a) {
  using W = WgradCfg<CIN, LAST>;
  constexpr int GSLOTS = W::GSLOTS, XSLOTS = W::XSLOTS, N = W::N;
  constexpr uint32_t IDESC = tc::idesc_bf16(128, N, true, true);
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t *gfull = reinterpret_cast<uint64_t *>(smem + W::bar_off), *gempty = gfull + GSLOTS, *xfull = gempty + GSLOTS,
           *xempty = xfull + XSLOTS, *done = xempty + XSLOTS;
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(done + 1);
  volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  // rows between the shifted copies meet only zero rows of X, but have to be finite
  for (uint32_t i = tid; i < W::bar_off / 16; i += W::THREADS)
    reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    for (int i = 0; i < GSLOTS; ++i) {
      tc::mbar_init(&gfull[i], 1);
      tc::mbar_init(&gempty[i], W::NY);
    }
    for (int i = 0; i < XSLOTS; ++i) {
      tc::mbar_init(&xfull[i], 1);
      tc::mbar_init(&xempty[i], W::NY);
    }
    tc::mbar_init(done, W::NY);
    *s_abort = 0;
    tc::mbar_fence_init();
  }
  if (warp == 5) {
    tc::tmem_alloc(s_tmem, W::TMEM_COLS);
    tc::tmem_relinquish();
  }
  tc::fence_proxy_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *s_tmem;
  pdl_wait();
  const int zc = a.zc, upp = kEdge / zc;
  const int64_t nunit = a.npatch * upp;
  const bool any = blockIdx.x < nunit;

  if (warp == 4) {
    if (lane == 0) {
      uint32_t qx = 0, qg = 0;
      bool ok = true;
      for (int64_t u = blockIdx.x; u < nunit && ok && !*s_abort; u += gridDim.x, ++qx) {
        const int64_t p = u / upp;
        const int z0 = int(u - p * upp) * zc;
        const uint32_t sx = qx % XSLOTS;
        if (qx >= XSLOTS && !tc::mbar_wait(&xempty[sx], (qx / XSLOTS - 1) & 1u, a.err)) ok = false;
        if (!ok) break;
        tc::mbar_arrive_expect_tx(&xfull[sx], (zc + 2) * W::x_plane);
        tc::bulk_load(smem + W::x_off + sx * W::x_bytes, a.x + plane_at(p, z0 - 1, 0, W::CPT), (zc + 2) * W::x_plane,
                      &xfull[sx]);
        for (int t = 0; t < zc; ++t, ++qg) {
          const uint32_t sg = qg % GSLOTS;
          if (qg >= GSLOTS && !tc::mbar_wait(&gempty[sg], (qg / GSLOTS - 1) & 1u, a.err)) {
            ok = false;
            break;
          }
          const __nv_bfloat16 *src = a.g + plane_at(p, z0 + t, 0, W::GCHUNKS);
          constexpr uint32_t bytes = LAST ? kPlaneChunkBytes : 4 * kPlaneChunkBytes;
          tc::mbar_arrive_expect_tx(&gfull[sg], W::COPIES * bytes);
#pragma unroll
          for (int j = 0; j < W::COPIES; ++j) {
            const int s = LAST ? (j / 3 - 1) * kPlaneLine + j % 3 - 1 : j - 1;  // row m of copy j = row m + s
            tc::bulk_load(smem + int(sg * W::g_bytes + j * W::copy_bytes) - 16 * s, src, bytes, &gfull[sg]);
          }
        }
      }
      if (!ok) *s_abort = 1;
      for (uint32_t k = qx > XSLOTS ? qx - XSLOTS : 0; k < qx; ++k)
        tc::mbar_wait(&xfull[k % XSLOTS], (k / XSLOTS) & 1u, nullptr);
      for (uint32_t k = qg > GSLOTS ? qg - GSLOTS : 0; k < qg; ++k)
        tc::mbar_wait(&gfull[k % GSLOTS], (k / GSLOTS) & 1u, nullptr);
    }
  } else if (warp >= 5) {
    const int dy = warp - 5;  // this warp's accumulator columns
    const uint32_t gbase = tc::smem_u32(smem), xbase = tc::smem_u32(smem + W::x_off);
    uint32_t qx = 0, qg = 0;
    IssueWait wait{a.err};
    for (int64_t u = blockIdx.x; u < nunit; u += gridDim.x, ++qx) {
      for (int t = 0; t < zc; ++t, ++qg) {
        // lane 1 watches the unit's input planes, the others the gradient plane
        wait(lane == 1 ? &xfull[qx % XSLOTS] : &gfull[qg % GSLOTS], (lane == 1 ? qx / XSLOTS : qg / GSLOTS) & 1u);
        tc::fence_after_sync();
        const int row = W::R0 + (W::NY == 3 ? (dy - 1) * kPlaneLine : 0);
        const uint64_t a0 = tc::smem_desc(gbase + (qg % GSLOTS) * W::g_bytes + W::R0 * 16, 128, W::a_stride);
        const uint64_t x0 =
            tc::smem_desc(xbase + (qx % XSLOTS) * W::x_bytes + t * W::x_plane + row * 16, 128, kPlaneChunkBytes);
#pragma unroll
        for (int ks = 0; ks < 7; ++ks)
          tc::mma_bf16_warp(tmem + uint32_t(dy * N), a0 + uint64_t(16 * ks), x0 + uint64_t(16 * ks), IDESC,
                            (qg > 0 || ks > 0) ? 1u : 0u);
        tc::mma_commit_warp(&gempty[qg % GSLOTS]);
      }
      tc::mma_commit_warp(&xempty[qx % XSLOTS]);
    }
    if (!wait.ok) *s_abort = 1;
    tc::mma_commit_warp(done);
  }
  pdl_trigger();
  // every accumulation has ended (bounded wait, one thread)
  if (tid == 160) tc::mbar_wait(done, 0, a.err);
  __syncwarp();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp < 4) {
    float *out = a.partial + int64_t(blockIdx.x) * (27 * CIN * W::NG);
    const int j = LAST ? tid >> 3 : tid >> 5, n = LAST ? tid & 7 : tid & 31;
    const bool keep = j < W::COPIES && n < W::NG;
#pragma unroll 1
    for (int dy = 0; dy < W::NY; ++dy)
#pragma unroll 1
      for (int h = 0; h < N / 16; ++h) {
        float v[16];
        tc::tmem_ld16(tmem + (uint32_t(warp * 32) << 16) + uint32_t(dy * N + h * 16), v);
        tc::tmem_wait_ld();
        if (keep) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int colm = h * 16 + i, dz = colm / CIN, c = colm % CIN;
            // copy j holds shift s_j: its tap steps back by s_j
            const int tap = LAST ? dz * 9 + 8 - j : dz * 9 + dy * 3 + 2 - j;
            if (dz < 3) out[(tap * CIN + c) * W::NG + n] = any ? v[i] : 0.f;
          }
        }
      }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 5) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, W::TMEM_COLS);
  }
}

}  // namespace net
}  // namespace gpg
