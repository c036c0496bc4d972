// convnet_infer.cuh -- the whole forward pass of the learned initial guess in
// one persistent kernel: one patch at a time per CTA, its activations resident
// in shared memory from the interpolated input to the predicted interior.
//
// Layout: the padded planes of convnet_kernels.cuh (136 rows of 16 bytes per
// plane and 8 channels, zero halo rows), ten planes of 32 channels.  A plane's
// window is multiplied by the weights of all three dz in one MMA (N = 96; 48 for
// the last layer) into the accumulators of planes w+1, w, w-1, which are adjacent
// TMEM columns.  Input plane w is read by window w alone and output plane z is
// complete after window z+1, so every layer's output replaces its input in
// place, and the next layer's first windows run while the last planes' epilogues
// do.  The first layer (8 channels, a tap pair per MMA, N = 32) reads its own
// buffer, which is filled for the next patch meanwhile.
//
// Roles (16 warps):
//   * issuing warp: all MMAs in order, 10 windows per layer;
//   * scout warp: waits for what the next window needs and passes the word on
//     through a named barrier.  An mbarrier poll takes 100-300 cycles while MMAs
//     saturate shared memory, longer than the queue of issued MMAs lasts;
//   * 8 epilogue warps in two groups (planes of either parity): bias, ReLU, BF16
//     into the planes; layer 4 writes (y + b) * s of output channel 0 on the 8^3
//     interior straight to the guess array; accumulators go back cleared;
//   * 4 input warps: interpolate the next patch's coarse potential (CQUAD, same
//     arithmetic as the SOR), s = max |shell|, layer-1 planes;
//   * loading lane: each layer's weights with one bulk copy (this CTA alone) into
//     one of two slots, as soon as the layer before last has been multiplied.
// Every operation and its order matches the per-layer kernels of
// convnet_kernels.cuh (same K order per output row, same epilogue arithmetic),
// so both paths produce the same guess.
//
// Per patch 680 MMAs of 43 to 56 cycles each (M 128: the operand reads bound
// them), 34.7k cycles: 0.49 ms for 4096 patches on 148 SMs.  Measured 0.65 ms;
// 1.88 ms with one MMA of N = 32 per tap, two activation buffers and each layer's
// epilogue after its last MMA.
#pragma once

#include <cstdint>

#include "convnet_kernels.cuh"
#include "interp.cuh"
#include "tc_common.cuh"

namespace gpg {
namespace net {

constexpr int kInferEpi = 8, kInferIn = 4;                      // epilogue and input warps
constexpr int kInferLoad = kInferEpi + kInferIn, kInferIssue = kInferLoad + 1, kInferScout = kInferLoad + 2;
constexpr int kInferThreads = (kInferScout + 1) * 32;
constexpr int kInferWindows = 4 * kEdge;                        // per patch
constexpr uint32_t kActPlane = 4 * kPlaneChunkBytes;
constexpr uint32_t kSlotBytes = 27 * 32 * 32 * 2;               // the largest layer's weights

struct InferSmem {
  static constexpr uint32_t act = 0;                            // [10 planes][4 chunks][136 rows][8]
  static constexpr uint32_t x0 = act + kEdge * kActPlane + kOverread;   // [12 planes][136 rows][8]
  static constexpr uint32_t w = x0 + kPlanes * kPlaneChunkBytes + kOverread;  // two slots
  static constexpr uint32_t bias = w + 2 * kSlotBytes;          // 32 + 32 + 32 + 16 floats
  static constexpr uint32_t cube = bias + 112 * 4;              // interpolated cube of the input warps
  static constexpr uint32_t scale = cube + kCells * 4;          // s of the last four patches
  static constexpr uint32_t red = scale + 4 * 4;                // one float per input warp
  static constexpr uint32_t bars = red + kInferIn * 4;
  // barriers: weights full x 2, input planes full, per plane epilogue done, layer-4 accumulators cleared x 8,
  // windows done, end, test hook
  static constexpr int kFullW = 0, kFullX = 2, kEpi = 3, kAcc4 = kEpi + kEdge, kDone = kAcc4 + 8,
                       kStop = kDone + kInferWindows, kProbe = kStop + 1, kBars = kProbe + 1;
  static constexpr uint32_t tmem_slot = bars + kBars * 8;
  static constexpr uint32_t flag = tmem_slot + 4;
  static constexpr uint32_t bytes = flag + 4;
};
static_assert(InferSmem::bytes <= 232448, "shared memory per CTA");
static_assert(InferSmem::bars % 8 == 0 && InferSmem::w % 128 == 0 && InferSmem::x0 % 16 == 0, "alignment");

struct InferArgs {
  const float *rho;              // [P][8]^3
  const float *pot_in;           // [P][8]^3 coarse potential
  float *guess;                  // [P][8]^3
  const __nv_bfloat16 *w[4];     // packed forward operands: layer 1 [28][32][8], then [(dy, dx)][chunk][dz, n][8]
  const float *bias[4];          // FP32 biases (32, 32, 32, 16)
  float cnst;                    // Poi_Coeff * dh^2
  float neg_zero;                // as in SolveArgs
  int64_t npatch;
  int *err;
  int probe_polls;               // > 0: thread 0 also waits that many polls on a barrier nothing signals
};

__host__ __device__ constexpr uint32_t infer_weight_bytes(int l) {
  return l == 0 ? KChunks<8>::KCH * 32 * 16 : 27u * 32 * (l == 3 ? 16 : 32) * 2;
}
static_assert(infer_weight_bytes(1) == kSlotBytes && infer_weight_bytes(0) <= kSlotBytes, "weight slots");

// Scout and issuing warp meet before every window; true when either passes
// true (a wait gave up: both stop).
__device__ __forceinline__ bool window_sync(bool stop) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, 2, 64, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(stop ? 1u : 0u)
      : "memory");
  return r != 0;
}

__global__ void __launch_bounds__(kInferThreads, 1) net_infer_kernel(const InferArgs a) {
  using S = InferSmem;
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + S::bars);
  uint64_t *wfull = bars + S::kFullW, *xfull = bars + S::kFullX, *epi = bars + S::kEpi, *acc4 = bars + S::kAcc4,
           *done = bars + S::kDone, *stop = bars + S::kStop;
  float *s_bias = reinterpret_cast<float *>(smem + S::bias), *s_scale = reinterpret_cast<float *>(smem + S::scale);
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(smem + S::tmem_slot);
  volatile int *s_abort = reinterpret_cast<volatile int *>(smem + S::flag);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  // planes start at zero; only cells are ever written, so the halo rows stay zero
  for (uint32_t i = tid; i < S::w / 16; i += kInferThreads)
    reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < 112; i += kInferThreads)
    s_bias[i] = i < 32 ? a.bias[0][i] : i < 64 ? a.bias[1][i - 32] : i < 96 ? a.bias[2][i - 64] : a.bias[3][i - 96];
  if (tid == 0) {
    for (int i = 0; i < S::kBars; ++i)
      tc::mbar_init(&bars[i], i >= S::kFullX && i < S::kDone ? 4 : 1);  // four warps fill, or hand back
    *s_abort = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(s_tmem, 512);
    tc::tmem_relinquish();
  }
  tc::fence_proxy_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *s_tmem;
  // accumulators: plane z of layers 1-3 at column (9 - z) * 32, of layer 4 at 320 + (8 - z) * 16
  constexpr uint32_t kCols4 = kEdge * 32;
  if (warp < kInferEpi) {
    for (int h = warp >> 2; h < 28; h += kInferEpi / 4)
      tc::tmem_zero16(tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(h * 16));
    tc::tmem_wait_st();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (a.probe_polls > 0 && tid == 0) {
    // test hook: a bounded wait on a barrier nothing arrives on gives up
    // after probe_polls polls, records the timeout and the kernel goes on
    tc::mbar_wait_polls(bars + S::kProbe, 0, a.err, uint32_t(a.probe_polls));
  }
  const uint32_t npatch = a.npatch > blockIdx.x ? uint32_t((a.npatch - 1 - blockIdx.x) / gridDim.x + 1) : 0u;
  auto patch_of = [&](uint32_t i) { return int64_t(blockIdx.x) + int64_t(i) * gridDim.x; };

  if (warp == kInferLoad) {
    if (lane == 0) {
      uint32_t j = 0;
      for (; j < 4 * npatch && !*s_abort; ++j) {
        const uint32_t slot = j & 1u, l = j & 3u, b = j - 2;  // b: the layer that had the slot before
        if (j >= 2 && !tc::mbar_wait(&done[(b & 3u) * kEdge + kEdge - 1], (b >> 2) & 1u, a.err)) {
          *s_abort = 1;
          break;
        }
        const uint32_t bytes = l == 0 ? infer_weight_bytes(0) : l == 3 ? infer_weight_bytes(3) : infer_weight_bytes(1);
        tc::mbar_arrive_expect_tx(&wfull[slot], bytes);
        tc::bulk_load(smem + S::w + slot * kSlotBytes, a.w[l], bytes, &wfull[slot]);
      }
      // the last copies land before the CTA leaves
      for (uint32_t k = j > 2 ? j - 2 : 0; k < j; ++k) tc::mbar_wait(&wfull[k & 1u], (k >> 1) & 1u, nullptr);
    }
  } else if (warp == kInferScout) {
    // while the issuing warp issues a window, wait for what the next one needs
    bool ok = true;
    for (uint32_t i = 0; i < npatch && ok; ++i)
      for (int l = 0; l < 4 && ok; ++l)
        for (int w = 0; w < kEdge && ok; ++w) {
          // one barrier per lane:
          //  1: a layer's weights (first window)
          //  2: layer 1: the patch's input planes; later: plane w's epilogue of the layer before
          //  3: the accumulator opened last is cleared: plane w (layer 1: by the patch before) or w + 1
          //  4: layer 4: its accumulator of plane w + 1, by the patch before
          uint64_t *bar = nullptr;
          uint32_t phase = 0;  // completions of the barrier before the one to wait for
          if (lane == 1 && w == 0) {
            bar = &wfull[l & 1], phase = (4 * i + l) >> 1;
          } else if (lane == 2) {
            if (l > 0)
              bar = &epi[w], phase = 3 * i + l - 1;
            else if (w == 0)
              bar = xfull, phase = i;
          } else if (lane == 3) {
            const int z = l == 0 ? w : w + 1;
            if (l < 3 && z < kEdge && (l > 0 || i > 0)) bar = &epi[z], phase = 3 * i + l - 1;
          } else if (lane == 4) {
            if (l == 3 && w < 8 && i > 0) bar = &acc4[w], phase = i - 1;
          }
          const bool got = !bar || (!*s_abort && tc::mbar_wait(bar, phase & 1u, a.err));
          ok = __all_sync(0xffffffffu, got);
          window_sync(!ok);
        }
    if (!ok) *s_abort = 1;
  } else if (warp == kInferIssue) {
    constexpr uint32_t IDESC1 = tc::idesc_bf16(128, 32, false, false);
    const uint32_t act = tc::smem_u32(smem + S::act), x0 = tc::smem_u32(smem + S::x0), wslot = tc::smem_u32(smem + S::w);
    bool end = false;
    for (uint32_t i = 0; i < npatch && !end; ++i) {
      // layer 1: tap pairs (2j, 2j+1); 27 is a tap of zero weights
      for (int t = 0; t < kEdge && !end; ++t) {
        end = window_sync(false);
        if (end) break;
        tc::fence_after_sync();
        const uint64_t b0 = tc::smem_desc(wslot, 32 * 16, 128);
        auto row_of = [&](int tap) {
          return (t + tap / 9) * kPlaneRows + kFirstRow + ((tap / 3) % 3 - 1) * kPlaneLine + tap % 3 - 1;
        };
#pragma unroll
        for (int j = 0; j < 14; ++j) {
          const int r0 = row_of(2 * j), lbo = j < 13 ? (row_of(2 * j + 1) - r0) * 16 : 16;
          tc::mma_bf16_warp(tmem + uint32_t((kEdge - 1 - t) * 32), tc::smem_desc(x0 + r0 * 16, lbo, 128),
                            b0 + uint64_t(j * 64), IDESC1, 1u);
        }
        tc::mma_commit_warp(&done[t]);
      }
      for (int l = 1; l < 4 && !end; ++l) {
        const uint32_t nout = l == 3 ? 16 : 32;
        const uint64_t b0 = tc::smem_desc(wslot + (l & 1) * kSlotBytes, 3 * nout * 16, 128);
        const int zmin = l == 3 ? 1 : 0, zmax = l == 3 ? 8 : 9;
        for (int w = 0; w < kEdge && !end; ++w) {
          end = window_sync(false);
          if (end) break;
          tc::fence_after_sync();
          const int hi = w + 1 < zmax ? w + 1 : zmax, lo = w - 1 > zmin ? w - 1 : zmin;
          const uint32_t d = tmem + (l == 3 ? kCols4 + uint32_t(8 - hi) * 16 : uint32_t(9 - hi) * 32);
          const uint32_t idesc = tc::idesc_bf16(128, 0, false, false) | (uint32_t(hi - lo + 1) * (nout / 8)) << 17;
          const uint64_t a0 = tc::smem_desc(act + w * kActPlane, kPlaneChunkBytes, 128);
          const uint64_t b = b0 + uint64_t((w - hi + 1) * nout);  // dz = w - z, from -1
          const uint32_t bstep = 2 * 3 * nout;
#pragma unroll
          for (int q = 0; q < 18; ++q) {
            const int yx = q / 2, h = q % 2, off = kFirstRow + (yx / 3 - 1) * kPlaneLine + yx % 3 - 1 + 2 * h * kPlaneRows;
            tc::mma_bf16_warp(d, a0 + uint64_t(off), b + uint64_t(q * bstep), idesc, 1u);
          }
          tc::mma_commit_warp(&done[l * kEdge + w]);
        }
      }
    }
    tc::mma_commit_warp(stop);
    tc::mbar_wait(stop, 0, nullptr);  // the MMAs have ended
  } else if (warp >= kInferEpi) {
    // ---- input planes, one patch ahead ---------------------------------------
    const int t = tid - kInferEpi * 32;
    float *cube = reinterpret_cast<float *>(smem + S::cube), *red = reinterpret_cast<float *>(smem + S::red);
    auto sync = []() { asm volatile("bar.sync 1, %0;" ::"n"(kInferIn * 32) : "memory"); };
    bool ok = true;
    for (uint32_t i = 0; i < npatch; ++i) {
      const int64_t p = patch_of(i);
      sync();  // the previous patch's cube is read
      interpolate<float, 1, kInferIn * 32>(a.pot_in + p * Geo<1>::PN3, t, 4, a.neg_zero,
                                           [cube](int x, int y, int z, float v) { cube[(z * 10 + y) * 10 + x] = v; });
      sync();
      float mx = 0.f;
      for (int v = t; v < kCells; v += kInferIn * 32) {
        const int x = v % 10, y = (v / 10) % 10, z = v / 100;
        if (x == 0 || y == 0 || z == 0 || x == 9 || y == 9 || z == 9) mx = fmaxf(mx, fabsf(cube[v]));
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane == 0) red[warp - kInferEpi] = mx;
      sync();
      float s = red[0];
      for (int w = 1; w < kInferIn; ++w) s = fmaxf(s, red[w]);
      if (!(s > 0.f)) s = 1.f;
      if (t == 0) s_scale[i & 3u] = s;
      // layer 1 of the patch before has read the planes
      int got = 1;
      if (lane == 0 && i > 0) got = !*s_abort && tc::mbar_wait(&done[kEdge - 1], (i - 1) & 1u, a.err);
      if (!__shfl_sync(0xffffffffu, got, 0)) ok = false;
      for (int v = t; ok && v < kCells; v += kInferIn * 32) {
        const int x = v % 10, y = (v / 10) % 10, z = v / 100;
        const bool shell = x == 0 || y == 0 || z == 0 || x == 9 || y == 9 || z == 9;
        __align__(16) __nv_bfloat16 o[8];
        const float r = shell ? 0.f : __fmul_rn(a.cnst, a.rho[p * 512 + ((z - 1) * 8 + (y - 1)) * 8 + (x - 1)]) / s;
        o[0] = __float2bfloat16_rn(r);
        o[1] = __float2bfloat16_rn(shell ? cube[v] / s : 0.f);
        o[2] = __float2bfloat16_rn(shell ? 0.f : 1.f);
#pragma unroll
        for (int e = 3; e < 8; ++e) o[e] = __float2bfloat16_rn(0.f);
        const int row = (z + 1) * kPlaneRows + (y + 1) * kPlaneLine + x + 1;
        *reinterpret_cast<uint4 *>(smem + S::x0 + row * 16) = *reinterpret_cast<const uint4 *>(o);
      }
      tc::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(xfull);
    }
    if (!ok) *s_abort = 1;
  } else {
    // ---- epilogues ------------------------------------------------------------
    const int group = warp >> 2;
    const uint32_t lanes = tmem + (uint32_t((warp & 3) * 32) << 16);
    const int r = kFirstRow + (tid & 127), cy = r / kPlaneLine - 1, cx = r - (cy + 1) * kPlaneLine - 1;
    const bool cell = cx >= 0 && r <= kLastRow;
    const bool inner = cell && cx >= 1 && cx <= 8 && cy >= 1 && cy <= 8;
    bool ok = true;
    for (uint32_t i = 0; i < npatch && ok; ++i) {
      for (int l = 0; l < 3 && ok; ++l) {
        const float *bias = s_bias + 32 * l;
        for (int z = group; z < kEdge && ok; z += kInferEpi / 4) {
          float acc[32];
          const int w = l == 0 || z == kEdge - 1 ? z : z + 1;  // the plane's last window
          ok = take_accumulator<32, true, false>(&done[l * kEdge + w], i & 1u, nullptr, lanes + (kEdge - 1 - z) * 32,
                                                 s_abort, a.err, lane, acc);
          if (ok && cell) {
            unsigned char *dst = smem + S::act + z * kActPlane + r * 16;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              __align__(16) __nv_bfloat16 o[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __float2bfloat16_rn(fmaxf(acc[8 * c + e] + bias[8 * c + e], 0.f));
              *reinterpret_cast<uint4 *>(dst + c * kPlaneChunkBytes) = *reinterpret_cast<const uint4 *>(o);
            }
          }
          tc::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&epi[z]);
        }
      }
      const int64_t p = patch_of(i);
      const float s = s_scale[i & 3u];
      for (int z = 1 + group; z < kEdge - 1 && ok; z += kInferEpi / 4) {
        float acc[16];
        ok = take_accumulator<16, true, true>(&done[3 * kEdge + z + 1], i & 1u, &acc4[z - 1], lanes + kCols4 + (8 - z) * 16,
                                              s_abort, a.err, lane, acc);
        if (ok && inner) a.guess[p * 512 + ((z - 1) * 8 + (cy - 1)) * 8 + (cx - 1)] = (acc[0] + s_bias[96]) * s;
      }
    }
    if (!ok) *s_abort = 1;
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
}

}  // namespace net
}  // namespace gpg
