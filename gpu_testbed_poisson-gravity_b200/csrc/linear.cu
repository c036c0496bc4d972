// linear.cu -- the learned linear correction of the interpolated SOR start
// (gpg_lin_* in include/gpg.h): the fused solve of lin_sor.cuh, the training
// features, and training by gradient descent (FP32 kernels below, Adam).
//
// Model (block space, see lin_sor.cuh): per patch the folded residual
// u[8][64] and, for training, the folded target t[8][64] = H(phi* - phi_i)/8,
// phi* the converged solution; the prediction of block b is
// v_b = W[class(b)] u_b with W[4][64][64] (row = output orbit, column = input
// orbit, both in the class representative's axes).  The features come scaled
// by the power of two that brings the patch's max|phi_i| into [2^16, 2^17): a
// linear model is indifferent to the scale, and the training loss, the mean
// over patches, blocks and rows of e^2 with e = v - t, then measures each
// patch's start error relative to its potential -- the quantity the solve is
// judged by.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/gpg.h"
#include "arena.cuh"
#include "args.cuh"
#include "lin_sor.cuh"
#include "optim.cuh"

namespace {

using gpg::lin::kK;
using gpg::lin::kParams;

thread_local std::string g_lin_error;

int lfail(int status, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_lin_error = buf;
  return status;
}

#define LIN_CUDA(call)                                                                                 \
  do {                                                                                                 \
    cudaError_t e_ = (call);                                                                           \
    if (e_ != cudaSuccess)                                                                             \
      return lfail(e_ == cudaErrorMemoryAllocation ? GPG_ERR_OOM : GPG_ERR_CUDA, "%s: %s (%s:%d)", #call, \
                   cudaGetErrorString(e_), __FILE__, __LINE__);                                        \
  } while (0)

// class of block b: number of odd axes
__host__ __device__ constexpr int class_of(int b) { return (b & 1) + ((b >> 1) & 1) + ((b >> 2) & 1); }

// four consecutive values, in one 128-bit load where the pointer allows it
__device__ __forceinline__ float4 load4(const float *p) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) return __ldg(reinterpret_cast<const float4 *>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// place of parameter i = (class, row, k) in the two stacked A tiles
// [kc][row 0..127][8]: tile 0 = (class 0 ; class 3), tile 1 = (class 1 ; class 2)
__device__ __forceinline__ int tile_index(int i) {
  const int cls = i / (kK * kK), r = (i / kK) % kK, k = i % kK;
  const int t = (cls == 1 || cls == 2) ? 1 : 0, row = r + (cls >= 2 ? kK : 0);
  return t * 128 * kK + ((k >> 3) * 128 + row) * 8 + (k & 7);
}

// W[4][64][64] (FP32) -> the A tiles (BF16)
__global__ void lin_pack_kernel(const float *__restrict__ w, __nv_bfloat16 *__restrict__ tiles) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kParams) tiles[tile_index(i)] = __float2bfloat16_rn(w[i]);
}

// one Adam step and the operand tiles of the new weights
__global__ void lin_adam_kernel(const gpg::AdamArgs a, __nv_bfloat16 *__restrict__ tiles) {
  gpg::pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kParams) tiles[tile_index(i)] = __float2bfloat16_rn(gpg::adam_update(a, i));
}

// ---------------------------------------------------------------------------
// Gradient of the loss.  Two dense FP32 products per block b of class c,
//   E = W[c] U^T - T    (64 rows x patches),    G = E U    (64 x 64),
// 0.27 GFLOP for 2048 patches (3.6 us at the FP32 peak) over 8.4 MB of
// features.  CTA (b, j) takes the patches j, j + grid.y, ... in chunks of 64:
// W[c] transposed stays in shared memory, E lives there between the two
// products (each thread 4 rows x 4 patches, then 4 rows x 4 columns), and the
// CTA's G stays in registers until its chunks are done; the next chunk's
// features are loaded while the current one is multiplied.  grid.y = 37 puts
// two CTAs on each of 148 SMs (8 x 37 = 296) and bounds the partial sums to 4.8
// MB, which the second kernel adds in a fixed order.
// Training step (gradient, Adam, operand tiles) of 2048 patches: 1212 -> 18.6
// us (24.6 without the launches' overlap, see launch_after).
// (A thread that walks all patches for its row and column, as before, waits
// for 6144 dependent steps.)
// The error e = W u - t sums k in order, as the single-row form did.
// ---------------------------------------------------------------------------
constexpr int kGradSplit = 37;               // CTAs that share a block's patches
constexpr int kChunk = 64;                   // patches per step
constexpr int kGradThreads = 256;
inline int grad_splits(int npatch) { return std::min(kGradSplit, (npatch + kChunk - 1) / kChunk); }
constexpr int kPitchW = kK + 4;              // row pitches (words) that keep the 128-bit accesses aligned
struct GradSmem {
  float wt[kK][kPitchW];                     // W[c]^T: [k][row]
  float u[kChunk][kPitchW];                  // [patch][k]
  float e[kChunk][kPitchW];                  // [patch][row]
  double loss[kGradThreads / 32];
};

__global__ void __launch_bounds__(kGradThreads) lin_grad_kernel(const float *__restrict__ u,
                                                                const float *__restrict__ t,
                                                                const float *__restrict__ w, int npatch,
                                                                float *__restrict__ part,
                                                                double *__restrict__ loss_part) {
  extern __shared__ __align__(16) unsigned char lin_smem[];
  GradSmem &sm = *reinterpret_cast<GradSmem *>(lin_smem);
  const int b = blockIdx.x, tid = threadIdx.x, c = class_of(b);
  gpg::pdl_wait();
  for (int i = tid; i < kK * kK; i += kGradThreads) sm.wt[i % kK][i / kK] = w[c * kK * kK + i];
  const int r0 = (tid & 15) * 4;             // 4 rows of E and of G
  const int p0 = (tid >> 4) * 4;             // 4 patches of E
  const int k0 = p0;                         // 4 columns of G
  float g[4][4] = {};
  double loss = 0.0;
  constexpr int NQ = kChunk * kK / 4 / kGradThreads;
  const int64_t step = int64_t(gridDim.y) * kChunk;
  float4 next[NQ];
  auto fetch = [&](int64_t from) {  // this thread's share of the chunk at `from`
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int i = tid + q * kGradThreads, p = i / (kK / 4), k = (i % (kK / 4)) * 4;
      next[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (from + p < npatch) next[q] = load4(u + ((from + p) * 8 + b) * kK + k);
    }
  };
  fetch(int64_t(blockIdx.y) * kChunk);
  for (int64_t first = int64_t(blockIdx.y) * kChunk; first < npatch; first += step) {
    __syncthreads();  // the previous chunk's u and e are read; wt is written
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int i = tid + q * kGradThreads;
      *reinterpret_cast<float4 *>(&sm.u[i / (kK / 4)][(i % (kK / 4)) * 4]) = next[q];
    }
    float4 want[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      want[q] = first + p0 + q < npatch ? load4(t + ((first + p0 + q) * 8 + b) * kK + r0)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
    fetch(first + step);
    __syncthreads();
    float e[4][4] = {};
#pragma unroll 4
    for (int k = 0; k < kK; k += 4) {
      float x[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 uk = *reinterpret_cast<const float4 *>(&sm.u[p0 + q][k]);
        x[q][0] = uk.x, x[q][1] = uk.y, x[q][2] = uk.z, x[q][3] = uk.w;
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const float4 wk = *reinterpret_cast<const float4 *>(&sm.wt[k + kk][r0]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          e[q][0] = fmaf(wk.x, x[q][kk], e[q][0]);
          e[q][1] = fmaf(wk.y, x[q][kk], e[q][1]);
          e[q][2] = fmaf(wk.z, x[q][kk], e[q][2]);
          e[q][3] = fmaf(wk.w, x[q][kk], e[q][3]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
      if (first + p0 + q < npatch) {
        const float4 x = want[q];
        d = make_float4(e[q][0] - x.x, e[q][1] - x.y, e[q][2] - x.z, e[q][3] - x.w);
        loss += double(d.x) * d.x + double(d.y) * d.y + (double(d.z) * d.z + double(d.w) * d.w);
      }
      *reinterpret_cast<float4 *>(&sm.e[p0 + q][r0]) = d;
    }
    __syncthreads();
#pragma unroll 8
    for (int p = 0; p < kChunk; ++p) {
      const float4 x = *reinterpret_cast<const float4 *>(&sm.e[p][r0]);
      const float4 y = *reinterpret_cast<const float4 *>(&sm.u[p][k0]);
      const float xe[4] = {x.x, x.y, x.z, x.w}, yu[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) g[i][j] = fmaf(xe[i], yu[j], g[i][j]);
    }
  }
  gpg::pdl_trigger();
  const int slot = blockIdx.y * 8 + b;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4 *>(part + (int64_t(slot) * kK + r0 + i) * kK + k0) =
        make_float4(g[i][0], g[i][1], g[i][2], g[i][3]);
  loss = gpg::warp_sum(loss);
  if ((tid & 31) == 0) sm.loss[tid >> 5] = loss;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int q = 0; q < kGradThreads / 32; ++q) s += sm.loss[q];
    loss_part[slot] = s;
  }
}

// grad[c] = 2 / (npatch 512) sum of its blocks' partial sums; the loss from
// the same kernel's partials (fixed orders).  Four threads share a value's
// partials, so that no thread waits for more than ten loads of a block.
__global__ void __launch_bounds__(256) lin_reduce_kernel(const float *__restrict__ part,
                                                         const double *__restrict__ loss_part, int nsplit, int npatch,
                                                         float *__restrict__ grad, float *__restrict__ loss) {
  __shared__ float sums[4][64];
  const int v = threadIdx.x & 63, q = threadIdx.x >> 6, i = blockIdx.x * 64 + v;
  const int c = i / (kK * kK), rk = i % (kK * kK);
  gpg::pdl_wait();
  gpg::pdl_trigger();
  float s = 0.f;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    if (class_of(b) != c) continue;
    float x[(kGradSplit + 3) / 4];  // all loads of a block in flight together
#pragma unroll
    for (int j = 0; j < (kGradSplit + 3) / 4; ++j)
      x[j] = q + 4 * j < nsplit ? part[int64_t((q + 4 * j) * 8 + b) * kK * kK + rk] : 0.f;
#pragma unroll
    for (int j = 0; j < (kGradSplit + 3) / 4; ++j) s += x[j];
  }
  sums[q][v] = s;
  __syncthreads();
  if (q == 0) grad[i] = ((sums[0][v] + sums[1][v]) + (sums[2][v] + sums[3][v])) * (2.f / (float(npatch) * 512.f));
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    double l = 0.0;
    for (int j = threadIdx.x; j < nsplit * 8; j += 32) l += loss_part[j];
    l = gpg::warp_sum(l);
    if (threadIdx.x == 0) *loss = float(l / (double(npatch) * 512.0));
  }
}

}  // namespace

struct gpg_lin {
  int device = 0;
  int max_batch = 0;
  int step = 0;
  int probe_polls = 0;
  void *block = nullptr;  // holds all arrays below
  float *params = nullptr, *grad = nullptr, *adam_m = nullptr, *adam_v = nullptr;
  float *part = nullptr, *loss = nullptr;  // partial gradients [kGradSplit * 8][64][64]
  double *loss_part = nullptr;
  __nv_bfloat16 *tiles = nullptr;
  int *err = nullptr;
  int variant = 0;                   // launch shape of the fused solve
  int grid[2] = {0, 0};              // persistent CTAs per shape (one per SM)
};

namespace {

int repack(gpg_lin *l, cudaStream_t s) {
  lin_pack_kernel<<<kParams / 256, 256, 0, s>>>(l->params, l->tiles);
  LIN_CUDA(cudaGetLastError());
  return GPG_OK;
}

// Launch shapes of the fused solve (identical results): 0 = two groups of 8
// teams with staged inputs, 1 = three groups of 8 teams reading their inputs
// from global memory.
constexpr int kLinVariants = 2;

template <bool FEATURES, int HALVES, bool STAGE>
int prepare(int *grid) {
  auto fn = gpg::lin::lin_sor_kernel<FEATURES, HALVES, STAGE>;
  using L = gpg::lin::Layout<HALVES, STAGE>;
  LIN_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(L::bytes)));
  LIN_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                int(cudaSharedmemCarveoutMaxShared)));
  if (grid) {
    int dev = 0, sms = 0;
    LIN_CUDA(cudaGetDevice(&dev));
    LIN_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    *grid = sms;  // one CTA per SM: its shared memory and TMEM take the whole SM
  }
  return GPG_OK;
}

// persistent CTAs for npatch patches: HALVES batches of 8 per CTA at a time
int lin_grid(int halves, int grid_max, int npatch) {
  const int64_t nbatch = (int64_t(npatch) + gpg::lin::kHalfWarps - 1) / gpg::lin::kHalfWarps;
  const int64_t need = (nbatch + halves - 1) / halves;
  return int(need < grid_max ? need : grid_max);
}

int check_solve_params(const gpg_params *p) {
  if (int rc = gpg_validate_params(p)) return lfail(rc, "%s", gpg_last_error());
  if (p->real_size != 4 || p->ghost != 1 || p->scheme != GPG_SOR || !p->poisson)
    return lfail(GPG_ERR_UNSUPPORTED, "the learned start covers ghost-size-1 FP32 SOR (real_size %d, ghost %d, scheme %d)",
                 p->real_size, p->ghost, p->scheme);
  return GPG_OK;
}

}  // namespace

extern "C" const char *gpg_lin_last_error(void) { return g_lin_error.c_str(); }

extern "C" int gpg_lin_param_count(int64_t *count) {
  if (!count) return lfail(GPG_ERR_INVALID, "count is NULL");
  *count = kParams;
  return GPG_OK;
}

extern "C" int gpg_lin_create(gpg_lin **out, int max_batch, int device_id) {
  if (!out) return lfail(GPG_ERR_INVALID, "lin is NULL");
  *out = nullptr;
  if (max_batch < 1 || max_batch > (1 << 22)) return lfail(GPG_ERR_INVALID, "max_batch %d", max_batch);
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device_id < 0 || device_id >= count)
    return lfail(GPG_ERR_NO_DEVICE, "device %d of %d", device_id, count);
  LIN_CUDA(cudaSetDevice(device_id));
  int major = 0, minor = 0;
  LIN_CUDA(gpg::compute_capability(device_id, &major, &minor));
  if (major != 10) return lfail(GPG_ERR_UNSUPPORTED, "tensor-core kernels need sm_100 (found sm_%d%d)", major, minor);
  gpg_lin *l = new gpg_lin;
  l->device = device_id;
  l->max_batch = max_batch;
  gpg::Arena arena;
  arena.add(l->err, 1);
  arena.add(l->params, kParams);
  arena.add(l->adam_m, kParams);
  arena.add(l->adam_v, kParams);
  arena.zeroed_to_here();
  arena.add(l->grad, kParams);
  arena.add(l->tiles, gpg::lin::kTileBytes);  // two tiles of 2-byte values
  const size_t splits = grad_splits(max_batch);
  arena.add(l->part, splits * 8 * kK * kK);
  arena.add(l->loss_part, splits * 8);
  arena.add(l->loss, 1);
  cudaError_t e = arena.allocate(&l->block);
  if (e != cudaSuccess) {
    gpg_lin_destroy(l);
    return lfail(e == cudaErrorMemoryAllocation ? GPG_ERR_OOM : GPG_ERR_CUDA, "allocation: %s", cudaGetErrorString(e));
  }
  // attributes here, so that a stream capture never sees first-use set-up
  int rc = prepare<false, 2, true>(&l->grid[0]);
  if (!rc) rc = prepare<false, 3, false>(&l->grid[1]);
  if (!rc) rc = prepare<true, 2, false>(nullptr);
  if (!rc && cudaFuncSetAttribute(lin_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(sizeof(GradSmem))) != cudaSuccess)
    rc = lfail(GPG_ERR_CUDA, "shared memory of the gradient kernel: %s", cudaGetErrorString(cudaGetLastError()));
  if (rc) {
    gpg_lin_destroy(l);
    return rc;
  }
  if (int rc = repack(l, 0)) {
    gpg_lin_destroy(l);
    return rc;
  }
  LIN_CUDA(cudaDeviceSynchronize());
  *out = l;
  return GPG_OK;
}

extern "C" int gpg_lin_destroy(gpg_lin *l) {
  if (!l) return GPG_OK;
  cudaSetDevice(l->device);
  cudaFree(l->block);
  delete l;
  return GPG_OK;
}

extern "C" int gpg_lin_get_params(gpg_lin *l, float *host) {
  if (!l || !host) return lfail(GPG_ERR_INVALID, "NULL argument");
  LIN_CUDA(cudaSetDevice(l->device));
  LIN_CUDA(cudaDeviceSynchronize());  // training steps on any stream
  LIN_CUDA(cudaMemcpy(host, l->params, kParams * 4, cudaMemcpyDeviceToHost));
  return GPG_OK;
}

extern "C" int gpg_lin_set_params(gpg_lin *l, const float *host) {
  if (!l || !host) return lfail(GPG_ERR_INVALID, "NULL argument");
  LIN_CUDA(cudaSetDevice(l->device));
  // calls before and after may be on streams that the default stream does not order
  LIN_CUDA(cudaDeviceSynchronize());
  LIN_CUDA(cudaMemcpy(l->params, host, kParams * 4, cudaMemcpyHostToDevice));
  LIN_CUDA(cudaMemset(l->adam_m, 0, kParams * 4));
  LIN_CUDA(cudaMemset(l->adam_v, 0, kParams * 4));
  l->step = 0;
  if (int rc = repack(l, 0)) return rc;
  LIN_CUDA(cudaDeviceSynchronize());
  return GPG_OK;
}

extern "C" int gpg_lin_solve_device(gpg_lin *l, const gpg_params *p, int npatch, const float *d_rho,
                                    const float *d_pot_in, float *d_pot_out, float *d_flu, int32_t *d_iters,
                                    double *d_resid, void *stream) {
  if (!l) return lfail(GPG_ERR_INVALID, "lin is NULL");
  if (int rc = check_solve_params(p)) return rc;
  if (npatch < 0) return lfail(GPG_ERR_INVALID, "npatch %d", npatch);
  if (npatch == 0) return GPG_OK;
  if (!d_rho || !d_pot_in || !d_pot_out || (p->gra_acc && !d_flu)) return lfail(GPG_ERR_INVALID, "NULL array");
  LIN_CUDA(cudaSetDevice(l->device));
  // the inputs are staged with bulk copies of whole patches
  if ((reinterpret_cast<uintptr_t>(d_rho) | reinterpret_cast<uintptr_t>(d_pot_in)) & 15)
    return lfail(GPG_ERR_INVALID, "d_rho and d_pot_in must be 16-byte aligned");
  gpg_params q = *p;
  q.init_mode = GPG_INIT_INTERP;  // the correction is added to the interpolated start
  gpg::lin::LinArgs a{};
  a.s = gpg::make_args<float>(q, npatch, d_rho, d_pot_in, d_pot_out, d_flu, nullptr, d_iters, d_resid);
  a.wtiles = l->tiles;
  a.err = l->err;
  a.probe_polls = l->probe_polls;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the set-up overlaps the end of the kernel before (300 patches, back to back:
  // 16.7 -> 13.6 us; 4096 28.7 -> 25.4)
  if (l->variant == 0) {
    using SH = gpg::lin::Shape<2, true>;
    LIN_CUDA(gpg::launch_after(gpg::lin::lin_sor_kernel<false, 2, true>, lin_grid(2, l->grid[0], npatch), SH::kThreads,
                               gpg::lin::Layout<2, true>::bytes, s, a));
  } else {
    using SH = gpg::lin::Shape<3, false>;
    LIN_CUDA(gpg::launch_after(gpg::lin::lin_sor_kernel<false, 3, false>, lin_grid(3, l->grid[1], npatch), SH::kThreads,
                               gpg::lin::Layout<3, false>::bytes, s, a));
  }
  return GPG_OK;
}

extern "C" int gpg_lin_features(gpg_lin *l, const gpg_params *p, int npatch, const float *d_rho,
                                const float *d_pot_in, const float *d_target, float *d_u, float *d_t,
                                void *stream) {
  if (!l) return lfail(GPG_ERR_INVALID, "lin is NULL");
  if (int rc = check_solve_params(p)) return rc;
  if (npatch < 0) return lfail(GPG_ERR_INVALID, "npatch %d", npatch);
  if (npatch == 0) return GPG_OK;
  if (!d_rho || !d_pot_in || !d_u || (d_target && !d_t)) return lfail(GPG_ERR_INVALID, "NULL array");
  LIN_CUDA(cudaSetDevice(l->device));
  gpg_params q = *p;
  q.init_mode = GPG_INIT_INTERP;
  q.gra_acc = 0;
  gpg::lin::LinArgs a{};
  a.s = gpg::make_args<float>(q, npatch, d_rho, d_pot_in, nullptr, nullptr, nullptr, nullptr, nullptr);
  a.u_out = d_u;
  a.t_out = d_t;
  a.target = d_target;
  a.err = l->err;
  gpg::lin::lin_sor_kernel<true, 2, false>
      <<<lin_grid(2, l->grid[0], npatch), gpg::lin::Shape<2, false>::kThreads, gpg::lin::Layout<2, false>::bytes,
         static_cast<cudaStream_t>(stream)>>>(a);
  LIN_CUDA(cudaGetLastError());
  return GPG_OK;
}

extern "C" int gpg_lin_gradients(gpg_lin *l, int npatch, const float *d_u, const float *d_t, float *d_grad,
                                 float *d_loss, void *stream) {
  if (!l) return lfail(GPG_ERR_INVALID, "lin is NULL");
  if (npatch < 1 || npatch > l->max_batch) return lfail(GPG_ERR_INVALID, "npatch %d (1..%d)", npatch, l->max_batch);
  if (!d_u || !d_t) return lfail(GPG_ERR_INVALID, "NULL array");
  LIN_CUDA(cudaSetDevice(l->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int nsplit = grad_splits(npatch);
  LIN_CUDA(gpg::launch_after(lin_grad_kernel, dim3(8, nsplit), kGradThreads, sizeof(GradSmem), s, d_u, d_t, l->params,
                             npatch, l->part, l->loss_part));
  LIN_CUDA(gpg::launch_after(lin_reduce_kernel, kParams / 64, 256, 0, s, l->part, l->loss_part, nsplit, npatch,
                             d_grad ? d_grad : l->grad, d_loss ? d_loss : l->loss));
  return GPG_OK;
}

namespace {
int lin_adam(gpg_lin *l, const float *grad, float lr, cudaStream_t s) {
  l->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, float(l->step)), c2 = 1.f - std::pow(b2, float(l->step));
  LIN_CUDA(gpg::launch_after(lin_adam_kernel, kParams / 256, 256, 0, s,
                             gpg::AdamArgs{l->params, l->adam_m, l->adam_v, grad, lr, b1, b2, 1e-8f, c1, c2}, l->tiles));
  return GPG_OK;
}
}  // namespace

extern "C" int gpg_lin_train_step(gpg_lin *l, int npatch, const float *d_u, const float *d_t, float lr,
                                  float *d_loss, void *stream) {
  if (int rc = gpg_lin_gradients(l, npatch, d_u, d_t, nullptr, d_loss, stream)) return rc;
  return lin_adam(l, l->grad, lr, static_cast<cudaStream_t>(stream));
}

extern "C" int gpg_lin_apply_gradient(gpg_lin *l, const float *d_grad, float lr, void *stream) {
  if (!l || !d_grad) return lfail(GPG_ERR_INVALID, "NULL argument");
  LIN_CUDA(cudaSetDevice(l->device));
  return lin_adam(l, d_grad, lr, static_cast<cudaStream_t>(stream));
}

extern "C" int gpg_lin_check(gpg_lin *l) {
  if (!l) return lfail(GPG_ERR_INVALID, "lin is NULL");
  LIN_CUDA(cudaSetDevice(l->device));
  int flag = 0;
  LIN_CUDA(cudaMemcpy(&flag, l->err, 4, cudaMemcpyDeviceToHost));
  if (flag) {
    LIN_CUDA(cudaMemset(l->err, 0, 4));
    return lfail(GPG_ERR_CUDA, "a tensor-core wait timed out");
  }
  return GPG_OK;
}

extern "C" int gpg_lin_variant_count(void) { return kLinVariants; }

extern "C" int gpg_lin_set_variant(gpg_lin *l, int variant) {
  if (!l) return lfail(GPG_ERR_INVALID, "lin is NULL");
  if (variant < 0 || variant >= kLinVariants) return lfail(GPG_ERR_INVALID, "variant %d", variant);
  l->variant = variant;
  return GPG_OK;
}

extern "C" int gpg_lin_set_wait_probe(gpg_lin *l, int polls) {
  if (!l) return lfail(GPG_ERR_INVALID, "lin is NULL");
  if (polls < 0) return lfail(GPG_ERR_INVALID, "polls %d", polls);
  l->probe_polls = polls;
  return GPG_OK;
}
