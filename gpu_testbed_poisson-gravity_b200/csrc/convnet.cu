// convnet.cu -- the learned initial guess for ghost-size-1 SOR: a 4-layer
// 3^3 convolution network (8 -> 32 -> 32 -> 32 -> 16 channels, ReLU, output
// channel 0 used) that maps a patch's density and interpolated boundary shell
// to its interior potential.  Forward, backward and the Adam update run on the
// tensor-core kernels of convnet_kernels.cuh and the small kernels below;
// weights are FP32 masters packed to BF16 for the MMAs.  C-ABI: gpg_net_* in
// include/gpg.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/gpg.h"
#include "arena.cuh"
#include "args.cuh"
#include "common.cuh"
#include "convnet_kernels.cuh"
#include "convnet_infer.cuh"
#include "interp.cuh"
#include "optim.cuh"

using gpg::net::ConvArgs;
using gpg::net::WgradArgs;
using gpg::net::kCells;
using gpg::net::KChunks;
using gpg::net::kEdge;
using gpg::net::plane_elems;

namespace {

thread_local std::string g_net_error;

int nfail(int status, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_net_error = buf;
  return status;
}

#define NET_CUDA(call)                                                                               \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess)                                                                           \
      return nfail(e_ == cudaErrorMemoryAllocation ? GPG_ERR_OOM : GPG_ERR_CUDA, "%s: %s (%s:%d)", #call, \
                   cudaGetErrorString(e_), __FILE__, __LINE__);                                      \
  } while (0)

// layer shapes (input channels padded to 8, output channels of the last layer to 16)
constexpr int kLayers = 4;
constexpr int kCin[kLayers] = {8, 32, 32, 32};
constexpr int kCout[kLayers] = {32, 32, 32, 16};
constexpr int kRealCin0 = 3;   // density, boundary shell, interior mask
constexpr int kRealCout3 = 1;  // the potential

constexpr int64_t w_count(int l) { return int64_t(27) * kCin[l] * kCout[l]; }
constexpr int64_t param_offset_w(int l) {
  int64_t o = 0;
  for (int i = 0; i < l; ++i) o += w_count(i) + kCout[i];
  return o;
}
constexpr int64_t param_offset_b(int l) { return param_offset_w(l) + w_count(l); }
constexpr int64_t kParams = param_offset_w(kLayers);

// ---------------------------------------------------------------------------
// small kernels
// ---------------------------------------------------------------------------

// Layer-1 input planes of one patch (one CTA): the interpolated cube (the SOR's
// initial cube), its scale s = max |shell potential|, and per cell the channels
// Const*rho / s (interior), phi / s (shell), interior mask
__global__ void __launch_bounds__(256) input_kernel(const float *__restrict__ rho, const float *__restrict__ pot_in,
                                                    __nv_bfloat16 *__restrict__ x0, float *__restrict__ scale,
                                                    float cnst, float neg_zero) {
  __shared__ float cube[kCells];
  __shared__ float red[8];
  const int64_t p = blockIdx.x;
  gpg::pdl_wait();
  gpg::interpolate<float, 1, 256>(pot_in + p * gpg::Geo<1>::PN3, threadIdx.x, 4, neg_zero,
                                  [](int x, int y, int z, float v) { cube[(z * 10 + y) * 10 + x] = v; });
  __syncthreads();
  float mx = 0.f;
  for (int v = threadIdx.x; v < kCells; v += 256) {
    const int x = v % 10, y = (v / 10) % 10, z = v / 100;
    const bool shell = x == 0 || y == 0 || z == 0 || x == 9 || y == 9 || z == 9;
    if (shell) mx = fmaxf(mx, fabsf(cube[v]));
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  float s = red[0];
  for (int w = 1; w < 8; ++w) s = fmaxf(s, red[w]);
  if (!(s > 0.f)) s = 1.f;
  gpg::pdl_trigger();
  if (threadIdx.x == 0) scale[p] = s;
  for (int v = threadIdx.x; v < kCells; v += 256) {
    const int x = v % 10, y = (v / 10) % 10, z = v / 100;
    const bool shell = x == 0 || y == 0 || z == 0 || x == 9 || y == 9 || z == 9;
    __align__(16) __nv_bfloat16 o[8];
    const float r = shell ? 0.f : __fmul_rn(cnst, rho[p * 512 + ((z - 1) * 8 + (y - 1)) * 8 + (x - 1)]) / s;
    o[0] = __float2bfloat16_rn(r);
    o[1] = __float2bfloat16_rn(shell ? cube[v] / s : 0.f);
    o[2] = __float2bfloat16_rn(shell ? 0.f : 1.f);
#pragma unroll
    for (int i = 3; i < 8; ++i) o[i] = __float2bfloat16_rn(0.f);
    const int row = (y + 1) * gpg::net::kPlaneLine + x + 1;
    *reinterpret_cast<uint4 *>(x0 + gpg::net::plane_at(p, z, 0, 1) + row * 8) = *reinterpret_cast<const uint4 *>(o);
  }
}

// Second stage of the gradients: parameter i = sum of the CTAs' partial sums of
// its layer (fixed order; four threads share a parameter's partials).  Layer
// 4's output channels 1..15 have no gradient.  The loss rides along.
struct ReduceArgs {
  const float *wpart[kLayers];  // [nw][27 * cin][kept channels]
  const float *bpart[kLayers];  // [nb][32]
  int nw[kLayers], nb[kLayers];
  int first[kLayers + 1], weights[kLayers];  // a layer's first parameter, its number of weights
  const double *loss_part;
  int nloss;
  float *grad, *loss;
};

__global__ void __launch_bounds__(256) reduce_kernel(const ReduceArgs a) {
  __shared__ float sums[4][64];
  const int v = threadIdx.x & 63, q = threadIdx.x >> 6;
  constexpr int kOut4 = 16;  // output channels of layer 4, padded
  const int i = blockIdx.x * 64 + v, total = a.first[kLayers];
  gpg::pdl_wait();
  gpg::pdl_trigger();
  float s = 0.f;
  if (i < total) {
    int l = 0;
    while (l + 1 < kLayers && i >= a.first[l + 1]) ++l;
    const int k = i - a.first[l], nw = a.weights[l];
    const float *src = nullptr;
    int64_t stride = 0;
    int n = 0;
    if (k >= nw) {
      if (l < 3 || k == nw) src = a.bpart[l] + (k - nw), stride = 32, n = a.nb[l];
    } else if (l < 3) {
      src = a.wpart[l] + k, stride = nw, n = a.nw[l];
    } else if (k % kOut4 == 0) {
      src = a.wpart[3] + k / kOut4, stride = nw / kOut4, n = a.nw[3];
    }
    for (int c0 = q; c0 < n; c0 += 4 * 37) {  // 37 loads in flight (148 CTAs: all of them)
      float x[37];
#pragma unroll
      for (int c = 0; c < 37; ++c) x[c] = c0 + 4 * c < n ? src[(c0 + 4 * c) * stride] : 0.f;
#pragma unroll
      for (int c = 0; c < 37; ++c) s += x[c];
    }
  }
  sums[q][v] = s;
  __syncthreads();
  if (q == 0 && i < total) a.grad[i] = (sums[0][v] + sums[1][v]) + (sums[2][v] + sums[3][v]);
  if (blockIdx.x == 0 && a.loss && threadIdx.x < 32) {
    double t = 0.0;
    for (int c = threadIdx.x; c < a.nloss; c += 32) t += a.loss_part[c];
    t = gpg::warp_sum(t);
    if (threadIdx.x == 0) *a.loss = float(t);
  }
}

// pack W[27][cin][cout] (FP32) into BF16 operands:
//   fwd  [KCH][cout][8], k = tap*cin + c  (layer 1: two taps per MMA)
//   fwd3 [(dy, dx)][cin/8][dz, n][8]      (the others: three dz per MMA)
//   bwd3 the same for the backward-data operand, W'[tap][n][c] = W[26-tap][c][n]:
//        [(dy, dx)][cout/8][dz, c][8]
__global__ void pack_kernel(const float *__restrict__ w, int cin, int cout, int kch_f, __nv_bfloat16 *__restrict__ fwd,
                            __nv_bfloat16 *__restrict__ fwd3, __nv_bfloat16 *__restrict__ bwd3) {
  const int nf = fwd ? kch_f * cout * 8 : 0, n3 = fwd3 ? 27 * cin * cout : 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf + 2 * n3; i += gridDim.x * blockDim.x) {
    if (i < nf) {
      const int chunk = i / (cout * 8), n = (i / 8) % cout, e = i % 8;
      const int k = chunk * 8 + e, tap = k / cin, c = k % cin;
      fwd[i] = __float2bfloat16_rn(tap < 27 ? w[(tap * cin + c) * cout + n] : 0.f);
    } else {
      const bool back = i >= nf + n3;
      const int j = i - nf - (back ? n3 : 0), in = back ? cout : cin, out = back ? cin : cout;
      const int e = j % 8, row = (j / 8) % (3 * out), chunk = j / (8 * 3 * out);
      const int yx = chunk / (in / 8), ch = (chunk % (in / 8)) * 8 + e;  // input channel
      const int tap = (row / out) * 9 + yx, o = row % out;               // output channel
      const float x = back ? w[((26 - tap) * cin + o) * cout + ch] : w[(tap * cin + ch) * cout + o];
      (back ? bwd3 : fwd3)[j] = __float2bfloat16_rn(x);
    }
  }
}

// kernel attributes belong to a device's context: set once per (kernel, device)
constexpr int kMaxDevices = 64;
struct DevOnce {
  std::once_flag once[kMaxDevices];
  cudaError_t err[kMaxDevices] = {};
};

int device_index() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
  return dev;
}

template <typename F>
int set_attr_once(F *fn, size_t bytes, DevOnce &st) {
  const int dev = device_index();
  if (dev < 0) return nfail(GPG_ERR_UNSUPPORTED, "current device out of range");
  std::call_once(st.once[dev], [&] {
    cudaError_t &err = st.err[dev];
    err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
  });
  if (st.err[dev] != cudaSuccess)
    return nfail(GPG_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(st.err[dev]));
  return GPG_OK;
}

// SM count of the current device (cached per device)
int sm_count() {
  static int n[kMaxDevices] = {};
  const int dev = device_index();
  if (dev < 0) return 148;
  if (!n[dev]) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    n[dev] = v > 0 ? v : 148;
  }
  return n[dev];
}

// Planes per unit: the most (fewest halo planes loaded twice) that still leaves
// four units per SM, so that the last round of units is a small part of the
// whole; 1 for the smallest batches.
int unit_planes(int64_t npatch, int nz, int zmax) {
  for (int zc = zmax; zc > 1; --zc)
    if (nz % zc == 0 && npatch * (nz / zc) >= 4 * int64_t(sm_count())) return zc;
  return 1;
}

// persistent CTAs: one per SM
int unit_grid(int64_t npatch, int nz, int zc) {
  return (int)std::min<int64_t>(npatch * (nz / zc), sm_count());
}

int launch_conv1(ConvArgs a, cudaStream_t s) {
  static DevOnce once;
  using C = gpg::net::Conv1Cfg;
  if (int rc = set_attr_once(gpg::net::conv1_kernel, C::bytes, once)) return rc;
  a.zc = unit_planes(a.npatch, kEdge, kEdge);
  NET_CUDA(gpg::launch_after(gpg::net::conv1_kernel, (unsigned)unit_grid(a.npatch, kEdge, a.zc), C::THREADS, C::bytes, s, a));
  return GPG_OK;
}

template <int CIN, int NOUT, int EPI>
int launch_conv(ConvArgs a, cudaStream_t s, int *grid_out = nullptr) {
  static DevOnce once;
  using C = gpg::net::ConvCfg<CIN, NOUT>;
  constexpr int nz = gpg::net::PlaneEpilogue<NOUT, EPI>::NZ;
  auto fn = gpg::net::conv_kernel<CIN, NOUT, EPI>;
  if (int rc = set_attr_once(fn, C::bytes, once)) return rc;
  a.zc = unit_planes(a.npatch, nz, nz);
  const int grid = unit_grid(a.npatch, nz, a.zc);
  if (grid_out) *grid_out = grid;
  NET_CUDA(gpg::launch_after(fn, (unsigned)grid, C::THREADS, C::bytes, s, a));
  return GPG_OK;
}

template <int CIN, bool LAST>
int launch_wgrad(WgradArgs a, cudaStream_t s, int *grid_out) {
  static DevOnce once;
  using W = gpg::net::WgradCfg<CIN, LAST>;
  auto fn = gpg::net::wgrad_kernel<CIN, LAST>;
  if (int rc = set_attr_once(fn, W::bytes, once)) return rc;
  a.zc = unit_planes(a.npatch, kEdge, W::ZMAX);
  const int grid = unit_grid(a.npatch, kEdge, a.zc);
  *grid_out = grid;
  NET_CUDA(gpg::launch_after(fn, (unsigned)grid, W::THREADS, W::bytes, s, a));
  return GPG_OK;
}

}  // namespace

// ===========================================================================
// network object
// ===========================================================================
struct gpg_net {
  int device = 0;
  int max_batch = 0;
  int probe_polls = 0;  // test hook of the inference kernel (gpg_net_set_wait_probe)
  int64_t step = 0;
  void *block = nullptr;  // holds all arrays below
  float *params = nullptr, *grad = nullptr, *adam_m = nullptr, *adam_v = nullptr;
  __nv_bfloat16 *wf0 = nullptr, *wf3[kLayers] = {}, *wb3[kLayers] = {};
  // planes: input, activations (each replaced by its gradient on the way back), loss gradient
  __nv_bfloat16 *x0 = nullptr, *act[3] = {}, *g4 = nullptr;
  float *scale = nullptr, *wpart[kLayers] = {}, *bpart[kLayers] = {};
  double *loss_part = nullptr;
  int *err = nullptr;
};

namespace {


int repack(gpg_net *n, cudaStream_t s) {
  for (int l = 0; l < kLayers; ++l) {
    pack_kernel<<<64, 256, 0, s>>>(n->params + param_offset_w(l), kCin[l], kCout[l], KChunks<kCin[0]>::KCH,
                                   l == 0 ? n->wf0 : nullptr, n->wf3[l], n->wb3[l]);
  }
  NET_CUDA(cudaGetLastError());
  return GPG_OK;
}

ConvArgs conv_args(gpg_net *n, int64_t npatch) {
  ConvArgs a{};
  a.scale = n->scale;
  a.inv = 1.0 / double(npatch * 512);
  a.loss_part = n->loss_part;
  a.npatch = npatch;
  a.err = n->err;
  return a;
}

// input planes and the activations of layers 1-3
// (the training kernels launch ahead of the end of the one before: barrier and
// TMEM set-up overlap its tail; a training step of 1024 patches 615 -> 590 us, of
// 333 308 -> 263, of 32 147 -> 110)
int forward_hidden(gpg_net *n, int64_t npatch, const float *rho, const float *pot_in, float cnst, cudaStream_t s) {
  NET_CUDA(gpg::launch_after(input_kernel, (unsigned)npatch, 256, 0, s, rho, pot_in, n->x0, n->scale, cnst, -0.f));
  ConvArgs a = conv_args(n, npatch);
  for (int l = 0; l < 3; ++l) {
    a.x = l == 0 ? n->x0 : n->act[l - 1];
    a.w = l == 0 ? n->wf0 : n->wf3[l];
    a.bias = n->params + param_offset_b(l);
    a.y = n->act[l];
    if (int rc = l == 0 ? launch_conv1(a, s) : launch_conv<32, 32, gpg::net::EPI_RELU>(a, s)) return rc;
  }
  return GPG_OK;
}

// Gradients of the batch into `grad`.  Going back, the gradient with respect to
// a layer's input replaces the activation in place (its only readers are the
// ReLU mask of that very value and the weight gradient, which has run).
int gradients(gpg_net *n, int64_t npatch, const float *rho, const float *pot_in, const float *target, float cnst,
              float *grad, float *loss, cudaStream_t s) {
  if (int rc = forward_hidden(n, npatch, rho, pot_in, cnst, s)) return rc;
  ReduceArgs r{};
  for (int l = 0; l < kLayers; ++l) {
    r.first[l] = int(param_offset_w(l));
    r.weights[l] = int(w_count(l));
  }
  r.first[kLayers] = int(kParams);
  r.loss_part = n->loss_part;
  r.grad = grad;
  r.loss = loss;
  {
    ConvArgs a = conv_args(n, npatch);
    a.x = n->act[2];
    a.w = n->wf3[3];
    a.bias = n->params + param_offset_b(3);
    a.y = n->g4;
    a.target = target;
    a.bias_part = n->bpart[3];
    if (int rc = launch_conv<32, 16, gpg::net::EPI_LOSS>(a, s, &r.nb[3])) return rc;
    r.nloss = r.nb[3];
  }
  for (int l = 3; l >= 0; --l) {
    const __nv_bfloat16 *g = l == 3 ? n->g4 : n->act[l];
    WgradArgs w{l == 0 ? n->x0 : n->act[l - 1], g, n->wpart[l], npatch, 0, n->err};
    if (int rc = l == 3   ? launch_wgrad<32, true>(w, s, &r.nw[l])
                 : l == 0 ? launch_wgrad<8, false>(w, s, &r.nw[l])
                          : launch_wgrad<32, false>(w, s, &r.nw[l]))
      return rc;
    r.wpart[l] = n->wpart[l];
    r.bpart[l] = n->bpart[l];
    if (l == 0) break;
    ConvArgs a = conv_args(n, npatch);
    a.x = g;
    a.w = n->wb3[l];
    a.y = n->act[l - 1];
    a.bias_part = n->bpart[l - 1];
    if (int rc = l == 3 ? launch_conv<16, 32, gpg::net::EPI_MASK>(a, s, &r.nb[l - 1])
                        : launch_conv<32, 32, gpg::net::EPI_MASK>(a, s, &r.nb[l - 1]))
      return rc;
  }
  NET_CUDA(gpg::launch_after(reduce_kernel, (unsigned)((kParams + 63) / 64), 256, 0, s, r));
  return GPG_OK;
}

void free_net(gpg_net *n) { cudaFree(n->block); }

}  // namespace

extern "C" const char *gpg_net_last_error(void) { return g_net_error.c_str(); }

extern "C" int gpg_net_param_count(int64_t *count) {
  if (!count) return nfail(GPG_ERR_INVALID, "count is NULL");
  *count = kParams;
  return GPG_OK;
}

extern "C" int gpg_net_create(gpg_net **out, int max_batch, uint64_t seed, int device_id) {
  if (!out) return nfail(GPG_ERR_INVALID, "net is NULL");
  *out = nullptr;
  if (max_batch < 1 || max_batch > (1 << 20)) return nfail(GPG_ERR_INVALID, "max_batch %d", max_batch);
  NET_CUDA(cudaSetDevice(device_id));
  int major = 0, minor = 0;
  NET_CUDA(gpg::compute_capability(device_id, &major, &minor));
  if (major != 10) return nfail(GPG_ERR_UNSUPPORTED, "tensor-core kernels need sm_100 (found sm_%d%d)", major, minor);
  auto *n = new gpg_net;
  n->device = device_id;
  n->max_batch = max_batch;
  gpg::Arena arena;
  arena.add(n->err, 1);
  arena.add(n->params, kParams);
  arena.add(n->grad, kParams);
  arena.add(n->adam_m, kParams);
  arena.add(n->adam_v, kParams);
  // the kernels write cells only, the planes' other rows stay zero
  arena.add(n->x0, size_t(max_batch) * plane_elems(8));
  for (auto &p : n->act) arena.add(p, size_t(max_batch) * plane_elems(32));
  arena.add(n->g4, size_t(max_batch) * plane_elems(16));
  arena.zeroed_to_here();
  arena.add(n->wf0, size_t(KChunks<kCin[0]>::KCH) * kCout[0] * 8);
  for (int l = 1; l < kLayers; ++l) {
    arena.add(n->wf3[l], size_t(w_count(l)));
    arena.add(n->wb3[l], size_t(w_count(l)));
  }
  arena.add(n->scale, size_t(max_batch));
  // partial sums of the CTAs: one per SM at most, and no more than there are planes
  const size_t ctas = std::min<size_t>(size_t(max_batch) * kEdge, sm_count());
  for (int l = 0; l < kLayers; ++l) {
    arena.add(n->wpart[l], ctas * 27 * kCin[l] * (l == 3 ? 1 : 32));
    arena.add(n->bpart[l], ctas * 32);
  }
  arena.add(n->loss_part, ctas);
  cudaError_t e = arena.allocate(&n->block);
  if (e != cudaSuccess) {
    free_net(n);
    delete n;
    return nfail(e == cudaErrorMemoryAllocation ? GPG_ERR_OOM : GPG_ERR_CUDA, "allocation: %s",
                 cudaGetErrorString(e));
  }
  // He-normal initialisation of the real weights (fixed seed); padded input
  // channels of layer 1 and output channels 1..15 of layer 4 stay zero
  std::vector<float> h(kParams, 0.f);
  uint64_t st = seed * 6364136223846793005ull + 1442695040888963407ull;
  auto uni = [&]() {
    st = st * 6364136223846793005ull + 1442695040888963407ull;
    return ((st >> 11) + 0.5) * (1.0 / 9007199254740992.0);
  };
  for (int l = 0; l < kLayers; ++l) {
    const int cin_real = l == 0 ? kRealCin0 : kCin[l];
    const int cout_real = l == 3 ? kRealCout3 : kCout[l];
    const double sd = std::sqrt(2.0 / (27.0 * cin_real)) * (l == 3 ? 0.1 : 1.0);
    for (int t = 0; t < 27; ++t)
      for (int c = 0; c < cin_real; ++c)
        for (int o = 0; o < cout_real; ++o) {
          const double z = std::sqrt(-2.0 * std::log(uni())) * std::cos(6.283185307179586 * uni());
          h[param_offset_w(l) + (int64_t(t) * kCin[l] + c) * kCout[l] + o] = float(sd * z);
        }
  }
  e = cudaMemcpy(n->params, h.data(), kParams * 4, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    free_net(n);
    delete n;
    return nfail(GPG_ERR_CUDA, "upload: %s", cudaGetErrorString(e));
  }
  int rc = repack(n, 0);
  // the fills and the packing run on the default stream, which other streams need not follow
  if (!rc && cudaStreamSynchronize(nullptr) != cudaSuccess)
    rc = nfail(GPG_ERR_CUDA, "set-up: %s", cudaGetErrorString(cudaGetLastError()));
  if (rc) {
    free_net(n);
    delete n;
    return rc;
  }
  *out = n;
  return GPG_OK;
}

extern "C" int gpg_net_destroy(gpg_net *n) {
  if (!n) return GPG_OK;
  cudaSetDevice(n->device);
  cudaDeviceSynchronize();
  free_net(n);
  delete n;
  return GPG_OK;
}

extern "C" int gpg_net_get_params(gpg_net *n, float *host) {
  if (!n || !host) return nfail(GPG_ERR_INVALID, "NULL argument");
  NET_CUDA(cudaSetDevice(n->device));
  NET_CUDA(cudaDeviceSynchronize());  // training steps on any stream
  NET_CUDA(cudaMemcpy(host, n->params, kParams * 4, cudaMemcpyDeviceToHost));
  return GPG_OK;
}

extern "C" int gpg_net_set_params(gpg_net *n, const float *host) {
  if (!n || !host) return nfail(GPG_ERR_INVALID, "NULL argument");
  NET_CUDA(cudaSetDevice(n->device));
  // calls before and after may be on streams that the default stream does not order
  NET_CUDA(cudaDeviceSynchronize());
  NET_CUDA(cudaMemcpy(n->params, host, kParams * 4, cudaMemcpyHostToDevice));
  NET_CUDA(cudaMemset(n->adam_m, 0, kParams * 4));
  NET_CUDA(cudaMemset(n->adam_v, 0, kParams * 4));
  n->step = 0;
  if (int rc = repack(n, 0)) return rc;
  NET_CUDA(cudaStreamSynchronize(nullptr));
  return GPG_OK;
}

extern "C" int gpg_net_check(gpg_net *n) {
  if (!n) return nfail(GPG_ERR_INVALID, "net is NULL");
  NET_CUDA(cudaSetDevice(n->device));
  int flag = 0;
  NET_CUDA(cudaMemcpy(&flag, n->err, 4, cudaMemcpyDeviceToHost));
  if (flag) {
    NET_CUDA(cudaMemset(n->err, 0, 4));  // reported once
    return nfail(GPG_ERR_CUDA, "a tensor-core wait timed out");
  }
  return GPG_OK;
}

extern "C" int gpg_net_set_wait_probe(gpg_net *n, int polls) {
  if (!n) return nfail(GPG_ERR_INVALID, "net is NULL");
  if (polls < 0) return nfail(GPG_ERR_INVALID, "polls %d", polls);
  n->probe_polls = polls;
  return GPG_OK;
}

extern "C" int gpg_net_predict(gpg_net *n, int npatch, const float *d_rho, const float *d_pot_in, float *d_guess,
                               double cnst, void *stream) {
  if (!n) return nfail(GPG_ERR_INVALID, "net is NULL");
  if (npatch < 0) return nfail(GPG_ERR_INVALID, "npatch %d", npatch);
  if (npatch && (!d_rho || !d_pot_in || !d_guess)) return nfail(GPG_ERR_INVALID, "NULL array");
  if (!npatch) return GPG_OK;
  NET_CUDA(cudaSetDevice(n->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  static DevOnce once;
  using gpg::net::InferSmem;
  if (int rc = set_attr_once(gpg::net::net_infer_kernel, InferSmem::bytes, once)) return rc;
  gpg::net::InferArgs a{};
  a.rho = d_rho;
  a.pot_in = d_pot_in;
  a.guess = d_guess;
  for (int l = 0; l < kLayers; ++l) {
    a.w[l] = l == 0 ? n->wf0 : n->wf3[l];
    a.bias[l] = n->params + param_offset_b(l);
  }
  a.cnst = float(cnst);
  a.neg_zero = -0.f;
  a.npatch = npatch;
  a.probe_polls = n->probe_polls;
  a.err = n->err;
  const int grid = std::min(npatch, sm_count());  // persistent: one CTA per SM (shared memory bound)
  gpg::net::net_infer_kernel<<<grid, gpg::net::kInferThreads, InferSmem::bytes, s>>>(a);
  NET_CUDA(cudaGetLastError());
  return GPG_OK;
}

extern "C" int gpg_net_predict_layers(gpg_net *n, int npatch, const float *d_rho, const float *d_pot_in,
                                      float *d_guess, double cnst, void *stream) {
  if (!n) return nfail(GPG_ERR_INVALID, "net is NULL");
  if (npatch < 0) return nfail(GPG_ERR_INVALID, "npatch %d", npatch);
  if (npatch && (!d_rho || !d_pot_in || !d_guess)) return nfail(GPG_ERR_INVALID, "NULL array");
  NET_CUDA(cudaSetDevice(n->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int64_t p0 = 0; p0 < npatch; p0 += n->max_batch) {
    const int64_t b = std::min<int64_t>(n->max_batch, npatch - p0);
    if (int rc = forward_hidden(n, b, d_rho + p0 * 512, d_pot_in + p0 * 512, float(cnst), s)) return rc;
    ConvArgs a = conv_args(n, b);
    a.x = n->act[2];
    a.w = n->wf3[3];
    a.bias = n->params + param_offset_b(3);
    a.guess = d_guess + p0 * 512;
    if (int rc = launch_conv<32, 16, gpg::net::EPI_GUESS>(a, s)) return rc;
  }
  return GPG_OK;
}

extern "C" int gpg_net_gradients(gpg_net *n, int npatch, const float *d_rho, const float *d_pot_in,
                                 const float *d_target, double cnst, float *d_grad, float *d_loss, void *stream) {
  if (!n) return nfail(GPG_ERR_INVALID, "net is NULL");
  if (npatch < 1 || npatch > n->max_batch) return nfail(GPG_ERR_INVALID, "npatch %d (1..%d)", npatch, n->max_batch);
  if (!d_rho || !d_pot_in || !d_target) return nfail(GPG_ERR_INVALID, "NULL array");
  NET_CUDA(cudaSetDevice(n->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return gradients(n, npatch, d_rho, d_pot_in, d_target, float(cnst), d_grad ? d_grad : n->grad, d_loss, s);
}

namespace {
// one Adam step (beta 0.9 / 0.999, eps 1e-8) with gradient `grad`, then the
// BF16 operands are repacked from the updated FP32 masters
int adam_step(gpg_net *n, const float *grad, float lr, cudaStream_t s) {
  n->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, float(n->step)), c2 = 1.f - std::pow(b2, float(n->step));
  gpg::adam_kernel<<<128, 256, 0, s>>>(
      gpg::AdamArgs{n->params, n->adam_m, n->adam_v, grad, lr, b1, b2, 1e-8f, c1, c2}, kParams);
  NET_CUDA(cudaGetLastError());
  return repack(n, s);
}
}  // namespace

extern "C" int gpg_net_train_step(gpg_net *n, int npatch, const float *d_rho, const float *d_pot_in,
                                  const float *d_target, double cnst, float lr, float *d_loss, void *stream) {
  if (int rc = gpg_net_gradients(n, npatch, d_rho, d_pot_in, d_target, cnst, nullptr, d_loss, stream)) return rc;
  return adam_step(n, n->grad, lr, static_cast<cudaStream_t>(stream));
}

extern "C" int gpg_net_apply_gradient(gpg_net *n, const float *d_grad, float lr, void *stream) {
  if (!n || !d_grad) return nfail(GPG_ERR_INVALID, "NULL argument");
  NET_CUDA(cudaSetDevice(n->device));
  return adam_step(n, d_grad, lr, static_cast<cudaStream_t>(stream));
}
