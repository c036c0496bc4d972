// gpg_api.cu -- C-ABI of libgpg (include/gpg.h): parameter handling, kernel
// dispatch, and the reference-shaped context API (device buffers, pinned host
// buffers, streams) that replaces GPU_API/CUAPI_*.cu.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <limits>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/gpg.h"
#include "args.cuh"
#include "batch_kernel.cuh"
#include "gravity.cuh"
#include "mg_kernel.cuh"
#include "sor_kernel.cuh"

namespace {

thread_local std::string g_last_error;

int fail(int status, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return status;
}

#define GPG_CUDA(call)                                                                      \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess)                                                                  \
      return fail(e_ == cudaErrorMemoryAllocation ? GPG_ERR_OOM : GPG_ERR_CUDA, "%s: %s (%s:%d)", \
                  #call, cudaGetErrorString(e_), __FILE__, __LINE__);                       \
  } while (0)

// ---------------------------------------------------------------------------
// launch configuration per (precision, ghost size)
// ---------------------------------------------------------------------------
// Kernel attributes, set once per (kernel instantiation, device) -- they
// belong to a device's context -- by the first call on that device (the
// caller owns the state): the dynamic shared memory size and the max-shared
// carveout (the reference's cudaFuncCachePreferShared,
// CUAPI_Set_Diagnose_Device.cu:274-285).
constexpr int kMaxDevices = 64;
struct AttrOnce {
  std::once_flag once[kMaxDevices];
  cudaError_t err[kMaxDevices] = {};
  int max_threads[kMaxDevices] = {};  // per block, given the kernel's registers
};

int current_device(int *dev) {
  GPG_CUDA(cudaGetDevice(dev));
  if (*dev < 0 || *dev >= kMaxDevices) return fail(GPG_ERR_UNSUPPORTED, "device %d (max %d)", *dev, kMaxDevices);
  return GPG_OK;
}

template <typename KernelFn>
int ensure_smem(KernelFn *fn, size_t bytes, AttrOnce &st, int *max_threads = nullptr) {
  int dev = 0;
  if (int rc = current_device(&dev)) return rc;
  std::call_once(st.once[dev], [&] {
    cudaError_t &err = st.err[dev];
    err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    cudaFuncAttributes fa;
    if (err == cudaSuccess) err = cudaFuncGetAttributes(&fa, fn);
    if (err == cudaSuccess) st.max_threads[dev] = fa.maxThreadsPerBlock;
  });
  if (st.err[dev] != cudaSuccess)
    return fail(GPG_ERR_CUDA, "cudaFuncSetAttribute(%zu bytes): %s", bytes, cudaGetErrorString(st.err[dev]));
  if (max_threads) *max_threads = st.max_threads[dev];
  return GPG_OK;
}

// SOR kernel variants: (teams per CTA, phased pass).  The table below holds
// the variant per (precision, ghost size); defaults are the fastest measured
// on B200, gpg_set_sor_variant / a tuning file override them.
// Variants 14-16: the layouts of 10, 11 and 13 in the staged persistent
// kernel (patches per CTA reported as 0: teams per CTA chosen per shape).
constexpr int kSorVariants = 17;
constexpr int kSorVariantPPC[kSorVariants] = {1, 1, 2, 2, 4, 4, 1, 1, 2, 2, 1, 1, 1, 1, 0, 0, 0};
constexpr bool kSorVariantPhased[kSorVariants] = {false, true, false, true, false, true, false, true,  false,
                                                  true,  false, true, false, true, false, true, true};
constexpr int kSorVariantSplit[kSorVariants] = {1, 1, 1, 1, 1, 1, 2, 2, 2, 2, 2, 2, 1, 1, 2, 2, 1};  // lanes per column
constexpr int kSorVariantRows[kSorVariants] = {1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 2, 2, 2, 2, 2, 2, 2};   // rows per lane
constexpr bool kSorVariantStaged[kSorVariants] = {false, false, false, false, false, false, false, false, false,
                                                  false, false, false, false, false, true,  true,  true};
constexpr int kSorDefault[2][6] = {
    // ghost:  -  1  2  3  4  5       (autotune.py on B200, 4096 patches, reference parameters;
    //   FP32 ghost 4: the whole column 138 us per launch, the split one 152; FP64 ghost 1
    //   height by height 105.4 us, phased 106.3, ghost 3 530 and 533, with gravity 548 and 554)
    {0, 11, 10, 10, 13, 11},   // float
    {0, 10, 13, 10, 10, 14},   // double
};
// atomic: gpg_set_sor_variant may run on one host thread while another launches
std::atomic<int> g_sor_variant[2][6] = {
    {kSorDefault[0][0], kSorDefault[0][1], kSorDefault[0][2], kSorDefault[0][3], kSorDefault[0][4], kSorDefault[0][5]},
    {kSorDefault[1][0], kSorDefault[1][1], kSorDefault[1][2], kSorDefault[1][3], kSorDefault[1][4], kSorDefault[1][5]},
};
// set once a variant was chosen explicitly (gpg_set_sor_variant or the tuning
// file): every launch then uses it, whatever its size
std::atomic<bool> g_sor_pinned[2][6] = {};
// Small launches: at a few thousand patches and fewer a launch leaves SMs short of
// teams, and other layouts finish each patch sooner: those that split each pair
// column between two lanes (twice the threads per patch), with one row per lane
// instead of two twice as many again; at FP64 ghost 4 the staged kernel, whose teams
// are as large but prefetch their inputs.  Each launch of up to max_npatch patches
// runs the variant below.  Both sides, us per launch with gravity (autotune.py
// --sizes, reference parameters; the variant below, then the one above the limit):
//   FP32 1: 256 patches 10.2 / 14.1, 1480 19.8 / 21.4, 2048 27.6 / 28.0, 2368 30.8 / 30.3
//        2: 256 10.2 / 13.2, 512 14.7 / 16.2, 740 17.0 / 18.7, 888 19.1 / 18.9
//        3: 256 15.6 / 16.1, 444 19.3 / 20.0, 512 20.9 / 19.9
//        4: v6, v11: 148 15.0 / 17.8, 200 20.1 / 20.0; v11, v13: 444 23.7 / 26.4, 740
//           32.8 / 34.6, 888 44.4 / 36.3, 1024 46.7 / 45.8
//        5: the large-launch layout at every size
//   FP64 1: 256 30.3 / 33.1, 370 33.6 / 33.7; 2: 256 37.2 / 50.6, 444 45.1 / 52.5
//        4: the staged kernel while each of its teams, two per SM, has one patch: 64
//           57.4 / 67.1, 148 59.0 / 68.6, 296 81.6 / 86.1; 310 124.5 / 108.7
//        5: 1024 337 / 348, 1184 384 / 353, but 888 292 / 266: the staged kernel hands
//           patches out at a fixed stride, and 1024 patches over its 296 teams leave some
//           teams a fourth patch, the size of the CUAPI path's four streams of 4096
//           patches; below it the unstaged v11 costs 2 to 9 %
// (512 at FP32 3 and 1024 at 4 were the crossings before the launches overlapped as
// they do now; 148 and 296 are one and two patches per SM.)
struct SorSmall {
  int max_npatch, variant;
};
constexpr SorSmall kSorSmall[2][6][2] = {
    // ghost 0 (none), 1, 2, 3, 4, 5; the smaller limit first, 0 none
    {{}, {{2048, 7}}, {{512, 6}}, {{512, 7}}, {{148, 6}, {1024, 11}}, {}},  // float
    {{}, {{256, 8}}, {{256, 7}}, {}, {{296, 14}}, {{1024, 11}}},            // double
};
std::once_flag g_tune_once;

void load_tune_file() {
  // optional text file, one "f32|f64 <ghost> <variant>" per line:
  // $GPG_TUNE_FILE, else sor_tune.txt beside libgpg.so (written by autotune.py)
  const char *path = std::getenv("GPG_TUNE_FILE");
  std::string p;
  if (path) {
    p = path;
  } else {
    Dl_info info;
    if (dladdr((void *)&load_tune_file, &info) && info.dli_fname) {
      p = info.dli_fname;
      p = p.substr(0, p.find_last_of('/') + 1) + "sor_tune.txt";
    }
  }
  if (p.empty()) return;
  FILE *f = std::fopen(p.c_str(), "r");
  if (!f) return;
  char prec[8];
  int g, v;
  while (std::fscanf(f, "%7s %d %d", prec, &g, &v) == 3) {
    const int t = std::strcmp(prec, "f64") == 0 ? 1 : (std::strcmp(prec, "f32") == 0 ? 0 : -1);
    if (t >= 0 && g >= 1 && g <= 5 && v >= 0 && v < kSorVariants) {
      g_sor_variant[t][g].store(v, std::memory_order_relaxed);
      g_sor_pinned[t][g].store(true, std::memory_order_relaxed);
    }
  }
  std::fclose(f);
}

template <typename T, int G, int PPC, bool PHASED, int Z, int Y>
AttrOnce &sor_attr() {
  static AttrOnce attr;
  return attr;
}

template <typename T, int G, int PPC, bool PHASED, int Z, int Y>
int launch_sor_v(const gpg::SolveArgs<T> &a, cudaStream_t s) {
  if constexpr (!gpg::SorCfg<T, G, Z, Y>::FITS) {
    return fail(GPG_ERR_UNSUPPORTED, "SOR variant holds more state per lane than registers allow");
  } else {
    using S = gpg::SorSmem<T, G, Z, Y>;
    constexpr int threads = PPC * gpg::SorCfg<T, G, Z, Y>::TEAM;
    const size_t smem = PPC * S::team_bytes;
    if (smem > 227 * 1024) return fail(GPG_ERR_UNSUPPORTED, "SOR variant needs %zu bytes of shared memory", smem);
    auto fn = gpg::sor_kernel<T, G, PPC, PHASED, Z, Y>;
    AttrOnce &attr = sor_attr<T, G, PPC, PHASED, Z, Y>();
    int max_threads = 0;
    if (int rc = ensure_smem(fn, smem, attr, &max_threads)) return rc;
    if (threads > max_threads)
      return fail(GPG_ERR_UNSUPPORTED, "SOR variant needs %d threads per CTA (registers allow %d)", threads,
                  max_threads);
    const int64_t grid = (a.npatch + PPC - 1) / PPC;
    GPG_CUDA(gpg::launch_after(fn, (unsigned)grid, threads, smem, s, a));
    return GPG_OK;
  }
}

// Kernel attributes of the SOR variant a (precision, ghost) solve will launch,
// set without launching (stream capture must not see first-use set-up).
template <typename T, int G, int PPC, bool PHASED, int Z, int Y>
int prepare_sor_v() {
  if constexpr (!gpg::SorCfg<T, G, Z, Y>::FITS) {
    return fail(GPG_ERR_UNSUPPORTED, "SOR variant holds more state per lane than registers allow");
  } else {
    auto fn = gpg::sor_kernel<T, G, PPC, PHASED, Z, Y>;
    static AttrOnce &attr = sor_attr<T, G, PPC, PHASED, Z, Y>();
    return ensure_smem(fn, PPC * gpg::SorSmem<T, G, Z, Y>::team_bytes, attr);
  }
}

// Staged persistent kernel: CTAs of about 128 threads, as many as fit on the
// device (per-device occupancy), at most one team per patch.  Inputs that are
// not 16-byte aligned (bulk copies need it) run the same layout unstaged.
template <typename T, int G, bool PHASED, int Z, int Y>
int launch_staged_v(const gpg::SolveArgs<T> &a, cudaStream_t s) {
  if constexpr (!gpg::SorCfg<T, G, Z, Y>::FITS) {
    return fail(GPG_ERR_UNSUPPORTED, "SOR variant holds more state per lane than registers allow");
  } else {
    constexpr int TEAM = gpg::SorCfg<T, G, Z, Y>::TEAM;
    constexpr int TPC = TEAM >= 128 ? 1 : 128 / TEAM;
    using SS = gpg::StagedSmem<T, G, Z, Y, TPC>;
    if ((reinterpret_cast<uintptr_t>(a.rho) | reinterpret_cast<uintptr_t>(a.pot_in)) & 15)
      return launch_sor_v<T, G, 1, PHASED, Z, Y>(a, s);
    if (SS::bytes > 227 * 1024) return fail(GPG_ERR_UNSUPPORTED, "staged SOR needs %zu bytes of shared memory", SS::bytes);
    auto fn = gpg::staged_sor_kernel<T, G, PHASED, Z, Y, TPC>;
    static AttrOnce attr;
    int max_threads = 0;
    if (int rc = ensure_smem(fn, SS::bytes, attr, &max_threads)) return rc;
    if (TPC * TEAM > max_threads)
      return fail(GPG_ERR_UNSUPPORTED, "staged SOR needs %d threads per CTA (registers allow %d)", TPC * TEAM,
                  max_threads);
    static int resident[kMaxDevices] = {};  // CTAs per device
    int dev = 0;
    if (int rc = current_device(&dev)) return rc;
    if (!resident[dev]) {
      int sms = 0, per = 0;
      GPG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      GPG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, TPC * TEAM, SS::bytes));
      if (per < 1) return fail(GPG_ERR_UNSUPPORTED, "staged SOR does not fit on an SM");
      resident[dev] = sms * per;
    }
    const int64_t need = (a.npatch + TPC - 1) / TPC;
    const int64_t grid = std::min<int64_t>(need, resident[dev]);
    GPG_CUDA(gpg::launch_after(fn, (unsigned)grid, TPC * TEAM, SS::bytes, s, a));
    return GPG_OK;
  }
}

template <typename T, int G, bool PHASED, int Z, int Y>
int prepare_staged_v() {
  if constexpr (!gpg::SorCfg<T, G, Z, Y>::FITS) {
    return fail(GPG_ERR_UNSUPPORTED, "SOR variant holds more state per lane than registers allow");
  } else {
    constexpr int TEAM = gpg::SorCfg<T, G, Z, Y>::TEAM;
    constexpr int TPC = TEAM >= 128 ? 1 : 128 / TEAM;
    using SS = gpg::StagedSmem<T, G, Z, Y, TPC>;
    if (SS::bytes > 227 * 1024) return fail(GPG_ERR_UNSUPPORTED, "staged SOR needs %zu bytes of shared memory", SS::bytes);
    static AttrOnce attr;
    if (int rc = ensure_smem(gpg::staged_sor_kernel<T, G, PHASED, Z, Y, TPC>, SS::bytes, attr)) return rc;
    return prepare_sor_v<T, G, 1, PHASED, Z, Y>();  // the unstaged fallback
  }
}

// Set on the host thread that prepares and captures a concurrent batch plan:
// its branches share the SMs, and a staged persistent kernel, whose CTAs take
// patches at a fixed stride, then finishes with a tail (65,536 mixed patches:
// 1.43 vs 1.34 ms per graph launch), so staged variants run as their unstaged
// layouts there.
thread_local bool t_shared_sms = false;
struct SharedSms {
  SharedSms() { t_shared_sms = true; }
  ~SharedSms() { t_shared_sms = false; }
};

// the variant a launch of npatch patches runs
inline int sor_variant_for(bool f64, int g, int64_t npatch) {
  int v = g_sor_variant[f64][g].load(std::memory_order_relaxed);
  if (!g_sor_pinned[f64][g].load(std::memory_order_relaxed)) {
    for (const SorSmall &sm : kSorSmall[f64][g])
      if (npatch <= sm.max_npatch) {
        v = sm.variant;
        break;
      }
  }
  if (t_shared_sms && kSorVariantStaged[v]) v = v == 14 ? 10 : (v == 15 ? 11 : 13);  // same layout, unstaged
  return v;
}

template <typename T, int G>
int launch_sor_variant(int variant, const gpg::SolveArgs<T> &a, cudaStream_t s) {
  switch (variant) {
    case 0: return launch_sor_v<T, G, 1, false, 1, 1>(a, s);
    case 1: return launch_sor_v<T, G, 1, true, 1, 1>(a, s);
    case 2: return launch_sor_v<T, G, 2, false, 1, 1>(a, s);
    case 3: return launch_sor_v<T, G, 2, true, 1, 1>(a, s);
    case 4: return launch_sor_v<T, G, 4, false, 1, 1>(a, s);
    case 5: return launch_sor_v<T, G, 4, true, 1, 1>(a, s);
    case 6: return launch_sor_v<T, G, 1, false, 2, 1>(a, s);
    case 7: return launch_sor_v<T, G, 1, true, 2, 1>(a, s);
    case 8: return launch_sor_v<T, G, 2, false, 2, 1>(a, s);
    case 9: return launch_sor_v<T, G, 2, true, 2, 1>(a, s);
    case 10: return launch_sor_v<T, G, 1, false, 2, 2>(a, s);
    case 11: return launch_sor_v<T, G, 1, true, 2, 2>(a, s);
    case 12: return launch_sor_v<T, G, 1, false, 1, 2>(a, s);
    case 13: return launch_sor_v<T, G, 1, true, 1, 2>(a, s);
    case 14: return launch_staged_v<T, G, false, 2, 2>(a, s);
    case 15: return launch_staged_v<T, G, true, 2, 2>(a, s);
    default: return launch_staged_v<T, G, true, 1, 2>(a, s);
  }
}

template <typename T, int G>
int launch_sor(const gpg::SolveArgs<T> &a, cudaStream_t s) {
  std::call_once(g_tune_once, load_tune_file);
  return launch_sor_variant<T, G>(sor_variant_for(sizeof(T) == 8, G, a.npatch), a, s);
}

template <typename T, int G>
int prepare_sor_variant(int variant) {
  switch (variant) {
    case 0: return prepare_sor_v<T, G, 1, false, 1, 1>();
    case 1: return prepare_sor_v<T, G, 1, true, 1, 1>();
    case 2: return prepare_sor_v<T, G, 2, false, 1, 1>();
    case 3: return prepare_sor_v<T, G, 2, true, 1, 1>();
    case 4: return prepare_sor_v<T, G, 4, false, 1, 1>();
    case 5: return prepare_sor_v<T, G, 4, true, 1, 1>();
    case 6: return prepare_sor_v<T, G, 1, false, 2, 1>();
    case 7: return prepare_sor_v<T, G, 1, true, 2, 1>();
    case 8: return prepare_sor_v<T, G, 2, false, 2, 1>();
    case 9: return prepare_sor_v<T, G, 2, true, 2, 1>();
    case 10: return prepare_sor_v<T, G, 1, false, 2, 2>();
    case 11: return prepare_sor_v<T, G, 1, true, 2, 2>();
    case 12: return prepare_sor_v<T, G, 1, false, 1, 2>();
    case 13: return prepare_sor_v<T, G, 1, true, 1, 2>();
    case 14: return prepare_staged_v<T, G, false, 2, 2>();
    case 15: return prepare_staged_v<T, G, true, 2, 2>();
    default: return prepare_staged_v<T, G, true, 1, 2>();
  }
}

// attributes of both variants a launch may pick (large and small batches)
template <typename T, int G>
int prepare_sor() {
  std::call_once(g_tune_once, load_tune_file);
  constexpr bool f64 = sizeof(T) == 8;
  if (int rc = prepare_sor_variant<T, G>(sor_variant_for(f64, G, std::numeric_limits<int64_t>::max()))) return rc;
  for (const SorSmall &sm : kSorSmall[f64][G])
    if (sm.max_npatch > 0)
      if (int rc = prepare_sor_variant<T, G>(sor_variant_for(f64, G, sm.max_npatch))) return rc;
  return GPG_OK;
}

template <typename T>
int prepare_sor_typed(int ghost) {
  switch (ghost) {
    case 1: return prepare_sor<T, 1>();
    case 2: return prepare_sor<T, 2>();
    case 3: return prepare_sor<T, 3>();
    case 4: return prepare_sor<T, 4>();
    default: return prepare_sor<T, 5>();
  }
}

// Attributes of the SOR kernel a solve with `q` launches (stream capture must
// not be the first use of a kernel).
int prepare_solve_kernels(const gpg_params &q) {
  return q.real_size == 4 ? prepare_sor_typed<float>(q.ghost) : prepare_sor_typed<double>(q.ghost);
}

// Launches of up to this many patches run the wide multigrid kernel: with one or
// two CTAs per SM the time is one patch's latency, which the helping threads
// shorten.  us per launch, as wide as level 0 / wide: 64 patches FP32 ghost 1 17.1 /
// 12.9, 2 14.8 / 12.8, 3 16.7 / 14.8, 5 29.2 / 21.3, FP64 ghost 1 60.0 / 53.8, 5 191 /
// 167; 296 patches FP32 17.0 / 13.1, 15.1 / 14.8, 17.2 / 16.8, 31.4 / 26.9, FP64 ghost
// 1 62.2 / 55.9, 5 217 / 334 (148: 193 / 169).  Elsewhere the wide form gains
// nothing (FP32 ghost 4) or spills (FP64 ghost 3 89 / 117 at 64 patches, 4 126 / 154).
template <typename T, int G>
constexpr int kMgWide = sizeof(T) == 4 ? (G == 4 ? 0 : 296) : (G == 1 ? 296 : (G == 5 ? 148 : 0));

template <typename T, int G, bool WIDE>
int prepare_mg() {
  static AttrOnce attr;
  return ensure_smem(gpg::mg_kernel<T, G, WIDE>, gpg::MgCfg<T, G, WIDE>::bytes, attr);
}

template <typename T, int G, bool WIDE>
int run_mg(const gpg::SolveArgs<T> &a, cudaStream_t s) {
  using K = gpg::MgCfg<T, G, WIDE>;
  GPG_CUDA(gpg::launch_after(gpg::mg_kernel<T, G, WIDE>, (unsigned)a.npatch, K::TEAM, K::bytes, s, a));
  return GPG_OK;
}

template <typename T, int G>
int launch_mg(const gpg::SolveArgs<T> &a, cudaStream_t s) {
  if (int rc = prepare_mg<T, G, false>()) return rc;
  if constexpr (kMgWide<T, G> > 0) {
    if (int rc = prepare_mg<T, G, true>()) return rc;
    if (a.npatch <= kMgWide<T, G>) return run_mg<T, G, true>(a, s);
  }
  return run_mg<T, G, false>(a, s);
}

template <typename T, int GG>
int launch_gravity(const gpg::SolveArgs<T> &a, cudaStream_t s) {
  gpg::gravity_kernel<T, GG><<<(unsigned)a.npatch, 256, 0, s>>>(a.flu, a.pot_out, a.npatch, a.gra_const, a.p5);
  GPG_CUDA(cudaGetLastError());
  return GPG_OK;
}


template <typename T>
int solve_typed(const gpg_params &p, int64_t npatch, const void *rho, const void *pin, void *pout, void *flu,
                const void *guess, int32_t *iters, double *resid, cudaStream_t s) {
  auto a = gpg::make_args<T>(p, npatch, rho, pin, pout, flu, guess, iters, resid);
  if (p.poisson) {
    // the fused kernel applies gravity itself when gra_acc is set
    if (p.scheme == GPG_SOR) {
      switch (p.ghost) {
        case 1: return launch_sor<T, 1>(a, s);
        case 2: return launch_sor<T, 2>(a, s);
        case 3: return launch_sor<T, 3>(a, s);
        case 4: return launch_sor<T, 4>(a, s);
        case 5: return launch_sor<T, 5>(a, s);
      }
    } else {
      switch (p.ghost) {
        case 1: return launch_mg<T, 1>(a, s);
        case 2: return launch_mg<T, 2>(a, s);
        case 3: return launch_mg<T, 3>(a, s);
        case 4: return launch_mg<T, 4>(a, s);
        case 5: return launch_mg<T, 5>(a, s);
      }
    }
    return fail(GPG_ERR_INVALID, "ghost %d", p.ghost);
  }
  if (p.gra_acc) {
    switch (p.gra_ghost) {
      case 1: return launch_gravity<T, 1>(a, s);
      case 2: return launch_gravity<T, 2>(a, s);
    }
  }
  return GPG_OK;
}

int check_ptr(const void *ptr, const char *name) {
  if (ptr == nullptr) return fail(GPG_ERR_INVALID, "%s is NULL", name);
  return GPG_OK;
}

}  // namespace

// ===========================================================================
// parameters
// ===========================================================================
extern "C" int gpg_abi_version(void) { return GPG_ABI_VERSION; }

extern "C" const char *gpg_last_error(void) { return g_last_error.c_str(); }

extern "C" int gpg_default_params(gpg_params *p, int real_size, int ghost, int scheme) {
  if (!p) return fail(GPG_ERR_INVALID, "params is NULL");
  if (real_size != 4 && real_size != 8) return fail(GPG_ERR_INVALID, "real_size %d (must be 4 or 8)", real_size);
  if (ghost < 1 || ghost > 5) return fail(GPG_ERR_INVALID, "ghost %d (must be 1..5)", ghost);
  if (scheme != GPG_SOR && scheme != GPG_MG) return fail(GPG_ERR_INVALID, "scheme %d", scheme);
  static const double omega[5] = {1.49, 1.57, 1.62, 1.65, 1.69};  // Main.cpp:1145
  std::memset(p, 0, sizeof *p);
  p->real_size = real_size;
  p->ghost = ghost;
  p->gra_ghost = 1;
  p->scheme = scheme;
  p->int_scheme = GPG_INT_CQUAD;
  p->p5_gradient = 0;
  p->poisson = 1;
  p->gra_acc = 1;
  p->dt = 1.0e-2;
  p->dh = 1.0;
  p->sor_min_iter = 10;
  p->sor_max_iter = real_size == 4 ? 60 : 100;
  p->sor_omega = omega[ghost - 1];
  p->mg_max_iter = real_size == 4 ? 10 : 20;
  p->mg_npre_smooth = 3;
  p->mg_npost_smooth = 3;
  p->init_mode = GPG_INIT_INTERP;
  p->mg_tolerated_error = real_size == 4 ? 1.0e-6 : 1.0e-15;
  p->poi_coeff = 4.0 * M_PI * 1.0e-5;
  p->stop_mode = GPG_STOP_REFERENCE;
  p->sor_tolerance = 0.0;
  return GPG_OK;
}

extern "C" int gpg_pot_tolerance(int real_size, int ghost, double *tol) {
  // oracle/calibrate_tol.py: 1024 seeded power-law patches per entry
  static const double kTol[2][5] = {{9.8e-7, 1.1e-6, 1.2e-6, 1.3e-6, 1.4e-6},
                                    {1.8e-15, 2.1e-15, 2.3e-15, 2.4e-15, 2.5e-15}};
  if ((real_size != 4 && real_size != 8) || ghost < 1 || ghost > 5 || !tol)
    return fail(GPG_ERR_INVALID, "real_size %d ghost %d", real_size, ghost);
  *tol = kTol[real_size == 8][ghost - 1];
  return GPG_OK;
}

extern "C" int gpg_validate_params(const gpg_params *p) {
  if (!p) return fail(GPG_ERR_INVALID, "params is NULL");
  if (p->real_size != 4 && p->real_size != 8) return fail(GPG_ERR_INVALID, "real_size %d", p->real_size);
  if (p->ghost < 1 || p->ghost > 5) return fail(GPG_ERR_INVALID, "ghost %d (must be 1..5)", p->ghost);
  if (p->gra_ghost < 0 || p->gra_ghost > 2 || p->gra_ghost > p->ghost)
    return fail(GPG_ERR_INVALID, "gra_ghost %d (must be 0..2 and <= ghost %d)", p->gra_ghost, p->ghost);
  if (p->poisson) {
    if (p->scheme != GPG_SOR && p->scheme != GPG_MG) return fail(GPG_ERR_INVALID, "scheme %d", p->scheme);
    // CUAPI_Asyn_PoissonGravitySolver.cu:134-135
    if (p->int_scheme != GPG_INT_CQUAD && p->int_scheme != GPG_INT_QUAD)
      return fail(GPG_ERR_INVALID, "incorrect parameter IntScheme = %d", p->int_scheme);
    if (p->scheme == GPG_SOR) {
      if (p->sor_max_iter < 0) return fail(GPG_ERR_INVALID, "sor_max_iter %d", p->sor_max_iter);
      if (p->init_mode < 0 || p->init_mode > 2) return fail(GPG_ERR_INVALID, "init_mode %d", p->init_mode);
      if (p->stop_mode < 0 || p->stop_mode > 3) return fail(GPG_ERR_INVALID, "stop_mode %d", p->stop_mode);
      if (p->stop_mode != GPG_STOP_REFERENCE && !(p->sor_tolerance >= 0.0))
        return fail(GPG_ERR_INVALID, "sor_tolerance %g", p->sor_tolerance);
    } else {
      if (p->mg_max_iter < 0 || p->mg_npre_smooth < 0 || p->mg_npost_smooth < 0)
        return fail(GPG_ERR_INVALID, "negative MG parameter");
    }
  }
  if (p->gra_acc) {
    if (p->gra_ghost < 1) return fail(GPG_ERR_INVALID, "gravity needs gra_ghost >= 1");
    // CUAPI_Asyn_PoissonGravitySolver.cu:137-140
    if (p->p5_gradient && p->gra_ghost != 2)
      return fail(GPG_ERR_INVALID, "incorrect parameter P5_Gradient = %d (needs gra_ghost 2)", p->p5_gradient);
  }
  return GPG_OK;
}

extern "C" int gpg_patch_sizes(const gpg_params *p, int64_t *rho, int64_t *pot_in, int64_t *pot_out, int64_t *flu) {
  if (!p) return fail(GPG_ERR_INVALID, "params is NULL");
  const int g = p->ghost, G = p->gra_ghost;
  if (g < 1 || g > 5 || G < 0 || G > 2) return fail(GPG_ERR_INVALID, "ghost %d / gra_ghost %d", g, G);
  const int64_t m = 8 + 2 * (g - 1), pn = 4 + 2 * ((g + 3) / 2), gn = 8 + 2 * G;
  if (rho) *rho = m * m * m;
  if (pot_in) *pot_in = pn * pn * pn;
  if (pot_out) *pot_out = gn * gn * gn;
  if (flu) *flu = 5 * 512;
  return GPG_OK;
}

// ===========================================================================
// stream-ordered device API
// ===========================================================================
extern "C" int gpg_poisson_gravity_device(const gpg_params *p, int npatch, const void *d_rho, const void *d_pot_in,
                                          void *d_pot_out, void *d_flu, const void *d_guess, int32_t *d_iters,
                                          double *d_resid, void *stream) {
  if (int rc = gpg_validate_params(p)) return rc;
  if (npatch < 0) return fail(GPG_ERR_INVALID, "npatch %d", npatch);
  if (npatch == 0) return GPG_OK;
  if (p->poisson) {
    if (int rc = check_ptr(d_rho, "d_rho")) return rc;
    if (int rc = check_ptr(d_pot_in, "d_pot_in")) return rc;
    if (p->scheme == GPG_SOR && p->init_mode == GPG_INIT_GUESS)
      if (int rc = check_ptr(d_guess, "d_guess")) return rc;
  }
  if (p->poisson || p->gra_acc)
    if (int rc = check_ptr(d_pot_out, "d_pot_out")) return rc;
  if (p->gra_acc)
    if (int rc = check_ptr(d_flu, "d_flu")) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p->real_size == 4)
    return solve_typed<float>(*p, npatch, d_rho, d_pot_in, d_pot_out, d_flu, d_guess, d_iters, d_resid, s);
  return solve_typed<double>(*p, npatch, d_rho, d_pot_in, d_pot_out, d_flu, d_guess, d_iters, d_resid, s);
}

// ===========================================================================
// reference-shaped context API
// ===========================================================================
struct gpg_context {
  int device = 0;
  int nstream = 1;
  std::vector<cudaStream_t> streams;
  gpg_params shape{};
  int64_t cap = 0;  // patches the buffers hold
  bool allocated = false;  // gpg_mem_allocate succeeded (cap may be 0)
  int64_t n_rho = 0, n_pin = 0, n_pout = 0, n_flu = 0;
  void *d_rho = nullptr, *d_pin = nullptr, *d_pout = nullptr, *d_flu = nullptr;
  int32_t *d_iters = nullptr;
  double *d_resid = nullptr;
  void *h_rho = nullptr, *h_pin = nullptr, *h_pout = nullptr, *h_flu = nullptr;
  int64_t last_npatch = 0;
};

extern "C" int gpg_set_diagnose_device(int *npgroup, int *nstream, int device_id) {
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0)
    return fail(GPG_ERR_NO_DEVICE, "no devices supporting CUDA (%s)", cudaGetErrorString(e));
  if (device_id < 0 || device_id >= count)
    return fail(GPG_ERR_NO_DEVICE, "Input GPU ID (%d) >= # of GPUs (%d)", device_id, count);
  GPG_CUDA(cudaSetDevice(device_id));
  cudaDeviceProp prop;
  GPG_CUDA(cudaGetDeviceProperties(&prop, device_id));
  if (prop.major != 10 || prop.minor != 0)
    return fail(GPG_ERR_UNSUPPORTED, "device \"%s\" is sm_%d%d; this library is built for sm_100a", prop.name,
                prop.major, prop.minor);
  if (nstream && *nstream == GPG_NULL_INT) *nstream = 4;
  if (npgroup && *npgroup == GPG_NULL_INT) *npgroup = 32 * prop.multiProcessorCount;
  return GPG_OK;
}

extern "C" int gpg_context_create(gpg_context **out, int device_id, int nstream) {
  if (!out) return fail(GPG_ERR_INVALID, "out is NULL");
  *out = nullptr;
  if (nstream < 1 || nstream > 1024) return fail(GPG_ERR_INVALID, "nstream %d", nstream);
  int ns = nstream, npg = 1;
  if (int rc = gpg_set_diagnose_device(&npg, &ns, device_id)) return rc;
  auto *ctx = new gpg_context;
  ctx->device = device_id;
  ctx->nstream = nstream;
  ctx->streams.resize(nstream);
  for (int s = 0; s < nstream; ++s) {
    cudaError_t e = cudaStreamCreateWithFlags(&ctx->streams[s], cudaStreamNonBlocking);
    if (e != cudaSuccess) {
      for (int t = 0; t < s; ++t) cudaStreamDestroy(ctx->streams[t]);
      delete ctx;
      return fail(GPG_ERR_CUDA, "cudaStreamCreate: %s", cudaGetErrorString(e));
    }
  }
  *out = ctx;
  return GPG_OK;
}

static void release_buffers(gpg_context *c) {
  cudaFree(c->d_rho);
  cudaFree(c->d_pin);
  cudaFree(c->d_pout);
  cudaFree(c->d_flu);
  cudaFree(c->d_iters);
  cudaFree(c->d_resid);
  c->d_rho = c->d_pin = c->d_pout = c->d_flu = nullptr;
  c->d_iters = nullptr;
  c->d_resid = nullptr;
  c->cap = 0;
  c->allocated = false;
  c->last_npatch = 0;  // gpg_last_iterations has nothing to read any more
}

extern "C" int gpg_mem_allocate(gpg_context *ctx, const gpg_params *shape, int npatch_group, void **h_rho,
                                void **h_pot_in, void **h_pot_out, void **h_flu) {
  if (!ctx) return fail(GPG_ERR_INVALID, "context is NULL");
  if (int rc = gpg_validate_params(shape)) return rc;
  if (npatch_group < 0) return fail(GPG_ERR_INVALID, "npatch_group %d", npatch_group);
  if (ctx->allocated) return fail(GPG_ERR_STATE, "buffers already allocated (call gpg_mem_free first)");
  GPG_CUDA(cudaSetDevice(ctx->device));
  ctx->shape = *shape;
  ctx->cap = 8 * (int64_t)npatch_group;
  gpg_patch_sizes(shape, &ctx->n_rho, &ctx->n_pin, &ctx->n_pout, &ctx->n_flu);
  const size_t es = shape->real_size, n = ctx->cap;
  const size_t b_rho = es * n * ctx->n_rho, b_pin = es * n * ctx->n_pin, b_pout = es * n * ctx->n_pout,
               b_flu = es * n * ctx->n_flu;
  auto chk = [&](cudaError_t e, const char *what) -> int {
    if (e == cudaSuccess) return GPG_OK;
    release_buffers(ctx);
    return fail(e == cudaErrorMemoryAllocation ? GPG_ERR_OOM : GPG_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  };
  if (int rc = chk(cudaMalloc(&ctx->d_rho, b_rho), "cudaMalloc rho")) return rc;
  if (int rc = chk(cudaMalloc(&ctx->d_pin, b_pin), "cudaMalloc pot_in")) return rc;
  if (int rc = chk(cudaMalloc(&ctx->d_pout, b_pout), "cudaMalloc pot_out")) return rc;
  if (int rc = chk(cudaMalloc(&ctx->d_flu, b_flu), "cudaMalloc flu")) return rc;
  if (int rc = chk(cudaMalloc(&ctx->d_iters, sizeof(int32_t) * (n ? n : 1)), "cudaMalloc iters")) return rc;
  if (int rc = chk(cudaMalloc(&ctx->d_resid, sizeof(double) * (n ? n : 1)), "cudaMalloc resid")) return rc;
  // pinned host arrays handed to the caller (CUAPI_MemAllocate_PoissonGravity.cu:66-69)
  void **outs[4] = {h_rho, h_pot_in, h_pot_out, h_flu};
  const size_t sizes[4] = {b_rho, b_pin, b_pout, b_flu};
  void *pinned[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int k = 0; k < 4; ++k) {
    if (!outs[k]) continue;
    cudaError_t e = cudaMallocHost(&pinned[k], sizes[k] ? sizes[k] : 16);
    if (e != cudaSuccess) {
      for (int t = 0; t < k; ++t) cudaFreeHost(pinned[t]);
      return chk(e, "cudaMallocHost");
    }
  }
  for (int k = 0; k < 4; ++k)
    if (outs[k]) *outs[k] = pinned[k];
  ctx->allocated = true;
  return GPG_OK;
}

extern "C" int gpg_mem_free(gpg_context *ctx, void **h_rho, void **h_pot_in, void **h_pot_out, void **h_flu) {
  if (!ctx) return fail(GPG_ERR_INVALID, "context is NULL");
  GPG_CUDA(cudaSetDevice(ctx->device));
  for (auto s : ctx->streams) cudaStreamSynchronize(s);
  release_buffers(ctx);
  void **outs[4] = {h_rho, h_pot_in, h_pot_out, h_flu};
  for (int k = 0; k < 4; ++k) {
    if (outs[k] && *outs[k]) {
      cudaError_t e = cudaFreeHost(*outs[k]);
      if (e != cudaSuccess) return fail(GPG_ERR_CUDA, "cudaFreeHost: %s", cudaGetErrorString(e));
      *outs[k] = nullptr;
    }
  }
  return GPG_OK;
}

extern "C" int gpg_context_destroy(gpg_context *ctx) {
  if (!ctx) return GPG_OK;
  cudaSetDevice(ctx->device);
  for (auto s : ctx->streams) cudaStreamSynchronize(s);
  release_buffers(ctx);
  for (auto s : ctx->streams) cudaStreamDestroy(s);
  delete ctx;
  return GPG_OK;
}

extern "C" int gpg_asyn_poisson_gravity_solver(gpg_context *ctx, const void *h_rho, void *h_pot_in, void *h_pot_out,
                                               void *h_flu, int npatch_group, const gpg_params *p, int nstream) {
  if (!ctx) return fail(GPG_ERR_INVALID, "context is NULL");
  if (int rc = gpg_validate_params(p)) return rc;
  if (!ctx->allocated) {
    if (npatch_group > 0) return fail(GPG_ERR_STATE, "no buffers (call gpg_mem_allocate first)");
  } else if (p->real_size != ctx->shape.real_size || p->ghost != ctx->shape.ghost ||
             p->gra_ghost != ctx->shape.gra_ghost) {
    return fail(GPG_ERR_INVALID, "parameters do not match the allocated shape");
  }
  if (p->poisson && p->init_mode == GPG_INIT_GUESS)
    return fail(GPG_ERR_UNSUPPORTED, "GPG_INIT_GUESS needs the device API");
  const int64_t npatch = 8 * (int64_t)npatch_group;
  if (npatch_group < 0 || npatch > ctx->cap)
    return fail(GPG_ERR_INVALID, "npatch_group %d exceeds the allocated %lld patches", npatch_group,
                (long long)ctx->cap);
  if (nstream < 1 || nstream > ctx->nstream)
    return fail(GPG_ERR_INVALID, "GPU_NStream %d (context has %d streams)", nstream, ctx->nstream);
  if (p->poisson && (!h_rho || !h_pot_in || !h_pot_out)) return fail(GPG_ERR_INVALID, "NULL host array");
  if (p->gra_acc && (!h_flu || !h_pot_out)) return fail(GPG_ERR_INVALID, "NULL host array");
  GPG_CUDA(cudaSetDevice(ctx->device));
  ctx->last_npatch = npatch;
  if (npatch == 0) return GPG_OK;

  // per-stream chunks, CUAPI_Asyn_PoissonGravitySolver.cu:151-164
  std::vector<int64_t> count(nstream), first(nstream);
  first[0] = 0;
  if (nstream == 1) {
    count[0] = npatch;
  } else {
    for (int s = 0; s < nstream - 1; ++s) {
      count[s] = npatch / nstream;
      first[s + 1] = first[s] + count[s];
    }
    count[nstream - 1] = npatch - first[nstream - 1];
  }
  const size_t es = p->real_size;
  auto bp = [](const void *base, int64_t off) { return (void *)((const char *)base + off); };
  for (int s = 0; s < nstream; ++s) {
    if (count[s] == 0) continue;
    cudaStream_t st = ctx->streams[s];
    const int64_t f = first[s], c = count[s];
    if (p->poisson) {
      GPG_CUDA(cudaMemcpyAsync(bp(ctx->d_rho, f * ctx->n_rho * es), bp(h_rho, f * ctx->n_rho * es),
                               c * ctx->n_rho * es, cudaMemcpyHostToDevice, st));
      GPG_CUDA(cudaMemcpyAsync(bp(ctx->d_pin, f * ctx->n_pin * es), bp(h_pot_in, f * ctx->n_pin * es),
                               c * ctx->n_pin * es, cudaMemcpyHostToDevice, st));
    }
    if (p->gra_acc) {
      if (!p->poisson)
        GPG_CUDA(cudaMemcpyAsync(bp(ctx->d_pout, f * ctx->n_pout * es), bp(h_pot_out, f * ctx->n_pout * es),
                                 c * ctx->n_pout * es, cudaMemcpyHostToDevice, st));
      GPG_CUDA(cudaMemcpyAsync(bp(ctx->d_flu, f * ctx->n_flu * es), bp(h_flu, f * ctx->n_flu * es),
                               c * ctx->n_flu * es, cudaMemcpyHostToDevice, st));
    }
  }
  for (int s = 0; s < nstream; ++s) {
    if (count[s] == 0) continue;
    const int64_t f = first[s];
    int rc = gpg_poisson_gravity_device(
        p, (int)count[s], bp(ctx->d_rho, f * ctx->n_rho * es), bp(ctx->d_pin, f * ctx->n_pin * es),
        bp(ctx->d_pout, f * ctx->n_pout * es), bp(ctx->d_flu, f * ctx->n_flu * es), nullptr,
        p->poisson ? ctx->d_iters + f : nullptr, p->poisson ? ctx->d_resid + f : nullptr, ctx->streams[s]);
    if (rc) return rc;
  }
  for (int s = 0; s < nstream; ++s) {
    if (count[s] == 0) continue;
    cudaStream_t st = ctx->streams[s];
    const int64_t f = first[s], c = count[s];
    if (p->poisson) {
      GPG_CUDA(cudaMemcpyAsync(bp(h_pot_out, f * ctx->n_pout * es), bp(ctx->d_pout, f * ctx->n_pout * es),
                               c * ctx->n_pout * es, cudaMemcpyDeviceToHost, st));
    }
    if (p->gra_acc)
      GPG_CUDA(cudaMemcpyAsync(bp(h_flu, f * ctx->n_flu * es), bp(ctx->d_flu, f * ctx->n_flu * es),
                               c * ctx->n_flu * es, cudaMemcpyDeviceToHost, st));
  }
  return GPG_OK;
}

extern "C" int gpg_synchronize(gpg_context *ctx) {
  if (ctx) {
    GPG_CUDA(cudaSetDevice(ctx->device));
    for (auto s : ctx->streams) GPG_CUDA(cudaStreamSynchronize(s));
  } else {
    GPG_CUDA(cudaDeviceSynchronize());
  }
  GPG_CUDA(cudaGetLastError());
  return GPG_OK;
}

extern "C" int gpg_last_iterations(gpg_context *ctx, int32_t *iters, double *resid, int npatch) {
  if (!ctx) return fail(GPG_ERR_INVALID, "context is NULL");
  if (npatch < 0 || npatch > ctx->last_npatch)
    return fail(GPG_ERR_INVALID, "npatch %d (last solve had %lld)", npatch, (long long)ctx->last_npatch);
  // read from the device on request: the per-call solve moves no per-patch
  // diagnostics over the host link
  GPG_CUDA(cudaSetDevice(ctx->device));
  for (auto s : ctx->streams) GPG_CUDA(cudaStreamSynchronize(s));
  if (iters && npatch)
    GPG_CUDA(cudaMemcpy(iters, ctx->d_iters, sizeof(int32_t) * npatch, cudaMemcpyDeviceToHost));
  if (resid && npatch) GPG_CUDA(cudaMemcpy(resid, ctx->d_resid, sizeof(double) * npatch, cudaMemcpyDeviceToHost));
  return GPG_OK;
}

// ===========================================================================
// SOR kernel variants (autotuning)
// ===========================================================================
extern "C" int gpg_sor_variant_count(void) { return kSorVariants; }

extern "C" int gpg_sor_variant_info(int variant, int *patches_per_cta, int *phased) {
  if (variant < 0 || variant >= kSorVariants) return fail(GPG_ERR_INVALID, "variant %d", variant);
  if (patches_per_cta) *patches_per_cta = kSorVariantPPC[variant];
  if (phased) *phased = kSorVariantPhased[variant];
  return GPG_OK;
}

extern "C" int gpg_sor_variant_staged(int variant, int *staged) {
  if (variant < 0 || variant >= kSorVariants) return fail(GPG_ERR_INVALID, "variant %d", variant);
  if (staged) *staged = kSorVariantStaged[variant];
  return GPG_OK;
}

extern "C" int gpg_sor_variant_layout(int variant, int *lanes_per_column, int *rows_per_lane) {
  if (variant < 0 || variant >= kSorVariants) return fail(GPG_ERR_INVALID, "variant %d", variant);
  if (lanes_per_column) *lanes_per_column = kSorVariantSplit[variant];
  if (rows_per_lane) *rows_per_lane = kSorVariantRows[variant];
  return GPG_OK;
}

namespace {
template <typename T, int G, int Z, int Y>
void sor_layout_fill(int *o) {
  using C = gpg::SorCfg<T, G, Z, Y>;
  const int v[GPG_SOR_LAYOUT_FIELDS] = {Z, Y, C::MH, C::R, C::P, C::PADZ, C::U, C::BLOCK, C::TEAM, C::PP, C::FITS};
  for (int i = 0; i < GPG_SOR_LAYOUT_FIELDS; ++i) o[i] = v[i];
}

template <typename T, int G>
void sor_layout_zy(int z, int y, int *o) {
  if (z == 1 && y == 1) sor_layout_fill<T, G, 1, 1>(o);
  else if (z == 2 && y == 1) sor_layout_fill<T, G, 2, 1>(o);
  else if (z == 2 && y == 2) sor_layout_fill<T, G, 2, 2>(o);
  else sor_layout_fill<T, G, 1, 2>(o);
}

template <typename T>
void sor_layout_g(int g, int z, int y, int *o) {
  switch (g) {
    case 1: return sor_layout_zy<T, 1>(z, y, o);
    case 2: return sor_layout_zy<T, 2>(z, y, o);
    case 3: return sor_layout_zy<T, 3>(z, y, o);
    case 4: return sor_layout_zy<T, 4>(z, y, o);
    default: return sor_layout_zy<T, 5>(z, y, o);
  }
}
}  // namespace

extern "C" int gpg_sor_layout(int real_size, int ghost, int variant, int *fields) {
  if ((real_size != 4 && real_size != 8) || ghost < 1 || ghost > 5 || variant < 0 || variant >= kSorVariants ||
      !fields)
    return fail(GPG_ERR_INVALID, "real_size %d ghost %d variant %d", real_size, ghost, variant);
  const int z = kSorVariantSplit[variant], y = kSorVariantRows[variant];
  if (real_size == 4)
    sor_layout_g<float>(ghost, z, y, fields);
  else
    sor_layout_g<double>(ghost, z, y, fields);
  return GPG_OK;
}

extern "C" int gpg_set_sor_variant(int real_size, int ghost, int variant) {
  std::call_once(g_tune_once, load_tune_file);
  if ((real_size != 4 && real_size != 8) || ghost < 1 || ghost > 5 || variant < -1 || variant >= kSorVariants)
    return fail(GPG_ERR_INVALID, "real_size %d ghost %d variant %d", real_size, ghost, variant);
  const int t = real_size == 8;
  // -1: back to the library's own choice (built-in table and small-batch rule)
  g_sor_variant[t][ghost].store(variant < 0 ? kSorDefault[t][ghost] : variant, std::memory_order_relaxed);
  g_sor_pinned[t][ghost].store(variant >= 0, std::memory_order_relaxed);
  return GPG_OK;
}

extern "C" int gpg_sor_variant_for_launch(int real_size, int ghost, int64_t npatch, int *variant) {
  std::call_once(g_tune_once, load_tune_file);
  if ((real_size != 4 && real_size != 8) || ghost < 1 || ghost > 5 || npatch < 0 || !variant)
    return fail(GPG_ERR_INVALID, "real_size %d ghost %d npatch %lld", real_size, ghost, (long long)npatch);
  *variant = sor_variant_for(real_size == 8, ghost, npatch);
  return GPG_OK;
}

extern "C" int gpg_get_sor_variant(int real_size, int ghost, int *variant) {
  std::call_once(g_tune_once, load_tune_file);
  if ((real_size != 4 && real_size != 8) || ghost < 1 || ghost > 5 || !variant)
    return fail(GPG_ERR_INVALID, "real_size %d ghost %d", real_size, ghost);
  *variant = g_sor_variant[real_size == 8][ghost].load(std::memory_order_relaxed);
  return GPG_OK;
}

// ===========================================================================
// batched mixed-ghost-size SOR (persistent kernel + device work queue)
// ===========================================================================
namespace {

const double kDefaultOmega[5] = {1.49, 1.57, 1.62, 1.65, 1.69};  // Main.cpp:1145

template <typename T>
struct BatchLaunchCfg {
  AttrOnce attr;
  std::once_flag occ_once[kMaxDevices];
  int blocks_per_sm[kMaxDevices] = {};
  int sms[kMaxDevices] = {};
  cudaError_t err[kMaxDevices] = {};
};

// attributes and occupancy of the persistent batch kernel on the current
// device; *grid_max = resident CTAs of the whole device
template <typename T>
int batch_prepare(int64_t *grid_max = nullptr) {
  static BatchLaunchCfg<T> cfg;
  const size_t smem = gpg::batch_smem_bytes<T>();
  if (int rc = ensure_smem(gpg::sor_batch_kernel<T>, smem, cfg.attr)) return rc;
  int dev = 0;
  if (int rc = current_device(&dev)) return rc;
  std::call_once(cfg.occ_once[dev], [&] {
    cudaError_t &err = cfg.err[dev];
    err = cudaDeviceGetAttribute(&cfg.sms[dev], cudaDevAttrMultiProcessorCount, dev);
    if (err == cudaSuccess)
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cfg.blocks_per_sm[dev], gpg::sor_batch_kernel<T>,
                                                          gpg::kBatchThreads, smem);
  });
  if (cfg.err[dev] != cudaSuccess) return fail(GPG_ERR_CUDA, "batch occupancy: %s", cudaGetErrorString(cfg.err[dev]));
  if (cfg.blocks_per_sm[dev] < 1) return fail(GPG_ERR_UNSUPPORTED, "batch kernel does not fit on an SM");
  if (grid_max) *grid_max = int64_t(cfg.sms[dev]) * cfg.blocks_per_sm[dev];
  return GPG_OK;
}

int validate_batch(const gpg_params *p, int ngroup, const gpg_batch_group *groups) {
  if (int rc = gpg_validate_params(p)) return rc;
  if (!p->poisson || p->scheme != GPG_SOR) return fail(GPG_ERR_UNSUPPORTED, "batched solve is SOR only");
  if (ngroup < 0 || ngroup > GPG_BATCH_MAX_GROUPS)
    return fail(GPG_ERR_INVALID, "ngroup %d (max %d)", ngroup, GPG_BATCH_MAX_GROUPS);
  if (ngroup && !groups) return fail(GPG_ERR_INVALID, "groups is NULL");
  for (int i = 0; i < ngroup; ++i) {
    const gpg_batch_group &g = groups[i];
    gpg_params q = *p;
    q.ghost = g.ghost;
    if (int rc = gpg_validate_params(&q)) return rc;
    if (g.npatch < 0) return fail(GPG_ERR_INVALID, "group %d: npatch %d", i, g.npatch);
    if (g.npatch == 0) continue;
    if (!g.d_rho || !g.d_pot_in || !g.d_pot_out) return fail(GPG_ERR_INVALID, "group %d: NULL array", i);
    if (p->gra_acc && !g.d_flu) return fail(GPG_ERR_INVALID, "group %d: d_flu is NULL", i);
    if (p->init_mode == GPG_INIT_GUESS && !g.d_guess) return fail(GPG_ERR_INVALID, "group %d: d_guess is NULL", i);
  }
  return GPG_OK;
}

template <typename T>
int solve_batch_typed(const gpg_params &p, int ngroup, const gpg_batch_group *groups, uint32_t *counter,
                      cudaStream_t s) {
  gpg::BatchArgs<T> b{};
  int order[gpg::kBatchMaxGroups];
  std::iota(order, order + ngroup, 0);
  // largest cubes first: their units are the longest, so they start earliest
  std::stable_sort(order, order + ngroup, [&](int x, int y) { return groups[x].ghost > groups[y].ghost; });
  int64_t u = 0;
  int k = 0;
  for (int n = 0; n < ngroup; ++n) {
    const int idx = order[n];
    const gpg_batch_group &gr = groups[idx];
    if (gr.npatch == 0) continue;
    gpg_params q = p;
    q.ghost = gr.ghost;
    q.sor_omega = gr.sor_omega > 0 ? gr.sor_omega : kDefaultOmega[gr.ghost - 1];
    b.grp[k] = gpg::make_args<T>(q, gr.npatch, gr.d_rho, gr.d_pot_in, gr.d_pot_out, gr.d_flu, gr.d_guess, gr.d_iters,
                            gr.d_resid);
    b.ghost[k] = gr.ghost;
    b.unit_start[k] = u;
    const int ppu = gpg::batch_patches_per_unit<T>(gr.ghost);
    u += (gr.npatch + ppu - 1) / ppu;
    ++k;
  }
  b.unit_start[k] = u;
  b.ngroup = k;
  b.nunit = u;
  b.counter = counter;
  if (u == 0) return GPG_OK;
  int64_t grid_max = 0;
  if (int rc = batch_prepare<T>(&grid_max)) return rc;
  const int64_t grid = std::min<int64_t>(u, grid_max);
  GPG_CUDA(cudaMemsetAsync(counter, 0, sizeof(uint32_t), s));
  gpg::sor_batch_kernel<T><<<(unsigned)grid, gpg::kBatchThreads, gpg::batch_smem_bytes<T>(), s>>>(b);
  GPG_CUDA(cudaGetLastError());
  return GPG_OK;
}

}  // namespace

extern "C" int gpg_solve_batch_device(const gpg_params *p, int ngroup, const gpg_batch_group *groups,
                                      uint32_t *d_counter, void *stream) {
  if (int rc = validate_batch(p, ngroup, groups)) return rc;
  if (!d_counter) return fail(GPG_ERR_INVALID, "d_counter is NULL");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return p->real_size == 4 ? solve_batch_typed<float>(*p, ngroup, groups, d_counter, s)
                           : solve_batch_typed<double>(*p, ngroup, groups, d_counter, s);
}

struct gpg_batch_plan {
  int device = 0;
  uint32_t *d_counter = nullptr;
  cudaStream_t capture = nullptr;
  cudaStream_t branch[GPG_BATCH_MAX_GROUPS] = {};
  cudaEvent_t fork = nullptr, join[GPG_BATCH_MAX_GROUPS] = {};
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

namespace {
// Per-ghost-size kernels of a batch as parallel branches of the capture:
// fork from `main`, one branch stream per group, join back.
int capture_concurrent(gpg_batch_plan *plan, const gpg_params *p, int ngroup, const gpg_batch_group *groups) {
  GPG_CUDA(cudaEventRecord(plan->fork, plan->capture));
  for (int i = 0; i < ngroup; ++i) {
    const gpg_batch_group &g = groups[i];
    GPG_CUDA(cudaStreamWaitEvent(plan->branch[i], plan->fork, 0));
    if (g.npatch > 0) {
      gpg_params q = *p;
      q.ghost = g.ghost;
      q.sor_omega = g.sor_omega > 0 ? g.sor_omega : kDefaultOmega[g.ghost - 1];
      if (int rc = gpg_poisson_gravity_device(&q, g.npatch, g.d_rho, g.d_pot_in, g.d_pot_out, g.d_flu, g.d_guess,
                                              g.d_iters, g.d_resid, plan->branch[i]))
        return rc;
    }
    GPG_CUDA(cudaEventRecord(plan->join[i], plan->branch[i]));
    GPG_CUDA(cudaStreamWaitEvent(plan->capture, plan->join[i], 0));
  }
  return GPG_OK;
}
}  // namespace

extern "C" int gpg_batch_plan_destroy(gpg_batch_plan *plan) {
  if (!plan) return GPG_OK;
  cudaSetDevice(plan->device);
  if (plan->exec) cudaGraphExecDestroy(plan->exec);
  if (plan->graph) cudaGraphDestroy(plan->graph);
  if (plan->capture) cudaStreamDestroy(plan->capture);
  for (int i = 0; i < GPG_BATCH_MAX_GROUPS; ++i) {
    if (plan->branch[i]) cudaStreamDestroy(plan->branch[i]);
    if (plan->join[i]) cudaEventDestroy(plan->join[i]);
  }
  if (plan->fork) cudaEventDestroy(plan->fork);
  if (plan->d_counter) cudaFree(plan->d_counter);
  delete plan;
  return GPG_OK;
}

extern "C" int gpg_batch_plan_create(gpg_batch_plan **out, const gpg_params *p, int ngroup,
                                     const gpg_batch_group *groups, int device_id, int mode) {
  if (!out) return fail(GPG_ERR_INVALID, "plan is NULL");
  *out = nullptr;
  if (mode != GPG_PLAN_PERSISTENT && mode != GPG_PLAN_CONCURRENT) return fail(GPG_ERR_INVALID, "mode %d", mode);
  if (int rc = validate_batch(p, ngroup, groups)) return rc;
  GPG_CUDA(cudaSetDevice(device_id));
  std::unique_ptr<SharedSms> shared(mode == GPG_PLAN_CONCURRENT ? new SharedSms : nullptr);
  if (mode == GPG_PLAN_CONCURRENT) {
    // every kernel the branches launch gets its attributes outside the capture
    for (int i = 0; i < ngroup; ++i) {
      if (groups[i].npatch == 0) continue;
      gpg_params q = *p;
      q.ghost = groups[i].ghost;
      if (int rc = gpg_poisson_gravity_device(&q, 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                              nullptr, nullptr))
        return rc;  // npatch 0: validates only
      if (int rc = prepare_solve_kernels(q)) return rc;
    }
  }
  // kernel attributes and occupancy are queried outside the capture
  if (int rc = p->real_size == 4 ? batch_prepare<float>() : batch_prepare<double>()) return rc;
  auto *plan = new gpg_batch_plan;
  plan->device = device_id;
  auto cleanup = [&](int rc) {
    gpg_batch_plan_destroy(plan);
    return rc;
  };
  cudaError_t e = cudaMalloc(&plan->d_counter, sizeof(uint32_t));
  if (e != cudaSuccess) return cleanup(fail(GPG_ERR_OOM, "cudaMalloc counter: %s", cudaGetErrorString(e)));
  e = cudaStreamCreateWithFlags(&plan->capture, cudaStreamNonBlocking);
  if (e != cudaSuccess) return cleanup(fail(GPG_ERR_CUDA, "cudaStreamCreate: %s", cudaGetErrorString(e)));
  if (mode == GPG_PLAN_CONCURRENT) {
    e = cudaEventCreateWithFlags(&plan->fork, cudaEventDisableTiming);
    for (int i = 0; e == cudaSuccess && i < ngroup; ++i) {
      e = cudaStreamCreateWithFlags(&plan->branch[i], cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&plan->join[i], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) return cleanup(fail(GPG_ERR_CUDA, "plan streams: %s", cudaGetErrorString(e)));
  }
  e = cudaStreamBeginCapture(plan->capture, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return cleanup(fail(GPG_ERR_CUDA, "cudaStreamBeginCapture: %s", cudaGetErrorString(e)));
  int rc;
  if (mode == GPG_PLAN_CONCURRENT)
    rc = capture_concurrent(plan, p, ngroup, groups);
  else
    rc = p->real_size == 4 ? solve_batch_typed<float>(*p, ngroup, groups, plan->d_counter, plan->capture)
                           : solve_batch_typed<double>(*p, ngroup, groups, plan->d_counter, plan->capture);
  e = cudaStreamEndCapture(plan->capture, &plan->graph);
  if (rc) return cleanup(rc);
  if (e != cudaSuccess) return cleanup(fail(GPG_ERR_CUDA, "cudaStreamEndCapture: %s", cudaGetErrorString(e)));
  e = cudaGraphInstantiate(&plan->exec, plan->graph, 0);
  if (e != cudaSuccess) return cleanup(fail(GPG_ERR_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(e)));
  *out = plan;
  return GPG_OK;
}

extern "C" int gpg_batch_plan_launch(gpg_batch_plan *plan, void *stream) {
  if (!plan || !plan->exec) return fail(GPG_ERR_INVALID, "plan is NULL");
  GPG_CUDA(cudaGraphLaunch(plan->exec, static_cast<cudaStream_t>(stream)));
  return GPG_OK;
}

// ===========================================================================
// batched SOR without any allocation by the library or the caller
// ===========================================================================
// For callers that may not allocate device memory when they solve: codes that
// hand all device memory to their own pool up front, solves issued while
// another runtime holds the allocator, or a fixed memory budget that must not
// move between steps.  The batch kernel's only scratch, its work-queue
// counter, lives here in a static device array instead of a caller buffer.
// Every GPU that loads libgpg holds this array until the process exits; all
// calls on one device share it.
namespace {

static __device__ __align__(256) unsigned int g_noalloc_queue[GPG_BATCH_NOALLOC_SCRATCH_WORDS];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned int *g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of g_noalloc_queue on the current device.  In host code the
// array's name only stands in for the symbol, so the address is looked up
// once per device (with that device current) and cached.
int noalloc_scratch(unsigned int **out) {
  int dev = 0;
  GPG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices)
    return fail(GPG_ERR_UNSUPPORTED, "device %d: at most %d devices supported", dev, kNoAllocMaxDevices);
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void *ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_queue);
    if (e != cudaSuccess || ptr == nullptr)
      return fail(GPG_ERR_CUDA, "cudaGetSymbolAddress(work-queue scratch): %s", cudaGetErrorString(e));
    g_noalloc_ptr[dev] = static_cast<unsigned int *>(ptr);
  }
  *out = g_noalloc_ptr[dev];
  return GPG_OK;
}

}  // namespace

extern "C" int gpg_solve_batch_device_noalloc(const gpg_params *p, int ngroup, const gpg_batch_group *groups,
                                              void *stream) {
  if (int rc = validate_batch(p, ngroup, groups)) return rc;
  int64_t total = 0;
  for (int i = 0; i < ngroup; ++i) total += groups[i].npatch;
  if (total > GPG_BATCH_NOALLOC_MAX_PATCHES)
    return fail(GPG_ERR_INVALID,
                "batch of %lld patches exceeds the %lld that one call without allocation may queue "
                "(its work-queue counter is a single 32-bit word)",
                (long long)total, (long long)GPG_BATCH_NOALLOC_MAX_PATCHES);
  unsigned int *counter = nullptr;
  if (int rc = noalloc_scratch(&counter)) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the counter is reset to zero on `stream` before the kernel reads it
  return p->real_size == 4 ? solve_batch_typed<float>(*p, ngroup, groups, counter, s)
                           : solve_batch_typed<double>(*p, ngroup, groups, counter, s);
}
