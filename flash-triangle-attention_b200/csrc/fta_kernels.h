// Internal launch interface between the C ABI (api.cu) and the kernels.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace fta {

// Records `cuda_error` (a cudaError_t) as the calling thread's last CUDA error, the value
// fta_last_cuda_error() reports, and clears the runtime's own record of it; returns FTA_ERR_CUDA.
int record_cuda_error(int cuda_error);

// Every launch_* function below returns cudaSuccess (0) or the cudaError_t of the call that failed
// (the launch itself or an attribute call before it), which the caller hands to record_cuda_error.

// cudaFuncAttributeMaxDynamicSharedMemorySize is a property of a kernel ON ONE DEVICE: a process
// that drives several GPUs has to set it once per device. One flag per device ordinal; two threads
// that race on the same device both make the (idempotent) call.
struct PerDeviceOnce {
  static constexpr int kMaxDevices = 64;
  std::atomic<unsigned char> done[kMaxDevices] = {};
};
template <typename Kernel>
inline cudaError_t ensure_dynamic_smem(PerDeviceOnce& once, Kernel kern, int bytes) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool tracked = dev >= 0 && dev < PerDeviceOnce::kMaxDevices;
  if (tracked && once.done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && tracked) once.done[dev].store(1, std::memory_order_release);
  return e;
}

// Launches `kern` so that it may start while the kernel before it on the stream still runs (programmatic stream
// serialization); `kern` calls grid_dependency_wait() before it touches memory.
template <typename Kernel, typename... Args>
inline cudaError_t launch_overlapped(Kernel kern, dim3 grid, int threads, int smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// SM count of the current device, looked up once per device (the attribute call costs more than the
// rest of a launch's host arithmetic).
inline int num_sms() {
  static std::atomic<int> cached[PerDeviceOnce::kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  const bool tracked = dev >= 0 && dev < PerDeviceOnce::kMaxDevices;
  if (tracked) {
    if (const int n = cached[dev].load(std::memory_order_relaxed)) return n;
  }
  int sms = 148;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && tracked)
    cached[dev].store(sms, std::memory_order_relaxed);
  return sms;
}

// The status word of a launch and its optional mirror in mapped host memory. A failed wait leaves its code
// in the word; the forward kernel (as it tears down) and the last kernel of a backward pass copy a word that
// is not zero to the mirror themselves, so the host can look for a failure without a copy or a
// synchronisation on the stream.
struct Status {
  int* word;
  int* mirror;  // nullptr: no mirror
};

struct FwdArgs {
  CUtensorMap tmQ, tmK, tmV, tmBias;
  void* o;
  void* o_resid;  // nullptr, or the rounding residual of O with O's strides
  float* lse;     // nullptr: no statistics (no backward pass will follow)
  Status status;
  int B, H, L1, L2, D;
  bool bf16;
  long long so[4];  // element strides of O (and of the residual) over (B, H, L1, L2)
  float sm_scale;
};
int launch_fwd(const FwdArgs& a, cudaStream_t stream);
// launch_fwd's kernel with tiles of 64 keys
int launch_fwd_quad(const FwdArgs& a, cudaStream_t stream);
// keys per K / V tile of the kernel that launch_fwd takes for a problem: the box height of FwdArgs::tmK and tmV
int fwd_key_block(int L2, int D);

struct BwdArgs {
  CUtensorMap tmQ, tmK, tmV, tmDO, tmBiasT;  // tmBiasT: over the key-major copy of the bias
  CUtensorMap tmDQ;    // the float32 dQ accumulator as (B*H*L1, L2, D), box 32 queries x 16 columns, 64 B swizzle: zeroed
                       // before, receives the sum over the key blocks of dS K (not used for L2 <= 128)
  CUtensorMap tmDK, tmDV, tmDQ16;  // the 16-bit outputs, boxes of 32 columns x 32 rows, 64 B swizzle (tmDQ16: L2 <= 128)
  CUtensorMap tmPlane; // the partial dBias planes as (nplanes*B*H, L2 keys, L2 queries) float32, box 128 keys x
                       // 32 queries, 128 B swizzle
  const float* lse;    // (3,B,H,L1,L2p), L2p = L2 rounded up to 128: -max, -log2(sum), combined (NaN where inexact)
  const float* delta;  // (B,H,L1,L2p)
  int* status;
  int B, H, L1, L2, D;
  int nplanes;  // bwd_num_planes()
  bool bf16;
  float sm_scale;
};
int launch_bwd(const BwdArgs& a, cudaStream_t stream);
int bwd_rows_per_cta(int D);
int bwd_num_planes(int B, int H, int L1, int L2, int D, int sms);

// delta[(b,h,i), j] = sum_d (O[.,d] + R[.,d]) * dO[.,d] for j < L2 and 0 up to `delta_pitch` (elements between rows
// (b,h,i) of delta: L2 rounded up to 128; the backward kernel reads whole 128-blocks)
struct PreArgs {
  const void* o;
  const void* o_resid;  // R, strides of O; may be nullptr
  const void* dout;
  float* delta;
  int delta_pitch, B, H, L1, L2, D;
  bool bf16;
  long long so[4], sdo[4];  // element strides of O, dO over (B, H, L1, L2)
};
int launch_preprocess(const PreArgs& a, cudaStream_t stream);

// out[b][h][q][k], (B, H, L2p, L2p) contiguous: the bias where q, k < L2 and the key is kept by
// `key_mask` ((B, L2) bytes, non-zero = keep; nullptr = keep all), -inf for every other key, 0 for
// the kept keys of the padding queries q >= L2. `sb`: element strides of the bias; 16-byte loads where they, L2
// and the pointers allow it, single elements otherwise
int launch_mask_bias(const void* bias, const long long sb[4], const uint8_t* key_mask, void* out, int B, int H, int L2,
                     int L2p, bool bf16, cudaStream_t stream);

// Backward prologue, one launch: bias_t[bh][k][q] = bias[b][h][q][k] (16-bit elements; `sb` = element
// strides of the bias) and zero-fill of the float32 dQ accumulator (`dq_elems` floats, a multiple of 4, or 0); with `pre`
// the preprocess too (three independent streams that share the launch)
int launch_bwd_prologue(const void* bias, const long long sb[4], void* bias_t, int B, int H, int L2, float* dq32,
                        long long dq_elems, const PreArgs* pre, cudaStream_t stream);

// Backward epilogue, one launch: dq[row, d] = (dtype)(scale * dq32[row, d]) (dq32 == nullptr: dq has been written
// already) and dbias_f32[bh][query][key] = sum_p planes[p][bh][key][query] in plane order, with an optional rounded
// copy, for the key-major planes that the backward kernel writes: (nplanes, B*H, key, query), rows of L2 rounded up to 8
// elements
int launch_bwd_epilogue(const float* dq32, void* dq, const long long sdq[4], int B, int H, int L1, int L2, int D,
                        float scale, const float* planes, int nplanes, float* dbias_f32, void* dbias_cast, bool bf16,
                        Status status, cudaStream_t stream);

// out = sum over r of parts[r][0..n) (rank order), float32 and / or rounded to 16 bits; `parts`: device
// array of `nranks` device pointers (peer mappings included); n a multiple of 8
// `flags` == nullptr: the caller has lined the ranks up; otherwise the kernel does (bounded wait, see the kernel)
int launch_dbias_sum_peers(const float* const* parts, int nranks, long long n, float* out_f32, void* out_cast,
                           bool bf16, int* const* flags, int rank, int epoch, unsigned long long limit_ns, int* status,
                           cudaStream_t stream);
// the same with the work split over the ranks: this rank sums its 1/nranks slice and stores the rounded
// result into every rank's buffer `outs[r]` (device array of nranks device pointers)
// `flags` == nullptr: the caller lines the ranks up before and after; otherwise the kernel does, and a
// one-block kernel behind it holds the stream until every rank's slice has arrived (`my_flags`: this
// rank's own flag array, 2 * nranks + 1 words)
int launch_dbias_sum_peers_sliced(const float* const* parts, void* const* outs, int nranks, int rank, long long n,
                                  bool bf16, int* const* flags, const int* my_flags, int epoch,
                                  unsigned long long limit_ns, int* status, cudaStream_t stream);
// dst[i] = (dtype) src[i], n a multiple of 4
int launch_dbias_cast(const float* src, long long n, void* dst, bool bf16, cudaStream_t stream);

}  // namespace fta
