// C ABI of libfta (declared in include/fta.h): argument validation, TMA tensor maps, launches.
// Nothing here allocates device memory; every buffer belongs to the caller.
#include "../../include/fta.h"

#include "fta_kernels.h"
#include "native_api.h"
#include "tmap.h"

namespace {

thread_local int g_last_cuda_error = 0;
thread_local cudaEvent_t g_prof_start = nullptr, g_prof_stop = nullptr;

// Every failed runtime call ends here. The runtime keeps its error until somebody asks, and the launches ask to learn
// how they went: what is reported here must not be found again by the next, healthy one.
int cuda_fail(cudaError_t e) {
  cudaGetLastError();
  g_last_cuda_error = static_cast<int>(e);
  return FTA_ERR_CUDA;
}
int cuda_fail(int e) { return cuda_fail(static_cast<cudaError_t>(e)); }

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// The C ABI takes L2 in multiples of 8 (its dBias buffers and biases have rows of L2 elements, read and written
// 16 bytes at a time); the native entry points stage the bias and take any L2.
int check_problem(const FtaProblem* p, bool any_l2 = false) {
  if (!p) return FTA_ERR_NULL;
  if (p->B <= 0 || p->H <= 0 || p->L1 <= 0 || p->L2 <= 0) return FTA_ERR_SHAPE;
  if (!any_l2 && p->L2 % 8 != 0) return FTA_ERR_SHAPE;
  if (p->D != 32 && p->D != 64) return FTA_ERR_HEAD_DIM;
  if (p->dtype != FTA_FP16 && p->dtype != FTA_BF16) return FTA_ERR_DTYPE;
  if (static_cast<long long>(p->B) * p->H > 65535) return FTA_ERR_TOO_LARGE;
  return FTA_OK;
}

int check_t5(const FtaTensor5* t) {
  if (!t || !t->ptr) return FTA_ERR_NULL;
  if (reinterpret_cast<uintptr_t>(t->ptr) % 16 != 0) return FTA_ERR_ALIGN;
  if (t->stride[4] != 1) return FTA_ERR_STRIDE;
  for (int i = 0; i < 4; ++i)
    if (t->stride[i] <= 0 || t->stride[i] % 8 != 0) return FTA_ERR_STRIDE;
  return FTA_OK;
}

int check_t4(const FtaTensor4* t) {
  if (!t || !t->ptr) return FTA_ERR_NULL;
  if (reinterpret_cast<uintptr_t>(t->ptr) % 16 != 0) return FTA_ERR_ALIGN;
  if (t->stride[3] != 1) return FTA_ERR_STRIDE;
  for (int i = 0; i < 3; ++i)
    if (t->stride[i] <= 0 || t->stride[i] % 8 != 0) return FTA_ERR_STRIDE;
  return FTA_OK;
}

// 5-D map over (D, L2, L1, H, B), tile = `box_rows` rows of L2 x D, swizzle = row bytes (64 or 128).
int map5(CUtensorMap* m, const FtaProblem* p, const FtaTensor5* t, uint32_t box_rows = 128) {
  const uint64_t dims[5] = {static_cast<uint64_t>(p->D), static_cast<uint64_t>(p->L2),
                            static_cast<uint64_t>(p->L1), static_cast<uint64_t>(p->H),
                            static_cast<uint64_t>(p->B)};
  const uint64_t str[5] = {0, static_cast<uint64_t>(t->stride[3]) * 2, static_cast<uint64_t>(t->stride[2]) * 2,
                           static_cast<uint64_t>(t->stride[1]) * 2, static_cast<uint64_t>(t->stride[0]) * 2};
  const uint32_t box[5] = {static_cast<uint32_t>(p->D), box_rows, 1, 1, 1};
  return fta::make_tmap_16bit(m, t->ptr, 5, dims, str, box, p->D * 2) == 0 ? FTA_OK : FTA_ERR_TENSOR_MAP;
}

// 5-D map over (D, L2, L1, H, B) for stores of 32 rows x 32 columns
int map5_out(CUtensorMap* m, const FtaProblem* p, const FtaTensor5* t) {
  const uint64_t dims[5] = {static_cast<uint64_t>(p->D), static_cast<uint64_t>(p->L2), static_cast<uint64_t>(p->L1),
                            static_cast<uint64_t>(p->H), static_cast<uint64_t>(p->B)};
  const uint64_t str[5] = {0, static_cast<uint64_t>(t->stride[3]) * 2, static_cast<uint64_t>(t->stride[2]) * 2,
                           static_cast<uint64_t>(t->stride[1]) * 2, static_cast<uint64_t>(t->stride[0]) * 2};
  const uint32_t box[5] = {32, 32, 1, 1, 1};
  return fta::make_tmap_16bit(m, t->ptr, 5, dims, str, box, 64) == 0 ? FTA_OK : FTA_ERR_TENSOR_MAP;
}

int padded_l2(const FtaProblem* p) { return (p->L2 + 127) / 128 * 128; }

// 4-D map over the bias (key, query, H, B); `box_k` keys x 128 queries per tile. The bias the kernels
// read always spans whole 128-blocks: the caller's tensor when L2 is a multiple of 128, else the
// padded copy made by fta_mask_bias.
int map_bias(CUtensorMap* m, const FtaProblem* p, const FtaTensor4* t, int box_k, int swizzle) {
  const uint64_t l2p = static_cast<uint64_t>(padded_l2(p));
  // a ragged problem must come with the padded copy: rows at least L2p apart, planes L2p rows apart
  if (l2p != static_cast<uint64_t>(p->L2) &&
      (static_cast<uint64_t>(t->stride[2]) < l2p || static_cast<uint64_t>(t->stride[1]) < l2p * l2p))
    return FTA_ERR_STRIDE;
  const uint64_t dims[4] = {l2p, l2p, static_cast<uint64_t>(p->H), static_cast<uint64_t>(p->B)};
  const uint64_t str[4] = {0, static_cast<uint64_t>(t->stride[2]) * 2, static_cast<uint64_t>(t->stride[1]) * 2,
                           static_cast<uint64_t>(t->stride[0]) * 2};
  const uint32_t box[4] = {static_cast<uint32_t>(box_k), 128, 1, 1};
  return fta::make_tmap_16bit(m, t->ptr, 4, dims, str, box, swizzle) == 0 ? FTA_OK : FTA_ERR_TENSOR_MAP;
}

size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

size_t plane_pitch(const FtaProblem* p) { return (static_cast<size_t>(p->L2) + 7) / 8 * 8; }  // elements of a plane row
size_t plane_bytes(const FtaProblem* p) {
  return static_cast<size_t>(p->B) * p->H * p->L2 * plane_pitch(p) * sizeof(float);
}
size_t dq32_bytes(const FtaProblem* p) {
  return static_cast<size_t>(p->B) * p->H * p->L1 * p->L2 * p->D * sizeof(float);
}
// float32 dQ accumulator, dBias planes, key-major copy of the bias (16-bit, whole blocks)
size_t workspace_bytes(const FtaProblem* p, int nplanes) {
  const size_t l2p = static_cast<size_t>(padded_l2(p));
  return align256(dq32_bytes(p)) + align256(plane_bytes(p) * nplanes) +
         align256(static_cast<size_t>(p->B) * p->H * l2p * l2p * 2);
}
int plan_planes(const FtaProblem* p) { return fta::bwd_num_planes(p->B, p->H, p->L1, p->L2, p->D, fta::num_sms()); }

int forward(const FtaProblem* prob, const FtaTensor5* q, const FtaTensor5* k, const FtaTensor5* v,
            const FtaTensor4* bias, float sm_scale, const FtaTensor5* o, void* o_resid, float* lse, fta::Status status,
            cudaStream_t stream) {
  int rc = check_problem(prob, true);
  if (rc) return rc;
  if ((rc = check_t5(q)) || (rc = check_t5(k)) || (rc = check_t5(v)) || (rc = check_t5(o)) || (rc = check_t4(bias)))
    return rc;
  if (!status.word) return FTA_ERR_NULL;
  if (!aligned16(lse) || !aligned16(o_resid)) return FTA_ERR_ALIGN;
  fta::FwdArgs a;
  const uint32_t keys = static_cast<uint32_t>(fta::fwd_key_block(prob->L2, prob->D));
  if ((rc = map5(&a.tmQ, prob, q)) || (rc = map5(&a.tmK, prob, k, keys)) || (rc = map5(&a.tmV, prob, v, keys)) ||
      (rc = map_bias(&a.tmBias, prob, bias, 64, 128)))
    return rc;
  a.o = o->ptr;
  a.o_resid = o_resid;
  a.lse = lse;
  a.status = status;
  a.B = prob->B;
  a.H = prob->H;
  a.L1 = prob->L1;
  a.L2 = prob->L2;
  a.D = prob->D;
  a.bf16 = prob->dtype == FTA_BF16;
  for (int i = 0; i < 4; ++i) a.so[i] = o->stride[i];
  a.sm_scale = sm_scale;
  if (const int e = fta::launch_fwd(a, stream)) return cuda_fail(e);
  return FTA_OK;
}

int fill_pre(fta::PreArgs* a, const FtaProblem* prob, const FtaTensor5* o, const void* o_resid, const FtaTensor5* dout,
             float* delta) {
  int rc;
  if ((rc = check_t5(o)) || (rc = check_t5(dout))) return rc;
  if (!delta) return FTA_ERR_NULL;
  if (!aligned16(o_resid)) return FTA_ERR_ALIGN;
  a->o = o->ptr;
  a->o_resid = o_resid;
  a->dout = dout->ptr;
  a->delta = delta;
  a->delta_pitch = padded_l2(prob);
  for (int i = 0; i < 4; ++i) {
    a->so[i] = o->stride[i];
    a->sdo[i] = dout->stride[i];
  }
  a->B = prob->B;
  a->H = prob->H;
  a->L1 = prob->L1;
  a->L2 = prob->L2;
  a->D = prob->D;
  a->bf16 = prob->dtype == FTA_BF16;
  return FTA_OK;
}

// `pre`: also run the preprocess it describes, in the launch of the prologue (nullptr: delta is there already)
int backward(const FtaProblem* prob, int nplanes, const fta::PreArgs* pre, const FtaTensor5* q, const FtaTensor5* k, const FtaTensor5* v,
             const FtaTensor4* bias, const FtaTensor5* dout, const float* lse, const float* delta, float sm_scale,
             const FtaTensor5* dq, const FtaTensor5* dk, const FtaTensor5* dv, float* dbias_f32, void* dbias_cast,
             void* workspace, size_t have_bytes, fta::Status status, cudaStream_t st) {
  int rc;
  if ((rc = check_t5(q)) || (rc = check_t5(k)) || (rc = check_t5(v)) || (rc = check_t5(dout)) ||
      (rc = check_t5(dq)) || (rc = check_t5(dk)) || (rc = check_t5(dv)) || (rc = check_t4(bias)))
    return rc;
  if (!lse || !delta || !dbias_f32 || !status.word || !workspace) return FTA_ERR_NULL;
  // the kernel fetches the statistics with 256-byte bulk copies and the epilogue writes dBias with
  // 16-byte stores
  if (!aligned16(lse) || !aligned16(delta) || !aligned16(dbias_f32) || !aligned16(dbias_cast)) return FTA_ERR_ALIGN;
  if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0 || have_bytes < workspace_bytes(prob, nplanes))
    return FTA_ERR_WORKSPACE;
  const size_t rows = static_cast<size_t>(prob->B) * prob->H * prob->L1 * prob->L2;
  float* dq32 = static_cast<float*>(workspace);
  float* planes = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + align256(dq32_bytes(prob)));
  void* bias_t = reinterpret_cast<uint8_t*>(planes) + align256(plane_bytes(prob) * nplanes);
  const bool bf16 = prob->dtype == FTA_BF16;
  const bool one_block = prob->L2 <= 128;  // one key block: the kernel writes dq itself

  fta::BwdArgs a;
  FtaTensor4 bt;  // key-major copy: (B, H, key, query) contiguous
  bt.ptr = bias_t;
  const int l2p = padded_l2(prob);
  bt.stride[0] = static_cast<int64_t>(prob->H) * l2p * l2p;
  bt.stride[1] = static_cast<int64_t>(l2p) * l2p;
  bt.stride[2] = l2p;
  bt.stride[3] = 1;
  // the backward kernel loads Q and dO by 64-query halves
  if ((rc = map5(&a.tmQ, prob, q, 64)) || (rc = map5(&a.tmK, prob, k)) || (rc = map5(&a.tmV, prob, v)) ||
      (rc = map5(&a.tmDO, prob, dout, 64)) || (rc = map5_out(&a.tmDK, prob, dk)) || (rc = map5_out(&a.tmDV, prob, dv)) ||
      (rc = map5_out(&a.tmDQ16, prob, dq)) || (rc = map_bias(&a.tmBiasT, prob, &bt, 64, 128)))
    return rc;
  {
    // dq32 seen as (B*H*L1, L2, D) float32; the kernel adds 32-query x 16-column tiles into it with
    // TMA reductions (the part of a ragged last query block beyond L2 is clipped)
    const uint64_t bhi = static_cast<uint64_t>(prob->B) * prob->H * prob->L1;
    if (bhi >= (1ull << 31)) return FTA_ERR_SHAPE;  // tile coordinates are signed 32-bit
    const uint64_t dims[3] = {static_cast<uint64_t>(prob->D), static_cast<uint64_t>(prob->L2), bhi};
    const uint64_t str[3] = {0, static_cast<uint64_t>(prob->D) * 4, static_cast<uint64_t>(prob->L2) * prob->D * 4};
    const uint32_t dq_box[3] = {16, 32, 1}, box[3] = {32, 128, 1};
    if (fta::make_tmap(&a.tmDQ, 4, dq32, 3, dims, str, dq_box, 64) != 0) return FTA_ERR_TENSOR_MAP;
    // the partial dBias planes, key-major: (nplanes * B*H, L2 keys, L2 queries) float32, clipped alike
    const uint64_t pdims[3] = {static_cast<uint64_t>(prob->L2), static_cast<uint64_t>(prob->L2),
                               static_cast<uint64_t>(nplanes) * prob->B * prob->H};
    const uint64_t pitch = plane_pitch(prob) * 4;
    const uint64_t pstr[3] = {0, pitch, prob->L2 * pitch};
    if (fta::make_tmap(&a.tmPlane, 4, planes, 3, pdims, pstr, box, 128) != 0) return FTA_ERR_TENSOR_MAP;
  }
  a.lse = lse;
  a.delta = delta;
  a.status = status.word;
  a.nplanes = nplanes;
  a.B = prob->B;
  a.H = prob->H;
  a.L1 = prob->L1;
  a.L2 = prob->L2;
  a.D = prob->D;
  a.bf16 = bf16;
  long long sdq[4];
  for (int i = 0; i < 4; ++i) {
    sdq[i] = dq->stride[i];
  }
  a.sm_scale = sm_scale;

  long long sb[4];
  for (int i = 0; i < 4; ++i) sb[i] = bias->stride[i];
  if (const int e = fta::launch_bwd_prologue(bias->ptr, sb, bias_t, prob->B, prob->H, l2p, dq32,
                                             one_block ? 0 : static_cast<long long>(rows) * prob->D, pre, st))
    return cuda_fail(e);
  if (g_prof_start) cudaEventRecord(g_prof_start, st);
  if (const int e = fta::launch_bwd(a, st)) return cuda_fail(e);
  if (g_prof_stop) cudaEventRecord(g_prof_stop, st);
  if (const int e = fta::launch_bwd_epilogue(one_block ? nullptr : dq32, dq->ptr, sdq, prob->B, prob->H, prob->L1, prob->L2, prob->D,
                                             sm_scale, planes, nplanes, dbias_f32, dbias_cast, bf16, status, st))
    return cuda_fail(e);
  return FTA_OK;
}


}  // namespace

namespace fta {

int record_cuda_error(int cuda_error) { return cuda_fail(cuda_error); }

int native_forward(const FtaProblem& prob, const FtaTensor5& q, const FtaTensor5& k, const FtaTensor5& v,
                   const FtaTensor4& bias, float sm_scale, const FtaTensor5& o, void* o_resid, float* lse,
                   StatusPair status, cudaStream_t stream) {
  return forward(&prob, &q, &k, &v, &bias, sm_scale, &o, o_resid, lse, {status.word, status.mirror}, stream);
}

int native_mask_bias(const FtaProblem& prob, const FtaTensor4& bias, const uint8_t* key_mask, void* out,
                     cudaStream_t stream) {
  if (const int rc = check_problem(&prob, true)) return rc;
  if (!bias.ptr || !out) return FTA_ERR_NULL;
  if (!aligned16(out)) return FTA_ERR_ALIGN;
  const long long sb[4] = {bias.stride[0], bias.stride[1], bias.stride[2], bias.stride[3]};
  if (const int e = fta::launch_mask_bias(bias.ptr, sb, key_mask, out, prob.B, prob.H, prob.L2, padded_l2(&prob),
                                          prob.dtype == FTA_BF16, stream))
    return cuda_fail(e);
  return FTA_OK;
}

int native_backward_plan(const FtaProblem& prob, BackwardPlan* plan) {
  if (const int rc = check_problem(&prob, true)) return rc;
  plan->nplanes = plan_planes(&prob);
  plan->workspace_bytes = workspace_bytes(&prob, plan->nplanes);
  plan->delta_bytes = sizeof(float) * static_cast<size_t>(prob.B) * prob.H * prob.L1 * padded_l2(&prob);
  return FTA_OK;
}

int native_backward(const FtaProblem& prob, const BackwardPlan& plan, const FtaTensor5& q, const FtaTensor5& k,
                    const FtaTensor5& v, const FtaTensor4& bias, const FtaTensor5& o, const void* o_resid,
                    const FtaTensor5& dout, const float* lse, float sm_scale, const FtaTensor5& dq,
                    const FtaTensor5& dk, const FtaTensor5& dv, float* dbias_f32, void* dbias_cast, void* workspace,
                    StatusPair status, cudaStream_t stream) {
  float* delta = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + plan.workspace_bytes);
  fta::PreArgs pre;
  if (const int rc = fill_pre(&pre, &prob, &o, o_resid, &dout, delta)) return rc;
  return backward(&prob, plan.nplanes, &pre, &q, &k, &v, &bias, &dout, lse, delta, sm_scale, &dq, &dk, &dv, dbias_f32,
                  dbias_cast, workspace, plan.workspace_bytes, {status.word, status.mirror}, stream);
}

}  // namespace fta

extern "C" {

int fta_version(void) { return 200; }

const char* fta_strerror(int code) {
  switch (code) {
    case FTA_OK: return "ok";
    case FTA_ERR_NULL: return "a required pointer is NULL";
    case FTA_ERR_SHAPE: return "bad shape: sizes must be positive and L2 a multiple of 8 (of 128 without fta_mask_bias)";
    case FTA_ERR_HEAD_DIM: return "unsupported head dimension: D must be 32 or 64";
    case FTA_ERR_DTYPE: return "unsupported dtype: fp16 or bf16 only";
    case FTA_ERR_STRIDE: return "bad stride: D stride must be 1, other strides positive multiples of 8 elements";
    case FTA_ERR_ALIGN: return "every device pointer must be 16-byte aligned";
    case FTA_ERR_WORKSPACE: return "workspace too small or misaligned";
    case FTA_ERR_TENSOR_MAP: return "the driver refused a TMA tensor map";
    case FTA_ERR_CUDA: return "a CUDA runtime call failed";
    case FTA_ERR_DEVICE: return "a bounded device-side wait ran out (status word non-zero)";
    case FTA_ERR_TOO_LARGE: return "size beyond a documented maximum";
    default: return "unknown error";
  }
}

int fta_last_cuda_error(void) { return g_last_cuda_error; }

int fta_forward(const FtaProblem* prob, const FtaTensor5* q, const FtaTensor5* k, const FtaTensor5* v,
                const FtaTensor4* bias, float sm_scale, const FtaTensor5* o, void* o_resid, float* lse,
                int32_t* status, void* stream) {
  if (const int rc = check_problem(prob)) return rc;
  if (!lse) return FTA_ERR_NULL;
  return forward(prob, q, k, v, bias, sm_scale, o, o_resid, lse, {status, nullptr}, static_cast<cudaStream_t>(stream));
}

int fta_bwd_preprocess(const FtaProblem* prob, const FtaTensor5* o, const void* o_resid, const FtaTensor5* dout,
                       float* delta, void* stream) {
  fta::PreArgs a;
  if (const int rc = check_problem(prob)) return rc;
  if (const int rc = fill_pre(&a, prob, o, o_resid, dout, delta)) return rc;
  if (const int e = fta::launch_preprocess(a, static_cast<cudaStream_t>(stream))) return cuda_fail(e);
  return FTA_OK;
}

int fta_mask_bias(const FtaProblem* prob, const FtaTensor4* bias, const uint8_t* key_mask, void* out, void* stream) {
  int rc = check_problem(prob);
  if (rc) return rc;
  if ((rc = check_t4(bias))) return rc;
  if (!out) return FTA_ERR_NULL;
  if (!aligned16(out) || reinterpret_cast<uintptr_t>(key_mask) % 8 != 0) return FTA_ERR_ALIGN;
  long long sb[4];
  for (int i = 0; i < 4; ++i) sb[i] = bias->stride[i];
  if (const int e = fta::launch_mask_bias(bias->ptr, sb, key_mask, out, prob->B, prob->H, prob->L2, padded_l2(prob),
                                          prob->dtype == FTA_BF16, static_cast<cudaStream_t>(stream)))
    return cuda_fail(e);
  return FTA_OK;
}

int fta_bwd_num_planes(const FtaProblem* prob) { return check_problem(prob) ? 0 : plan_planes(prob); }

size_t fta_bwd_workspace_bytes(const FtaProblem* prob) {
  return check_problem(prob) ? 0 : workspace_bytes(prob, plan_planes(prob));
}

int fta_backward(const FtaProblem* prob, const FtaTensor5* q, const FtaTensor5* k, const FtaTensor5* v,
                 const FtaTensor4* bias, const FtaTensor5* dout, const float* lse, const float* delta,
                 float sm_scale, const FtaTensor5* dq, const FtaTensor5* dk, const FtaTensor5* dv,
                 float* dbias_f32, void* dbias_cast, void* workspace, size_t workspace_bytes, int32_t* status,
                 void* stream) {
  if (const int rc = check_problem(prob)) return rc;
  return backward(prob, plan_planes(prob), nullptr, q, k, v, bias, dout, lse, delta, sm_scale, dq, dk, dv, dbias_f32, dbias_cast,
                  workspace, workspace_bytes, {status, nullptr}, static_cast<cudaStream_t>(stream));
}

int fta_dbias_cast(const float* src, void* dst, int64_t n, int32_t dtype, void* stream) {
  if (!src || !dst) return FTA_ERR_NULL;
  if (n <= 0 || n % 4 != 0) return FTA_ERR_SHAPE;
  if (dtype != FTA_FP16 && dtype != FTA_BF16) return FTA_ERR_DTYPE;
  if (!aligned16(src) || !aligned16(dst)) return FTA_ERR_ALIGN;
  if (const int e = fta::launch_dbias_cast(src, n, dst, dtype == FTA_BF16, static_cast<cudaStream_t>(stream)))
    return cuda_fail(e);
  return FTA_OK;
}

int fta_dbias_sum_peers(const float* const* parts, int32_t nranks, int64_t n, float* out_f32, void* out_cast,
                        int32_t dtype, void* stream) {
  if (!parts || (!out_f32 && !out_cast)) return FTA_ERR_NULL;
  if (nranks < 1 || nranks > 64 || n <= 0 || n % 8 != 0) return FTA_ERR_SHAPE;
  if (dtype != FTA_FP16 && dtype != FTA_BF16) return FTA_ERR_DTYPE;
  if ((reinterpret_cast<uintptr_t>(parts) & 7u) || (out_f32 && !aligned16(out_f32)) || (out_cast && !aligned16(out_cast)))
    return FTA_ERR_ALIGN;
  if (const int e = fta::launch_dbias_sum_peers(parts, nranks, n, out_f32, out_cast, dtype == FTA_BF16, nullptr, 0, 0, 0,
                                                nullptr, static_cast<cudaStream_t>(stream)))
    return cuda_fail(e);
  return FTA_OK;
}

int fta_dbias_sum_peers_sync(const float* const* parts, int32_t* const* flags, int32_t nranks, int32_t rank,
                             int32_t epoch, int64_t n, float* out_f32, void* out_cast, int32_t dtype,
                             uint64_t wait_limit_ns, int32_t* status, void* stream) {
  if (!parts || !flags || !status || (!out_f32 && !out_cast)) return FTA_ERR_NULL;
  if (nranks < 1 || nranks > 64 || rank < 0 || rank >= nranks || epoch <= 0 || n <= 0 || n % 8 != 0) return FTA_ERR_SHAPE;
  if (dtype != FTA_FP16 && dtype != FTA_BF16) return FTA_ERR_DTYPE;
  if ((reinterpret_cast<uintptr_t>(parts) & 7u) || (reinterpret_cast<uintptr_t>(flags) & 7u) ||
      (out_f32 && !aligned16(out_f32)) || (out_cast && !aligned16(out_cast)))
    return FTA_ERR_ALIGN;
  if (wait_limit_ns == 0) wait_limit_ns = 1000000000ull;
  if (const int e = fta::launch_dbias_sum_peers(parts, nranks, n, out_f32, out_cast, dtype == FTA_BF16, flags, rank, epoch,
                                                wait_limit_ns, status, static_cast<cudaStream_t>(stream)))
    return cuda_fail(e);
  return FTA_OK;
}

int fta_dbias_sum_peers_sliced(const float* const* parts, void* const* outs, int32_t nranks, int32_t rank, int64_t n,
                               int32_t dtype, void* stream) {
  if (!parts || !outs) return FTA_ERR_NULL;
  if (nranks < 1 || nranks > 64 || rank < 0 || rank >= nranks || n <= 0 || n % 8 != 0) return FTA_ERR_SHAPE;
  if (dtype != FTA_FP16 && dtype != FTA_BF16) return FTA_ERR_DTYPE;
  if ((reinterpret_cast<uintptr_t>(parts) & 7u) || (reinterpret_cast<uintptr_t>(outs) & 7u)) return FTA_ERR_ALIGN;
  if (const int e = fta::launch_dbias_sum_peers_sliced(parts, outs, nranks, rank, n, dtype == FTA_BF16, nullptr, nullptr, 0,
                                                       0, nullptr, static_cast<cudaStream_t>(stream)))
    return cuda_fail(e);
  return FTA_OK;
}

int fta_dbias_sum_peers_sliced_sync(const float* const* parts, void* const* outs, int32_t* const* flags,
                                    const int32_t* my_flags, int32_t nranks, int32_t rank, int32_t epoch, int64_t n,
                                    int32_t dtype, uint64_t wait_limit_ns, int32_t* status, void* stream) {
  if (!parts || !outs || !flags || !my_flags || !status) return FTA_ERR_NULL;
  if (nranks < 1 || nranks > 31 || rank < 0 || rank >= nranks || epoch <= 0 || n <= 0 || n % 8 != 0) return FTA_ERR_SHAPE;
  if (dtype != FTA_FP16 && dtype != FTA_BF16) return FTA_ERR_DTYPE;
  if ((reinterpret_cast<uintptr_t>(parts) & 7u) || (reinterpret_cast<uintptr_t>(outs) & 7u) ||
      (reinterpret_cast<uintptr_t>(flags) & 7u) || (reinterpret_cast<uintptr_t>(my_flags) & 3u))
    return FTA_ERR_ALIGN;
  if (wait_limit_ns == 0) wait_limit_ns = 1000000000ull;
  if (const int e = fta::launch_dbias_sum_peers_sliced(parts, outs, nranks, rank, n, dtype == FTA_BF16, flags, my_flags, epoch,
                                                       wait_limit_ns, status, static_cast<cudaStream_t>(stream)))
    return cuda_fail(e);
  return FTA_OK;
}

int fta_memcpy_2d(void* dst, size_t dst_pitch_bytes, const void* src, size_t src_pitch_bytes, size_t width_bytes,
                  size_t rows, void* stream) {
  if (!dst || !src) return FTA_ERR_NULL;
  if (width_bytes == 0 || rows == 0) return FTA_ERR_SHAPE;
  if (dst_pitch_bytes < width_bytes || src_pitch_bytes < width_bytes) return FTA_ERR_STRIDE;
  const cudaError_t e = cudaMemcpy2DAsync(dst, dst_pitch_bytes, src, src_pitch_bytes, width_bytes, rows,
                                          cudaMemcpyDefault, static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? FTA_OK : cuda_fail(e);
}

int fta_profile_backward_kernel(void* start_event, void* stop_event) {
  g_prof_start = static_cast<cudaEvent_t>(start_event);
  g_prof_stop = static_cast<cudaEvent_t>(stop_event);
  return FTA_OK;
}

int fta_read_status(const int32_t* status, int32_t* code_out, void* stream) {
  if (!status) return FTA_ERR_NULL;
  int32_t host = 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(&host, status, sizeof(host), cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e);
  if (code_out) *code_out = host;
  return host == 0 ? FTA_OK : FTA_ERR_DEVICE;
}

}  // extern "C"
