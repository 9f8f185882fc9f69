// C++ entry points of libfta.so for the torch extension that ships beside it (torch_binding.cpp). They run
// the same validation and launches as the C ABI (include/fta.h); what they add is what a caller that owns
// both passes can use: any L2 (with a staged bias; the C ABI takes multiples of 8), a host mirror of the status
// word, a forward pass without statistics, and the whole backward pass (preprocess included) as one call
// planned once.
#pragma once

#include "../../include/fta.h"

#include <cuda_runtime.h>
#include <stddef.h>

#define FTA_NATIVE __attribute__((visibility("default")))

namespace fta {

struct StatusPair {
  int* word;    // device memory
  int* mirror;  // mapped host memory, or nullptr
};

// fta_forward; `lse` may be nullptr (nothing is saved for a backward pass)
FTA_NATIVE int native_forward(const FtaProblem& prob, const FtaTensor5& q, const FtaTensor5& k, const FtaTensor5& v,
                              const FtaTensor4& bias, float sm_scale, const FtaTensor5& o, void* o_resid, float* lse,
                              StatusPair status, cudaStream_t stream);

// fta_mask_bias for any L2, any strides and any alignment of the bias and the mask
FTA_NATIVE int native_mask_bias(const FtaProblem& prob, const FtaTensor4& bias, const uint8_t* key_mask, void* out,
                                cudaStream_t stream);

// What fta_backward and fta_bwd_preprocess need in scratch memory for `prob`, planned once per call
struct BackwardPlan {
  int nplanes;
  size_t workspace_bytes;  // of fta_backward
  size_t delta_bytes;      // of fta_bwd_preprocess's output
};
FTA_NATIVE int native_backward_plan(const FtaProblem& prob, BackwardPlan* plan);

// fta_bwd_preprocess + fta_backward; `workspace`: plan.workspace_bytes (256-byte aligned) followed by
// plan.delta_bytes
FTA_NATIVE int native_backward(const FtaProblem& prob, const BackwardPlan& plan, const FtaTensor5& q,
                               const FtaTensor5& k, const FtaTensor5& v, const FtaTensor4& bias, const FtaTensor5& o,
                               const void* o_resid, const FtaTensor5& dout, const float* lse, float sm_scale,
                               const FtaTensor5& dq, const FtaTensor5& dk, const FtaTensor5& dv, float* dbias_f32,
                               void* dbias_cast, void* workspace, StatusPair status, cudaStream_t stream);

}  // namespace fta
