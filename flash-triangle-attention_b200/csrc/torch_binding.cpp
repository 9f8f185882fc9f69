// The torch side of attention(): argument checks, allocations, launches and the autograd node, natively.
//
// A call of a small problem is bound by host time: with ctypes, a Python autograd.Function and one Python
// allocation per buffer, a forward call took 63 us and a training step 253 us at B1 H4 L64 D32 on a B200
// host, of which the kernels are a fraction. Here a call is one C++ function, backward runs on the autograd
// thread without the interpreter, and scratch memory is one allocation per pass.
//
// Everything is launched through libfta.so (native_api.h); nothing here is a fallback for it.
#include "native_api.h"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <cstdio>
#include <mutex>

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------------
// per-device status word and its mirror (the tensors belong to the Python module)
// ------------------------------------------------------------------------------------------------
struct DeviceStatus {
  at::Tensor word, mirror;
  volatile int* host = nullptr;  // the mirror, as the host reads it
  fta::StatusPair pair{nullptr, nullptr};
};
constexpr int kMaxDevices = 64;
DeviceStatus g_status[kMaxDevices];
bool g_save_o_residual = true;

at::Tensor g_last_dbias_f32;  // of the most recent backward call, any thread
std::mutex g_last_mu;

// What was there before dies after the lock is given back: if Python has seen that tensor, its end takes the
// interpreter's lock, which a thread that waits for ours may hold.
void set_last_dbias_f32(at::Tensor t) {
  std::lock_guard<std::mutex> lock(g_last_mu);
  std::swap(t, g_last_dbias_f32);
}
std::optional<at::Tensor> last_dbias_f32() {
  std::lock_guard<std::mutex> lock(g_last_mu);
  if (!g_last_dbias_f32.defined()) return std::nullopt;
  return g_last_dbias_f32;
}

// Called with a device index the first time attention() meets that device: has the Python module create
// and register its status word. Never released (it lives as long as the interpreter).
py::object* g_make_status = nullptr;

void set_status(int64_t device, at::Tensor word, at::Tensor mirror) {
  TORCH_CHECK(device >= 0 && device < kMaxDevices, "device index out of range");
  DeviceStatus& s = g_status[device];
  s.word = word;
  s.mirror = mirror;
  s.host = mirror.data_ptr<int>();
  s.pair = {word.data_ptr<int>(), mirror.data_ptr<int>()};
}

[[noreturn]] void raise_status(DeviceStatus& s, int code) {
  s.word.zero_();
  s.mirror.zero_();
  char msg[160];
  std::snprintf(msg, sizeof(msg),
                "flash_tt_attn: device status 0x%x (a bounded device-side wait ran out in an earlier call; its "
                "outputs are incomplete)", code);
  throw std::runtime_error(msg);
}

// An earlier launch's failed wait, seen through the mirror without touching the stream.
DeviceStatus& status_of(c10::DeviceIndex device) {
  TORCH_CHECK(device >= 0 && device < kMaxDevices, "device index out of range");
  DeviceStatus& s = g_status[device];
  TORCH_CHECK(s.host != nullptr, "flash_tt_attn: no status word registered for this device");
  const int code = *s.host;
  if (C10_UNLIKELY(code != 0)) raise_status(s, code);
  return s;
}

// The same for the launches just made: waits for them.
void check_status_now(const c10::Device& device) {
  const c10::cuda::CUDAGuard guard(device);
  DeviceStatus& s = status_of(device.index());
  if (const int code = s.word.item<int>()) raise_status(s, code);
}

void ensure_status(const c10::Device& device) {
  const int i = device.index();
  TORCH_CHECK(i >= 0 && i < kMaxDevices, "device index out of range");
  if (C10_UNLIKELY(g_status[i].host == nullptr)) (*g_make_status)(i);
}

// FtaError, from whichever thread this is
void check_rc(int rc, const char* where) {
  if (C10_LIKELY(rc == FTA_OK)) return;
  py::gil_scoped_acquire gil;
  py::module_::import("_cabi").attr("check")(rc, where);
}

// ------------------------------------------------------------------------------------------------
// tensors as the kernels take them
// ------------------------------------------------------------------------------------------------
// Unit stride in the last dimension, the others positive multiples of 8 elements, 16-byte aligned: addressed
// in place. (The stride of a dimension of size 1 carries no meaning.) Anything else is copied.
bool addressable(const at::Tensor& t) {
  const auto sizes = t.sizes();
  const auto strides = t.strides();
  const int n = static_cast<int>(sizes.size());
  if (strides[n - 1] != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return false;
  for (int i = 0; i < n - 1; ++i)
    if (sizes[i] > 1 && (strides[i] <= 0 || strides[i] % 8 != 0)) return false;
  return true;
}
at::Tensor dense(const at::Tensor& t) {
  return addressable(t) ? t : t.clone(at::MemoryFormat::Contiguous);
}

template <typename View, int N>
View view_of(const at::Tensor& t) {
  View v;
  v.ptr = t.data_ptr();
  const auto sizes = t.sizes();
  const auto strides = t.strides();
  int64_t span = 1;  // a valid stride for dimensions of size 1
  for (int i = N - 1; i >= 0; --i) {
    v.stride[i] = (sizes[i] > 1 || i == N - 1) ? strides[i] : (span + 7) / 8 * 8;
    const int64_t s = v.stride[i] * sizes[i];
    span = s > span ? s : span;
  }
  return v;
}
FtaTensor5 v5(const at::Tensor& t) { return view_of<FtaTensor5, 5>(t); }
FtaTensor4 v4(const at::Tensor& t) { return view_of<FtaTensor4, 4>(t); }

int64_t padded(int64_t l2) { return (l2 + 127) / 128 * 128; }

FtaProblem problem_of(const at::Tensor& q) {
  FtaProblem p;
  p.B = static_cast<int32_t>(q.size(0));
  p.H = static_cast<int32_t>(q.size(1));
  p.L1 = static_cast<int32_t>(q.size(2));
  p.L2 = static_cast<int32_t>(q.size(3));
  p.D = static_cast<int32_t>(q.size(4));
  p.dtype = q.scalar_type() == at::kBFloat16 ? FTA_BF16 : FTA_FP16;
  return p;
}

at::Tensor bytes_like(const at::Tensor& q, int64_t n) { return at::empty({n}, q.options().dtype(at::kByte)); }

int64_t align256(int64_t x) { return (x + 255) & ~int64_t(255); }

// ------------------------------------------------------------------------------------------------
// the two passes
// ------------------------------------------------------------------------------------------------
struct ForwardOut {
  at::Tensor q, k, v, bias;  // as the kernels read them (bias: the padded, masked copy where one is needed)
  at::Tensor o;
  at::Tensor saved;          // statistics and, with bf16, the rounding residual of O; undefined without `keep`
};

// `keep`: a backward pass will follow
ForwardOut run_forward(const at::Tensor& q_, const at::Tensor& k_, const at::Tensor& v_, const at::Tensor& bias_,
                       double sm_scale, const std::optional<at::Tensor>& key_mask, bool keep) {
  const c10::cuda::CUDAGuard guard(q_.device());
  DeviceStatus& st = status_of(q_.device().index());
  ForwardOut r;
  r.q = dense(q_);
  r.k = dense(k_);
  r.v = dense(v_);
  const FtaProblem prob = problem_of(q_);
  const int64_t l2p = padded(prob.L2);
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
  r.o = at::empty(q_.sizes(), q_.options().memory_format(at::MemoryFormat::Contiguous));
  if (key_mask.has_value() || l2p != prob.L2) {
    // Ragged L2 and / or a boolean key mask: only this bias-sized tensor is staged (whole 128-blocks,
    // -inf on padding and masked keys); q, k, v are read in place.
    at::Tensor km;
    if (key_mask.has_value()) km = key_mask->to(q_.device()).contiguous();
    r.bias = at::empty({prob.B, prob.H, l2p, l2p}, q_.options());
    FtaTensor4 b4;
    b4.ptr = bias_.data_ptr();
    for (int i = 0; i < 4; ++i) b4.stride[i] = bias_.stride(i);
    check_rc(fta::native_mask_bias(prob, b4, km.defined() ? static_cast<const uint8_t*>(km.data_ptr()) : nullptr,
                                   r.bias.data_ptr(), stream), "fta_mask_bias");
  } else {
    r.bias = dense(bias_);
  }
  float* lse = nullptr;
  void* resid = nullptr;
  if (keep) {
    const int64_t stats = align256(int64_t(3) * prob.B * prob.H * prob.L1 * l2p * 4);
    const bool want_resid = g_save_o_residual && prob.dtype == FTA_BF16;
    r.saved = bytes_like(q_, stats + (want_resid ? r.o.numel() * 2 : 0));
    lse = static_cast<float*>(r.saved.data_ptr());
    if (want_resid) resid = static_cast<uint8_t*>(r.saved.data_ptr()) + stats;
  }
  check_rc(fta::native_forward(prob, v5(r.q), v5(r.k), v5(r.v), v4(r.bias), static_cast<float>(sm_scale), v5(r.o), resid,
                               lse, st.pair, stream), "fta_forward");
  return r;
}

struct BackwardOut {
  at::Tensor dq, dk, dv, dbias, dbias_f32;
};

// `cast`: also round dBias to the bias dtype (not when it is summed over a process group first)
BackwardOut run_backward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                         const at::Tensor& o, const at::Tensor& saved, const at::Tensor& dout_, double sm_scale,
                         bool cast) {
  const c10::cuda::CUDAGuard guard(q.device());
  DeviceStatus& st = status_of(q.device().index());
  const at::Tensor dout = dense(dout_);
  const FtaProblem prob = problem_of(q);
  const int64_t l2p = padded(prob.L2);
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
  const int64_t stats = align256(int64_t(3) * prob.B * prob.H * prob.L1 * l2p * 4);
  const void* resid = saved.numel() > stats ? static_cast<const uint8_t*>(saved.data_ptr()) + stats : nullptr;
  fta::BackwardPlan plan;
  check_rc(fta::native_backward_plan(prob, &plan), "fta_backward");
  const at::Tensor ws = bytes_like(q, static_cast<int64_t>(plan.workspace_bytes + plan.delta_bytes));
  BackwardOut r;
  const auto dense_opts = q.options().memory_format(at::MemoryFormat::Contiguous);
  r.dq = at::empty(q.sizes(), dense_opts);
  r.dk = at::empty(q.sizes(), dense_opts);
  r.dv = at::empty(q.sizes(), dense_opts);
  r.dbias = at::empty({prob.B, prob.H, prob.L2, prob.L2}, q.options());
  r.dbias_f32 = at::empty({prob.B, prob.H, prob.L2, prob.L2}, q.options().dtype(at::kFloat));
  check_rc(fta::native_backward(prob, plan, v5(q), v5(k), v5(v), v4(bias), v5(o), resid, v5(dout),
                                static_cast<const float*>(saved.data_ptr()), static_cast<float>(sm_scale), v5(r.dq),
                                v5(r.dk), v5(r.dv), r.dbias_f32.data_ptr<float>(), cast ? r.dbias.data_ptr() : nullptr,
                                ws.data_ptr(), st.pair, stream), "fta_backward");
  set_last_dbias_f32(r.dbias_f32);
  return r;
}

struct Attention : public torch::autograd::Function<Attention> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                            const at::Tensor& bias, double sm_scale, const std::optional<at::Tensor>& key_mask, bool debug) {
    ForwardOut r = run_forward(q, k, v, bias, sm_scale, key_mask, true);
    ctx->save_for_backward({r.q, r.k, r.v, r.bias, r.o, r.saved});
    ctx->saved_data["sm_scale"] = sm_scale;
    if (debug) ctx->saved_data["debug"] = true;
    return r.o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    TORCH_CHECK(grads[0].scalar_type() == s[0].scalar_type(), "the gradient of O must have O's dtype");
    BackwardOut r = run_backward(s[0], s[1], s[2], s[3], s[4], s[5], grads[0], ctx->saved_data["sm_scale"].toDouble(), true);
    if (C10_UNLIKELY(ctx->saved_data.count("debug") != 0)) check_status_now(s[0].device());
    return {r.dq, r.dk, r.dv, r.dbias, at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

void require(bool ok, const char* msg) {
  if (C10_LIKELY(ok)) return;
  PyErr_SetString(PyExc_AssertionError, msg);
  throw py::error_already_set();
}

void check_arguments(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                     const std::optional<at::Tensor>& key_mask) {
  // a trace would record the allocation of O and not the launches that fill it
  require(!torch::jit::tracer::isTracing(), "flash_tt_attn.attention cannot be recorded by torch.jit.trace");
  require(q.dim() == 5 && q.size(4) == k.size(-1) && k.size(-1) == v.size(-1), "q, k, v must be 5-D with one head dimension");
  require(q.size(4) == 32 || q.size(4) == 64, "head dimension must be 32 or 64");
  const auto dt = q.scalar_type();
  require(dt == k.scalar_type() && dt == v.scalar_type() && dt == bias.scalar_type(), "q, k, v and the bias must have one dtype");
  require(dt == at::kHalf || dt == at::kBFloat16, "fp16 or bf16 only");
  require(q.is_cuda(), "flash_tt_attn.attention needs CUDA tensors (there is no CPU path)");
  require(q.sizes() == k.sizes() && q.sizes() == v.sizes(), "q, k, v must have one shape");
  const int64_t l2 = q.size(3);
  require(bias.sizes() == at::IntArrayRef({q.size(0), q.size(1), l2, l2}), "bias must be (B, H, L2, L2)");
  require(k.device() == q.device() && v.device() == q.device() && bias.device() == q.device(), "q, k, v and the bias must be on one device");
  if (key_mask.has_value())
    require(key_mask->scalar_type() == at::kBool && key_mask->sizes() == at::IntArrayRef({q.size(0), l2}), "key_mask: bool (B, L2)");
  ensure_status(q.device());
}

bool has_tangent(const at::Tensor& t) { return t._fw_grad(/*level=*/0).defined(); }

// `debug`: the backward pass waits for its launches and raises if one of them failed
at::Tensor attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                     double sm_scale, const std::optional<at::Tensor>& key_mask, bool debug) {
  check_arguments(q, k, v, bias, key_mask);
  py::gil_scoped_release no_gil;  // as torch's own operators do: an allocation or a full launch queue may wait
  const bool keep = at::GradMode::is_enabled() &&
                    (q.requires_grad() || k.requires_grad() || v.requires_grad() || bias.requires_grad());
  // A forward-mode tangent on any input goes through the autograd function whatever the mode: it has no formula for
  // tangents and says so, where the bare pass would drop them.
  const bool dual = has_tangent(q) || has_tangent(k) || has_tangent(v) || has_tangent(bias);
  if (!keep && !dual) return run_forward(q, k, v, bias, sm_scale, key_mask, false).o;
  return Attention::apply(q, k, v, bias, sm_scale, key_mask, debug);
}

// For the Python autograd node of the sharded call (it puts a collective between the passes).
py::tuple forward_pass(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                       double sm_scale, const std::optional<at::Tensor>& key_mask) {
  check_arguments(q, k, v, bias, key_mask);
  ForwardOut r;
  {
    py::gil_scoped_release no_gil;
    r = run_forward(q, k, v, bias, sm_scale, key_mask, true);
  }
  return py::make_tuple(r.q, r.k, r.v, r.bias, r.o, r.saved);
}
py::tuple backward_pass(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias,
                        const at::Tensor& o, const at::Tensor& saved, const at::Tensor& dout, double sm_scale, bool cast) {
  require(dout.scalar_type() == q.scalar_type(), "the gradient of O must have O's dtype");
  BackwardOut r;
  {
    py::gil_scoped_release no_gil;
    r = run_backward(q, k, v, bias, o, saved, dout, sm_scale, cast);
  }
  return py::make_tuple(r.dq, r.dk, r.dv, r.dbias, r.dbias_f32);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("attention", &attention);
  m.def("forward_pass", &forward_pass);
  m.def("backward_pass", &backward_pass);
  m.def("on_new_device", [](py::object make_status) { g_make_status = new py::object(std::move(make_status)); });
  m.def("set_status", &set_status);
  m.def("set_save_o_residual", [](bool on) { g_save_o_residual = on; });
  m.def("last_dbias_f32", &last_dbias_f32);
  m.def("set_last_dbias_f32", &set_last_dbias_f32);
  // the saved tensor must not outlive the allocator it came from
  py::module_::import("atexit").attr("register")(py::cpp_function([] {
    set_last_dbias_f32(at::Tensor());
    for (auto& s : g_status) s = DeviceStatus();
  }));
}
