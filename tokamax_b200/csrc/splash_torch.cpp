// The host side of a call in native code: reads the tensors' addresses, sizes and strides, allocates the results
// and fills the C ABI's argument structs (include/splash_b200.h), which python did field by field through ctypes.
// forward() takes 12 us and backward() 25 (three launches), launches included; a whole forward pass of 256 tokens went
// from 39 to 21 us, a training step of 2 x 1024 from 176 to 114.  attention() is the autograd function in native code too, for
// calls without segment ids, sinks and a fixed maximum: a whole pass of those two 21.0 -> 16.5 and 118.8 -> 93.1 us.  The checks of
// arguments, the schedules and the autograd function of the other calls are in splash_attention_kernel.py.
#include <torch/csrc/utils/pybind.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>

#include <ATen/ATen.h>
#include <c10/core/DeviceGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <memory>
#include <optional>
#include <tuple>
#include <vector>

#include "../../include/splash_b200.h"

namespace {

// entry points of libsplash_b200.so, as ctypes resolved them
struct Library {
  int (*fwd)(const SplashFwdArgs*, const SplashShards*, void*) = nullptr;
  int (*bwd)(const SplashBwdArgs*, const SplashShards*, void*) = nullptr;
  size_t (*workspace_bytes)(int64_t, int64_t, int64_t) = nullptr;
  size_t (*fused_workspace_bytes)(int64_t, int64_t, int64_t) = nullptr;
} lib;

void bind_library(uintptr_t fwd, uintptr_t bwd, uintptr_t workspace_bytes, uintptr_t fused_workspace_bytes) {
  lib.fwd = reinterpret_cast<decltype(lib.fwd)>(fwd);
  lib.bwd = reinterpret_cast<decltype(lib.bwd)>(bwd);
  lib.workspace_bytes = reinterpret_cast<decltype(lib.workspace_bytes)>(workspace_bytes);
  lib.fused_workspace_bytes = reinterpret_cast<decltype(lib.fused_workspace_bytes)>(fused_workspace_bytes);
}

// `t` if the kernels can read it in place, else a contiguous copy
at::Tensor usable(const at::Tensor& t) {
  TORCH_CHECK(t.dim() == 4, "expected a tensor of rank 4, got rank ", t.dim());
  bool ok = t.stride(3) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  for (int i = 0; i < 3; ++i) ok = ok && t.stride(i) % 8 == 0;
  return ok ? t : t.contiguous();
}

// The kernels follow every address that they are given: each must be one of their own device, that of `q`.
void require_beside(const at::Tensor& t, const at::Tensor& q) {
  TORCH_CHECK(t.device() == q.device(), "expected all tensors on the device of q, ", q.device(), ", got one on ", t.device());
}

SplashTensor describe(const at::Tensor& t, const at::Tensor& q) {
  TORCH_CHECK(t.dim() == 4, "expected a tensor of rank 4, got rank ", t.dim());
  TORCH_CHECK(t.scalar_type() == at::kBFloat16, "expected bfloat16 operands, got ", t.scalar_type());
  require_beside(t, q);
  SplashTensor d{};
  d.data = t.data_ptr();
  d.dtype = SPLASH_BF16;
  for (int i = 0; i < 4; ++i) d.size[i] = t.size(i), d.stride[i] = t.stride(i);
  return d;
}

template <typename T>
T* pointer(const at::Tensor& t, const at::Tensor& q) {
  require_beside(t, q);
  return static_cast<T*>(t.data_ptr());
}
template <typename T>
T* pointer(const std::optional<at::Tensor>& t, const at::Tensor& q) {
  return t.has_value() ? pointer<T>(*t, q) : nullptr;
}

template <typename T>
const T& at_address(uintptr_t a) {
  return *reinterpret_cast<const T*>(a);
}

using Maybe = std::optional<at::Tensor>;

// Gives the interpreter's lock up, where this thread holds it.
class WithoutGil {
  std::optional<pybind11::gil_scoped_release> release_;

 public:
  WithoutGil() {
    if (PyGILState_Check()) release_.emplace();
  }
};

// `sched`, `mask_fn`, `o_peer`: addresses of the structs (o_peer: 0 for none).  Returns the status, the operands as
// the kernel read them, and the results.
std::tuple<int, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor> forward(
    const at::Tensor& q_in, const at::Tensor& k_in, const at::Tensor& v_in, const Maybe& q_seg, const Maybe& kv_seg,
    const Maybe& q_sequence, const Maybe& sinks, const Maybe& max_logit, const at::Tensor& error_record, uintptr_t sched,
    uintptr_t mask_fn, double scale, double mask_value, double soft_cap, int head_shards, int q_shards, uintptr_t o_peer) {
  const at::Tensor q = usable(q_in), k = usable(k_in), v = usable(v_in);
  const int64_t b = q.size(0), hq = q.size(1), sq = q.size(2);
  // (like q, it keeps q's dense stride order, e.g. [B,T,H,D] storage stays [B,T,H,D])
  const at::Tensor o = v.size(3) == q.size(3) ? at::empty_like(q) : at::empty({b, hq, sq, v.size(3)}, q.options());
  const auto f32 = q.options().dtype(at::kFloat);
  const at::Tensor lse = at::empty({b, hq, sq}, f32), max_logits = at::empty({b, hq, sq}, f32);
  SplashFwdArgs a{};
  a.q = describe(q, q);
  a.k = describe(k, q);
  a.v = describe(v, q);
  a.o = describe(o, q);
  a.logsumexp = pointer<float>(lse, q);
  a.max_logits = static_cast<float*>(max_logits.data_ptr());
  a.q_segment_ids = pointer<int32_t>(q_seg, q);
  a.kv_segment_ids = pointer<int32_t>(kv_seg, q);
  a.q_sequence = pointer<int32_t>(q_sequence, q);
  a.sched = at_address<SplashDeviceSchedule>(sched);
  a.mask_fn = at_address<SplashMaskFn>(mask_fn);
  a.scale = (float)scale;
  a.mask_value = (float)mask_value;
  a.error_record = pointer<uint32_t>(error_record, q);
  a.sinks = pointer<float>(sinks, q);
  a.max_logit_value = pointer<float>(max_logit, q);
  a.soft_cap = (float)soft_cap;
  if (o_peer != 0) a.o_peer = at_address<SplashPeerOutput>(o_peer);
  const SplashShards shards{head_shards, q_shards};
  int status;
  {
    const WithoutGil release;
    const c10::OptionalDeviceGuard guard(q.device());
    status = lib.fwd(&a, &shards, c10::cuda::getCurrentCUDAStream(q.device().index()).stream());
  }
  return {status, q, k, v, o, lse, max_logits};
}

// `peers`: addresses of three SplashPeerOutput, or zeros.  Returns the status, the gradients and the workspace.
std::tuple<int, at::Tensor, at::Tensor, at::Tensor, at::Tensor> backward(
    const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& lse,
    const at::Tensor& d_o_in, const Maybe& q_seg, const Maybe& kv_seg, const Maybe& q_sequence, const at::Tensor& error_record,
    uintptr_t sched_dq, uintptr_t sched_dkv, uintptr_t mask_fn, double scale, double soft_cap, bool fused, int head_shards,
    int q_shards, uintptr_t dq_peer, uintptr_t dk_peer, uintptr_t dv_peer) {
  const at::Tensor d_o = usable(d_o_in);
  const at::Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  SplashBwdArgs a{};
  a.q = describe(q, q);
  a.k = describe(k, q);
  a.v = describe(v, q);
  a.o = describe(o, q);
  a.d_o = describe(d_o, q);
  a.dq = describe(dq, q);
  a.dk = describe(dk, q);
  a.dv = describe(dv, q);
  const size_t bytes = (fused ? lib.fused_workspace_bytes : lib.workspace_bytes)(q.size(0), q.size(1), q.size(2));
  const at::Tensor workspace = at::empty({(int64_t)bytes}, q.options().dtype(at::kByte));
  a.flags = fused ? SPLASH_BWD_FUSED_DQ : 0;
  a.logsumexp = pointer<float>(lse, q);
  a.q_segment_ids = pointer<int32_t>(q_seg, q);
  a.kv_segment_ids = pointer<int32_t>(kv_seg, q);
  a.q_sequence = pointer<int32_t>(q_sequence, q);
  a.sched_dq = at_address<SplashDeviceSchedule>(sched_dq);
  a.sched_dkv = at_address<SplashDeviceSchedule>(sched_dkv);
  a.mask_fn = at_address<SplashMaskFn>(mask_fn);
  a.scale = (float)scale;
  a.workspace = workspace.data_ptr();
  a.workspace_bytes = bytes;
  a.error_record = pointer<uint32_t>(error_record, q);
  a.soft_cap = (float)soft_cap;
  if (dq_peer != 0) a.dq_peer = at_address<SplashPeerOutput>(dq_peer);
  if (dk_peer != 0) a.dk_peer = at_address<SplashPeerOutput>(dk_peer);
  if (dv_peer != 0) a.dv_peer = at_address<SplashPeerOutput>(dv_peer);
  const SplashShards shards{head_shards, q_shards};
  int status;
  {
    const WithoutGil release;
    const c10::OptionalDeviceGuard guard(q.device());
    status = lib.bwd(&a, &shards, c10::cuda::getCurrentCUDAStream(q.device().index()).stream());
  }
  return {status, dq, dk, dv, workspace};
}

// The schedules of one kernel object on one device, with the tensors that hold them.
struct Tables {
  SplashDeviceSchedule fwd, dq, dkv;
  std::vector<at::Tensor> held;
  at::Tensor error_record;
  Maybe q_sequence;
  int q_shards;

  Tables(uintptr_t fwd, uintptr_t dq, uintptr_t dkv, std::vector<at::Tensor> held, at::Tensor error_record, Maybe q_sequence,
         int q_shards)
      : fwd(at_address<SplashDeviceSchedule>(fwd)),
        dq(at_address<SplashDeviceSchedule>(dq)),
        dkv(at_address<SplashDeviceSchedule>(dkv)),
        held(std::move(held)),
        error_record(std::move(error_record)),
        q_sequence(std::move(q_sequence)),
        q_shards(q_shards) {}
};

// What the backward of a call needs beside its tensors.
struct Call : torch::CustomClassHolder {
  std::shared_ptr<const Tables> tables;
  SplashMaskFn mask_fn;
  double scale, mask_value, soft_cap;
  bool fused;
  int head_shards;
};

// `_native.check`, held for the life of the process: raises the package's exception for a status that is not zero
PyObject* check_status = nullptr;

// From a thread that does not hold the interpreter's lock, as python's own exception.
void raise_status(int status, const char* what) {
  pybind11::gil_scoped_acquire gil;
  Py_XDECREF(PyObject_CallFunction(check_status, "is", status, what));
  python_error error;
  error.persist();
  throw std::move(error);
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// As _SplashFunction of splash_attention_kernel.py.
struct Attention : torch::autograd::Function<Attention> {
  static variable_list forward(AutogradContext* ctx, const at::Tensor& q_in, const at::Tensor& k_in, const at::Tensor& v_in,
                               const c10::intrusive_ptr<Call>& call) {
    const Tables& t = *call->tables;
    auto [status, q, k, v, o, lse, max_logits] = ::forward(
        q_in, k_in, v_in, {}, {}, t.q_sequence, {}, {}, t.error_record, reinterpret_cast<uintptr_t>(&t.fwd),
        reinterpret_cast<uintptr_t>(&call->mask_fn), call->scale, call->mask_value, call->soft_cap, call->head_shards, t.q_shards, 0);
    if (status != 0) raise_status(status, "splash_fwd");
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["call"] = c10::IValue::make_capsule(call);
    ctx->mark_non_differentiable({lse, max_logits});
    ctx->set_materialize_grads(false);  // no zeros made up for the gradients of lse and max_logits
    return {o, lse, max_logits};
  }

  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list saved = ctx->get_saved_variables();
    const at::Tensor &q = saved[0], &k = saved[1], &v = saved[2], &o = saved[3], &lse = saved[4];
    const auto call = c10::static_intrusive_pointer_cast<Call>(ctx->saved_data["call"].toCapsule());
    const Tables& t = *call->tables;
    const at::Tensor d_o = grads[0].defined() ? grads[0] : at::zeros_like(o);  // an undefined gradient of o is zero
    auto [status, dq, dk, dv, workspace] = ::backward(
        q, k, v, o, lse, d_o, {}, {}, t.q_sequence, t.error_record, reinterpret_cast<uintptr_t>(&t.dq),
        reinterpret_cast<uintptr_t>(&t.dkv), reinterpret_cast<uintptr_t>(&call->mask_fn), call->scale, call->soft_cap,
        call->fused, call->head_shards, t.q_shards, 0, 0, 0);
    if (status != 0) raise_status(status, "splash_bwd");
    return {dq, dk, dv, at::Tensor()};
  }
};

// Output, logsumexp and max_logits, the output differentiable.
std::tuple<at::Tensor, at::Tensor, at::Tensor> attention(const std::shared_ptr<Tables>& tables, const at::Tensor& q,
                                                         const at::Tensor& k, const at::Tensor& v, uintptr_t mask_fn,
                                                         double scale, double mask_value, double soft_cap, bool fused,
                                                         int head_shards) {
  auto call = c10::make_intrusive<Call>();
  call->tables = tables;
  call->mask_fn = at_address<SplashMaskFn>(mask_fn);
  call->scale = scale;
  call->mask_value = mask_value;
  call->soft_cap = soft_cap;
  call->fused = fused;
  call->head_shards = head_shards;
  variable_list out;
  {
    pybind11::gil_scoped_release release;
    out = Attention::apply(q, k, v, call);
  }
  return {out[0], out[1], out[2]};
}

}  // namespace

PYBIND11_MODULE(_splash_torch, m) {
  m.def("bind_library", &bind_library);
  m.def("forward", torch::wrap_pybind_function(forward));
  m.def("backward", torch::wrap_pybind_function(backward));
  m.def("bind_check", [](pybind11::object check) { check_status = check.release().ptr(); });
  pybind11::class_<Tables, std::shared_ptr<Tables>>(m, "Tables")
      .def(pybind11::init<uintptr_t, uintptr_t, uintptr_t, std::vector<at::Tensor>, at::Tensor, Maybe, int>());
  m.def("attention", torch::wrap_pybind_function(attention));
}
