// Host path of the public operators: from torch tensors to the C ABI and back, with the autograd node, in one native call.
//
// What bounds a small call is not the GPU: building the argument block in Python, the ctypes transition and a Python
// autograd.Function cost 49 us per forward and about 210 us per forward + backward (measured on 200-token and 1243-token
// calls), several times the kernels' own time.  Everything between the public Python function and the launches is
// therefore here.  The kernels stay behind the C ABI (include/sb_b200.h); nothing in this file computes.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <atomic>
#include <mutex>

#include "../../include/sb_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using torch::autograd::variable_list;

std::atomic<long long> g_launches{0};   // process-wide: the backward runs on autograd's threads

// What one call is, apart from its tensors.
struct Call {
  bool fixed, fused, leading_zero;
  int32_t max_seqlen, attend_current, flags;
  float scale;
};

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return SB_DTYPE_F32;
    case at::kBFloat16: return SB_DTYPE_BF16;
    case at::kHalf: return SB_DTYPE_F16;
    default: TORCH_CHECK_VALUE(false, "unsupported dtype ", t);
  }
  return -1;
}

// One int32[4] status word per device, written by kernels that find a problem; lives as long as the process.
Tensor status_word(int device) {
  static std::mutex mu;
  static std::array<Tensor, 64> words;
  std::lock_guard<std::mutex> guard(mu);
  TORCH_CHECK(device >= 0 && device < (int)words.size(), "device ordinal ", device, " not supported");
  Tensor &w = words[device];
  if (!w.defined()) w = at::zeros({4}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
  return w;
}
int32_t *status_ptr(int device) {
  static std::array<std::atomic<int32_t *>, 64> ptrs{};
  if (device < 0 || device >= (int)ptrs.size()) return static_cast<int32_t *>(status_word(device).data_ptr());
  int32_t *p = ptrs[device].load(std::memory_order_acquire);
  if (p == nullptr) {
    p = static_cast<int32_t *>(status_word(device).data_ptr());
    ptrs[device].store(p, std::memory_order_release);
  }
  return p;
}

// Unit innermost stride, 16-byte aligned base and outer strides (what TMA and the vector accesses need) and, for the types
// the tensor maps are for, no axis that repeats its elements (an expanded tensor: a key head shared by several heads, the
// gradient of a sum); copies only where that does not hold, so that forward and backward take the same kernels whatever
// the strides.  Rows that are no multiple of 16 bytes take the CUDA-core kernels: any stride will do.
Tensor tma_ready(const Tensor &t) {
  const int64_t mult = 16 / t.element_size(), nd = t.dim();
  bool ok = t.stride(-1) == 1;
  if (ok && t.size(-1) % mult == 0) {
    ok = reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
    for (int64_t i = 0; ok && i + 1 < nd; ++i) ok = t.size(i) == 1 || (t.stride(i) % mult == 0 && (t.stride(i) > 0 || mult < 8));
  }
  return ok ? t : t.contiguous();
}

Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor &like) {
  return at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt);
}
// Same sizes and, for a dense tensor (permuted views included), the same strides: torch.empty_like without the dispatcher.
Tensor empty_as(const Tensor &t) {
  if (t.is_non_overlapping_and_dense()) return at::detail::empty_strided_cuda(t.sizes(), t.strides(), t.scalar_type(), t.device());
  return at::empty_like(t);
}

SbTensor arg(const Tensor &t, bool fixed) {
  return fixed ? SbTensor{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)} : SbTensor{t.data_ptr(), 0, t.stride(0), t.stride(1)};
}

void check_inputs(const Tensor &q, const Tensor &k, const Tensor &v, const std::optional<Tensor> &cu, const Call &c) {
  TORCH_CHECK_VALUE(q.is_cuda(), "stick-breaking attention runs on a CUDA device only (no CPU path)");
  dtype_code(q.scalar_type());
  TORCH_CHECK_VALUE(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "q, k, v must share a dtype");
  TORCH_CHECK_VALUE(q.sizes() == k.sizes() && q.sizes() == v.sizes(), "q, k, v must share a shape");
  TORCH_CHECK_VALUE(q.device() == k.device() && q.device() == v.device(), "q, k, v must share a device");
  TORCH_CHECK_VALUE(q.dim() == (c.fixed ? 4 : 3), "expected (B,H,T,d) for sb_attn and (H,T,d) for sb_attn_varlen");
  if (!c.fixed) {
    TORCH_CHECK_VALUE(cu->is_cuda() && cu->dim() == 1, "cu_seqlens must be a 1-D CUDA tensor");
    TORCH_CHECK_VALUE(cu->device() == q.device(), "cu_seqlens must be on the device of q, k, v");
    TORCH_CHECK_VALUE(cu->scalar_type() == at::kInt || cu->scalar_type() == at::kLong, "cu_seqlens must be int32 or int64");
    TORCH_CHECK_VALUE(cu->numel() <= 1 || cu->stride(0) == 1, "cu_seqlens must be contiguous");
  }
}

// The backward's own inputs: the kernels go by the shapes of q.
void check_gradients(const Tensor &dout, const Tensor &drem, const Tensor &q) {
  if (dout.defined())
    TORCH_CHECK_VALUE(dout.device() == q.device() && dout.sizes() == q.sizes(), "the gradient of o must have the shape and device of q");
  if (drem.defined())
    TORCH_CHECK_VALUE(drem.device() == q.device() && drem.numel() * q.size(-1) == q.numel(),
                      "the gradient of rem must have one value per row of q, on its device");
}
void check_log_rem(const Tensor &log_rem, const Tensor &q) {
  TORCH_CHECK_VALUE(log_rem.scalar_type() == at::kDouble && log_rem.is_contiguous() && log_rem.device() == q.device() &&
                        log_rem.numel() * q.size(-1) == q.numel(),
                    "log_rem must be what the forward returned: fp64, contiguous, one value per row of q");
}

void fill(SbParams &p, const Tensor &q, const Tensor &k, const Tensor &v, const std::optional<Tensor> &cu, const Call &c) {
  memset(&p, 0, sizeof(p));
  p.struct_bytes = (int32_t)sizeof(SbParams);
  p.dtype = dtype_code(q.scalar_type());
  const int64_t nd = q.dim();
  p.batch = c.fixed ? (int32_t)q.size(0) : 1;
  p.heads = (int32_t)q.size(nd - 3);
  p.tokens = q.size(nd - 2);
  p.head_dim = (int32_t)q.size(nd - 1);
  if (!c.fixed) {   // the C ABI takes the sequence ends only
    const int64_t skip = c.leading_zero ? 1 : 0;
    p.num_seq = (int32_t)(cu->numel() - skip);
    p.cu_seqlens = static_cast<const char *>(cu->data_ptr()) + skip * cu->element_size();
    p.cu_seqlens_int64 = cu->scalar_type() == at::kLong;
  }
  p.max_seqlen = c.max_seqlen;
  p.attend_current = c.attend_current;
  p.logit_scale = c.scale;
  p.flags = c.flags | (c.leading_zero && !c.fixed ? SB_FLAG_CHECK_LEADING_ZERO : 0) | (c.fused ? SB_FLAG_FUSE_REM_V : 0);
  p.q = arg(q, c.fixed);
  p.k = arg(k, c.fixed);
  p.v = arg(v, c.fixed);
}

// An error the library reported; reaches Python as _cabi.SbError (see set_python_error).
struct LibraryError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
[[noreturn]] void raise_library_error(const char *what, int rc) {
  if (rc < 0) throw LibraryError(std::string("invalid parameters: ") + sb_last_error());
  throw LibraryError(std::string(what) + " failed with status " + std::to_string(rc) + ": " + sb_last_error());
}
void set_python_error(const LibraryError &e) {   // with the GIL held
  const py::object type = py::module_::import("stickbreaking_attention_b200._cabi").attr("SbError");
  PyErr_SetString(type.ptr(), e.what());
}

size_t workspace_bytes(const SbParams &p, bool backward) {
  const size_t need = sb_workspace_bytes(&p, backward);
  if (need == (size_t)-1) raise_library_error("sb_workspace_bytes", -1);
  return need < 256 ? 256 : need;
}

void launch(SbParams &p, bool backward, char *workspace, size_t bytes, const Tensor &q) {
  p.workspace = workspace;
  p.workspace_bytes = bytes;
  p.status = status_ptr(q.get_device());
  void *stream = at::cuda::getCurrentCUDAStream(q.get_device()).stream();
  const int rc = backward ? sb_bwd(&p, stream) : sb_fwd(&p, stream);
  if (rc != SB_OK) raise_library_error(backward ? "sb_bwd" : "sb_fwd", rc);
  g_launches.fetch_add(sb_last_launch_count(), std::memory_order_relaxed);
}

// `state`: what the backward needs, one fp64 buffer -- log_rem (batch, heads, tokens) and, where the call keeps them, the
// int32 tile starts (batch * heads, ceil(tokens / 32)) behind it.
struct Forward { Tensor out, rem, state; };

void attach_state(SbParams &p, double *state, bool tile_starts) {
  const int64_t rows = (int64_t)p.batch * p.heads;
  p.log_rem = state;
  if (tile_starts) {
    p.tile_start = reinterpret_cast<int32_t *>(state + rows * p.tokens);
    p.tile_start_stride = (p.tokens + 31) / 32;
  }
}
int64_t state_doubles(const SbParams &p) {
  const int64_t rows = (int64_t)p.batch * p.heads;
  return rows * p.tokens + (rows * ((p.tokens + 31) / 32) + 1) / 2;
}

// kLogRem: log_rem over all keys, as a tensor of the rows' shape; kState: the operator's own saved state; kNothing: no
// backward will come, and the state is scratch like the rest and shares its allocation.
enum class Keep { kNothing, kState, kLogRem };

Forward run_forward(const Tensor &q_in, const Tensor &k_in, const Tensor &v_in, const std::optional<Tensor> &cu, const Call &c,
                    Keep keep) {
  check_inputs(q_in, k_in, v_in, cu, c);
  c10::cuda::CUDAGuard guard(q_in.device());
  const Tensor q = tma_ready(q_in), k = tma_ready(k_in), v = tma_ready(v_in);
  Forward f;
  f.out = empty_as(q);
  const auto row_sizes = q.sizes().slice(0, q.dim() - 1);
  f.rem = empty_cuda(row_sizes, q.scalar_type(), q);
  SbParams p;
  fill(p, q, k, v, cu, c);
  p.o = arg(f.out, c.fixed);
  p.rem = f.rem.data_ptr();
  const size_t ws = (workspace_bytes(p, false) + 255) / 256 * 256;
  size_t bytes = ws;
  if (keep == Keep::kLogRem) f.state = empty_cuda(row_sizes, at::kDouble, q);
  else if (keep == Keep::kState) f.state = empty_cuda({state_doubles(p)}, at::kDouble, q);
  else bytes += sizeof(double) * (size_t)state_doubles(p);
  // freed on return: the caching allocator hands the block out again only behind this stream's work
  const Tensor scratch = empty_cuda({(int64_t)bytes}, at::kByte, q);
  char *base = static_cast<char *>(scratch.data_ptr());
  attach_state(p, f.state.defined() ? static_cast<double *>(f.state.data_ptr()) : reinterpret_cast<double *>(base + ws),
               keep != Keep::kLogRem);
  launch(p, false, base, ws, q);
  return f;
}

std::array<Tensor, 3> run_backward(const Tensor &dout_in, const Tensor &drem_in, const Tensor &q_in, const Tensor &k_in, const Tensor &v_in,
                                   const std::optional<Tensor> &cu, const Tensor &state, bool tile_starts, const Call &c) {
  check_inputs(q_in, k_in, v_in, cu, c);
  check_gradients(dout_in, drem_in, q_in);
  c10::cuda::CUDAGuard guard(q_in.device());
  const Tensor q = tma_ready(q_in), k = tma_ready(k_in), v = tma_ready(v_in);
  const Tensor dout = dout_in.defined() ? tma_ready(dout_in.scalar_type() == q.scalar_type() ? dout_in : dout_in.to(q.scalar_type()))
                                        : at::zeros_like(q);
  Tensor drem;
  if (drem_in.defined()) drem = drem_in.to(q.scalar_type()).contiguous();
  else if (!c.fused) drem = at::zeros(q.sizes().slice(0, q.dim() - 1), q.options());
  const Tensor dq = empty_as(q), dk = empty_as(k), dv = empty_as(v);
  SbParams p;
  fill(p, q, k, v, cu, c);
  attach_state(p, static_cast<double *>(state.data_ptr()), tile_starts);
  p.d_o = arg(dout, c.fixed);
  p.d_rem = drem.defined() ? drem.data_ptr() : nullptr;
  p.dq = arg(dq, c.fixed);
  p.dk = arg(dk, c.fixed);
  p.dv = arg(dv, c.fixed);
  size_t bytes = workspace_bytes(p, true);
  Tensor scratch;
  try {
    scratch = empty_cuda({(int64_t)bytes}, at::kByte, q);
  } catch (const c10::OutOfMemoryError &) {
    // the stored-tiles backward asks for up to the scratch budget; where that does not fit, the recomputing kernels and
    // their few MB do the same work instead of failing
    if (p.flags & SB_FLAG_BWD_RECOMPUTE) throw;
    p.flags |= SB_FLAG_BWD_RECOMPUTE;
    bytes = workspace_bytes(p, true);
    scratch = empty_cuda({(int64_t)bytes}, at::kByte, q);
  }
  launch(p, true, static_cast<char *>(scratch.data_ptr()), bytes, q);
  return {dq, dk, dv};
}

// The operator's node in the autograd graph (reference: StickBreakingAttention.backward, sb_varlen/__init__.py:48-68).
struct StickBreakingAttentionBackward : public torch::autograd::Node {
  torch::autograd::SavedVariable q, k, v, state, cu;
  Call call{};
  bool released = false;

  std::string name() const override { return "StickBreakingAttentionBackward"; }
  void release_variables() override {
    q.reset_data(); k.reset_data(); v.reset_data(); state.reset_data(); cu.reset_data();
    released = true;
  }
  variable_list apply(variable_list &&grads) override {
    TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
    // Saved-tensor hooks run here and may record operations of their own (activation checkpointing runs the forward again).
    const Tensor sq = q.unpack(), sk = k.unpack(), sv = v.unpack(), saved = state.unpack();
    std::optional<Tensor> ends;
    if (!call.fixed) ends = cu.unpack();
    at::AutoDispatchBelowADInplaceOrView below;   // plain tensors from here on: conversions and copies record nothing
    std::array<Tensor, 3> g;
    try {
      g = run_backward(grads[0], grads.size() > 1 ? grads[1] : Tensor(), sq, sk, sv, ends, saved, true, call);
    } catch (const LibraryError &e) {   // on an autograd thread: the exception keeps its Python type on its way to the caller
      py::gil_scoped_acquire gil;
      set_python_error(e);
      python_error err;
      err.persist();
      throw std::move(err);
    }
    variable_list out(3);
    for (size_t i = 0; i < 3; ++i)
      if (task_should_compute_output(i)) out[i] = std::move(g[i]);
    return out;
  }
};

Call make_call(bool fixed, std::optional<int64_t> max_seqlens, double scale, bool attend_current, bool leading_zero, bool fused,
               int64_t flags) {
  Call c;
  c.fixed = fixed;
  c.fused = fused;
  c.leading_zero = leading_zero;
  c.max_seqlen = (int32_t)max_seqlens.value_or(0);
  c.attend_current = attend_current;
  c.flags = (int32_t)flags;
  c.scale = (float)scale;
  return c;
}

// The differentiable operator: (out, rem), or (out,) with out = o + rem * v.
variable_list attention(const Tensor &q, const Tensor &k, const Tensor &v, const std::optional<Tensor> &cu,
                        std::optional<int64_t> max_seqlens, double scale, bool attend_current, bool leading_zero, bool fused,
                        int64_t flags) {
  const Call c = make_call(!cu.has_value(), max_seqlens, scale, attend_current, leading_zero, fused, flags);
  for (const Tensor *t : {&q, &k, &v})
    TORCH_CHECK_NOT_IMPLEMENTED(!t->_fw_grad(0).defined(), "stick-breaking attention has no forward-mode derivative");
  const bool grad = torch::autograd::compute_requires_grad(q, k, v);
  Forward f;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    f = run_forward(q, k, v, cu, c, grad ? Keep::kState : Keep::kNothing);
  }
  if (grad) {
    auto node = std::shared_ptr<StickBreakingAttentionBackward>(new StickBreakingAttentionBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
    node->call = c;
    node->q = torch::autograd::SavedVariable(q, false);
    node->k = torch::autograd::SavedVariable(k, false);
    node->v = torch::autograd::SavedVariable(v, false);
    node->state = torch::autograd::SavedVariable(f.state, false);
    if (cu.has_value()) node->cu = torch::autograd::SavedVariable(*cu, false);
    torch::autograd::set_history(f.out, node);
    if (!fused) torch::autograd::set_history(f.rem, node);
  }
  if (fused) return {f.out};
  return {f.out, f.rem};
}

// The launchers: no autograd, the saved state handed out and back in.
std::tuple<Tensor, Tensor, Tensor> forward(const Tensor &q, const Tensor &k, const Tensor &v, const std::optional<Tensor> &cu,
                                           std::optional<int64_t> max_seqlens, double scale, bool attend_current, bool leading_zero,
                                           bool fused, int64_t flags) {
  at::AutoDispatchBelowADInplaceOrView below;
  Forward f = run_forward(q, k, v, cu, make_call(!cu.has_value(), max_seqlens, scale, attend_current, leading_zero, fused, flags),
                          Keep::kLogRem);
  return {f.out, f.rem, f.state};
}
std::tuple<Tensor, Tensor, Tensor> backward(const Tensor &dout, const std::optional<Tensor> &drem, const Tensor &q, const Tensor &k,
                                            const Tensor &v, const std::optional<Tensor> &cu, std::optional<int64_t> max_seqlens,
                                            const Tensor &log_rem, double scale, bool attend_current, bool leading_zero, bool fused,
                                            int64_t flags) {
  at::AutoDispatchBelowADInplaceOrView below;
  check_log_rem(log_rem, q);
  std::array<Tensor, 3> g = run_backward(dout, drem.value_or(Tensor()), q, k, v, cu, log_rem, false,
                                         make_call(!cu.has_value(), max_seqlens, scale, attend_current, leading_zero, fused, flags));
  return {g[0], g[1], g[2]};
}

}  // namespace

PYBIND11_MODULE(_sb_torch, m) {
  py::register_exception_translator([](std::exception_ptr e) {
    try {
      if (e) std::rethrow_exception(e);
    } catch (const LibraryError &err) {
      set_python_error(err);
    }
  });
  m.def("attention", &attention, py::call_guard<py::gil_scoped_release>());
  m.def("forward", &forward, py::call_guard<py::gil_scoped_release>());
  m.def("backward", &backward, py::call_guard<py::gil_scoped_release>());
  m.def("tma_ready", &tma_ready);
  m.def("status_word", &status_word, py::call_guard<py::gil_scoped_release>());
  m.def("launches", [] { return g_launches.load(); });
}
