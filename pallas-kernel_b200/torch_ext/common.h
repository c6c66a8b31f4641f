// What the host paths share: errors, allocations on the first tensor's GPU and stream, autograd nodes.
#pragma once
#include <torch/extension.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <optional>
#include <vector>

#include "tops_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

namespace tops_torch {


inline PyObject* g_module = nullptr;   // tops_b200._lib: TopsError, CHECK_DEVICE

// Raises a Python exception, also from a node that runs on an autograd thread without the GIL: the engine carries a
// python_error over to the thread that called backward().
[[noreturn]] inline void raise_py(PyObject* type, const std::string& text) {
  const bool held = PyGILState_Check();
  py::gil_scoped_acquire gil;
  PyErr_SetString(type, text.c_str());
  if (held) throw py::error_already_set();
  python_error e;
  e.persist();
  throw e;
}
[[noreturn]] inline void raise_tops(const std::string& text) {
  py::gil_scoped_acquire gil;
  raise_py(py::handle(g_module).attr("TopsError").ptr(), text);
}
[[noreturn]] inline void raise_assertion(const std::string& text) { raise_py(PyExc_AssertionError, text); }
inline void check(int rc, const char* what) {
  if (rc == 0) return;
  std::string text = std::string(what) + ": " + tops_b200_strerror(rc) + " (code " + std::to_string(rc) + ")";
  if (rc == TOPS_E_CUDA) {
    char buf[256] = "";
    tops_b200_last_cuda_error(buf, sizeof buf);
    text += std::string(" [") + buf + "]";
  }
  raise_tops(text);
}
inline void check_device_word(const char* what) {
  {
    py::gil_scoped_acquire gil;
    if (!py::handle(g_module).attr("CHECK_DEVICE").cast<bool>()) return;
  }
  int code = 0;
  check(tops_b200_device_error(&code), "device_error");
  if (code == 0) return;
  tops_b200_device_error_reset();
  raise_tops(std::string(what) + ": a kernel gave up on a bounded device-side wait (code " + std::to_string(code) +
             "); its outputs are invalid");
}

inline int code_of(at::ScalarType t) {
  if (t == at::kFloat) return TOPS_F32;
  if (t == at::kBFloat16) return TOPS_BF16;
  if (t == at::kHalf) return TOPS_F16;
  raise_assertion("unsupported dtype (fp32, bf16, fp16 only)");
}
inline int code_of(const Tensor& t) { return code_of(t.scalar_type()); }

// a call runs on the first tensor's GPU; every other tensor is checked to be on a GPU
struct Call {
  c10::Device dev;
  c10::cuda::CUDAGuard guard;
  explicit Call(const Tensor& t) : dev(t.device()), guard(need_cuda(t)) {}
  static c10::Device need_cuda(const Tensor& t) {
    if (!t.is_cuda()) raise_assertion("tops_b200 ops take CUDA tensors; there is no CPU path");
    return t.device();
  }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
  Tensor empty(at::IntArrayRef sizes, at::ScalarType t) const { return Tensor(at::detail::empty_cuda(sizes, t, dev, std::nullopt)); }
  Tensor empty_as(const Tensor& t) const { return empty(t.sizes(), t.scalar_type()); }
  Tensor bytes(size_t n) const { return empty({(int64_t)(n < 256 ? 256 : n)}, at::kByte); }
  // a tensor that is updated where it lies (fp32 and contiguous by the caller's checks)
  float* state(const Tensor& t) const {
    need_cuda(t);
    return t.data_ptr<float>();
  }
  // contiguous, on a GPU, on a 16-byte boundary (which a view into a larger tensor may not be, and what moves 16 bytes per
  // access asks for)
  Tensor in(const Tensor& t) const {
    if (!t.defined()) return t;
    need_cuda(t);
    if (!t.is_contiguous()) return t.contiguous();
    return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0 ? t : t.clone();
  }
  Tensor in(const OptTensor& t) const { return t.has_value() ? in(*t) : Tensor(); }
  Tensor in_as(const Tensor& t, at::ScalarType type) const { return t.defined() ? in(t.scalar_type() == type ? t : t.to(type)) : t; }
};
template <class T = void> T* ptr(const Tensor& t) { return t.defined() ? reinterpret_cast<T*>(t.data_ptr()) : nullptr; }
inline Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

template <class... Ts> bool wants_grad(const Ts&... ts) {
  return at::GradMode::is_enabled() && ((ts.defined() && ts.requires_grad()) || ...);
}

// A node whose saved tensors are given back after use.
struct OpNode : public Node {
  std::vector<SavedVariable> saved;
  bool released = false;
  void keep(std::initializer_list<Tensor> ts) {
    saved.reserve(ts.size());
    for (const Tensor& t : ts) saved.emplace_back(t, false);
  }
  variable_list unpack() {
    TORCH_CHECK(!released, "Trying to backward through the graph a second time (or directly access saved tensors after they "
                           "have already been freed): specify retain_graph=True");
    variable_list r;
    r.reserve(saved.size());
    for (auto& s : saved) r.push_back(s.unpack());
    return r;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    saved.clear();
    released = true;
  }
};
template <class N, class... Ts> std::shared_ptr<N> make_node(const Ts&... inputs) {
  auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  return node;
}
inline void attach(const Tensor& out, const std::shared_ptr<Node>& node) {
  if (out.defined()) torch::autograd::set_history(out, node);
}
inline Tensor cotangent(const Tensor& g, const Tensor& like_sizes_of, at::ScalarType type, const Call& c) {
  if (!g.defined()) return at::zeros(like_sizes_of.sizes(), at::TensorOptions().dtype(type).device(c.dev));
  return c.in_as(g, type);
}


struct ChunkShape {
  int kind = 0, chunk = 64, N = 0;
  double scale = 1.0;
  std::vector<int32_t> cu;
};

std::tuple<Tensor, OptTensor> gla_layer(const Tensor& x, const Tensor& Wq, const Tensor& Wk, const Tensor& Wv, const Tensor& Wg,
                                        const Tensor& Wlow, const Tensor& Wgk, const Tensor& bgk, const OptTensor& norm_weight,
                                        const Tensor& Wo, int heads, double eps, double normalizer, std::optional<double> clamp,
                                        const OptTensor& state, bool want_state, std::vector<int32_t> cu, bool recurrent);
bool gla_layer_takes(const Tensor& x, const Tensor& Wq, const Tensor& Wk, const Tensor& Wv, const Tensor& Wg, const Tensor& Wlow,
                     const Tensor& Wgk, const Tensor& bgk, const OptTensor& norm_weight, const Tensor& Wo, int heads, bool recurrent);

}  // namespace tops_torch
