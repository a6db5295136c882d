// The host side of the Python products, in native code: what SO3part.py and SO3vec.py do around one C-ABI call -- output
// type, output tensors, zero-filled gradients, descriptors, device, stream -- for operands that need nothing special.  Each
// function returns None, having done nothing, when an operand is not plain (not on a CUDA device, not complex64, lazily
// conjugated, more than two grid dimensions, two parts of one l, ...), when sizes do not fit together, and when the library
// skips the call: the Python code then takes it from the start and says what there is to say.
#include <ATen/ATen.h>
#include <ATen/ops/_foreach_zero.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <climits>
#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/gelib_b200.h"

namespace {

using Tensors = std::vector<at::Tensor>;

// A plain Python int of 32 bits.  Others are left to the Python code too: through ctypes the low 32 bits of a larger maxl count
// (sys.maxsize: every l), and what is not an int is refused there.
std::optional<int> plain_int(pybind11::handle h) {
  if (!PyLong_CheckExact(h.ptr())) return std::nullopt;
  int overflow = 0;
  const long v = PyLong_AsLongAndOverflow(h.ptr(), &overflow);
  if (overflow || v < INT_MIN || v > INT_MAX) return std::nullopt;
  return static_cast<int>(v);
}

// The tensor in canonical form, core/Gpart.hpp:450-469 of GElib; false when it is not plain.
bool describe(const at::Tensor& t, c10::Device device, gelib_tensor5* d) {
  if (!t.defined() || !t.is_cuda() || t.device() != device || t.scalar_type() != at::kComplexFloat || t.is_conj()) return false;
  const int dim = static_cast<int>(t.dim());
  if (dim < 3 || dim > 5) return false;
  const auto sizes = t.sizes();
  const auto strides = t.strides();
  for (int k = 0; k < dim; k++)
    if (sizes[k] > INT_MAX) return false;
  d->base = static_cast<float*>(t.data_ptr());
  const int at[5] = {0, dim > 3 ? 1 : -1, dim > 4 ? 2 : -1, dim - 2, dim - 1};
  for (int k = 0; k < 5; k++) {
    d->dims[k] = at[k] < 0 ? 1 : static_cast<int32_t>(sizes[at[k]]);
    d->strides[k] = at[k] < 0 ? 0 : 2 * strides[at[k]];  // in floats
  }
  return true;
}

// The parts of a vector, described in ascending l.
struct Vec {
  std::vector<gelib_tensor5> d;
  std::vector<int> l, n;
  int size() const { return static_cast<int>(d.size()); }
};
bool describe_all(const Tensors& parts, c10::Device device, Vec* v) {
  std::vector<std::pair<int, const at::Tensor*>> order;
  order.reserve(parts.size());
  for (const auto& t : parts) {
    if (!t.defined() || t.dim() < 3 || t.size(-2) > INT_MAX) return false;
    order.emplace_back(static_cast<int>((t.size(-2) - 1) / 2), &t);
  }
  std::sort(order.begin(), order.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
  for (size_t i = 0; i < order.size(); i++) {
    if (i > 0 && order[i].first == order[i - 1].first) return false;
    gelib_tensor5 t;
    if (!describe(*order[i].second, device, &t)) return false;
    v->d.push_back(t);
    v->l.push_back(order[i].first);
    v->n.push_back(t.dims[4]);
  }
  return true;
}

// Makes the call without the interpreter lock (a first call of a signature builds its plan).  True: done; false: the library
// skipped it.  Errors raise, as in _lib.check.
template <class F>
bool call(F f) {
  int status;
  std::string message;
  {
    pybind11::gil_scoped_release release;
    status = f();
    if (status != GELIB_OK && status != GELIB_SKIPPED) message = gelib_last_error();
  }
  if (!message.empty()) throw std::runtime_error(message);
  return status == GELIB_OK;
}

void* stream_of(c10::Device device) { return c10::cuda::getCurrentCUDAStream(device.index()).stream(); }

// Batch and grid of a product; false when the batches do not fit, or an operand is empty (the kernels then write nothing).
bool lead_dims(const at::Tensor& x, const at::Tensor& y, std::vector<int64_t>* lead) {
  const int64_t bx = x.size(0), by = y.size(0);
  if ((bx > 1 && by > 1 && bx != by) || x.numel() == 0 || y.numel() == 0) return false;
  lead->push_back(std::max(bx, by));
  const int64_t gx = x.dim() - 3, gy = y.dim() - 3;
  for (int64_t k = 1; k <= std::max(gx, gy); k++)  // size-1 grid dimensions are broadcast against the other operand's
    lead->push_back(gx == gy ? std::max(x.size(k), y.size(k)) : (gx > gy ? x : y).size(k));
  return true;
}

at::Tensor output(std::vector<int64_t> lead, int64_t l, int64_t n, c10::Device device) {
  lead.push_back(2 * l + 1);
  lead.push_back(n);
  return at::empty(lead, at::TensorOptions().dtype(at::kComplexFloat).device(device));
}

Tensors zeros_like_all(const Tensors& v) {
  Tensors r;
  r.reserve(v.size());
  for (const auto& t : v) r.push_back(at::empty_like(t));
  at::_foreach_zero_(r);
  return r;
}

std::optional<Tensors> vec_forward(const Tensors& x, const Tensors& y, pybind11::handle max_l, bool diag) {
  const auto maxl = plain_int(max_l);
  if (!maxl || x.empty() || y.empty() || !x[0].defined() || !x[0].is_cuda()) return std::nullopt;
  const auto device = x[0].device();
  Vec dx, dy, dr;
  std::vector<int64_t> lead;
  if (!describe_all(x, device, &dx) || !describe_all(y, device, &dy) || !lead_dims(x[0], y[0], &lead)) return std::nullopt;
  const int cap = dx.l.back() + dy.l.back() + 1;
  std::vector<int> l(cap), n(cap);
  const int k = gelib_SO3type_CGproduct(dx.size(), dx.l.data(), dx.n.data(), dy.size(), dy.l.data(), dy.n.data(), *maxl, diag, cap, l.data(), n.data());
  if (k <= 0) return std::nullopt;
  c10::cuda::CUDAGuard guard(device);
  Tensors r;
  for (int i = 0; i < k; i++) r.push_back(output(lead, l[i], n[i], device));
  if (!describe_all(r, device, &dr)) return std::nullopt;
  void* s = stream_of(device);
  const auto f = diag ? gelib_SO3vec_addDiagCGproduct : gelib_SO3vec_addCGproduct;
  if (!call([&] { return f(dr.size(), dr.d.data(), dx.size(), dx.d.data(), dy.size(), dy.d.data(), GELIB_OVERWRITE, s); })) return std::nullopt;
  return r;
}

// The gradients asked for, those of x first.
std::optional<Tensors> vec_backward(const Tensors& x, const Tensors& y, const Tensors& g, bool need_x, bool need_y, bool diag) {
  if (x.empty() || y.empty() || g.empty() || !(need_x || need_y) || !x[0].defined() || !x[0].is_cuda()) return std::nullopt;
  const auto device = x[0].device();
  Vec dx, dy, dg, dxg, dyg;
  if (!describe_all(x, device, &dx) || !describe_all(y, device, &dy) || !describe_all(g, device, &dg)) return std::nullopt;
  Tensors wanted;
  if (need_x) wanted.insert(wanted.end(), x.begin(), x.end());
  if (need_y) wanted.insert(wanted.end(), y.begin(), y.end());
  c10::cuda::CUDAGuard guard(device);
  Tensors r = zeros_like_all(wanted);
  const auto split = r.begin() + (need_x ? x.size() : 0);
  if (!describe_all(Tensors(r.begin(), split), device, &dxg) || !describe_all(Tensors(split, r.end()), device, &dyg)) return std::nullopt;
  void* s = stream_of(device);
  const bool ok = call([&] {
    if (need_x && need_y)
      return (diag ? gelib_SO3vec_addDiagCGproduct_back01 : gelib_SO3vec_addCGproduct_back01)(
          dxg.size(), dxg.d.data(), dyg.size(), dyg.d.data(), dg.size(), dg.d.data(), dx.d.data(), dy.d.data(), 0, s);
    if (need_x)
      return (diag ? gelib_SO3vec_addDiagCGproduct_back0 : gelib_SO3vec_addCGproduct_back0)(dxg.size(), dxg.d.data(), dg.size(), dg.d.data(),
                                                                                           dy.size(), dy.d.data(), 0, s);
    return (diag ? gelib_SO3vec_addDiagCGproduct_back1 : gelib_SO3vec_addCGproduct_back1)(dyg.size(), dyg.d.data(), dg.size(), dg.d.data(),
                                                                                         dx.size(), dx.d.data(), 0, s);
  });
  if (!ok) return std::nullopt;
  return r;
}

std::optional<at::Tensor> part_forward(const at::Tensor& x, const at::Tensor& y, pybind11::handle out_l, bool diag) {
  const auto l = plain_int(out_l);
  if (!l || !x.defined() || !x.is_cuda() || *l < 0) return std::nullopt;
  const auto device = x.device();
  gelib_tensor5 dx, dy, dr;
  std::vector<int64_t> lead;
  if (!describe(x, device, &dx) || !describe(y, device, &dy) || !lead_dims(x, y, &lead)) return std::nullopt;
  if (diag && x.size(-1) != y.size(-1)) return std::nullopt;
  c10::cuda::CUDAGuard guard(device);
  at::Tensor r = output(lead, *l, diag ? x.size(-1) : x.size(-1) * y.size(-1), device);
  if (!describe(r, device, &dr)) return std::nullopt;
  void* s = stream_of(device);
  const auto f = diag ? gelib_SO3part_addDiagCGproduct : gelib_SO3part_addCGproduct;
  if (!call([&] { return f(&dr, &dx, &dy, 0, GELIB_OVERWRITE, s); })) return std::nullopt;
  return r;
}

std::optional<Tensors> part_backward(const at::Tensor& x, const at::Tensor& y, const at::Tensor& g, bool need_x, bool need_y, bool diag) {
  if (!x.defined() || !x.is_cuda() || !(need_x || need_y)) return std::nullopt;
  const auto device = x.device();
  gelib_tensor5 dx, dy, dg, dw[2];
  if (!describe(x, device, &dx) || !describe(y, device, &dy) || !describe(g, device, &dg)) return std::nullopt;
  Tensors wanted;
  if (need_x) wanted.push_back(x);
  if (need_y) wanted.push_back(y);
  c10::cuda::CUDAGuard guard(device);
  Tensors r = zeros_like_all(wanted);
  for (size_t i = 0; i < r.size(); i++)
    if (!describe(r[i], device, &dw[i])) return std::nullopt;
  void* s = stream_of(device);
  const bool ok = call([&] {
    if (need_x && need_y) return (diag ? gelib_SO3part_addDiagCGproduct_back01 : gelib_SO3part_addCGproduct_back01)(&dw[0], &dw[1], &dg, &dx, &dy, 0, 0, s);
    if (need_x) return (diag ? gelib_SO3part_addDiagCGproduct_back0 : gelib_SO3part_addCGproduct_back0)(&dw[0], &dg, &dy, 0, 0, s);
    return (diag ? gelib_SO3part_addDiagCGproduct_back1 : gelib_SO3part_addCGproduct_back1)(&dw[0], &dg, &dx, 0, 0, s);
  });
  if (!ok) return std::nullopt;
  return r;
}

// x gathered along array dimension d (tensor dimension d + 1) by a map of n_in cells into n_out.
std::optional<at::Tensor> gather(const at::Tensor& x0, const at::Tensor& row_ptr, const at::Tensor& col, int n_in, int n_out, pybind11::handle dim) {
  const auto array_dim = plain_int(dim);
  if (!array_dim || !x0.defined() || !x0.is_cuda() || x0.scalar_type() != at::kComplexFloat || x0.is_conj()) return std::nullopt;
  const auto device = x0.device();
  const int d = *array_dim;
  if (d < 0 || d + 1 >= x0.dim() || x0.size(d + 1) != n_in || row_ptr.device() != device || col.device() != device) return std::nullopt;
  c10::cuda::CUDAGuard guard(device);
  const at::Tensor x = x0.detach().contiguous();
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
  shape[d + 1] = n_out;
  int64_t outer = 1, inner = 1;
  for (int k = 0; k <= d; k++) outer *= shape[k];
  for (size_t k = d + 2; k < shape.size(); k++) inner *= shape[k];
  at::Tensor r = at::zeros(shape, at::TensorOptions().dtype(at::kComplexFloat).device(device));
  void* s = stream_of(device);
  float* rp = static_cast<float*>(r.data_ptr());
  const float* xp = static_cast<const float*>(x.data_ptr());
  const int *pp = row_ptr.data_ptr<int>(), *cp = col.data_ptr<int>();
  if (!call([&] { return gelib_add_gather(rp, xp, outer, n_out, n_in, inner, pp, cp, s); })) return std::nullopt;
  return r;
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.attr("torch_version") = GELIB_TORCH_VERSION;
  m.def("vec_forward", torch::wrap_pybind_function(&vec_forward));
  m.def("vec_backward", torch::wrap_pybind_function(&vec_backward));
  m.def("part_forward", torch::wrap_pybind_function(&part_forward));
  m.def("part_backward", torch::wrap_pybind_function(&part_backward));
  m.def("gather", torch::wrap_pybind_function(&gather));
}
