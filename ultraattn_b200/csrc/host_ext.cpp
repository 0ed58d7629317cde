// What a single-device attention call does on the host between Python and the kernel library, as one native call:
// output and workspace tensors, checks, the argument block, the launches.
//
// In Python these took 12 us of the forward and 25 of the backward, twice that on the autograd thread, whose
// caches are cold: a training call of 512 tokens waited for the host for two thirds of its time. Only this
// part is native. The autograd functions stay in Python, and so does every case that is not the plain one: a function
// here answers None, having done nothing, for tensors that it does not take, and the caller goes on as before.
//
// The library is not linked; its entry points are handed over as addresses (init).
#include <ATen/ATen.h>
#include <torch/csrc/utils/pybind.h>

#include "arg_blocks.h"

namespace {

int (*fwd_dense_parts)(int, int, int, int, int, int, int);
int (*fwd_dense)(const UaDenseFwd*, int, float, int, float*, int*, void*);
int (*bwd_local)(const UaLocalBwd*, float, int*, void*);
const char* (*last_error)();

void init(uintptr_t parts, uintptr_t dense, uintptr_t local, uintptr_t error) {
  fwd_dense_parts = reinterpret_cast<decltype(fwd_dense_parts)>(parts);
  fwd_dense = reinterpret_cast<decltype(fwd_dense)>(dense);
  bwd_local = reinterpret_cast<decltype(bwd_local)>(local);
  last_error = reinterpret_cast<decltype(last_error)>(error);
}

constexpr int64_t D = 128;

// [batch, tokens, heads, 128] bf16 on `dev`, head dim contiguous
bool takes(const at::Tensor& t, const at::Device& dev) {
  return t.dim() == 4 && t.scalar_type() == at::kBFloat16 && t.device() == dev && t.size(3) == D && t.stride(3) == 1;
}
// ... whose heads lie side by side (an axis of one may have any stride)
bool takes_rows(const at::Tensor& t, const at::Device& dev) { return takes(t, dev) && (t.stride(2) == D || t.size(2) == 1); }

UaTensorSrc src(const at::Tensor& t) {
  return UaTensorSrc{t.data_ptr(), t.size(1), t.size(2), t.size(0), t.stride(1), t.stride(2), t.stride(0)};
}

void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + " failed: " + last_error());
}

// (o, lse, kernels launched): all queries against all keys
py::object dense_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, bool causal, double scale, uintptr_t status,
                         uintptr_t stream) {
  const at::Device dev = q.device();
  if (!dev.is_cuda() || !takes(q, dev) || !takes(k, dev) || !takes(v, dev)) return py::none();
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2);
  const at::Tensor o = at::empty_like(q);
  if (o.stride(2) != D || o.stride(3) != 1) return py::none();
  const auto f32 = q.options().dtype(at::kFloat);
  const at::Tensor lse = at::empty({B, H, S}, f32);
  const int parts = fwd_dense_parts(static_cast<int>(B), static_cast<int>(S), static_cast<int>(k.size(1)), static_cast<int>(H),
                                    static_cast<int>(k.size(2)), causal, 0);
  at::Tensor ws;
  if (parts > 0) ws = at::empty({parts * B * S * H * (D + 1)}, f32);
  const UaDenseFwd a{src(q), src(k), src(v),
                     {o.data_ptr(), static_cast<float*>(lse.data_ptr()), o.stride(1), o.stride(0), lse.stride(1), lse.stride(0)}};
  {
    py::gil_scoped_release nogil;
    check(fwd_dense(&a, causal, static_cast<float>(scale), 0, parts > 0 ? static_cast<float*>(ws.data_ptr()) : nullptr,
                    reinterpret_cast<int*>(status), reinterpret_cast<void*>(stream)),
          "ua_attn_fwd_dense");
  }
  return py::make_tuple(o, lse, parts > 0 ? 2 : 1);
}

// (dq, dk, dv): the whole backward, under a plan (device tables) or dense = 1 / 2: without a mask / causal
py::object local_backward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& lse,
                          const at::Tensor& d_o, uintptr_t cols, uintptr_t segs, uintptr_t tiles, int64_t n_tiles, int64_t dense,
                          int64_t skewed, double scale, uintptr_t status, uintptr_t stream) {
  const at::Device dev = q.device();
  if (!dev.is_cuda() || !takes(q, dev) || !takes(k, dev) || !takes(v, dev) || !takes_rows(o, dev) || !takes_rows(d_o, dev)) return py::none();
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2);
  if (o.sizes() != q.sizes() || d_o.sizes() != q.sizes() || k.sizes() != v.sizes() || lse.dim() != 3 || lse.device() != dev ||
      lse.scalar_type() != at::kFloat || lse.size(0) != B || lse.size(1) != H || lse.size(2) != S || !lse.is_contiguous())
    return py::none();
  const at::Tensor dq = at::empty(q.sizes(), q.options());
  const at::Tensor dk = at::empty_like(k), dv = at::empty_like(v);
  if (!takes_rows(dk, dev) || dk.strides() != dv.strides()) return py::none();
  const auto f32 = q.options().dtype(at::kFloat);
  const at::Tensor dvec = at::empty({B, H, S}, f32), dq32 = at::empty({B * S * H * D}, f32);
  const UaLocalBwd a{src(q), src(k), src(v), src(d_o), o.data_ptr(), o.stride(1), o.stride(0), static_cast<float*>(lse.data_ptr()),
                     static_cast<float*>(dvec.data_ptr()), static_cast<float*>(dq32.data_ptr()), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                     dk.stride(1), dk.stride(0), reinterpret_cast<void*>(cols), reinterpret_cast<void*>(segs), reinterpret_cast<void*>(tiles),
                     n_tiles, dense, skewed};
  {
    py::gil_scoped_release nogil;
    check(bwd_local(&a, static_cast<float>(scale), reinterpret_cast<int*>(status), reinterpret_cast<void*>(stream)), "ua_attn_bwd_local");
  }
  return py::make_tuple(dq, dk, dv);
}

}  // namespace

PYBIND11_MODULE(ua_host, m) {
  m.def("init", &init);
  m.def("dense_forward", &dense_forward);
  m.def("local_backward", &local_backward);
}
