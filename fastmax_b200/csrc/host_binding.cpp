// torch C++ module `fastmax_b200._host`: the host side of the package's most frequent calls -- the attention module, the
// model's call site and a decode step -- as C++ autograd functions over the C ABI.  Small problems are bound by the
// host; the same work in Python (argument checks, allocations, ctypes calls, a Python frame in the backward thread)
// takes longer than their kernels.  Forward and backward through the module, 8 heads x 197 in bf16: 147 -> 98 us, 16 x 1024
// in float32 153 -> 104.
//
// Every entry returns None for arguments outside the plain case (other types, layouts, devices, shapes that do not match):
// the Python functions of the same purpose serve those, and raise the errors.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <cstdint>
#include <optional>
#include <tuple>
#include <vector>

#include "fastmax_b200.h"

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// what an error code of the library becomes: an argument error is a ValueError, as in Python
void check_rc(int rc, const char* what) {
  TORCH_CHECK_VALUE(rc != FASTMAX_E_ARG, what, ": ", fastmax_b200_last_error());
  TORCH_CHECK(rc == FASTMAX_OK, what, " failed (code ", rc, "): ", fastmax_b200_last_error());
}

Tensor bytes_like(size_t n, const Tensor& like) {
  return at::empty({(int64_t)(n < 1 ? 1 : n)}, like.options().dtype(torch::kUInt8));
}
// Scratch of the wanted size, or of the least the call runs with where the device has no room for more.
Tensor scratch(size_t want, size_t least, const Tensor& like) {
  try {
    return bytes_like(want, like);
  } catch (const c10::OutOfMemoryError&) {
    if (least >= want) throw;
  }
  return bytes_like(least, like);
}

struct Args {
  bool mask, normalize;
  double temperature, a0, a1, a2, lim;
  int64_t p;
};

bool kind_ok(const Tensor& t) {
  return t.is_cuda() && (t.scalar_type() == torch::kFloat32 || t.scalar_type() == torch::kBFloat16);
}

// q (.., nq, d) and k (.., nk, d) over one or two leading axes
fastmax_problem problem_of(const Tensor& q, const Tensor& k, const Args& a) {
  fastmax_problem pr = {};
  pr.dtype = q.scalar_type() == torch::kFloat32 ? FASTMAX_F32 : FASTMAX_BF16;
  pr.bh = (int32_t)(q.dim() == 4 ? q.size(0) * q.size(1) : q.size(0));
  pr.bhkv = (int32_t)(k.dim() == 4 ? k.size(0) * k.size(1) : k.size(0));
  pr.nq = (int32_t)q.size(-2);
  pr.nk = (int32_t)k.size(-2);
  pr.d = (int32_t)q.size(-1);
  pr.mask = a.mask;
  pr.normalize = a.normalize;
  pr.p = (int32_t)a.p;
  pr.impl = FASTMAX_IMPL_AUTO;
  pr.a0 = (float)a.a0;
  pr.a1 = (float)a.a1;
  pr.a2 = (float)a.a2;
  pr.lim = (float)a.lim;
  pr.temperature = (float)a.temperature;
  pr.chunk = 0;
  return pr;
}

cudaStream_t stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

void keep(AutogradContext* ctx, const Args& a) {
  ctx->saved_data["s"] = std::vector<double>{(double)a.mask, (double)a.normalize, a.temperature, a.a0, a.a1, a.a2, a.lim,
                                             (double)a.p};
}
Args kept(AutogradContext* ctx) {
  const auto s = ctx->saved_data["s"].toDoubleVector();
  return Args{s[0] != 0, s[1] != 0, s[2], s[3], s[4], s[5], s[6], (int64_t)s[7]};
}

// forward of contiguous q, k, v: out (q's shape, or (batch, nq, heads, d) when bt_heads > 0), den, stats
std::tuple<Tensor, Tensor, Tensor> run_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Args& a, int bt_heads) {
  const fastmax_problem pr = problem_of(q, k, a);
  const c10::cuda::CUDAGuard guard(q.device());
  const size_t want = fastmax_b200_forward_workspace_bytes(&pr), least = fastmax_b200_forward_workspace_least_bytes(&pr);
  const size_t words = fastmax_b200_stats_bytes(&pr);
  Tensor out = bt_heads ? at::empty({pr.bh / bt_heads, pr.nq, bt_heads, pr.d}, q.options()) : at::empty(q.sizes(), q.options());
  Tensor den = at::empty({pr.bh, pr.nq}, q.options().dtype(torch::kFloat32));
  Tensor stats = bytes_like(words < 8 ? 8 : words, q);
  Tensor ws;
  if (want) ws = scratch(want, least, q);
  void* wp = ws.defined() ? ws.data_ptr() : nullptr;
  const size_t wb = ws.defined() ? (size_t)ws.numel() : 0;
  if (bt_heads)
    check_rc(fastmax_b200_forward_bt(&pr, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), (float*)den.data_ptr(),
                                     stats.data_ptr(), bt_heads, wp, wb, stream_of(q)), "fastmax_b200_forward_bt");
  else
    check_rc(fastmax_b200_forward(&pr, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), (float*)den.data_ptr(),
                                  stats.data_ptr(), wp, wb, stream_of(q)), "fastmax_b200_forward");
  return {out, den, stats};
}

std::tuple<Tensor, Tensor, Tensor> run_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out,
                                                const Tensor& den, const Tensor& stats, const Tensor& go, const Args& a,
                                                int bt_heads) {
  const fastmax_problem pr = problem_of(q, k, a);
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor gq = at::empty(q.sizes(), q.options()), gk = at::empty(k.sizes(), k.options()), gv = at::empty(v.sizes(), v.options());
  Tensor ws = scratch(fastmax_b200_backward_workspace_bytes(&pr), fastmax_b200_backward_workspace_least_bytes(&pr), q);
  if (bt_heads)
    check_rc(fastmax_b200_backward_bt(&pr, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                                      (const float*)den.data_ptr(), stats.data_ptr(), go.data_ptr(), bt_heads, gq.data_ptr(),
                                      gk.data_ptr(), gv.data_ptr(), ws.data_ptr(), (size_t)ws.numel(), stream_of(q)),
             "fastmax_b200_backward_bt");
  else
    check_rc(fastmax_b200_backward(&pr, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                                   (const float*)den.data_ptr(), stats.data_ptr(), go.data_ptr(), gq.data_ptr(),
                                   gk.data_ptr(), gv.data_ptr(), ws.data_ptr(), (size_t)ws.numel(), stream_of(q)),
             "fastmax_b200_backward");
  if (a.temperature != 1.0) gk = gk / a.temperature;      // as the reference wrapper does (example.py:80)
  return {gq, gk, gv};
}

// ---- the attention module -------------------------------------------------------------------------------------
struct Attention : public torch::autograd::Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Args& a) {
    const Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous();
    auto [out, den, stats] = run_forward(q, k, v, a, 0);
    ctx->save_for_backward({q, k, v, out, den, stats});
    keep(ctx, a);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    Tensor go = grads[0].contiguous();
    if (go.scalar_type() != s[0].scalar_type()) go = go.to(s[0].scalar_type());
    auto [gq, gk, gv] = run_backward(s[0], s[1], s[2], s[3], s[4], s[5], go, kept(ctx), 0);
    return {gq, gk, gv, Tensor()};
  }
};

std::optional<Tensor> attention(const Tensor& q, const Tensor& k, const Tensor& v, bool mask, bool normalize,
                                double temperature, double a0, double a1, double a2, double lim, int64_t p) {
  if (!kind_ok(q) || (q.dim() != 3 && q.dim() != 4) || (k.dim() != 3 && k.dim() != 4) || k.sizes() != v.sizes() ||
      q.size(-1) != k.size(-1) || k.device() != q.device() || v.device() != q.device() ||
      k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type())
    return std::nullopt;
  py::gil_scoped_release no_gil;
  return Attention::apply(q, k, v, Args{mask, normalize, temperature, a0, a1, a2, lim, p});
}

// ---- the model's call site --------------------------------------------------------------------------------------
struct FromQKV : public torch::autograd::Function<FromQKV> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& cs, const Tensor& sn, int64_t groups,
                        int64_t qper, int64_t rope, const Args& a) {
    const int64_t b = qkv.size(0), n = qkv.size(1), heads = groups * qper, d = qkv.size(2) / (groups * (qper + 2));
    const c10::cuda::CUDAGuard guard(qkv.device());
    const int dt = qkv.scalar_type() == torch::kFloat32 ? FASTMAX_F32 : FASTMAX_BF16;
    Tensor q = at::empty({b * heads, n, d}, qkv.options()), k = at::empty({b * groups, n, d}, qkv.options());
    Tensor v = at::empty({b * groups, n, d}, qkv.options());
    const float* cp = rope ? (const float*)cs.data_ptr() : nullptr;
    const float* sp = rope ? (const float*)sn.data_ptr() : nullptr;
    check_rc(fastmax_b200_qkv_split_rope(qkv.data_ptr(), cp, sp, q.data_ptr(), k.data_ptr(), v.data_ptr(), b, n, (int)groups,
                                         (int)qper, (int)d, (int)rope, dt, stream_of(qkv)), "fastmax_b200_qkv_split_rope");
    const fastmax_problem pr = problem_of(q, k, a);
    const bool bt = fastmax_b200_bt_layout_supported(&pr, (int)heads) != 0;    // the attention kernel writes (B, T, H, hs) itself
    auto [out, den, stats] = run_forward(q, k, v, a, bt ? (int)heads : 0);
    // without a rotation the tables are not part of the problem: the caller may go on changing them
    ctx->save_for_backward({q, k, v, out, den, stats, rope ? cs : Tensor(), rope ? sn : Tensor()});
    keep(ctx, a);
    ctx->saved_data["d"] = std::vector<int64_t>{b, n, groups, qper, d, rope, bt ? 1 : 0};
    if (bt) return out.view({b, n, heads * d});
    Tensor y = at::empty({b, n, heads * d}, qkv.options());
    check_rc(fastmax_b200_swap_middle_axes(out.data_ptr(), y.data_ptr(), b, heads, n, (int)d, dt, stream_of(qkv)),
             "fastmax_b200_swap_middle_axes");
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const auto dims = ctx->saved_data["d"].toIntVector();
    const int64_t b = dims[0], n = dims[1], groups = dims[2], qper = dims[3], d = dims[4], rope = dims[5], heads = groups * qper;
    const bool bt = dims[6] != 0;
    const Tensor& q = s[0];
    const c10::cuda::CUDAGuard guard(q.device());
    const int dt = q.scalar_type() == torch::kFloat32 ? FASTMAX_F32 : FASTMAX_BF16;
    Tensor gy = grads[0].to(q.scalar_type()).contiguous();
    if (!bt) {
      Tensor go = at::empty({b * heads, n, d}, q.options());
      check_rc(fastmax_b200_swap_middle_axes(gy.data_ptr(), go.data_ptr(), b, n, heads, (int)d, dt, stream_of(q)),
               "fastmax_b200_swap_middle_axes");
      gy = go;
    }
    auto [gq, gk, gv] = run_backward(q, s[1], s[2], s[3], s[4], s[5], gy, kept(ctx), bt ? (int)heads : 0);
    Tensor gqkv = at::empty({b, n, groups * (qper + 2) * d}, q.options());
    check_rc(fastmax_b200_qkv_merge_rope_grad(gq.data_ptr(), gk.data_ptr(), gv.data_ptr(),
                                              rope ? (const float*)s[6].data_ptr() : nullptr,
                                              rope ? (const float*)s[7].data_ptr() : nullptr, gqkv.data_ptr(), b, n,
                                              (int)groups, (int)qper, (int)d, (int)rope, dt, stream_of(q)),
             "fastmax_b200_qkv_merge_rope_grad");
    return {gqkv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// qkv (B, T, groups * (qper + 2) * d) contiguous; cos, sin (T, rope) float32 contiguous on its device, or empty
std::optional<Tensor> from_qkv(const Tensor& qkv, const Tensor& cs, const Tensor& sn, int64_t groups, int64_t qper,
                               int64_t d, int64_t rope, bool mask, bool normalize, double temperature, double a0, double a1,
                               double a2, double lim, int64_t p) {
  if (!kind_ok(qkv) || qkv.dim() != 3 || !qkv.is_contiguous() || groups < 1 || qper < 1 || d < 1 ||
      qkv.size(2) != groups * (qper + 2) * d)
    return std::nullopt;
  if (rope)
    for (const Tensor* t : {&cs, &sn})
      if (t->device() != qkv.device() || t->scalar_type() != torch::kFloat32 || !t->is_contiguous() || t->dim() != 2 ||
          t->size(0) != qkv.size(1) || t->size(1) != rope)
        return std::nullopt;
  py::gil_scoped_release no_gil;
  return FromQKV::apply(qkv, cs, sn, groups, qper, rope, Args{mask, normalize, temperature, a0, a1, a2, lim, p});
}

// ---- a decode step ------------------------------------------------------------------------------------------------
// problem: address of the caller's fastmax_problem
std::optional<Tensor> decode_step(uintptr_t problem, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& state,
                                  const Tensor& scratch) {
  const fastmax_problem& pr = *reinterpret_cast<const fastmax_problem*>(problem);
  const auto dtype = pr.dtype == FASTMAX_BF16 ? torch::kBFloat16 : torch::kFloat32;
  auto row_ok = [&](const Tensor& t, int64_t heads) {
    return t.dim() == 3 && t.size(0) == heads && t.size(1) == 1 && t.size(2) == pr.d && t.scalar_type() == dtype &&
           t.device() == state.device() && t.is_contiguous();
  };
  if (!row_ok(q, pr.bh) || !row_ok(k, pr.bhkv) || !row_ok(v, pr.bhkv)) return std::nullopt;
  py::gil_scoped_release no_gil;       // a launch waits while the device's queue is full
  const c10::cuda::CUDAGuard guard(state.device());
  Tensor out = at::empty(q.sizes(), q.options());
  check_rc(fastmax_b200_decode_step(&pr, q.data_ptr(), k.data_ptr(), v.data_ptr(), state.data_ptr(), scratch.data_ptr(),
                                    out.data_ptr(), stream_of(q)), "fastmax_b200_decode_step");
  return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("attention", &attention);
  m.def("from_qkv", &from_qkv);
  m.def("decode_step", &decode_step);
}
