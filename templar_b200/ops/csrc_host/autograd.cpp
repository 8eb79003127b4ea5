// Autograd nodes of the decoder block's operators, host side.
//
// The same sequences of kernel launches as the Python nodes in functional.py (_RMSNorm, _AddRMSNorm, _Linear, _FeedForward,
// _AttentionBlock), for bf16 CUDA operands that those nodes would hand to the own kernels.  A Python node costs its
// interpreter time twice (the backward half on the autograd thread, behind the interpreter lock): for one residual add and
// norm of a small batch that was 115 us around 9 us of kernels.  Here it is 80 us, most of it the engine's own.
//
// functional.py decides which calls come here (operand types, strides and alignment) and keeps its nodes for all others.
// Tensors are saved as saved variables only; the gradient buffers of the flat store are held by reference as there.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>

#include "../csrc/entries.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
typedef long long ll;

std::atomic<ll> g_launches{0};

// C entry points of the kernel library
struct Entries {
  decltype(&tplr_add_rmsnorm_fwd) add_rmsnorm_fwd;
  decltype(&tplr_add_rmsnorm_bwd_v2) add_rmsnorm_bwd;
  decltype(&tplr_gemm2_bf16) gemm;
  decltype(&tplr_gemm2_acc_splits) acc_splits;
  decltype(&tplr_gemm2_acc_split) acc_split;
  decltype(&tplr_gemm2_out_splits) out_splits;
  decltype(&tplr_gemm2_bf16_split) gemm_split;
  decltype(&tplr_gemm2_swiglu) swiglu;
  decltype(&tplr_gemm2_swiglu_bwd) swiglu_bwd;
  decltype(&tplr_gemm2_rope) gemm_rope;
  decltype(&tplr_attention_fwd) attention_fwd;
  decltype(&tplr_gemm2_attn_dout) attn_dout;
  decltype(&tplr_attention_bwd_scratch_cols) bwd_scratch_cols;
  decltype(&tplr_attention_bwd_unrope_delta) attention_bwd;
} E;

void bind(const std::string& path) {
  void* so = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(so, "cannot open ", path, ": ", dlerror());
  auto get = [&](auto& fn, const char* name) {
    void* p = dlsym(so, name);
    TORCH_CHECK(p, name, " is missing in ", path);
    fn = reinterpret_cast<std::decay_t<decltype(fn)>>(p);
  };
  decltype(&tplr_abi) abi;
  get(abi, "tplr_abi");
  TORCH_CHECK(abi() == TPLR_ABI, path, " was built from other entry declarations than the autograd nodes; build both again");
  get(E.add_rmsnorm_fwd, "tplr_add_rmsnorm_fwd");
  get(E.add_rmsnorm_bwd, "tplr_add_rmsnorm_bwd_v2");
  get(E.gemm, "tplr_gemm2_bf16");
  get(E.acc_splits, "tplr_gemm2_acc_splits");
  get(E.acc_split, "tplr_gemm2_acc_split");
  get(E.out_splits, "tplr_gemm2_out_splits");
  get(E.gemm_split, "tplr_gemm2_bf16_split");
  get(E.swiglu, "tplr_gemm2_swiglu");
  get(E.swiglu_bwd, "tplr_gemm2_swiglu_bwd");
  get(E.gemm_rope, "tplr_gemm2_rope");
  get(E.attention_fwd, "tplr_attention_fwd");
  get(E.attn_dout, "tplr_gemm2_attn_dout");
  get(E.bwd_scratch_cols, "tplr_attention_bwd_scratch_cols");
  get(E.attention_bwd, "tplr_attention_bwd_unrope_delta");
}

void check(int err, const char* what) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  TORCH_CHECK(err == 0, what, " failed with CUDA error ", err);
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
// the device's status word, as the kernels take it; the nodes keep the tensor and no pointer into it
unsigned* word(const Tensor& status) { return reinterpret_cast<unsigned*>(status.data_ptr()); }

// A gradient as the kernels read it: dense, on a 16-byte boundary.
Tensor dense(const Tensor& t) {
  Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 ? c.clone() : c;
}
Tensor f32(at::IntArrayRef shape, const Tensor& like) { return at::empty(shape, like.options().dtype(at::kFloat)); }
Tensor bf16(at::IntArrayRef shape, const Tensor& like) { return at::empty(shape, like.options()); }

// a tensor that takes no part in differentiation (a gradient buffer, the rotary tables); may be undefined
struct Aside { Tensor t; };
Tensor aside(AutogradContext* ctx, const char* key) {
  auto it = ctx->saved_data.find(key);
  return it == ctx->saved_data.end() ? Tensor() : it->second.toTensor();
}
void keep(AutogradContext* ctx, const char* key, const Aside& a) {
  if (a.t.defined()) ctx->saved_data[key] = a.t;
}

// out = op(a) op(b)^T as functional.gemm; epi 0: store bf16, 1: add into fp32
void gemm(const Tensor& a, const Tensor& b, const Tensor& out, bool a_mn, bool b_mn, int epi, const Tensor& status) {
  const ll M = a_mn ? a.size(1) : a.size(0), K = a_mn ? a.size(0) : a.size(1), N = b_mn ? b.size(1) : b.size(0);
  const ll plane = (M + 31) / 32 * 32 * N;             // workspace of one part of K, where K is cut
  if (epi == 0) {
    if (const ll parts = E.out_splits((int)M, (int)N, (int)K); parts > 1) {
      Tensor ws = f32({parts * plane}, a);
      check(E.gemm_split(a.data_ptr(), b.data_ptr(), out.data_ptr(), ws.data_ptr<float>(), (int)M, (int)N, (int)K, a.stride(0),
                         b.stride(0), out.stride(0), a_mn, b_mn, word(status), stream()),
            "tplr_gemm2_bf16_split");
      return;
    }
  } else if (reinterpret_cast<uintptr_t>(out.data_ptr()) % 16 == 0) {
    if (const ll parts = E.acc_splits((int)M, (int)N, (int)K); parts > 1) {
      Tensor ws = f32({(parts - 1) * plane}, a);
      check(E.acc_split(a.data_ptr(), b.data_ptr(), out.data_ptr<float>(), ws.data_ptr<float>(), (int)M, (int)N, (int)K, a.stride(0),
                        b.stride(0), out.stride(0), a_mn, b_mn, word(status), stream()),
            "tplr_gemm2_acc_split");
      return;
    }
  }
  check(E.gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, a.stride(0), b.stride(0), out.stride(0), a_mn,
               b_mn, epi, word(status), 0, stream()),
        "tplr_gemm_bf16");
}
// dW of y = x W^T: added into the gradient buffer when there is one, else returned when wanted
Tensor weight_grad(const Tensor& buffer, const Tensor& dy2, const Tensor& x2, const Tensor& w, bool wanted, const Tensor& status) {
  if (buffer.defined()) {
    gemm(dy2, x2, buffer, true, true, 1, status);
    return Tensor();
  }
  if (!wanted) return Tensor();
  Tensor dw = bf16(w.sizes(), w);
  gemm(dy2, x2, dw, true, true, 0, status);
  return dw;
}
Tensor rows(const Tensor& t) { return t.reshape({-1, t.size(-1)}); }
// rows of a tensor whose last dimension is D; an integer division by zero would end the process
ll count_rows(const Tensor& t, ll D) {
  TORCH_CHECK(D > 0, "rows of no elements");
  return t.numel() / D;
}

// ------------------------------------------------------------------------------------------ norms
// inputs: x (or res, delta), w, buffer, eps, status
variable_list norm_backward(AutogradContext* ctx, const Tensor& dh, const Tensor& dy_in, const Tensor& h, const Tensor& w,
                            const Tensor& rstd, int w_index) {
  const Tensor status = aside(ctx, "status");
  const Tensor buffer = aside(ctx, "buffer");
  const ll D = h.size(-1), T = count_rows(h, D);
  const Tensor dy = dy_in.defined() ? dense(dy_in) : at::zeros_like(h);
  const Tensor dres = dh.defined() ? dense(dh) : Tensor();
  Tensor dx = at::empty_like(h);
  Tensor dw = buffer.defined() ? buffer : at::zeros({D}, h.options().dtype(at::kFloat));
  check(E.add_rmsnorm_bwd(dy.data_ptr(), h.data_ptr(), w.data_ptr(), rstd.data_ptr<float>(), dres.defined() ? dres.data_ptr() : nullptr,
                          dx.data_ptr(), dw.data_ptr<float>(), T, (int)D, word(status), stream()),
        "add_rmsnorm_bwd");
  return {dx, buffer.defined() || !ctx->needs_input_grad(w_index) ? Tensor() : dw.to(w.scalar_type())};
}

struct RMSNorm : Function<RMSNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, Aside buffer, double eps, Aside status) {
    const ll D = x.size(-1), T = count_rows(x, D);
    Tensor y = at::empty_like(x), rstd = f32({T}, x);
    check(E.add_rmsnorm_fwd(x.data_ptr(), nullptr, w.data_ptr(), nullptr, y.data_ptr(), rstd.data_ptr<float>(), T, (int)D, (float)eps,
                            stream()),
          "rmsnorm_fwd");
    ctx->save_for_backward({x, w, rstd});
    keep(ctx, "buffer", buffer);
    keep(ctx, "status", status);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    auto r = norm_backward(ctx, Tensor(), g[0], s[0], s[1], s[2], 1);
    return {r[0], r[1], Tensor(), Tensor(), Tensor()};
  }
};

struct AddRMSNorm : Function<AddRMSNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& res, const Tensor& delta, const Tensor& w, Aside buffer, double eps,
                               Aside status) {
    const ll D = res.size(-1), T = count_rows(res, D);
    Tensor h = at::empty_like(res), y = at::empty_like(res), rstd = f32({T}, res);
    check(E.add_rmsnorm_fwd(res.data_ptr(), delta.data_ptr(), w.data_ptr(), h.data_ptr(), y.data_ptr(), rstd.data_ptr<float>(), T,
                            (int)D, (float)eps, stream()),
          "add_rmsnorm_fwd");
    ctx->save_for_backward({h, w, rstd});
    keep(ctx, "buffer", buffer);
    keep(ctx, "status", status);
    return {h, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    auto r = norm_backward(ctx, g[0], g[1], s[0], s[1], s[2], 2);
    return {r[0], r[0], r[1], Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------ projections
struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, Aside buffer, Aside status) {
    auto shape = x.sizes().vec();
    shape.back() = w.size(0);
    Tensor y = bf16(shape, x);
    gemm(rows(x), w, y.view({-1, w.size(0)}), false, false, 0, status.t);
    ctx->save_for_backward({x, w});
    keep(ctx, "buffer", buffer);
    keep(ctx, "status", status);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    const Tensor status = aside(ctx, "status");
    const Tensor dy2 = dense(rows(g[0])), x2 = rows(s[0]);
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      dx = bf16(s[0].sizes(), s[0]);
      gemm(dy2, s[1], dx.view({-1, s[1].size(1)}), false, true, 0, status);
    }
    return {dx, weight_grad(aside(ctx, "buffer"), dy2, x2, s[1], ctx->needs_input_grad(1), status), Tensor(), Tensor()};
  }
};

struct FeedForward : Function<FeedForward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w13, const Tensor& w2, Aside buffer13, Aside buffer2,
                        Aside status) {
    const Tensor x2 = rows(x);
    const ll T = x2.size(0), F2 = w13.size(0), F = F2 / 2;
    Tensor gu = bf16({T, F2}, x), h = bf16({T, F}, x);
    check(E.swiglu(x2.data_ptr(), w13.data_ptr(), gu.data_ptr(), h.data_ptr(), (int)T, (int)F, (int)x2.size(1), x2.stride(0),
                   w13.stride(0), F2, F, word(status.t), stream()),
          "gemm2_swiglu");
    auto shape = x.sizes().vec();
    shape.back() = w2.size(0);
    Tensor y = bf16(shape, x);
    gemm(h, w2, y.view({-1, w2.size(0)}), false, false, 0, status.t);
    ctx->save_for_backward({x, w13, w2, gu, h});
    keep(ctx, "buffer13", buffer13);
    keep(ctx, "buffer2", buffer2);
    keep(ctx, "status", status);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &w13 = s[1], &w2 = s[2], &gu = s[3], &h = s[4];
    const Tensor status = aside(ctx, "status");
    const Tensor dy2 = dense(rows(g[0])), x2 = rows(x);
    const ll T = gu.size(0), F = gu.size(1) / 2;
    Tensor dgu = at::empty_like(gu);
    check(E.swiglu_bwd(dy2.data_ptr(), w2.data_ptr(), gu.data_ptr(), dgu.data_ptr(), (int)T, (int)F, (int)dy2.size(1), dy2.stride(0),
                       w2.stride(0), gu.stride(0), dgu.stride(0), word(status), stream()),
          "gemm2_swiglu_bwd");
    Tensor dw2 = weight_grad(aside(ctx, "buffer2"), dy2, h, w2, ctx->needs_input_grad(2), status);
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      dx = bf16(x.sizes(), x);
      gemm(dgu, w13, dx.view({-1, w13.size(1)}), false, true, 0, status);
    }
    Tensor dw13 = weight_grad(aside(ctx, "buffer13"), dgu, x2, w13, ctx->needs_input_grad(1), status);
    return {dx, dw13, dw2, Tensor(), Tensor(), Tensor()};
  }
};

struct AttentionBlock : Function<AttentionBlock> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& wqkv, const Tensor& wo, Aside buffer_qkv, Aside buffer_o,
                        Aside cos, Aside sin, int64_t heads, int64_t kv, int64_t hd, Aside status) {
    const ll B = x.size(0), S = x.size(1), C = wqkv.size(0), N = heads * hd;
    const Tensor x2 = rows(x);
    Tensor qkv = bf16({B, S, C}, x);
    check(E.gemm_rope(x2.data_ptr(), wqkv.data_ptr(), qkv.data_ptr(), (int)x2.size(0), (int)C, (int)x2.size(1), x2.stride(0),
                      wqkv.stride(0), C, cos.t.data_ptr<float>(), sin.t.data_ptr<float>(), (int)S, (int)((heads + kv) * hd), (int)hd,
                      word(status.t), stream()),
          "gemm2_rope");
    Tensor out = bf16({B, S, N}, x), lse = f32({B, heads, S}, x);
    check(E.attention_fwd(qkv.data_ptr(), out.data_ptr(), lse.data_ptr<float>(), (int)B, (int)S, (int)heads, (int)kv, (int)hd, C, N,
                          (float)std::pow((double)hd, -0.5), word(status.t), stream()),
          "attention_fwd");
    Tensor y = bf16({B, S, wo.size(0)}, x);
    gemm(out.view({-1, N}), wo, y.view({-1, wo.size(0)}), false, false, 0, status.t);
    ctx->save_for_backward({x, wqkv, wo, qkv, out, lse, cos.t, sin.t});
    keep(ctx, "buffer_qkv", buffer_qkv);
    keep(ctx, "buffer_o", buffer_o);
    keep(ctx, "status", status);
    ctx->saved_data["dims"] = std::vector<int64_t>{heads, kv, hd};
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &wqkv = s[1], &wo = s[2], &qkv = s[3], &out = s[4], &lse = s[5], &cos = s[6], &sin = s[7];
    const auto dims = ctx->saved_data["dims"].toIntVector();
    const int64_t heads = dims[0], kv = dims[1], hd = dims[2];
    const Tensor status = aside(ctx, "status");
    const ll B = qkv.size(0), S = qkv.size(1), C = qkv.size(2), T = B * S, N = heads * hd;
    const Tensor dy2 = dense(rows(g[0])), out2 = out.view({T, N});
    Tensor dO = bf16({T, N}, qkv), delta = f32({B, heads, S}, qkv);
    check(E.attn_dout(dy2.data_ptr(), wo.data_ptr(), out2.data_ptr(), dO.data_ptr(), delta.data_ptr<float>(), (int)T, (int)N,
                      (int)dy2.size(1), (int)S, (int)hd, dy2.stride(0), wo.stride(0), out2.stride(0), dO.stride(0), word(status),
                      stream()),
          "gemm2_attn_dout");
    Tensor dwo = weight_grad(aside(ctx, "buffer_o"), dy2, out2, wo, ctx->needs_input_grad(2), status);
    Tensor dqkv = at::empty_like(qkv);
    {
      Tensor scratch = f32({T * E.bwd_scratch_cols((int)B, (int)S, (int)heads, (int)kv, (int)hd)}, qkv);
      scratch.narrow(0, 0, T * N).zero_();                   // dQ accumulates; the parts behind it are written whole
      check(E.attention_bwd(qkv.data_ptr(), out.data_ptr(), dO.data_ptr(), lse.data_ptr<float>(), delta.data_ptr<float>(),
                            scratch.data_ptr<float>(), dqkv.data_ptr(), (int)B, (int)S, (int)heads, (int)kv, (int)hd, C, N,
                            (float)std::pow((double)hd, -0.5), cos.data_ptr<float>(), sin.data_ptr<float>(), word(status), stream()),
            "attention_bwd_unrope_delta");
    }
    const Tensor d2 = dqkv.view({T, C}), x2 = rows(x);
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      dx = bf16(x.sizes(), x);
      gemm(d2, wqkv, dx.view({-1, wqkv.size(1)}), false, true, 0, status);
    }
    Tensor dwqkv = weight_grad(aside(ctx, "buffer_qkv"), d2, x2, wqkv, ctx->needs_input_grad(1), status);
    return {dx, dwqkv, dwo, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Aside opt(const std::optional<Tensor>& t) { return Aside{t ? *t : Tensor()}; }

}  // namespace

PYBIND11_MODULE(tplr_host, m) {
  typedef py::call_guard<py::gil_scoped_release> nogil;
  m.def("bind", &bind);
  m.def("launches", [] { return g_launches.load(std::memory_order_relaxed); });
  m.def("rmsnorm", [](const Tensor& x, const Tensor& w, const std::optional<Tensor>& buffer, double eps, const Tensor& status) {
    return RMSNorm::apply(x, w, opt(buffer), eps, Aside{status});
  }, nogil());
  m.def("add_rmsnorm", [](const Tensor& res, const Tensor& delta, const Tensor& w, const std::optional<Tensor>& buffer, double eps,
                          const Tensor& status) {
    auto r = AddRMSNorm::apply(res, delta, w, opt(buffer), eps, Aside{status});
    return std::make_tuple(r[0], r[1]);
  }, nogil());
  m.def("linear", [](const Tensor& x, const Tensor& w, const std::optional<Tensor>& buffer, const Tensor& status) {
    return Linear::apply(x, w, opt(buffer), Aside{status});
  }, nogil());
  m.def("feed_forward", [](const Tensor& x, const Tensor& w13, const Tensor& w2, const std::optional<Tensor>& b13,
                           const std::optional<Tensor>& b2, const Tensor& status) {
    return FeedForward::apply(x, w13, w2, opt(b13), opt(b2), Aside{status});
  }, nogil());
  m.def("attention_block", [](const Tensor& x, const Tensor& wqkv, const Tensor& wo, const std::optional<Tensor>& bq,
                              const std::optional<Tensor>& bo, const Tensor& cos, const Tensor& sin, int64_t heads, int64_t kv,
                              int64_t hd, const Tensor& status) {
    return AttentionBlock::apply(x, wqkv, wo, opt(bq), opt(bo), Aside{cos}, Aside{sin}, heads, kv, hd, Aside{status});
  }, nogil());
}
