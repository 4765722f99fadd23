// Host path of the differentiable ops: the autograd nodes of ops/functional.py in C++, calling the same kernels of liblightron_b200.so.
//
// Why: a small call is bound by its host work.  Of 395 us for one attention layer of 4 x 128 tokens forward and backward, 61 are kernels; an
// autograd function written in Python costs some 20 us forward and 60 us backward besides its launches (6 us each), a node here about 5.
//
// Every function takes the plain case (exact tensors or parameters, CUDA, bf16, contiguous, adjacent weights) and answers
// NotImplemented for anything else, as also under function transforms, forward-mode derivatives, tracing and dispatch or function modes: the
// caller then runs the autograd function in Python, which accepts, refuses and traces what it always did.  Outputs, streams, version checks and
// error types are the same in both forms, and saved-tensor hooks see the same tensors (an input in its own shape, not flattened to rows).  What such hooks
// give back is looked at again in backward (operand(), fused_rows()).  Weights whose gradients go straight into the optimizer's arena stay with
// the Python form.
#include <Python.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <atomic>
#include <climits>
#include <cstdlib>
#include <cstring>

namespace {
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

// ---- the kernels' entry points -------------------------------------------------------------------
typedef const void* P;
typedef void* W;
typedef long long L;
struct Api {
  int (*lb_rmsnorm_fwd)(P, P, P, W, W, W, int, int, float, W);
  int (*lb_rmsnorm_bwd_blocks)(int, int);
  int (*lb_rmsnorm_bwd)(P, P, P, P, P, W, W, W, int, int, int, W);
  int (*lb_rope)(W, P, P, P, int, int, int, int, L, int, W);
  int (*lb_gemm_grouped_epi)(int, const P*, const P*, const W*, const int*, const int*, const int*, const L*, const L*, const L*, const int*,
                             const int*, const int*, const int*, const W*, const L*, const int*, W);
  int (*lb_flash_fwd_tc)(P, P, P, W, W, int, int, int, int, int, int, L, L, L, L, float, int, W);
  L (*lb_flash_bwd_ws_bytes_kv)(int, int, int, int, int, int, int);
  int (*lb_flash_bwd_tc_ws)(P, P, P, P, P, P, W, L, W, W, W, int, int, int, int, int, int, L, L, L, L, L, L, L, L, float, int, W);
  int (*lb_flash_bwd)(P, P, P, P, P, P, W, W, W, W, W, int, int, int, int, int, int, L, L, L, L, L, L, L, L, float, int, W);
  int (*lb_embedding_fwd)(P, P, W, int, int, int, int, W);
  int (*lb_clear)(W, L, W);
  int (*lb_embedding_bwd)(P, P, W, int, int, int, int, W);
  int (*lb_ce_stats)(P, P, W, W, W, int, int, L, int, W);
  int (*lb_ce_loss)(P, W, P, P, W, W, int, float, int, W);
  int (*lb_ce_grad)(P, P, P, W, P, int, int, L, int, float, int, W);
  int (*lb_gemm_rope)(P, P, W, int, int, int, P, P, P, int, int, int, W);
} api;
PyObject* raise_error = nullptr;                 // (name, code): raises the error of ops/native.py
PyObject* direct_grad = nullptr;                 // the attribute of a weight whose gradient the optimizer keeps
std::atomic<unsigned long long> g_launches{0};

void check(const char* name, int rc) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (rc == 0) return;
  pybind11::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(raise_error, "si", name, rc);
  Py_XDECREF(r);
  python_error err;
  err.persist();
  throw err;
}
#define LB_CALL(fn, ...) check(#fn, api.fn(__VA_ARGS__))

W stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
bool env_is_tc(const char* name) {
  const char* v = std::getenv(name);
  return v == nullptr || std::strcmp(v, "tc") == 0;
}
Tensor empty(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options()); }
Tensor empty_f32(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().dtype(at::kFloat)); }

// ---- GEMM launches -------------------------------------------------------------------------------
struct Gemms {
  int n = 0;
  P A[2], B[2];
  W C[2], C2[2];
  int M[2], N[2], K[2], a_mn[2], b_mn[2], acc[2], epi[2], half[2];
  L lda[2], ldb[2], ldc[2], ldc2[2];
  // C [m, n] = op(a) op(b)^T, all matrices contiguous; epilogues as in gemm_grouped.cu
  void add(const Tensor& a, const Tensor& b, const Tensor& c, L m, L nn, L k, bool amn, bool bmn, int e = 0, const Tensor* c2 = nullptr, L hf = 0) {
    const int i = n++;
    A[i] = a.const_data_ptr(); B[i] = b.const_data_ptr(); C[i] = c.mutable_data_ptr();
    M[i] = (int)m; N[i] = (int)nn; K[i] = (int)k;
    a_mn[i] = amn; b_mn[i] = bmn; acc[i] = 0; epi[i] = e; half[i] = (int)hf;
    lda[i] = amn ? m : k; ldb[i] = bmn ? nn : k; ldc[i] = e == 2 ? 2 * hf : nn;
    C2[i] = c2 ? c2->mutable_data_ptr() : nullptr;
    ldc2[i] = e == 1 ? hf : (e == 2 ? 2 * hf : 0);
  }
  void run() { LB_CALL(lb_gemm_grouped_epi, n, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, acc, epi, C2, ldc2, half, stream()); }
};

L rows_of(const Tensor& t) { return t.numel() / t.size(-1); }
std::vector<int64_t> with_last(const Tensor& x, int64_t n) {
  std::vector<int64_t> s = x.sizes().vec();
  s.back() = n;
  return s;
}

// ---- saved tensors -------------------------------------------------------------------------------
// Saved-tensor hooks (and an assignment to a parameter's .data) may put another tensor in the place of a saved one, which a kernel would
// read past its end.  Copies and other strides are fine; other sizes, types or devices are refused.  `last`: size of the last dimension, or -1.
void check_saved(const Tensor& t, const Tensor& grad, at::ScalarType type, L numel, L last) {
  TORCH_CHECK(t.defined() && t.has_storage() && t.device() == grad.device() && t.scalar_type() == type && t.numel() == numel &&
                  (last < 0 || (t.dim() > 0 && t.size(-1) == last)),
              "a tensor saved for backward has come back with another size, type or device");
}
Tensor operand(const Tensor& t, const Tensor& grad, L numel, L last, at::ScalarType type = at::kBFloat16) {
  check_saved(t, grad, type, numel, last);
  return t.contiguous();
}
// [n_i, K] matrices back to back in one buffer
bool rows_adjacent(const Tensor* const* ws, size_t n) {
  for (size_t i = 0; i + 1 < n; i++) {
    const Tensor &a = *ws[i], &b = *ws[i + 1];
    if (a.storage().data() != b.storage().data()) return false;
    if (static_cast<const char*>(a.const_data_ptr()) + a.numel() * 2 != b.const_data_ptr()) return false;
  }
  return true;
}
// The matrix [W_0; W_1; ...] of n rows that the forward pass read, given by the first of its parts.  Parts that no longer follow one another
// (each unpacked into memory of its own, as save_on_cpu() does) are refused, as the Python form's view of them is.
Tensor fused_rows(const Tensor* ws, size_t nw, const Tensor& grad, L n, L K) {
  const Tensor* p[3];
  L rows = 0;
  for (size_t i = 0; i < nw; i++) {
    check_saved(ws[i], grad, at::kBFloat16, ws[i].defined() ? ws[i].numel() : -1, K);
    TORCH_CHECK(ws[i].dim() == 2 && (nw == 1 || ws[i].is_contiguous()), "a weight saved for backward has come back with other strides");
    rows += ws[i].size(0);
    p[i] = &ws[i];
  }
  TORCH_CHECK(rows == n && rows_adjacent(p, nw), "adjacent weights saved for backward have come back as separate tensors");
  return ws[0].contiguous();
}

// Gradients of y = x [W_0; W_1; ...]^T: dx (or undefined), then one per weight
variable_list linear_backward(const Tensor& saved_x, const Tensor* ws, size_t nw, const Tensor& dy, bool need_x, bool need_w) {
  const L n = dy.size(-1), T = rows_of(dy), K = saved_x.size(-1);
  const Tensor x = operand(saved_x, dy, T * K, K);
  variable_list out(1 + nw);
  Gemms g;
  Tensor dw;
  if (need_w) {          // first: its tiles are the longest
    dw = empty({n, K}, x);
    g.add(dy, x, dw, n, K, T, true, true);
  }
  Tensor w;
  if (need_x) {
    w = fused_rows(ws, nw, dy, n, K);
    out[0] = at::empty(x.sizes(), x.options());
    g.add(dy, w, out[0], T, K, n, false, true);
  }
  if (g.n) g.run();
  L off = 0;
  for (size_t i = 0; need_w && i < nw; i++) {
    out[1 + i] = nw == 1 ? dw : dw.narrow(0, off, ws[i].size(0));
    off += ws[i].size(0);
  }
  return out;
}

struct Linear : Function<Linear> {
  template <typename... Ts>                      // one argument per weight: autograd gives a list of tensors no edges
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w0, const Ts&... ws) {
    const L n = (w0.size(0) + ... + ws.size(0));
    Tensor y = empty(with_last(x, n), x);
    Gemms g;
    g.add(x, w0, y, rows_of(x), n, x.size(-1), false, false);
    g.run();
    ctx->save_for_backward({x, w0, ws...});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    bool need_w = false;
    for (size_t i = 1; i < s.size(); i++) need_w |= ctx->needs_input_grad(i);
    return linear_backward(s[0], s.data() + 1, s.size() - 1, grads[0].contiguous(), ctx->needs_input_grad(0), need_w);
  }
};

struct SwiGLUMLP : Function<SwiGLUMLP> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const Tensor& w3, const Tensor& w2) {
    const L T = rows_of(x), I = w1.size(0);
    Tensor gu = empty({T, 2 * I}, x), h = empty({T, I}, x), y = empty(with_last(x, w2.size(0)), x);
    Gemms g;
    g.add(x, w1, gu, T, 2 * I, x.size(-1), false, false, 1, &h, I);
    g.run();
    Gemms d;
    d.add(h, w2, y, T, w2.size(0), I, false, false);
    d.run();
    ctx->save_for_backward({x, gu, h, w1, w3, w2});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor& x = s[0];
    const Tensor dy = grads[0].contiguous();
    const L T = rows_of(dy), I = s[2].size(-1), H = dy.size(-1);
    const Tensor gu = operand(s[1], dy, T * 2 * I, 2 * I), h = operand(s[2], dy, T * I, I), w2 = operand(s[5], dy, H * I, I);
    Tensor dgu = at::empty(gu.sizes(), gu.options()), dw2;
    Gemms g;
    if (ctx->needs_input_grad(3)) {
      dw2 = empty({H, I}, x);
      g.add(dy, h, dw2, H, I, T, true, true);
    }
    g.add(dy, w2, dgu, T, I, H, false, true, 2, &gu, I);
    g.run();
    variable_list r = linear_backward(x, s.data() + 3, 2, dgu, ctx->needs_input_grad(0), ctx->needs_input_grad(1) || ctx->needs_input_grad(2));
    r.push_back(dw2);
    return r;
  }
};

// ---- RMSNorm -------------------------------------------------------------------------------------
variable_list rmsnorm_backward(const variable_list& saved, const Tensor* dh, const Tensor& dy) {
  const int rows = (int)rows_of(dy), cols = (int)dy.size(-1), nblk = api.lb_rmsnorm_bwd_blocks(rows, cols);
  const Tensor src = operand(saved[0], dy, dy.numel(), cols), w = operand(saved[1], dy, cols, cols), rstd = operand(saved[2], dy, rows, rows, at::kFloat);
  const Tensor dyc = dy.contiguous(), dhc = dh ? dh->contiguous() : Tensor();
  Tensor partial = empty_f32({nblk, cols}, src), dx = at::empty(src.sizes(), src.options()), dw = at::empty(w.sizes(), w.options());
  LB_CALL(lb_rmsnorm_bwd, dyc.const_data_ptr(), src.const_data_ptr(), w.const_data_ptr(), rstd.const_data_ptr(),
          dh ? dhc.const_data_ptr() : nullptr, dx.mutable_data_ptr(), partial.mutable_data_ptr(), dw.mutable_data_ptr(), rows, cols, nblk, stream());
  return {dx, dw};
}
struct RMSNorm : Function<RMSNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    Tensor y = at::empty(x.sizes(), x.options()), rstd = empty_f32({rows_of(x)}, x);
    LB_CALL(lb_rmsnorm_fwd, x.const_data_ptr(), nullptr, w.const_data_ptr(), nullptr, y.mutable_data_ptr(), rstd.mutable_data_ptr(),
            (int)rows_of(x), (int)x.size(-1), (float)eps, stream());
    ctx->save_for_backward({x, w, rstd});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    variable_list r = rmsnorm_backward(s, nullptr, grads[0]);
    r.push_back(Tensor());
    return r;
  }
};
struct AddRMSNorm : Function<AddRMSNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& res, const Tensor& w, double eps) {
    Tensor h = at::empty(x.sizes(), x.options()), y = at::empty(x.sizes(), x.options()), rstd = empty_f32({rows_of(x)}, x);
    LB_CALL(lb_rmsnorm_fwd, x.const_data_ptr(), res.const_data_ptr(), w.const_data_ptr(), h.mutable_data_ptr(), y.mutable_data_ptr(),
            rstd.mutable_data_ptr(), (int)rows_of(x), (int)x.size(-1), (float)eps, stream());
    ctx->save_for_backward({h, w, rstd});
    return {h, y};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    const variable_list r = rmsnorm_backward(s, &grads[0], grads[1]);
    return {r[0], r[0], r[1], Tensor()};
  }
};

// ---- attention -----------------------------------------------------------------------------------
// [B, S, h, d] with unit inner stride, head stride d, batch stride S * token stride, 16-byte rows
bool layout_ok(const Tensor& t) {
  return t.stride(3) == 1 && t.stride(2) == t.size(3) && (t.size(0) == 1 || t.stride(0) == t.size(1) * t.stride(1)) && t.stride(1) % 8 == 0 &&
         ((uintptr_t)t.const_data_ptr() & 15) == 0;
}
Tensor fix_layout(const Tensor& t) { return layout_ok(t) ? t : t.contiguous(); }

struct Heads { P p; L ts; };                     // first element and token stride of [B, S, heads, d]
struct AttnDims { int B, Sq, Sk, hq, hkv, d, causal; float scale; };

void attention_forward(const Heads& q, const Heads& k, const Heads& v, const Tensor& o, const Tensor& lse, const AttnDims& m) {
  LB_CALL(lb_flash_fwd_tc, q.p, k.p, v.p, o.mutable_data_ptr(), lse.mutable_data_ptr(), m.B, m.Sq, m.Sk, m.hq, m.hkv, m.d, q.ts, k.ts, v.ts,
          (L)m.hq * m.d, m.scale, m.causal, stream());
}
void attention_backward(const Heads& q, const Heads& k, const Heads& v, const Tensor& saved_o, const Tensor& saved_lse, const Tensor& grad,
                        const Heads& dout, W dq, W dk, W dv, L dq_ts, L dk_ts, L dv_ts, const AttnDims& m) {
  const L o_ts = (L)m.hq * m.d, rows = (L)m.B * m.Sq;
  const Tensor o = operand(saved_o, grad, rows * o_ts, -1), lse = operand(saved_lse, grad, rows * m.hq, m.Sq, at::kFloat);
  if (env_is_tc("LIGHTRON_FA_BWD")) {
    const L bytes = api.lb_flash_bwd_ws_bytes_kv(m.B, m.Sq, m.Sk, m.hq, m.hkv, m.d, m.causal);
    Tensor ws = at::empty({bytes}, o.options().dtype(at::kByte));
    LB_CALL(lb_flash_bwd_tc_ws, q.p, k.p, v.p, o.const_data_ptr(), dout.p, lse.const_data_ptr(), ws.mutable_data_ptr(), bytes, dq, dk, dv, m.B, m.Sq,
            m.Sk, m.hq, m.hkv, m.d, q.ts, k.ts, v.ts, o_ts, dout.ts, dq_ts, dk_ts, dv_ts, m.scale, m.causal, stream());
  } else {
    Tensor delta = empty_f32({m.B, m.hq, m.Sq}, o), acc = at::zeros({(L)m.B * m.Sq * m.hq * m.d}, o.options().dtype(at::kFloat));
    LB_CALL(lb_flash_bwd, q.p, k.p, v.p, o.const_data_ptr(), dout.p, lse.const_data_ptr(), delta.mutable_data_ptr(), acc.mutable_data_ptr(), dq, dk,
            dv, m.B, m.Sq, m.Sk, m.hq, m.hkv, m.d, q.ts, k.ts, v.ts, o_ts, dout.ts, dq_ts, dk_ts, dv_ts, m.scale, m.causal, stream());
  }
}

AttnDims dims_of(const Tensor& q, const Tensor& k, bool causal, double scale) {
  return {(int)q.size(0), (int)q.size(1), (int)k.size(1), (int)q.size(2), (int)k.size(2), (int)q.size(3), causal ? 1 : 0, (float)scale};
}
struct Attention : Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q0, const Tensor& k0, const Tensor& v0, bool causal, double scale) {
    const Tensor q = fix_layout(q0), k = fix_layout(k0), v = fix_layout(v0);
    const AttnDims m = dims_of(q, k, causal, scale);
    Tensor o = empty(q0.sizes(), q0), lse = empty_f32({m.B, m.hq, m.Sq}, q0);
    attention_forward({q.const_data_ptr(), q.stride(1)}, {k.const_data_ptr(), k.stride(1)}, {v.const_data_ptr(), v.stride(1)}, o, lse, m);
    ctx->save_for_backward({q0, k0, v0, o, lse});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor& g = grads[0];
    check_saved(s[0], g, at::kBFloat16, g.numel(), g.size(3));
    for (int i = 1; i < 3; i++) check_saved(s[i], g, at::kBFloat16, s[1].defined() ? s[1].numel() : -1, g.size(3));
    TORCH_CHECK(s[0].sizes().equals(g.sizes()) && s[1].dim() == 4 && s[2].sizes().equals(s[1].sizes()) && s[1].size(0) == g.size(0) &&
                    s[1].numel() > 0 && g.size(2) % s[1].size(2) == 0,
                "q, k or v saved for backward has come back with another shape");
    const Tensor q = fix_layout(s[0]), k = fix_layout(s[1]), v = fix_layout(s[2]), dout = fix_layout(g);
    const AttnDims m = dims_of(q, k, ctx->saved_data["causal"].toBool(), ctx->saved_data["scale"].toDouble());
    Tensor dq = empty(q.sizes(), q), dk = empty(k.sizes(), k), dv = empty(v.sizes(), v);
    attention_backward({q.const_data_ptr(), q.stride(1)}, {k.const_data_ptr(), k.stride(1)}, {v.const_data_ptr(), v.stride(1)}, s[3], s[4], g,
                       {dout.const_data_ptr(), dout.stride(1)}, dq.mutable_data_ptr(), dk.mutable_data_ptr(), dv.mutable_data_ptr(), dq.stride(1),
                       dk.stride(1), dv.stride(1), m);
    return {dq, dk, dv, Tensor(), Tensor()};
  }
};

// RoPE + causal attention on the fused projection's output, which is rotated in place without telling autograd (the caller hands it over)
struct Dims { int64_t v[5]; };                   // B, S, hq, hkv, d (one argument to autograd; a vector would count as five)
struct RopeAttention : Function<RopeAttention> {
  static W at_head(const Tensor& t, L head, L d) { return static_cast<char*>(t.mutable_data_ptr()) + head * d * 2; }
  static void rope(const Tensor& t, const Tensor& cos, const Tensor& sin, const Tensor& positions, L S, L heads, L d, L row, int inverse) {
    LB_CALL(lb_rope, t.mutable_data_ptr(), cos.const_data_ptr(), sin.const_data_ptr(), positions.defined() ? positions.const_data_ptr() : nullptr,
            (int)(t.numel() / row), (int)S, (int)heads, (int)d, row, inverse, stream());
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& cos, const Tensor& sin, const std::optional<Tensor>& positions,
                        Dims dims, double scale) {
    const L B = dims.v[0], S = dims.v[1], hq = dims.v[2], hkv = dims.v[3], d = dims.v[4], row = (hq + 2 * hkv) * d;
    const Tensor pos = positions.value_or(Tensor());
    rope(qkv, cos, sin, pos, S, hq + hkv, d, row, 0);
    Tensor o = empty({B * S, hq * d}, qkv), lse = empty_f32({B, hq, S}, qkv);
    const AttnDims m{(int)B, (int)S, (int)S, (int)hq, (int)hkv, (int)d, 1, (float)scale};
    attention_forward({at_head(qkv, 0, d), row}, {at_head(qkv, hq, d), row}, {at_head(qkv, hq + hkv, d), row}, o, lse, m);
    ctx->save_for_backward({qkv, o, lse, cos, sin, pos});
    ctx->saved_data["dims"] = std::vector<int64_t>{B, S, hq, hkv, d, cos.numel(), sin.numel()};
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    const std::vector<int64_t> dims = ctx->saved_data["dims"].toIntVector();
    const L B = dims[0], S = dims[1], hq = dims[2], hkv = dims[3], d = dims[4], row = (hq + 2 * hkv) * d;
    const AttnDims m{(int)B, (int)S, (int)S, (int)hq, (int)hkv, (int)d, 1, (float)ctx->saved_data["scale"].toDouble()};
    const Tensor& g = grads[0];
    const Tensor qkv = operand(s[0], g, B * S * row, row), cos = operand(s[3], g, dims[5], d / 2, at::kFloat), sin = operand(s[4], g, dims[6], d / 2, at::kFloat);
    const Tensor pos = s[5].defined() ? operand(s[5], g, S, -1, at::kInt) : Tensor();
    const Tensor dout = fix_layout(g.reshape({B, S, hq, d}));
    Tensor dqkv = at::empty(qkv.sizes(), qkv.options());
    attention_backward({at_head(qkv, 0, d), row}, {at_head(qkv, hq, d), row}, {at_head(qkv, hq + hkv, d), row}, s[1], s[2], g,
                       {dout.const_data_ptr(), dout.stride(1)}, at_head(dqkv, 0, d), at_head(dqkv, hq, d), at_head(dqkv, hq + hkv, d), row, row, row, m);
    rope(dqkv, cos, sin, pos, S, hq + hkv, d, row, 1);
    return {dqkv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- embedding, loss -----------------------------------------------------------------------------
struct Embedding : Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& tok, const Tensor& w, int64_t v0) {
    const L H = w.size(1);
    std::vector<int64_t> sizes = tok.sizes().vec();
    sizes.push_back(H);
    Tensor out = empty(sizes, w);
    LB_CALL(lb_embedding_fwd, tok.const_data_ptr(), w.const_data_ptr(), out.mutable_data_ptr(), (int)tok.numel(), (int)H, (int)v0,
            (int)(v0 + w.size(0)), stream());
    ctx->save_for_backward({tok});
    ctx->saved_data["shape"] = std::vector<int64_t>{w.size(0), H, v0};
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const std::vector<int64_t> s = ctx->saved_data["shape"].toIntVector();
    const Tensor dy = grads[0].contiguous(), tok = operand(ctx->get_saved_variables()[0], dy, dy.numel() / s[1], -1, at::kLong);
    Tensor dw = empty({s[0], s[1]}, dy);
    LB_CALL(lb_clear, dw.mutable_data_ptr(), (L)dw.nbytes(), stream());
    LB_CALL(lb_embedding_bwd, tok.const_data_ptr(), dy.const_data_ptr(), dw.mutable_data_ptr(), (int)tok.numel(), (int)s[1], (int)s[2],
            (int)(s[2] + s[0]), stream());
    return {Tensor(), dw, Tensor()};
  }
};

struct CrossEntropy : Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& tgt, int64_t v0, int64_t n_valid, int64_t ignore) {
    const L T = logits.size(0), V = logits.size(1);
    Tensor mx = empty_f32({T}, logits), se = empty_f32({T}, logits), tl = empty_f32({T}, logits), lse = empty_f32({T}, logits), loss = empty_f32({}, logits);
    LB_CALL(lb_ce_stats, logits.const_data_ptr(), tgt.const_data_ptr(), mx.mutable_data_ptr(), se.mutable_data_ptr(), tl.mutable_data_ptr(), (int)T,
            (int)V, logits.stride(0), (int)v0, stream());
    LB_CALL(lb_ce_loss, mx.const_data_ptr(), se.mutable_data_ptr(), tl.const_data_ptr(), tgt.const_data_ptr(), lse.mutable_data_ptr(),
            loss.mutable_data_ptr(), (int)T, inv_n(n_valid), (int)ignore, stream());
    ctx->save_for_backward({logits, tgt, lse});
    ctx->saved_data["meta"] = std::vector<int64_t>{v0, n_valid, ignore, T, V};
    return loss;
  }
  static float inv_n(int64_t n) { return (float)(1.0 / (double)std::max<int64_t>(n, 1)); }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const variable_list s = ctx->get_saved_variables();
    const std::vector<int64_t> m = ctx->saved_data["meta"].toIntVector();
    const Tensor dl = grads[0].to(at::kFloat).reshape({1}).contiguous();         // read on the device: no host sync
    const L T = m[3], V = m[4];
    check_saved(s[0], grads[0], at::kBFloat16, T * V, V);
    TORCH_CHECK(s[0].dim() == 2, "logits saved for backward have come back with another shape");
    const Tensor logits = s[0].stride(1) == 1 ? s[0] : s[0].contiguous();
    const Tensor tgt = operand(s[1], grads[0], T, T, at::kLong), lse = operand(s[2], grads[0], T, T, at::kFloat);
    // the gradient overwrites the logits, which are dead after the loss
    LB_CALL(lb_ce_grad, logits.const_data_ptr(), tgt.const_data_ptr(), lse.const_data_ptr(), logits.mutable_data_ptr(), dl.const_data_ptr(), (int)T,
            (int)V, logits.stride(0), (int)m[0], inv_n(m[1]), (int)m[2], stream());
    return {logits, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- what is plain -------------------------------------------------------------------------------
const Tensor* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

// CUDA, bf16, dense, without a forward-mode derivative
bool plain(const Tensor* t, bool contiguous = true) {
  return t && t->defined() && t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->layout() == at::kStrided && !t->is_neg() &&
         (!contiguous || t->is_contiguous()) && t->numel() > 0 && !t->_fw_grad(0).defined();
}
bool fits_int(std::initializer_list<int64_t> v) {
  for (int64_t x : v) if (x < 0 || x > INT_MAX) return false;
  return true;
}
// Nothing looks at the calls of this thread that only an autograd function in Python would show them
bool unobserved() {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() || torch::jit::tracer::isTracing()) return false;
  const auto keys = c10::impl::tls_local_dispatch_key_set().included_;
  return !keys.has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode,
                                            c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize, c10::DispatchKey::Python}));
}
// A weight that the optimizer's arena backs: its gradient is accumulated by the Python form
bool in_arena(PyObject* o, const Tensor& w) {
  if (!w.requires_grad() || !at::GradMode::is_enabled()) return false;
  PyObject* a = PyObject_GetAttr(o, direct_grad);
  if (!a) { PyErr_Clear(); return false; }
  const int yes = PyObject_IsTrue(a);
  Py_DECREF(a);
  if (yes < 0) PyErr_Clear();                    // the Python form asks again, and raises
  return yes != 0;
}
bool weight_ok(const Tensor* w, int64_t K) {
  return plain(w) && w->dim() == 2 && w->size(1) == K && w->size(0) % 8 == 0 && w->size(0) <= INT_MAX;
}
#define LB_NOT_PLAIN Py_RETURN_NOTIMPLEMENTED
// Runs a node without the interpreter's lock, as torch's own ops run: allocations and launches may block.  The node takes its tensors by value.
template <typename F>
auto unlocked(F f) {
  pybind11::gil_scoped_release release;
  return f();
}

PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 2 || n > 4 || !unobserved()) LB_NOT_PLAIN;
  const Tensor* x = tensor(a[0]);
  if (!plain(x) || x->dim() < 1) LB_NOT_PLAIN;
  const int64_t K = x->size(-1);
  if (K % 8 || !fits_int({K, rows_of(*x)})) LB_NOT_PLAIN;
  const Tensor* ws[3];
  const size_t nw = (size_t)n - 1;
  int64_t total = 0;
  for (size_t i = 0; i < nw; i++) {
    ws[i] = tensor(a[1 + i]);
    if (!weight_ok(ws[i], K) || in_arena(a[1 + i], *ws[i])) LB_NOT_PLAIN;
    total += ws[i]->size(0);
  }
  if (!rows_adjacent(ws, nw) || !fits_int({total})) LB_NOT_PLAIN;
  const Tensor w0 = *ws[0], w1 = nw > 1 ? *ws[1] : Tensor(), w2 = nw > 2 ? *ws[2] : Tensor();
  return THPVariable_Wrap(unlocked([&, x = *x] {
    return nw == 1 ? Linear::apply(x, w0) : nw == 2 ? Linear::apply(x, w0, w1) : Linear::apply(x, w0, w1, w2);
  }));
  END_HANDLE_TH_ERRORS
}

PyObject* py_swiglu_mlp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !unobserved()) LB_NOT_PLAIN;
  const Tensor *x = tensor(a[0]), *w1 = tensor(a[1]), *w3 = tensor(a[2]), *w2 = tensor(a[3]);
  if (!plain(x) || x->dim() < 1 || x->size(-1) % 8 || !fits_int({x->size(-1), rows_of(*x)})) LB_NOT_PLAIN;
  if (!weight_ok(w1, x->size(-1)) || !weight_ok(w3, x->size(-1)) || w1->size(0) != w3->size(0) || !weight_ok(w2, w1->size(0))) LB_NOT_PLAIN;
  const Tensor* up[2] = {w1, w3};
  if (!rows_adjacent(up, 2) || !fits_int({2 * w1->size(0)}) || in_arena(a[1], *w1) || in_arena(a[2], *w3) || in_arena(a[3], *w2)) LB_NOT_PLAIN;
  return THPVariable_Wrap(unlocked([x = *x, w1 = *w1, w3 = *w3, w2 = *w2] { return SwiGLUMLP::apply(x, w1, w3, w2); }));
  END_HANDLE_TH_ERRORS
}

// (x, res or None, w, eps) -> y, or (h, y)
PyObject* py_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !PyFloat_Check(a[3]) || !unobserved()) LB_NOT_PLAIN;
  const Tensor *x = tensor(a[0]), *res = a[1] == Py_None ? nullptr : tensor(a[1]), *w = tensor(a[2]);
  if (!plain(x) || x->dim() < 1 || !fits_int({x->size(-1), rows_of(*x)}) || !plain(w) || w->dim() != 1 || w->size(0) != x->size(-1)) LB_NOT_PLAIN;
  if (a[1] != Py_None && (!plain(res) || !res->sizes().equals(x->sizes()))) LB_NOT_PLAIN;
  const double eps = PyFloat_AsDouble(a[3]);
  if (!res) return THPVariable_Wrap(unlocked([x = *x, w = *w, eps] { return RMSNorm::apply(x, w, eps); }));
  variable_list r = unlocked([x = *x, res = *res, w = *w, eps] { return AddRMSNorm::apply(x, res, w, eps); });
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  for (int i = 0; i < 2; i++) PyTuple_SET_ITEM(t, i, THPVariable_Wrap(std::move(r[i])));
  return t;
  END_HANDLE_TH_ERRORS
}

bool attention_plain(const Tensor* t) { return plain(t, false) && t->dim() == 4; }

PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5 || !PyBool_Check(a[3]) || !PyFloat_Check(a[4]) || !unobserved() || !env_is_tc("LIGHTRON_FA")) LB_NOT_PLAIN;
  const Tensor *q = tensor(a[0]), *k = tensor(a[1]), *v = tensor(a[2]);
  if (!attention_plain(q) || !attention_plain(k) || !attention_plain(v)) LB_NOT_PLAIN;
  const int64_t d = q->size(3);
  const bool causal = a[3] == Py_True;
  if ((d != 64 && d != 128) || k->size(3) != d || !v->sizes().equals(k->sizes()) || k->size(0) != q->size(0) || q->size(2) % k->size(2) ||
      (causal && k->size(1) < q->size(1)) || !fits_int({q->size(0) * q->size(1), k->size(0) * k->size(1)})) LB_NOT_PLAIN;
  const double scale = PyFloat_AsDouble(a[4]);
  return THPVariable_Wrap(unlocked([q = *q, k = *k, v = *v, causal, scale] { return Attention::apply(q, k, v, causal, scale); }));
  END_HANDLE_TH_ERRORS
}

bool table_ok(const Tensor* t, int64_t d) {
  return t && t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->dim() == 2 && t->size(1) == d / 2 && !t->requires_grad() &&
         !t->_fw_grad(0).defined();
}

// (qkv, cos, sin, positions or None, B, S, hq, hkv, d, scale)
PyObject* py_rope_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 10 || !PyFloat_Check(a[9]) || !unobserved() || !env_is_tc("LIGHTRON_FA")) LB_NOT_PLAIN;
  const Tensor *qkv = tensor(a[0]), *cos = tensor(a[1]), *sin = tensor(a[2]), *pos = a[3] == Py_None ? nullptr : tensor(a[3]);
  Dims dims;
  for (int i = 0; i < 5; i++) {
    if (!PyLong_CheckExact(a[4 + i])) LB_NOT_PLAIN;
    dims.v[i] = PyLong_AsLongLong(a[4 + i]);
    if (PyErr_Occurred()) return nullptr;
    if (dims.v[i] < 1 || dims.v[i] > (1 << 24)) LB_NOT_PLAIN;
  }
  const int64_t B = dims.v[0], S = dims.v[1], hq = dims.v[2], hkv = dims.v[3], d = dims.v[4];
  if (!plain(qkv) || qkv->dim() != 2 || qkv->size(0) != B * S || qkv->size(1) != (hq + 2 * hkv) * d || hq % hkv || (d != 64 && d != 128) ||
      !fits_int({B * S}) || !table_ok(cos, d) || !table_ok(sin, d) || ((uintptr_t)qkv->const_data_ptr() & 15)) LB_NOT_PLAIN;
  if (a[3] != Py_None) {
    if (!pos || !pos->is_cuda() || pos->scalar_type() != at::kInt || !pos->is_contiguous() || pos->numel() != S) LB_NOT_PLAIN;
  } else if (cos->size(0) < S || sin->size(0) < S) {
    LB_NOT_PLAIN;
  }
  const double scale = PyFloat_AsDouble(a[9]);
  return THPVariable_Wrap(unlocked([qkv = *qkv, cos = *cos, sin = *sin, pos = pos ? std::optional<Tensor>(*pos) : std::nullopt, dims, scale] {
    return RopeAttention::apply(qkv, cos, sin, pos, dims, scale);
  }));
  END_HANDLE_TH_ERRORS
}

PyObject* py_embedding(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || !PyLong_CheckExact(a[2]) || !unobserved()) LB_NOT_PLAIN;
  const Tensor *tok = tensor(a[0]), *w = tensor(a[1]);
  const long long v0 = PyLong_AsLongLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  if (!tok || !tok->is_cuda() || tok->scalar_type() != at::kLong || !tok->is_contiguous() || tok->numel() == 0 || !plain(w) || w->dim() != 2 ||
      !fits_int({tok->numel(), w->size(1), v0, v0 + w->size(0)})) LB_NOT_PLAIN;
  return THPVariable_Wrap(unlocked([tok = *tok, w = *w, v0 = (int64_t)v0] { return Embedding::apply(tok, w, v0); }));
  END_HANDLE_TH_ERRORS
}

// (logits [T, V], targets, vocab_start, n_valid, ignore_index), one vocabulary on this rank
PyObject* py_cross_entropy(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5 || !unobserved()) LB_NOT_PLAIN;
  int64_t v[3];
  for (int i = 0; i < 3; i++) {
    if (!PyLong_CheckExact(a[2 + i])) LB_NOT_PLAIN;
    v[i] = PyLong_AsLongLong(a[2 + i]);
    if (PyErr_Occurred()) return nullptr;
  }
  const Tensor *x = tensor(a[0]), *t = tensor(a[1]);
  if (!plain(x, false) || x->dim() != 2 || x->stride(1) != 1 || !fits_int({x->size(0), x->size(1), v[0], v[1]}) || v[2] < INT_MIN || v[2] > INT_MAX ||
      !t || !t->is_cuda() || t->scalar_type() != at::kLong || t->dim() != 1 || !t->is_contiguous() || t->size(0) != x->size(0)) LB_NOT_PLAIN;
  return THPVariable_Wrap(unlocked([x = *x, t = *t, v0 = v[0], nv = v[1], ig = v[2]] { return CrossEntropy::apply(x, t, v0, nv, ig); }));
  END_HANDLE_TH_ERRORS
}

// ---- a run of decoder layers without gradients -----------------------------------------------------
// What models/llama.py does for one GPU with seven ops a layer, in one call: seven launches a layer (the rotation is in the projection's
// epilogue, g | u are not stored), intermediate results in one workspace.  12 layers of 768 columns over 128 tokens, embedding and
// head included, were bound by the host's 8 us an op: 808 us, now 516 (kernels 486).
struct DecoderLayer { Tensor norm1, wqkv, wo, norm2, w13, w2; double eps1, eps2; L I; };

std::pair<Tensor, Tensor> decoder_layers(Tensor h, Tensor delta, const Tensor& cos, const Tensor& sin, const Tensor& positions, Dims dims, double scale,
                                         const std::vector<DecoderLayer>& layers) {
  const L B = dims.v[0], S = dims.v[1], hq = dims.v[2], hkv = dims.v[3], d = dims.v[4], T = h.size(0), H = h.size(1), nqkv = (hq + 2 * hkv) * d;
  L I = 0;
  for (const DecoderLayer& l : layers) I = std::max(I, l.I);
  // Of a layer: the normed rows throughout; then qkv, o, the log-sum-exp and the attention's output, and in their place the activation
  auto up = [](L bytes) { return (bytes + 255) / 256 * 256; };
  const L at_rstd = up(2 * T * H), at_qkv = at_rstd + up(4 * T), at_o = at_qkv + up(2 * T * nqkv), at_lse = at_o + up(2 * T * hq * d),
          at_a = at_lse + up(4 * T * hq), end = std::max(at_a + up(2 * T * H), at_qkv + up(2 * T * I));
  const Tensor ws = at::empty({end}, h.options().dtype(at::kByte));
  char* base = static_cast<char*>(ws.mutable_data_ptr());
  W x = base, rstd = base + at_rstd, qkv = base + at_qkv, o = base + at_o, lse = base + at_lse, a = base + at_a, act = qkv;
  auto head = [&](L n) { return base + at_qkv + n * d * 2; };
  const Tensor own[2] = {empty({T, H}, h), empty({T, H}, h)};      // the residual stream, each sum in the one that does not hold the last
  Tensor f = empty({T, H}, h);
  int turn = 0;
  auto norm = [&](P add, const Tensor& w, double eps) {            // h (+)= add, x = norm(h)
    if (add) {
      LB_CALL(lb_rmsnorm_fwd, add, h.const_data_ptr(), w.const_data_ptr(), own[turn].mutable_data_ptr(), x, rstd, (int)T, (int)H, (float)eps, stream());
      h = own[turn];
      turn ^= 1;
    } else {
      LB_CALL(lb_rmsnorm_fwd, h.const_data_ptr(), nullptr, w.const_data_ptr(), nullptr, x, rstd, (int)T, (int)H, (float)eps, stream());
    }
  };
  auto gemm = [&](P in, const Tensor& w, W out, L n, L k, int epi = 0, W c2 = nullptr) {
    const P A[1] = {in}, Bw[1] = {w.const_data_ptr()};
    const W C[1] = {out}, C2[1] = {c2};
    const int M[1] = {(int)T}, N[1] = {(int)n}, K[1] = {(int)k}, no[1] = {0}, ep[1] = {epi}, half[1] = {(int)(n / 2)};
    const L lda[1] = {k}, ldc[1] = {n}, ldc2[1] = {n / 2};
    LB_CALL(lb_gemm_grouped_epi, 1, A, Bw, C, M, N, K, lda, lda, ldc, no, no, no, ep, C2, ldc2, half, stream());
  };
  for (const DecoderLayer& l : layers) {
    norm(delta.defined() ? delta.const_data_ptr() : nullptr, l.norm1, l.eps1);
    LB_CALL(lb_gemm_rope, x, l.wqkv.const_data_ptr(), qkv, (int)T, (int)nqkv, (int)H, cos.const_data_ptr(), sin.const_data_ptr(),
            positions.defined() ? positions.const_data_ptr() : nullptr, (int)S, (int)d, (int)((hq + hkv) * d), stream());
    LB_CALL(lb_flash_fwd_tc, head(0), head(hq), head(hq + hkv), o, lse, (int)B, (int)S, (int)S, (int)hq, (int)hkv, (int)d, nqkv, nqkv, nqkv, hq * d,
            (float)scale, 1, stream());
    gemm(o, l.wo, a, H, hq * d);
    norm(a, l.norm2, l.eps2);
    gemm(x, l.w13, nullptr, 2 * l.I, H, 1, act);
    gemm(act, l.w2, f.mutable_data_ptr(), H, l.I);
    delta = f;                                                     // (the next layer's first norm reads it before its last GEMM writes it)
  }
  return {h, delta};
}

// (h, delta or None, cos, sin, positions or None, B, S, hq, hkv, d, scale, layers) -> (h, delta).  layers: a list with, per layer, a tuple (attention norm's weight, eps,
// wq, wk, wv, wo, feed-forward norm's weight, eps, w1, w3, w2).  Without gradients only.
PyObject* py_decoder_layers(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 12 || at::GradMode::is_enabled() || !PyFloat_Check(a[10]) || !PyList_CheckExact(a[11]) || PyList_GET_SIZE(a[11]) == 0 || !unobserved() ||
      !env_is_tc("LIGHTRON_FA")) LB_NOT_PLAIN;
  const Tensor *h = tensor(a[0]), *delta = a[1] == Py_None ? nullptr : tensor(a[1]), *cos = tensor(a[2]), *sin = tensor(a[3]),
               *pos = a[4] == Py_None ? nullptr : tensor(a[4]);
  Dims dims;
  for (int i = 0; i < 5; i++) {
    if (!PyLong_CheckExact(a[5 + i])) LB_NOT_PLAIN;
    dims.v[i] = PyLong_AsLongLong(a[5 + i]);
    if (PyErr_Occurred()) return nullptr;
    if (dims.v[i] < 1 || dims.v[i] > (1 << 24)) LB_NOT_PLAIN;
  }
  const int64_t B = dims.v[0], S = dims.v[1], hq = dims.v[2], hkv = dims.v[3], d = dims.v[4];
  auto aligned = [](const Tensor& t) { return ((uintptr_t)t.const_data_ptr() & 15) == 0; };
  if (!plain(h) || h->dim() != 2 || h->size(0) != B * S || h->size(1) % 8 || !aligned(*h) || hq % hkv || (d != 64 && d != 128) ||
      !fits_int({B * S, h->size(1), (hq + 2 * hkv) * d}) || !table_ok(cos, d) || !table_ok(sin, d)) LB_NOT_PLAIN;
  if (a[1] != Py_None && (!plain(delta) || !delta->sizes().equals(h->sizes()) || !aligned(*delta))) LB_NOT_PLAIN;
  if (a[4] != Py_None) {
    if (!pos || !pos->is_cuda() || pos->scalar_type() != at::kInt || !pos->is_contiguous() || pos->numel() != S) LB_NOT_PLAIN;
  } else if (cos->size(0) < S || sin->size(0) < S) {
    LB_NOT_PLAIN;
  }
  const int64_t H = h->size(1);
  std::vector<DecoderLayer> layers((size_t)PyList_GET_SIZE(a[11]));
  for (size_t i = 0; i < layers.size(); i++) {
    PyObject* t = PyList_GET_ITEM(a[11], (Py_ssize_t)i);
    if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 11) LB_NOT_PLAIN;
    const Tensor* w[11];
    for (int j = 0; j < 11; j++) {
      PyObject* o = PyTuple_GET_ITEM(t, j);
      if (j == 1 || j == 7) {
        if (!PyFloat_Check(o)) LB_NOT_PLAIN;
        continue;
      }
      w[j] = tensor(o);
      if (!plain(w[j]) || !aligned(*w[j]) || w[j]->device() != h->device()) LB_NOT_PLAIN;
    }
    for (int j : {0, 6})
      if (w[j]->dim() != 1 || w[j]->size(0) != H) LB_NOT_PLAIN;
    for (int j : {2, 3, 4, 8, 9})
      if (!weight_ok(w[j], H)) LB_NOT_PLAIN;
    if (w[2]->size(0) != hq * d || w[3]->size(0) != hkv * d || w[4]->size(0) != hkv * d || !weight_ok(w[5], hq * d) || w[5]->size(0) != H ||
        w[8]->size(0) != w[9]->size(0) || !weight_ok(w[10], w[8]->size(0)) || w[10]->size(0) != H || !fits_int({2 * w[8]->size(0)})) LB_NOT_PLAIN;
    if (!rows_adjacent(w + 2, 3) || !rows_adjacent(w + 8, 2)) LB_NOT_PLAIN;
    layers[i] = {*w[0], *w[2], *w[5], *w[6], *w[8], *w[10], PyFloat_AsDouble(PyTuple_GET_ITEM(t, 1)), PyFloat_AsDouble(PyTuple_GET_ITEM(t, 7)), w[8]->size(0)};
  }
  const double scale = PyFloat_AsDouble(a[10]);
  std::pair<Tensor, Tensor> r = unlocked([&, h = *h, delta = delta ? *delta : Tensor(), cos = *cos, sin = *sin, pos = pos ? *pos : Tensor()] {
    return decoder_layers(h, delta, cos, sin, pos, dims, scale, layers);
  });
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(r.first)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(r.second)));
  return t;
  END_HANDLE_TH_ERRORS
}

PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromUnsignedLongLong(g_launches.load(std::memory_order_relaxed)); }

// init(addresses: dict of name -> int, raise_error): the kernels' entry points of the library that ops/native.py has loaded
PyObject* py_init(PyObject*, PyObject* args) {
  PyObject *table, *fn;
  if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &table, &fn)) return nullptr;
  bool ok = true;
  auto take = [&](const char* name, void* slot) {
    PyObject* v = PyDict_GetItemString(table, name);
    void* p = v ? PyLong_AsVoidPtr(v) : nullptr;
    if (!p) { ok = false; return; }
    std::memcpy(slot, &p, sizeof(p));
  };
#define LB_TAKE(name) take(#name, &api.name)
  LB_TAKE(lb_rmsnorm_fwd); LB_TAKE(lb_rmsnorm_bwd_blocks); LB_TAKE(lb_rmsnorm_bwd); LB_TAKE(lb_rope); LB_TAKE(lb_gemm_grouped_epi);
  LB_TAKE(lb_flash_fwd_tc); LB_TAKE(lb_flash_bwd_ws_bytes_kv); LB_TAKE(lb_flash_bwd_tc_ws); LB_TAKE(lb_flash_bwd); LB_TAKE(lb_embedding_fwd); LB_TAKE(lb_clear);
  LB_TAKE(lb_embedding_bwd); LB_TAKE(lb_ce_stats); LB_TAKE(lb_ce_loss); LB_TAKE(lb_ce_grad); LB_TAKE(lb_gemm_rope);
  if (!ok) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "an entry point of the kernels is missing");
    return nullptr;
  }
  Py_INCREF(fn);
  Py_XSETREF(raise_error, fn);
  Py_RETURN_NONE;
}

#define LB_FAST(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {LB_FAST(linear), LB_FAST(swiglu_mlp), LB_FAST(rmsnorm), LB_FAST(attention), LB_FAST(rope_attention), LB_FAST(embedding),
                         LB_FAST(cross_entropy), LB_FAST(decoder_layers), {"launches", py_launches, METH_NOARGS, nullptr}, {"init", py_init, METH_VARARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// Read from the file by csrc/build.py before the module is loaded.
extern "C" __attribute__((used, visibility("default"))) const char lb_host_ops_built_for[] = LB_BUILT_FOR;

PyMODINIT_FUNC PyInit__host_ops() {
  direct_grad = PyUnicode_InternFromString("_lb_direct_grad");
  return direct_grad ? PyModule_Create(&module) : nullptr;
}
