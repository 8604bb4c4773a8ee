// Autograd bindings of the sm_100a kernels: each op allocates its outputs, launches the kernels of
// ../kernels on the current CUDA stream and records one C++ autograd node whose backward does the
// same.  There is no eager fallback.
//
// Why native: a GPT-2 small layer (2 x 1024 tokens, forward + backward) was about fifty launches of a
// few microseconds each.  Issued from Python autograd functions through ctypes they took 1.14 ms of
// host time against 0.57 ms on the device, so every layer up to that size ran at the speed of the
// interpreter.  It is 20 launches and 0.23 ms now, as one node (Block).
//
// Conventions shared by all ops
//   * tensors are 16-bit (the kernels refuse other types) and live on the current device;
//   * weight gradients: a parameter whose .grad already holds a contiguous, 16-byte aligned tensor of its
//     shape and type (the engine's gradient buffer) gets the product accumulated into it by the GEMM
//     epilogue and the node returns no gradient for it; otherwise the gradient is returned as usual, also to a
//     backward pass for chosen inputs, which changes the .grad of no other;
//   * gains and biases likewise, where autograd would do nothing but add (see row_sum);
//   * saved tensors go through save_for_backward, so saved-tensor hooks see them;
//   * a tensor is made for what is allocated, returned or saved; parts and reshapes of one that only a kernel sees are
//     an address and a stride (a view costs a microsecond or more, and a small layer made 45 of them a pass);
//   * Python's interpreter lock is released for the duration of a call.
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/functions/accumulate_grad.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/extension.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <string>

namespace py = pybind11;
using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// C entry points of libft_cuda.so (loaded globally before this module)
extern "C" {
int64_t ft_gemm_ws_bytes(int M, int N, int K, int c_dtype);
int ft_gemm_ws(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int64_t ldc,
               int c_dtype, int accumulate, const void* R, int64_t ldr, const void* bias, int M, int N, int K,
               int ab_dtype, void* workspace, int64_t workspace_bytes, cudaStream_t stream);
int ft_gemm_dw_db(const void* dy, int64_t ld_dy, const void* x, int64_t ld_x, void* dw, int64_t ld_dw, int add_dw,
                  void* db, int add_db, int T, int N, int K, int dtype, cudaStream_t stream);
int ft_gemm_backward(const void* dy, int64_t ld_dy, const void* w, int64_t ld_w, const void* x, int64_t ld_x, void* dx,
                     int64_t ld_dx, void* dw, int64_t ld_dw, int add_dw, void* db, int add_db, int t, int n, int k, int dtype,
                     cudaStream_t stream);
int ft_sum_parts(int n, const float* const* part, void* const* out, const int* parts, const int* N, const int* add, int dt,
                 cudaStream_t s);
int ft_embedding_add(const int64_t* tokens, const void* dy, void* grad, int64_t n, int H, int64_t V, int dt, cudaStream_t s);
int ft_gemm_swiglu(const void* X, int64_t ldx, const void* W, int64_t ldw, void* act, int64_t ld_act, void* gu,
                   int64_t ld_gu, int M, int F, int K, int dtype, cudaStream_t stream);
int ft_swiglu_fwd(const void* gu, void* out, int64_t rows, int F, int dt, cudaStream_t s);
int ft_swiglu_bwd(const void* gu, const void* dout, void* dgu, int64_t rows, int F, int dt, cudaStream_t s);
int ft_add_norm_fwd(const void* x, const void* res, void* sum_out, const void* w, const void* b, void* y, float* mean,
                    float* rstd, int64_t rows, int H, float eps, int layernorm, int dt, cudaStream_t s);
int ft_norm_bwd_parts(int64_t rows, int H);
int ft_norm_bwd_into(const void* x, const void* w, const void* dy, const void* dres, const float* mean,
                     const float* rstd, void* dx, void* dx_copy, void* dw, void* db, float* dw_part, float* db_part,
                     int64_t rows, int H, int layernorm, int accumulate, int dt, cudaStream_t s);
int ft_bias_act_fwd(const void* x, const void* bias, void* y, int64_t rows, int N, int act, int dt, cudaStream_t s);
int ft_bias_act_bwd_parts(int64_t rows, int N);
int ft_bias_act_bwd(const void* dy, const void* x, const void* bias, void* dx, void* dbias, float* db_part,
                    int64_t rows, int N, int act, int accumulate, int dt, cudaStream_t s);
int ft_rope(const void* x, int64_t x_tok_stride, void* y, int64_t y_tok_stride, const float* cos_t, const float* sin_t,
            int64_t tokens, int heads, int D, int seq_len, float sin_sign, int dt, cudaStream_t s);
int ft_attn_fwd(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v, int64_t v_stride,
                void* o, float* lse, int B, int S, int Hq, int Hkv, int D, float scale, int dtype,
                cudaStream_t stream);
int ft_attn_bwd_parts(int B, int S, int Hq, int Hkv, int D);
int ft_attn_bwd_split(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v,
                      int64_t v_stride, const void* o, const void* d_o, int64_t do_stride, const float* lse,
                      float* delta, float* dq_acc, float* kv_part, int splits, void* dq, int64_t dq_stride, void* dk,
                      int64_t dk_stride, void* dv, int64_t dv_stride, int B, int S, int Hq, int Hkv, int D,
                      float scale, int dtype, cudaStream_t stream, long long* trace, int trace_cta, int trace_it0);
}

namespace {

cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + " failed (code " + std::to_string(rc) + ")");
}

int dtype_code(const Tensor& t) {                    // csrc/kernels/common.cuh, DType
  switch (t.scalar_type()) {
    case at::kFloat: return 0;
    case at::kBFloat16: return 1;
    case at::kHalf: return 2;
    default:
      throw py::type_error(std::string("native kernels support fp32/bf16/fp16, not ") + c10::toString(t.scalar_type()));
  }
}

// The kernels take sizes from one operand; the others have to have what they will read.
void fits(bool ok, const char* what) {
  if (!ok) throw py::value_error(what);
}

bool vector_of(const Tensor& v, int64_t n, const Tensor& like) {
  return v.numel() == n && v.is_contiguous() && v.scalar_type() == like.scalar_type();
}

const void* opt_ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* f32(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }

Tensor empty_f32(int64_t n, const Tensor& like) { return at::empty({n}, like.options().dtype(at::kFloat)); }

// Whether this is a backward pass that ends in adding to .grad in place: not one that returns the gradients of
// chosen inputs (autograd.grad, backward(inputs=...)), nor one that records a graph of itself.
bool plain_backward() {
  const auto* chosen = torch::autograd::get_current_graph_task_exec_info();
  return !at::GradMode::is_enabled() && (chosen == nullptr || chosen->empty());
}

// Where autograd takes the gradient of the running node's `input`-th tensor: its accumulation, or nullptr.
torch::autograd::AccumulateGrad* leaf_of_input(size_t input) {
  const auto node = torch::autograd::get_current_node();
  if (!node || input >= node->num_outputs()) return nullptr;
  return dynamic_cast<torch::autograd::AccumulateGrad*>(node->next_edge(input).function.get());
}

// A kernel will write into t: to autograd a change in place, as its own addition to .grad is.
void written(const Tensor& t) {
  if (!t.is_inference()) torch::autograd::impl::bump_version(t);
}

// Where a gain's or a bias's gradient, a sum over `rows` rows, is written; the kernels leave it alone for none.
// Into the parameter's .grad where autograd would add it there with a kernel of its own for a few kilobytes (112
// launches of 508 in a GPT-2 small of 12 layers): a leaf whose accumulation nobody watches, on this node's stream.
struct RowSum {
  Tensor out;
  bool added = false;
  Tensor gradient() const { return added ? Tensor() : out; }
};

RowSum vector_for(const Tensor& like, int64_t rows) {
  return {rows > 0 ? at::empty_like(like) : at::zeros_like(like)};
}

// Where the gradient of the running node's `input`-th tensor, which looks like `like`, may be added by a kernel: its .grad, or nothing.
Tensor grad_to_add_to(size_t input, const Tensor& like) {
  namespace ag = torch::autograd;
  auto* sink = plain_backward() ? leaf_of_input(input) : nullptr;
  if (sink == nullptr) return Tensor();
  const Tensor &p = sink->variable, &g = p.grad();
  const auto s = sink->stream();
  if (g.defined() && g.layout() == at::kStrided && g.sizes() == like.sizes() && g.is_contiguous() &&
      g.scalar_type() == like.scalar_type() && g.device() == like.device() && !g.requires_grad() &&
      ag::impl::hooks(p).empty() && !ag::impl::post_acc_grad_hooks(p) && sink->pre_hooks().empty() &&
      sink->post_hooks().empty() && (!s || *s == c10::cuda::getCurrentCUDAStream(like.device().index()).unwrap()))
    return g;
  return Tensor();
}

// The parameter is the running node's `input`-th tensor and looks like `like`.
RowSum row_sum(size_t input, const Tensor& like, int64_t rows) {
  const Tensor g = grad_to_add_to(input, like);
  if (!g.defined()) return vector_for(like, rows);
  written(g);
  return {g, true};
}

// Whether two contiguous tensors share memory.
bool overlap(const Tensor& a, const Tensor& b) {
  const auto *pa = static_cast<const char*>(a.data_ptr()), *pb = static_cast<const char*>(b.data_ptr());
  return pa < pb + b.nbytes() && pb < pa + a.nbytes();
}

// Whether the running node's first two inputs are leaves that keep the gradient they are given, so that one
// tensor for both would be cloned.
bool feeds_two_leaves() {
  const auto *a = leaf_of_input(0), *b = leaf_of_input(1);
  return plain_backward() && a != nullptr && b != nullptr && a != b && !a->variable.grad().defined() &&
         !b->variable.grad().defined();
}

std::vector<int64_t> with_last(c10::IntArrayRef shape, int64_t last) {
  std::vector<int64_t> s(shape.begin(), shape.end());
  s.back() = last;
  return s;
}

// [rows, k] of x [..., k]
Tensor as_rows(const Tensor& x, int64_t k) {
  if (x.dim() == 2 && x.size(1) == k) return x;
  return k > 0 && x.is_contiguous() ? x.view({x.numel() / k, k}) : x.reshape({-1, k});
}

// [rows, k] with unit inner stride and 16-byte aligned rows (what a TMA descriptor wants)
Tensor gemm_rows(const Tensor& x, int64_t k) {
  Tensor x2 = as_rows(x, k);
  if (x2.stride(1) != 1 || (x2.stride(0) * x2.element_size()) % 16 != 0) x2 = x2.contiguous();
  return x2;
}

constexpr int kWorkspaceWanted = -5;                 // gemm_tcgen05.cu

// A 16-bit matrix whose rows have unit inner stride
struct Rows {
  void* ptr = nullptr;
  int64_t ld = 0;
};

Rows rows_of(const Tensor& t) { return t.defined() ? Rows{t.data_ptr(), t.stride(0)} : Rows{}; }

// out[m, n] (+)= sum_k A(m, k) B(n, k) (+ add) (+ bias); *_mn: the operand is stored with k as its rows.  Types are codes, `like`
// says where scratch belongs.
int product(Rows a, bool a_mn, Rows b, bool b_mn, int64_t m, int64_t n, int64_t k, Rows out, int type, int out_type,
            const Tensor& like, bool accumulate = false, Rows add = {}, const void* bias = nullptr) {
  const auto launch = [&](void* ws, int64_t bytes) {
    return ft_gemm_ws(a.ptr, a_mn, a.ld, b.ptr, b_mn, b.ld, out.ptr, out.ld, out_type, accumulate, add.ptr, add.ld, bias,
                      (int)m, (int)n, (int)k, type, ws, bytes, stream());
  };
  int rc = launch(nullptr, -1);
  if (rc == kWorkspaceWanted) {
    // scratch for partial sums: the product is divided along k, or runs whole where there is no memory for them
    int64_t bytes = ft_gemm_ws_bytes((int)m, (int)n, (int)k, out_type);
    Tensor ws;
    try {
      ws = at::empty({bytes}, like.options().dtype(at::kByte));
    } catch (const c10::OutOfMemoryError&) {
      bytes = 0;
    }
    rc = launch(const_cast<void*>(opt_ptr(ws)), bytes);
  }
  return rc;
}

// The same of tensors; out is [m, n] or contiguous [..., n]
void gemm(const Tensor& a, bool a_mn, const Tensor& b, bool b_mn, int64_t m, int64_t n, int64_t k, const Tensor& out,
          bool accumulate = false, const Tensor& add = Tensor(), const Tensor& bias = Tensor()) {
  const auto t = a.scalar_type();
  if (t != b.scalar_type() || (t != at::kBFloat16 && t != at::kHalf))
    throw py::type_error("gemm operands must both be bf16 or both fp16");
  if (m == 0 || n == 0 || k == 0) return;            // nor has a tensor of nothing strides to look at
  if (a.stride(-1) != 1 || b.stride(-1) != 1) throw py::value_error("gemm operands need unit inner stride");
  if (add.defined() && (add.size(0) != m || add.size(1) != n || add.scalar_type() != out.scalar_type() ||
                        add.stride(-1) != 1))
    throw py::value_error("gemm: `add` must be [m, n] of the output's type with unit inner stride");
  if (bias.defined() && (bias.dim() != 1 || bias.size(0) != n || bias.scalar_type() != out.scalar_type() ||
                         !bias.is_contiguous()))
    throw py::value_error("gemm: `bias` must be a contiguous [n] of the output's type");
  check(product(rows_of(a), a_mn, rows_of(b), b_mn, m, n, k, {out.data_ptr(), out.dim() == 2 ? out.stride(0) : n},
                dtype_code(a), dtype_code(out), out, accumulate, rows_of(add), opt_ptr(bias)),
        bias.defined() ? "ft_gemm_bias" : add.defined() ? "ft_gemm_add" : "ft_gemm");
}

// dX = dY W of the given shape, [..., columns of w]
Tensor data_gradient(const Tensor& dy2, const Tensor& w, c10::IntArrayRef shape) {
  Tensor dx = at::empty(shape, dy2.options());
  gemm(dy2, false, w, true, dy2.size(0), w.size(1), w.size(0), dx);
  return dx;
}

// column sums of dy, contiguous [rows, n]
Tensor bias_gradient(const void* dy, int64_t rows, int64_t n, const Tensor& bias, size_t input) {
  Tensor part = empty_f32(ft_bias_act_bwd_parts(rows, (int)n) * n, bias);
  const RowSum db = row_sum(input, bias, rows);
  check(ft_bias_act_bwd(dy, nullptr, nullptr, nullptr, db.out.data_ptr(), f32(part), rows, (int)n, 0, db.added,
                        dtype_code(bias), stream()),
        "ft_bias_act_bwd");
  return db.gradient();
}

Tensor bias_gradient(const Tensor& dy, const Tensor& bias, size_t input) {
  const Tensor dy2 = dy.contiguous();
  return bias_gradient(dy2.data_ptr(), dy2.size(0), dy2.size(1), bias, input);
}

// dW = dY^T X, into the engine's buffer where the parameter has one (then nothing is returned)
struct WeightGradient {
  Tensor dw;
  bool held = false;
  Tensor gradient() const { return held ? Tensor() : dw; }
};

WeightGradient weight_buffer(const Tensor& w, int64_t rows, c10::TensorOptions options) {
  const Tensor g = w.is_leaf() && plain_backward() ? w.grad() : Tensor();
  const bool held = g.defined() && g.sizes() == w.sizes() && g.is_contiguous() && g.scalar_type() == w.scalar_type() &&
                    reinterpret_cast<uintptr_t>(g.data_ptr()) % 16 == 0;
  return {held ? g : rows > 0 ? at::empty(w.sizes(), options) : at::zeros(w.sizes(), options), held};
}

// dW and the gradient `db` of `bias`, the running node's `input`-th tensor, in one product; false where that cannot sum.
bool weight_and_bias(Rows dy, Rows x, int64_t rows, const WeightGradient& g, const Tensor& bias, size_t input, Tensor& db) {
  const RowSum sum = row_sum(input, bias, rows);
  const int rc = ft_gemm_dw_db(dy.ptr, dy.ld, x.ptr, x.ld, g.dw.data_ptr(), g.dw.size(1), g.held, sum.out.data_ptr(), sum.added,
                               (int)rows, (int)g.dw.size(0), (int)g.dw.size(1), dtype_code(bias), stream());
  if (rc == -4) return false;
  check(rc, "ft_gemm_dw_db");
  db = sum.gradient();
  return true;
}

// dX, dW and, with `bias` (the running node's `input`-th tensor), db in one launch; false where that is no better than one each.
bool both_gradients(Rows dy, Rows x, int64_t rows, const Tensor& w, Rows dx, const WeightGradient& g, const Tensor& bias, size_t input,
                    Tensor& db) {
  if (rows == 0) return false;
  const RowSum sum = bias.defined() ? row_sum(input, bias, rows) : RowSum();
  const int rc = ft_gemm_backward(dy.ptr, dy.ld, w.data_ptr(), w.stride(0), x.ptr, x.ld, dx.ptr, dx.ld, g.dw.data_ptr(), g.dw.size(1),
                                  g.held, const_cast<void*>(opt_ptr(sum.out)), sum.added, (int)rows, (int)w.size(0), (int)w.size(1),
                                  dtype_code(w), stream());
  if (rc == -4) return false;
  check(rc, "ft_gemm_backward");
  if (bias.defined()) db = sum.gradient();
  return true;
}

// With `bias`, the running node's `input`-th tensor, its gradient `db` too, in the same product where that can sum.
// `made`: where dW goes, if that is known already.
Tensor weight_gradient(const Tensor& dy2, const Tensor& x2, const Tensor& w, const Tensor& bias = Tensor(),
                       size_t input = 0, Tensor* db = nullptr, const WeightGradient* made = nullptr) {
  const int64_t n = w.size(0), k = w.size(1), m = dy2.size(0);
  const WeightGradient g = made != nullptr ? *made : weight_buffer(w, m, dy2.options());
  const bool alike = bias.defined() && m > 0 && dy2.scalar_type() == x2.scalar_type() && bias.scalar_type() == dy2.scalar_type();
  if (!(alike && weight_and_bias(rows_of(dy2), rows_of(x2), m, g, bias, input, *db))) {
    gemm(dy2, true, x2, true, n, k, m, g.dw, g.held);
    if (bias.defined()) *db = bias_gradient(dy2, bias, input);
  }
  return g.gradient();
}

// ------------------------------------------------------------------ products
// x w^T (+ bias) (+ res), the additions in the GEMM's epilogue.  Saved: x2, w, bias.
// `done`: the product, where another kernel has already formed it (no additions then), a tensor of the
// caller's without history.  It becomes the output as a modified input does: an input that is returned
// without the mark comes back as a view, and the next op of a block (rope, bias) may not change that in place.
struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias,
                        const OptTensor& res, const OptTensor& done) {
    const int64_t k = x.size(-1);
    fits(w.dim() == 2 && w.size(1) == k, "linear: w must be [n, k] for x [..., k]");
    const int64_t n = w.size(0);
    Tensor x2 = gemm_rows(x, k), y;
    if (done) {
      y = *done;
      ctx->mark_dirty({y});
    } else {
      y = at::empty(with_last(x.sizes(), n), x.options());
      Tensor r2;
      if (res) {
        r2 = as_rows(*res, n);
        if (r2.stride(1) != 1) r2 = r2.contiguous();
      }
      gemm(x2, false, w, false, x2.size(0), n, k, y, false, r2, bias ? *bias : Tensor());
    }
    ctx->save_for_backward({x2, w, bias ? *bias : Tensor()});
    ctx->saved_data["res"] = res.has_value();
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &w = saved[1];
    const bool biased = saved[2].defined();              // an absent tensor has no edge: res comes third without a bias
    const int need = ctx->needs_input_grad(0) | ctx->needs_input_grad(1) << 1 | (biased && ctx->needs_input_grad(2)) << 2 |
                     (ctx->saved_data["res"].toBool() && ctx->needs_input_grad(biased ? 3 : 2)) << 3;
    const Tensor dy2 = gemm_rows(grads[0], w.size(0));
    Tensor dx, dw, db, dr;
    const Tensor bias = need & 4 ? saved[2] : Tensor();
    const auto type = w.scalar_type();
    if ((need & 3) == 3 && (type == at::kBFloat16 || type == at::kHalf) && dy2.scalar_type() == type && x2.scalar_type() == type &&
        w.stride(1) == 1 && (!bias.defined() || bias.scalar_type() == type)) {
      dx = at::empty(with_last(grads[0].sizes(), w.size(1)), dy2.options());
      const WeightGradient g = weight_buffer(w, dy2.size(0), dy2.options());
      if (both_gradients(rows_of(dy2), rows_of(x2), dy2.size(0), w, {dx.data_ptr(), w.size(1)}, g, bias, 2, db))
        return {dx, g.gradient(), db, need & 8 ? grads[0] : Tensor(), Tensor()};
      gemm(dy2, false, w, true, dy2.size(0), w.size(1), w.size(0), dx);
      dw = weight_gradient(dy2, x2, w, bias, 2, &db, &g);
      return {dx, dw, db, need & 8 ? grads[0] : Tensor(), Tensor()};
    }
    if (need & 1) {
      dx = data_gradient(dy2, w, with_last(grads[0].sizes(), w.size(1)));
    }
    if (need & 2) dw = weight_gradient(dy2, x2, w, bias, 2, &db);
    else if (need & 4) db = bias_gradient(dy2, bias, 2);
    if (need & 8) dr = grads[0];
    return {dx, dw, db, dr, Tensor()};
  }
};

// swiglu(x w^T), w = [w_gate ; w_up], with the activation in the GEMM's epilogue.  The projection is
// kept for the backward only when there will be one.  Saved: x2, w, gu.
struct LinearSwiGLU : Function<LinearSwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, bool need_gu) {
    const int64_t k = x.size(-1);
    fits(w.dim() == 2 && w.size(1) == k && w.size(0) % 2 == 0 && w.scalar_type() == x.scalar_type(),
         "linear_swiglu: w must be [2 f, k] for x [..., k], of one type");
    const int64_t f = w.size(0) / 2;
    Tensor x2 = gemm_rows(x, k);
    const int64_t rows = x2.size(0);
    Tensor act = at::empty({rows, f}, x.options()), gu;
    if (need_gu) gu = at::empty({rows, 2 * f}, x.options());
    const int dt = dtype_code(x);
    const int rc = ft_gemm_swiglu(x2.data_ptr(), x2.stride(0), w.data_ptr(), w.stride(0), act.data_ptr(), f,
                                  const_cast<void*>(opt_ptr(gu)), 2 * f, (int)rows, (int)f, (int)k, dt, stream());
    if (rc == -4) {                                  // shape outside the fused kernel: two steps
      gu = at::empty({rows, 2 * f}, x.options());
      gemm(x2, false, w, false, rows, 2 * f, k, gu);
      check(ft_swiglu_fwd(gu.data_ptr(), act.data_ptr(), rows, (int)f, dt, stream()), "ft_swiglu_fwd");
    } else {
      check(rc, "ft_gemm_swiglu");
    }
    if (need_gu) ctx->save_for_backward({x2, w, gu});
    return act.view(with_last(x.sizes(), f));
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &w = saved[1], &gu = saved[2];
    const int64_t rows = gu.size(0), f2 = gu.size(1);
    const Tensor d2 = grads[0].reshape({rows, f2 / 2}).contiguous();
    Tensor dgu = at::empty_like(gu), dx, dw;
    check(ft_swiglu_bwd(gu.data_ptr(), d2.data_ptr(), dgu.data_ptr(), rows, (int)(f2 / 2), dtype_code(gu), stream()),
          "ft_swiglu_bwd");
    if (ctx->needs_input_grad(0)) dx = data_gradient(dgu, w, with_last(grads[0].sizes(), w.size(1)));
    if (ctx->needs_input_grad(1)) dw = weight_gradient(dgu, x2, w);
    return {dx, dw, Tensor()};
  }
};

struct SwiGLU : Function<SwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gate_up) {
    const int64_t f = gate_up.size(-1) / 2;
    Tensor g2 = gate_up.reshape({-1, 2 * f}).contiguous();
    Tensor out = at::empty(with_last(gate_up.sizes(), f), gate_up.options());
    check(ft_swiglu_fwd(g2.data_ptr(), out.data_ptr(), g2.size(0), (int)f, dtype_code(gate_up), stream()),
          "ft_swiglu_fwd");
    ctx->save_for_backward({g2});
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor g2 = ctx->get_saved_variables()[0];
    const int64_t rows = g2.size(0), f2 = g2.size(1);
    const Tensor d2 = grads[0].reshape({rows, f2 / 2}).contiguous();
    Tensor dgu = at::empty_like(g2);
    check(ft_swiglu_bwd(g2.data_ptr(), d2.data_ptr(), dgu.data_ptr(), rows, (int)(f2 / 2), dtype_code(g2), stream()),
          "ft_swiglu_bwd");
    return {dgu.view(with_last(grads[0].sizes(), f2))};
  }
};

// --------------------------------------------------------------------- norms
struct NormGradients { Tensor dx, dx_copy, dw, db; };

// Sums of partial rows that wait for the end of a node's backward, to be formed in one launch.
struct LaterSums {
  const int type;
  int n = 0, parts[6], widths[6], add[6];
  const float* part[6];
  void* out[6];
  std::array<Tensor, 6> scratch, outs;

  // The sums of one launch read and write side by side: one that is added to memory which another adds to (a gain of both norms)
  // goes into the next launch.
  void keep(const Tensor& rows, int64_t offset, const RowSum& sum, int64_t count, int64_t width) {
    for (int i = 0; i < n && sum.added; ++i)
      if (add[i] && overlap(outs[i], sum.out)) form();
    scratch[n] = rows;
    outs[n] = sum.out;
    part[n] = f32(rows) + offset;
    out[n] = sum.out.data_ptr();
    parts[n] = (int)count;
    widths[n] = (int)width;
    add[n++] = sum.added;
  }
  void form() {
    check(ft_sum_parts(n, part, out, parts, widths, add, type, stream()), "ft_sum_parts");
    n = 0;
  }
};

// The gradients of a gain (the running node's `gain`-th tensor, like w) and, for LayerNorm, of the bias behind it, with dx (and
// dx_copy) written where the caller says; `ds`: a gradient that reaches the rows past the norm, or nullptr.
NormGradients norm_backward(const void* x, const Tensor& w, const float* mean, const float* rstd, const void* ds,
                            const void* dy, void* dx, void* dx_copy, int64_t rows, int64_t h, size_t gain,
                            LaterSums* later = nullptr) {
  const bool ln = mean != nullptr;
  const RowSum dw = row_sum(gain, w, rows);
  RowSum db = ln ? row_sum(gain + 1, w, rows) : RowSum();
  if (dw.added && db.added && overlap(dw.out, db.out)) db = vector_for(w, rows);      // one kernel adds to both
  const int64_t parts = ft_norm_bwd_parts(rows, (int)h);
  Tensor part = empty_f32((ln ? 2 : 1) * parts * h, w);
  check(ft_norm_bwd_into(x, w.data_ptr(), dy, ds, mean, rstd, dx, dx_copy, later ? nullptr : dw.out.data_ptr(),
                         later ? nullptr : const_cast<void*>(opt_ptr(db.out)), f32(part), ln ? f32(part) + parts * h : nullptr, rows, (int)h,
                         ln, dw.added | db.added << 1, dtype_code(w), stream()),
        "ft_norm_bwd_into");
  if (later != nullptr) {
    later->keep(part, 0, dw, parts, h);
    if (ln) later->keep(part, parts * h, db, parts, h);
  }
  return {Tensor(), Tensor(), dw.gradient(), db.gradient()};
}

// saved: the normalised rows [..., h], w, their rstd and (LayerNorm) mean, [1 or 2, rows].  `ds`: as above, or
// undefined.  `gain`: which input w is (b follows).  `twice`: dx in two buffers.
NormGradients norm_backward(const variable_list& saved, const Tensor& ds, const Tensor& dy, size_t gain, bool twice) {
  const Tensor &x = saved[0], &w = saved[1], &stats = saved[2];
  const int64_t rows = stats.size(1), h = x.size(-1);
  const float* rstd = f32(stats);
  const Tensor dy2 = dy.contiguous(), ds2 = ds.defined() ? ds.contiguous() : ds;
  Tensor dx = at::empty_like(x), dx_copy;
  if (twice) dx_copy = at::empty_like(x);
  NormGradients g = norm_backward(x.data_ptr(), w, stats.size(0) == 2 ? rstd + rows : nullptr, rstd, opt_ptr(ds2),
                                  dy2.data_ptr(), dx.data_ptr(), const_cast<void*>(opt_ptr(dx_copy)), rows, h, gain);
  g.dx = dx;
  g.dx_copy = dx_copy;
  return g;
}

// LayerNorm (b given) or RMSNorm through the row-resident kernels.  Saved: x, w, rstd with mean.
struct Norm : Function<Norm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& b, double eps) {
    const int64_t h = x.size(-1);
    fits(h > 0 && vector_of(w, h, x) && (!b || vector_of(*b, h, x)), "norm: gain and bias must have the width and type of x");
    const Tensor xc = x.contiguous();
    const int64_t rows = x.numel() / h;
    Tensor y = at::empty(x.sizes(), x.options()), stats = at::empty({b ? 2 : 1, rows}, x.options().dtype(at::kFloat));
    check(ft_add_norm_fwd(xc.data_ptr(), nullptr, nullptr, w.data_ptr(), b ? b->data_ptr() : nullptr, y.data_ptr(),
                          b ? f32(stats) + rows : nullptr, f32(stats), rows, (int)h, (float)eps, b.has_value(),
                          dtype_code(x), stream()),
          "ft_norm_fwd");
    ctx->save_for_backward({xc, w, stats});
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto d = norm_backward(ctx->get_saved_variables(), Tensor(), grads[0], 1, false);
    return {d.dx, d.dw, d.db, Tensor()};
  }
};

// x itself and y = norm(x), for a block that needs both: the gradient that arrives at x along the residual branch is
// added inside the norm's backward kernel (autograd's addition is a launch and three passes over the activations).
// Saved as Norm.
struct ResidualNorm : Function<ResidualNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& b, double eps) {
    ctx->set_materialize_grads(false);
    return {x, Norm::forward(ctx, x, w, b, eps)};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (!grads[1].defined()) return {grads[0], Tensor(), Tensor(), Tensor()};
    const auto d = norm_backward(ctx->get_saved_variables(), grads[0], grads[1], 1, false);
    return {d.dx, d.dw, d.db, Tensor()};
  }
};

// s = x + r and y = norm(s) in one kernel (LayerNorm with b, RMSNorm without); the backward adds the
// gradient that arrives at s from its other consumer inside the norm's backward kernel.
// Saved: s, w, rstd with mean.
struct AddNorm : Function<AddNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& r, const Tensor& w,
                               const OptTensor& b, double eps) {
    const int64_t h = x.size(-1);
    fits(h > 0 && vector_of(w, h, x) && (!b || vector_of(*b, h, x)), "norm: gain and bias must have the width and type of x");
    fits(r.numel() == x.numel() && r.scalar_type() == x.scalar_type(), "add_norm: x and r must have one shape and type");
    const Tensor xc = x.contiguous(), rc = r.contiguous();
    const int64_t rows = x.numel() / h;
    Tensor s = at::empty(x.sizes(), x.options()), y = at::empty(x.sizes(), x.options()),
           stats = at::empty({b ? 2 : 1, rows}, x.options().dtype(at::kFloat));
    check(ft_add_norm_fwd(xc.data_ptr(), rc.data_ptr(), s.data_ptr(), w.data_ptr(), b ? b->data_ptr() : nullptr,
                          y.data_ptr(), b ? f32(stats) + rows : nullptr, f32(stats), rows, (int)h, (float)eps,
                          b.has_value(), dtype_code(x), stream()),
          "ft_add_norm_fwd");
    ctx->save_for_backward({s, w, stats});
    return {s, y};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto d = norm_backward(ctx->get_saved_variables(), grads[0], grads[1], 2, feeds_two_leaves());
    return {d.dx, d.dx_copy.defined() ? d.dx_copy : d.dx, d.dw, d.db, Tensor()};
  }
};

// ---------------------------------------------------------- bias + activation
// act(x + bias) over the last dimension; act 0 adds the bias in place, act 1 is the tanh GELU.
// Saved: bias, and x for act 1.
struct BiasAct : Function<BiasAct> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& bias, int64_t act) {
    const int64_t n = x.size(-1);
    fits(n > 0 && vector_of(bias, n, x), "bias must have the width and type of x");
    const Tensor x2 = x.contiguous();
    const bool in_place = act == 0 && x2.data_ptr() == x.data_ptr();
    const Tensor y = in_place ? x2 : at::empty(x.sizes(), x.options());
    check(ft_bias_act_fwd(x2.data_ptr(), bias.data_ptr(), y.data_ptr(), x.numel() / n, (int)n, (int)act, dtype_code(x),
                          stream()),
          "ft_bias_act_fwd");
    ctx->saved_data["act"] = act;
    if (act == 0) ctx->save_for_backward({bias});
    else ctx->save_for_backward({bias, x2});
    if (in_place) {
      ctx->mark_dirty({x});
      return x;
    }
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const int64_t act = ctx->saved_data["act"].toInt();
    const Tensor& bias = saved[0];
    const int64_t n = bias.size(0);
    const Tensor dy2 = grads[0].contiguous();
    if (act == 0) return {dy2, bias_gradient(as_rows(dy2, n), bias, 1), Tensor()};
    const int64_t rows = dy2.numel() / n;
    Tensor part = empty_f32(ft_bias_act_bwd_parts(rows, (int)n) * n, dy2), dx2 = at::empty_like(dy2);
    const RowSum db = row_sum(1, bias, rows);
    check(ft_bias_act_bwd(dy2.data_ptr(), saved[1].data_ptr(), bias.data_ptr(), dx2.data_ptr(), db.out.data_ptr(),
                          f32(part), rows, (int)n, (int)act, db.added, dtype_code(dy2), stream()),
          "ft_bias_act_bwd");
    return {dx2, db.gradient(), Tensor()};
  }
};

// ---------------------------------------------------------------------- RoPE
// Rotates the first `heads` heads of every row of x [B, S, W] in place.  Saved: the tables.
struct RopeHeads : Function<RopeHeads> {
  static void launch(const Tensor& x, int64_t stride, const Tensor& cos, const Tensor& sin, int64_t heads, int64_t d,
                     float sign) {
    const int64_t b = x.size(0), s = x.size(1);
    check(ft_rope(x.data_ptr(), stride, x.data_ptr(), stride, cos.data_ptr<float>(), sin.data_ptr<float>(),
                  b * s, (int)heads, (int)d, (int)s, sign, dtype_code(x), stream()),
          "ft_rope");
  }

  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& cos, const Tensor& sin, int64_t heads,
                        int64_t d) {
    fits(heads * d <= x.size(2) && cos.numel() >= x.size(1) * (d / 2) && sin.numel() >= x.size(1) * (d / 2),
         "rope: x must be at least heads * d wide, the tables at least [S, d / 2]");
    launch(x, x.stride(1), cos, sin, heads, d, 1.f);
    ctx->mark_dirty({x});
    ctx->save_for_backward({cos, sin});
    ctx->saved_data["heads"] = heads;
    ctx->saved_data["d"] = d;
    return x;
  }

  // The gradient is rotated where it lies only if nobody else can see it, as after the attention of a
  // block; a caller's tensor, a hook's or one that another branch of the graph receives too is copied.
  // (`grads` by reference: a copy of the list would count as an owner.)
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto saved = ctx->get_saved_variables();
    const bool ours = grads[0].is_contiguous() && grads[0].use_count() == 1 && grads[0].storage().use_count() == 1;
    Tensor dy = ours ? grads[0] : grads[0].clone(at::MemoryFormat::Contiguous);
    launch(dy, dy.size(2), saved[0], saved[1], ctx->saved_data["heads"].toInt(), ctx->saved_data["d"].toInt(), -1.f);
    return {dy, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ----------------------------------------------------------------- attention
// Elements from one token to the next of [B, S, H, D].  A dimension of size 1 may have any stride, so with
// one token a sequence it is the batch's.
int64_t token_stride(const Tensor& t) {
  return t.size(1) > 1 ? t.stride(1) : t.size(0) > 1 ? t.stride(0) : t.size(2) * t.size(3);
}

// [B, S, H, D] with unit stride inside a head, adjacent heads, one token stride and 16-byte alignment, as
// every contiguous tensor has
bool token_rows(const Tensor& t, bool check_base) {
  return t.stride(3) == 1 && (t.size(2) == 1 || t.stride(2) == t.size(3)) &&
         (t.size(0) == 1 || t.size(1) == 1 || t.stride(0) == t.size(1) * t.stride(1)) &&
         (token_stride(t) * t.element_size()) % 16 == 0 &&
         (!check_base || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0);
}

// Heads of q, k or v (or their gradients) as the kernels address them.
struct Heads { void* ptr; int64_t stride, heads; };
struct AttentionShape { int64_t b, s, d; double scale; };

Heads heads_of(const Tensor& t) { return {t.data_ptr(), token_stride(t), t.size(2)}; }

void attention_forward(const AttentionShape& n, Heads q, Heads k, Heads v, void* o, float* lse, int type) {
  check(ft_attn_fwd(q.ptr, q.stride, k.ptr, k.stride, v.ptr, v.stride, o, lse, (int)n.b, (int)n.s, (int)q.heads,
                    (int)k.heads, (int)n.d, (float)n.scale, type, stream()),
        "ft_attn_fwd");
}

void attention_backward(const AttentionShape& n, Heads q, Heads k, Heads v, const void* o, const float* lse,
                        const void* d_o, int64_t do_stride, Heads dq, Heads dk, Heads dv, const Tensor& like) {
  const int splits = ft_attn_bwd_parts((int)n.b, (int)n.s, (int)q.heads, (int)k.heads, (int)n.d);
  // one scratch tensor: dq's sums, those of dk and dv where they are divided, delta
  const int64_t dq_sums = n.b * n.s * q.heads * n.d, kv_sums = splits > 1 ? 2 * splits * n.b * n.s * k.heads * n.d : 0;
  const Tensor scratch = empty_f32(dq_sums + kv_sums + n.b * q.heads * n.s, like);
  float* sums = f32(scratch);
  check(ft_attn_bwd_split(q.ptr, q.stride, k.ptr, k.stride, v.ptr, v.stride, o, d_o, do_stride, lse,
                          sums + dq_sums + kv_sums, sums, kv_sums ? sums + dq_sums : nullptr, splits, dq.ptr, dq.stride,
                          dk.ptr, dk.stride, dv.ptr, dv.stride, (int)n.b, (int)n.s, (int)q.heads, (int)k.heads,
                          (int)n.d, (float)n.scale, dtype_code(like), stream(), nullptr, 0, 0),
        "ft_attn_bwd");
}

struct Attention : Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale) {
    fits(q_.dim() == 4 && k_.dim() == 4 && v_.dim() == 4, "attention: q, k and v must be [B, S, H, D]");
    fits(k_.size(0) == q_.size(0) && k_.size(1) == q_.size(1) && k_.size(3) == q_.size(3) && v_.sizes() == k_.sizes() &&
             k_.scalar_type() == q_.scalar_type() && v_.scalar_type() == q_.scalar_type(),
         "attention: q, k and v must have the same B, S, D and type, k and v the same heads");
    const Tensor q = token_rows(q_, true) ? q_ : q_.contiguous(), k = token_rows(k_, true) ? k_ : k_.contiguous(),
                 v = token_rows(v_, true) ? v_ : v_.contiguous();
    Tensor o = at::empty(q.sizes(), q.options());
    Tensor lse = at::empty({q.size(0), q.size(2), q.size(1)}, q.options().dtype(at::kFloat));
    attention_forward({q.size(0), q.size(1), q.size(3), scale}, heads_of(q), heads_of(k), heads_of(v), o.data_ptr(), f32(lse),
                      dtype_code(o));
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["scale"] = scale;
    return o;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    Tensor dq = at::empty(s[0].sizes(), s[0].options()), dk = at::empty(s[1].sizes(), s[0].options()),
           dv = at::empty(s[1].sizes(), s[0].options());
    const Tensor d_o = token_rows(grads[0], false) ? grads[0] : grads[0].contiguous();
    attention_backward({s[0].size(0), s[0].size(1), s[0].size(3), ctx->saved_data["scale"].toDouble()}, heads_of(s[0]),
                       heads_of(s[1]), heads_of(s[2]), s[3].data_ptr(), f32(s[4]), d_o.data_ptr(), token_stride(d_o),
                       heads_of(dq), heads_of(dk), heads_of(dv), s[3]);
    return {dq, dk, dv, Tensor()};
  }
};

// Attention over a packed qkv [B, S, (Hq + 2 Hkv) D] whose q and k heads are already rotated; the
// backward writes one packed gradient.  Saved: qkv (a copy where the kernels cannot address its parts: both
// directions read the same tensor), o, lse.
struct PackedAttention : Function<PackedAttention> {
  // q, k and v inside qkv, an address each
  static int64_t stride_of(const Tensor& t) {
    return t.size(1) > 1 ? t.stride(1) : t.size(0) > 1 ? t.stride(0) : t.size(2);
  }

  static std::array<Heads, 3> split(const Tensor& qkv, int64_t hq, int64_t hkv, int64_t d) {
    const int64_t stride = stride_of(qkv);
    auto part = [&](int64_t first, int64_t n) {
      return Heads{static_cast<char*>(qkv.data_ptr()) + first * d * qkv.element_size(), stride, n};
    };
    return {part(0, hq), part(hq, hkv), part(hq + hkv, hkv)};
  }

  // What token_rows asks of a part: unit stride inside a token, one aligned stride from token to token
  static bool one_stride(const Tensor& t) {
    return t.stride(2) == 1 && (t.size(0) == 1 || t.size(1) == 1 || t.stride(0) == t.size(1) * t.stride(1)) &&
           (stride_of(t) * t.element_size()) % 16 == 0;
  }

  static bool addressable(const Tensor& qkv, const std::array<Heads, 3>& p) {
    const auto misaligned = [](const Heads& h) { return reinterpret_cast<uintptr_t>(h.ptr) % 16 != 0; };
    return one_stride(qkv) && !misaligned(p[0]) && !misaligned(p[1]) && !misaligned(p[2]);
  }

  static Tensor forward(AutogradContext* ctx, const Tensor& qkv_, int64_t hq, int64_t hkv, int64_t d, double scale) {
    fits(qkv_.dim() == 3 && qkv_.size(2) == (hq + 2 * hkv) * d, "attention_packed: qkv must be [B, S, (hq + 2 * hkv) * d]");
    const int64_t b = qkv_.size(0), s = qkv_.size(1);
    Tensor qkv = qkv_;
    auto p = split(qkv, hq, hkv, d);
    if (!addressable(qkv, p)) {
      qkv = qkv.contiguous();
      p = split(qkv, hq, hkv, d);
    }
    Tensor o = at::empty({b, s, hq * d}, qkv.options());
    Tensor lse = at::empty({b, hq, s}, qkv.options().dtype(at::kFloat));
    attention_forward({b, s, d, scale}, p[0], p[1], p[2], o.data_ptr(), f32(lse), dtype_code(o));
    ctx->save_for_backward({qkv, o, lse});
    ctx->saved_data["hq"] = hq;
    ctx->saved_data["hkv"] = hkv;
    ctx->saved_data["scale"] = scale;
    return o;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &qkv = saved[0], &o = saved[1], &lse = saved[2];
    const int64_t hq = ctx->saved_data["hq"].toInt(), hkv = ctx->saved_data["hkv"].toInt(),
                  d = qkv.size(2) / (hq + 2 * hkv);
    Tensor dqkv = at::empty(qkv.sizes(), qkv.options());
    const auto p = split(qkv, hq, hkv, d), g = split(dqkv, hq, hkv, d);
    const Tensor d_o = one_stride(grads[0]) ? grads[0] : grads[0].contiguous();
    attention_backward({qkv.size(0), qkv.size(1), d, ctx->saved_data["scale"].toDouble()}, p[0], p[1], p[2],
                       o.data_ptr(), f32(lse), d_o.data_ptr(), stride_of(d_o), g[0], g[1], g[2], o);
    return {dqkv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ----------------------------------------------------------------- embedding
// Rows of a table by token.  The backward adds to the table's .grad where autograd would do nothing else with a gradient of the whole
// table that is zero but for the tokens' rows.  Saved: tokens.
struct Embedding : Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& tokens, const Tensor& w) {
    ctx->save_for_backward({tokens});
    ctx->saved_data["rows"] = w.size(0);
    return at::embedding(w, tokens);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor tokens = ctx->get_saved_variables()[0], &dy = grads[0];
    const int64_t rows = ctx->saved_data["rows"].toInt();
    const auto* table = leaf_of_input(1);
    const bool covered = table != nullptr && tokens.scalar_type() == at::kLong &&
                         tokens.is_contiguous() && (dy.scalar_type() == at::kBFloat16 || dy.scalar_type() == at::kHalf) &&
                         table->variable.scalar_type() == dy.scalar_type();
    const Tensor g = covered ? grad_to_add_to(1, table->variable) : Tensor();
    if (g.defined()) {
      const Tensor dy2 = dy.contiguous();
      const int rc = ft_embedding_add(tokens.data_ptr<int64_t>(), dy2.data_ptr(), g.data_ptr(), tokens.numel(), (int)g.size(1), rows,
                                      dtype_code(g), stream());
      if (rc != -4) {
        check(rc, "ft_embedding_add");
        written(g);
        return {Tensor(), Tensor()};
      }
    }
    return {Tensor(), at::embedding_dense_backward(dy, tokens, rows, -1, false)};
  }
};

// ------------------------------------------------------------------- a block
// A GPT block (models/gpt.py) as one node, for blocks that the host bounds: the same kernels in the same order as its eight ops, with
// one tensor for all that they leave one another instead of one each, and one node instead of eight.  Two sequences of 128
// tokens at width 256, forward + backward: 332 -> 228 us, a GPT-2 small of 2 x 512 tokens 3883 -> 2872.
// Saved: x, the parameters without the norms' biases, the 16-bit and the 32-bit intermediates.
struct Block : Function<Block> {
  enum Input { X, LN1_W, LN1_B, WQKV, BQKV, WO, BO, LN2_W, LN2_B, W_FC, B_FC, W_PROJ, B_PROJ, INPUTS };

  // Offsets of the intermediates, 16-bit (rows of 16-byte aligned widths) and 32-bit
  struct Layout {
    int64_t t, h, f, h1, qkv, o, s, h2, u, g, end, stats1, stats2, lse, end32;
    Layout(int64_t t_, int64_t h_, int64_t f_, int64_t heads) : t(t_), h(h_), f(f_) {
      h1 = 0, qkv = h1 + t * h, o = qkv + 3 * t * h, s = o + t * h, h2 = s + t * h, u = h2 + t * h;
      g = u + t * std::max(f, h), end = g + t * f;     // the attention's projection lies where u will, until the second norm has read it
      stats1 = 0, stats2 = 2 * t, lse = 4 * t, end32 = 4 * t + heads * t;
    }
  };

  struct Parts {                                     // addresses in a tensor of 16-bit values
    char* base;
    Rows operator()(int64_t offset, int64_t ld) const { return {base + 2 * offset, ld}; }
  };

  static std::array<Heads, 3> heads_in(Rows qkv, int64_t heads, int64_t d) {
    char* p = static_cast<char*>(qkv.ptr);
    return {Heads{p, qkv.ld, heads}, Heads{p + 2 * heads * d, qkv.ld, heads}, Heads{p + 4 * heads * d, qkv.ld, heads}};
  }

  static void norm(const void* x, const void* res, void* sum, const Tensor& w, const Tensor& b, Rows y, float* stats,
                   const Layout& at, double eps) {
    check(ft_add_norm_fwd(x, res, sum, w.data_ptr(), b.data_ptr(), y.ptr, stats + at.t, stats, at.t, (int)at.h, (float)eps, 1,
                          dtype_code(w), stream()),
          "ft_add_norm_fwd");
  }

  // x w^T + bias (+ add)
  static void forward_product(Rows x, const Tensor& w, const void* bias, Rows out, int64_t rows, Rows add = {}) {
    check(product(x, false, rows_of(w), false, rows, w.size(0), w.size(1), out, dtype_code(w), dtype_code(w), w, false, add, bias),
          bias ? "ft_gemm_bias" : "ft_gemm");
  }

  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& ln1_w, const Tensor& ln1_b, const Tensor& wqkv,
                        const Tensor& bqkv, const Tensor& wo, const Tensor& bo, const Tensor& ln2_w, const Tensor& ln2_b,
                        const Tensor& w_fc, const Tensor& b_fc, const Tensor& w_proj, const Tensor& b_proj, int64_t heads,
                        double eps) {
    const Tensor xc = x.contiguous();
    const int64_t b = x.size(0), s = x.size(1), d = x.size(2) / heads;
    const Layout at(b * s, x.size(2), w_fc.size(0), heads);
    const Tensor mid = at::empty({at.end}, x.options()), mid32 = empty_f32(at.end32, x);
    Tensor y = at::empty(x.sizes(), x.options());
    const Parts part{static_cast<char*>(mid.data_ptr())};
    float* m32 = f32(mid32);
    const Rows h1 = part(at.h1, at.h), qkv = part(at.qkv, 3 * at.h), o = part(at.o, at.h), a = part(at.u, at.h),
               sum = part(at.s, at.h), h2 = part(at.h2, at.h), u = part(at.u, at.f), g = part(at.g, at.f);
    const int dt = dtype_code(x);
    norm(xc.data_ptr(), nullptr, nullptr, ln1_w, ln1_b, h1, m32 + at.stats1, at, eps);
    forward_product(h1, wqkv, bqkv.data_ptr(), qkv, at.t);
    const auto p = heads_in(qkv, heads, d);
    attention_forward({b, s, d, 1.0 / std::sqrt((double)d)}, p[0], p[1], p[2], o.ptr, m32 + at.lse, dt);
    forward_product(o, wo, bo.data_ptr(), a, at.t);
    norm(xc.data_ptr(), a.ptr, sum.ptr, ln2_w, ln2_b, h2, m32 + at.stats2, at, eps);
    forward_product(h2, w_fc, nullptr, u, at.t);
    check(ft_bias_act_fwd(u.ptr, b_fc.data_ptr(), g.ptr, at.t, (int)at.f, 1, dt, stream()), "ft_bias_act_fwd");
    forward_product(g, w_proj, b_proj.data_ptr(), {y.data_ptr(), at.h}, at.t, sum);
    // not the norms' biases, which their ops do not keep either: the program may change them
    ctx->save_for_backward({xc, ln1_w, Tensor(), wqkv, bqkv, wo, bo, ln2_w, Tensor(), w_fc, b_fc, w_proj, b_proj, mid, mid32});
    ctx->saved_data["heads"] = heads;
    return y;
  }

  // Which inputs the running backward pass wants the gradients of.  They are numbered along the forward pass, so the backward ends
  // with the `first` of them.
  struct Wanted {
    bool input[INPUTS];
    int first = INPUTS;
    explicit Wanted(const AutogradContext* ctx) {
      for (int i = INPUTS - 1; i >= 0; --i)
        if ((input[i] = ctx->needs_input_grad(i))) first = i;
    }
  };

  // What is wanted of dX, dW and db of a projection; no `bias`: not its
  static void projection_backward(const variable_list& in, const Wanted& wanted, Rows dy, Rows x, int64_t rows, int w, bool bias, Rows dx,
                                  variable_list& out) {
    const int64_t n = in[w].size(0), k = in[w].size(1);
    const int dt = dtype_code(in[w]);
    const bool data = wanted.first < w, weight = wanted.input[w], sums = bias && wanted.input[w + 1];
    WeightGradient g;
    if (weight) {
      g = weight_buffer(in[w], rows, in[w].options());
      out[w] = g.gradient();
    }
    if (data && weight && both_gradients(dy, x, rows, in[w], dx, g, sums ? in[w + 1] : Tensor(), w + 1, out[w + 1])) return;
    if (data) check(product(dy, false, rows_of(in[w]), true, rows, k, n, dx, dt, dt, in[w]), "ft_gemm");
    if (weight && sums && weight_and_bias(dy, x, rows, g, in[w + 1], w + 1, out[w + 1])) return;
    if (weight) check(product(dy, true, x, true, n, k, rows, rows_of(g.dw), dt, dt, in[w], g.held), "ft_gemm");
    if (sums) out[w + 1] = bias_gradient(dy.ptr, rows, n, in[w + 1], w + 1);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto in = ctx->get_saved_variables();
    const Wanted wanted(ctx);
    const Tensor &x = in[X], dy = grads[0].contiguous();
    const int64_t heads = ctx->saved_data["heads"].toInt(), b = x.size(0), s = x.size(1), d = x.size(2) / heads;
    const Layout at(b * s, x.size(2), in[W_FC].size(0), heads);
    const int64_t t = at.t, h = at.h, f = at.f;
    const Parts mid{static_cast<char*>(in[INPUTS].data_ptr())};
    const float* m32 = f32(in[INPUTS + 1]);
    // dg and du, and where they lay do, dqkv and dh1; behind them dh2 and ds
    const int64_t behind = t * std::max(2 * f, 5 * h);
    const Tensor scratch = at::empty({behind + 2 * t * h}, x.options());
    const Parts tmp{static_cast<char*>(scratch.data_ptr())};
    const Rows dg = tmp(0, f), du = tmp(t * f, f), d_o = tmp(0, h), dqkv = tmp(t * h, 3 * h), dh1 = tmp(4 * t * h, h),
               dh2 = tmp(behind, h), ds = tmp(behind + t * h, h), dy2{dy.data_ptr(), h};
    variable_list out(INPUTS + 2);
    const int dt = dtype_code(x);
    LaterSums later{dt};
    projection_backward(in, wanted, dy2, mid(at.g, f), t, W_PROJ, true, dg, out);
    if (wanted.first <= B_FC) {
      const int64_t parts = ft_bias_act_bwd_parts(t, (int)f);
      Tensor part = empty_f32(parts * f, x);
      const RowSum db = row_sum(B_FC, in[B_FC], t);
      check(ft_bias_act_bwd(dg.ptr, mid(at.u, f).ptr, in[B_FC].data_ptr(), du.ptr, nullptr, f32(part), t, (int)f, 1, 0, dt, stream()),
            "ft_bias_act_bwd");
      later.keep(part, 0, db, parts, f);
      out[B_FC] = db.gradient();
    }
    if (wanted.first <= W_FC) projection_backward(in, wanted, du, mid(at.h2, h), t, W_FC, false, dh2, out);
    if (wanted.first <= LN2_B) {
      const auto n2 = norm_backward(mid(at.s, h).ptr, in[LN2_W], m32 + at.stats2 + t, m32 + at.stats2, dy.data_ptr(), dh2.ptr, ds.ptr,
                                    nullptr, t, h, LN2_W, &later);
      out[LN2_W] = n2.dw, out[LN2_B] = n2.db;
    }
    if (wanted.first <= BO) projection_backward(in, wanted, ds, mid(at.o, h), t, WO, true, d_o, out);
    if (wanted.first <= BQKV) {
      const auto p = heads_in(mid(at.qkv, 3 * h), heads, d), g = heads_in(dqkv, heads, d);
      attention_backward({b, s, d, 1.0 / std::sqrt((double)d)}, p[0], p[1], p[2], mid(at.o, h).ptr, m32 + at.lse, d_o.ptr, h, g[0],
                         g[1], g[2], x);
      projection_backward(in, wanted, dqkv, mid(at.h1, h), t, WQKV, true, dh1, out);
    }
    if (wanted.first <= LN1_B) {
      Tensor dx = at::empty(x.sizes(), x.options());
      const auto n1 = norm_backward(x.data_ptr(), in[LN1_W], m32 + at.stats1 + t, m32 + at.stats1, ds.ptr, dh1.ptr, dx.data_ptr(),
                                    nullptr, t, h, LN1_W, &later);
      out[X] = dx, out[LN1_W] = n1.dw, out[LN1_B] = n1.db;
    }
    if (later.n > 0) later.form();
    return out;
  }
};

// What the node takes: a training pass in which every parameter learns, tensors as the eight ops would hand them to their
// kernels, and a width of up to kBlockWork operations forward.  There a pass takes the device some 0.4 ms, longer than it takes the host
// either way, and the ops give their activations back one by one during backward.
constexpr double kBlockWork = 1e11;

bool block_covers(const Tensor& x, const std::vector<Tensor>& params, int64_t heads) {
  if (!at::GradMode::is_enabled() || x.dim() != 3 || x.numel() == 0) return false;
  const auto type = x.scalar_type();
  const int64_t h = x.size(2), f = params[Block::W_FC - 1].size(0);
  if ((type != at::kBFloat16 && type != at::kHalf) || heads <= 0 || h % heads || h % 8 || f % 8 || f == 0) return false;
  if (h / heads != 64 && h / heads != 128) return false;
  if (2.0 * (double)x.numel() * (double)(4 * h + 2 * f) > kBlockWork) return false;
  const int64_t rows[] = {h, h, 3 * h, 3 * h, h, h, h, h, f, f, h, h}, cols[] = {0, 0, h, 0, h, 0, 0, 0, h, 0, f, 0};
  for (size_t i = 0; i < params.size(); ++i) {
    const Tensor& p = params[i];
    if (!p.requires_grad() || !p.is_contiguous() || p.scalar_type() != type || p.device() != x.device() || p.size(0) != rows[i] ||
        p.dim() != (cols[i] ? 2 : 1) || (cols[i] && p.size(1) != cols[i]) || reinterpret_cast<uintptr_t>(p.data_ptr()) % 16)
      return false;
  }
  return reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 || !x.is_contiguous();
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using guard = py::call_guard<py::gil_scoped_release>;
  m.def("plain_backward", &plain_backward);            // of the pass that is running, for nodes written in Python
  m.def("linear", [](const Tensor& x, const Tensor& w, const OptTensor& bias, const OptTensor& res,
                     const OptTensor& done) { return Linear::apply(x, w, bias, res, done); }, guard());
  m.def("linear_swiglu", [](const Tensor& x, const Tensor& w) {
    const bool grad = at::GradMode::is_enabled() && (x.requires_grad() || w.requires_grad());
    return LinearSwiGLU::apply(x, w, grad);
  }, guard());
  m.def("swiglu", [](const Tensor& gate_up) { return SwiGLU::apply(gate_up); }, guard());
  m.def("norm", [](const Tensor& x, const Tensor& w, const OptTensor& b, double eps) {
    return Norm::apply(x, w, b, eps);
  }, guard());
  m.def("residual_norm", [](const Tensor& x, const Tensor& w, const OptTensor& b, double eps) {
    if (!at::GradMode::is_enabled()) return std::make_tuple(x, Norm::apply(x, w, b, eps));
    auto out = ResidualNorm::apply(x, w, b, eps);
    return std::make_tuple(out[0], out[1]);
  }, guard());
  m.def("add_norm", [](const Tensor& x, const Tensor& r, const Tensor& w, const OptTensor& b, double eps) {
    auto out = AddNorm::apply(x, r, w, b, eps);
    return std::make_tuple(out[0], out[1]);
  }, guard());
  m.def("bias_act", [](const Tensor& x, const Tensor& bias, int64_t act) { return BiasAct::apply(x, bias, act); },
        guard());
  m.def("rope_heads", [](const Tensor& x, const Tensor& cos, const Tensor& sin, int64_t heads, int64_t d) {
    return RopeHeads::apply(x, cos, sin, heads, d);
  }, guard());
  m.def("attention", [](const Tensor& q, const Tensor& k, const Tensor& v, double scale) {
    return Attention::apply(q, k, v, scale);
  }, guard());
  m.def("embedding", [](const Tensor& tokens, const Tensor& w) { return Embedding::apply(tokens, w); }, guard());
  // nothing where the block is not the node's
  m.def("gpt_block", [](const Tensor& x, const std::vector<Tensor>& p, int64_t heads, double eps) -> OptTensor {
    if (p.size() != Block::INPUTS - 1) throw py::value_error("gpt_block: twelve parameters");
    if (!block_covers(x, p, heads)) return std::nullopt;
    return Block::apply(x, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8], p[9], p[10], p[11], heads, eps);
  }, guard());
  m.def("attention_packed", [](const Tensor& qkv, int64_t hq, int64_t hkv, int64_t d, double scale) {
    return PackedAttention::apply(qkv, hq, hkv, d, scale);
  }, guard());
}
