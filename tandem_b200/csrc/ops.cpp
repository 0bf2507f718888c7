// The operators' host side for eager calls: the autograd functions of tandem_b200.ops, issued natively.
//
// A small layer's kernels take 5 - 10 us each, and a Python autograd function 20 - 40 us per call between its checks, its
// ctypes calls and the interpreter lock, which backward's threads wait for in turn.  Each function here does what the
// function of the same name in tandem_b200/ops does -- the same checks, allocations, kernels, streams and saved tensors -- without
// entering the interpreter.  The Python functions stay for what only they can answer: functorch transforms,
// forward-mode differentiation, tracing, and a weight whose all-gather rides in its GEMM.
// Measured on B200, us: linear forward + backward of 1537 x 768 x 1003 182 -> 94; one eager step of a model of two small blocks 2165 -> 1287;
// a forward pass of 24 blocks over 5 x 512 tokens 3571 -> 2511.
//
// The kernels are taken from libtb200_cuda.so at bind(), so that this library has no CUDA code of its own.
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../cuda/operators.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ---------------------------------------------------------------- the kernel library
// Types from the declarations that the kernels' own sources include, names from the same words.
#define TB_KERNELS(X)                                                                                                      \
  X(gemm, tb_gemm_bf16) X(gemm_workspace, tb_gemm_workspace_bytes) X(gemm_error_text, tb_gemm_last_error)                  \
  X(col_sum, tb_col_sum) X(ln_fwd, tb_layernorm_fwd) X(ln_bwd_slices, tb_layernorm_bwd_blocks)                             \
  X(ln_bwd, tb_layernorm_bwd_add) X(attn_fwd, tb_attn_fwd) X(attn_bwd, tb_attn_bwd)                                        \
  X(embed_fwd, tb_embed_fwd) X(embed_bwd, tb_embed_bwd) X(xent_fwd, tb_xent_fwd)                                           \
  X(xent_bwd, tb_xent_bwd) X(stream_wait, tb_stream_wait) X(error_string, tb_error_string)                                 \
  X(last_error, tb_last_error)

typedef cudaStream_t Stream;
struct Kernels {
#define MEMBER(member, name) decltype(&name) member;
  TB_KERNELS(MEMBER)
#undef MEMBER
};
Kernels K;

void bind(const std::string& path) {
  void* lib = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (lib == nullptr) throw std::runtime_error(dlerror());
  auto find = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(lib, name));
    if (fn == nullptr) throw std::runtime_error(std::string("libtb200_cuda.so lacks ") + name);
  };
#define FIND(member, name) find(K.member, #name);
  TB_KERNELS(FIND)
#undef FIND
}

void check(int rc, const char* what) {
  if (rc == 0) return;
  const std::string text = rc > 0 ? K.error_string(rc) : "code " + std::to_string(rc);
  throw std::runtime_error(std::string(what) + " failed: " + text + " (" + K.last_error() + ")");
}

// The current stream of t's device; host tensors are refused before a launch.
Stream stream_of(const Tensor& t) {
  if (!t.is_cuda()) throw py::value_error("Expected a cuda device, but got: " + t.device().str());
  return c10::cuda::getCurrentCUDAStream(t.get_device()).stream();
}

// ---------------------------------------------------------------- tensors
constexpr int BIAS = 1, GELU = 2, RESIDUAL = 4, DGELU = 8;

int64_t pad8(int64_t n) { return (n + 7) / 8 * 8; }

// A [rows, cols] view of [rows, pad8(cols)] storage: every row starts 16-byte aligned.
Tensor empty_padded(int64_t rows, int64_t cols, const at::TensorOptions& options) {
  const int64_t ld = pad8(cols);
  Tensor t = at::empty({rows, ld}, options);
  return ld == cols ? t : t.slice(1, 0, cols);
}

// The kernels take addresses and sizes: what would read beyond an operand is refused here, before a launch.
void need(bool ok, const char* what) {
  if (!ok) throw py::value_error(what);
}
void need_bf16(std::initializer_list<Tensor> tensors) {
  const Tensor* first = nullptr;
  for (const Tensor& t : tensors) {
    if (!t.defined()) continue;
    if (!t.is_cuda() || t.scalar_type() != at::kBFloat16)
      throw py::type_error("the sm_100a operators take bf16 CUDA tensors (cast the model with .bfloat16())");
    if (first == nullptr) first = &t;
    need(t.device() == first->device(), "the operands lie on different devices");
  }
}
void need_ids(const Tensor& ids, const Tensor& beside) {
  if (!ids.is_cuda() || ids.scalar_type() != at::kLong) throw py::type_error("token ids and targets are int64 CUDA tensors");
  need(ids.device() == beside.device(), "the operands lie on different devices");
}
// x . w^T + bias: of w's rows only their distance is free.
void need_product(const Tensor& x, const Tensor& w, const Tensor& bias) {
  need(x.dim() > 0 && w.dim() == 2, "a product takes an input of rows and a 2-D weight");
  need(x.size(-1) == w.size(1), "the input's width is not the weight's");
  need(w.stride(1) == 1 || w.size(1) == 1, "the weight's rows have to be contiguous");
  need(!bias.defined() || bias.numel() == w.size(0), "the bias has not one value per output");
}

bool misaligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0; }
// t, or a copy of it, for kernels that read it as a run of 16-byte vectors
Tensor vectors_of(const Tensor& t) {
  const Tensor c = t.contiguous();
  return misaligned(c) ? c.clone() : c;
}
void* data(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

struct Rows {
  Tensor t;
  int64_t ld;
};
// The 2-D view of a tensor whose last dimension is contiguous and whose rows are evenly strided (else a copy), and its row stride.
Rows rows_of(const Tensor& t) {
  Tensor t2 = t.dim() != 2 ? t.reshape({-1, t.size(-1)}) : t;
  if (t2.stride(1) != 1 || (t2.size(0) > 1 && t2.stride(0) % 8) || misaligned(t2)) {
    Tensor copy = empty_padded(t2.size(0), t2.size(1), t2.options());
    copy.copy_(t2);
    t2 = copy;
  }
  return {t2, t2.size(0) > 1 ? t2.stride(0) : pad8(t2.size(1))};
}

// t2's rows under the leading dimensions of `shape`.
Tensor with_rows_of(const Tensor& t2, at::IntArrayRef shape, int64_t width) {
  if (t2.is_contiguous()) {
    std::vector<int64_t> full(shape.begin(), shape.end());
    full.back() = width;
    return t2.view(full);
  }
  return t2.unflatten(0, shape.slice(0, shape.size() - 1));
}

// ---------------------------------------------------------------- products
// out[M, N] = op(a) . op(b) (+ epilogue); out and workspace are allocated here unless given, `on` overrides the stream.
Tensor gemm(const Tensor& a, const Tensor& b, int64_t M, int64_t N, int64_t k, int64_t lda, int64_t ldb, bool a_mn, bool b_mn, int flags,
            const Tensor& bias_in, Tensor aux_in, const Tensor& aux_out, Tensor out = {}, Tensor workspace = {}, Stream on = nullptr) {
  if (!out.defined()) out = empty_padded(M, N, a.options());
  if (k == 0) {  // a sum over nothing, as the weight gradient of an empty batch is: the kernel writes nothing
    need(flags == 0, "a product over no columns takes no bias and no other operand");
    return out.zero_();
  }
  const int64_t ldc = M > 1 ? out.stride(0) : pad8(N);
  const Tensor bias = bias_in.defined() ? bias_in.contiguous() : bias_in;
  if (aux_in.defined() && misaligned(aux_in)) aux_in = aux_in.clone();  // it is read in 16-byte vectors
  if (aux_in.defined() && M > 1 && aux_in.stride(0) != ldc) throw std::invalid_argument("aux_in must share the output's row stride");
  const long long need = K.gemm_workspace((int)M, (int)N, (int)k);
  if (need && !workspace.defined()) workspace = at::empty({need}, a.options().dtype(at::kByte));
  const int rc = K.gemm(data(a), data(b), data(out), (int)M, (int)N, (int)k, (int)lda, (int)ldb, (int)ldc, a_mn, b_mn, flags, data(bias),
                        data(aux_in), data(aux_out), 0, need ? data(workspace) : nullptr, need, on != nullptr ? on : stream_of(a));
  if (rc == -11 || rc == -12)
    throw std::runtime_error("gemm: operand not addressable by TMA (M=" + std::to_string(M) + " N=" + std::to_string(N) + " K=" + std::to_string(k) +
                             " lda=" + std::to_string(lda) + " ldb=" + std::to_string(ldb) + "): " + K.gemm_error_text());
  check(rc, "gemm");
  return out;
}

Tensor forward_product(const Rows& x, const Tensor& w, const Tensor& bias, int flags, const Tensor& aux_in, const Tensor& aux_out) {
  if (bias.defined()) flags |= BIAS;
  return gemm(x.t, w, x.t.size(0), w.size(0), x.t.size(1), x.ld, w.stride(0), false, false, flags, bias, aux_in, aux_out);
}

// dX[M, K] = dY[M, N] . W[N, K]
Tensor grad_input(const Rows& dy, const Rows& w, int flags = 0, const Tensor& aux_in = {}) {
  return gemm(dy.t, w.t, dy.t.size(0), w.t.size(1), dy.t.size(1), dy.ld, w.ld, false, true, flags, {}, aux_in, {});
}

// dW[N, K] = dY[M, N]^T . X[M, K]
Tensor grad_weight(const Rows& dy, const Rows& x) {
  return gemm(dy.t, x.t, dy.t.size(1), x.t.size(1), dy.t.size(0), dy.ld, x.ld, true, true, 0, {}, {}, {}).contiguous();
}

void column_sums(const Rows& dy, const Tensor& out, const Tensor& scratch, Stream on) {
  check(K.col_sum(data(dy.t), (int)dy.t.size(0), (int)dy.t.size(1), (int)dy.ld, data(out), (float*)data(scratch), on), "col_sum");
}

// One second stream per device for the parameter gradients of small layers.
Stream side_stream(int device) {
  static std::mutex lock;
  static std::vector<std::optional<c10::cuda::CUDAStream>> streams;
  std::lock_guard<std::mutex> hold(lock);
  if ((int)streams.size() <= device) streams.resize(device + 1);
  if (!streams[device]) streams[device] = c10::cuda::getStreamFromPool(false, device);
  return streams[device]->stream();
}

// dW = dY^T . X and dB = column sums of dY, beside the input gradient on a second stream where a layer has few rows (neither
// fills the GPU by itself).  Everything that the second stream touches is allocated on the caller's stream beforehand and is
// released after join(), which makes that stream wait: the caching allocator never sees a block used by a stream that it does not know about.
// The fork is made by start(), not by a constructor: one that throws leaves no object to join.
struct ParameterGrads {
  Tensor dw, db;
  Tensor scratch, workspace;
  Stream main = nullptr, beside = nullptr;

  void start(const Rows& dy, const Rows& x, bool want_w, bool want_b, int64_t side_below) {
    const int64_t M = dy.t.size(0), N = dy.t.size(1), k = x.t.size(1);
    if (!want_w && !want_b) return;
    const auto options = dy.t.options();
    if (want_b) {
      db = at::empty({N}, options);
      scratch = at::empty({32 * N}, options.dtype(at::kFloat));
    }
    if (M >= side_below) {
      if (want_w) dw = grad_weight(dy, x);
      if (want_b) column_sums(dy, db, scratch, stream_of(dy.t));
      return;
    }
    if (want_w && pad8(k) != k) {  // a padded product needs a compaction copy afterwards: keep that case on one stream
      dw = grad_weight(dy, x);
      want_w = false;
    } else if (want_w) {
      dw = at::empty({N, k}, options);
      const long long need = K.gemm_workspace((int)N, (int)k, (int)M);
      if (need) workspace = at::empty({need}, options.dtype(at::kByte));
    }
    main = stream_of(dy.t);
    Stream side = side_stream((int)dy.t.get_device());
    check(K.stream_wait(side, main), "stream wait");
    beside = side;
    if (want_w) gemm(dy.t, x.t, N, k, M, dy.ld, x.ld, true, true, 0, {}, {}, {}, dw, workspace, beside);
    if (want_b) column_sums(dy, db, scratch, beside);
  }
  void join() {
    if (beside != nullptr) check(K.stream_wait(main, beside), "stream wait");
    beside = nullptr;
  }
  ~ParameterGrads() {  // a call that ends in an exception joins too, before its buffers are given back
    if (beside != nullptr) K.stream_wait(main, beside);
  }
};

Tensor undefined_if_none(const std::optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }

// ---------------------------------------------------------------- functions
// What backward needs beside the saved tensors.  Not their strides: a saved-tensor hook may answer with others (save_on_cpu does).
enum { NEEDS = 0, SIDE = 1, SHAPE = 2 };

struct Linear : torch::autograd::Function<Linear> {
  static Tensor run(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& residual, int64_t side_below) {
    need_bf16({x, w, bias, residual});
    need_product(x, w, bias);
    const Rows x2 = rows_of(x);
    Tensor res2;
    if (residual.defined()) {
      res2 = residual.reshape({-1, residual.size(-1)});
      if (pad8(w.size(0)) != w.size(0) || !res2.is_contiguous())
        throw py::value_error("a fused residual needs a contiguous tensor whose width is a multiple of 8");
      need(res2.size(0) == x2.t.size(0) && res2.size(1) == w.size(0), "the residual has not the output's shape");
    }
    const Tensor y = forward_product(x2, w, bias, residual.defined() ? RESIDUAL : 0, res2, {});
    if (ctx != nullptr) {
      ctx->save_for_backward({x2.t, w});
      const auto wants = [](const Tensor& t) { return t.defined() && t.requires_grad(); };
      std::vector<int64_t> keep{wants(x) | wants(w) << 1 | wants(bias) << 2 | wants(residual) << 3, side_below};
      keep.insert(keep.end(), x.sizes().begin(), x.sizes().end());
      ctx->saved_data["keep"] = std::move(keep);
    }
    return with_rows_of(y, x.sizes(), w.size(0));
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const std::optional<Tensor>& bias,
                        const std::optional<Tensor>& residual, int64_t side_below) {
    return run(ctx, x, w, undefined_if_none(bias), undefined_if_none(residual), side_below);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const std::vector<int64_t> keep = ctx->saved_data["keep"].toIntVector();
    const Rows x = rows_of(saved[0]), w = rows_of(saved[1]), dy = rows_of(grads[0]);
    ParameterGrads parameters;
    parameters.start(dy, x, keep[NEEDS] & 2, keep[NEEDS] & 4, keep[SIDE]);
    Tensor dx;
    if (keep[NEEDS] & 1) dx = with_rows_of(grad_input(dy, w), at::IntArrayRef(keep).slice(SHAPE), w.t.size(1));
    parameters.join();
    return {dx, parameters.dw, parameters.db, keep[NEEDS] & 8 ? grads[0] : Tensor(), Tensor()};
  }
};

struct MLP : torch::autograd::Function<MLP> {
  static Tensor run(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const Tensor& b1, const Tensor& w2, const Tensor& b2,
                    const Tensor& residual, int64_t side_below) {
    need_bf16({x, w1, b1, w2, b2, residual});
    if (!residual.defined()) throw py::value_error("ops.mlp adds its input stream: pass the residual tensor");
    if (w1.size(0) % 8 || w2.size(0) % 8) throw py::value_error("ops.mlp needs hidden and output widths that are multiples of 8 (16-byte rows)");
    need_product(x, w1, b1);
    need(w2.dim() == 2 && w2.size(1) == w1.size(0), "the second weight's width is not the hidden one");
    need(w2.stride(1) == 1 || w2.size(1) == 1, "the weight's rows have to be contiguous");
    need(!b2.defined() || b2.numel() == w2.size(0), "the bias has not one value per output");
    const Rows x2 = rows_of(x);
    const Tensor res2 = residual.reshape({-1, residual.size(-1)});
    need(res2.size(0) == x2.t.size(0) && res2.size(1) == w2.size(0) && res2.stride(1) == 1, "the residual has not the output's shape");
    const Tensor slope = empty_padded(x2.t.size(0), w1.size(0), x.options());  // gelu'(W1 . x + b1), written by the same epilogue
    const Tensor h = forward_product(x2, w1, b1, GELU, {}, slope);
    const Tensor y = forward_product({h, h.stride(0)}, w2, b2, RESIDUAL, res2, {});
    if (ctx != nullptr) {
      ctx->save_for_backward({x2.t, w1, w2, slope, h});
      const auto wants = [](const Tensor& t) { return t.defined() && t.requires_grad(); };
      std::vector<int64_t> keep{wants(x) | wants(w1) << 1 | wants(b1) << 2 | wants(w2) << 3 | wants(b2) << 4 | wants(residual) << 5, side_below};
      keep.insert(keep.end(), x.sizes().begin(), x.sizes().end());
      ctx->saved_data["keep"] = std::move(keep);
    }
    return with_rows_of(y, x.sizes(), w2.size(0));
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const std::optional<Tensor>& b1, const Tensor& w2,
                        const std::optional<Tensor>& b2, const Tensor& residual, int64_t side_below) {
    return run(ctx, x, w1, undefined_if_none(b1), w2, undefined_if_none(b2), residual, side_below);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const std::vector<int64_t> keep = ctx->saved_data["keep"].toIntVector();
    const int64_t needs = keep[NEEDS];
    const Rows x = rows_of(saved[0]), w1 = rows_of(saved[1]), w2 = rows_of(saved[2]), hidden = rows_of(saved[4]), dy = rows_of(grads[0]);
    const Tensor slope = saved[3].contiguous();
    ParameterGrads second;
    second.start(dy, hidden, needs & 8, needs & 16, keep[SIDE]);
    const Tensor dpre = grad_input(dy, w2, DGELU, slope);  // (dY . W2) * gelu'(pre)
    second.join();
    const Rows pre{dpre, dpre.stride(0)};
    ParameterGrads first;
    first.start(pre, x, needs & 2, needs & 4, keep[SIDE]);
    Tensor dx;
    if (needs & 1) dx = with_rows_of(grad_input(pre, w1), at::IntArrayRef(keep).slice(SHAPE), w1.t.size(1));
    first.join();
    return {dx, first.dw, first.db, second.dw, second.db, needs & 32 ? grads[0] : Tensor(), Tensor()};
  }
};

// x -> LayerNorm(x), its rows' mean and 1 / std
struct Normed {
  Tensor x2, y, stats;
};
Normed normalize(const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
  need_bf16({x, w, b});
  need(x.dim() > 0 && w.numel() == x.size(-1) && b.numel() == x.size(-1), "layer_norm takes a weight and a bias with one value per column");
  Normed n;
  n.x2 = vectors_of(x.reshape({-1, x.size(-1)}));
  const int64_t M = n.x2.size(0);
  n.y = at::empty_like(n.x2);
  n.stats = at::empty({2, M}, x.options().dtype(at::kFloat));
  float* stats = (float*)data(n.stats);
  const Tensor gain = vectors_of(w), shift = vectors_of(b);
  check(K.ln_fwd(data(n.x2), data(gain), data(shift), data(n.y), stats, stats + M, (int)M, (int)n.x2.size(1), (float)eps, stream_of(x)),
        "layernorm forward");
  return n;
}
variable_list normalize_backward(const variable_list& saved, const Tensor& dy, const Tensor& second) {
  const Tensor x2 = vectors_of(saved[0]), w = saved[1], stats = saved[2].contiguous();
  const int64_t M = x2.size(0), D = x2.size(1);
  const Tensor dy2 = vectors_of(dy.reshape({-1, D})), add = second.defined() ? vectors_of(second.reshape({-1, D})) : Tensor(), gain = vectors_of(w);
  const Tensor dx = at::empty_like(x2), dw = at::empty_like(w, at::MemoryFormat::Contiguous), db = at::empty_like(dw);
  const Tensor scratch = at::empty({(int64_t)K.ln_bwd_slices((int)M) * 2 * D}, x2.options().dtype(at::kFloat));
  const float* mean = (const float*)data(stats);
  check(K.ln_bwd(data(dy2), data(x2), data(gain), mean, mean + M, data(add), data(dx), data(dw), data(db), (float*)data(scratch), (int)M, (int)D,
                 stream_of(x2)),
        "layernorm backward");
  return {dx.view(dy.sizes()), dw, db, Tensor()};
}

struct LayerNorm : torch::autograd::Function<LayerNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
    const Normed n = normalize(x, w, b, eps);
    if (ctx != nullptr) ctx->save_for_backward({n.x2, w, n.stats});
    return n.y.view(x.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return normalize_backward(ctx->get_saved_variables(), grads[0], {});
  }
};

struct ResidualLayerNorm : torch::autograd::Function<ResidualLayerNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
    const Normed n = normalize(x, w, b, eps);
    if (ctx != nullptr) ctx->save_for_backward({n.x2, w, n.stats});
    return {x.view_as(x), n.y.view(x.sizes())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (!grads[1].defined()) return {grads[0], Tensor(), Tensor(), Tensor()};
    return normalize_backward(ctx->get_saved_variables(), grads[1], grads[0]);
  }
};

struct CausalAttention : torch::autograd::Function<CausalAttention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv_in, int64_t heads) {
    need_bf16({qkv_in});
    if (qkv_in.dim() != 3) throw py::value_error("causal_attention takes [batch, time, 3 * dim]");
    const int64_t B = qkv_in.size(0), T = qkv_in.size(1), d = qkv_in.size(2) / 3, hd = d / heads;
    if (T % 128 || (hd != 64 && hd != 128))
      throw py::value_error("causal_attention kernels need T % 128 == 0 and head dim 64 or 128 (got T=" + std::to_string(T) + ", head dim " +
                            std::to_string(hd) + ")");
    need(qkv_in.size(2) == 3 * heads * hd, "causal_attention takes queries, keys and values of heads * head dim columns each");
    const Tensor qkv = qkv_in.contiguous();
    const Tensor out = at::empty({B, T, d}, qkv.options()), lse = at::empty({B, heads, T}, qkv.options().dtype(at::kFloat));
    check(K.attn_fwd(data(qkv), data(out), (float*)data(lse), (int)B, (int)T, (int)heads, (int)hd, stream_of(qkv)), "attention forward");
    if (ctx != nullptr) {
      ctx->save_for_backward({qkv, out, lse});
      ctx->saved_data["heads"] = heads;
    }
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor qkv = vectors_of(saved[0]), out = vectors_of(saved[1]), lse = vectors_of(saved[2]);
    const int64_t B = qkv.size(0), T = qkv.size(1), d = qkv.size(2) / 3, heads = ctx->saved_data["heads"].toInt();
    const Tensor d_out = vectors_of(grads[0]), dqkv = at::empty_like(qkv), delta = at::empty({B * heads * T}, qkv.options().dtype(at::kFloat));
    check(K.attn_bwd(data(qkv), data(out), data(d_out), (const float*)data(lse), data(dqkv), (float*)data(delta), (int)B, (int)T, (int)heads,
                     (int)(d / heads), stream_of(qkv)),
          "attention backward");
    return {dqkv, Tensor()};
  }
};

struct Embedding : torch::autograd::Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& idx_in, const Tensor& tok, const Tensor& pos) {
    need_bf16({tok, pos});
    if (idx_in.dim() != 2) throw py::value_error("embedding takes [batch, time] token ids");
    need_ids(idx_in, tok);
    need(tok.dim() == 2 && pos.dim() == 2 && tok.size(1) == pos.size(1), "embedding takes two 2-D tables of one width");
    need(idx_in.size(1) <= pos.size(0), "more positions than the table has rows");
    const int64_t B = idx_in.size(0), T = idx_in.size(1), D = tok.size(1);
    const Tensor idx = idx_in.contiguous(), tokens = vectors_of(tok), positions = vectors_of(pos);
    const Tensor out = at::empty({B, T, D}, tok.options());
    check(K.embed_fwd((const long long*)data(idx), data(tokens), data(positions), data(out), (int)(B * T), (int)T, (int)D, stream_of(tok)), "embedding forward");
    if (ctx != nullptr) {
      ctx->save_for_backward({idx});
      ctx->saved_data["sizes"] = std::vector<int64_t>{tok.size(0), D, pos.size(0)};
    }
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor idx = ctx->get_saved_variables()[0].contiguous();
    const std::vector<int64_t> sizes = ctx->saved_data["sizes"].toIntVector();
    const int64_t B = idx.size(0), T = idx.size(1), V = sizes[0], D = sizes[1], S = sizes[2];
    const Tensor dy = vectors_of(grads[0]);
    const auto bf16 = dy.options().dtype(at::kBFloat16);
    const Tensor dtok32 = at::zeros({V, D}, dy.options().dtype(at::kFloat)), dtok = at::empty({V, D}, bf16), dpos = at::zeros({S, D}, bf16);
    check(K.embed_bwd((const long long*)data(idx), data(dy), (float*)data(dtok32), data(dtok), data(dpos), (int)B, (int)T, (int)D, (int)V,
                      stream_of(dy)),
          "embedding backward");
    return {Tensor(), dtok, dpos};
  }
};

// Backward writes rows of logits where they lie: none may share memory with another.
Tensor rows_apart(const Tensor& t) { return t.stride(1) != 1 || (t.size(0) > 1 && t.stride(0) < t.size(1)) ? t.contiguous() : t; }

struct CrossEntropy : torch::autograd::Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits_in, const Tensor& targets_in) {
    need_bf16({logits_in});
    if (logits_in.dim() != 2) throw py::value_error("cross_entropy takes [rows, vocab] logits");
    need_ids(targets_in, logits_in);
    const int64_t rows = logits_in.size(0), V = logits_in.size(1);
    need(targets_in.numel() == rows, "cross_entropy takes one target per row");
    const Tensor logits = rows_apart(logits_in);
    const int64_t ld = rows > 1 ? logits.stride(0) : V;
    const Tensor targets = targets_in.contiguous();
    const auto f32 = logits.options().dtype(at::kFloat);
    const Tensor lse = at::empty({rows}, f32), row_loss = at::empty({rows}, f32), loss = at::empty({}, f32);
    check(K.xent_fwd(data(logits), (const long long*)data(targets), (float*)data(lse), (float*)data(row_loss), (float*)data(loss), (int)rows, (int)V,
                     (int)ld, stream_of(logits)),
          "cross-entropy forward");
    if (ctx != nullptr) ctx->save_for_backward({logits, targets, lse});
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor logits = rows_apart(saved[0]), targets = saved[1].contiguous(), lse = saved[2].contiguous();
    const int64_t rows = logits.size(0), V = logits.size(1), ld = rows > 1 ? logits.stride(0) : V;
    const Tensor scale = grads[0].detach().reshape({1}).to(at::kFloat).contiguous();
    // In place: the saved logits become their own gradient (they are not needed again).  The columns [V, ld) of a row are cleared
    // too when they belong to this tensor's storage (a padded allocation).
    const int64_t last = logits.storage_offset() + (rows - 1) * logits.stride(0) + ld;
    const bool owns = last <= (int64_t)(logits.storage().nbytes() / logits.element_size());
    check(K.xent_bwd(data(logits), (const long long*)data(targets), (const float*)data(lse), (const float*)data(scale), (int)rows, (int)V, (int)ld,
                     (int)(ld - V < 8 && owns ? ld : V), stream_of(logits)),
          "cross-entropy backward");
    return {logits, Tensor()};
  }
};

// Where gradients are off nothing can ask for the node: the forward alone.  Without the interpreter lock: an allocation or a launch
// may have to wait for the GPU, and other threads go on meanwhile, as they do beside ctypes (saved-tensor hooks take the lock themselves).
template <typename F, typename... Args>
auto call(const Args&... args) {
  py::gil_scoped_release unlocked;
  return at::GradMode::is_enabled() ? F::apply(args...) : F::forward(nullptr, args...);
}

// Looked for in the file by the build, which cannot import a library of another torch.
__attribute__((used)) const char built_for[] = BUILT_FOR;

}  // namespace

PYBIND11_MODULE(_ops, m) {
  using Maybe = std::optional<Tensor>;
  m.def("bind", &bind);
  m.def("linear", [](const Tensor& x, const Tensor& w, const Maybe& bias, const Maybe& residual, int64_t side_below) {
    return call<Linear>(x, w, bias, residual, side_below);
  });
  m.def("mlp", [](const Tensor& x, const Tensor& w1, const Maybe& b1, const Tensor& w2, const Maybe& b2, const Tensor& residual, int64_t side_below) {
    return call<MLP>(x, w1, b1, w2, b2, residual, side_below);
  });
  m.def("layer_norm", [](const Tensor& x, const Tensor& w, const Tensor& b, double eps) { return call<LayerNorm>(x, w, b, eps); });
  m.def("residual_layer_norm", [](const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
    const variable_list out = call<ResidualLayerNorm>(x, w, b, eps);
    return py::make_tuple(out[0], out[1]);
  });
  m.def("causal_attention", [](const Tensor& qkv, int64_t heads) { return call<CausalAttention>(qkv, heads); });
  m.def("embedding", [](const Tensor& idx, const Tensor& tok, const Tensor& pos) { return call<Embedding>(idx, tok, pos); });
  m.def("cross_entropy", [](const Tensor& logits, const Tensor& targets) { return call<CrossEntropy>(logits, targets); });
}
