// Eager calls of the fused layers and losses, as autograd functions in C++.
//
// A layer that is not replayed from a CUDA graph costs its host more than its device: an autograd function in Python, its
// allocations and some twenty foreign-function arguments per launch took 20 to 60 us where the kernels behind them take 5 to 25
// (a bottleneck block, forward and backward: 51 launches, 378 us on the device, 1110 on the host).  Here a call of Python's is one
// node of the graph, whose backward does not enter the interpreter at all, and a convolution and its BatchNorm are one node.  The
// kernels, their order and their results are those of the functions of the same names in `tspipe_b200/ops`, which stay in use
// where a stage is being recorded (they add small gradients in place there), under a functorch transform or a trace, and for all
// that the conditions at the callers leave out.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>

#include "../tspipe_kernels.h"

#define TSP_DTYPE_F32 0
#define TSP_DTYPE_BF16 1

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

std::atomic<int64_t> g_launches{0};
std::atomic<bool> g_accumulate{true};        // conv.set_accumulate_in_place

void check(int code, const char* what) { TORCH_CHECK(code == 0, what, " failed with code ", code); }
cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? TSP_DTYPE_BF16 : TSP_DTYPE_F32; }
bool aligned(const Tensor& t) { return ((uintptr_t)t.data_ptr() & 15) == 0; }
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const float* fptr(const Tensor& t) { return static_cast<const float*>(ptr(t)); }
at::TensorOptions f32_like(const Tensor& t) { return t.options().dtype(at::kFloat); }
Tensor zeroed_f32(int64_t n, const Tensor& like, cudaStream_t st) {
  Tensor t = at::empty({n}, f32_like(like));
  check((int)cudaMemsetAsync(t.data_ptr(), 0, n * sizeof(float), st), "cudaMemsetAsync");
  return t;
}

// A tensor whose memory a kernel can read: no batched or otherwise wrapped stand-in.
bool plain(const Tensor& t) {
  constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                         c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
                                         c10::DispatchKey::Batched});
  return t.defined() && t.is_cuda() && !t.key_set().has_any(wrapped);
}

// [N, C, H, W] with channels innermost, which a single pixel's are in either format
bool nhwc(const Tensor& t) {
  if (t.dim() != 4) return false;
  const int64_t c = t.size(1), h = t.size(2), w = t.size(3);
  if (h * w == 1 && t.is_contiguous()) return true;
  return t.stride(1) == 1 && t.stride(3) == c && t.stride(2) == w * c && t.stride(0) == h * w * c;
}
// (rows, channels) of a matrix with channels innermost, or (0, 0)
std::pair<int64_t, int64_t> rows_of(const Tensor& t) {
  if (t.dim() == 2 && t.is_contiguous()) return {t.size(0), t.size(1)};
  if (nhwc(t)) return {t.size(0) * t.size(2) * t.size(3), t.size(1)};
  return {0, 0};
}
// A gradient of `like` as the kernels read it.
Tensor gradient_like(Tensor g, const Tensor& like) {
  if (g.scalar_type() != like.scalar_type() || rows_of(g) != rows_of(like))
    g = g.to(like.scalar_type()).contiguous(like.dim() == 4 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::Contiguous);
  return aligned(g) ? g : g.clone(at::MemoryFormat::Preserve);
}

bool owns_saved() { return !at::SavedTensorDefaultHooks::get_hooks().has_value(); }

// Whether autograd's accumulation of p's gradient runs on `st`.  Autograd orders the accumulation, and the caller of backward()
// behind it, by the stream on which the accumulating node was made, and for the gradients that this node is handed; an
// addition that a backward launches itself is in that order on that very stream and on no other.
bool accumulates_on(const Tensor& p, cudaStream_t st) {
  const auto node = torch::autograd::impl::try_get_grad_accumulator(p);
  const auto own = node ? node->stream() : std::nullopt;
  return own.has_value() && own->device() == p.device() && c10::cuda::CUDAStream(*own).stream() == st;
}

// The fp32 gradient of a leaf that a kernel on `st` can add to in place: the weight's elements in the order [rows][taps][columns].
Tensor grad_target(const Tensor& weight, cudaStream_t st) {
  if (!g_accumulate.load(std::memory_order_relaxed) || !weight.is_leaf() || !accumulates_on(weight, st)) return {};
  const Tensor& g = weight.grad();
  if (!g.defined() || g.scalar_type() != at::kFloat || g.sizes() != weight.sizes() || g.layout() != at::kStrided || !g.is_cuda())
    return {};
  if (weight.dim() == 4) return g.permute({0, 2, 3, 1}).is_contiguous() ? g : Tensor();
  return g.is_contiguous() && aligned(g) ? g : Tensor();
}

// The fp32 gradient of a vector parameter that a backward may add to itself on `st`, in place of the node that accumulates it: in a
// backward() over the whole graph (one that was asked for gradients by name lists what to execute), without a recorded graph of
// its own, for a leaf with a gradient whose hooks want to see nothing and no search for NaN, on the stream of the accumulation.  (The
// kernels read, add and write: two of them on two streams would lose one's sums.)  The caller bumps its version, as the node would have.
Tensor accumulated(const Tensor& p, cudaStream_t st) {
  namespace ag = torch::autograd;
  const auto* listed = ag::get_current_graph_task_exec_info();
  if (!g_accumulate.load(std::memory_order_relaxed) || ag::AnomalyMode::is_enabled()) return {};
  if (listed == nullptr || !listed->empty() || at::GradMode::is_enabled() || !p.is_leaf() || !p.requires_grad()) return {};
  const Tensor& g = p.grad();
  if (!g.defined() || !plain(g) || g.layout() != at::kStrided || g.scalar_type() != at::kFloat || g.sizes() != p.sizes() || !g.is_contiguous() ||
      g.get_device() != p.get_device())
    return {};
  if (!ag::impl::hooks(p).empty() || ag::impl::post_acc_grad_hooks(p) != nullptr) return {};
  if (const auto node = ag::impl::try_get_grad_accumulator(p);
      node && !(node->pre_hooks().empty() && node->post_hooks().empty() && node->tensor_pre_hooks().empty()))
    return {};
  return accumulates_on(p, st) ? g : Tensor();
}

struct ConvGeom {
  int n, h, w, cin, cout, k, s, ho, wo;
  ConvGeom(const Tensor& x, const Tensor& weight, int64_t stride)
      : n(x.size(0)), h(x.size(2)), w(x.size(3)), cin(x.size(1)), cout(weight.size(0)), k(weight.size(2)), s(stride) {
    const int pad = (k - 1) / 2;
    ho = (h + 2 * pad - k) / s + 1;
    wo = (w + 2 * pad - k) / s + 1;
  }
  int64_t pixels() const { return (int64_t)n * ho * wo; }
};

// The accumulators of a BatchNorm layer (see `batchnorm.py: BatchNormGroup`).
struct Accumulators {
  float *sum, *sumsq, *count;
  int64_t stride;
};

// Forward of a training-mode BatchNorm from its statistics [segs][sum | sum of squares] at `sums`; [segs][mean | rstd] follow.
void bn_apply(const Tensor& x, const Tensor& res, const Tensor& y, float* sums, const Tensor& w, const Tensor& b,
              const Accumulators& acc, int64_t m, int c, double eps, bool relu, int segs, cudaStream_t st) {
  check(tsp_bn_apply(ptr(x), ptr(res), ptr(y), sums, nullptr, fptr(w), fptr(b), sums + (int64_t)segs * 2 * c, acc.sum, acc.sumsq,
                     acc.count, acc.stride, m, c, (float)eps, relu ? 1 : 0, dtype_code(x), segs, st),
        "tsp_bn_apply");
  g_launches += 1;
}

struct BnGrads {
  Tensor dx, dres, dw, db;      // dres: the residual's gradient; dw, db: undefined where they have been added to w's and b's
};
// Backward of it; `y`: the output, where its sign tells what the ReLU passed (with a residual).
BnGrads bn_backward(const Tensor& dy, const Tensor& x, const Tensor& y, const float* mean_rstd, const Tensor& w, const Tensor& b,
                    bool relu, bool has_res, bool params, int64_t m, int c, int segs, cudaStream_t st) {
  BnGrads g;
  Tensor add_w = params ? accumulated(w, st) : Tensor(), add_b = params ? accumulated(b, st) : Tensor();
  const bool add = add_w.defined() && add_b.defined();
  if (add) {
    torch::autograd::impl::bump_version(add_w);
    torch::autograd::impl::bump_version(add_b);
  }
  g.dx = at::empty_like(x);
  const bool masked = has_res && relu;
  if (masked) g.dres = at::empty_like(x);
  // (the sums over all views: behind theirs)
  const bool behind = segs > 1 && !add;
  const Tensor sums = zeroed_f32((int64_t)(behind ? segs + 1 : segs) * 2 * c, x, st);
  float* s = sums.data_ptr<float>();
  float* gw = add ? add_w.data_ptr<float>() : behind ? s + (int64_t)(segs * 2 + 1) * c : nullptr;
  float* gb = add ? add_b.data_ptr<float>() : behind ? s + (int64_t)segs * 2 * c : nullptr;
  check(tsp_bn_bwd_reduce(ptr(dy), ptr(x), ptr(y), ptr(g.dres), mean_rstd, fptr(w), fptr(b), relu ? 1 : 0, m, c, dtype_code(x), s,
                          segs, st),
        "tsp_bn_bwd_reduce");
  check(tsp_bn_bwd_apply(masked ? ptr(g.dres) : ptr(dy), ptr(x), masked ? nullptr : ptr(y), mean_rstd, fptr(w), fptr(b),
                         masked ? 0 : (relu ? 1 : 0), s, ptr(g.dx), gw, gb, m, c, dtype_code(x), segs, st),
        "tsp_bn_bwd_apply");
  g_launches += 3;
  if (!add) {
    const int64_t at = behind ? (int64_t)segs * 2 * c : 0;
    g.db = sums.narrow(0, at, c);
    g.dw = sums.narrow(0, at + c, c);
  }
  if (has_res && !masked) g.dres = dy;
  return g;
}

// relu(bn(conv(x)) + residual), 1x1 or 3x3; with `fork`, x is handed on as a second output, whose gradient the data gradient
// takes along.
struct ConvBnAct : Function<ConvBnAct> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& w16,
                               const Tensor& bn_w, const Tensor& bn_b, const std::optional<Tensor>& res, const Tensor& acc_sum,
                               const Tensor& acc_sumsq, const Tensor& acc_count, int64_t acc_stride, double eps, bool relu,
                               int64_t stride, int64_t segs, bool stats, bool fork, const Tensor& status) {
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t st = stream_of(x);
    const ConvGeom g(x, weight, stride);
    const Tensor y = at::empty({g.n, g.cout, g.ho, g.wo}, x.options(), at::MemoryFormat::ChannelsLast);
    const Tensor out = at::empty_like(y);
    const Tensor sums = at::empty({segs * 4 * g.cout}, f32_like(x));
    float* s = sums.data_ptr<float>();
    int* word = status.data_ptr<int>();
    if (stats) check((int)cudaMemsetAsync(s, 0, segs * 2 * g.cout * sizeof(float), st), "cudaMemsetAsync");
    check(tsp_conv_fprop(ptr(x), ptr(w16), ptr(y), stats ? s : nullptr, (int)segs, g.n, g.h, g.w, g.cin, g.cout, g.k, g.s, word,
                         st),
          "tsp_conv_fprop");
    if (!stats) check(tsp_bn_stats(ptr(y), g.pixels(), g.cout, TSP_DTYPE_BF16, s, (int)segs, st), "tsp_bn_stats");
    g_launches += stats ? 1 : 3;
    const Accumulators acc = {acc_sum.data_ptr<float>(), acc_sumsq.data_ptr<float>(), acc_count.data_ptr<float>(), acc_stride};
    const bool has_res = res.has_value();
    bn_apply(y, res.value_or(Tensor()), out, s, bn_w, bn_b, acc, g.pixels(), g.cout, eps, relu, (int)segs, st);
    ctx->set_materialize_grads(false);
    // The convolution's output is for the first half of the backward alone and is let go behind it (hooks on saved tensors get
    // it as all others).
    const bool own = owns_saved();
    if (own) ctx->saved_data["y"] = y;
    ctx->save_for_backward({x, weight, bn_w, bn_b, own ? Tensor() : y, sums, relu && has_res ? out : Tensor()});
    ctx->saved_data["w16"] = w16;             // (not for hooks on saved tensors, which may hand back copies)
    ctx->saved_data["status"] = status;
    ctx->saved_data["o"] = std::vector<int64_t>{stride, segs, relu, has_res, fork};
    if (fork) return {out, x.view_as(x)};
    return {out};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list r(17);
    const auto o = ctx->saved_data["o"].toIntVector();
    const bool fork = o[4] != 0;
    const Tensor dskip = fork ? grads[1] : Tensor();
    if (!grads[0].defined()) {
      r[0] = dskip;
      return r;
    }
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &weight = saved[1], &bn_w = saved[2], &bn_b = saved[3], &sums = saved[5], &out = saved[6],
                 w16 = ctx->saved_data["w16"].toTensor();
    Tensor y = saved[4];
    if (!y.defined()) {
      y = ctx->saved_data["y"].toTensor();
      if (!torch::autograd::get_current_graph_task_keep_graph()) ctx->saved_data.erase("y");
    }
    int* word = ctx->saved_data["status"].toTensor().data_ptr<int>();
    const int segs = (int)o[1];
    const bool relu = o[2] != 0, has_res = o[3] != 0;
    const at::NoGradGuard no_grad;
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t st = stream_of(x);
    const ConvGeom g(x, weight, o[0]);
    const BnGrads b = bn_backward(gradient_like(grads[0], y), y, out, sums.data_ptr<float>() + (int64_t)segs * 2 * g.cout, bn_w,
                                  bn_b, relu, has_res, ctx->needs_input_grad(3) && ctx->needs_input_grad(4), g.pixels(), g.cout, segs, st);
    y = Tensor();
    if (ctx->needs_input_grad(3)) r[3] = b.dw;
    if (ctx->needs_input_grad(4)) r[4] = b.db;
    r[5] = b.dres;
    if (ctx->needs_input_grad(0)) {
      const bool fits = dskip.defined() && dskip.scalar_type() == x.scalar_type() && nhwc(dskip) && aligned(dskip);
      Tensor dx = at::empty_like(x);
      check(tsp_conv_dgrad(ptr(b.dx), ptr(w16), fits ? ptr(dskip) : nullptr, ptr(dx), g.n, g.h, g.w, g.cin, g.cout, g.k, g.s, word,
                           st),
            "tsp_conv_dgrad");
      g_launches += g.s == 2 && g.k == 3 ? 4 : 1;
      r[0] = dskip.defined() && !fits ? dx + dskip : dx;
    }
    if (ctx->needs_input_grad(1)) {
      Tensor target = grad_target(weight, st);
      if (!target.defined()) {
        target = zeroed_f32((int64_t)g.cout * g.k * g.k * g.cin, x, st);
        r[1] = target.view({g.cout, g.k, g.k, g.cin}).permute({0, 3, 1, 2});
      }
      check(tsp_conv_wgrad(ptr(x), ptr(b.dx), target.data_ptr<float>(), g.n, g.h, g.w, g.cin, g.cout, g.k, g.s, word, st),
            "tsp_conv_wgrad");
      g_launches += 1;
      if (r[1].defined() && weight.scalar_type() != at::kFloat) r[1] = r[1].to(weight.scalar_type());
    }
    return r;
  }
};

// relu(bn(x) + residual) over rows with channels innermost.
struct BnAct : Function<BnAct> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& bn_w, const Tensor& bn_b,
                        const std::optional<Tensor>& res, const Tensor& acc_sum, const Tensor& acc_sumsq, const Tensor& acc_count, int64_t acc_stride, double eps,
                        bool relu, int64_t segs) {
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t st = stream_of(x);
    const auto [m, c] = rows_of(x);
    const Tensor out = at::empty_like(x), sums = at::empty({segs * 4 * c}, f32_like(x));
    float* s = sums.data_ptr<float>();
    check(tsp_bn_stats(ptr(x), m, (int)c, dtype_code(x), s, (int)segs, st), "tsp_bn_stats");
    g_launches += 2;
    const Accumulators acc = {acc_sum.data_ptr<float>(), acc_sumsq.data_ptr<float>(), acc_count.data_ptr<float>(), acc_stride};
    const bool has_res = res.has_value();
    bn_apply(x, res.value_or(Tensor()), out, s, bn_w, bn_b, acc, m, (int)c, eps, relu, (int)segs, st);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x, bn_w, bn_b, sums, relu && has_res ? out : Tensor()});
    ctx->saved_data["o"] = std::vector<int64_t>{segs, relu, has_res};
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list r(11);
    if (!grads[0].defined()) return r;
    const auto o = ctx->saved_data["o"].toIntVector();
    const auto saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];
    const at::NoGradGuard no_grad;
    const c10::cuda::CUDAGuard guard(x.device());
    const auto [m, c] = rows_of(x);
    const BnGrads b = bn_backward(gradient_like(grads[0], x), x, saved[4], saved[3].data_ptr<float>() + o[0] * 2 * c, saved[1],
                                  saved[2], o[1] != 0, o[2] != 0, ctx->needs_input_grad(1) && ctx->needs_input_grad(2), m, (int)c,
                                  (int)o[0], stream_of(x));
    r[0] = b.dx;
    if (ctx->needs_input_grad(1)) r[1] = b.dw;
    if (ctx->needs_input_grad(2)) r[2] = b.db;
    r[3] = b.dres;
    return r;
  }
};

// x W^T + b on the CTA-pair products.
struct LinearBias : Function<LinearBias> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& w16,
                        const std::optional<Tensor>& bias, const Tensor& status) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t n = weight.size(0), k = weight.size(1);
    Tensor x2 = x.reshape({-1, k});
    if (x2.scalar_type() != at::kBFloat16 || !x2.is_contiguous()) x2 = x2.to(at::kBFloat16).contiguous();
    const int64_t m = x2.size(0);
    auto shape = x.sizes().vec();
    shape.back() = n;
    const Tensor y = at::empty(shape, x2.options());
    check(tsp_gemm_bf16_tn_2cta(ptr(x2), ptr(w16), ptr(y), bias.has_value() ? fptr(*bias) : nullptr, (int)m, (int)n, (int)k, (int)k,
                                (int)k, (int)n, TSP_DTYPE_BF16, bias.has_value() ? 1 : 0, status.data_ptr<int>(), stream_of(x)),
          "tsp_gemm_bf16_tn");
    g_launches += 1;
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x2, weight});
    if (bias.has_value()) ctx->saved_data["bias"] = *bias;
    ctx->saved_data["w16"] = w16;
    ctx->saved_data["status"] = status;
    ctx->saved_data["s"] = x.sizes().vec();
    ctx->saved_data["o"] = std::vector<int64_t>{bias.has_value(), (int64_t)x.scalar_type()};
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list r(5);
    if (!grads[0].defined()) return r;
    const auto o = ctx->saved_data["o"].toIntVector();
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &weight = saved[1], w16 = ctx->saved_data["w16"].toTensor();
    int* word = ctx->saved_data["status"].toTensor().data_ptr<int>();
    const at::NoGradGuard no_grad;
    const c10::cuda::CUDAGuard guard(x2.device());
    const cudaStream_t st = stream_of(x2);
    const int64_t m = x2.size(0), n = weight.size(0), k = weight.size(1);
    Tensor dy = grads[0].reshape({-1, n});
    if (dy.scalar_type() != at::kBFloat16 || !dy.is_contiguous()) dy = dy.to(at::kBFloat16).contiguous();
    if (!aligned(dy)) dy = dy.clone();
    const void* src[1] = {ptr(dy)};
    if (ctx->needs_input_grad(0)) {
      Tensor dx = at::empty(ctx->saved_data["s"].toIntVector(), x2.options());
      check(tsp_gemm_bf16_nn_2cta(src, 1, ptr(w16), ptr(dx), (int)m, (int)k, (int)n, (int)n, (int)k, (int)k, word, st),
            "tsp_gemm_bf16_nn_2cta");
      g_launches += 1;
      const auto want = (at::ScalarType)o[1];
      r[0] = want == at::kBFloat16 ? dx : dx.to(want);
    }
    if (ctx->needs_input_grad(1)) {
      Tensor target = grad_target(weight, st);
      if (!target.defined()) {
        target = zeroed_f32(n * k, x2, st).view({n, k});
        r[1] = target;
      }
      check(tsp_gemm_bf16_wgrad_2cta(src, 1, ptr(x2), target.data_ptr<float>(), (int)n, (int)k, (int)m, (int)n, (int)k, (int)k,
                                     word, st),
            "tsp_gemm_bf16_wgrad_2cta");
      g_launches += 1;
      if (r[1].defined() && weight.scalar_type() != at::kFloat) r[1] = r[1].to(weight.scalar_type());
    }
    if (o[0] != 0 && ctx->needs_input_grad(3)) {
      if (n % 8 != 0 || n > 8192 || m < 2) {
        r[3] = dy.sum(0, false, at::kFloat);
      } else {
        const Tensor add = accumulated(ctx->saved_data["bias"].toTensor(), st);
        if (add.defined()) torch::autograd::impl::bump_version(add);
        const Tensor out = add.defined() ? add : at::empty({n}, f32_like(x2));
        check(tsp_col_sums(ptr(dy), m, (int)n, TSP_DTYPE_BF16, out.data_ptr<float>(), add.defined() ? 1 : 0, st), "tsp_col_sums");
        g_launches += 1;
        if (!add.defined()) r[3] = out;
      }
    }
    return r;
  }
};

// g * gout for a gradient that the forward has computed and saved, and the loss's gradient (a scalar): `fused.py: _scaled`.
Tensor scaled(const Tensor& g, const Tensor& gout, bool own) {
  if (at::GradMode::is_enabled() || !plain(gout) || !plain(g) || gout.scalar_type() != at::kFloat || gout.dim() != 0 ||
      gout.get_device() != g.get_device() || !g.is_contiguous() || !aligned(g))
    return g * gout.to(g.scalar_type());
  const c10::cuda::CUDAGuard guard(g.device());
  const cudaStream_t st = stream_of(g);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  check((int)cudaStreamIsCapturing(st, &capture), "cudaStreamIsCapturing");
  own = own && !torch::autograd::get_current_graph_task_keep_graph() && capture == cudaStreamCaptureStatusNone;
  const Tensor out = own ? g : at::empty_like(g);
  check(tsp_scale(ptr(g), fptr(gout), ptr(out), g.numel(), dtype_code(g), st), "tsp_scale");
  g_launches += 1;
  return out;
}

// Both directions of a symmetric loss: forward leaves the loss and [2][n][d] gradients of the two students.
variable_list pair_backward(AutogradContext* ctx, const variable_list& grads, int args) {
  variable_list r(args);
  if (!grads[0].defined()) return r;
  const Tensor g = scaled(ctx->get_saved_variables()[0], grads[0], ctx->saved_data["own"].toBool());
  if (ctx->needs_input_grad(0)) r[0] = g.select(0, 0);
  if (ctx->needs_input_grad(1)) r[1] = g.select(0, 1);
  return r;
}

struct ByolPair : Function<ByolPair> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x1, const Tensor& x2, const Tensor& y1, const Tensor& y2,
                        double scale) {
    const c10::cuda::CUDAGuard guard(x1.device());
    const int64_t n = x1.size(0), d = x1.size(1);
    const Tensor loss = at::empty({}, f32_like(x1)), total = at::empty({2}, x1.options().dtype(at::kDouble)),
                 gx = at::empty({2, n, d}, x1.options());
    check(tsp_byol_loss_pair(ptr(x1), ptr(y1), ptr(x2), ptr(y2), (int)n, (int)d, dtype_code(x1), (float)scale,
                             total.data_ptr<double>(), loss.data_ptr<float>(), ptr(gx), stream_of(x1)),
          "tsp_byol_loss_pair");
    g_launches += 1;
    ctx->save_for_backward({gx});
    ctx->saved_data["own"] = owns_saved();
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) { return pair_backward(ctx, grads, 5); }
};

struct NcePair : Function<NcePair> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q1, const Tensor& q2, const Tensor& k1, const Tensor& k2,
                        double temp, int64_t chunk, int64_t chunks, const Tensor& status) {
    const c10::cuda::CUDAGuard guard(q1.device());
    const int64_t n = q1.size(0), d = q1.size(1);
    // unit rows of the queries and the keys, the chunks' sums of keys, their log-sum-exps and the loss's 64-bit sum
    const int64_t q_bytes = 2 * n * d * 2, k_bytes = 2 * chunks * chunk * d * 2, o_bytes = 2 * chunks * n * d * 4,
                  l_bytes = (2 * chunks * n + 4) * 4;
    auto up = [](int64_t b) { return (b + 255) / 256 * 256; };
    const Tensor scratch = at::empty({up(q_bytes) + up(k_bytes) + up(o_bytes) + l_bytes}, q1.options().dtype(at::kByte));
    uint8_t* q16 = scratch.data_ptr<uint8_t>();
    uint8_t *k16 = q16 + up(q_bytes), *o = k16 + up(k_bytes), *lse = o + up(o_bytes);
    const Tensor loss = at::empty({}, f32_like(q1)), gq = at::empty({2, n, d}, q1.options());
    check(tsp_nce_pair(ptr(q1), ptr(k1), ptr(q2), ptr(k2), (int)n, dtype_code(q1), (int)chunk, (int)chunks, (float)temp, q16, k16,
                       (float*)o, (float*)lse, loss.data_ptr<float>(), ptr(gq), status.data_ptr<int>(), stream_of(q1)),
          "tsp_nce_pair");
    g_launches += 3;
    ctx->save_for_backward({gq});
    ctx->saved_data["own"] = owns_saved();
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) { return pair_backward(ctx, grads, 8); }
};

// What every function here takes: parameters in fp32 as the kernels read them.
bool vector_f32(const Tensor& t) { return plain(t) && t.scalar_type() == at::kFloat && t.is_contiguous() && aligned(t); }
bool row_matrix(const Tensor& t, const Tensor& like) {
  return plain(t) && t.scalar_type() == like.scalar_type() && t.sizes() == like.sizes() && rows_of(t).first > 0 && aligned(t) &&
         t.get_device() == like.get_device();
}

// None where the call is not one for these functions.
std::optional<variable_list> conv_bn_act(const Tensor& x, const Tensor& weight, const Tensor& w16, const Tensor& bn_w,
                                         const Tensor& bn_b, const std::optional<Tensor>& residual, const Tensor& acc_sum,
                                         const Tensor& acc_sumsq, const Tensor& acc_count, int64_t acc_stride, double eps,
                                         bool relu, int64_t stride, int64_t segs, bool stats, bool fork, const Tensor& status) {
  if (!plain(x) || !plain(weight) || !vector_f32(bn_w) || !vector_f32(bn_b)) return std::nullopt;
  const ConvGeom g(x, weight, stride);
  if (residual.has_value() && !(plain(*residual) && residual->scalar_type() == at::kBFloat16 && nhwc(*residual) &&
                                residual->size(0) == g.n && residual->size(1) == g.cout && residual->size(2) == g.ho &&
                                residual->size(3) == g.wo && aligned(*residual) && residual->get_device() == x.get_device()))
    return std::nullopt;
  return ConvBnAct::apply(x, weight, w16, bn_w, bn_b, residual, acc_sum, acc_sumsq, acc_count, acc_stride, eps,
                          relu, stride, segs, stats, fork, status);
}

std::optional<Tensor> bn_act(const Tensor& x, const Tensor& bn_w, const Tensor& bn_b, const std::optional<Tensor>& residual,
                             const Tensor& acc_sum, const Tensor& acc_sumsq, const Tensor& acc_count, int64_t acc_stride,
                             double eps, bool relu, int64_t segs) {
  if (!plain(x) || rows_of(x).first == 0 || !aligned(x) || !vector_f32(bn_w) || !vector_f32(bn_b) ||
      (residual.has_value() && !row_matrix(*residual, x)))
    return std::nullopt;
  return BnAct::apply(x, bn_w, bn_b, residual, acc_sum, acc_sumsq, acc_count, acc_stride, eps, relu, segs);
}

std::optional<Tensor> linear(const Tensor& x, const Tensor& weight, const Tensor& w16, const std::optional<Tensor>& bias,
                             const Tensor& status) {
  if (!plain(x) || !plain(weight) || (bias.has_value() && !vector_f32(*bias)) ||
      !(x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kFloat))
    return std::nullopt;
  return LinearBias::apply(x, weight, w16, bias, status);
}

bool pair_ok(const Tensor& a, const Tensor& b, const Tensor& c, const Tensor& d) {
  if (!plain(a) || a.dim() != 2 || a.size(0) == 0 || !(a.scalar_type() == at::kBFloat16 || a.scalar_type() == at::kFloat))
    return false;
  for (const Tensor* t : {&a, &b, &c, &d})
    if (!plain(*t) || t->sizes() != a.sizes() || t->scalar_type() != a.scalar_type() || t->get_device() != a.get_device() ||
        !t->is_contiguous())
      return false;
  return true;
}

std::optional<Tensor> byol_pair(const Tensor& x1, const Tensor& x2, const Tensor& y1, const Tensor& y2) {
  if (!pair_ok(x1, x2, y1, y2)) return std::nullopt;
  return ByolPair::apply(x1, x2, y1.detach(), y2.detach(), 1.0 / (double)x1.size(0));
}

std::optional<Tensor> nce_pair(const Tensor& q1, const Tensor& q2, const Tensor& k1, const Tensor& k2, double temp, int64_t chunk,
                               int64_t chunks, const Tensor& status) {
  if (!pair_ok(q1, q2, k1, k2) || !aligned(q1) || !aligned(q2) || !aligned(k1) || !aligned(k2)) return std::nullopt;
  return NcePair::apply(q1, q2, k1.detach(), k2.detach(), temp, chunk, chunks, status);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  // (other threads run while a launch waits for room in its stream's queue)
  using release = pybind11::call_guard<pybind11::gil_scoped_release>;
  m.def("conv_bn_act", &conv_bn_act, release());
  m.def("bn_act", &bn_act, release());
  m.def("linear", &linear, release());
  m.def("byol_pair", &byol_pair, release());
  m.def("nce_pair", &nce_pair, release());
  m.def("launches", [] { return g_launches.load(); });
  m.def("set_accumulate", [](bool on) { g_accumulate = on; });
}
