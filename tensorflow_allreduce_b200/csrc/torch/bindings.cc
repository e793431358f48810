// Native call paths of the small operations: the parts of the Python front end that stand between a call and its kernel
// launches (tensor checks, output allocation, the autograd node, the GEMMs around a recurrent layer), as one extension
// module over the C ABI of libbcoll (csrc/bcoll.h).
//
// Why: batch norm with the clipped ReLU on [5, 32, 41, 175], forward and backward, was 22 us of kernels behind 155 us of
// interpreter work.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>
#include <map>
#include <mutex>

#include "../bcoll.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

void check(int rc, const char* what) {
  if (rc >= 0) return;
  const char* e = bc_last_error();
  throw std::runtime_error(e && *e ? e : std::string("native call failed: ") + what);
}

float* ptr(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// Something that follows torch's operators does not see the kernels: a trace would hold this call's values as constants,
// forward-mode derivatives would stop here, the batches and gradients of torch.func and tensors without storage have no memory to
// hand to them.
bool traced() { return torch::jit::tracer::isTracing(); }
bool has_tangent(const Tensor& t) { return torch::autograd::isFwGradDefined(t); }
bool plain(const Tensor& t) {
  constexpr c10::DispatchKeySet wrappers({c10::DispatchKey::Batched, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                          c10::DispatchKey::Functionalize, c10::DispatchKey::Python});
  return !traced() && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !t.key_set().has_any(wrappers) && !has_tangent(t);
}

// ---- batch norm + clipped ReLU -----------------------------------------------------------------

std::atomic<long long> g_bn_launches{0};

// Scratch doubles of the kernels (partial sums), then batch mean and reciprocal deviation of every channel.
int64_t bn_doubles(int64_t c) { return 2 * (c + 1024); }

struct BnClip : torch::autograd::Function<BnClip> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& bias, const c10::optional<Tensor>& running_mean,
                        const c10::optional<Tensor>& running_var, const c10::optional<Tensor>& batches, double eps, double momentum, double clip) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t n = x.size(0), c = x.size(1), hw = x.numel() / (n * c);
    Tensor y = at::empty_like(x);
    Tensor work = at::empty({bn_doubles(c) + c}, x.options().dtype(at::kDouble));
    double* acc = work.data_ptr<double>();
    float* stats = reinterpret_cast<float*>(acc + bn_doubles(c));
    check(bc_bn_clip_forward(ptr(x), ptr(y), ptr(weight), ptr(bias), running_mean ? ptr(*running_mean) : nullptr,
                             running_var ? ptr(*running_var) : nullptr,
                             batches ? reinterpret_cast<long long*>(batches->data_ptr<int64_t>()) : nullptr, stats, stats + c, acc, (int)n, (int)c,
                             (int)hw, (float)eps, (float)momentum, (float)clip, stream_of(x)),
          "bc_bn_clip_forward");
    g_bn_launches++;
    ctx->save_for_backward({x, weight, bias, work});
    ctx->saved_data["clip"] = clip;
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &weight = saved[1], &bias = saved[2], &work = saved[3];
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t n = x.size(0), c = x.size(1), hw = x.numel() / (n * c);
    const Tensor dy = grads[0].contiguous();
    Tensor dx = at::empty_like(x), dw = at::empty_like(weight), db = at::empty_like(bias);
    double* acc = work.data_ptr<double>();          // the forward pass's partial sums are not needed any more
    const float* stats = reinterpret_cast<const float*>(acc + bn_doubles(c));
    check(bc_bn_clip_backward(ptr(x), ptr(dy), ptr(weight), ptr(bias), stats, stats + c, ptr(dx), ptr(dw), ptr(db), acc, (int)n, (int)c, (int)hw,
                              (float)ctx->saved_data["clip"].toDouble(), stream_of(x)),
          "bc_bn_clip_backward");
    g_bn_launches++;
    return {dx, dw, db, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor bn_clip(const Tensor& x, const Tensor& weight, const Tensor& bias, const c10::optional<Tensor>& running_mean,
               const c10::optional<Tensor>& running_var, const c10::optional<Tensor>& batches, double eps, double momentum, double clip) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && x.scalar_type() == at::kFloat && x.dim() >= 2 && x.numel() > 0,
              "bn_clip needs a contiguous fp32 CUDA tensor");
  // The kernels take the channels' values, and update the counter of batches, where they lie: in memory of this device.
  auto fits = [&](const c10::optional<Tensor>& t) {
    return !t || (t->device() == x.device() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == x.size(1));
  };
  if (traced() || !fits(weight) || !fits(bias) || !fits(running_mean) || !fits(running_var)) {
    if (batches) Tensor(*batches).add_(1);
    return at::hardtanh(at::batch_norm(x, weight, bias, running_mean, running_var, true, momentum, eps, at::globalContext().userEnabledCuDNN()), 0.0, clip);
  }
  if (batches && (batches->device() != x.device() || batches->scalar_type() != at::kLong)) {
    Tensor(*batches).add_(1);
    return BnClip::apply(x, weight, bias, running_mean, running_var, c10::nullopt, eps, momentum, clip);
  }
  return BnClip::apply(x, weight, bias, running_mean, running_var, batches, eps, momentum, clip);
}

// ---- persistent GRU layers ---------------------------------------------------------------------

std::atomic<long long> g_gru_launches{0};
double g_gru_timeout_s = 10.0;
std::mutex g_gru_mu;
std::map<int, Tensor> g_gru_status;                              // per device: the kernels' status word
std::map<std::pair<int, void*>, Tensor> g_gru_scratch;           // per device and stream

bool capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  C10_CUDA_CHECK(cudaStreamIsCapturing(stream, &status));
  return status != cudaStreamCaptureStatusNone;
}

// Made by the first call on the device. If that is a captured one the word is made outside the capture, for good: memory of the graph
// would be cleared by every replay, and hold anything before the first.
int* gru_status(const Tensor& like) {
  std::lock_guard<std::mutex> g(g_gru_mu);
  Tensor& t = g_gru_status[like.device().index()];
  if (!t.defined()) {
    const auto options = like.options().dtype(at::kInt);
    if (capturing((cudaStream_t)stream_of(like))) {
      const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
      void* word = nullptr;
      cudaStream_t aside = nullptr;
      C10_CUDA_CHECK(cudaMalloc(&word, sizeof(int)));
      C10_CUDA_CHECK(cudaStreamCreateWithFlags(&aside, cudaStreamNonBlocking));
      C10_CUDA_CHECK(cudaMemsetAsync(word, 0, sizeof(int), aside));
      C10_CUDA_CHECK(cudaStreamSynchronize(aside));
      C10_CUDA_CHECK(cudaStreamDestroy(aside));
      t = at::from_blob(word, {1}, options);
    } else {
      t = at::zeros({1}, options);
    }
  }
  return t.data_ptr<int>();
}

// Memory through which the blocks of a launch exchange operands and partial sums. Every word says which step it belongs to
// and a launch clears its part first, so the contents only have to be zero once. Kernels on one stream use it one after the
// other: one buffer per device and stream, for the 16 streams that came last. The caller holds it until its launch is queued: another
// thread's call on the stream may want a larger one in the meantime. A captured launch has its own, cleared by the graph: two graphs may
// run at a time, on any streams, and the second before the first.
constexpr size_t kScratchStreams = 16;
Tensor gru_scratch(const Tensor& like, void* stream, int64_t T, int64_t B, int64_t H, int64_t nd) {
  const int64_t need = bc_gru_scratch_bytes((int)T, (int)B, (int)H, (int)nd);
  auto make = [&] { return at::zeros({need}, like.options().dtype(at::kByte)); };
  if (capturing((cudaStream_t)stream)) return make();
  std::lock_guard<std::mutex> g(g_gru_mu);
  const std::pair<int, void*> key{like.device().index(), stream};
  if (g_gru_scratch.size() >= kScratchStreams && !g_gru_scratch.count(key)) g_gru_scratch.clear();
  Tensor& t = g_gru_scratch[key];
  if (!t.defined() || t.numel() < need) t = make();
  return t;
}

Tensor aligned(const Tensor& t, uintptr_t bytes = 16) {
  Tensor c = t.contiguous();
  return (reinterpret_cast<uintptr_t>(c.data_ptr()) & (bytes - 1)) == 0 ? c : c.clone();
}

// One layer: output, and what its backward pass needs (x, all input weights, y, factors of dh, recurrent weights).
// `w` holds w_ih, w_hh, b_ih, b_hh of every direction.
Tensor gru_run(const Tensor& x, at::TensorList w, bool save, variable_list* keep) {
  const int64_t T = x.size(0), B = x.size(1), I = x.size(2), nd = (int64_t)w.size() / 4, H = w[1].size(1);
  const Tensor w_ih = nd > 1 ? at::cat({w[0], w[4]}) : w[0], b_ih = nd > 1 ? at::cat({w[2], w[6]}) : w[2];
  Tensor w_hh[2], b_hh[2];
  for (int64_t d = 0; d < nd; d++) {
    w_hh[d] = aligned(w[4 * d + 1]);
    b_hh[d] = w[4 * d + 3].contiguous();
  }
  // input projections of both directions in one GEMM: [T*B, nd*3H]
  const Tensor gx = at::addmm(b_ih, x.reshape({T * B, I}), w_ih.t());
  Tensor y = at::empty({T, B, nd * H}, x.options());
  Tensor fac;
  if (save) fac = at::empty({nd, T, B, 5, H}, x.options());
  void* s = stream_of(x);
  const Tensor scratch = gru_scratch(x, s, T, B, H, nd);
  check(bc_gru_forward_factors((int)T, (int)B, (int)H, (int)nd, ptr(w_hh[0]), ptr(w_hh[nd - 1]), ptr(b_hh[0]), ptr(b_hh[nd - 1]), ptr(gx), ptr(y),
                               ptr(fac), scratch.data_ptr(), (unsigned*)gru_status(x), g_gru_timeout_s, s),
        "bc_gru_forward_factors");
  g_gru_launches++;
  if (save) {
    *keep = {x, w_ih, y, fac, w_hh[0]};
    if (nd > 1) keep->push_back(w_hh[1]);
  }
  return y;
}

struct GruLayer : torch::autograd::Function<GruLayer> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, at::TensorList w) {
    const c10::cuda::CUDAGuard guard(x.device());
    variable_list keep;
    Tensor y = gru_run(x, w, true, &keep);
    ctx->save_for_backward(keep);
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w_ih = saved[1], &y = saved[2];
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t nd = (int64_t)saved.size() - 4, T = x.size(0), B = x.size(1), I = x.size(2), H = saved[4].size(1), H3 = 3 * H;
    const Tensor dy = grads[0].contiguous(), fac = aligned(saved[3], 32);      // hooks of saved tensors may return views
    // gradients of the pre-activations: (dr, dz, dn) of every direction, then dn * r of every direction
    Tensor dg = at::empty({T * B, nd * 4 * H}, x.options()), db = at::empty({nd, 2, H3}, x.options());
    void* s = stream_of(x);
    const Tensor scratch = gru_scratch(x, s, T, B, H, nd);
    check(bc_gru_backward_factors((int)T, (int)B, (int)H, (int)nd, ptr(saved[4]), ptr(saved[3 + nd]), ptr(fac), ptr(dy), ptr(dg), ptr(db),
                                  scratch.data_ptr(), (unsigned*)gru_status(x), g_gru_timeout_s, s),
          "bc_gru_backward_factors");
    g_gru_launches++;
    const Tensor dgx = dg.narrow(1, 0, nd * H3);
    variable_list out(1 + 4 * nd);
    if (ctx->needs_input_grad(0)) out[0] = at::mm(dgx, w_ih).view({T, B, I});
    bool any_ih = false;
    for (int64_t d = 0; d < nd; d++) any_ih = any_ih || ctx->needs_input_grad(1 + 4 * d);
    Tensor dw_ih;
    if (any_ih) dw_ih = at::mm(dgx.t(), x.reshape({T * B, I}));
    for (int64_t d = 0; d < nd; d++) {
      if (ctx->needs_input_grad(1 + 4 * d)) out[1 + 4 * d] = nd > 1 ? dw_ih.narrow(0, d * H3, H3) : dw_ih;
      if (ctx->needs_input_grad(2 + 4 * d)) {
        Tensor dw = at::empty({H3, H}, x.options());
        if (T > 1) {
          // direction 0: h_{t-1} = y[t-1]; direction 1 runs backwards in time: h_prev = y[t+1]
          const int64_t rows = (T - 1) * B;
          const Tensor g = dg.narrow(0, d == 0 ? B : 0, rows);
          const Tensor h = y.view({T * B, nd * H}).narrow(0, d == 0 ? 0 : B, rows).narrow(1, d * H, H);
          Tensor upper = dw.narrow(0, 0, 2 * H), lower = dw.narrow(0, 2 * H, H);
          at::mm_out(upper, g.narrow(1, d * H3, 2 * H).t(), h);
          at::mm_out(lower, g.narrow(1, nd * H3 + d * H, H).t(), h);
        } else {
          dw.zero_();
        }
        out[2 + 4 * d] = dw;
      }
      if (ctx->needs_input_grad(3 + 4 * d)) out[3 + 4 * d] = db.select(0, d).select(0, 0);
      if (ctx->needs_input_grad(4 + 4 * d)) out[4 + 4 * d] = db.select(0, d).select(0, 1);
    }
    return out;
  }
};

// A stack of layers; `weights` holds w_ih, w_hh, b_ih, b_hh of every layer and direction.
Tensor gru_stack(Tensor x, const std::vector<Tensor>& weights, int64_t layers) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 3, "the persistent GRU kernels take fp32 CUDA tensors [T, B, features]");
  const size_t per = weights.size() / layers;
  x = x.contiguous();
  for (int64_t l = 0; l < layers; l++) {
    const at::TensorList w(weights.data() + l * per, per);
    bool grad = at::GradMode::is_enabled() && x.requires_grad();
    bool tangent = has_tangent(x);
    for (const Tensor& t : w) {
      grad = grad || (at::GradMode::is_enabled() && t.requires_grad());
      tangent = tangent || has_tangent(t);
    }
    TORCH_CHECK(!tangent, "the persistent GRU kernels have no forward-mode derivative");
    if (grad) {
      x = GruLayer::apply(x, w);
    } else {
      const c10::cuda::CUDAGuard guard(x.device());
      x = gru_run(x, w, false, nullptr);
    }
  }
  return x;
}

// Status of the kernels on `device` since the last call, on all of its streams (waits for the device); 0 = fine.
int gru_take_status(int device) {
  std::lock_guard<std::mutex> g(g_gru_mu);
  auto it = g_gru_status.find(device);
  if (it == g_gru_status.end()) return 0;
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  c10::cuda::device_synchronize();
  const int code = it->second.item<int>();
  if (code) {                     // what a launch that gave up has left in the exchange memory is not used again
    it->second.zero_();
    for (auto s = g_gru_scratch.begin(); s != g_gru_scratch.end();) s = s->first.first == device ? g_gru_scratch.erase(s) : std::next(s);
    c10::cuda::device_synchronize();
  }
  return code;
}

std::vector<int> gru_devices() {
  std::lock_guard<std::mutex> g(g_gru_mu);
  std::vector<int> out;
  for (auto& kv : g_gru_status) out.push_back(kv.first);
  return out;
}

// ---- row convolutions ---------------------------------------------------------------------------

std::atomic<long long> g_conv_launches{0};

struct Conv {
  int v[9];
  Conv(const Tensor& x, const Tensor& w, int64_t ph, int64_t pw)
      : v{(int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), (int)w.size(2), (int)w.size(3), (int)ph, (int)pw, x.size(1) == 1 ? 2 : 1} {}
  int64_t Ho() const { return (v[2] + 2 * v[6] - v[4]) / 2 + 1; }
  int64_t Wo() const { return (v[3] + 2 * v[7] - v[5]) / v[8] + 1; }
  Tensor scratch(const Tensor& like) const { return at::empty({(int64_t)bc_conv_scratch_bytes(v)}, like.options().dtype(at::kByte)); }
};

struct ConvRows : torch::autograd::Function<ConvRows> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, int64_t ph, int64_t pw) {
    const c10::cuda::CUDAGuard guard(x.device());
    const Conv c(x, w, ph, pw);
    const Tensor wc = w.contiguous(), scratch = c.scratch(x);
    Tensor y = at::empty({x.size(0), 32, c.Ho(), c.Wo()}, x.options());
    check(bc_conv_forward(c.v, ptr(x), ptr(wc), ptr(y), scratch.data_ptr(), (unsigned*)gru_status(x), g_gru_timeout_s, stream_of(x)), "bc_conv_forward");
    g_conv_launches++;
    ctx->save_for_backward({x, w});
    ctx->saved_data["ph"] = ph;
    ctx->saved_data["pw"] = pw;
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t ph = ctx->saved_data["ph"].toInt(), pw = ctx->saved_data["pw"].toInt();
    const Conv c(x, saved[1], ph, pw);
    auto by_torch = [&](bool need_x, bool need_w) {
      return at::convolution_backward(grads[0], x, saved[1], c10::nullopt, {2, c.v[8]}, {ph, pw}, {1, 1}, false, {0, 0}, 1, {need_x, need_w, false});
    };
    if (at::GradMode::is_enabled() || !plain(grads[0])) {      // the gradients are to be differentiated again, or are many
      const auto d = by_torch(ctx->needs_input_grad(0), ctx->needs_input_grad(1));
      return {std::get<0>(d), std::get<1>(d), Tensor(), Tensor()};
    }
    const Tensor w = saved[1].contiguous(), dy = grads[0].contiguous(), scratch = c.scratch(x);
    unsigned* status = (unsigned*)gru_status(x);
    Tensor dx, dw;
    if (ctx->needs_input_grad(1)) {
      dw = at::empty_like(w);
      check(bc_conv_backward_weight(c.v, ptr(x), ptr(dy), ptr(dw), scratch.data_ptr(), status, g_gru_timeout_s, stream_of(x)), "bc_conv_backward_weight");
      g_conv_launches++;
    }
    if (ctx->needs_input_grad(0)) {
      if (x.size(1) == 32) {
        dx = at::empty_like(x);
        check(bc_conv_backward_input(c.v, ptr(dy), ptr(w), ptr(dx), scratch.data_ptr(), status, g_gru_timeout_s, stream_of(x)), "bc_conv_backward_input");
        g_conv_launches++;
      } else {       // the spectrogram's gradient is not part of training
        dx = std::get<0>(by_torch(true, false));
      }
    }
    return {dx, dw, Tensor(), Tensor()};
  }
};

// The operands are TF32: not where fp32 convolutions are asked for, by the flag of all of cuDNN or by that of its convolutions, and not
// where cuDNN is off, since torch's own convolutions are fp32.
bool tf32_allowed() { return at::globalContext().userEnabledCuDNN() && at::globalContext().allowTF32CuDNN(at::Float32Op::CONV); }

bool conv_supported(const Tensor& x, const Tensor& w, int64_t ph, int64_t pw) {
  if (!x.is_cuda() || !w.is_cuda() || x.scalar_type() != at::kFloat || w.scalar_type() != at::kFloat || x.dim() != 4 || w.dim() != 4 ||
      !x.is_contiguous() || w.size(0) != 32 || w.size(1) != x.size(1) || x.size(0) > 65535 || !tf32_allowed() || !plain(x) || !plain(w))
    return false;
  const Conv c(x, w, ph, pw);
  return bc_conv_supported(x.device().index(), c.v) == 1;
}

Tensor conv_rows(const Tensor& x, const Tensor& w, int64_t ph, int64_t pw) {
  TORCH_CHECK(conv_supported(x, w, ph, pw), "conv_rows does not cover this convolution");
  return ConvRows::apply(x, w, ph, pw);
}

// ---- CTC loss -----------------------------------------------------------------------------------

std::atomic<long long> g_ctc_launches{0};

const long long* longs(const Tensor& t) { return reinterpret_cast<const long long*>(t.data_ptr<int64_t>()); }

struct CtcMean : torch::autograd::Function<CtcMean> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logp, const Tensor& labels, const Tensor& lens) {
    const c10::cuda::CUDAGuard guard(logp.device());
    const int64_t t = logp.size(0), b = logp.size(1), c = logp.size(2), l = labels.size(1), chains = 2 * b * t * (2 * l + 1);
    Tensor work = at::empty({chains + b}, logp.options()), loss = at::empty({}, logp.options());
    check(bc_ctc_forward(ptr(logp), longs(labels), l, longs(lens), ptr(work), ptr(work) + chains, ptr(loss), (int)t, (int)b, (int)c, (int)l,
                         stream_of(logp)),
          "bc_ctc_forward");
    g_ctc_launches++;
    ctx->save_for_backward({logp, labels, lens, work});
    return loss;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &logp = saved[0], &labels = saved[1], &lens = saved[2], &work = saved[3];
    const c10::cuda::CUDAGuard guard(logp.device());
    const int64_t t = logp.size(0), b = logp.size(1), c = logp.size(2), l = labels.size(1), chains = 2 * b * t * (2 * l + 1);
    const bool one = plain(grads[0]);          // else a batch of them
    const Tensor dloss = one ? grads[0].contiguous() : at::ones({}, logp.options());
    Tensor dlogp = at::empty_like(logp);
    check(bc_ctc_backward(ptr(logp), longs(labels), l, longs(lens), ptr(work), ptr(work) + chains, ptr(dloss), ptr(dlogp), (int)t, (int)b, (int)c,
                          (int)l, stream_of(logp)),
          "bc_ctc_backward");
    g_ctc_launches++;
    if (at::GradMode::is_enabled())        // there is no second derivative, in torch's loss either: asking for it is an error
      torch::autograd::set_history(dlogp, std::make_shared<torch::autograd::Error>("the CTC loss cannot be differentiated twice",
                                                                                  torch::autograd::collect_next_edges(logp, grads[0])));
    return {one ? dlogp : dlogp * grads[0], Tensor(), Tensor()};
  }
};

Tensor ctc_mean(const Tensor& logp, const Tensor& labels, const Tensor& lens) {
  TORCH_CHECK(logp.is_cuda() && logp.scalar_type() == at::kFloat && logp.dim() == 3 && logp.numel() > 0 && labels.device() == logp.device() &&
                  labels.scalar_type() == at::kLong && labels.dim() == 2 && labels.size(0) == logp.size(1) && lens.device() == logp.device() &&
                  lens.scalar_type() == at::kLong && lens.dim() == 1 && lens.size(0) == logp.size(1),
              "ctc_mean takes fp32 CUDA log-probabilities [T, B, C], labels [B, L] and lengths [B] on the same device");
  return CtcMean::apply(logp.contiguous(), labels.contiguous(), lens.contiguous());
}

// ---- activations of a convolution, time first ---------------------------------------------------

// [B, ..., T] -> [T, B, features] of contiguous fp32 activations.
struct TimeMajor : torch::autograd::Function<TimeMajor> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t b = x.size(0), t = x.size(-1), k = x.numel() / (b * t);
    ctx->saved_data["shape"] = x.sizes().vec();
    Tensor y = at::empty({t, b, k}, x.options());
    check(bc_transpose(ptr(x), ptr(y), (int)b, (int)k, (int)t, t, k * t, b * k, k, stream_of(x)), "bc_transpose");
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (at::GradMode::is_enabled() || !plain(grads[0]))        // the gradient is to be differentiated again, or is many
      return {grads[0].permute({1, 2, 0}).reshape(ctx->saved_data["shape"].toIntVector())};
    const Tensor dy = grads[0].contiguous();
    const c10::cuda::CUDAGuard guard(dy.device());
    const int64_t t = dy.size(0), b = dy.size(1), k = dy.size(2);
    Tensor dx = at::empty(ctx->saved_data["shape"].toIntVector(), dy.options());
    check(bc_transpose(ptr(dy), ptr(dx), (int)b, (int)t, (int)k, b * k, k, t, k * t, stream_of(dy)), "bc_transpose");
    return {dx};
  }
};

Tensor time_major(const Tensor& x) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && x.scalar_type() == at::kFloat && x.dim() >= 2 && x.numel() > 0 && x.size(0) <= 65535,
              "time_major takes contiguous fp32 CUDA activations");
  if (!plain(x)) return (x.dim() == 2 ? x.unsqueeze(1) : x.flatten(1, -2)).permute({2, 0, 1}).contiguous();
  return TimeMajor::apply(x);
}

// ---- collectives of a group of one --------------------------------------------------------------

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return 0;
    case at::kInt: return 1;
    case at::kLong: return 2;
    case at::kBFloat16: return 3;
    case at::kHalf: return 4;
    case at::kDouble: return 5;
    case at::kByte: return 6;
    default: return -1;
  }
}

// The reduction of a GPU tensor over a group of one rank, on the caller's stream; none if the call has to be negotiated.
c10::optional<Tensor> allreduce_alone(const std::string& name, const Tensor& tensor, bool average, int red) {
  const int dt = dtype_code(tensor.scalar_type());
  if (dt < 0 || !tensor.is_cuda() || tensor.layout() != at::kStrided) return c10::nullopt;
  const c10::cuda::CUDAGuard guard(tensor.device());
  at::NoGradGuard no_grad;
  const Tensor t = tensor.detach().contiguous();
  Tensor out = at::empty_like(t);
  const int rc = bc_allreduce_alone(name.c_str(), t.data_ptr(), out.data_ptr(), dt, t.numel(), t.device().index(), average, red, stream_of(t));
  check(rc, "allreduce");
  if (rc == 0) return c10::nullopt;
  return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("plain", &plain);
  m.def("bn_clip", &bn_clip);
  m.def("bn_launches", [] { return g_bn_launches.load(); });
  m.def("gru_stack", &gru_stack);
  m.def("gru_launches", [] { return g_gru_launches.load(); });
  m.def("gru_set_timeout", [](double s) { g_gru_timeout_s = s; });
  m.def("gru_take_status", &gru_take_status);
  m.def("gru_devices", &gru_devices);
  m.def("conv_supported", &conv_supported);
  m.def("conv_rows", &conv_rows);
  m.def("conv_launches", [] { return g_conv_launches.load(); });
  m.def("ctc_mean", &ctc_mean);
  m.def("ctc_launches", [] { return g_ctc_launches.load(); });
  m.def("time_major", &time_major);
  m.def("allreduce_alone", &allreduce_alone);
}
