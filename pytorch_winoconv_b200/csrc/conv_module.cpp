#include "conv_module.h"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>

#include <algorithm>
#include <cstring>

namespace {

int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return WINOCONV_F32;
    case at::kHalf: return WINOCONV_F16;
    case at::kBFloat16: return WINOCONV_BF16;
    default: return -1;
  }
}
at::ScalarType type_of(int code) { return code == WINOCONV_F32 ? at::kFloat : code == WINOCONV_F16 ? at::kHalf : at::kBFloat16; }

void check_abi(int st, const char *what) {
  if (st == WINOCONV_OK) return;
  char buf[1024];
  winoconv_last_error(buf, sizeof buf);
  TORCH_CHECK(false, what, " failed (", winoconv_status_string(st), "): ", buf);
}
void *stream_of() { return (void *)at::cuda::getCurrentCUDAStream().stream(); }

ConvRunner::Stamp stamp_of(const at::Tensor &w, const std::optional<at::Tensor> &b) {
  ConvRunner::Stamp s;
  s.w_ref = ConvRunner::Stamp::Ref(w.getIntrusivePtr());
  s.w = w.data_ptr();
  s.w_version = (int64_t)w._version();
  s.w_dtype = (int)w.scalar_type();
  if (b) {
    s.b_ref = ConvRunner::Stamp::Ref(b->getIntrusivePtr());
    s.b = b->data_ptr();
    s.b_version = (int64_t)b->_version();
  }
  return s;
}

// Whether an [N, C, spatial...] tensor lies channels last in memory (dimensions of one element may have any stride).
bool lies_channels_last(const at::Tensor &t) {
  const auto sizes = t.sizes(), strides = t.strides();
  const int nd = (int)sizes.size();
  int64_t want = 1;
  auto ok = [&](int d) {
    if (sizes[d] != 1 && strides[d] != want) return false;
    want *= sizes[d];
    return true;
  };
  if (!ok(1)) return false;
  for (int d = nd - 1; d >= 2; --d)
    if (!ok(d)) return false;
  return ok(0);
}

at::Tensor empty_bytes(uint64_t bytes, const at::Tensor &like) {
  return at::empty({(int64_t)bytes}, like.options().dtype(at::kByte).requires_grad(false));
}

// An [N, C, spatial...] tensor in torch's contiguous order as a channels-last one of another element type.
at::Tensor turned_channels_last(const at::Tensor &t, at::ScalarType type, void *stream) {
  const int nd = (int)t.dim() - 2;
  at::Tensor out = at::empty(t.sizes(), t.options().dtype(type).requires_grad(false), nd == 2 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::ChannelsLast3d);
  const int64_t pixels = t.numel() / (t.size(0) * t.size(1));
  const int st = (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) ? WINOCONV_ERR_UNSUPPORTED
                 : winoconv_to_channels_last(t.data_ptr(), code_of(t.scalar_type()), out.data_ptr(), code_of(type), (int)t.size(0), (int)t.size(1), pixels, (int)t.size(1), stream);
  if (st == WINOCONV_ERR_UNSUPPORTED) out.copy_(t);
  else check_abi(st, "winoconv_to_channels_last");
  return out;
}

// The tensor itself where it is of `type` and lies channels last without gaps, else a copy that does.  (Tensor::to would hand a
// crop, a channel slice or the gradient behind a concatenation back as it is: it looks at the order of the strides only.)
at::Tensor dense_channels_last(const at::Tensor &t, at::ScalarType type, void *stream) {
  if (t.scalar_type() == type && lies_channels_last(t)) return t;
  if (t.is_contiguous() && t.size(1) > 1 && code_of(t.scalar_type()) >= 0 && t.size(0) <= 65535) return turned_channels_last(t, type, stream);
  at::Tensor out = at::empty(t.sizes(), t.options().dtype(type).requires_grad(false), t.dim() == 4 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::ChannelsLast3d);
  return out.copy_(t);
}

// The tensor itself where it starts on 16 bytes, as TMA and the C ABI want it; else a copy in the same order.
at::Tensor aligned(const at::Tensor &t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) ? t.clone() : t; }

// The last dimension of a channels-last buffer zero-extended to `c` channels; the tensor itself where it has them.
at::Tensor pad_channels(const at::Tensor &t, int64_t c) {
  const int nd = (int)t.dim();
  if (t.size(1) == c) return t;
  at::Tensor cl = t.movedim(1, nd - 1);
  return at::constant_pad_nd(cl, {0, c - t.size(1)}).contiguous().movedim(nd - 1, 1);
}

// The graph capture the stream takes part in, 0 outside of one.  (The default stream takes part in none, and needs no query.)
unsigned long long capture_of(cudaStream_t stream) {
  if (stream == nullptr) return 0;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  C10_CUDA_CHECK(cudaStreamGetCaptureInfo(stream, &status, &id));
  return status == cudaStreamCaptureStatusNone ? 0 : id;
}

struct ConvFn : public torch::autograd::Function<ConvFn> {
  static at::Tensor forward(torch::autograd::AutogradContext *ctx, const c10::intrusive_ptr<ConvRunner> &runner, const at::Tensor &x,
                            const at::Tensor &x_cl, const std::shared_ptr<ConvRunner::Entry> &entry, const at::Tensor &weight,
                            const std::optional<at::Tensor> &bias, bool relu) {
    at::Tensor y = runner->run(*entry, x_cl, weight, bias, weight.requires_grad());
    ctx->save_for_backward({x, relu ? y : at::Tensor()});
    ctx->saved_data["runner"] = c10::IValue::make_capsule(runner);
    ctx->saved_data["weight"] = weight;
    if (bias) ctx->saved_data["bias"] = *bias;
    return y;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
    torch::autograd::variable_list out(7);
    if (!grads[0].defined()) return out;
    auto saved = ctx->get_saved_variables();
    auto runner = c10::static_intrusive_pointer_cast<ConvRunner>(ctx->saved_data["runner"].toCapsule());
    const at::Tensor weight = ctx->saved_data["weight"].toTensor();
    std::optional<at::Tensor> bias;
    auto b = ctx->saved_data.find("bias");
    if (b != ctx->saved_data.end()) bias = b->second.toTensor();
    // numbered by the tensors among the arguments of apply: x, x_cl, weight, bias
    const bool nx = ctx->needs_input_grad(0), nw = ctx->needs_input_grad(2), nb = bias && ctx->needs_input_grad(3);
    auto g = runner->backward(grads[0], saved[0], saved[1], weight, bias, nx, nw, nb);
    out[1] = g[0];
    out[4] = g[1];
    out[5] = g[2];
    return out;
  }
};

}  // namespace

ConvRunner::ConvRunner(int64_t nd, std::vector<int64_t> stride, std::vector<int64_t> padding, int64_t tile_m, int64_t algo, bool relu,
                       bool pool, int64_t compute, int64_t max_plans)
    : nd_((int)nd), tile_m_((int)tile_m), algo_((int)algo), compute_((int)compute), relu_(relu), pool_(pool), max_plans_((size_t)max_plans) {
  TORCH_CHECK((nd == 2 || nd == 3) && (int64_t)stride.size() == nd && (int64_t)padding.size() == nd, "ConvRunner: bad rank");
  for (int i = 0; i < 3; ++i) { stride_[i] = 1; pad_[i] = 0; }
  for (int i = 0; i < nd; ++i) { stride_[3 - nd + i] = (int)stride[i]; pad_[3 - nd + i] = (int)padding[i]; }
}

std::shared_ptr<ConvRunner::Entry> ConvRunner::entry_for(const at::Tensor &x, const at::Tensor &weight, const std::optional<at::Tensor> &bias,
                                                         int dtype, bool first) {
  int64_t shape[5] = {x.size(0), 1, 1, 1, x.size(1)};
  for (int i = 0; i < nd_; ++i) shape[4 - nd_ + i] = x.size(2 + i);
  int64_t w_shape[4] = {weight.size(0), 1, 1, 1};
  for (int i = 0; i < nd_; ++i) w_shape[4 - nd_ + i] = weight.size(2 + i);
  const int device = x.get_device(), bias_type = bias ? (int)bias->scalar_type() : -1;
  std::lock_guard<std::mutex> lock(mu_);
  for (size_t i = entries_.size(); i-- > 0;) {
    Entry &e = *entries_[i];
    if (e.dtype == dtype && e.device == device && e.bias_type == bias_type && e.first == first && std::memcmp(e.shape, shape, sizeof shape) == 0 &&
        std::memcmp(e.w_shape, w_shape, sizeof w_shape) == 0) {
      auto hit = entries_[i];
      if (i + 1 != entries_.size()) {
        entries_.erase(entries_.begin() + i);
        entries_.push_back(hit);
      }
      return hit;
    }
  }
  auto e = std::make_shared<Entry>();
  std::memcpy(e->shape, shape, sizeof shape);
  std::memcpy(e->w_shape, w_shape, sizeof w_shape);
  e->dtype = dtype;
  e->device = device;
  e->bias_type = bias_type;
  e->first = first;
  winoconv_desc_t &d = e->desc;
  std::memset(&d, 0, sizeof d);
  d.ndim = nd_;
  for (int64_t s : {shape[0], shape[1], shape[2], shape[3], shape[4], w_shape[0], w_shape[1], w_shape[2], w_shape[3]})
    if (s <= 0 || s > 0x7fffffffLL) return nullptr;
  d.batch = (int)shape[0]; d.c_in = (int)shape[4]; d.k_out = (int)w_shape[0];
  for (int i = 0; i < 3; ++i) {
    d.in_size[i] = (int)shape[1 + i];
    d.ker_size[i] = (int)w_shape[1 + i];
    d.stride[i] = stride_[i];
    d.pad[i] = pad_[i];
  }
  d.tile_m = tile_m_;
  d.dtype = dtype;
  d.epilogue = (bias ? WINOCONV_EPI_BIAS : 0u) | (relu_ ? WINOCONV_EPI_RELU : 0u) | (pool_ ? WINOCONV_EPI_POOL2 : 0u);
  d.algo = algo_;
  d.x_channels_first = first ? 2 : 0;
  d.bias_f32 = dtype != WINOCONV_F32 && bias && bias->scalar_type() == at::kFloat;      // read as it is where the kernel can
  if (winoconv_plan(&d, &e->info) != WINOCONV_OK) {
    d.bias_f32 = 0;
    if (winoconv_plan(&d, &e->info) != WINOCONV_OK) return nullptr;
  }
  entries_.push_back(e);
  while (entries_.size() > max_plans_) entries_.erase(entries_.begin());      // each entry holds its own transformed filter
  return e;
}

at::Tensor ConvRunner::run(Entry &e, const at::Tensor &x, const at::Tensor &weight, const std::optional<at::Tensor> &bias, bool learns) {
  const at::ScalarType type = type_of(e.dtype);
  const auto here = at::cuda::getCurrentCUDAStream();
  void *s = (void *)here.stream();
  const Stamp now = stamp_of(weight, bias);
  at::Tensor u, b;
  {
    std::lock_guard<std::mutex> lock(mu_);
    if (!(e.stamp == now) || !e.written.usable_on(here, learns, e.u, e.bias)) {
      at::AutoDispatchBelowADInplaceOrView guard;
      // a new buffer, not the old one, which launches may still be queued to read (the allocator knows on which streams)
      const at::Tensor fresh = empty_bytes(e.info.filter_bytes, weight);
      at::Tensor w = weight.is_contiguous() ? weight : weight.contiguous();
      if (winoconv_filter_transform_from(&e.desc, w.data_ptr(), code_of(w.scalar_type()), fresh.data_ptr(), s) != WINOCONV_OK) {
        w = w.to(type);
        check_abi(winoconv_filter_transform(&e.desc, w.data_ptr(), fresh.data_ptr(), s), "winoconv_filter_transform");
      }
      e.u = fresh;
      e.bias = bias ? bias->detach().to(e.desc.bias_f32 ? at::kFloat : type).contiguous() : at::Tensor();
      e.written.on(here);
      e.stamp = now;
      e.serial = ++serial_;
      newest_ = now;
    }
    u = e.u;
    b = e.bias;
    if (e.written.capture == 0 && capture_of(here) != 0 &&
        std::none_of(in_graphs_.begin(), in_graphs_.end(), [&](const auto &t) { return t.first.is_same(u); }))
      in_graphs_.emplace_back(u, b);
  }
  int64_t sizes[5] = {e.shape[0], (int64_t)e.desc.k_out, 0, 0, 0};
  for (int i = 0; i < nd_; ++i) sizes[2 + i] = e.info.out_size[3 - nd_ + i];
  at::Tensor y = at::empty(at::IntArrayRef(sizes, nd_ + 2), x.options().dtype(type).requires_grad(false),
                           nd_ == 2 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::ChannelsLast3d);
  at::Tensor v, m;
  if (e.info.direct != 1) {
    if (e.info.input_ws_bytes) v = empty_bytes(e.info.input_ws_bytes, x);
    if (!e.info.direct && e.info.product_ws_bytes) m = empty_bytes(e.info.product_ws_bytes, x);
  }
  check_abi(winoconv_forward(&e.desc, x.data_ptr(), u.data_ptr(), b.defined() ? b.data_ptr() : nullptr, y.data_ptr(),
                             v.defined() ? v.data_ptr() : nullptr, e.info.input_ws_bytes, m.defined() ? m.data_ptr() : nullptr,
                             e.info.product_ws_bytes, s),
            "winoconv_forward");
  return y;
}

std::optional<at::Tensor> ConvRunner::forward(const at::Tensor &x, const at::Tensor &weight, const std::optional<at::Tensor> &bias, bool training) {
  if (!x.is_cuda() || x.dim() != nd_ + 2 || weight.dim() != nd_ + 2 || !weight.is_cuda() || weight.get_device() != x.get_device() ||
      x.size(1) != weight.size(1) || x.numel() == 0 || code_of(weight.scalar_type()) < 0 ||
      (bias && (!bias->is_cuda() || bias->get_device() != x.get_device() || bias->numel() != weight.size(0))))
    return std::nullopt;
  if (weight.is_inference() || (bias && bias->is_inference())) return std::nullopt;      // no version to tell a new value by
  const int dtype = compute_ >= 0 ? compute_ : code_of(x.scalar_type());
  if (dtype < 0) return std::nullopt;
  const bool grad = at::GradMode::is_enabled() && (x.requires_grad() || (weight.requires_grad() && training));
  if (grad && (pool_ || dtype == WINOCONV_F32)) return std::nullopt;
  c10::cuda::CUDAGuard guard(x.device());
  std::shared_ptr<Entry> e;
  if (!grad && dtype != WINOCONV_F32 && tile_m_ == 0 && algo_ == WINOCONV_ALGO_AUTO && x.scalar_type() == type_of(dtype) && x.is_contiguous() &&
      x.size(1) * weight.size(-1) <= 64 && x.size(1) > 1 && !lies_channels_last(x) && (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15u) == 0) {
    // few channels in torch's contiguous order: the kernel gathers them as they lie where that beats a copy
    e = entry_for(x, weight, bias, dtype, true);
    if (e) {
      at::AutoDispatchBelowADInplaceOrView no_graph;
      return run(*e, x, weight, bias, false);
    }
  }
  e = entry_for(x, weight, bias, dtype, false);
  if (!e) return std::nullopt;
  if (!grad) {
    at::AutoDispatchBelowADInplaceOrView no_graph;
    return run(*e, dense_channels_last(x, type_of(dtype), stream_of()), weight, bias, false);
  }
  if (!backward_covered(*e)) return std::nullopt;
  at::Tensor x_cl;
  {
    at::AutoDispatchBelowADInplaceOrView no_graph;
    x_cl = dense_channels_last(x, type_of(dtype), stream_of());
    if (x_cl.is_same(x)) x_cl = x.detach();
  }
  return ConvFn::apply(c10::intrusive_ptr<ConvRunner>::reclaim_copy(this), x, x_cl, e, weight, bias, relu_);
}

void ConvRunner::Written::on(const c10::cuda::CUDAStream &here) {
  stream = here;
  capture = capture_of(here);
  recorded = finished = false;
}

bool ConvRunner::Written::usable_on(const c10::cuda::CUDAStream &here, bool learns, const at::Tensor &a, const at::Tensor &b) {
  if (!stream) return false;
  if (capture == 0 && *stream == here && !learns) return true;
  const unsigned long long current = capture_of(here);
  if ((capture != 0 || learns) && capture != current) return false;
  if (*stream == here) return true;
  if (!finished) {
    c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);      // a query is no part of anyone's capture
    if (!recorded && capture_of(*stream) != capture) return false;      // being captured now: it tells nothing of the work before that
    finished = capture == 0 && (recorded ? event.query() : stream->query());
    if (!finished && !recorded) {
      event.record(*stream);
      recorded = true;
    }
  }
  if (!finished) {
    if (capture != current) return false;
    event.block(here);
  }
  for (const at::Tensor *t : {&a, &b})
    if (t->defined()) t->record_stream(here);
  return true;
}

bool ConvRunner::backward_covered(Entry &e) {
  std::lock_guard<std::mutex> lock(mu_);
  if (!e.back_known) {
    winoconv_backward_info_t info;
    bool ok = winoconv_backward_plan(&e.desc, &info) == WINOCONV_OK && info.data_ok && info.weight_ok;
    for (int i = 0; i < 3; ++i) ok = ok && pad_[i] < e.desc.ker_size[i];      // the Python path refuses the data gradient
    e.back_ok = ok;
    e.back_known = true;
  }
  return e.back_ok;
}

std::vector<at::Tensor> ConvRunner::backward(const at::Tensor &gy_in, const at::Tensor &x_in, const at::Tensor &y, const at::Tensor &weight,
                                             const std::optional<at::Tensor> &bias, bool need_x, bool need_w, bool need_b) {
  at::AutoDispatchBelowADInplaceOrView no_graph;
  c10::cuda::CUDAGuard guard(x_in.device());
  const int dtype = compute_ >= 0 ? compute_ : code_of(x_in.scalar_type());
  const at::ScalarType type = type_of(dtype);
  std::shared_ptr<Entry> e = entry_for(x_in, weight, bias, dtype, false);
  TORCH_CHECK(e, "winoconv backward: no plan");
  const auto here = at::cuda::getCurrentCUDAStream();
  void *s = (void *)here.stream();
  at::Tensor gy = gy_in;
  if (y.defined()) gy = gy * (y > 0).to(gy.scalar_type());
  gy = aligned(dense_channels_last(gy, type, s));
  winoconv_desc_t d = e->desc;
  d.epilogue = need_b ? WINOCONV_EPI_BIAS : 0u;
  winoconv_backward_info_t info;
  check_abi(winoconv_backward_plan(&d, &info), "winoconv_backward_plan");
  const at::Tensor gyp = pad_channels(gy, info.k_stride);
  at::Tensor gx, gw, gb;
  const at::Tensor w = weight.is_contiguous() ? weight : weight.contiguous();
  if (need_x) {
    at::Tensor u;
    const Stamp now = stamp_of(weight, std::nullopt);
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (!(e->back_stamp == now) || !e->back_written.usable_on(here, weight.requires_grad(), e->u_back, at::Tensor())) {
        const at::Tensor fresh = empty_bytes(std::max<uint64_t>(info.data_filter_bytes, 16), w);
        at::Tensor wt = w;
        if (code_of(w.scalar_type()) != WINOCONV_F32 && code_of(w.scalar_type()) != dtype) wt = w.to(type);
        check_abi(winoconv_backward_filter_transform(&d, wt.data_ptr(), code_of(wt.scalar_type()), fresh.data_ptr(), s),
                  "winoconv_backward_filter_transform");
        e->u_back = fresh;
        e->back_written.on(here);
        e->back_stamp = now;
      }
      u = e->u_back;
    }
    gx = at::empty(x_in.sizes(), x_in.options().dtype(type).requires_grad(false), nd_ == 2 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::ChannelsLast3d);
    check_abi(winoconv_backward_data(&d, gyp.data_ptr(), u.data_ptr(), gx.data_ptr(), s), "winoconv_backward_data");
    if (x_in.scalar_type() != type) gx = gx.to(x_in.scalar_type());
  }
  if (need_w) {
    const at::Tensor xp = aligned(pad_channels(dense_channels_last(x_in, type, s), info.c_stride));
    gw = at::empty(weight.sizes(), weight.options().requires_grad(false));
    if (need_b) gb = at::empty({weight.size(0)}, weight.options().dtype(at::kFloat).requires_grad(false));
    const at::Tensor ws = empty_bytes(info.weight_ws_bytes, w);
    check_abi(winoconv_backward_weight(&d, xp.data_ptr(), gyp.data_ptr(), gw.data_ptr(), code_of(gw.scalar_type()),
                                       need_b ? gb.data_ptr<float>() : nullptr, ws.data_ptr(), info.weight_ws_bytes, s),
              "winoconv_backward_weight");
  } else if (need_b) {
    std::vector<int64_t> dims{0};
    for (int i = 0; i < nd_; ++i) dims.push_back(2 + i);
    gb = gy.to(at::kFloat).sum(dims);
  }
  if (gb.defined() && gb.scalar_type() != bias->scalar_type()) gb = gb.to(bias->scalar_type());
  return {gx, gw, gb};
}

std::vector<std::tuple<std::vector<int64_t>, int64_t, int64_t, at::Tensor, int64_t, std::string>> ConvRunner::entries() {
  std::lock_guard<std::mutex> lock(mu_);
  std::vector<std::tuple<std::vector<int64_t>, int64_t, int64_t, at::Tensor, int64_t, std::string>> out;
  for (auto &e : entries_) {
    if (!e->u.defined() || !(e->stamp == newest_)) continue;
    std::vector<int64_t> shape{e->shape[0]};
    for (int i = 4 - nd_; i < 5; ++i) shape.push_back(e->shape[i]);
    out.emplace_back(shape, e->dtype, e->device, e->u, e->serial, std::string(reinterpret_cast<const char *>(&e->info), sizeof e->info));
  }
  return out;
}

std::optional<at::Tensor> conv_call(const at::Tensor &x_in, const at::Tensor &weight_in, const std::optional<at::Tensor> &bias,
                                    std::vector<int64_t> stride, std::vector<int64_t> padding, int64_t compute, bool out_f32, int64_t tile_m) {
  const int nd = (int)x_in.dim() - 2;
  if (!x_in.is_cuda() || (nd != 2 && nd != 3) || weight_in.dim() != nd + 2 || x_in.size(1) != weight_in.size(1) || x_in.numel() == 0 ||
      weight_in.numel() == 0 || (int)stride.size() != nd || (int)padding.size() != nd || (bias && bias->numel() != weight_in.size(0)))
    return std::nullopt;
  // bias with a graph: its gradient is the caller's addition
  if (bias && at::GradMode::is_enabled() && bias->requires_grad()) return std::nullopt;
  const int dtype = compute >= 0 ? (int)compute : code_of(x_in.scalar_type());
  if (dtype < 0 || code_of(x_in.scalar_type()) < 0 || code_of(weight_in.scalar_type()) < 0) return std::nullopt;
  at::AutoDispatchBelowADInplaceOrView no_graph;
  c10::cuda::CUDAGuard guard(x_in.device());
  const at::ScalarType type = type_of(dtype);
  winoconv_desc_t d;
  std::memset(&d, 0, sizeof d);
  d.ndim = nd;
  for (int64_t v : x_in.sizes())
    if (v > 0x7fffffffLL) return std::nullopt;
  d.batch = (int)x_in.size(0); d.c_in = (int)x_in.size(1); d.k_out = (int)weight_in.size(0);
  for (int i = 0; i < 3; ++i) {
    const int a = i - (3 - nd);
    d.in_size[i] = a < 0 ? 1 : (int)x_in.size(2 + a);
    d.ker_size[i] = a < 0 ? 1 : (int)weight_in.size(2 + a);
    d.stride[i] = a < 0 ? 1 : (int)stride[a];
    d.pad[i] = a < 0 ? 0 : (int)padding[a];
  }
  d.dtype = dtype;
  const bool bias_after = bias && out_f32 && dtype != WINOCONV_F32;
  d.epilogue = bias && !bias_after ? WINOCONV_EPI_BIAS : 0u;
  // direct taps, unless the tile asked for does the layer in fewer multiplies than its traffic is worth: F(2,3) of wide fp32 3x3 layers
  // (us direct / F(2,3) on B200 at 28 x 28, N = 8: 128 -> 256 36 / 35, 416 -> 256 103 / 86, 128 -> 96 21 / 27; F(4x4,3x3), which AUTO
  // weighs for the modules, crosses earlier)
  winoconv_plan_info_t info;
  const bool wide_f32 = dtype == WINOCONV_F32 && nd == 2 && d.ker_size[1] == 3 && d.ker_size[2] == 3 && d.stride[1] == 1 && d.stride[2] == 1 &&
                        (int64_t)d.c_in * d.k_out > 128 * 128;
  d.tile_m = 1;
  if (tile_m != 2 || wide_f32 || winoconv_plan(&d, &info) != WINOCONV_OK) {
    d.tile_m = (int)tile_m;
    if (winoconv_plan(&d, &info) != WINOCONV_OK) return std::nullopt;
  }
  void *s = stream_of();
  at::Tensor x = aligned(dense_channels_last(x_in, type, s));
  at::Tensor w = weight_in.to(x.device()).contiguous();
  at::Tensor u = empty_bytes(info.filter_bytes, x);
  if (winoconv_filter_transform_from(&d, w.data_ptr(), code_of(w.scalar_type()), u.data_ptr(), s) != WINOCONV_OK) {
    w = w.to(type);
    check_abi(winoconv_filter_transform(&d, w.data_ptr(), u.data_ptr(), s), "winoconv_filter_transform");
  }
  at::Tensor b;
  if (bias) b = bias->to(x.device(), bias_after ? at::kFloat : type).contiguous();
  at::Tensor v, m;
  if (info.direct != 1) {
    if (info.input_ws_bytes) v = empty_bytes(info.input_ws_bytes, x);
    if (!info.direct && info.product_ws_bytes) m = empty_bytes(info.product_ws_bytes, x);
  }
  int64_t sizes[5] = {d.batch, d.k_out, 0, 0, 0};
  for (int i = 0; i < nd; ++i) sizes[2 + i] = info.out_size[3 - nd + i];
  const at::IntArrayRef out_sizes(sizes, nd + 2);
  at::Tensor y = at::empty(out_sizes, x.options().requires_grad(false), nd == 2 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::ChannelsLast3d);
  check_abi(winoconv_forward(&d, x.data_ptr(), u.data_ptr(), d.epilogue ? b.data_ptr() : nullptr, y.data_ptr(), v.defined() ? v.data_ptr() : nullptr,
                             info.input_ws_bytes, m.defined() ? m.data_ptr() : nullptr, info.product_ws_bytes, s),
            "winoconv_forward");
  const at::ScalarType out_type = out_f32 ? at::kFloat : type;
  at::Tensor out = at::empty(out_sizes, x.options().dtype(out_type).requires_grad(false), at::MemoryFormat::Contiguous);
  const int st = winoconv_to_channels_first(y.data_ptr(), dtype, out.data_ptr(), code_of(out_type), bias_after ? b.data_ptr<float>() : nullptr, d.batch, d.k_out,
                                            y.numel() / ((int64_t)d.batch * d.k_out), s);
  if (st == WINOCONV_ERR_UNSUPPORTED) {
    out.copy_(y);
    if (bias_after) {
      std::vector<int64_t> shape(nd + 2, 1);
      shape[1] = d.k_out;
      out.add_(b.view(shape));
    }
  } else check_abi(st, "winoconv_to_channels_first");
  return out;
}
