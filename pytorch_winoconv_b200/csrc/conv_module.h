// Native forward and backward of the convolution modules (conv.py): plan and filter cache, layout, launches and the autograd
// node without a trip through Python per call.
#pragma once

#include <cstdint>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <utility>
#include <vector>

#include <ATen/cuda/CUDAEvent.h>
#include <torch/extension.h>

#include "winoconv_b200.h"

// One call of the reference's functional operators: x and weight in torch order, the filter transformed on the spot.  compute:
// the dtype of operands and products' result (-1: x's own); the result is in torch order, in fp32 where out_f32 is set (bias
// added in fp32 after the rounding to the compute dtype), else in the compute dtype.  tile_m as in winoconv_desc_t where the
// direct-tap kernel does not take the layer.  Nothing where the caller's own path has to decide.
std::optional<at::Tensor> conv_call(const at::Tensor &x, const at::Tensor &weight, const std::optional<at::Tensor> &bias,
                                    std::vector<int64_t> stride, std::vector<int64_t> padding, int64_t compute, bool out_f32, int64_t tile_m);

// One per module.  Every entry is the plan of an input and a weight shape with its transformed filters; they follow the weights
// (storage, version, dtype), and the least recently used one goes when there are more than `max_plans`.
class ConvRunner : public torch::CustomClassHolder {
 public:
  ConvRunner(int64_t nd, std::vector<int64_t> stride, std::vector<int64_t> padding, int64_t tile_m, int64_t algo, bool relu, bool pool,
             int64_t compute, int64_t max_plans);

  // The module's forward, or nothing where the Python path has to decide (an error to raise, a gradient the kernels do not cover).
  std::optional<at::Tensor> forward(const at::Tensor &x, const at::Tensor &weight, const std::optional<at::Tensor> &bias, bool training);

  // (input shape channels last, dtype code, device index, transformed filter, serial of its transform, plan bytes) of every entry
  // whose filter belongs to the newest weights, least recently used first
  std::vector<std::tuple<std::vector<int64_t>, int64_t, int64_t, at::Tensor, int64_t, std::string>> entries();

  // What a transformed filter was made from.  The weak references keep the tensors' headers (not their memory) from being
  // reused, so that a new tensor at an old one's address is another one: a parametrised module computes its weight per call.
  struct Stamp {
    using Ref = c10::weak_intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl>;
    Ref w_ref{c10::intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl>()}, b_ref{c10::intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl>()};
    const void *w = nullptr, *b = nullptr;
    int64_t w_version = -1, b_version = -1;
    int w_dtype = -1;
    bool operator==(const Stamp &o) const {
      return w_ref == o.w_ref && b_ref == o.b_ref && w == o.w && b == o.b && w_version == o.w_version && b_version == o.b_version && w_dtype == o.w_dtype;
    }
  };
  // Where an entry's buffers were written.  The first call on another stream records an event there (whoever stays on one stream
  // pays for none), waits for it and tells the allocator that it reads them.  A graph capture cannot wait for work outside of it:
  // it uses them once that work has finished, else it makes its own; and what a capture writes holds its values only when the
  // graph runs, so nobody outside of that capture uses it.
  struct Written {
    std::optional<c10::cuda::CUDAStream> stream;
    at::cuda::CUDAEvent event;
    bool recorded = false, finished = false;
    unsigned long long capture = 0;
    void on(const c10::cuda::CUDAStream &here);      // they are written by what is queued on that stream so far
    // false: write them anew; learns: of weights that change between two runs of a graph, which then writes them itself
    bool usable_on(const c10::cuda::CUDAStream &here, bool learns, const at::Tensor &a, const at::Tensor &b);
  };
  struct Entry {
    int64_t shape[5] = {0, 0, 0, 0, 0};      // N, D, H, W, C of the input
    int64_t w_shape[4] = {0, 0, 0, 0};       // K, kD, kH, kW of the weight: a module's weight may be replaced by one of another shape
    int dtype = -1, device = -1, bias_type = -1;   // bias_type: scalar type of the bias, -1 without one
    winoconv_desc_t desc;
    winoconv_plan_info_t info;
    at::Tensor u, bias;                      // transformed filter, bias in the compute dtype
    Stamp stamp;
    Written written;
    int64_t serial = 0;
    bool first = false;                      // x in torch's contiguous order
    at::Tensor u_back;                       // filter of the data gradient
    Stamp back_stamp;
    Written back_written;
    bool back_known = false, back_ok = false;
  };

  at::Tensor run(Entry &e, const at::Tensor &x_cl, const at::Tensor &weight, const std::optional<at::Tensor> &bias, bool learns);
  // Gradients of one layer call; undefined where not asked for.
  std::vector<at::Tensor> backward(const at::Tensor &gy, const at::Tensor &x, const at::Tensor &y, const at::Tensor &weight,
                                   const std::optional<at::Tensor> &bias, bool need_x, bool need_w, bool need_b);

 private:
  std::shared_ptr<Entry> entry_for(const at::Tensor &x, const at::Tensor &weight, const std::optional<at::Tensor> &bias, int dtype, bool first);
  bool backward_covered(Entry &e);      // whether the native gradients take the layer

  int nd_, stride_[3], pad_[3], tile_m_, algo_, compute_;
  bool relu_, pool_;
  size_t max_plans_;
  std::mutex mu_;
  std::vector<std::shared_ptr<Entry>> entries_;     // most recently used last
  std::vector<std::pair<at::Tensor, at::Tensor>> in_graphs_;      // filters and biases that a captured graph reads: kept as long as the module
  Stamp newest_;
  int64_t serial_ = 0;
};
