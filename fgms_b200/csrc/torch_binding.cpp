// PyTorch side of the library: the operator calls and the autograd function as a CPython extension module
// (fgms_b200._native) over the C ABI of libfgms_b200.so.
//
// Argument checks, the choice of the current stream and the kernel launches of a call are a few microseconds of host
// time here; the same steps in Python took 15-20 us per call (20 us for a forward of a few hundred voxels whose
// kernel runs 6 us; 56 us per layer and pass through the autograd engine), which is what bounded every layer of up to
// about a hundred thousand voxels.  Error types are those of the reference's binding: ValueError for what pybind11
// maps from std::invalid_argument, TypeError for an argument that is no tensor, RuntimeError for a CUDA failure.
#include <array>
#include <atomic>
#include <vector>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>
#include <pybind11/pybind11.h>

#include "../../include/fgms_b200.h"

namespace {

using at::Tensor;

void check_status(int rc) {
  if (rc == FGMS_OK) return;
  const char* msg = fgms_b200_last_error();
  if (rc == FGMS_ERR_CHANNEL_MISMATCH || rc == FGMS_ERR_INVALID_ARG || rc == FGMS_ERR_UNSUPPORTED || rc == FGMS_ERR_WORKSPACE)
    TORCH_CHECK_VALUE(false, msg);
  TORCH_CHECK(false, "fgms_b200 error ", rc, ": ", msg);
}

void check_feat(const char* name, const Tensor& t, int64_t dim) {
  TORCH_CHECK_VALUE(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK_VALUE(t.dim() == dim, name, " must have ", dim, " dimensions, got ", t.dim());
  TORCH_CHECK_VALUE(t.is_contiguous(), name, " must be contiguous");
}
void check_feat(const char* name, const Tensor& t, int64_t dim, const Tensor& like) {
  check_feat(name, t, dim);
  TORCH_CHECK_VALUE(t.scalar_type() == like.scalar_type(), name, " must have dtype ", like.scalar_type(), ", got ", t.scalar_type());
}
void check_index(const char* name, const Tensor& t, const Tensor& like, int64_t min_len) {
  TORCH_CHECK_VALUE(t.scalar_type() == at::kInt, name, " must be an int32 tensor");
  TORCH_CHECK_VALUE(t.is_cuda() && t.device() == like.device(), name, " must live on ", like.device());
  TORCH_CHECK_VALUE(t.is_contiguous(), name, " must be contiguous");
  TORCH_CHECK_VALUE(t.numel() >= min_len, name, " needs at least ", min_len, " entries, got ", t.numel());
}

struct Arith { int dtype, math; };
Arith arith(const Tensor& t, bool arch80) {
  if (t.scalar_type() == at::kHalf) return {FGMS_DTYPE_F16, FGMS_MATH_F16};
  TORCH_CHECK_VALUE(t.scalar_type() == at::kFloat, "unsupported feature dtype ", t.scalar_type(), ": the operator takes float16 or float32");
  return {FGMS_DTYPE_F32, arch80 ? FGMS_MATH_TF32 : FGMS_MATH_FP32};
}

void* ptr(const Tensor& t) { return t.numel() > 0 ? t.data_ptr() : nullptr; }
const int32_t* iptr(const Tensor& t) { return static_cast<const int32_t*>(ptr(t)); }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// checks shared by every pass over a pair list; returns k_vol
int check_common(const Tensor& feats, const Tensor& kernel, const Tensor& kpos, const Tensor& in_map, const Tensor& out_map) {
  check_feat("in_feats", feats, 2);
  check_feat("kernel", kernel, 3, feats);
  const int64_t k_vol = kernel.size(0);
  check_index("kpos", kpos, feats, k_vol + 1);
  check_index("in_map", in_map, feats, 0);
  check_index("out_map", out_map, feats, 0);
  TORCH_CHECK_VALUE(in_map.numel() == out_map.numel(), "in_map and out_map differ in length");
  return (int)k_vol;
}

void fusion_fwd(const Tensor& in_feats, const Tensor& kernel, int64_t sum_nnz, const Tensor& out, const Tensor& kpos,
                const Tensor* qkpos, const Tensor& in_map, const Tensor& out_map, bool separate_mid, bool arch80) {
  const int k_vol = check_common(in_feats, kernel, kpos, in_map, out_map);
  check_feat("out_feats", out, 2, in_feats);
  if (qkpos) check_index("qkpos", *qkpos, in_feats, k_vol + 1);
  TORCH_CHECK_VALUE(out.size(1) == kernel.size(2), "out_feats width differs from the kernel's output channels");
  const Arith a = arith(in_feats, arch80);
  c10::cuda::CUDAGuard guard(in_feats.device());
  check_status(fgms_b200_fusion_fwd(ptr(in_feats), ptr(kernel), ptr(out), iptr(kpos), qkpos ? iptr(*qkpos) : nullptr, iptr(in_map),
                                    iptr(out_map), in_map.numel(), (int)in_feats.size(0), (int)out.size(0), (int)in_feats.size(1),
                                    (int)kernel.size(1), (int)kernel.size(2), k_vol, sum_nnz, a.dtype, a.math, separate_mid,
                                    stream_of(in_feats)));
}

void seq_fwd(const Tensor& in_feats, const Tensor& kernel, int64_t sum_nnz, const Tensor& out, const Tensor& kernel_nnz,
             const Tensor& kpos, const Tensor& in_map, const Tensor& out_map, bool separate_mid, bool arch80) {
  const int k_vol = check_common(in_feats, kernel, kpos, in_map, out_map);
  check_feat("out_feats", out, 2, in_feats);
  TORCH_CHECK_VALUE(kernel_nnz.scalar_type() == at::kInt, "kernel_nnz must be an int32 tensor");
  TORCH_CHECK_VALUE(!kernel_nnz.is_cuda(), "kernel_nnz must be a CPU tensor");
  TORCH_CHECK_VALUE(kernel_nnz.is_contiguous(), "kernel_nnz must be contiguous");
  TORCH_CHECK_VALUE(kernel_nnz.numel() >= k_vol, "kernel_nnz needs at least ", k_vol, " entries, got ", kernel_nnz.numel());
  TORCH_CHECK_VALUE(out.size(1) == kernel.size(2), "out_feats width differs from the kernel's output channels");
  const Arith a = arith(in_feats, arch80);
  c10::cuda::CUDAGuard guard(in_feats.device());
  check_status(fgms_b200_seq_fwd(ptr(in_feats), ptr(kernel), ptr(out), kernel_nnz.data_ptr<int32_t>(), iptr(kpos), iptr(in_map),
                                 iptr(out_map), in_map.numel(), (int)in_feats.size(0), (int)out.size(0), (int)in_feats.size(1),
                                 (int)kernel.size(1), (int)kernel.size(2), k_vol, sum_nnz, a.dtype, a.math, separate_mid,
                                 stream_of(in_feats)));
}

// fp32 sums of an fp16 weight gradient that has no single-launch form (or was asked for in fp32 sums): from PyTorch's
// caching allocator, so that calls on different streams or threads never share one
Tensor wgrad_workspace(const Tensor& kernel_grad, const Arith& a, bool fp32_sums) {
  if (a.dtype != FGMS_DTYPE_F16) return {};
  const int c_in = (int)kernel_grad.size(1), c_out = (int)kernel_grad.size(2), k_vol = (int)kernel_grad.size(0);
  if (!fp32_sums && k_vol >= 1 && fgms_b200_kernel_family(2, c_in, c_out, k_vol, a.dtype, a.math) == 1) return {};
  const int64_t n = std::max<int64_t>((int64_t)(fgms_b200_wgrad_workspace_bytes(c_in, c_out, k_vol, a.dtype) / 4), 64);
  return at::empty({n}, kernel_grad.options().dtype(at::kFloat));
}

// The same for both gradients in one call: also where the library is faster with one.  A call whose pointers are not 16-byte aligned
// gets none, nor one for which there is no memory, as it has another way without.
Tensor bwd_workspace(const void* grad_out, const void* feats, const void* kernel, const void* in_grad, const Tensor& kernel_grad, int64_t pairs,
                     const Arith& a, bool fp32_sums) {
  if (const Tensor ws = wgrad_workspace(kernel_grad, a, fp32_sums); ws.defined() || a.dtype != FGMS_DTYPE_F16) return ws;
  const int c_in = (int)kernel_grad.size(1), c_out = (int)kernel_grad.size(2), k_vol = (int)kernel_grad.size(0);
  const size_t bytes = fgms_b200_bwd_workspace_bytes(pairs, c_in, c_out, k_vol, a.dtype, a.math);
  uintptr_t at = 0;
  for (const void* p : {grad_out, feats, kernel, in_grad, (const void*)kernel_grad.data_ptr()}) at |= reinterpret_cast<uintptr_t>(p);
  if (bytes == 0 || (at & 15) != 0) return {};
  try {
    return at::empty({(int64_t)(bytes / 4)}, kernel_grad.options().dtype(at::kFloat));
  } catch (const c10::OutOfMemoryError&) {
    return {};
  }
}

void bwd(const Tensor& grad_out, const Tensor& in_feats, const Tensor& kernel, int64_t sum_nnz, const Tensor& in_grad,
         const Tensor& kernel_grad, const Tensor& kpos, const Tensor* qkpos, const Tensor& in_map, const Tensor& out_map,
         bool separate_mid, bool arch80, bool fp32_sums) {
  const int k_vol = check_common(in_feats, kernel, kpos, in_map, out_map);
  check_feat("out_feats_grad", grad_out, 2, in_feats);
  check_feat("in_feats_grad", in_grad, 2, in_feats);
  check_feat("kernel_grad", kernel_grad, 3, in_feats);
  if (in_feats.size(1) == kernel.size(1)) {  // a channel mismatch is the library's own error below
    TORCH_CHECK_VALUE(in_grad.sizes() == in_feats.sizes() && kernel_grad.sizes() == kernel.sizes(),
                      "gradient buffers must have the shapes of in_feats and kernel");
    TORCH_CHECK_VALUE(grad_out.size(1) == kernel.size(2), "out_feats_grad width differs from the kernel's output channels");
  }
  const Arith a = arith(in_feats, arch80);
  c10::cuda::CUDAGuard guard(in_feats.device());
  const Tensor ws = in_feats.size(1) == kernel.size(1)
                        ? bwd_workspace(ptr(grad_out), ptr(in_feats), ptr(kernel), ptr(in_grad), kernel_grad, in_map.numel(), a, fp32_sums)
                        : Tensor();
  check_status(fgms_b200_bwd(ptr(grad_out), ptr(in_feats), ptr(kernel), ptr(in_grad), ptr(kernel_grad), iptr(kpos),
                             qkpos ? iptr(*qkpos) : nullptr, iptr(in_map), iptr(out_map), in_map.numel(), (int)in_feats.size(0),
                             (int)grad_out.size(0), (int)in_feats.size(1), (int)kernel.size(1), (int)kernel.size(2), k_vol, sum_nnz,
                             a.dtype, a.math, separate_mid, ws.defined() ? ws.data_ptr() : nullptr,
                             ws.defined() ? (size_t)ws.numel() * 4 : 0, stream_of(in_feats)));
}

// ---------------------------------------------------------------------------------------------
// autograd
// ---------------------------------------------------------------------------------------------
// backend.WGRAD_FP32_SUMS.  A backward follows the switch of its own time, not of the forward's; it runs on a thread of the
// autograd engine without the GIL, so the switch is kept here and the module's attribute reads and sets it.
std::atomic<bool> g_fp32_sums{false};

size_t bytes_of(const Tensor& t) { return (size_t)t.numel() * t.element_size(); }

struct SparseConv : torch::autograd::Function<SparseConv> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& feats_, const Tensor& weight_, const Tensor& kpos,
                        const Tensor& imap, const Tensor& omap, int64_t n_out, bool arch80) {
    const Tensor feats = feats_.contiguous(), weight = weight_.contiguous();
    TORCH_CHECK_VALUE(feats.is_cuda(), "in_feats must be a CUDA tensor");
    TORCH_CHECK_VALUE(weight.dim() == 3, "kernel must have 3 dimensions, got ", weight.dim());
    c10::cuda::CUDAGuard guard(feats.device());
    Tensor out = at::empty({n_out, weight.size(2)}, feats.options().requires_grad(false));
    check_status(fgms_b200_zero2(ptr(out), bytes_of(out), nullptr, 0, stream_of(feats)));
    fusion_fwd(feats, weight, 0, out, kpos, nullptr, imap, omap, false, arch80);
    ctx->save_for_backward({feats, weight, kpos, imap, omap});
    ctx->saved_data["arch80"] = arch80;
    return out;
  }

  // Only the gradients that something needs are computed: the first layer of a network has no input gradient, a
  // frozen layer no weight gradient.
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &feats = saved[0], &weight = saved[1], &kpos = saved[2], &imap = saved[3], &omap = saved[4];
    const bool arch80 = ctx->saved_data["arch80"].toBool();
    const Tensor grad_out = grads[0].contiguous();
    const bool need_in = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
    // saved tensors come back through whatever hooks were installed when they were saved: as good as new arguments
    const int k_vol = check_common(feats, weight, kpos, imap, omap);
    check_feat("out_feats_grad", grad_out, 2, feats);
    TORCH_CHECK_VALUE(feats.size(1) == weight.size(1), "Input feature size and kernel size mismatch");
    TORCH_CHECK_VALUE(grad_out.size(1) == weight.size(2), "out_feats_grad width differs from the kernel's output channels");
    c10::cuda::CUDAGuard guard(feats.device());
    void* st = stream_of(feats);
    Tensor in_grad, w_grad;
    if (need_in) in_grad = at::empty_like(feats);
    if (need_w) w_grad = at::empty_like(weight);
    const Arith a = arith(feats, arch80);
    const int n_in = (int)feats.size(0), n_out = (int)grad_out.size(0), c_in = (int)weight.size(1), c_out = (int)weight.size(2);
    check_status(fgms_b200_zero2(need_in ? ptr(in_grad) : nullptr, need_in ? bytes_of(in_grad) : 0, need_w ? ptr(w_grad) : nullptr,
                                 need_w ? bytes_of(w_grad) : 0, st));
    if (need_in && need_w) {  // in one call, which lets them run side by side
      const Tensor ws = bwd_workspace(ptr(grad_out), ptr(feats), ptr(weight), ptr(in_grad), w_grad, imap.numel(), a,
                                      g_fp32_sums.load(std::memory_order_relaxed));
      check_status(fgms_b200_bwd(ptr(grad_out), ptr(feats), ptr(weight), ptr(in_grad), ptr(w_grad), iptr(kpos), nullptr, iptr(imap),
                                 iptr(omap), imap.numel(), n_in, n_out, c_in, c_in, c_out, k_vol, 0, a.dtype, a.math, 0,
                                 ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? (size_t)ws.numel() * 4 : 0, st));
    } else if (need_in) {
      check_status(fgms_b200_dgrad(ptr(grad_out), ptr(weight), ptr(in_grad), iptr(kpos), iptr(imap), iptr(omap), imap.numel(), n_in,
                                   n_out, c_in, c_out, k_vol, a.dtype, a.math, st));
    } else if (need_w) {
      const Tensor ws = wgrad_workspace(w_grad, a, g_fp32_sums.load(std::memory_order_relaxed));
      check_status(fgms_b200_wgrad(ptr(feats), ptr(grad_out), ptr(w_grad), iptr(kpos), iptr(imap), iptr(omap), imap.numel(), n_in,
                                   n_out, c_in, c_out, k_vol, a.dtype, a.math, ws.defined() ? ws.data_ptr() : nullptr,
                                   ws.defined() ? (size_t)ws.numel() * 4 : 0, 1, st));
    }
    return {in_grad, w_grad, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---------------------------------------------------------------------------------------------
// a stack of layers as one node
// ---------------------------------------------------------------------------------------------
// A node per layer costs 14 us of the engine's host time on top of its launches, and a fill of its own for the output and for the
// gradients: 1100 us for the 25 layers of an encoder-decoder on 8 k voxels whose kernels run 500 us.  Here the layers' values lie in one
// allocation, their gradients in another, each cleared by one launch, and the backward is a loop.  The arithmetic is the one of
// a node per layer: every layer adds into zeros, a skip connection and its gradient are sums rounded once.
//
// A node per layer needs less memory: it hands back its input and its output's gradient as the backward goes on.  So beyond STACK_BYTES
// of values, and where there is no memory for one allocation, values and gradients are allocated and cleared one by one and dropped in the
// same way.  Training steps of the 25 layers, peaks above what is there before: 120 k voxels, 59 MB of values, a node per layer 66 MB, two
// allocations 123; 240 k voxels, 113 MB, 129 MB a node per layer and one by one, 231 in two allocations.  By then the device is
// busy for longer than the further allocations and launches take the host: 1970 us a node per layer, 1080-1150 one by one, 965 in two.
//
// Value 0 is the input, value l + 1 what layer l produces.
struct StackLayer { int64_t src, skip /* -1: none */, map, n_in, n_out; };
using StackPlan = std::vector<int64_t>;  // StackLayer by StackLayer
constexpr int64_t STACK_FIELDS = 5;
constexpr int64_t STACK_BYTES = 64 << 20;
StackLayer layer_of(const StackPlan& plan, size_t l) {
  const int64_t* f = plan.data() + l * STACK_FIELDS;
  return {f[0], f[1], f[2], f[3], f[4]};
}

// What every layer's own call would accept, and what one node can hold: each value but the last is used, by one layer at most.
// False: the caller runs layer by layer, and meets its errors there.
bool stack_suits(const Tensor& feats, at::TensorList weights, at::TensorList maps, const StackPlan& plan, bool arch80) {
  const size_t n = weights.size();
  const auto dtype = feats.scalar_type();
  if (n == 0 || plan.size() != n * STACK_FIELDS || maps.size() % 3 != 0) return false;
  if (!feats.is_cuda() || feats.dim() != 2 || !feats.is_contiguous() || (dtype != at::kHalf && dtype != at::kFloat)) return false;
  auto aligned = [](const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; };
  if (feats.numel() == 0 || !aligned(feats)) return false;
  for (const Tensor& m : maps)
    if (m.scalar_type() != at::kInt || m.device() != feats.device() || !m.is_contiguous() || m.requires_grad()) return false;
  struct Value { int64_t rows, width; int convs, skips; };
  std::vector<Value> value(1, {feats.size(0), feats.size(1), 0, 0});
  value.reserve(n + 1);
  for (size_t l = 0; l < n; ++l) {
    const StackLayer s = layer_of(plan, l);
    const Tensor& w = weights[l];
    const int64_t known = (int64_t)value.size();
    if (w.scalar_type() != dtype || w.device() != feats.device() || w.dim() != 3 || !w.is_contiguous() || w.numel() == 0 || !aligned(w)) return false;
    if (s.src < 0 || s.src >= known || s.skip >= known || s.map < 0 || 3 * s.map + 2 >= (int64_t)maps.size() || s.n_out < 1) return false;
    const Tensor &kpos = maps[3 * s.map], &imap = maps[3 * s.map + 1], &omap = maps[3 * s.map + 2];
    Value& from = value[s.src];
    if (from.rows != s.n_in || from.width != w.size(1) || kpos.numel() != w.size(0) + 1 || imap.numel() != omap.numel()) return false;
    if (from.convs++ > 0) return false;
    value.push_back({s.n_out, w.size(2), 0, 0});
    if (s.skip >= 0) {
      Value& add = value[s.skip];
      if (add.rows != s.n_out || add.width != w.size(2)) return false;
      ++add.skips;
    }
  }
  for (size_t v = 1; v < n; ++v)
    if (value[v].convs + value[v].skips == 0) return false;
  return true;
}

struct SparseStack : torch::autograd::Function<SparseStack> {
  // What the node keeps, in elements: the values that layers 0 .. n - 2 produce (slots 1 .. n - 1) and, where the input's few fp16
  // channels are padded to a multiple of 16 (8-byte rows cannot be gathered in 16-byte pieces and would run on the CUDA cores: 4 -> 32
  // on 84 k pairs 16.6 / 45 us forward / weight gradient, padded 4.9 / 6.2), the padded input (slot 0) and the weights that go with it (slot n).
  struct Layout {
    std::vector<int64_t> count, at;  // of a slot; its place in a block of all of them, from a 256-byte boundary
    int64_t end = 0;                 // of that block
    int64_t pad = 0;                 // channels of the padded input, 0: as it is
    template <typename Kept>
    Layout(const Tensor& feats, at::TensorList kernels, const StackPlan& plan, bool padding, Kept kept) {
      const size_t n = kernels.size();
      count.resize(n + 1);
      at.resize(n + 1);
      for (size_t l = 0; l + 1 < n; ++l)
        if (kept(l + 1)) count[l + 1] = layer_of(plan, l).n_out * kernels[l].size(2);
      const Tensor* reader = nullptr;  // the layer of the input
      padding = padding && feats.scalar_type() == at::kHalf && feats.size(1) % 16 != 0 && feats.size(1) <= 256;
      for (size_t l = 0; padding && l < n; ++l) {
        padding = layer_of(plan, l).skip != 0;
        if (layer_of(plan, l).src == 0) reader = &kernels[l];
      }
      if (padding && reader && reader->size(2) % 16 == 0 && reader->size(2) <= 256) {
        pad = (feats.size(1) + 15) / 16 * 16;
        count[0] = feats.size(0) * pad;
        count[n] = reader->size(0) * pad * reader->size(2);
      }
      for (size_t i = 0; i <= n; ++i) {
        at[i] = end;
        end += (count[i] + 127) / 128 * 128;
      }
    }
  };
  // The slots of a layout: in one block, or by themselves (each until it is dropped).
  struct Slots {
    const Layout& layout;
    at::TensorOptions options;
    Tensor block;
    std::vector<Tensor> own;
    Slots(const Layout& l, const Tensor& like) : layout(l), options(like.options().requires_grad(false)) {}
    bool apart() const { return !own.empty(); }
    // a block where there is memory for one and `may` says so
    void take(bool may) {
      if (may) {
        try {
          block = at::empty({layout.end}, options);
          return;
        } catch (const c10::OutOfMemoryError&) {
        }
      }
      own.resize(layout.count.size());
    }
    const Tensor& make(size_t i) { return own[i] = at::empty({layout.count[i]}, options); }
    void drop(size_t i) { if (apart()) own[i].reset(); }
    void* of(size_t i) const {
      return apart() ? own[i].data_ptr() : static_cast<uint8_t*>(block.data_ptr()) + layout.at[i] * block.element_size();
    }
  };
  // the input and its layer's weights with further channels of zeros, into cleared slots
  static void pad_input(const Slots& slots, const Tensor& feats, const Tensor& w, int dtype, void* st) {
    const int64_t pad = slots.layout.pad, c_in = feats.size(1);
    check_status(fgms_b200_copy_rows_f16(ptr(feats), c_in, dtype, slots.of(0), pad, feats.size(0), (int)c_in, st));
    check_status(fgms_b200_copy_rows_f16(ptr(w), c_in * w.size(2), dtype, slots.of(slots.layout.at.size() - 1), pad * w.size(2), w.size(0), (int)(c_in * w.size(2)), st));
  }

  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& feats, at::TensorList weights, at::TensorList maps,
                        const StackPlan& plan, bool arch80) {
    const size_t n = weights.size();
    c10::cuda::CUDAGuard guard(feats.device());
    void* st = stream_of(feats);
    const Arith a = arith(feats, arch80);
    const Layout in(feats, weights, plan, true, [](size_t) { return true; });
    Slots values(in, feats);
    values.take(in.end * (int64_t)feats.element_size() <= STACK_BYTES);
    Tensor out = at::empty({layer_of(plan, n - 1).n_out, weights[n - 1].size(2)}, values.options);
    auto cleared = [&](const Tensor& t) { check_status(fgms_b200_zero2(ptr(t), bytes_of(t), nullptr, 0, st)); };
    if (values.apart()) cleared(out);
    else check_status(fgms_b200_zero2(ptr(values.block), bytes_of(values.block), ptr(out), bytes_of(out), st));
    auto make = [&](size_t i) {
      if (values.apart()) cleared(values.make(i));
    };
    auto value = [&](int64_t v) -> void* {
      if (v == 0) return in.pad ? values.of(0) : feats.data_ptr();
      return v == (int64_t)n ? out.data_ptr() : values.of(v);
    };
    for (size_t l = 0; l < n; ++l) {
      const StackLayer s = layer_of(plan, l);
      const Tensor &w = weights[l], &imap = maps[3 * s.map + 1];
      const bool padded = s.src == 0 && in.pad;
      if (padded) {
        make(0);
        make(n);
        pad_input(values, feats, w, a.dtype, st);
      }
      if (l + 1 < n) make(l + 1);
      const int c_in = padded ? (int)in.pad : (int)w.size(1);
      check_status(fgms_b200_fusion_fwd(value(s.src), padded ? values.of(n) : ptr(w), value(l + 1), iptr(maps[3 * s.map]), nullptr, iptr(imap),
                                        iptr(maps[3 * s.map + 2]), imap.numel(), (int)s.n_in, (int)s.n_out, c_in, c_in, (int)w.size(2), (int)w.size(0), 0,
                                        a.dtype, a.math, 0, st));
      if (s.skip >= 0) check_status(fgms_b200_add(value(l + 1), value(s.skip), s.n_out * w.size(2), a.dtype, st));
      if (padded) {  // made again for the backward
        values.drop(0);
        values.drop(n);
      }
    }
    torch::autograd::variable_list saved;
    saved.reserve(2 + n + maps.size());
    saved.push_back(feats);
    saved.push_back(values.block);
    saved.insert(saved.end(), weights.begin(), weights.end());
    saved.insert(saved.end(), maps.begin(), maps.end());
    ctx->save_for_backward(std::move(saved));
    if (values.apart()) ctx->saved_data["values"] = values.own;
    ctx->saved_data["plan"] = plan;
    ctx->saved_data["arch80"] = arch80;
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const StackPlan plan = ctx->saved_data["plan"].toIntVector();
    const bool arch80 = ctx->saved_data["arch80"].toBool();
    const size_t n = plan.size() / STACK_FIELDS;
    const Tensor& feats = saved[0];
    const at::TensorList weights(saved.data() + 2, n), maps(saved.data() + 2 + n, saved.size() - 2 - n);
    TORCH_CHECK_VALUE(stack_suits(feats, weights, maps, plan, arch80), "saved tensors of the stack are not the ones it was run with");
    Tensor grad_out = grads[0].contiguous();
    check_feat("out_feats_grad", grad_out, 2, feats);
    if (reinterpret_cast<uintptr_t>(grad_out.data_ptr()) & 15) grad_out = grad_out.clone();
    c10::cuda::CUDAGuard guard(feats.device());
    void* st = stream_of(feats);
    const Arith a = arith(feats, arch80);
    TORCH_CHECK_VALUE(grad_out.size(0) == layer_of(plan, n - 1).n_out && grad_out.size(1) == weights[n - 1].size(2),
                      "out_feats_grad has another shape than the output");
    const Layout in(feats, weights, plan, true, [](size_t) { return true; });
    Slots values(in, feats);
    values.block = saved[1];
    if (const auto kept = ctx->saved_data.find("values"); kept != ctx->saved_data.end()) {
      // the last backward hands them back on the way
      values.own = kept->second.toTensorVector();
      if (!torch::autograd::get_current_graph_task_keep_graph()) ctx->saved_data.erase(kept);
    } else {
      const Tensor& block = values.block;
      TORCH_CHECK_VALUE(block.defined() && block.scalar_type() == feats.scalar_type() && block.device() == feats.device() && block.is_contiguous() &&
                        block.numel() == in.end && (reinterpret_cast<uintptr_t>(block.data_ptr()) & 15) == 0, "saved values of the stack are not the ones it was run with");
    }
    // gradients that something needs: a value's, if a weight before it or the input needs one
    std::vector<char> need(n + 1, 0), need_w(n);
    need[0] = ctx->needs_input_grad(0);
    for (size_t l = 0; l < n; ++l) {
      const StackLayer s = layer_of(plan, l);
      need_w[l] = ctx->needs_input_grad(1 + l);
      need[l + 1] = need_w[l] || need[s.src] || (s.skip >= 0 && need[s.skip]);
    }
    const Layout out(feats, weights, plan, false, [&](size_t v) { return need[v] != 0; });
    torch::autograd::variable_list result(1 + n + maps.size() + 2);
    Slots g_values(out, feats);
    g_values.take(!values.apart());
    Tensor g_input;
    auto make_g_input = [&] { return at::empty({feats.size(0), in.pad ? in.pad : feats.size(1)}, values.options); };
    if (!g_values.apart()) {  // otherwise each when it is first used
      std::vector<void*> clear;
      std::vector<size_t> bytes;
      auto add = [&](const Tensor& t) { clear.push_back(ptr(t)); bytes.push_back(bytes_of(t)); };
      add(g_values.block);
      if (need[0]) add(g_input = make_g_input());
      for (size_t l = 0; l < n; ++l)
        if (need_w[l]) add(result[1 + l] = at::empty_like(weights[l]));
      check_status(fgms_b200_zero_list(clear.data(), bytes.data(), (int)clear.size(), st));
    }
    auto cleared = [&](const Tensor& t) { check_status(fgms_b200_zero2(ptr(t), bytes_of(t), nullptr, 0, st)); };
    auto value = [&](int64_t v) -> void* { return v == 0 && !in.pad ? feats.data_ptr() : values.of(v); };
    auto grad = [&](int64_t v) -> void* {
      if (v == (int64_t)n) return grad_out.data_ptr();
      if (v == 0) {
        if (!g_input.defined()) cleared(g_input = make_g_input());
        return g_input.data_ptr();
      }
      if (g_values.apart() && !g_values.own[v].defined()) cleared(g_values.make(v));
      return g_values.of(v);
    };
    std::vector<std::vector<int64_t>> added(n + 1);  // values whose gradient is part of a value's, through a skip connection
    auto finish = [&](int64_t v, int64_t count) {    // its layer's input gradient is in it
      for (int64_t from : added[v]) {
        check_status(fgms_b200_add(grad(v), grad(from), count, a.dtype, st));
        if (from < (int64_t)n) g_values.drop(from);
      }
    };
    const bool fp32_sums = g_fp32_sums.load(std::memory_order_relaxed);
    // both gradients of a layer
    auto layer = [&](size_t l, const StackLayer& s) {
      const Tensor &w = weights[l], &imap = maps[3 * s.map + 1];
      const int32_t *kpos = iptr(maps[3 * s.map]), *im = iptr(imap), *om = iptr(maps[3 * s.map + 2]);
      const int c_in = (int)w.size(1), c_out = (int)w.size(2), k_vol = (int)w.size(0), n_in = (int)s.n_in, n_out = (int)s.n_out;
      if (need_w[l] && !result[1 + l].defined()) cleared(result[1 + l] = at::empty_like(w));
      if (s.src == 0 && in.pad) {
        const int pad = (int)in.pad;
        if (values.apart()) {
          cleared(values.make(0));
          cleared(values.make(n));
          pad_input(values, feats, w, a.dtype, st);
        }
        if (need_w[l]) {  // fp32 sums, of which the rows of the real channels are rounded
          const Tensor sums = at::empty({(int64_t)k_vol * pad * c_out}, w.options().dtype(at::kFloat).requires_grad(false));
          check_status(fgms_b200_wgrad(value(0), grad(l + 1), nullptr, kpos, im, om, imap.numel(), n_in, n_out, pad, c_out, k_vol, a.dtype, a.math,
                                       sums.data_ptr(), bytes_of(sums), 0, st));
          check_status(fgms_b200_copy_rows_f16(sums.data_ptr(), pad * c_out, FGMS_DTYPE_F32, result[1 + l].data_ptr(), c_in * c_out, k_vol, c_in * c_out, st));
        }
        if (need[0])
          check_status(fgms_b200_dgrad(grad(l + 1), values.of(n), grad(0), kpos, im, om, imap.numel(), n_in, n_out, pad, c_out, k_vol, a.dtype, a.math, st));
        return;
      }
      const Tensor ws = !need_w[l] ? Tensor()
                        : need[s.src] ? bwd_workspace(grad(l + 1), value(s.src), ptr(w), grad(s.src), result[1 + l], imap.numel(), a, fp32_sums)
                                      : wgrad_workspace(result[1 + l], a, fp32_sums);
      void* ws_ptr = ws.defined() ? ws.data_ptr() : nullptr;
      const size_t ws_bytes = ws.defined() ? bytes_of(ws) : 0;
      if (need[s.src] && need_w[l])
        check_status(fgms_b200_bwd(grad(l + 1), value(s.src), ptr(w), grad(s.src), result[1 + l].data_ptr(), kpos, nullptr, im, om, imap.numel(), n_in,
                                   n_out, c_in, c_in, c_out, k_vol, 0, a.dtype, a.math, 0, ws_ptr, ws_bytes, st));
      else if (need[s.src])
        check_status(fgms_b200_dgrad(grad(l + 1), ptr(w), grad(s.src), kpos, im, om, imap.numel(), n_in, n_out, c_in, c_out, k_vol, a.dtype, a.math, st));
      else if (need_w[l])
        check_status(fgms_b200_wgrad(value(s.src), grad(l + 1), result[1 + l].data_ptr(), kpos, im, om, imap.numel(), n_in, n_out, c_in, c_out, k_vol,
                                     a.dtype, a.math, ws_ptr, ws_bytes, 1, st));
    };
    for (size_t l = n; l-- > 0;) {
      const StackLayer s = layer_of(plan, l);
      if (need[l + 1]) {
        if (l + 1 < n) finish(l + 1, s.n_out * weights[l].size(2));
        layer(l, s);
        if (s.skip >= 0 && need[s.skip]) added[s.skip].push_back(l + 1);
        else if (l + 1 < n) g_values.drop(l + 1);
      }
      values.drop(s.src);  // no other layer reads it
    }
    if (need[0]) {
      finish(0, feats.numel());
      grad(0);
      result[0] = in.pad ? g_input.narrow(1, 0, feats.size(1)).contiguous() : g_input;
    }
    return result;
  }
};

// output-stationary forward into `out`; nbr is the table fgms_b200_build_neighbor_table fills
void fwd_os(const Tensor& in_feats, const Tensor& kernel, const Tensor& out, const Tensor& nbr, bool arch80, const Tensor* bias,
            bool relu, bool accumulate) {
  check_feat("in_feats", in_feats, 2);
  check_feat("kernel", kernel, 3, in_feats);
  check_feat("out_feats", out, 2, in_feats);
  TORCH_CHECK_VALUE(kernel.size(1) == in_feats.size(1), "Input feature size and kernel size mismatch");
  TORCH_CHECK_VALUE(out.size(1) == kernel.size(2), "out_feats width differs from the kernel's output channels");
  const int64_t k_vol = kernel.size(0), stride = (out.size(0) + 127) / 128 * 128;
  TORCH_CHECK_VALUE(nbr.scalar_type() == at::kInt && nbr.is_contiguous() && nbr.device() == in_feats.device() && nbr.numel() == k_vol * stride,
                    "nbr must be the contiguous int32 table build_neighbor_table returns for these sizes");
  if (bias) {
    check_feat("bias", *bias, 1, in_feats);
    TORCH_CHECK_VALUE(bias->numel() == kernel.size(2), "bias length differs from the kernel's output channels");
  }
  const Arith a = arith(in_feats, arch80);
  c10::cuda::CUDAGuard guard(in_feats.device());
  check_status(fgms_b200_fwd_output_stationary(ptr(in_feats), ptr(kernel), ptr(out), iptr(nbr), (int)in_feats.size(0), (int)out.size(0),
                                               (int)in_feats.size(1), (int)kernel.size(2), (int)k_vol, a.dtype, a.math,
                                               bias ? ptr(*bias) : nullptr, relu, accumulate, stream_of(in_feats)));
}

// ---------------------------------------------------------------------------------------------
// kernel maps
// ---------------------------------------------------------------------------------------------
struct Pyramid {
  bool fits = false;
  std::vector<int64_t> voxels;                  // per level
  std::vector<std::array<Tensor, 3>> maps;      // kpos, imap, omap
  std::vector<Tensor> out_coords;               // level 1 ..
};

// The maps of `what` (see fgms_b200_pyramid_plan) of the cloud and its coarser levels.  One wait, for the sizes (two if the
// box turns out larger than the first workspace has room for); the Python objects around the maps are made while the last
// kernel runs.
Pyramid try_pyramid(const Tensor& coords, int levels, int what) {
  TORCH_CHECK_VALUE(coords.is_cuda() && coords.scalar_type() == at::kInt && coords.dim() == 2 && coords.size(1) == 3 && coords.is_contiguous(),
                    "coords must be a contiguous CUDA int32 tensor of shape [n, 3]");
  Pyramid r;
  const int64_t n64 = coords.size(0);
  if (n64 < 1 || n64 > 0x7fffffffll / 27) return r;
  const int n = (int)n64;
  size_t bytes = fgms_b200_pyramid_workspace_bytes(n, levels, what);
  if (bytes == 0) return r;
  c10::cuda::CUDAGuard guard(coords.device());
  void* st = stream_of(coords);
  const auto ints = coords.options();
  const int n_maps = ((what & 1) ? levels : 0) + ((what & 2) ? levels - 1 : 0) + ((what & 4) ? levels - 1 : 0);
  const Tensor host = at::empty({64}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
  const int32_t* sizes = host.data_ptr<int32_t>();
  Tensor ws, kpos;
  std::vector<int32_t*> coord_ptrs;
  for (int attempt = 0;; ++attempt) {
    ws = Tensor();  // before the larger one
    ws = at::empty({(int64_t)bytes}, ints.dtype(at::kByte));
    if (attempt == 0) {
      kpos = at::empty({n_maps * 28}, ints);
      for (int l = 1; l < levels; ++l) {
        r.out_coords.push_back(at::empty({n64, 3}, ints));
        coord_ptrs.push_back(r.out_coords.back().data_ptr<int32_t>());
      }
    }
    int rc;
    {
      pybind11::gil_scoped_release unlock;  // this waits for the device
      rc = fgms_b200_pyramid_plan(iptr(coords), n, levels, what, kpos.data_ptr<int32_t>(), coord_ptrs.data(), ws.data_ptr(), bytes,
                                  host.data_ptr<int32_t>(), st);
    }
    check_status(rc);
    if (sizes[0] == 0) break;
    if (sizes[1] == 0 || attempt > 0) return Pyramid();
    bytes = (size_t)sizes[1] * 256;
  }
  r.fits = true;
  for (int l = 0; l < levels; ++l) r.voxels.push_back(sizes[1 + l]);
  // Both sides of a map in one allocation, each on a 256-byte boundary; a map has memory of its own, so that one that is kept does not
  // keep the others.  The device waits for the addresses only: they become tensors while it writes the maps, one TensorImpl a side
  // (13 maps of 120 k voxels: at::empty here and narrow there 112 us, so 91).
  c10::Allocator* memory = c10::cuda::CUDACachingAllocator::get();
  auto padded = [&](int j) { return ((int64_t)sizes[1 + levels + j] + 64) / 64 * 64; };
  std::vector<c10::DataPtr> flat;
  std::vector<int32_t*> in_maps, out_maps;
  flat.reserve(n_maps);
  for (int j = 0; j < n_maps; ++j) {
    flat.push_back(memory->allocate(2 * padded(j) * sizeof(int32_t)));
    in_maps.push_back(static_cast<int32_t*>(flat[j].get()));
    out_maps.push_back(in_maps[j] + padded(j));
  }
  check_status(fgms_b200_pyramid_emit(iptr(coords), n, levels, what, kpos.data_ptr<int32_t>(), coord_ptrs.data(), in_maps.data(),
                                      out_maps.data(), ws.data_ptr(), bytes, st));
  for (int j = 0; j < n_maps; ++j) {
    const c10::Storage storage(c10::Storage::use_byte_size_t(), 2 * padded(j) * sizeof(int32_t), std::move(flat[j]), memory, true);
    auto side = [&](int64_t offset) {
      Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(storage), c10::DispatchKeySet(c10::DispatchKey::CUDA), caffe2::TypeMeta::Make<int32_t>());
      t.unsafeGetTensorImpl()->set_storage_offset(offset);
      t.unsafeGetTensorImpl()->set_sizes_contiguous({(int64_t)sizes[1 + levels + j]});
      return t;
    };
    const bool subm = (what & 1) && j < levels;
    r.maps.push_back({kpos.narrow(0, j * 28, subm ? 28 : 9), side(0), side(padded(j))});
  }
  for (int l = 1; l < levels; ++l) r.out_coords[l - 1] = r.out_coords[l - 1].narrow(0, 0, r.voxels[l]);
  return r;
}

// A cloud for whose bitmaps there is no memory does not fit either: the other builders need less.
Pyramid build_pyramid(const Tensor& coords, int levels, int what) {
  try {
    return try_pyramid(coords, levels, what);
  } catch (const c10::OutOfMemoryError&) {
    return Pyramid();
  }
}

// ---------------------------------------------------------------------------------------------
// Python entry points (positional arguments only; the functions of backend.py / nn.py give them their names)
// ---------------------------------------------------------------------------------------------
const Tensor& feat_arg(PyObject* o, const char* name) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a torch.Tensor");
  return THPVariable_Unpack(o);
}
const Tensor& index_arg(PyObject* o, const char* name) {
  TORCH_CHECK_VALUE(THPVariable_Check(o), name, " must be an int32 tensor");
  return THPVariable_Unpack(o);
}
const Tensor* optional_arg(PyObject* o, const char* name) { return o == Py_None ? nullptr : &index_arg(o, name); }
int64_t int_arg(PyObject* o) {  // like int(o): a Python or NumPy integer, or a tensor of one element
  PyObject* n = PyLong_CheckExact(o) ? Py_NewRef(o) : PyNumber_Long(o);
  if (!n) throw python_error();
  const long long v = PyLong_AsLongLong(n);
  Py_DECREF(n);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
bool bool_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
void expect(Py_ssize_t got, Py_ssize_t want) { TORCH_CHECK_TYPE(got == want, "expected ", want, " arguments, got ", got); }

PyObject* py_fusion_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 10);
  const Tensor &in_feats = feat_arg(a[0], "in_feats"), &kernel = feat_arg(a[1], "kernel"), &out = feat_arg(a[3], "out_feats");
  const Tensor &kpos = index_arg(a[4], "kpos"), *qkpos = optional_arg(a[5], "qkpos");
  const Tensor &in_map = index_arg(a[6], "in_map"), &out_map = index_arg(a[7], "out_map");
  fusion_fwd(in_feats, kernel, int_arg(a[2]), out, kpos, qkpos, in_map, out_map, bool_arg(a[8]), bool_arg(a[9]));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
PyObject* py_seq_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 10);
  const Tensor &in_feats = feat_arg(a[0], "in_feats"), &kernel = feat_arg(a[1], "kernel"), &out = feat_arg(a[3], "out_feats");
  const Tensor &nnz = index_arg(a[4], "kernel_nnz"), &kpos = index_arg(a[5], "kpos");
  const Tensor &in_map = index_arg(a[6], "in_map"), &out_map = index_arg(a[7], "out_map");
  seq_fwd(in_feats, kernel, int_arg(a[2]), out, nnz, kpos, in_map, out_map, bool_arg(a[8]), bool_arg(a[9]));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
PyObject* py_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 13);
  const Tensor &grad_out = feat_arg(a[0], "out_feats_grad"), &in_feats = feat_arg(a[1], "in_feats"), &kernel = feat_arg(a[2], "kernel");
  const Tensor &in_grad = feat_arg(a[4], "in_feats_grad"), &kernel_grad = feat_arg(a[5], "kernel_grad");
  const Tensor &kpos = index_arg(a[6], "kpos"), *qkpos = optional_arg(a[7], "qkpos");
  const Tensor &in_map = index_arg(a[8], "in_map"), &out_map = index_arg(a[9], "out_map");
  bwd(grad_out, in_feats, kernel, int_arg(a[3]), in_grad, kernel_grad, kpos, qkpos, in_map, out_map, bool_arg(a[10]), bool_arg(a[11]),
      bool_arg(a[12]));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
PyObject* py_sparse_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 7);
  const Tensor &feats = feat_arg(a[0], "in_feats"), &weight = feat_arg(a[1], "kernel");
  const Tensor &kpos = index_arg(a[2], "kpos"), &imap = index_arg(a[3], "in_map"), &omap = index_arg(a[4], "out_map");
  return THPVariable_Wrap(SparseConv::apply(feats, weight, kpos, imap, omap, int_arg(a[5]), bool_arg(a[6])));
  END_HANDLE_TH_ERRORS
}
// (in_feats, [kernels], [kpos, in_map, out_map of every map], [src, skip, map, n_in, n_out of every layer], arch80) -> the last layer's
// output, or None where the layers are to be run one by one
PyObject* py_sparse_stack(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 5);
  const Tensor& feats = feat_arg(a[0], "in_feats");
  auto tensors = [](PyObject* list, const char* name) {
    TORCH_CHECK_TYPE(PyList_Check(list), name, " must be a list");
    std::vector<Tensor> out;
    out.reserve(PyList_GET_SIZE(list));
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) out.push_back(feat_arg(PyList_GET_ITEM(list, i), name));
    return out;
  };
  const std::vector<Tensor> weights = tensors(a[1], "kernels"), maps = tensors(a[2], "maps");
  TORCH_CHECK_TYPE(PyList_Check(a[3]), "plan must be a list");
  StackPlan plan;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(a[3]); ++i) plan.push_back(int_arg(PyList_GET_ITEM(a[3], i)));
  const bool arch80 = bool_arg(a[4]);
  if (!stack_suits(feats, weights, maps, plan, arch80)) Py_RETURN_NONE;
  return THPVariable_Wrap(SparseStack::apply(feats, at::TensorList(weights), at::TensorList(maps), plan, arch80));
  END_HANDLE_TH_ERRORS
}
PyObject* py_wgrad_fp32_sums(PyObject*, PyObject* const* a, Py_ssize_t n) {  // () -> the switch; (value) sets it
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n <= 1, "expected at most 1 argument, got ", n);
  if (n == 1) g_fp32_sums.store(bool_arg(a[0]), std::memory_order_relaxed);
  return PyBool_FromLong(g_fp32_sums.load(std::memory_order_relaxed));
  END_HANDLE_TH_ERRORS
}
PyObject* py_fwd_os(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 8);
  const Tensor &in_feats = feat_arg(a[0], "in_feats"), &kernel = feat_arg(a[1], "kernel"), &out = feat_arg(a[2], "out_feats");
  const Tensor &nbr = index_arg(a[3], "nbr"), *bias = a[5] == Py_None ? nullptr : &feat_arg(a[5], "bias");
  fwd_os(in_feats, kernel, out, nbr, bool_arg(a[4]), bias, bool_arg(a[6]), bool_arg(a[7]));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// (voxels per level, [(kpos, imap, omap) ...], [coords of level 1 ...]), or None for a cloud that does not suit
PyObject* py_build_pyramid(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 3);
  const Pyramid r = build_pyramid(index_arg(a[0], "coords"), (int)int_arg(a[1]), (int)int_arg(a[2]));
  if (!r.fits) Py_RETURN_NONE;
  PyObject *voxels = PyList_New(r.voxels.size()), *maps = PyList_New(r.maps.size()), *coords = PyList_New(r.out_coords.size());
  for (size_t i = 0; i < r.voxels.size(); ++i) PyList_SET_ITEM(voxels, i, PyLong_FromLongLong(r.voxels[i]));
  for (size_t i = 0; i < r.maps.size(); ++i) {
    PyObject* t = PyTuple_New(3);
    for (int k = 0; k < 3; ++k) PyTuple_SET_ITEM(t, k, THPVariable_Wrap(r.maps[i][k]));
    PyList_SET_ITEM(maps, i, t);
  }
  for (size_t i = 0; i < r.out_coords.size(); ++i) PyList_SET_ITEM(coords, i, THPVariable_Wrap(r.out_coords[i]));
  return Py_BuildValue("(NNN)", voxels, maps, coords);
  END_HANDLE_TH_ERRORS
}

#define FGMS_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FGMS_METHOD("fusion_fwd", py_fusion_fwd), FGMS_METHOD("seq_fwd", py_seq_fwd),         FGMS_METHOD("bwd", py_bwd),
    FGMS_METHOD("fwd_os", py_fwd_os),         FGMS_METHOD("sparse_conv", py_sparse_conv),
    FGMS_METHOD("sparse_stack", py_sparse_stack),
    FGMS_METHOD("wgrad_fp32_sums", py_wgrad_fp32_sums),
    FGMS_METHOD("build_pyramid", py_build_pyramid), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module_def); }
