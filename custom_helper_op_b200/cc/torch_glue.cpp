// The differentiable op functions of python/ops/custom_helper_ops.py in native code: argument checks, output
// allocation, the C-ABI call and the autograd node of each op.
//
// Why: a small training step (c0: 27 us of kernels) spent 185 us in Python - ctypes marshalling, two
// torch.autograd.Function trampolines, and the gradient's Python code run on the autograd engine's thread, which has to
// wait for the interpreter lock first.  Here a node is a torch::autograd::Node whose apply() runs without the
// interpreter, and an undefined gradient of the int32 mask is never materialised (that was a fill of the whole mask per
// step).  Messages and exception types are those of the raw Python functions.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/chop.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// ---- errors ----------------------------------------------------------------------------------------------
// the reference reports these through OP_REQUIRES -> InvalidArgumentError; ValueError in Python
inline void require(bool cond, const char* msg) {
  if (!cond) throw std::invalid_argument(msg);
}

// A status of the C ABI becomes _lib.ChopError, also on the autograd engine's thread.
void check(int status, const char* what) {
  if (status == 0) return;
  py::gil_scoped_acquire gil;
  py::object cls = py::module_::import("custom_helper_op_b200._lib").attr("ChopError");
  py::object err = cls(status, what);
  PyErr_SetObject(cls.ptr(), err.ptr());
  python_error e;
  e.persist();
  throw e;
}

// The same for the checks of a gradient: what apply() throws reaches Python through the engine, as a RuntimeError unless it
// is a Python exception.
template <typename F>
auto in_engine(F&& f) -> decltype(f()) {
  try {
    return f();
  } catch (const std::invalid_argument& x) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(PyExc_ValueError, x.what());
    python_error e;
    e.persist();
    throw e;
  }
}

// python_error crosses the pybind boundary as the exception that it holds
template <typename F>
auto guarded(F&& f) -> decltype(f()) {
  try {
    return f();
  } catch (python_error& e) {
    py::gil_scoped_acquire gil;
    e.restore();
    throw py::error_already_set();
  }
}

// What the nodes below do not implement is refused, not dropped: a forward-mode tangent (torch.autograd.Function without a
// jvp raises the same type) and the wrapped tensors of torch.func's transforms (vmap, grad, jvp), which have no memory.
void refuse_transforms(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts) {
    if (!t->defined()) continue;
    if (t->key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper})))
      throw std::runtime_error("custom_helper_op: the ops do not support torch.func transforms (vmap, grad, jvp, ...)");
    if (t->_fw_grad(/*level=*/0).defined()) {
      py::gil_scoped_acquire gil;
      PyErr_SetString(PyExc_NotImplementedError, "custom_helper_op: the ops do not implement forward mode AD (jvp)");
      python_error e;
      e.persist();
      throw e;
    }
  }
}

// ---- small helpers ---------------------------------------------------------------------------------------
int chop_dtype_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return CHOP_F32;
    case at::kDouble: return CHOP_F64;
    case at::kBFloat16: return CHOP_BF16;
    default: throw std::invalid_argument("dtype must be float32, float64 or bfloat16");
  }
}
// depths, cameras, costs and gradients of bfloat16 features are float32
at::ScalarType real_of(at::ScalarType t) { return t == at::kBFloat16 ? at::kFloat : t; }

// contiguous tensor of the given type on the given device; the common case costs no dispatch
Tensor as(const Tensor& t, at::ScalarType dt, at::Device dev) {
  if (t.scalar_type() == dt && t.device() == dev && t.is_contiguous()) return t;
  return t.to(dev, dt).contiguous();
}
Tensor fresh(at::IntArrayRef shape, at::ScalarType dt, at::Device dev) {
  return at::detail::empty_cuda(shape, dt, dev, std::nullopt);
}
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* cuda_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
bool has_shape(const Tensor& t, std::initializer_list<int64_t> s) { return t.sizes() == at::IntArrayRef(s.begin(), s.size()); }

// What a forward pass saved for its gradient: hooks on saved tensors may have brought back another layout or device, and
// the kernels index these by the problem's sizes.
Tensor saved_as(const Tensor& t, at::ScalarType dt, int64_t n, at::Device dev, const char* msg) {
  require(t.scalar_type() == dt && t.numel() == n, msg);
  return as(t, dt, dev);
}

// float32 gradients as the features' type: bfloat16 ones in one launch, otherwise what the tensor library does
void as_features(const Tensor& g0, const Tensor* g1, at::ScalarType ft, Tensor* out0, Tensor* out1) {
  if (g0.scalar_type() == at::kFloat && ft == at::kBFloat16) {
    const at::Device dev = g0.device();
    if (out0) *out0 = fresh(g0.sizes(), ft, dev);
    if (out1) *out1 = fresh(g1->sizes(), ft, dev);
    check(chop_narrow_bf16(out0 ? g0.const_data_ptr<float>() : nullptr, out0 ? ptr(*out0) : nullptr, out0 ? g0.numel() : 0,
                           out1 ? g1->const_data_ptr<float>() : nullptr, out1 ? ptr(*out1) : nullptr, out1 ? g1->numel() : 0,
                           cuda_stream()),
          "chop_narrow_bf16");
    return;
  }
  if (out0) *out0 = g0.scalar_type() == ft ? g0 : g0.to(ft);
  if (out1) *out1 = g1->scalar_type() == ft ? *g1 : g1->to(ft);
}

// A node with the inputs that its gradient needs.  Backward passes from several threads can share a node, one of them
// releasing what another reads: both take the node's lock, as torch's own nodes do.
struct SavingNode : public Node {
  std::vector<SavedVariable> saved;
  void save(std::initializer_list<Tensor> ts) {
    saved.reserve(ts.size());
    for (const Tensor& t : ts) saved.emplace_back(t, /*is_output=*/false);
  }
  std::vector<Tensor> unpack() {
    std::lock_guard<std::mutex> lock(mutex_);
    std::vector<Tensor> ts;
    ts.reserve(saved.size());
    for (auto& s : saved) ts.push_back(s.unpack());
    return ts;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto& s : saved) s.reset_data();
  }
  bool wanted(size_t i) const { return task_should_compute_output(i); }
  // an upstream gradient that nothing defined counts as zeros, as in torch.autograd.Function
  variable_list apply(variable_list&& grads) final {
    return in_engine([&] { return gradient(grads[0].defined() ? grads[0] : input_metadata(0).zeros_like()); });
  }
  virtual variable_list gradient(const Tensor& grad) = 0;
};
template <typename N, typename... Ts>
std::shared_ptr<N> make_node(const Ts&... inputs) {
  std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
  n->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  return n;
}

// ---- cost volume family -------------------------------------------------------------------------------------
struct CvConf {
  int kind, reduce;
  int64_t groups;
  bool half_centor;
};
struct CvArgs {
  Tensor ref, src, depth, offsets, Rs, Ts;
  chop_cv_desc d;
  at::ScalarType real;
};

CvArgs cv_prepare(const CvConf& c, const Tensor& ref, const Tensor& src, const Tensor& depth, const Tensor& offsets,
                  const Tensor& Rs, const Tensor& Ts) {
  require(ref.is_cuda(), "cost volume ops run on CUDA tensors only (no CPU kernel is registered)");
  CvArgs a;
  const at::ScalarType dt = ref.scalar_type();
  a.d = chop_cv_desc{};
  a.d.dtype = chop_dtype_of(dt);
  a.real = real_of(dt);
  const at::Device dev = ref.device();
  a.ref = as(ref, dt, dev);
  a.src = as(src, dt, dev);
  a.depth = as(depth, a.real, dev);
  if (offsets.defined()) a.offsets = as(offsets, a.real, dev);
  a.Rs = as(Rs, a.real, dev);
  a.Ts = as(Ts, a.real, dev);
  require(a.ref.dim() == 4, "ref image must have rank 4");
  const int64_t B = a.ref.size(0), H = a.ref.size(1), W = a.ref.size(2), C = a.ref.size(3);
  require(a.src.dim() == 5 && has_shape(a.src, {B, a.src.size(1), H, W, C}),
          "src_images must have rank 5, and must compate to ref_image");
  const int64_t N = a.src.size(1);
  int64_t D;
  if (c.kind == CHOP_COST_VOLUME_V2) {
    require(a.depth.dim() == 4 && has_shape(a.depth, {B, H, W, a.depth.size(3)}),
            "depth_grid must have rank 4, and must compate to ref_image");
    D = a.depth.size(3);
  } else {
    require(has_shape(a.depth, {B, H, W, 1}), "base_plane must have rank 4, and must compate to ref_image");
    require(a.offsets.defined() && a.offsets.dim() == 2 && a.offsets.size(0) == B,
            "offsets must have rank 2, and must compate to ref_image");
    D = a.offsets.size(1);
  }
  require(has_shape(a.Rs, {B, N, 3, 3}), "Rs must have rank 4, and must compate to ref_image");
  require(has_shape(a.Ts, {B, N, 3}), "Ts must have rank 3, and must compate to ref_image");
  if (c.kind == CHOP_COST_VOLUME_V2 || c.kind == CHOP_COST_VOLUME_V3)
    require(c.groups >= 1 && C % c.groups == 0, "channels must be divisible by groups");
  if (c.kind == CHOP_COST_VOLUME_V3)   // cost_volume_kernels_v3.cc:110-111
    require(C / c.groups <= 8, "image_channels / groups_ less than MAX_SUBCHANNELS_SIZE(8)");
  a.d.kind = c.kind;
  a.d.reduce = c.reduce;
  a.d.half_centor = c.half_centor;
  a.d.groups = (int32_t)(c.groups ? c.groups : 1);
  a.d.B = B; a.d.H = a.d.Hs = H; a.d.W = a.d.Ws = W; a.d.C = C; a.d.D = D; a.d.N = N;
  return a;
}

int64_t cv_channels(const CvArgs& a) {
  return a.d.kind == CHOP_COST_VOLUME ? a.d.C : a.d.kind == CHOP_COST_VOLUME_V2 ? a.d.groups : 1;
}
int64_t cv_mask_channels(const CvArgs& a) {
  if (a.d.reduce == CHOP_REDUCE_MEAN) return 1;
  return a.d.kind == CHOP_COST_VOLUME_V3 ? 3 : cv_channels(a);   // v3 MIN: (view, reference group, source group)
}

struct CvNode : public SavingNode {
  CvConf conf;
  std::string name() const override { return "CostVolumeGrad"; }
  variable_list gradient(const Tensor& grad) override {
    variable_list out(6);
    const auto t = unpack();
    const CvArgs a = cv_prepare(conf, t[0], t[1], t[2], t[3], t[4], t[5]);
    c10::cuda::CUDAGuard guard(a.ref.device());
    const at::Device dev = a.ref.device();
    const int64_t voxels = a.d.B * a.d.H * a.d.W * a.d.D;
    const Tensor cg = as(grad, a.real, dev);
    require(cg.numel() == voxels * cv_channels(a), "cost_grad must have rank 5, and must compate to ref_image");
    const Tensor mask = saved_as(t[6], at::kInt, voxels * cv_mask_channels(a), dev, "cost_mask must be the int32 mask returned by the forward op");
    Tensor winners;
    if (t[7].defined())
      winners = saved_as(t[7], at::kByte, (int64_t)chop_cost_volume_saved_bytes(&a.d), dev, "the winners must be those that the forward op recorded");
    Tensor rg = fresh(a.ref.sizes(), a.real, dev);
    Tensor sg = fresh(a.src.sizes(), a.real, dev);
    Tensor dg = fresh(a.depth.sizes(), a.real, dev);
    check(chop_cost_volume_bwd_saved(&a.d, ptr(a.ref), ptr(a.src), ptr(a.depth), ptr(a.offsets), ptr(a.Rs), ptr(a.Ts),
                                     ptr(cg), static_cast<const int32_t*>(ptr(mask)), ptr(winners), ptr(rg), ptr(sg), ptr(dg),
                                     cuda_stream()),
          "chop_cost_volume_bwd");
    as_features(rg, &sg, a.ref.scalar_type(), wanted(0) ? &out[0] : nullptr, wanted(1) ? &out[1] : nullptr);
    out[2] = dg.sizes() == t[2].sizes() ? dg : dg.view_as(t[2]);
    return out;
  }
};

// (cost, cost_mask) of CostVolume / CostVolumeV2 / CostVolumeV3 / CostAggregate, differentiable in ref, src and depth
std::tuple<Tensor, Tensor> cost_op(int kind, const std::string& reduce, int64_t groups, bool half_centor, const Tensor& ref,
                                   const Tensor& src, const Tensor& depth, const std::optional<Tensor>& offsets,
                                   const Tensor& Rs, const Tensor& Ts) {
  return guarded([&] {
    if (reduce != "MEAN" && reduce != "MIN")
      throw std::invalid_argument("Invalid reduce method " + reduce + ". Supported types: MEAN, MIN");
    const CvConf conf{kind, reduce == "MIN" ? CHOP_REDUCE_MIN : CHOP_REDUCE_MEAN, groups, half_centor};
    const Tensor offs = offsets ? *offsets : Tensor();
    refuse_transforms({&ref, &src, &depth, &offs, &Rs, &Ts});
    const bool train = torch::autograd::compute_requires_grad(ref, src, depth, offs, Rs, Ts);
    Tensor cost, mask, saved;   // saved: for the gradient only
    {
      at::AutoDispatchBelowADInplaceOrView below;
      const CvArgs a = cv_prepare(conf, ref, src, depth, offs, Rs, Ts);
      const at::Device dev = a.ref.device();
      c10::cuda::CUDAGuard guard(dev);
      const chop_cv_desc& d = a.d;
      if (kind == CHOP_COST_AGGREGATE) {
        cost = fresh({d.B, d.H, d.W, d.D}, a.real, dev);
        mask = fresh({d.B, d.H, d.W, d.D}, at::kInt, dev);
      } else {
        cost = fresh({d.B, d.H, d.W, d.D, cv_channels(a)}, a.real, dev);
        mask = fresh({d.B, d.H, d.W, d.D, cv_mask_channels(a)}, at::kInt, dev);
      }
      if (train && kind == CHOP_COST_VOLUME_V3)
        if (const size_t n = chop_cost_volume_saved_bytes(&d)) saved = fresh({(int64_t)n}, at::kByte, dev);
      check(chop_cost_volume_fwd_save(&d, ptr(a.ref), ptr(a.src), ptr(a.depth), ptr(a.offsets), ptr(a.Rs), ptr(a.Ts),
                                      ptr(cost), static_cast<int32_t*>(ptr(mask)), ptr(saved), cuda_stream()),
            "chop_cost_volume_fwd");
    }
    if (train) {
      auto node = make_node<CvNode>(ref, src, depth, offs, Rs, Ts);
      node->conf = conf;
      node->save({ref, src, depth, offs, Rs, Ts, mask, saved});
      torch::autograd::set_history(cost, node);
    }
    return std::make_tuple(cost, mask);
  });
}

// ---- FeatureAggregate -----------------------------------------------------------------------------------------
struct FaArgs {
  Tensor src, base, offsets, Rs, Ts;
  chop_cv_desc d;
  at::ScalarType real;
};
FaArgs fa_prepare(bool half_centor, const Tensor& src, const Tensor& base, const Tensor& offsets, const Tensor& Rs,
                  const Tensor& Ts) {
  require(src.is_cuda(), "feature_aggregate runs on CUDA tensors only (no CPU kernel is registered)");
  FaArgs a;
  a.d = chop_cv_desc{};
  const at::ScalarType dt = src.scalar_type();
  a.d.dtype = chop_dtype_of(dt);
  a.real = real_of(dt);
  require(src.dim() == 5, "src image must have rank 5");
  const at::Device dev = src.device();
  a.src = as(src, dt, dev);
  a.base = as(base, a.real, dev);
  a.offsets = as(offsets, a.real, dev);
  a.Rs = as(Rs, a.real, dev);
  a.Ts = as(Ts, a.real, dev);
  const int64_t B = a.src.size(0), N = a.src.size(1);
  require(a.base.dim() == 4 && a.base.size(0) == B && a.base.size(3) == 1,
          "base_plane must have rank 4, and must compate to src_images");
  require(a.offsets.dim() == 2 && a.offsets.size(0) == B, "offsets must have rank 2, and must compate to src_images");
  require(has_shape(a.Rs, {B, N, 3, 3}), "Rs must have rank 4, and must compate to src_images");
  require(has_shape(a.Ts, {B, N, 3}), "Ts must have rank 3, and must compate to src_images");
  a.d.groups = 1;
  a.d.half_centor = half_centor;
  a.d.B = B; a.d.N = N; a.d.Hs = a.src.size(2); a.d.Ws = a.src.size(3); a.d.C = a.src.size(4);
  a.d.H = a.base.size(1); a.d.W = a.base.size(2); a.d.D = a.offsets.size(1);
  return a;
}
struct FaNode : public SavingNode {
  bool half_centor;
  std::string name() const override { return "FeatureAggregateGrad"; }
  variable_list gradient(const Tensor& grad) override {
    variable_list out(5);
    const auto t = unpack();
    const FaArgs a = fa_prepare(half_centor, t[0], t[1], t[2], t[3], t[4]);
    c10::cuda::CUDAGuard guard(a.src.device());
    const at::Device dev = a.src.device();
    const int64_t samples = a.d.B * a.d.H * a.d.W * a.d.D * a.d.N;
    const Tensor mg = as(grad, a.real, dev);
    require(mg.numel() == samples * a.d.C, "mapped_feature_grad must compate to the forward output");
    const Tensor mask = saved_as(t[5], at::kInt, samples, dev, "mapped_mask must be the int32 mask returned by the forward op");
    Tensor sg = fresh(a.src.sizes(), a.real, dev);
    Tensor bg = fresh(a.base.sizes(), a.real, dev);
    check(chop_feature_aggregate_bwd(&a.d, ptr(a.src), ptr(a.base), ptr(a.offsets), ptr(a.Rs), ptr(a.Ts), ptr(mg),
                                     static_cast<const int32_t*>(ptr(mask)), ptr(sg), ptr(bg), cuda_stream()),
          "chop_feature_aggregate_bwd");
    // gradients for src_images and base_plane only (reference: custom_helper_ops.py:192)
    const at::ScalarType ft = t[0].scalar_type(), bt = t[1].scalar_type();
    if (wanted(0)) as_features(sg, nullptr, ft, &out[0], nullptr);
    if (wanted(1)) out[1] = bt == a.real ? bg : bg.to(bt);
    return out;
  }
};
std::tuple<Tensor, Tensor> feature_aggregate(bool half_centor, const Tensor& src, const Tensor& base, const Tensor& offsets,
                                             const Tensor& Rs, const Tensor& Ts) {
  return guarded([&] {
    refuse_transforms({&src, &base, &offsets, &Rs, &Ts});
    Tensor mapped, mask;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      const FaArgs a = fa_prepare(half_centor, src, base, offsets, Rs, Ts);
      const at::Device dev = a.src.device();
      c10::cuda::CUDAGuard guard(dev);
      const chop_cv_desc& d = a.d;
      mapped = fresh({d.B, d.H, d.W, d.D, d.N, d.C}, a.real, dev);
      mask = fresh({d.B, d.H, d.W, d.D, d.N, 1}, at::kInt, dev);
      check(chop_feature_aggregate_fwd(&d, ptr(a.src), ptr(a.base), ptr(a.offsets), ptr(a.Rs), ptr(a.Ts), ptr(mapped),
                                       static_cast<int32_t*>(ptr(mask)), cuda_stream()),
            "chop_feature_aggregate_fwd");
    }
    if (torch::autograd::compute_requires_grad(src, base, offsets, Rs, Ts)) {
      auto node = make_node<FaNode>(src, base, offsets, Rs, Ts);
      node->half_centor = half_centor;
      node->save({src, base, offsets, Rs, Ts, mask});
      torch::autograd::set_history(mapped, node);
    }
    return std::make_tuple(mapped, mask);
  });
}

// ---- manifold convolution ----------------------------------------------------------------------------------------
using Ints = std::vector<int64_t>;
struct ScConf {
  bool transpose, dynamic_default;
  Ints output_size;   // transposed form: the fine grid
  int32_t strides[3], dilations[3];
};
struct ScArgs {
  Tensor images, filters, def, base;
  chop_sc_desc d;
  std::array<int64_t, 5> out_shape;
};

// Before a call that may take tensor-core kernels (bfloat16 and float32): raise if a kernel of an EARLIER call gave up a bounded
// wait on its MMA barrier.  Reads one int of pinned host memory (chop_umma_watch); only the first call per device does more.
void umma_watch(at::ScalarType dt) {
  if (dt != at::kBFloat16 && dt != at::kFloat) return;
  const int n = chop_umma_watch();
  if (n > 0)
    throw std::runtime_error("custom_helper_op: " + std::to_string(n) +
                             " tensor-core convolution wait(s) timed out on the device; results of the manifold-convolution "
                             "calls since the previous check are incomplete");
}

ScArgs sc_prepare(const ScConf& c, const Tensor& images, const Tensor& filters, const Tensor& def, const Tensor& base) {
  ScArgs a;
  a.d = chop_sc_desc{};
  require(images.is_cuda(), c.transpose ? "sparse_conv3d_transpose_fast runs on CUDA tensors only (no CPU kernel is registered)"
                                        : "sparse_conv3d_fast runs on CUDA tensors only (no CPU kernel is registered)");
  const at::ScalarType dt = images.scalar_type();
  a.d.dtype = chop_dtype_of(dt);
  const at::Device dev = images.device();
  require(filters.device() == dev && base.device() == dev, "filters and base_plane must be on the device of images");
  a.images = as(images, dt, dev);
  a.filters = filters.scalar_type() == dt ? filters.contiguous() : filters.to(dt).contiguous();
  a.def = as(def, dt, dev);
  a.base = base.contiguous();
  require(images.dim() == 5, "images must have rank 5");
  require(filters.dim() == 5, "filter must have rank 5");
  require(images.size(4) == filters.size(c.transpose ? 4 : 3), "images channel size wrong");
  chop_sc_desc& d = a.d;
  d.dynamic_default = c.dynamic_default;
  d.B = images.size(0);
  d.Cin = filters.size(3);
  d.Cout = filters.size(4);
  for (int i = 0; i < 3; ++i) {
    d.filter[i] = (int32_t)filters.size(i);
    d.strides[i] = c.strides[i];
    d.dilations[i] = c.dilations[i];
  }
  auto coarse = [&](int64_t n, int i) { return (n + d.strides[i] - 1) / d.strides[i]; };
  if (c.transpose) {
    // the forward convolution whose transpose is taken (sparse_conv3d_fast_op.cc:78-146): output_size is the fine grid
    d.H = c.output_size[0]; d.W = c.output_size[1]; d.D = c.output_size[2];
    require(images.size(1) == coarse(d.H, 0) && images.size(2) == coarse(d.W, 1) && images.size(3) == coarse(d.D, 2),
            "images shape and output_shape does not compate");
    a.out_shape = {d.B, d.H, d.W, d.D, d.Cin};
  } else {
    d.H = images.size(1); d.W = images.size(2); d.D = images.size(3);
    a.out_shape = {d.B, coarse(d.H, 0), coarse(d.W, 1), coarse(d.D, 2), d.Cout};
  }
  require(base.scalar_type() == at::kInt && has_shape(base, {d.B, d.H, d.W, 1}),
          "base_plane must have rank 4, and must compate to ref_image");
  return a;
}

struct ScNode : public SavingNode {
  ScConf conf;
  std::string name() const override { return conf.transpose ? "SparseConv3DTransposeFastGrad" : "SparseConv3DFastGrad"; }
  variable_list gradient(const Tensor& grad) override {
    variable_list out(4);
    const auto t = unpack();
    const ScArgs a = sc_prepare(conf, t[0], t[1], t[2], t[3]);
    const at::Device dev = a.images.device();
    const at::ScalarType dt = a.images.scalar_type(), wdt = real_of(dt);
    c10::cuda::CUDAGuard guard(dev);
    const Tensor og = as(grad, dt, dev);
    require(og.sizes() == at::IntArrayRef(a.out_shape), "out_grad must have rank 5, and must compate to ref_image");
    Tensor ig = fresh(a.images.sizes(), dt, dev);
    Tensor fg = fresh(a.filters.sizes(), wdt, dev);
    const size_t need = conf.transpose ? chop_sparse_conv3d_transpose_bwd_workspace_size(&a.d)
                                       : chop_sparse_conv3d_bwd_workspace_size(&a.d);
    const int64_t nbytes = (int64_t)std::max<size_t>(need, 16);
    Tensor ws = fresh({nbytes}, at::kByte, dev);
    umma_watch(dt);
    const int32_t* bp = static_cast<const int32_t*>(ptr(a.base));
    if (conf.transpose) {
      check(chop_sparse_conv3d_transpose_bwd(&a.d, ptr(a.images), ptr(a.filters), ptr(a.def), bp, ptr(og), ptr(ig), ptr(fg),
                                             ptr(ws), (size_t)nbytes, cuda_stream()),
            "chop_sparse_conv3d_transpose_bwd");
    } else {
      Tensor dg = fresh({}, wdt, dev);
      check(chop_sparse_conv3d_bwd(&a.d, ptr(a.images), ptr(a.filters), ptr(a.def), bp, ptr(og), ptr(ig), ptr(fg), ptr(dg),
                                   ptr(ws), (size_t)nbytes, cuda_stream()),
            "chop_sparse_conv3d_bwd");
      // the reference drops the default-value gradient unless dynamic_default (custom_helper_ops.py:284-286)
      if (conf.dynamic_default && wanted(2)) out[2] = dg.to(t[2].scalar_type());
    }
    if (wanted(0)) out[0] = ig;
    if (wanted(1)) as_features(fg, nullptr, t[1].scalar_type(), &out[1], nullptr);
    return out;
  }
};

// sparse_conv3d_fast (output_size absent) or sparse_conv3d_transpose_fast; `def` is a device scalar of the images' type
Tensor sparse_conv(const Tensor& images, const Tensor& filters, const Tensor& def, const Tensor& base, const Ints& strides,
                   const Ints& dilations, bool dynamic_default, const std::optional<Ints>& output_size) {
  return guarded([&] {
    refuse_transforms({&images, &filters, &def, &base});
    ScConf conf{output_size.has_value(), dynamic_default, output_size ? *output_size : Ints(), {}, {}};
    require(strides.size() == 3, "strides must be a vector have 3 element");
    require(dilations.size() == 3, "dilations must be a vector have 3 element");
    if (conf.transpose) require(conf.output_size.size() == 3, "output_shape must be an 1-D vector of (height, width, depth)");
    for (int i = 0; i < 3; ++i) {
      conf.strides[i] = (int32_t)strides[i];
      conf.dilations[i] = (int32_t)dilations[i];
      require(conf.strides[i] > 0, "strides must be positive");
    }
    Tensor out;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      const ScArgs a = sc_prepare(conf, images, filters, def, base);
      const at::Device dev = a.images.device();
      c10::cuda::CUDAGuard guard(dev);
      out = fresh(a.out_shape, a.images.scalar_type(), dev);
      umma_watch(a.images.scalar_type());
      const int32_t* bp = static_cast<const int32_t*>(ptr(a.base));
      if (conf.transpose)
        check(chop_sparse_conv3d_transpose_fwd(&a.d, ptr(a.images), ptr(a.filters), ptr(a.def), bp, ptr(out), cuda_stream()),
              "chop_sparse_conv3d_transpose_fwd");
      else
        check(chop_sparse_conv3d_fwd(&a.d, ptr(a.images), ptr(a.filters), ptr(a.def), bp, ptr(out), cuda_stream()),
              "chop_sparse_conv3d_fwd");
    }
    if (torch::autograd::compute_requires_grad(images, filters, def, base)) {
      auto node = make_node<ScNode>(images, filters, def, base);
      node->conf = std::move(conf);
      node->save({images, filters, def, base});
      torch::autograd::set_history(out, node);
    }
    return out;
  });
}

// ---- SparsePad ---------------------------------------------------------------------------------------------------
struct PadArgs {
  Tensor base;
  int32_t strides[3];
  std::array<int64_t, 5> coarse, fine;
  int dtype;
};
PadArgs pad_prepare(at::IntArrayRef shape, at::ScalarType dt, at::Device dev, const Tensor& base, const int32_t* strides) {
  PadArgs a;
  a.dtype = chop_dtype_of(dt);
  require(base.device() == dev, "base_plane must be on the device of images");
  a.base = base.contiguous();
  std::copy(shape.begin(), shape.end(), a.coarse.begin());
  std::copy(strides, strides + 3, a.strides);
  a.fine = {shape[0], shape[1] * strides[0], shape[2] * strides[1], shape[3] * strides[2], shape[4]};
  require(base.scalar_type() == at::kInt && has_shape(base, {a.fine[0], a.fine[1], a.fine[2], 1}),
          "base_plane must have rank 4, and must compate to ref_image");
  return a;
}
struct PadNode : public SavingNode {
  std::array<int64_t, 5> coarse;   // the gradient needs the images' shape and type only
  at::ScalarType dt;
  at::Device dev = at::kCPU;
  int32_t strides[3];
  std::string name() const override { return "SparsePadGrad"; }
  variable_list gradient(const Tensor& grad) override {
    variable_list out(2);
    const auto t = unpack();
    const PadArgs a = pad_prepare(coarse, dt, dev, t[0], strides);
    c10::cuda::CUDAGuard guard(dev);
    const Tensor og = as(grad, dt, dev);
    require(og.sizes() == at::IntArrayRef(a.fine), "out_grad must compate to the padded shape");
    Tensor ig = fresh(coarse, dt, dev);
    check(chop_sparse_pad_bwd(a.dtype, coarse[0], coarse[1], coarse[2], coarse[3], coarse[4], a.strides,
                              static_cast<const int32_t*>(ptr(a.base)), ptr(og), ptr(ig), cuda_stream()),
          "chop_sparse_pad_bwd");
    out[0] = ig;
    return out;
  }
};
Tensor sparse_pad(const Tensor& images, const Tensor& base, const Ints& strides) {
  return guarded([&] {
    refuse_transforms({&images, &base});
    require(images.is_cuda(), "sparse_pad runs on CUDA tensors only");
    require(images.dim() == 5, "images must have rank 5");
    require(strides.size() == 3, "strides must be a vector have 3 element");
    const int32_t s[3] = {(int32_t)strides[0], (int32_t)strides[1], (int32_t)strides[2]};
    Tensor out;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      const Tensor im = images.contiguous();
      const PadArgs a = pad_prepare(im.sizes(), im.scalar_type(), im.device(), base, s);
      c10::cuda::CUDAGuard guard(im.device());
      out = fresh(a.fine, im.scalar_type(), im.device());
      check(chop_sparse_pad_fwd(a.dtype, a.coarse[0], a.coarse[1], a.coarse[2], a.coarse[3], a.coarse[4], a.strides, ptr(im),
                                static_cast<const int32_t*>(ptr(a.base)), ptr(out), cuda_stream()),
            "chop_sparse_pad_fwd");
    }
    if (torch::autograd::compute_requires_grad(images, base)) {
      auto node = make_node<PadNode>(images, base);
      std::copy(images.sizes().begin(), images.sizes().end(), node->coarse.begin());
      node->dt = images.scalar_type();
      node->dev = images.device();
      std::copy(s, s + 3, node->strides);
      node->save({base});
      torch::autograd::set_history(out, node);
    }
    return out;
  });
}

}  // namespace

// Allocation, launch (which waits while the stream's queue is full) and the first chop_umma_watch() run without the
// interpreter lock, as the ctypes calls of the raw functions do; what needs the lock takes it (check, guarded, hooks).
PYBIND11_MODULE(_torch_glue, m) {
  using unlocked = py::call_guard<py::gil_scoped_release>;
  m.def("cost_op", &cost_op, unlocked());
  m.def("feature_aggregate", &feature_aggregate, unlocked());
  m.def("sparse_conv", &sparse_conv, unlocked());
  m.def("sparse_pad", &sparse_pad, unlocked());
}
