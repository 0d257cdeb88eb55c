// Native host path of the Python operators: eligibility checks, output and workspace allocation, the C-ABI call and the
// autograd node, in one call from Python.
//
// What bounds a window or ViT-at-224 training step is the host, not the GPU: at (512,3,49,32) fp16 with a bias the kernels
// take 57 us, while the same step through a Python autograd.Function with ctypes took 160 us (argument lists, a Python
// frame on the autograd thread, the GIL hand-over to it).  Here a forward is one C call, and the backward node runs on the
// autograd thread without Python.
//
// Every function returns None when the call is not the plain case it covers (tensor subclasses, function transforms,
// dispatch modes, a wrong shape, dtype or device): the Python operators then take their general path, which also raises
// the errors.  Layout rules are those of elsa_b200/attention.py: operands are read in place when the D axis is
// contiguous and rows start on 16-byte boundaries, otherwise copied first; `out` follows q's axis order in memory.
#define PY_SSIZE_T_CLEAN
#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>

#include "../../include/elsa_b200.h"

namespace {

using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// the C ABI, by address: the library itself is loaded by elsa_b200/_lib.py (which also honours ELSA_B200_LIB)
decltype(&elsa_forward_workspace_bytes) f_fwd_ws = nullptr;
decltype(&elsa_twopass_forward) f_fwd = nullptr;
decltype(&elsa_twopass_forward_strided) f_fwd_strided = nullptr;
decltype(&elsa_backward_workspace_bytes) f_bwd_ws = nullptr;
decltype(&elsa_twopass_backward) f_bwd = nullptr;
decltype(&elsa_twopass_backward_strided) f_bwd_strided = nullptr;
decltype(&elsa_strerror) f_strerror = nullptr;
decltype(&elsa_last_cuda_error) f_last_cuda_error = nullptr;

void check_status(int rc, const char* what) {
  if (rc == ELSA_OK) return;
  std::string msg = std::string(what) + ": " + f_strerror(rc);
  if (rc == ELSA_ERR_CUDA) msg += " [cudaError " + std::to_string(f_last_cuda_error()) + "]";
  if (rc == ELSA_ERR_INVALID_ARGUMENT || rc == ELSA_ERR_UNSUPPORTED) TORCH_CHECK_VALUE(false, msg);
  throw std::runtime_error(msg);
}

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? ELSA_F32 : t == at::kHalf ? ELSA_F16 : t == at::kBFloat16 ? ELSA_BF16 : -1;
}

struct Call {                 // the problem, as the C ABI wants it
  int batch, heads, n, d, dt, sdt, causal, part_width, q_chunk;
};

struct View {                 // a [B, H, N, D] operand: first element and {batch, head, row} element strides
  char* p = nullptr;
  int64_t st[3] = {0, 0, 0};
};

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

char* data_of(const at::Tensor& t) { return static_cast<char*>(const_cast<void*>(t.const_data_ptr())); }

// fills *v; true when the kernels can read `t` in place
bool in_place_view(const at::Tensor& t, View* v) {
  const auto sz = t.sizes();
  const auto st = t.strides();
  v->p = data_of(t);
  for (int i = 0; i < 3; ++i) v->st[i] = sz[i] > 1 ? st[i] : sz[3] * 8;   // (a size-1 axis may have any stride)
  if ((sz[3] > 1 && st[3] != 1) || !aligned16(v->p)) return false;
  return ((v->st[0] | v->st[1] | v->st[2]) % 8 == 0) && v->st[0] > 0 && v->st[1] > 0 && v->st[2] >= sz[3];
}

at::Tensor aligned(const at::Tensor& t) {
  at::Tensor c = t.contiguous();
  return aligned16(c.const_data_ptr()) ? c : c.clone();
}

at::Tensor new_tensor(at::IntArrayRef sizes, const at::Tensor& like, at::ScalarType dtype) {
  return at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt);
}

// an uninitialised [B, H, N, D] tensor in row-major [B, N, H, D] memory
at::Tensor new_bnhd(const at::Tensor& like, int64_t b, int64_t h, int64_t n, int64_t d) {
  return at::detail::empty_strided_cuda({b, h, n, d}, {n * h * d, d, h * d, 1}, like.scalar_type(), like.device());
}

// an uninitialised tensor of t's shape whose axis order in memory follows t
at::Tensor new_like_layout(const at::Tensor& t, const View& v) {
  if (t.size(1) > 1 && t.size(2) > 1 && v.st[1] < v.st[2]) return new_bnhd(t, t.size(0), t.size(1), t.size(2), t.size(3));
  return new_tensor(t.sizes(), t, t.scalar_type());
}

bool plain(const at::Tensor& t) {
  // wrappers of function transforms, Python-dispatched and functional tensors keep to the general path
  constexpr c10::DispatchKeySet special({c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::FuncTorchBatched,
                                         c10::DispatchKey::FuncTorchVmapMode, c10::DispatchKey::Python,
                                         c10::DispatchKey::Functionalize, c10::DispatchKey::Batched});
  // (a forward-mode tangent too: the autograd functions of the general path refuse it, a result without one would be wrong)
  return t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has_any(special) && !t._fw_grad(/*level=*/0).defined();
}

// dispatch modes, and torch.jit.trace: the general path's autograd functions are recorded as operations of the graph, while
// the output of a native call would be recorded as a constant
bool modes_active() { return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::tracer::impl::is_dispatch_enabled(); }

struct Bias {
  at::Tensor t;               // fp32, contiguous: [B|1, H|1, N, N] up to leading axes of size 1
  int64_t sb = 0, sh = 0, sq = 0, sk = 0;
  const float* ptr() const { return t.defined() ? t.const_data_ptr<float>() : nullptr; }
};

// Called below autograd.  A contiguous fp32 bias is used as it is: no view is made of it, so its version counter is the
// caller's, and a change between forward and backward is found.
bool canonical_bias(const at::Tensor& bias, const Call& c, c10::Device dev, Bias* out) {
  if (!bias.defined()) return true;
  const int64_t dim = bias.dim(), n = c.n;
  if (bias.device() != dev || dim < 2 || dim > 4 || bias.size(dim - 2) != n || bias.size(dim - 1) != n) return false;
  const int64_t lh = dim >= 3 ? bias.size(dim - 3) : 1, lb = dim == 4 ? bias.size(0) : 1;
  if ((lh != 1 && lh != c.heads) || (lb != 1 && lb != c.batch)) return false;
  out->t = (bias.scalar_type() == at::kFloat ? bias : bias.to(at::kFloat)).contiguous();
  out->sb = lb == 1 ? 0 : lh * n * n;
  out->sh = lh == 1 ? 0 : n * n;
  out->sq = n;
  out->sk = 1;
  return true;
}

int64_t padded_rows(const Call& c) { return (static_cast<int64_t>(c.batch) * c.heads * c.n + 63) / 64 * 64; }

c10::DataPtr workspace(int64_t bytes) { return c10::cuda::CUDACachingAllocator::get()->allocate(static_cast<size_t>(bytes)); }

// row_m and row_z in one allocation, the second at a 256-byte boundary
at::Tensor new_state(const Call& c, const at::Tensor& like) { return new_tensor({2 * padded_rows(c)}, like, at::kFloat); }

void run_forward(const View (&in)[3], const View& out, bool strided, const Bias& bias, const at::Tensor& state, const Call& c, c10::Device dev) {
  const int64_t need = f_fwd_ws(c.dt, c.sdt, c.batch, c.heads, c.n, c.d, bias.t.defined(), c.causal, c.part_width, c.q_chunk, 0u);
  TORCH_CHECK_VALUE(need >= 0, "elsa_b200: unsupported problem size for the forward");
  const int64_t bytes = std::max<int64_t>(need, 256);
  c10::cuda::CUDAGuard guard(dev);
  c10::DataPtr ws = workspace(bytes);
  float* rm = state.defined() ? state.mutable_data_ptr<float>() : nullptr;
  float* rz = rm ? rm + padded_rows(c) : nullptr;
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int rc =
      strided ? f_fwd_strided(in[0].p, in[1].p, in[2].p, in[0].st, in[1].st, in[2].st, bias.ptr(), bias.sb, bias.sh, bias.sq, bias.sk,
                              out.p, out.st, rm, rz, ws.get(), bytes, c.dt, c.sdt, c.batch, c.heads, c.n, c.d, c.causal,
                              c.part_width, c.q_chunk, 0u, stream)
              : f_fwd(in[0].p, in[1].p, in[2].p, bias.ptr(), bias.sb, bias.sh, bias.sq, bias.sk, out.p, rm, rz, ws.get(), bytes,
                      c.dt, c.sdt, c.batch, c.heads, c.n, c.d, c.causal, c.part_width, c.q_chunk, 0u, stream);
  check_status(rc, "elsa_twopass_forward");
}

// t: q, k, v, out, dout, dq, dk, dv
void run_backward(const View (&t)[8], bool strided, const Bias& bias, const at::Tensor& dbias, const at::Tensor& state, const Call& c,
                  c10::Device dev) {
  const unsigned flags = at::globalContext().deterministicAlgorithms() ? ELSA_FLAG_REPEATABLE : 0u;
  const int64_t need = f_bwd_ws(c.dt, c.batch, c.heads, c.n, c.d, bias.t.defined(), c.causal, flags);
  TORCH_CHECK_VALUE(need >= 0, "elsa_b200: unsupported problem size for the backward");
  const int64_t bytes = std::max<int64_t>(need, 256);
  c10::DataPtr ws = workspace(bytes);
  const float* rm = state.const_data_ptr<float>();
  const float* rz = rm + padded_rows(c);
  float* db = dbias.defined() ? dbias.mutable_data_ptr<float>() : nullptr;
  const int64_t ds[4] = {db ? bias.sb : 0, db ? bias.sh : 0, db ? bias.sq : 0, db ? bias.sk : 0};
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  int rc;
  if (strided) {
    int64_t st[24];
    for (int i = 0; i < 8; ++i)
      for (int j = 0; j < 3; ++j) st[3 * i + j] = t[i].st[j];
    rc = f_bwd_strided(t[0].p, t[1].p, t[2].p, t[3].p, t[4].p, st, rm, rz, bias.ptr(), bias.sb, bias.sh, bias.sq, bias.sk, t[5].p,
                       t[6].p, t[7].p, db, ds[0], ds[1], ds[2], ds[3], ws.get(), bytes, c.dt, c.batch, c.heads, c.n, c.d,
                       c.causal, flags, stream);
  } else {
    rc = f_bwd(t[0].p, t[1].p, t[2].p, t[3].p, t[4].p, rm, rz, bias.ptr(), bias.sb, bias.sh, bias.sq, bias.sk, t[5].p, t[6].p,
               t[7].p, db, ds[0], ds[1], ds[2], ds[3], ws.get(), bytes, c.dt, c.batch, c.heads, c.n, c.d, c.causal, flags, stream);
  }
  check_status(rc, "elsa_twopass_backward");
}

// q, k, v (and out, dout) as the kernels will see them, copied first where they have to be; true when the strided entry
// points are needed
template <size_t N>
bool pick_layouts(std::array<at::Tensor, N>& t, View* v) {
  bool strided = false;
  for (auto& x : t) strided = strided || !x.is_contiguous();
  if (strided && t[0].size(3) % 8 == 0) {
    strided = false;
    for (size_t i = 0; i < N; ++i) {
      if (!in_place_view(t[i], &v[i])) {
        t[i] = aligned(t[i]);
        in_place_view(t[i], &v[i]);
      }
      strided = strided || !t[i].is_contiguous();
    }
    if (strided) return true;
  }
  for (size_t i = 0; i < N; ++i) {
    t[i] = aligned(t[i]);
    in_place_view(t[i], &v[i]);
  }
  return false;
}

// the three views of a contiguous packed [B, N, 3, H, D] tensor
void packed_views(char* base, const Call& c, int64_t esize, View* v) {
  const int64_t hd = static_cast<int64_t>(c.heads) * c.d;
  for (int i = 0; i < 3; ++i) {
    v[i].p = base + i * hd * esize;
    v[i].st[0] = c.n * 3 * hd;
    v[i].st[1] = c.d;
    v[i].st[2] = 3 * hd;
  }
}

void bnhd_view(char* base, const Call& c, View* v) {
  const int64_t hd = static_cast<int64_t>(c.heads) * c.d;
  v->p = base;
  v->st[0] = c.n * hd;
  v->st[1] = c.d;
  v->st[2] = hd;
}

// A saved tensor as the backward may use it: saved-tensor hooks may return the values in another memory layout (a copy
// built from the sizes alone, an unaligned slice), so nothing but the values is taken for granted.
void check_unpacked(const at::Tensor& t, at::IntArrayRef sizes, at::ScalarType dtype, c10::Device dev) {
  TORCH_CHECK(t.defined() && plain(t) && t.device() == dev && t.scalar_type() == dtype && t.sizes() == sizes,
              "a saved tensor of the attention came back from its unpack hook with another shape, dtype or device");
}

// what a backward needs beside the saved tensors
struct BackwardPlan {
  Call c{};
  bool packed = false, bias_grad = false;
  at::ScalarType dtype = at::kFloat, bias_dtype = at::kFloat, saved_bias_dtype = at::kFloat;
  std::vector<int64_t> bias_sizes, saved_bias_sizes;

  // the same as plain numbers and back, for compiled autograd
  std::vector<int64_t> numbers() const {
    std::vector<int64_t> x{c.batch, c.heads, c.n, c.d, c.dt, c.sdt, c.causal, c.part_width, c.q_chunk, packed, bias_grad,
                           static_cast<int64_t>(dtype), static_cast<int64_t>(bias_dtype), static_cast<int64_t>(saved_bias_dtype)};
    for (const auto* sizes : {&bias_sizes, &saved_bias_sizes}) {
      x.push_back(static_cast<int64_t>(sizes->size()));
      x.insert(x.end(), sizes->begin(), sizes->end());
    }
    return x;
  }
  static BackwardPlan of_numbers(const std::vector<int64_t>& x) {
    BackwardPlan p;
    size_t i = 0;
    for (int* f : {&p.c.batch, &p.c.heads, &p.c.n, &p.c.d, &p.c.dt, &p.c.sdt, &p.c.causal, &p.c.part_width, &p.c.q_chunk}) *f = static_cast<int>(x.at(i++));
    p.packed = x.at(i++) != 0;
    p.bias_grad = x.at(i++) != 0;
    for (at::ScalarType* f : {&p.dtype, &p.bias_dtype, &p.saved_bias_dtype}) *f = static_cast<at::ScalarType>(x.at(i++));
    for (auto* sizes : {&p.bias_sizes, &p.saved_bias_sizes}) {
      sizes->resize(x.at(i++));
      for (int64_t& n : *sizes) n = x.at(i++);
    }
    return p;
  }

  // packed: q is the packed tensor, k and v stay undefined, bias is the one in fp32; else bias is the caller's (a 16-bit or
  // expanded bias is kept as it is, and converted again by the backward)
  struct Saved { at::Tensor q, k, v, out, state, bias; };

  variable_list gradients(Saved s, at::Tensor go) const {
    variable_list result(packed ? 2 : 4);
    const int64_t B = c.batch, H = c.heads, N = c.n, D = c.d;
    const std::array<int64_t, 5> packed_sizes{B, N, 3, H, D};
    const std::array<int64_t, 4> sizes{B, H, N, D};
    const c10::Device dev = go.device();
    check_unpacked(s.q, packed ? at::IntArrayRef(packed_sizes) : at::IntArrayRef(sizes), dtype, dev);
    check_unpacked(s.out, sizes, dtype, dev);
    check_unpacked(s.state, {2 * padded_rows(c)}, at::kFloat, dev);
    const at::Tensor state = aligned(s.state);
    Bias bias;
    if (!saved_bias_sizes.empty()) {
      check_unpacked(s.bias, saved_bias_sizes, saved_bias_dtype, dev);
      canonical_bias(s.bias, c, dev, &bias);
    }
    if (go.scalar_type() != dtype) go = go.to(dtype);
    c10::cuda::CUDAGuard guard(dev);
    at::Tensor dbias;
    if (bias_grad) {
      // Sums over a broadcast axis and pairs that the causal rule leaves out need zeros.  Otherwise the kernels store every
      // element once, and clearing the tensor first is one more pass over it (537 MB at (1,8,4096,64)).
      const bool summed = (bias.sb == 0 && c.batch > 1) || (bias.sh == 0 && c.heads > 1);
      dbias = new_tensor(bias_sizes, go, at::kFloat);
      if (summed || c.causal) dbias.zero_();
    }
    View t[8];
    if (packed) {
      if (!in_place_view(go, &t[4])) {
        go = aligned(go);
        in_place_view(go, &t[4]);
      }
      const at::Tensor q = aligned(s.q);
      if (!in_place_view(s.out, &t[3])) {
        s.out = aligned(s.out);
        in_place_view(s.out, &t[3]);
      }
      result[0] = new_tensor(q.sizes(), q, dtype);
      packed_views(data_of(q), c, q.element_size(), &t[0]);
      packed_views(data_of(result[0]), c, q.element_size(), &t[5]);
      run_backward(t, true, bias, dbias, state, c, dev);
    } else {
      check_unpacked(s.k, sizes, dtype, dev);
      check_unpacked(s.v, sizes, dtype, dev);
      std::array<at::Tensor, 5> in{s.q, s.k, s.v, s.out, go};
      const bool strided = pick_layouts(in, t);
      for (int i = 0; i < 3; ++i) {
        result[i] = strided ? new_like_layout(in[i], t[i]) : new_tensor(sizes, go, dtype);
        in_place_view(result[i], &t[5 + i]);
      }
      run_backward(t, strided, bias, dbias, state, c, dev);
    }
    if (bias_grad) {
      result.back() = dbias.scalar_type() == bias_dtype ? dbias : dbias.to(bias_dtype);
    }
    return result;
  }
};

struct AttentionBackward : public torch::autograd::Node {
  BackwardPlan plan;
  SavedVariable q_, k_, v_, out_, state_, bias_;    // see BackwardPlan::Saved

  std::string name() const override { return plan.packed ? "TwopassAttentionQkvpackedBackward" : "TwopassAttentionBackward"; }

  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q_, &k_, &v_, &out_, &state_, &bias_}) s->reset_data();
  }

  BackwardPlan::Saved unpack() {
    return {q_.unpack(), k_.unpack(), v_.unpack(), out_.unpack(shared_from_this()), state_.unpack(), bias_.unpack()};
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return variable_list(plan.packed ? 2 : 4);
    // Unpacking runs the user's hooks, with autograd in force: a checkpoint repeats the forward in there, and the repeated
    // forward has to record and save what the first one did.
    BackwardPlan::Saved s = unpack();
    at::AutoDispatchBelowADInplaceOrView below;
    return plan.gradients(std::move(s), std::move(grads[0]));
  }

  // Compiled autograd: the node is one opaque call of its graph, on the saved tensors and the plan.
  void compiled_args(torch::dynamo::autograd::CompiledNodeArgs& args) const override {
    args.collect(plan.numbers());
    for (const SavedVariable* s : {&q_, &k_, &v_, &state_, &bias_}) args.collect(*s, false);
    args.collect(out_, true);
  }

  variable_list apply_with_saved(const variable_list& grads, torch::dynamo::autograd::SwapSavedVariables& saved) override {
    SavedVariable* const all[] = {&q_, &k_, &v_, &state_, &bias_, &out_};
    for (SavedVariable* s : all) saved.before(*s);
    BackwardPlan::Saved s = unpack();
    torch::dynamo::autograd::PackedArgs packed;
    std::vector<at::TypePtr> schema;
    auto add = [&](const auto& x) {
      packed.pack(x);
      schema.emplace_back(torch::dynamo::autograd::IValuePacker<std::decay_t<decltype(x)>>::packed_type());
    };
    add(plan.numbers());
    for (const at::Tensor* t : {&s.q, &s.k, &s.v, &s.out, &s.state, &s.bias}) add(*t);
    const auto& compiler = torch::dynamo::autograd::getPyCompilerInterface();
    const std::string fn = compiler->bind_function(saved.get_py_compiler(), name(), &call_packed, schema, /*is_custom_function=*/true, /*is_traceable=*/false);
    variable_list result = compiler->call_function(saved.get_py_compiler(), "apply_functional", fn, grads, packed.vec(), output_metadata());
    for (SavedVariable* s : all) saved.after(*s);
    return result;
  }

  static variable_list call_packed(const variable_list& grads, const std::vector<c10::IValue>& values) {
    torch::dynamo::autograd::PackedArgs packed(values);
    const BackwardPlan plan = BackwardPlan::of_numbers(packed.unpack<std::vector<int64_t>>());
    BackwardPlan::Saved s;
    for (at::Tensor* t : {&s.q, &s.k, &s.v, &s.out, &s.state, &s.bias}) *t = packed.unpack<at::Tensor>();
    if (!grads[0].defined()) return variable_list(plan.packed ? 2 : 4);
    at::AutoDispatchBelowADInplaceOrView below;
    return plan.gradients(std::move(s), grads[0]);
  }

  // shape, type and device of every input of the forward that gets a gradient
  c10::IValue output_metadata() const {
    return torch::dynamo::autograd::IValuePacker<std::vector<std::optional<torch::autograd::InputMetadata>>>::pack(
        torch::dynamo::autograd::get_input_metadata(next_edges()));
  }
};

bool fill_call(Call* c, const at::Tensor& q, int64_t b, int64_t h, int64_t n, int64_t d) {
  c->dt = dtype_code(q.scalar_type());
  if (c->dt < 0 || b <= 0 || h <= 0 || n <= 0 || d <= 0 || d > 128 || b > 65535 || h > 65535 || b * h > 65535 || n >= (1 << 30)) return false;
  c->batch = static_cast<int>(b);
  c->heads = static_cast<int>(h);
  c->n = static_cast<int>(n);
  c->d = static_cast<int>(d);
  if (c->sdt < 0) c->sdt = c->dt;
  return true;
}

template <typename... V>
std::shared_ptr<AttentionBackward> new_node(const Call& c, bool packed, const at::Tensor& bias, const Bias& canon, const V&... inputs) {
  std::shared_ptr<AttentionBackward> node(new AttentionBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(inputs..., bias));
  BackwardPlan& p = node->plan;
  p.c = c;
  p.packed = packed;
  p.dtype = c.dt == ELSA_F32 ? at::kFloat : c.dt == ELSA_F16 ? at::kHalf : at::kBFloat16;
  if (bias.defined()) {
    const at::Tensor& saved = packed ? canon.t : bias;
    p.bias_grad = bias.requires_grad();
    p.bias_dtype = bias.scalar_type();
    p.bias_sizes = bias.sizes().vec();
    p.saved_bias_dtype = saved.scalar_type();
    p.saved_bias_sizes = saved.sizes().vec();
    node->bias_ = SavedVariable(saved, false);
  }
  return node;
}

// out of the unpacked operator, or an undefined tensor when the call is not covered
at::Tensor attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& bias, Call c, bool train) {
  if (q.dim() != 4 || q.sizes() != k.sizes() || q.sizes() != v.sizes() || !plain(q) || !plain(k) || !plain(v) ||
      k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type() || k.device() != q.device() || v.device() != q.device() ||
      (bias.defined() && !plain(bias)) || modes_active() || !fill_call(&c, q, q.size(0), q.size(1), q.size(2), q.size(3)))
    return {};
  const bool record = train && at::GradMode::is_enabled() &&
                      (q.requires_grad() || k.requires_grad() || v.requires_grad() || (bias.defined() && bias.requires_grad()));
  Bias canon;
  std::array<at::Tensor, 3> in{q, k, v};
  at::Tensor out, state;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (!canonical_bias(bias, c, q.device(), &canon)) return {};
    View t[3], o;
    const bool strided = pick_layouts(in, t);
    out = strided ? new_like_layout(in[0], t[0]) : new_tensor(q.sizes(), q, q.scalar_type());
    in_place_view(out, &o);
    if (record) state = new_state(c, q);
    run_forward(t, o, strided, canon, state, c, q.device());
  }
  if (record) {
    auto node = new_node(c, false, bias, canon, q, k, v);
    node->q_ = SavedVariable(in[0], false);
    node->k_ = SavedVariable(in[1], false);
    node->v_ = SavedVariable(in[2], false);
    node->state_ = SavedVariable(state, false);
    torch::autograd::set_history(out, node);
    node->out_ = SavedVariable(out, true);
  }
  return out;
}

// the same on a packed [B, N, 3, H, D] tensor; out is a [B, H, N, D] tensor in [B, N, H, D] memory
at::Tensor attention_packed(const at::Tensor& qkv, const at::Tensor& bias, Call c, bool train) {
  if (qkv.dim() != 5 || qkv.size(2) != 3 || !plain(qkv) || !qkv.is_contiguous() || qkv.size(4) % 8 != 0 || (bias.defined() && !plain(bias)) ||
      modes_active() || !fill_call(&c, qkv, qkv.size(0), qkv.size(3), qkv.size(1), qkv.size(4)) || !aligned16(qkv.const_data_ptr()))
    return {};
  const bool record = train && at::GradMode::is_enabled() && (qkv.requires_grad() || (bias.defined() && bias.requires_grad()));
  Bias canon;
  at::Tensor out, state;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (!canonical_bias(bias, c, qkv.device(), &canon)) return {};
    out = new_bnhd(qkv, c.batch, c.heads, c.n, c.d);
    View in[3], o;
    packed_views(data_of(qkv), c, qkv.element_size(), in);
    bnhd_view(data_of(out), c, &o);
    if (record) state = new_state(c, qkv);
    run_forward(in, o, true, canon, state, c, qkv.device());
  }
  if (record) {
    auto node = new_node(c, true, bias, canon, qkv);
    node->q_ = SavedVariable(qkv, false);
    node->state_ = SavedVariable(state, false);
    torch::autograd::set_history(out, node);
    node->out_ = SavedVariable(out, true);
  }
  return out;
}

// ---- Python -----------------------------------------------------------------------------------
// (positional arguments only: the Python operators resolve the keywords)

bool get_tensor(PyObject* o, at::Tensor* t) {
  if (o == Py_None) return true;
  if (!THPVariable_CheckExact(o)) return false;
  *t = THPVariable_Unpack(o);
  return true;
}

bool get_call(PyObject* const* a, Call* c) {          // causal, summary dtype code, part_width, q_chunk
  const int causal = PyObject_IsTrue(a[0]);
  if (causal < 0) return false;
  c->causal = causal;
  c->sdt = static_cast<int>(PyLong_AsLong(a[1]));
  c->part_width = static_cast<int>(PyLong_AsLong(a[2]));
  c->q_chunk = static_cast<int>(PyLong_AsLong(a[3]));
  return !PyErr_Occurred();
}

struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

// attention(q, k, v, bias, causal, summary, part_width, q_chunk, train)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  at::Tensor q, k, v, bias, out;
  Call c{};
  TORCH_CHECK_TYPE(n == 9, "attention takes 9 arguments");
  if (!get_call(a + 4, &c)) return nullptr;
  if (!get_tensor(a[0], &q) || !get_tensor(a[1], &k) || !get_tensor(a[2], &v) || !get_tensor(a[3], &bias) || !q.defined() || !k.defined() || !v.defined())
    Py_RETURN_NONE;
  {
    NoGil no_gil;
    out = attention(q, k, v, bias, c, a[8] == Py_True);
  }
  if (!out.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// attention_packed(qkv, bias, causal, summary, part_width, q_chunk, train)
PyObject* py_attention_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  at::Tensor qkv, bias, out;
  Call c{};
  TORCH_CHECK_TYPE(n == 7, "attention_packed takes 7 arguments");
  if (!get_call(a + 2, &c)) return nullptr;
  if (!get_tensor(a[0], &qkv) || !get_tensor(a[1], &bias) || !qkv.defined()) Py_RETURN_NONE;
  {
    NoGil no_gil;
    out = attention_packed(qkv, bias, c, a[6] == Py_True);
  }
  if (!out.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind({name: address}): the C ABI of the loaded library
PyObject* py_bind(PyObject*, PyObject* d) {
  HANDLE_TH_ERRORS
  auto at_name = [&](const char* name) -> void* {
    PyObject* o = PyDict_GetItemString(d, name);
    TORCH_CHECK_VALUE(o != nullptr, "missing address of ", name);
    return PyLong_AsVoidPtr(o);
  };
  f_fwd_ws = reinterpret_cast<decltype(f_fwd_ws)>(at_name("elsa_forward_workspace_bytes"));
  f_fwd = reinterpret_cast<decltype(f_fwd)>(at_name("elsa_twopass_forward"));
  f_fwd_strided = reinterpret_cast<decltype(f_fwd_strided)>(at_name("elsa_twopass_forward_strided"));
  f_bwd_ws = reinterpret_cast<decltype(f_bwd_ws)>(at_name("elsa_backward_workspace_bytes"));
  f_bwd = reinterpret_cast<decltype(f_bwd)>(at_name("elsa_twopass_backward"));
  f_bwd_strided = reinterpret_cast<decltype(f_bwd_strided)>(at_name("elsa_twopass_backward_strided"));
  f_strerror = reinterpret_cast<decltype(f_strerror)>(at_name("elsa_strerror"));
  f_last_cuda_error = reinterpret_cast<decltype(f_last_cuda_error)>(at_name("elsa_last_cuda_error"));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention)), METH_FASTCALL, nullptr},
    {"attention_packed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention_packed)), METH_FASTCALL, nullptr},
    {"bind", py_bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&kModule);
  if (m && PyModule_AddStringConstant(m, "torch_version", ELSA_TORCH_VERSION) < 0) Py_CLEAR(m);
  return m;
}
