// The host side of the two ops: argument canonicalisation, allocation from torch's caching allocator, the C-ABI calls
// and autograd, as one Python extension.
//
// The same steps in Python -- descriptor structs over ctypes, a Python autograd Function, a dozen small tensor calls --
// took about 65 us per call, which is what a call on a small pair tensor costs in all (its kernels take 10).  Here a call
// without gradients goes straight to the library, and the backward runs on autograd's thread without the interpreter.
//
// Semantics follow the reference's public wrappers (geometric_nn_ops_torch/triangle/_triattn.py:23-106, _trimul.py:39-88).
// The library is reached through function pointers taken from the one that the ctypes binding loaded.
#include <ATen/autocast_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <initializer_list>
#include <optional>
#include <vector>

#include "../../include/tri_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

struct Api {
  decltype(&tri_last_error) last_error;
  decltype(&tri_last_path) last_path;
  decltype(&tri_ws_status) ws_status;
  decltype(&tri_attn_ws_bytes) attn_ws_bytes;
  decltype(&tri_attn_fwd) attn_fwd;
  decltype(&tri_attn_bwd) attn_bwd;
  decltype(&tri_attn_project_bias) attn_project_bias;
  decltype(&tri_gate_mul) gate_mul;
  decltype(&tri_gated_linear_after) gated_linear_after;
  decltype(&tri_mul_saved_bytes) mul_saved_bytes;
  decltype(&tri_mul_ws_bytes) mul_ws_bytes;
  decltype(&tri_mul_fwd) mul_fwd;
  decltype(&tri_mul_fwd_residual) mul_fwd_residual;
  decltype(&tri_mul_bwd) mul_bwd;
} api;

void bind(const std::string& path) {
  void* lib = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(lib != nullptr, "cannot load ", path, ": ", dlerror());
  auto get = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(lib, name));
    TORCH_CHECK(fn != nullptr, path, " has no ", name);
  };
  get(api.last_error, "tri_last_error"); get(api.last_path, "tri_last_path"); get(api.ws_status, "tri_ws_status");
  get(api.attn_ws_bytes, "tri_attn_ws_bytes"); get(api.attn_fwd, "tri_attn_fwd"); get(api.attn_bwd, "tri_attn_bwd");
  get(api.mul_fwd_residual, "tri_mul_fwd_residual");
  get(api.attn_project_bias, "tri_attn_project_bias"); get(api.gate_mul, "tri_gate_mul"); get(api.gated_linear_after, "tri_gated_linear_after");
  get(api.mul_saved_bytes, "tri_mul_saved_bytes"); get(api.mul_ws_bytes, "tri_mul_ws_bytes");
  get(api.mul_fwd, "tri_mul_fwd"); get(api.mul_bwd, "tri_mul_bwd");
}

void ok(int code, const char* what) {
  TORCH_CHECK(code == 0, what, " failed with code ", code, ": ", api.last_error());
}
// with TRI_B200_CHECK=1, read back the tensor-core kernels' status (synchronises the stream)
void check_device(const Tensor& ws, cudaStream_t st) {
  const char* e = std::getenv("TRI_B200_CHECK");
  if (e != nullptr && std::strcmp(e, "1") == 0 && std::strcmp(api.last_path(), "tcgen05") == 0)
    ok(api.ws_status(ws.data_ptr(), reinterpret_cast<tri_stream_t>(st)), "device status");
}

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return TRI_F32;
    case at::kBFloat16: return TRI_BF16;
    case at::kHalf: return TRI_F16;
    default: TORCH_CHECK_TYPE(false, "unsupported dtype torch.", at::toString(t.scalar_type()));
  }
}
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
Tensor bytes(size_t n, const Tensor& like) {
  return at::empty({(int64_t)std::max<size_t>(n, 1)}, like.options().dtype(at::kByte));
}
// Without gradients the torch calls of a function need no autograd bookkeeping (about half a microsecond each).  Tensors that are
// handed out must not be views made under this.
struct NoRecord {
  std::optional<at::AutoDispatchBelowADInplaceOrView> guard;
  explicit NoRecord(bool on) { if (on) guard.emplace(); }
};
// Is a derivative taken through any of these: recorded for a backward, or carried along in forward mode?
bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(0).defined(); }
bool wants_grad(std::initializer_list<const Tensor*> tensors) {
  const bool mode = at::GradMode::is_enabled();
  for (const Tensor* t : tensors)
    if ((mode && t->defined() && t->requires_grad()) || has_tangent(*t)) return true;
  return false;
}
void refuse_tangents(std::initializer_list<const Tensor*> tensors, const char* op) {
  for (const Tensor* t : tensors) TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent(*t), op, " has no forward-mode derivative");
}
Tensor or_undefined(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

tri_stream_t stream_of(const Tensor& t) {
  return reinterpret_cast<tri_stream_t>(c10::cuda::getCurrentCUDAStream(t.get_device()).stream());
}

// --------------------------------------------------------------------------------------------------- attention

// a tensor whose last axis has stride 1 (copied only if it does not)
Tensor inner_contiguous(const Tensor& t) { return t.stride(-1) == 1 || t.size(-1) == 1 ? t : t.contiguous(); }

// an output with t's layout where t is a permutation of a dense block, else contiguous
Tensor like(const Tensor& t) {
  if (t.is_contiguous()) return at::empty(t.sizes(), t.options());
  bool dense = t.stride(-1) == 1;
  if (dense) {
    std::vector<std::pair<int64_t, int64_t>> ax;   // (stride, size)
    for (int64_t i = 0; i < t.dim(); ++i)
      if (t.size(i) != 1) ax.emplace_back(t.stride(i), t.size(i));
    std::sort(ax.begin(), ax.end());
    int64_t expect = 1;
    for (auto& a : ax) {
      if (a.first != expect) { dense = false; break; }
      expect *= a.second;
    }
  }
  return dense ? at::empty_strided(t.sizes(), t.strides(), t.options()) : at::empty(t.sizes(), t.options());
}

void st4(int64_t (&dst)[4], const Tensor& t) {
  for (int i = 0; i < 4; ++i) dst[i] = t.stride(i);
}

TriAttnDesc attn_desc(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& bias, const Tensor& mask,
                      double scale, int64_t precision) {
  TriAttnDesc d{};
  d.B = q.size(0); d.n_seq = q.size(1); d.n_res = q.size(2); d.H = q.size(3); d.D = q.size(4);
  d.dtype = dtype_code(q); d.precision = (int)precision; d.scale = (float)scale;
  st4(d.q_st, q); st4(d.k_st, k); st4(d.v_st, v); st4(d.o_st, o);
  if (bias.defined()) { d.bias_st[0] = bias.stride(0); d.bias_st[1] = bias.stride(2); d.bias_st[2] = bias.stride(3); }
  else d.bias_st[1] = d.bias_st[2] = 8;   // (strides that need no copy: no room for one)
  if (mask.defined()) { d.mask_st[0] = mask.stride(0); d.mask_st[1] = mask.stride(1); }
  return d;
}

// the workspace of a call; a bias that starts off a 16-byte boundary is copied into it
size_t attn_ws_bytes(const TriAttnDesc& d, const Tensor& bias, int is_bwd) {
  const size_t n = api.attn_ws_bytes(&d, is_bwd);
  if (!bias.defined() || reinterpret_cast<uintptr_t>(bias.data_ptr()) % 16 == 0) return n;
  return n + (size_t)bias.element_size() * d.B * d.H * d.n_res * (d.n_res + 7) + 256;
}

struct AttnCall { Tensor q, k, v, bias, mask, o, stats; };   // mask: bytes [B, S, N]

// q, k, v [B, S, N, H, D], bias [B, 1, H, N, N], mask [B, S, 1, 1, N]
// (`rows`: o contiguous in that order of axes, else laid out like q; or like `model`)
AttnCall attn_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& bias_, const Tensor& mask_, double scale,
                      int64_t precision, bool rows, bool record = false, const Tensor& model = Tensor()) {
  TORCH_CHECK_VALUE(q_.dim() == 5 && k_.sizes() == q_.sizes() && v_.sizes() == q_.sizes(),
                    "q, k and v must have one shape, got ", q_.sizes(), ", ", k_.sizes(), " and ", v_.sizes());
  TORCH_CHECK_VALUE(k_.device() == q_.device() && v_.device() == q_.device() && (!bias_.defined() || bias_.device() == q_.device()) &&
                    (!mask_.defined() || mask_.device() == q_.device()), "q, k, v, bias and mask must be on one device");
  const NoRecord fast(!record);   // (views that are saved for a backward share their base's version counter)
  AttnCall c;
  c.q = inner_contiguous(q_); c.k = inner_contiguous(k_); c.v = inner_contiguous(v_);
  if (bias_.defined()) c.bias = inner_contiguous(bias_);
  const int64_t B = c.q.size(0), S = c.q.size(1), N = c.q.size(2), H = c.q.size(3);
  if (mask_.defined()) c.mask = mask_.reshape({B, S, N}).contiguous();
  c.o = model.defined() ? at::empty_strided(model.sizes(), model.strides(), c.q.options())
                        : (rows ? at::empty(c.q.sizes(), c.q.options()) : like(c.q));
  c.stats = at::empty({2, B, S, H, N}, c.q.options().dtype(at::kFloat));
  const TriAttnDesc d = attn_desc(c.q, c.k, c.v, c.o, c.bias, c.mask, scale, precision);
  const c10::cuda::CUDAGuard guard(c.q.device());
  const size_t n = attn_ws_bytes(d, c.bias, 0);
  const Tensor ws = bytes(n, c.q);
  const tri_stream_t st = stream_of(c.q);
  ok(api.attn_fwd(&d, ptr(c.q), ptr(c.k), ptr(c.v), ptr(c.bias), static_cast<const uint8_t*>(ptr(c.mask)), ptr(c.o),
                  static_cast<float*>(ptr(c.stats)), ptr(ws), n, st), "tri_attn_fwd");
  check_device(ws, reinterpret_cast<cudaStream_t>(st));
  return c;
}

// (an autograd Function takes an absent tensor as an empty optional; needs_input_grad counts the tensors that are there)
OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }

struct AttnFn : torch::autograd::Function<AttnFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& bias,
                               const OptTensor& mask, double scale, int64_t precision, bool rows) {
    const AttnCall c = attn_forward(q, k, v, or_undefined(bias), or_undefined(mask), scale, precision, rows, /*record=*/true);
    ctx->save_for_backward({c.q, c.k, c.v, c.bias, c.mask, c.o, c.stats});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["precision"] = precision;
    ctx->mark_non_differentiable({c.stats});
    ctx->set_materialize_grads(false);   // (no zeros for the statistics)
    return {c.o, c.stats};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &bias = s[3], &mask = s[4], &o = s[5], &stats = s[6];
    const Tensor d_o = grads[0].defined() ? inner_contiguous(grads[0]) : at::zeros_like(o);
    const int64_t B = q.size(0), N = q.size(2), H = q.size(3);
    Tensor dq = like(q), dk = like(k), dv = like(v), dbias;
    if (bias.defined() && ctx->needs_input_grad(3)) dbias = at::empty({B, H, N, N}, q.options().dtype(at::kFloat));
    TriAttnDesc d = attn_desc(q, k, v, o, bias, mask, ctx->saved_data["scale"].toDouble(), ctx->saved_data["precision"].toInt());
    st4(d.do_st, d_o); st4(d.dq_st, dq); st4(d.dk_st, dk); st4(d.dv_st, dv);
    const c10::cuda::CUDAGuard guard(q.device());
    const size_t n = attn_ws_bytes(d, bias, 1);
    const Tensor ws = bytes(n, q);
    const tri_stream_t st = stream_of(q);
    ok(api.attn_bwd(&d, ptr(q), ptr(k), ptr(v), ptr(bias), static_cast<const uint8_t*>(ptr(mask)), ptr(o),
                    static_cast<const float*>(ptr(stats)), ptr(d_o), ptr(dq), ptr(dk), ptr(dv), static_cast<float*>(ptr(dbias)),
                    ptr(ws), n, st), "tri_attn_bwd");
    check_device(ws, reinterpret_cast<cudaStream_t>(st));
    if (dbias.defined()) dbias = dbias.to(bias.scalar_type()).view({B, 1, H, N, N});
    return {dq, dk, dv, dbias, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// residual + attention, laid out like the residual; q, k, v, residual [B, S, N, H, D], bias [B, 1, H, N, N]; inference only
Tensor attention_residual(const Tensor& residual, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias, const Tensor& mask,
                          int64_t precision) {
  TORCH_CHECK(residual.is_cuda() && residual.sizes() == q.sizes() && residual.scalar_type() == q.scalar_type() &&
              residual.is_non_overlapping_and_dense() && residual.stride(-1) == 1, "residual must be dense and of q's shape and dtype");
  refuse_tangents({&residual, &q, &k, &v, &bias}, "triangle_attention");
  const at::NoGradGuard no_grad;
  // (the sum in the kernel's epilogue was slower, 0.25 ms per 1024 x 1024 x 4 x 32 call against 0.12: its softmax warps wait for it)
  return attn_forward(q, k, v, bias, mask, 1.0 / std::sqrt((double)q.size(4)), precision, false, false, residual).o.add_(residual);
}

// leading axes folded (or added) to rank 5
Tensor rank5(const Tensor& t) {
  if (t.dim() == 5) return t;
  std::vector<int64_t> s(t.sizes().begin(), t.sizes().end());
  if (t.dim() < 5) {
    s.insert(s.begin(), 5 - t.dim(), 1);
    return t.reshape(s);
  }
  return t.reshape({-1, s[s.size() - 4], s[s.size() - 3], s[s.size() - 2], s[s.size() - 1]});
}

// o and the statistics, recorded for the backward where a gradient is wanted
std::pair<Tensor, Tensor> attn_any(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias, const Tensor& mask, double scale,
                                   int64_t precision, bool rows) {
  refuse_tangents({&q, &k, &v, &bias}, "triangle_attention");
  if (wants_grad({&q, &k, &v, &bias})) {
    const variable_list r = AttnFn::apply(q, k, v, opt(bias), opt(mask), scale, precision, rows);
    return {r[0], r[1]};
  }
  const AttnCall c = attn_forward(q, k, v, bias, mask, scale, precision, rows);
  return {c.o, c.stats};
}

py::object attention(const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& bias_, const OptTensor& mask_,
                     std::optional<double> scale_, int64_t precision, bool return_aux) {
  TORCH_CHECK(q_.is_cuda(), "triangle_attention needs CUDA tensors: there is no CPU implementation");
  dtype_code(q_);
  const bool canonical = q_.dim() == 5;
  Tensor o, stats;
  {
    Tensor bias = or_undefined(bias_), mask;
    const NoRecord fast(!wants_grad({&q_, &k_, &v_, &bias}));
    const Tensor q = rank5(q_);
    Tensor k = rank5(k_), v = rank5(v_);
    if (k.scalar_type() != q.scalar_type()) k = k.to(q.scalar_type());
    if (v.scalar_type() != q.scalar_type()) v = v.to(q.scalar_type());
    const int64_t B = q.size(0), S = q.size(1), N = q.size(2), H = q.size(3);
    if (bias.defined()) {
      if (bias.dim() == 4) bias = bias.unsqueeze(-4);
      else if (bias.dim() > 5) bias = rank5(bias);
      bias = bias.expand({B, 1, H, N, N});
      if (bias.scalar_type() != q.scalar_type()) bias = bias.to(q.scalar_type());
    }
    if (mask_.has_value()) {
      mask = *mask_;
      if (mask.dim() > 5) mask = rank5(mask);
      mask = mask.expand({B, S, 1, 1, N});
    }
    const double scale = scale_.has_value() ? *scale_ : 1.0 / std::sqrt((double)q.size(4));
    std::tie(o, stats) = attn_any(q, k, v, bias, mask, scale, precision, false);
  }
  if (!canonical) o = o.reshape(q_.sizes());
  if (!return_aux) return py::cast(o);
  const Tensor m = stats.select(0, 0);
  return py::make_tuple(o, (m + stats.select(0, 1)).unsqueeze(-1), m.unsqueeze(-1));
}

// ------------------------------------------------------------------------------------- multiplicative update

constexpr int kWeights = 12;   // in the order of TriMulWeights
using Weights = std::array<Tensor, kWeights>;
static_assert(sizeof(TriMulWeights) == kWeights * sizeof(void*) && sizeof(TriMulWeightGrads) == kWeights * sizeof(void*));
const char* const kNames[kWeights] = {"norm_in_weight", "norm_in_bias", "p_in_weight", "p_in_bias", "g_in_weight", "g_in_bias",
                                      "norm_out_weight", "norm_out_bias", "p_out_weight", "p_out_bias", "g_out_weight", "g_out_bias"};

// contiguous and 16-byte aligned (TMA and the vector loads need it); copied only if it must be
Tensor aligned(const Tensor& t_) {
  const Tensor t = t_.contiguous();
  return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone();
}

TriMulWeights weight_ptrs(const Weights& w) {
  TriMulWeights p;
  const void* a[kWeights];
  for (int i = 0; i < kWeights; ++i) a[i] = ptr(w[i]);
  std::memcpy(&p, a, sizeof p);
  return p;
}

struct MulCall { TriMulDesc d; Tensor x, mask, saved, out; Weights w; };

// `residual`: out is x + update
MulCall mul_forward(const Tensor& x, const Tensor& mask, const Weights& weights, bool outgoing, double eps, int64_t precision, bool keep,
                    bool residual = false) {
  TORCH_CHECK(x.is_cuda(), "triangle_multiplicative_update needs CUDA tensors: there is no CPU implementation");
  const NoRecord fast(!keep);   // as in attn_forward
  MulCall c{};
  c.d.dtype = dtype_code(x);
  for (int i : {2, 4, 8, 10}) TORCH_CHECK_VALUE(weights[i].defined(), kNames[i], " is required");
  for (int i = 0; i < kWeights; ++i)
    TORCH_CHECK_VALUE(!weights[i].defined() || weights[i].device() == x.device(), kNames[i], " is on ", weights[i].device(), ", x on ", x.device());
  TORCH_CHECK_VALUE(!mask.defined() || mask.device() == x.device(), "mask is on ", mask.device(), ", x on ", x.device());
  TORCH_CHECK_VALUE(x.dim() >= 3 && x.size(-2) == x.size(-3), "x must be [*, N, N, C], got ", x.sizes());
  const int64_t N = x.size(-2), C = x.size(-1);
  c.x = aligned(x.dim() == 4 ? x : x.reshape({-1, N, N, C}));
  const int64_t B = c.x.size(0);
  if (mask.defined()) c.mask = aligned(mask.to(x.scalar_type()).expand(x.sizes().slice(0, x.dim() - 1)).reshape({B, N, N}));
  for (int i = 0; i < kWeights; ++i)
    if (weights[i].defined()) c.w[i] = aligned(weights[i].scalar_type() == x.scalar_type() ? weights[i].detach() : weights[i].detach().to(x.scalar_type()));
  const int64_t Ch = c.w[2].size(0) / 2;
  const int64_t rows[kWeights] = {C, C, 2 * Ch, 2 * Ch, 2 * Ch, 2 * Ch, Ch, Ch, C, C, C, C};
  const int64_t cols[kWeights] = {0, 0, C, 0, C, 0, 0, 0, Ch, 0, C, 0};
  for (int i = 0; i < kWeights; ++i) {
    if (!c.w[i].defined()) continue;
    const auto s = c.w[i].sizes();
    const bool fits = cols[i] ? s.size() == 2 && s[0] == rows[i] && s[1] == cols[i] : s.size() == 1 && s[0] == rows[i];
    TORCH_CHECK_VALUE(fits, kNames[i], " has shape ", s, ", expected [", rows[i], cols[i] ? ", " + std::to_string(cols[i]) : std::string(), "]");
  }
  c.d.B = B; c.d.N = N; c.d.C = C; c.d.Ch = Ch; c.d.precision = (int)precision;
  c.d.direction = outgoing ? TRI_OUTGOING : TRI_INCOMING; c.d.eps = (float)eps;
  const c10::cuda::CUDAGuard guard(x.device());
  if (keep) c.saved = bytes(api.mul_saved_bytes(&c.d), x);
  const size_t n = api.mul_ws_bytes(&c.d, 0);
  const Tensor ws = bytes(n, x);
  c.out = at::empty(c.x.sizes(), c.x.options());
  const TriMulWeights w = weight_ptrs(c.w);
  const tri_stream_t st = stream_of(x);
  bool add = residual;
  if (add) {
    const int code = api.mul_fwd_residual(&c.d, ptr(c.x), ptr(c.mask), &w, ptr(c.x), ptr(c.out), ptr(ws), n, st);
    if (code != TRI_ERR_UNSUPPORTED) { ok(code, "tri_mul_fwd_residual"); add = false; }
  }
  if (!residual || add) ok(api.mul_fwd(&c.d, ptr(c.x), ptr(c.mask), &w, ptr(c.out), ptr(c.saved), ptr(ws), n, st), "tri_mul_fwd");
  if (add) c.out.add_(c.x);
  check_device(ws, reinterpret_cast<cudaStream_t>(st));
  return c;
}

struct MulFn : torch::autograd::Function<MulFn> {
  using O = const OptTensor&;
  static Tensor forward(AutogradContext* ctx, const Tensor& x, O mask, O w0, O w1, O w2, O w3, O w4, O w5, O w6, O w7, O w8, O w9, O w10,
                        O w11, bool outgoing, double eps, int64_t precision) {
    Weights in;
    int n = 0;
    for (O w : {std::cref(w0), std::cref(w1), std::cref(w2), std::cref(w3), std::cref(w4), std::cref(w5), std::cref(w6), std::cref(w7),
                std::cref(w8), std::cref(w9), std::cref(w10), std::cref(w11)})
      in[n++] = or_undefined(w);
    const MulCall c = mul_forward(x, or_undefined(mask), in, outgoing, eps, precision, /*keep=*/true);
    variable_list keep = {c.x, c.mask, c.saved};
    std::vector<int64_t> dtypes(kWeights, -1);
    for (int i = 0; i < kWeights; ++i) {
      keep.push_back(c.w[i]);
      if (in[i].defined()) dtypes[i] = (int64_t)in[i].scalar_type();
    }
    ctx->save_for_backward(keep);
    ctx->saved_data["desc"] = std::string(reinterpret_cast<const char*>(&c.d), sizeof c.d);
    ctx->saved_data["dtypes"] = dtypes;
    ctx->saved_data["shape"] = x.sizes().vec();
    return c.out.reshape(x.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &mask = s[1], &saved = s[2];
    TriMulDesc d;
    std::memcpy(&d, ctx->saved_data["desc"].toStringRef().data(), sizeof d);
    const auto dtypes = ctx->saved_data["dtypes"].toIntVector();
    Weights w;
    for (int i = 0; i < kWeights; ++i) w[i] = s[3 + i];
    // the weight gradients, fp32 as the library writes them, side by side: one conversion to the weights' dtype for all
    std::array<int64_t, kWeights> at_{};
    int64_t total = 0, one = -1;
    bool same = true;
    size_t input = mask.defined() ? 2 : 1;   // x, the mask, then the weights that are there
    for (int i = 0; i < kWeights; ++i) {
      at_[i] = -1;
      if (!w[i].defined() || !ctx->needs_input_grad(input++)) continue;
      at_[i] = total;
      total += (w[i].numel() + 15) / 16 * 16;
      if (one >= 0 && one != dtypes[i]) same = false;
      one = dtypes[i];
    }
    Tensor flat = at::empty({total}, x.options().dtype(at::kFloat));
    void* g_ptr[kWeights];
    for (int i = 0; i < kWeights; ++i) g_ptr[i] = at_[i] < 0 ? nullptr : flat.data_ptr<float>() + at_[i];
    TriMulWeightGrads g;
    std::memcpy(&g, g_ptr, sizeof g);
    const Tensor d_out = aligned(grads[0].reshape(x.sizes()).to(x.scalar_type()));
    Tensor dx = at::empty(x.sizes(), x.options());
    const c10::cuda::CUDAGuard guard(x.device());
    const size_t n = api.mul_ws_bytes(&d, 1);
    const Tensor ws = bytes(n, x);
    const TriMulWeights wp = weight_ptrs(w);
    const tri_stream_t st = stream_of(x);
    ok(api.mul_bwd(&d, ptr(x), ptr(mask), &wp, ptr(saved), ptr(d_out), ptr(dx), &g, ptr(ws), n, st), "tri_mul_bwd");
    check_device(ws, reinterpret_cast<cudaStream_t>(st));
    variable_list out(2 + kWeights + 3);
    if (ctx->needs_input_grad(0)) out[0] = dx.reshape(ctx->saved_data["shape"].toIntVector());
    if (same && one >= 0) flat = flat.to((at::ScalarType)one);
    for (int i = 0; i < kWeights; ++i) {
      if (at_[i] < 0) continue;
      Tensor t = flat.narrow(0, at_[i], w[i].numel()).view(w[i].sizes());
      out[2 + i] = same ? t : t.to((at::ScalarType)dtypes[i]);
    }
    return out;
  }
};

Tensor multiplicative_update(const Tensor& x, const OptTensor& mask_, bool outgoing, double eps, int64_t precision,
                             const std::vector<OptTensor>& weights) {
  TORCH_CHECK(weights.size() == kWeights, "expected ", kWeights, " weights");
  Weights w;
  const Tensor mask = or_undefined(mask_);
  refuse_tangents({&x, &mask}, "triangle_multiplicative_update");
  bool grad = wants_grad({&x});
  for (int i = 0; i < kWeights; ++i) {
    w[i] = or_undefined(weights[i]);
    refuse_tangents({&w[i]}, "triangle_multiplicative_update");
    grad = grad || wants_grad({&w[i]});
  }
  if (grad)
    return MulFn::apply(x, mask_, weights[0], weights[1], weights[2], weights[3], weights[4], weights[5], weights[6], weights[7], weights[8],
                        weights[9], weights[10], weights[11], outgoing, eps, precision);
  return mul_forward(x, mask, w, outgoing, eps, precision, /*keep=*/false).out.reshape(x.sizes());
}

// x + update, inference only
Tensor multiplicative_update_residual(const Tensor& x, const OptTensor& mask, bool outgoing, double eps, int64_t precision,
                                      const std::vector<OptTensor>& weights) {
  TORCH_CHECK(weights.size() == kWeights, "expected ", kWeights, " weights");
  Weights w;
  refuse_tangents({&x}, "triangle_multiplicative_update");
  for (int i = 0; i < kWeights; ++i) {
    w[i] = or_undefined(weights[i]);
    refuse_tangents({&w[i]}, "triangle_multiplicative_update");
  }
  const at::NoGradGuard no_grad;
  return mul_forward(x, or_undefined(mask), w, outgoing, eps, precision, /*keep=*/false, /*residual=*/true).out.reshape(x.sizes());
}

// ---------------------------------------------------------------------------------------------------- pair bias

// z [B, U, V, Zc] -> LayerNorm (weight only) -> projection to H heads -> [B, H, U, V].  One kernel where it has the shape (16-bit
// types, 128 channels, at most 16 heads) and neither gradients nor autocast are in force, else torch's operations.
bool pair_bias_fits(const Tensor& z, const OptTensor& ln_w, const Tensor& w) {
  const auto dt = z.scalar_type();
  const bool fits = z.is_cuda() && z.dim() == 4 && (dt == at::kBFloat16 || dt == at::kHalf) && z.size(3) == 128 && w.dim() == 2 &&
                    w.size(1) == 128 && w.size(0) >= 1 && w.size(0) <= 16 && w.scalar_type() == dt && w.device() == z.device() &&
                    (!ln_w.has_value() || (ln_w->scalar_type() == dt && ln_w->dim() == 1 && ln_w->size(0) == 128 && ln_w->device() == z.device()));
  const Tensor lw = or_undefined(ln_w);
  return fits && !wants_grad({&z, &w, &lw}) && z.numel() >= 128 && z.numel() / 128 < (1LL << 31) - 128 && !at::autocast::is_autocast_enabled(at::kCUDA);
}
// (`status`: the kernel's workspace, whose first word later kernels on the stream may report to; undefined where torch ran)
Tensor pair_bias_of(const Tensor& z, const OptTensor& ln_w, const Tensor& w, double eps, Tensor* status) {
  if (!pair_bias_fits(z, ln_w, w))
    return at::linear(at::layer_norm(z, {z.size(-1)}, ln_w, {}, eps), w).permute({0, 3, 1, 2}).contiguous();
  TriAttnProjDesc d{};
  d.M = z.numel() / 128; d.C = 128; d.H = (int32_t)w.size(0); d.dtype = dtype_code(z); d.eps = (float)eps;
  const c10::cuda::CUDAGuard guard(z.device());
  const Tensor zc = aligned(z), wc = aligned(w), lw = ln_w.has_value() ? ln_w->contiguous() : Tensor(), ws = bytes(256, z);
  const Tensor out = at::empty({z.size(0), w.size(0), z.size(1), z.size(2)}, z.options());
  const tri_stream_t st = stream_of(z);
  ok(api.attn_project_bias(&d, z.size(1) * z.size(2), ptr(zc), ptr(lw), nullptr, ptr(wc), ptr(out), ptr(ws), st), "tri_attn_project_bias");
  check_device(ws, reinterpret_cast<cudaStream_t>(st));
  *status = ws;
  return out;
}
Tensor pair_bias(const Tensor& z, const OptTensor& ln_w, const Tensor& w, double eps) {
  Tensor status;
  return pair_bias_of(z, ln_w, w, eps, &status);
}

// Whether (o * sigmoid(s g_w^T)) o_w^T can run as two products of this package: dense operands of one 16-bit type, no biases.
bool gated_linear_fits(const Tensor& s, const Tensor& o, const Tensor& g_w, const Tensor& o_w) {
  const auto dt = s.scalar_type();
  if ((dt != at::kBFloat16 && dt != at::kHalf) || s.numel() == 0 || g_w.size(1) != s.size(-1) || g_w.size(0) != o.size(-1) ||
      o_w.size(1) != o.size(-1) || s.numel() / s.size(-1) != o.numel() / o.size(-1) || s.numel() / s.size(-1) >= (1LL << 31) - 128)
    return false;
  for (const Tensor* t : {&s, &o, &g_w, &o_w})
    if (t->scalar_type() != dt || t->device() != s.device() || !t->is_contiguous() || reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 != 0) return false;
  return g_w.size(1) % 8 == 0 && g_w.size(0) % 8 == 0 && o_w.size(0) % 8 == 0 && o_w.size(0) > 0;
}

// o * sigmoid(gate)
Tensor gated(const Tensor& o, const Tensor& gate) {
  if (wants_grad({&o, &gate}) || !o.is_contiguous() || !gate.is_contiguous() || o.scalar_type() != gate.scalar_type() || o.sizes() != gate.sizes())
    return o * at::sigmoid(gate);
  const c10::cuda::CUDAGuard guard(o.device());
  const Tensor out = at::empty(o.sizes(), o.options());
  ok(api.gate_mul(dtype_code(o), o.numel(), ptr(o), ptr(gate), ptr(out), stream_of(o)), "tri_gate_mul");
  return out;
}

// The whole of attention_pair_bias where its softmax core runs on the kernels (the Python function decides); returns the
// output and the projected bias.  About fifteen torch calls, which took 100 us from Python and whose kernels take a third of that.
std::pair<Tensor, Tensor> attention_pair_bias(const Tensor& s, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& z,
                                              const Tensor& g_w, const OptTensor& g_b, const Tensor& o_w, const OptTensor& o_b,
                                              const OptTensor& z_w, const OptTensor& ln_w, const OptTensor& mask_, double scale, double eps,
                                              int64_t precision) {
  const int64_t BM = q.size(0), H = q.size(1), U = q.size(2), D = q.size(3), B = z.size(0), M = BM / B;
  const Tensor gb = or_undefined(g_b), ob = or_undefined(o_b), zw = or_undefined(z_w), lw = or_undefined(ln_w);
  const bool grad = wants_grad({&s, &q, &k, &v, &z, &g_w, &o_w, &gb, &ob, &zw, &lw});
  const NoRecord fast(!grad);
  Tensor status;
  const Tensor pz = z_w.has_value() ? pair_bias_of(z, ln_w, *z_w, eps, &status) : z;
  // (BM, H, U, D) -> rows = multiplicity: [B, M, U, H, D] as a strided view (no copy)
  auto rows = [&](const Tensor& t) { return inner_contiguous(t.reshape({B, M, H, U, D}).transpose(2, 3)); };
  Tensor mask;
  if (mask_.has_value()) mask = at::ne(*mask_, 0).reshape({B, -1, 1, 1, U}).expand({B, M, 1, 1, U});
  const Tensor bias = (pz.scalar_type() == q.scalar_type() ? pz : pz.to(q.scalar_type())).unsqueeze(1).expand({B, 1, H, U, U});
  const Tensor o = attn_any(rows(q), rows(k), rows(v), bias, mask, scale, precision, true).first.reshape({BM, U, H * D}).to(s.scalar_type());
  if (grad || s.dim() != 3 || !s.is_contiguous() || g_w.dim() != 2 || o_w.dim() != 2)
    return {at::linear(gated(o, at::linear(s, g_w, g_b)), o_w, o_b), pz};
  if (status.defined() && !g_b.has_value() && !o_b.has_value() && gated_linear_fits(s, o, g_w, o_w)) {
    const c10::cuda::CUDAGuard guard(s.device());
    const int64_t W = H * D, N = o_w.size(0);
    const Tensor gated = at::empty({BM, U, W}, s.options()), out = at::empty({BM, U, N}, s.options());
    const tri_stream_t st = stream_of(s);
    // (the last call of the library is the attention, and s and the weights are the caller's: older than it)
    ok(api.gated_linear_after(dtype_code(s), BM * U, (int32_t)s.size(2), (int32_t)W, (int32_t)N, ptr(s), ptr(g_w), ptr(o), ptr(o_w), ptr(gated),
                              ptr(out), ptr(status), st), "tri_gated_linear_after");
    check_device(status, reinterpret_cast<cudaStream_t>(st));
    return {out, pz};
  }
  // the same products on two dimensions
  auto linear = [](const Tensor& x, const Tensor& w, const OptTensor& b) { return b.has_value() ? at::addmm(*b, x, w.t()) : at::mm(x, w.t()); };
  const Tensor gate = linear(s.view({-1, s.size(2)}), g_w, g_b);
  const Tensor out = linear(gated(o.reshape({-1, H * D}), gate), o_w, o_b);
  return {at::_unsafe_view(out, {BM, U, o_w.size(0)}), pz};   // (the product's own storage, and no view of a tensor that is kept)
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("bind", &bind);
  m.def("attention", &attention);
  m.def("multiplicative_update", &multiplicative_update);
  m.def("attention_residual", &attention_residual);
  m.def("multiplicative_update_residual", &multiplicative_update_residual);
  m.def("pair_bias", &pair_bias);
  m.def("pair_bias_fits", &pair_bias_fits);
  m.def("attention_pair_bias", &attention_pair_bias);
}
