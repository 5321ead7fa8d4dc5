// Native host path of the ops: argument checks of the common case, output and workspace allocation, the
// autograd nodes and the calls into the C ABI (include/slinoss_b200.h).
//
// What bounds the small calls is the host: a Python autograd.Function, ctypes argument conversion and torch's
// operator dispatch together took 110-260 us per scan or layer call, several times the kernels of a short
// sequence (one token of decode: 213 us for 8 us of kernels).  Here a call costs the allocations and the launches.
//
// Every entry point takes the form in which programs normally call the op (one device, contiguous, 16-byte aligned,
// matching shapes and dtypes) and returns None for anything else; the Python function above it then raises the
// error, or converts the arguments and calls again.  The interpreter lock is not held meanwhile: an allocation or a full
// launch queue may wait for the GPU, and what it waits for may be another thread's to launch.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <optional>
#include <tuple>
#include <vector>

#include "../../../include/slinoss_b200.h"

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

namespace {

int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return SLX_F32;
    case at::kBFloat16: return SLX_BF16;
    case at::kHalf: return SLX_F16;
    default: return -1;
  }
}
at::ScalarType type_of(int code) { return code == SLX_BF16 ? at::kBFloat16 : code == SLX_F16 ? at::kHalf : at::kFloat; }

// A non-zero status as the exception the reference would raise.
void check(int status, const char *what) {
  if (status == SLX_OK) return;
  const char *msg = slx_last_error_string();
  if (status == SLX_E_DTYPE) TORCH_CHECK_TYPE(false, what, ": ", msg);
  if (status < 0) TORCH_CHECK_VALUE(false, what, ": ", msg);
  TORCH_CHECK(false, what, ": CUDA error ", status, ": ", msg);
}

Tensor empty(at::IntArrayRef sizes, at::ScalarType t, const at::Device &dev) {
  return Tensor(at::detail::empty_cuda(sizes, t, dev, std::nullopt));
}
void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }
const void *cptr(const OptTensor &t) { return t ? t->data_ptr() : nullptr; }
float *fptr(const Tensor &t) { return t.defined() ? static_cast<float *>(t.data_ptr()) : nullptr; }
bool aligned(const Tensor &t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
void *stream_of(const at::Device &dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
bool is(const Tensor &t, const at::Device &dev) { return t.defined() && t.device() == dev; }
bool shaped(const Tensor &t, at::IntArrayRef sizes) { return t.sizes() == sizes; }

// a tensor in the dtype and layout the kernels read
Tensor as_read(const Tensor &g, at::ScalarType t) {
  Tensor r = g.scalar_type() == t ? g : g.to(t);
  r = r.contiguous();
  return aligned(r) ? r : r.clone();
}
Tensor saved(SavedVariable &v) { return v.unpack(); }
// Forward-mode derivatives are not implemented: an error, not an output without its tangent.
void refuse_tangent(const Tensor &t) {
  TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(0).defined(),
                              "slinoss_b200 ops have no forward-mode derivative; use reverse mode.");
}
template <typename... T>
void refuse_tangents(const T &...t) {
  (refuse_tangent(t), ...);
}
Tensor or_undefined(const OptTensor &t) { return t.value_or(Tensor()); }
SavedVariable keep(const Tensor &t) { return t.defined() ? SavedVariable(t, false) : SavedVariable(); }
// A small tensor that its owner may overwrite before the backward runs (a stream's carried rows, in place; parameters): a
// half one is kept by value, an fp32 one by reference, so that autograd reports the overwriting.
SavedVariable keep_value(const Tensor &t) { return keep(t.scalar_type() == at::kFloat ? t : t.detach().clone()); }

template <typename N>
std::shared_ptr<N> make_node(torch::autograd::edge_list edges) {
  std::shared_ptr<N> node(new N(), torch::autograd::deleteNode);
  node->set_next_edges(std::move(edges));
  return node;
}

// ------------------------------------------------------------------------------------------------------------
// chunked scan
// ------------------------------------------------------------------------------------------------------------
struct ScanDims {
  int64_t b, h, T, P, D, L, NC;
  slx_scan_shape s;
  at::Device dev = at::kCUDA;
  at::ScalarType act;
};

// starts_dtype (the code in which chunk starts are held, and with it the kernel family): that of chunk starts in hand, or
// the library's current choice for the shape.
ScanDims scan_dims(const Tensor &U, const Tensor &B, int64_t L, std::optional<int> starts_dtype = std::nullopt) {
  ScanDims d;
  d.b = U.size(0);
  d.h = U.size(1);
  d.T = U.size(2);
  d.P = U.size(3);
  d.D = B.size(3);
  d.L = L;
  d.NC = (d.T + L - 1) / L;
  d.dev = U.device();
  d.act = U.scalar_type();
  d.s = slx_scan_shape{(int32_t)(d.b * d.h), (int32_t)d.T, (int32_t)d.P, (int32_t)(d.D / 2), (int32_t)L,
                       code_of(d.act), SLX_F32};
  d.s.starts_dtype = starts_dtype ? *starts_dtype : slx_scan_starts_dtype(&d.s);
  return d;
}

struct ScanForward {
  Tensor Y, final32, final_copy, B_last, U_last, starts, mch;
};

ScanForward scan_forward(const ScanDims &d, const Tensor &U, const Tensor &M, const Tensor &K, const Tensor &B,
                         const Tensor &C, const OptTensor &init, const OptTensor &Bp, const OptTensor &Up,
                         bool want_final32, bool want_state, at::ScalarType final_type) {
  ScanForward r;
  const at::ScalarType st = type_of(d.s.starts_dtype);
  const int64_t chunk_sizes[5] = {d.b, d.h, d.NC, d.P, d.D};
  const int64_t state_sizes[4] = {d.b, d.h, d.P, d.D};
  r.Y = empty(U.sizes(), d.act, d.dev);
  r.starts = empty(chunk_sizes, st, d.dev);
  r.mch = empty({d.b, d.h, d.NC, 2}, at::kFloat, d.dev);
  // separate increment buffer (stored like the chunk starts): the two-buffer state pass is about 2.5x faster than
  // the in-place one
  Tensor inc = empty(chunk_sizes, st, d.dev);
  slx_scan_ends e{};
  if (want_state && final_type == at::kFloat) want_final32 = true;
  if (want_final32) r.final32 = empty(state_sizes, at::kFloat, d.dev);
  if (want_state) {
    if (final_type == at::kFloat) {
      r.final_copy = r.final32;
    } else {
      r.final_copy = empty(state_sizes, final_type, d.dev);
      e.final_copy = ptr(r.final_copy);
      e.final_dtype = code_of(final_type);
    }
    r.B_last = empty({d.b, d.h, d.D}, d.act, d.dev);
    r.U_last = empty({d.b, d.h, d.P}, d.act, d.dev);
    e.B_last = ptr(r.B_last);
    e.U_last = ptr(r.U_last);
  }
  if (init) {
    e.initial_states = init->data_ptr();
    e.initial_dtype = code_of(init->scalar_type());
  }
  if (Bp) {
    e.B_prev = Bp->data_ptr();
    e.U_prev = Up->data_ptr();
    e.prev_dtype = code_of(Bp->scalar_type());
  }
  c10::cuda::CUDAGuard guard(d.dev);
  check(slx_v2x2ssd_fwd_stream(&d.s, ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), &e, ptr(r.Y), fptr(r.final32),
                               ptr(r.starts), fptr(r.mch), ptr(inc), stream_of(d.dev)),
        "v2x2ssd forward");
  return r;
}

struct ScanGrads {
  Tensor dU, dM, dK, dB, dC, d_init, dBp, dUp;
};

ScanGrads scan_backward(const ScanDims &d, const Tensor &U, const Tensor &M, const Tensor &K, const Tensor &B,
                        const Tensor &C, const Tensor &Bp, const Tensor &Up, const Tensor &starts, const Tensor &mch,
                        const Tensor &final32, const Tensor &dY, const Tensor &d_final, std::optional<at::ScalarType> init_type,
                        bool want_prev, const OptTensor &workspace) {
  ScanGrads g;
  g.dU = empty(U.sizes(), d.act, d.dev);
  g.dB = empty(B.sizes(), d.act, d.dev);
  g.dC = empty(C.sizes(), d.act, d.dev);
  g.dM = empty(M.sizes(), at::kFloat, d.dev);
  g.dK = empty(K.sizes(), at::kFloat, d.dev);
  slx_scan_grad_ends e{};
  if (Bp.defined()) {
    e.B_prev = ptr(Bp);
    e.U_prev = ptr(Up);
    e.prev_dtype = code_of(Bp.scalar_type());
  }
  if (d_final.defined()) {
    e.d_final = ptr(d_final);
    e.d_final_dtype = code_of(d_final.scalar_type());
  }
  if (init_type) {
    g.d_init = empty({d.b, d.h, d.P, d.D}, *init_type, d.dev);
    e.d_initial = ptr(g.d_init);
    e.d_initial_dtype = code_of(*init_type);
  }
  if (want_prev) {
    const at::ScalarType t = Bp.scalar_type();
    g.dBp = empty({d.b, d.h, d.D}, t, d.dev);
    g.dUp = empty({d.b, d.h, d.P}, t, d.dev);
    e.dB_prev = ptr(g.dBp);
    e.dU_prev = ptr(g.dUp);
    e.d_prev_dtype = code_of(t);
  }
  const size_t nbytes = slx_v2x2ssd_bwd_workspace_bytes(&d.s);
  Tensor ws = workspace ? *workspace : empty({(int64_t)nbytes}, at::kByte, d.dev);
  c10::cuda::CUDAGuard guard(d.dev);
  if (!workspace) {
    check(slx_v2x2ssd_bwd_stream(&d.s, ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), &e, ptr(starts), fptr(mch),
                                 fptr(final32), ptr(dY), ptr(g.dU), fptr(g.dM), fptr(g.dK), ptr(g.dB), ptr(g.dC),
                                 ptr(ws), nbytes, stream_of(d.dev)),
          "v2x2ssd backward");
  } else {  // dZ0 is already in the workspace; this form takes fp32 streaming tensors
    check(slx_v2x2ssd_bwd_finish(&d.s, ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), fptr(Bp), fptr(Up), ptr(starts),
                                 fptr(mch), fptr(final32), ptr(dY), fptr(d_final), ptr(g.dU), fptr(g.dM), fptr(g.dK),
                                 ptr(g.dB), ptr(g.dC), fptr(g.d_init), fptr(g.dBp), fptr(g.dUp), ptr(ws), nbytes,
                                 stream_of(d.dev)),
          "v2x2ssd backward");
  }
  return g;
}

struct ScanBackward : public Node {
  int64_t L = 0;
  bool recompute = false;
  SavedVariable U_, M_, K_, B_, C_, mch_, starts_, final_, init_, Bp_, Up_;
  std::optional<at::ScalarType> init_type;  // of the initial states, where there are any
  bool has_prev = false;
  std::string name() const override { return "V2x2ssdBackward"; }

  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable *v : {&U_, &M_, &K_, &B_, &C_, &mch_, &starts_, &final_, &init_, &Bp_, &Up_}) v->reset_data();
  }

  variable_list apply(variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(8);
    const Tensor dY_in = grads[0];
    const Tensor d_fin_in = grads.size() > 1 ? grads[1] : Tensor();
    Tensor U = saved(U_), B = saved(B_);
    if (dY_in.defined() || d_fin_in.defined()) {
      Tensor M = saved(M_), K = saved(K_), C = saved(C_), mch = saved(mch_), final32 = saved(final_);
      Tensor Bp, Up;
      if (has_prev) {
        Bp = saved(Bp_);
        Up = saved(Up_);
      }
      const ScanDims d = scan_dims(U, B, L);
      Tensor dY = dY_in.defined() ? as_read(dY_in, d.act) : at::zeros_like(U);
      Tensor d_fin;
      if (d_fin_in.defined())
        d_fin = as_read(d_fin_in, code_of(d_fin_in.scalar_type()) < 0 ? at::kFloat : d_fin_in.scalar_type());
      Tensor starts;
      if (recompute) {
        const at::ScalarType st = type_of(d.s.starts_dtype);
        const int64_t sizes[5] = {d.b, d.h, d.NC, d.P, d.D};
        starts = empty(sizes, st, d.dev);
        Tensor inc = empty(sizes, st, d.dev), m2 = empty({d.b, d.h, d.NC, 2}, at::kFloat, d.dev);
        slx_scan_ends e{};
        Tensor init;
        if (init_type) {
          init = saved(init_);
          e.initial_states = ptr(init);
          e.initial_dtype = code_of(init.scalar_type());
        }
        if (has_prev) {
          e.B_prev = ptr(Bp);
          e.U_prev = ptr(Up);
          e.prev_dtype = code_of(Bp.scalar_type());
        }
        c10::cuda::CUDAGuard guard(d.dev);
        check(slx_v2x2ssd_fwd_stream(&d.s, ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), &e, nullptr, nullptr, ptr(starts),
                                     fptr(m2), ptr(inc), stream_of(d.dev)),
              "v2x2ssd chunk starts");
      } else {
        // the process may have chosen other kernels since the forward, which hold chunk starts in another dtype
        starts = as_read(saved(starts_), type_of(d.s.starts_dtype));
      }
      ScanGrads g = scan_backward(d, U, M, K, B, C, Bp, Up, starts, mch, final32, dY, d_fin, init_type, has_prev,
                                  std::nullopt);
      out = {g.dU, g.dM, g.dK, g.dB, g.dC, g.d_init, g.dBp, g.dUp};
    }
    // cotangents of the carried-on rows (they are copies of row T-1 of B and U)
    auto add_last = [](Tensor &acc, const Tensor &like, const Tensor &g) {
      if (!g.defined()) return;
      if (!acc.defined()) acc = at::zeros_like(like);
      acc.select(2, -1).add_(g.to(acc.scalar_type()));
    };
    if (grads.size() > 2) add_last(out[3], B, grads[2]);
    if (grads.size() > 3) add_last(out[0], U, grads[3]);
    return out;
  }
};

bool scan_inputs_plain(const Tensor &U, const Tensor &M, const Tensor &K, const Tensor &B, const Tensor &C,
                       const OptTensor &init, const OptTensor &Bp, const OptTensor &Up) {
  if (!U.is_cuda() || U.dim() != 4 || B.dim() != 4) return false;
  const at::Device dev = U.device();
  const at::ScalarType act = U.scalar_type();
  const int64_t b = U.size(0), h = U.size(1), T = U.size(2), P = U.size(3), D = B.size(3);
  if (code_of(act) < 0 || b == 0 || h == 0 || T == 0 || P == 0 || D == 0 || D % 2 != 0) return false;
  const int64_t bsz[4] = {b, h, T, D}, msz[4] = {b, h, T, 2}, ksz[5] = {b, h, T, 2, 2};
  if (!shaped(B, bsz) || !shaped(C, bsz) || !shaped(M, msz) || !shaped(K, ksz)) return false;
  if (B.scalar_type() != act || C.scalar_type() != act || M.scalar_type() != at::kFloat || K.scalar_type() != at::kFloat)
    return false;
  for (const Tensor *t : {&U, &M, &K, &B, &C})
    if (t->device() != dev || !t->is_contiguous() || !aligned(*t)) return false;
  if (init) {
    const int64_t sz[4] = {b, h, P, D};
    if (!is(*init, dev) || !shaped(*init, sz) || !init->is_contiguous() || !aligned(*init) ||
        code_of(init->scalar_type()) < 0)
      return false;
  }
  if (Bp.has_value() != Up.has_value()) return false;
  if (Bp) {
    const int64_t sb[3] = {b, h, D}, su[3] = {b, h, P};
    if (!is(*Bp, dev) || !is(*Up, dev) || !shaped(*Bp, sb) || !shaped(*Up, su) || !Bp->is_contiguous() ||
        !Up->is_contiguous() || !aligned(*Bp) || !aligned(*Up) || (Bp->scalar_type() != act && Bp->scalar_type() != at::kFloat) ||
        Bp->scalar_type() != Up->scalar_type())
      return false;
  }
  return true;
}

// Tiling of the CUDA-core chunk kernels.  Their work per token is least at 64 tokens: at 128 the causal triangle doubles
// and one CTA fills an SM (2, 8, T 2048, N 64, forward + backward: 466 us against 286), below it the chunk states and
// the state pass weigh more (32 tokens: 320).  A CTA's time is proportional to its tokens, though, so calls with less
// than a chunk of 64 per SM are tiled in 32 (1, 2, T 500, N 64: 99 -> 66 us; 1, 8, T 1024: 109 -> 105).
int64_t cuda_core_chunk(int64_t heads, int64_t T, const at::Device &dev) {
  return heads * ((T + 63) / 64) < at::cuda::getDeviceProperties(dev.index())->multiProcessorCount ? 32 : 64;
}

// (U, M, K, B, C) -> [Y] or [Y, final, B_last, U_last] in the activation dtype, with autograd.  None: not the
// plain case.
std::optional<std::vector<Tensor>> v2x2ssd(const Tensor &U, const Tensor &M, const Tensor &K, const Tensor &B, const Tensor &C, int64_t L,
                   const OptTensor &init, const OptTensor &Bp, const OptTensor &Up, bool return_state, bool retile,
                   bool recompute, std::optional<at::ScalarType> final_type_in) {
  if (!scan_inputs_plain(U, M, K, B, C, init, Bp, Up)) return std::nullopt;
  const int64_t P = U.size(3), D = B.size(3);
  // chunk_size only says how the sequence is tiled; the tcgen05 kernels tile in 128 tokens
  const bool tensor_cores = U.scalar_type() != at::kFloat && P == 64 && D % 64 == 0 && D <= 256;
  if (L > 0 && retile && tensor_cores) L = 128;
  if (L != 16 && L != 32 && L != 64 && L != 128) return std::nullopt;
  if (retile && !tensor_cores) L = cuda_core_chunk(U.size(0) * U.size(1), U.size(2), U.device());
  const at::ScalarType final_type = final_type_in.value_or(U.scalar_type());
  if (code_of(final_type) < 0) return std::nullopt;
  const ScanDims d = scan_dims(U, B, L);
  refuse_tangents(U, M, K, B, C, or_undefined(init), or_undefined(Bp), or_undefined(Up));
  const bool grad =
      torch::autograd::compute_requires_grad(U, M, K, B, C, or_undefined(init), or_undefined(Bp), or_undefined(Up));
  ScanForward r = scan_forward(d, U, M, K, B, C, init, Bp, Up, grad, return_state, final_type);
  if (grad) {
    auto node = make_node<ScanBackward>(torch::autograd::collect_next_edges(
        U, M, K, B, C, or_undefined(init), or_undefined(Bp), or_undefined(Up)));
    node->L = L;
    node->recompute = recompute;
    node->U_ = keep(U);
    node->M_ = keep(M);
    node->K_ = keep(K);
    node->B_ = keep(B);
    node->C_ = keep(C);
    node->mch_ = keep(r.mch);
    node->final_ = keep(r.final32.is_same(r.final_copy) ? r.final32.detach() : r.final32);
    // What is kept of the chunk-start states, the largest residual: as the kernels exchange them, or (recompute)
    // nothing: the backward rebuilds them with one more chunk-increment and state pass, from the initial states.
    if (!recompute) node->starts_ = keep(r.starts);
    if (init) node->init_type = init->scalar_type();
    if (init && recompute) node->init_ = keep_value(*init);
    node->has_prev = Bp.has_value();
    if (Bp) {
      node->Bp_ = keep_value(*Bp);
      node->Up_ = keep_value(*Up);
    }
    torch::autograd::set_history(r.Y, node);
    if (return_state)
      for (Tensor *t : {&r.final_copy, &r.B_last, &r.U_last}) torch::autograd::set_history(*t, node);
  }
  if (!return_state) return std::vector<Tensor>{r.Y};
  return std::vector<Tensor>{r.Y, r.final_copy, r.B_last, r.U_last};
}

// building blocks of the context-parallel mode: fp32 streaming tensors, no autograd
using Parts4 = std::tuple<Tensor, Tensor, Tensor, Tensor>;
Parts4 scan_fwd_parts(const Tensor &U, const Tensor &M, const Tensor &K, const Tensor &B, const Tensor &C,
                         const OptTensor &init, const OptTensor &Bp, const OptTensor &Up, int64_t L) {
  ScanForward r = scan_forward(scan_dims(U, B, L), U, M, K, B, C, init, Bp, Up, true, false, at::kFloat);
  return {r.Y, r.final32, r.starts, r.mch};
}
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> scan_bwd_parts(const Tensor &U, const Tensor &M, const Tensor &K, const Tensor &B, const Tensor &C,
                         const OptTensor &Bp, const OptTensor &Up, const Tensor &starts, const Tensor &mch,
                         const Tensor &final32, const Tensor &dY, const OptTensor &d_final, int64_t L,
                         bool want_initial, bool want_prev, const OptTensor &workspace) {
  std::optional<at::ScalarType> it;
  if (want_initial) it = at::kFloat;
  // (the stage entry points convert the chunk starts to the current kernels' dtype first)
  ScanGrads g = scan_backward(scan_dims(U, B, L, code_of(starts.scalar_type())), U, M, K, B, C, or_undefined(Bp), or_undefined(Up), starts,
                              mch, final32, dY, or_undefined(d_final), it, want_prev && Bp.has_value(), workspace);
  return {g.dU, g.dM, g.dK, g.dB, g.dC, g.d_init, g.dBp, g.dUp};  // (undefined tensors arrive as None)
}

// ------------------------------------------------------------------------------------------------------------
// scan preparation
// ------------------------------------------------------------------------------------------------------------
constexpr int kParamDim = 13;

// Elements between the rows of a (b, T, ...) tensor whose rows are dense inside and equally spaced over (b, T), or 0.
// The stride of an axis of one element means nothing (and contiguous() leaves it as it is), so it is not looked at.
int64_t row_stride(const Tensor &x) {
  int64_t width = 1;
  for (int64_t i = x.dim() - 1; i >= 2; --i) {
    if (x.size(i) != 1 && x.stride(i) != width) return 0;
    width *= x.size(i);
  }
  const int64_t b = x.size(0), T = x.size(1);
  if (b == 1 && T == 1) return width;
  const int64_t s = x.stride(T > 1 ? 1 : 0);
  return s < width || (b > 1 && T > 1 && x.stride(0) != T * s) ? 0 : s;
}
// x itself where its rows are like that, else a copy
Tensor with_rows(const Tensor &x) { return row_stride(x) ? x : x.detach().contiguous(); }

struct PrepConfig {
  int64_t H, N, P;
  bool normalize;
  float dt_min, dt_max, r_min, r_max, theta_bound, k_max, eps;
};
using Hyper = std::tuple<double, double, double, double, double, double, double>;

PrepConfig prep_config(int64_t H, int64_t N, int64_t P, bool normalize, const Hyper &hp) {
  return PrepConfig{H, N, P, normalize, (float)std::get<0>(hp), (float)std::get<1>(hp), (float)std::get<2>(hp),
                    (float)std::get<3>(hp), (float)std::get<4>(hp), (float)std::get<5>(hp), (float)std::get<6>(hp)};
}
slx_prep_shape prep_shape(const PrepConfig &c, int64_t b, int64_t T, int dtype, int64_t vs, int64_t ps, int64_t bs) {
  return slx_prep_shape{(int32_t)b, (int32_t)T, (int32_t)c.H, (int32_t)c.P, (int32_t)c.N, dtype, c.normalize ? 1 : 0,
                        c.dt_min, c.dt_max, c.r_min, c.r_max, c.theta_bound, c.k_max, c.eps, vs, ps, bs};
}

// The nine parameter tensors in one dtype: as they are where they agree, as fp32 copies otherwise.
bool prep_params_plain(const std::vector<Tensor> &pars, bool normalize, const at::Device &dev, int64_t H, int64_t N) {
  const size_t n = normalize ? 9 : 7;
  if (pars.size() < n) return false;
  for (size_t i = 0; i < n; ++i) {
    const Tensor &t = pars[i];
    if (!t.defined() || t.device() != dev || code_of(t.scalar_type()) < 0) return false;
    // biases (H) or (1, H), scales (H, 2, N) or (H, 2 N)
    const int64_t n_dim = t.dim();
    const bool ok = i < 7 ? n_dim >= 1 && t.size(-1) == H && t.numel() == H
                          : t.numel() == 2 * H * N && ((n_dim == 3 && t.size(0) == H && t.size(1) == 2) ||
                                                       (n_dim == 2 && t.size(0) == H));
    if (!ok) return false;
  }
  return true;
}
std::vector<Tensor> uniform_params(const std::vector<Tensor> &pars, bool normalize) {
  const size_t n = normalize ? 9 : 7;
  const at::ScalarType t0 = pars[0].scalar_type();
  bool same = true;
  for (size_t i = 0; i < n; ++i)
    same = same && pars[i].scalar_type() == t0 && pars[i].is_contiguous() && (i < 7 || aligned(pars[i]));
  if (same) return pars;
  std::vector<Tensor> r(pars.size());
  for (size_t i = 0; i < n; ++i) {
    r[i] = pars[i].detach().to(at::kFloat).contiguous();
    if (!aligned(r[i])) r[i] = r[i].clone();
  }
  return r;
}
slx_prep_params params_struct(const std::vector<Tensor> &p, bool normalize) {
  slx_prep_params s{};
  for (int i = 0; i < 7; ++i) s.bias[i] = ptr(p[i]);
  if (normalize) {
    s.b_scale = ptr(p[7]);
    s.c_scale = ptr(p[8]);
  }
  s.dtype = code_of(p[0].scalar_type());
  return s;
}

// The same parameters by value, in one tensor: [scales of B and C,] biases.  What the backward keeps: a program may
// update them before it runs.
Tensor flat_params(const std::vector<Tensor> &p, bool normalize) {
  at::AutoDispatchBelowAutograd no_graph;
  std::vector<Tensor> flat;
  for (int i = normalize ? 7 : 9; i < 9; ++i) flat.push_back(p[i].view({-1}));
  for (int i = 0; i < 7; ++i) flat.push_back(p[i].dim() == 1 ? p[i] : p[i].view({-1}));
  return at::cat(flat);
}
slx_prep_params flat_params_struct(const Tensor &flat, bool normalize, int64_t H, int64_t N) {
  slx_prep_params s{};
  const char *at = static_cast<const char *>(flat.data_ptr());
  const int64_t size = flat.element_size();
  if (normalize) {
    s.b_scale = at;
    s.c_scale = at + 2 * H * N * size;
    at += 4 * H * N * size;
  }
  for (int i = 0; i < 7; ++i) s.bias[i] = at + i * H * size;
  s.dtype = code_of(flat.scalar_type());
  return s;
}

struct PrepBackward : public Node {
  PrepConfig cfg{};
  int64_t b = 0, T = 0;
  std::vector<int64_t> bc_sizes;
  SavedVariable params_, bc_, pars_;  // pars_: the parameters by value, as flat_params lays them out
  std::vector<at::ScalarType> par_types;
  std::string name() const override { return "ScanPrepBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    params_.reset_data();
    bc_.reset_data();
    pars_.reset_data();
  }
  variable_list apply(variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    Tensor params = with_rows(saved(params_)), bc = with_rows(saved(bc_));
    const Tensor pars = saved(pars_);
    const at::ScalarType act = params.scalar_type(), pt = pars.scalar_type();
    const at::Device dev = params.device();
    auto in = [&](size_t i, at::IntArrayRef sizes, at::ScalarType t) {
      return grads[i].defined() ? as_read(grads[i], t) : at::zeros(sizes, at::TensorOptions().dtype(t).device(dev));
    };
    const int64_t H = cfg.H, N = cfg.N, P = cfg.P;
    Tensor dU = in(0, {b, H, T, P}, act), dM = in(1, {b, H, T, 2}, at::kFloat), dK = in(2, {b, H, T, 2, 2}, at::kFloat),
           dB = in(3, {b, H, T, 2 * N}, act), dC = in(4, {b, H, T, 2 * N}, act);
    Tensor d_value = empty({b, T, H * P}, act, dev), d_params = empty({b, T, H * kParamDim}, act, dev);
    Tensor d_bc = empty(bc_sizes, act, dev), d_bias = empty({7, H}, pt, dev), d_bs, d_cs;
    if (cfg.normalize) {
      d_bs = empty({H, 2, N}, pt, dev);
      d_cs = empty({H, 2, N}, pt, dev);
    }
    const slx_prep_shape s = prep_shape(cfg, b, T, code_of(act), H * P, row_stride(params), row_stride(bc));
    const slx_prep_params pp = flat_params_struct(pars, cfg.normalize, H, N);
    const size_t nbytes = slx_scanprep_bwd_workspace_bytes(&s);
    Tensor ws = empty({(int64_t)nbytes}, at::kByte, dev);
    {
      c10::cuda::CUDAGuard guard(dev);
      check(slx_scanprep_bwd_params(&s, ptr(params), ptr(bc), &pp, ptr(dU), fptr(dM), fptr(dK), ptr(dB), ptr(dC),
                                    ptr(d_value), ptr(d_params), ptr(d_bc), ptr(d_bias), ptr(d_bs), ptr(d_cs), ptr(ws),
                                    nbytes, stream_of(dev)),
            "scanprep backward");
    }
    variable_list out(12);
    out[0] = d_value;
    out[1] = d_params;
    out[2] = d_bc;
    for (int i = 0; i < 7; ++i) {
      if (!task_should_compute_output(3 + i)) continue;
      Tensor g = d_bias.select(0, i);
      out[3 + i] = par_types[i] == pt ? g : g.to(par_types[i]);
    }
    if (cfg.normalize) {
      out[10] = par_types[7] == pt ? d_bs : d_bs.to(par_types[7]);
      out[11] = par_types[8] == pt ? d_cs : d_cs.to(par_types[8]);
    }
    return out;
  }
};

// value (b,T,H*P), params (b,T,H*13), bc (b,T,H,4,N); pars = the seven biases, then b_scale, c_scale
std::optional<std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>> scanprep(const Tensor &value, const Tensor &params, const Tensor &bc, int64_t H, int64_t N, int64_t P,
                    bool normalize, const Hyper &hp, const std::vector<Tensor> &pars) {
  if (!value.is_cuda() || value.dim() != 3 || params.dim() != 3 || bc.dim() != 5) return std::nullopt;
  const at::Device dev = value.device();
  const at::ScalarType act = value.scalar_type();
  const int64_t b = value.size(0), T = value.size(1);
  if (b == 0 || T == 0 || H <= 0 || N <= 0 || P <= 0 || code_of(act) < 0) return std::nullopt;
  const int64_t vsz[3] = {b, T, H * P}, psz[3] = {b, T, H * kParamDim}, bsz[5] = {b, T, H, 4, N};
  if (!shaped(value, vsz) || !shaped(params, psz) || !shaped(bc, bsz)) return std::nullopt;
  if (params.scalar_type() != act || bc.scalar_type() != act || params.device() != dev || bc.device() != dev)
    return std::nullopt;
  if (!prep_params_plain(pars, normalize, dev, H, N)) return std::nullopt;
  refuse_tangents(value, params, bc);
  for (const Tensor &t : pars) refuse_tangent(t);
  const Tensor v = with_rows(value), p = with_rows(params), c = with_rows(bc);
  const PrepConfig cfg = prep_config(H, N, P, normalize, hp);
  Tensor U = empty({b, H, T, P}, act, dev), M = empty({b, H, T, 2}, at::kFloat, dev),
         K = empty({b, H, T, 2, 2}, at::kFloat, dev), B = empty({b, H, T, 2 * N}, act, dev),
         C = empty({b, H, T, 2 * N}, act, dev);
  const slx_prep_shape s = prep_shape(cfg, b, T, code_of(act), row_stride(v), row_stride(p), row_stride(c));
  const std::vector<Tensor> up = uniform_params(pars, normalize);
  const slx_prep_params pp = params_struct(up, normalize);
  {
    c10::cuda::CUDAGuard guard(dev);
    check(slx_scanprep_fwd_params(&s, ptr(v), ptr(p), ptr(c), &pp, ptr(U), fptr(M), fptr(K), ptr(B), ptr(C),
                                  stream_of(dev)),
          "scanprep forward");
  }
  bool grad = torch::autograd::compute_requires_grad(value, params, bc);
  if (!grad && at::GradMode::is_enabled())
    for (const Tensor &t : pars) grad = grad || (t.defined() && t.requires_grad());
  if (grad) {
    torch::autograd::edge_list edges = torch::autograd::collect_next_edges(value, params, bc);
    for (size_t i = 0; i < 9; ++i)
      edges.push_back(i < pars.size() && pars[i].defined() ? torch::autograd::impl::gradient_edge(pars[i])
                                                           : torch::autograd::Edge());
    auto node = make_node<PrepBackward>(std::move(edges));
    node->cfg = cfg;
    node->b = b;
    node->T = T;
    node->bc_sizes.assign(bsz, bsz + 5);
    node->params_ = keep(p);
    node->bc_ = keep(c);
    node->pars_ = keep(flat_params(up, normalize));
    for (size_t i = 0; i < (normalize ? 9 : 7); ++i) node->par_types.push_back(pars[i].scalar_type());
    for (Tensor *t : {&U, &M, &K, &B, &C}) torch::autograd::set_history(*t, node);
  }
  return std::make_tuple(U, M, K, B, C);
}

// ------------------------------------------------------------------------------------------------------------
// one-token decode step
// ------------------------------------------------------------------------------------------------------------
// value, gate (b,H,P), params (b,H,13), bc (b,H,4,N): rows dense inside a batch, any batch stride.
bool dense_batch(const Tensor &x, int64_t inner) {
  int64_t want = 1;
  for (int64_t i = x.dim() - 1; i >= 1; --i) {
    if (x.size(i) != 1 && x.stride(i) != want) return false;
    want *= x.size(i);
  }
  return x.size(0) == 1 || x.stride(0) >= inner;
}
std::optional<Parts4> decode_step(const Tensor &value, const Tensor &params, const Tensor &bc, const Tensor &gate,
                       const Tensor &skip, const OptTensor &state_in, const OptTensor &Bp, const OptTensor &Up,
                       bool normalize, const Hyper &hp, const std::vector<Tensor> &pars, const OptTensor &state_out_in,
                       const OptTensor &b_last_in, const OptTensor &u_last_in) {
  if (!value.is_cuda() || value.dim() != 3 || bc.dim() != 4) return std::nullopt;
  const at::Device dev = value.device();
  const at::ScalarType act = value.scalar_type();
  const int64_t b = value.size(0), H = value.size(1), P = value.size(2), N = bc.size(3);
  if (code_of(act) < 0 || b == 0 || H == 0 || P == 0 || N == 0) return std::nullopt;
  const int64_t vsz[3] = {b, H, P}, psz[3] = {b, H, kParamDim}, bsz[4] = {b, H, 4, N}, ssz[4] = {b, H, P, 2 * N},
                lsz[3] = {b, H, 2 * N};
  if (!shaped(params, psz) || !shaped(bc, bsz) || !shaped(gate, vsz) || skip.numel() != H * P) return std::nullopt;
  for (const Tensor *t : {&params, &bc, &gate, &skip})
    if (t->device() != dev) return std::nullopt;
  for (const Tensor *t : {&params, &bc, &gate})
    if (t->scalar_type() != act) return std::nullopt;
  if (code_of(skip.scalar_type()) < 0 || !skip.is_contiguous()) return std::nullopt;
  if (!dense_batch(value, H * P) || !dense_batch(params, H * kParamDim) || !dense_batch(bc, H * 4 * N) ||
      !dense_batch(gate, H * P))
    return std::nullopt;
  if (!prep_params_plain(pars, normalize, dev, H, N)) return std::nullopt;
  auto fits = [&](const OptTensor &t, at::IntArrayRef sz, at::ScalarType ty) {
    return !t || (is(*t, dev) && shaped(*t, sz) && t->is_contiguous() && t->scalar_type() == ty);
  };
  if (Bp.has_value() != Up.has_value()) return std::nullopt;
  if (!fits(state_in, ssz, at::kFloat) || !fits(Bp, lsz, act) || !fits(Up, vsz, act) ||
      !fits(state_out_in, ssz, at::kFloat) || !fits(b_last_in, lsz, act) || !fits(u_last_in, vsz, act))
    return std::nullopt;
  Tensor out = empty({b, H * P}, act, dev);
  Tensor state_out = state_out_in ? *state_out_in : empty(ssz, at::kFloat, dev);
  Tensor b_last = b_last_in ? *b_last_in : empty(lsz, act, dev);
  Tensor u_last = u_last_in ? *u_last_in : empty(vsz, act, dev);
  const PrepConfig c = prep_config(H, N, P, normalize, hp);
  const slx_decode_shape s{(int32_t)b, (int32_t)H, (int32_t)P, (int32_t)N, code_of(act), normalize ? 1 : 0,
                           c.dt_min, c.dt_max, c.r_min, c.r_max, c.theta_bound, c.k_max, c.eps};
  const std::vector<Tensor> up = uniform_params(pars, normalize);
  const slx_prep_params pp = params_struct(up, normalize);
  const int64_t strides[4] = {value.stride(0), params.stride(0), bc.stride(0), gate.stride(0)};
  c10::cuda::CUDAGuard guard(dev);
  check(slx_decode_step_params(&s, ptr(value), ptr(params), ptr(bc), ptr(gate), strides, ptr(skip),
                               code_of(skip.scalar_type()), &pp, static_cast<const float *>(cptr(state_in)), cptr(Bp),
                               cptr(Up), ptr(out), fptr(state_out), ptr(b_last), ptr(u_last), stream_of(dev)),
        "decode step");
  return Parts4{out, state_out, b_last, u_last};
}

// ------------------------------------------------------------------------------------------------------------
// causal conv
// ------------------------------------------------------------------------------------------------------------
Tensor as_type(const Tensor &t, at::ScalarType ty) {
  return (t.scalar_type() == ty ? t : t.detach().to(ty)).contiguous();
}

struct ConvBackward : public Node {
  bool silu = false, has_bias = false, has_state = false;
  at::ScalarType w_type, b_type, s_type;
  SavedVariable x_, w_, bias_, state_;
  std::string name() const override { return "CConv1dBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable *v : {&x_, &w_, &bias_, &state_}) v->reset_data();
  }
  variable_list apply(variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    Tensor x = saved(x_);
    const at::ScalarType act = x.scalar_type();
    const at::Device dev = x.device();
    Tensor w = saved(w_), bias, state;  // in x's dtype
    if (has_bias) bias = saved(bias_);
    if (has_state) state = saved(state_);
    const int64_t b = x.size(0), T = x.size(1), C = x.size(2), W = w.size(1);
    Tensor dy = grads[0].defined() ? as_read(grads[0], act)
                                   : at::zeros({b, T, C}, at::TensorOptions().dtype(act).device(dev));
    Tensor dn;
    if (grads[1].defined()) dn = as_type(grads[1], act);
    // the fp32 sums are rounded once, to the dtype of the parameter they belong to
    const bool one_type = (!has_bias || b_type == w_type) && (!has_state || s_type == w_type) && code_of(w_type) >= 0;
    const at::ScalarType gt = one_type ? w_type : at::kFloat;
    Tensor dx = empty({b, T, C}, act, dev), dw = empty({C, W}, gt, dev), db, ds;
    if (has_bias) db = empty({C}, gt, dev);
    if (has_state) ds = empty({b, C, W - 1}, gt, dev);
    const slx_conv_shape s{(int32_t)b, (int32_t)T, (int32_t)C, (int32_t)W, code_of(act), silu ? 1 : 0,
                           std::max<int64_t>(x.stride(1), C), x.stride(0)};
    const size_t nbytes = slx_cconv1d_bwd_workspace_bytes(&s);
    Tensor ws = empty({(int64_t)nbytes}, at::kByte, dev);
    {
      c10::cuda::CUDAGuard guard(dev);
      check(slx_cconv1d_bwd_as(&s, ptr(x), ptr(w), ptr(bias), ptr(state), ptr(dy), ptr(dn), ptr(dx), ptr(dw), ptr(db),
                               ptr(ds), code_of(gt), ptr(ws), nbytes, stream_of(dev)),
            "cconv1d backward");
    }
    auto back = [&](const Tensor &t, at::ScalarType ty) { return t.defined() && ty != gt ? t.to(ty) : t; };
    return {dx, back(dw, w_type), back(db, b_type), back(ds, s_type)};
  }
};

std::optional<std::tuple<Tensor, Tensor>> cconv1d(const Tensor &x_in, const Tensor &weight, const OptTensor &bias, const OptTensor &state, bool silu) {
  if (!x_in.is_cuda() || x_in.dim() != 3 || weight.dim() != 2) return std::nullopt;
  const at::Device dev = x_in.device();
  const at::ScalarType act = x_in.scalar_type();
  const int64_t b = x_in.size(0), T = x_in.size(1), C = x_in.size(2), W = weight.size(1);
  if (code_of(act) < 0 || b == 0 || T == 0 || C == 0 || W < 2 || W > 4 || weight.size(0) != C || weight.device() != dev)
    return std::nullopt;
  if (bias && (!is(*bias, dev) || bias->numel() != C)) return std::nullopt;
  const int64_t ssz[3] = {b, C, W - 1};
  if (state && (!is(*state, dev) || !shaped(*state, ssz))) return std::nullopt;
  refuse_tangents(x_in, weight, or_undefined(bias), or_undefined(state));
  // a column slice of a wider matrix is read where it is; anything else is copied
  const bool rows = x_in.stride(2) == 1 && (T == 1 || x_in.stride(1) >= C);
  const Tensor x = rows ? x_in : x_in.detach().contiguous();
  const Tensor w = as_type(weight, act), bs = bias ? as_type(*bias, act) : Tensor(),
               st = state ? as_type(*state, act) : Tensor();
  Tensor y = empty({b, T, C}, act, dev), nxt = empty(ssz, act, dev);
  const slx_conv_shape s{(int32_t)b, (int32_t)T, (int32_t)C, (int32_t)W, code_of(act), silu ? 1 : 0,
                         std::max<int64_t>(x.stride(1), C), x.stride(0)};
  {
    c10::cuda::CUDAGuard guard(dev);
    check(slx_cconv1d_fwd(&s, ptr(x), ptr(w), ptr(bs), ptr(st), ptr(y), ptr(nxt), stream_of(dev)), "cconv1d forward");
  }
  if (torch::autograd::compute_requires_grad(x_in, weight, or_undefined(bias), or_undefined(state))) {
    auto node = make_node<ConvBackward>(
        torch::autograd::collect_next_edges(x_in, weight, or_undefined(bias), or_undefined(state)));
    node->silu = silu;
    node->has_bias = bias.has_value();
    node->has_state = state.has_value();
    node->w_type = weight.scalar_type();
    if (bias) node->b_type = bias->scalar_type();
    if (state) node->s_type = state->scalar_type();
    node->x_ = keep(x);
    node->w_ = keep(w);
    node->bias_ = keep(bs);
    node->state_ = keep(st);
    torch::autograd::set_history(y, node);
    torch::autograd::set_history(nxt, node);
  }
  return std::make_tuple(y, nxt);
}

// x (b,C), rolling state (b,C,W-1) -> (y, next state); `inplace`: the state tensor itself is rolled
std::optional<std::tuple<Tensor, Tensor>> cconv1d_update(const Tensor &x_in, const Tensor &weight, const OptTensor &bias, const OptTensor &state,
                          bool silu, bool inplace) {
  if (!x_in.is_cuda() || x_in.dim() != 2 || weight.dim() != 2) return std::nullopt;
  const at::Device dev = x_in.device();
  const at::ScalarType act = x_in.scalar_type();
  const int64_t b = x_in.size(0), C = x_in.size(1), W = weight.size(1);
  if (code_of(act) < 0 || b == 0 || C == 0 || W < 2 || W > 4 || weight.size(0) != C || weight.device() != dev)
    return std::nullopt;
  if (bias && (!is(*bias, dev) || bias->numel() != C)) return std::nullopt;
  const int64_t ssz[3] = {b, C, W - 1};
  if (state && (!is(*state, dev) || !shaped(*state, ssz))) return std::nullopt;
  if (inplace && (!state || state->scalar_type() != act || !state->is_contiguous())) return std::nullopt;
  const Tensor x = x_in.stride(1) == 1 ? x_in : x_in.contiguous();
  const Tensor w = as_type(weight, act), bs = bias ? as_type(*bias, act) : Tensor(),
               st = state ? as_type(*state, act) : Tensor();
  Tensor y = empty({b, C}, act, dev), nxt = inplace ? *state : empty(ssz, act, dev);
  const slx_conv_shape s{(int32_t)b, 1, (int32_t)C, (int32_t)W, code_of(act), silu ? 1 : 0, C, x.stride(0)};
  c10::cuda::CUDAGuard guard(dev);
  check(slx_cconv1d_update(&s, ptr(x), ptr(w), ptr(bs), ptr(st), ptr(y), ptr(nxt), stream_of(dev)), "cconv1d update");
  return std::make_tuple(y, nxt);
}

// ------------------------------------------------------------------------------------------------------------
// skip and gate
// ------------------------------------------------------------------------------------------------------------
// Strides of the gate over (tokens, batch): it may be a column slice of a wider row, with rows on 16-byte boundaries.
// As in row_stride, an axis of one element has the stride that a dense tensor would have.
struct GateRows {
  int64_t token, batch;
};
GateRows gate_rows(const Tensor &g) {
  GateRows r;
  r.token = g.size(1) > 1 ? g.stride(1) : g.size(2);
  r.batch = g.size(0) > 1 ? g.stride(0) : g.size(1) * r.token;
  return r;
}
Tensor with_gate_rows(const Tensor &g) {
  const GateRows r = gate_rows(g);
  const bool ok = g.stride(2) == 1 && r.token % 8 == 0 && r.batch % 8 == 0 && r.token >= g.size(2) && aligned(g);
  if (ok) return g;
  Tensor c = g.detach().contiguous();
  return aligned(c) ? c : c.clone();
}

struct GateBackward : public Node {
  SavedVariable y_, u_, gate_, skip_;
  at::ScalarType u_type, g_type, s_type;
  std::vector<int64_t> skip_sizes;
  std::string name() const override { return "GateSkipBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable *v : {&y_, &u_, &gate_, &skip_}) v->reset_data();
  }
  variable_list apply(variable_list &&grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return variable_list(4);
    Tensor y = saved(y_), u = saved(u_), gate = with_gate_rows(saved(gate_)), skip = saved(skip_);
    const int64_t b = y.size(0), H = y.size(1), T = y.size(2), P = y.size(3);
    const at::ScalarType act = y.scalar_type();
    const at::Device dev = y.device();
    Tensor go = as_read(grads[0], act);
    const at::ScalarType kt = code_of(s_type) >= 0 ? s_type : at::kFloat;
    Tensor dy = empty(y.sizes(), act, dev), du = empty(y.sizes(), act, dev), dg = empty({b, T, H * P}, act, dev),
           dsk = empty(skip_sizes, kt, dev);
    const slx_glue_shape s{(int32_t)b, (int32_t)T, (int32_t)H, (int32_t)P, code_of(act), gate_rows(gate).token,
                           gate_rows(gate).batch};
    const size_t nbytes = slx_gate_skip_bwd_workspace_bytes(&s);
    Tensor ws = empty({(int64_t)nbytes}, at::kByte, dev);
    {
      c10::cuda::CUDAGuard guard(dev);
      check(slx_gate_skip_bwd_as(&s, ptr(y), ptr(u), ptr(gate), ptr(skip), code_of(skip.scalar_type()), ptr(go), ptr(dy),
                                 ptr(du), ptr(dg), ptr(dsk), ptr(ws), nbytes, stream_of(dev)),
            "gate_skip backward");
    }
    auto back = [](const Tensor &t, at::ScalarType ty) { return t.scalar_type() == ty ? t : t.to(ty); };
    return {dy, back(du, u_type), back(dg, g_type), back(dsk, s_type)};
  }
};

OptTensor gate_skip(const Tensor &y_in, const Tensor &u_in, const Tensor &gate_in, const Tensor &skip_in) {
  if (!y_in.is_cuda() || y_in.dim() != 4 || gate_in.dim() != 3) return std::nullopt;
  const at::Device dev = y_in.device();
  const at::ScalarType act = y_in.scalar_type();
  const int64_t b = y_in.size(0), H = y_in.size(1), T = y_in.size(2), P = y_in.size(3);
  const int64_t gsz[3] = {b, T, H * P};
  if (code_of(act) < 0 || b == 0 || T == 0 || H == 0 || P == 0 || P % 8 != 0 || !shaped(u_in, y_in.sizes()) ||
      !shaped(gate_in, gsz) || skip_in.numel() != H * P)
    return std::nullopt;
  for (const Tensor *t : {&u_in, &gate_in, &skip_in})
    if (t->device() != dev) return std::nullopt;
  refuse_tangents(y_in, u_in, gate_in, skip_in);
  auto plain = [&](const Tensor &t) {
    Tensor r = as_type(t, act);
    return aligned(r) ? r : r.clone();
  };
  const Tensor y = plain(y_in), u = plain(u_in);
  const Tensor gate = with_gate_rows(gate_in.scalar_type() == act ? gate_in : gate_in.detach().to(act));
  Tensor skip = skip_in;
  if (code_of(skip.scalar_type()) < 0) skip = skip.detach().to(at::kFloat);
  if (!skip.is_contiguous()) skip = skip.detach().contiguous();
  Tensor out = empty(gsz, act, dev);
  const slx_glue_shape s{(int32_t)b, (int32_t)T, (int32_t)H, (int32_t)P, code_of(act), gate_rows(gate).token,
                         gate_rows(gate).batch};
  {
    c10::cuda::CUDAGuard guard(dev);
    check(slx_gate_skip_fwd_as(&s, ptr(y), ptr(u), ptr(gate), ptr(skip), code_of(skip.scalar_type()), ptr(out),
                               stream_of(dev)),
          "gate_skip forward");
  }
  if (torch::autograd::compute_requires_grad(y_in, u_in, gate_in, skip_in)) {
    auto node = make_node<GateBackward>(torch::autograd::collect_next_edges(y_in, u_in, gate_in, skip_in));
    node->y_ = keep(y);
    node->u_ = keep(u);
    node->gate_ = keep(gate);
    node->skip_ = keep_value(skip);
    node->u_type = u_in.scalar_type();
    node->g_type = gate_in.scalar_type();
    node->s_type = skip_in.scalar_type();
    node->skip_sizes = skip_in.sizes().vec();
    torch::autograd::set_history(out, node);
  }
  return out;
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.def("v2x2ssd", torch::wrap_pybind_function_no_gil(&v2x2ssd));
  m.def("scan_fwd_parts", torch::wrap_pybind_function_no_gil(&scan_fwd_parts));
  m.def("scan_bwd_parts", torch::wrap_pybind_function_no_gil(&scan_bwd_parts));
  m.def("scanprep", torch::wrap_pybind_function_no_gil(&scanprep));
  m.def("row_stride", torch::wrap_pybind_function(&row_stride));
  m.def("decode_step", torch::wrap_pybind_function_no_gil(&decode_step));
  m.def("cconv1d", torch::wrap_pybind_function_no_gil(&cconv1d));
  m.def("cconv1d_update", torch::wrap_pybind_function_no_gil(&cconv1d_update));
  m.def("gate_skip", torch::wrap_pybind_function_no_gil(&gate_skip));
}
