// Host path of the torch operators: argument checks, allocation, the library calls and the autograd nodes in native code.
//
// The small calls (a decode step, a short prompt, a correctness run) take less time on the GPU than a Python autograd
// function and a foreign-function call with twenty arguments take on the host, so the whole path from the Python
// signature to the launches is here.  Every operator returns None for arguments that are not of its plain form; the
// Python wrapper then repeats the checks one by one and raises the error that says which one failed.
// No kernel and no arithmetic lives here: everything goes through the C ABI of include/gla_b200.h.
#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/cuda/CUDAFunctions.h>
#include <cmath>
#include "../../include/gla_b200.h"

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

PyObject* g_error = nullptr;      // gla_jax_b200._lib.GlaError

[[noreturn]] void raise(const std::string& msg) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(g_error ? g_error : PyExc_RuntimeError, msg.c_str());
  python_error e;
  e.persist();
  throw e;
}
void check(int status, const char* what) {
  if (status == 0) return;
  std::string m = std::string(what) + ": " + gla_status_string(status);
  if (status == GLA_ERR_LAUNCH) m += " (cudaError " + std::to_string(gla_last_cuda_error()) + ")";
  raise(m);
}
int dt_of(const Tensor& t) {
  return t.scalar_type() == torch::kFloat32 ? GLA_F32 : t.scalar_type() == torch::kBFloat16 ? GLA_BF16 : -1;
}
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* stream_of(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
bool here(const Tensor& t) { return t.is_cuda() && t.device().index() == c10::cuda::current_device(); }
Tensor bytes(const Tensor& like, size_t n) {
  return n ? torch::empty({(int64_t)n}, like.options().dtype(torch::kUInt8)) : Tensor();
}
// as much as the faster form of a call takes, or `least` where that does not fit the device (0 bytes: undefined)
Tensor bytes_or(const Tensor& like, size_t n, size_t least) {
  try {
    return bytes(like, n);
  } catch (const c10::OutOfMemoryError&) {
    if (n <= least) throw;
    return bytes(like, least);
  }
}
size_t size_of(const Tensor& t) { return t.defined() ? (size_t)t.numel() : 0; }
Tensor f32(const Tensor& g) { return (g.scalar_type() == torch::kFloat32 ? g : g.to(torch::kFloat32)).contiguous(); }
bool wants_any(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts) if (t->requires_grad()) return true;
  return false;
}
bool wants_grad(std::initializer_list<const Tensor*> ts) { return torch::GradMode::is_enabled() && wants_any(ts); }
// There is no forward-mode formula: refuse a dual tensor (which need not require a gradient) instead of returning outputs
// without a tangent.
void no_forward_mode(const char* what, std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->defined() && t->_fw_grad(/*level=*/0).defined())
      TORCH_CHECK_NOT_IMPLEMENTED(false, what, ": forward-mode differentiation (jvp) is not implemented");
}
// a gradient that may be absent, in the dtype and layout the library takes
Tensor grad_or_zeros(const Tensor& g, const Tensor& like) {
  return g.defined() ? g.to(like.scalar_type()).contiguous() : torch::zeros(like.sizes(), like.options().requires_grad(false));
}

struct Dims { int64_t B, T, H, D; int dt; };
// (T,H,D) or (B,T,H,D) arrays of one dtype with a matching state; false: let the wrapper say what is wrong
bool dims_of(const Tensor& h, const Tensor& g, const Tensor& v, const Tensor& k, const Tensor& q, Dims& d) {
  if (!v.defined() || !here(v) || (v.dim() != 3 && v.dim() != 4)) return false;
  for (const Tensor* t : {&h, &g, &k, &q}) if (!t->defined() || t->device() != v.device()) return false;
  if (g.sizes() != v.sizes() || k.sizes() != v.sizes() || q.sizes() != v.sizes()) return false;
  d.dt = dt_of(v);
  if (d.dt < 0 || k.scalar_type() != v.scalar_type() || q.scalar_type() != v.scalar_type() || h.scalar_type() != v.scalar_type()) return false;
  const int b = v.dim() == 4;
  d.B = b ? v.size(0) : 1; d.T = v.size(b); d.H = v.size(b + 1); d.D = v.size(b + 2);
  if (h.dim() != 3 + b || (b && h.size(0) != d.B)) return false;
  return h.size(b) == d.H && h.size(b + 1) == d.D && h.size(b + 2) == d.D;
}
std::string shape_text(const Dims& d, int64_t chunk, const Tensor& v) {
  return "T=" + std::to_string(d.T) + " H=" + std::to_string(d.H) + " D=" + std::to_string(d.D) + " chunk=" + std::to_string(chunk) +
         " dtype=" + (d.dt == GLA_F32 ? "torch.float32" : "torch.bfloat16");
}

// ---- chunk_gla ---------------------------------------------------------------------------------------------------
variable_list chunk_forward(const Dims& d, const Tensor& h, const Tensor& g, const Tensor& v, const Tensor& k, const Tensor& q,
                            int64_t chunk, int64_t impl, bool residuals) {
  size_t n = gla_chunk_fwd_workspace_bytes(d.B, d.T, d.H, d.D, chunk, d.dt, (int)impl);
  if (n == 0) raise("chunk_gla: unsupported configuration " + shape_text(d, chunk, v));
  if (residuals) n = gla_chunk_training_workspace_bytes(d.B, d.T, d.H, d.D, chunk, d.dt, (int)impl, 0);
  Tensor saved = residuals ? bytes(v, gla_chunk_saved_bytes(d.B, d.T, d.H, d.D, chunk, d.dt, (int)impl)) : Tensor();
  Tensor ws = bytes(v, n), hf = torch::empty_like(h), out = torch::empty_like(v);
  check(gla_chunk_fwd(stream_of(v), d.B, d.T, d.H, d.D, chunk, d.dt, (int)impl, ptr(h), (const float*)ptr(g), ptr(v), ptr(k), ptr(q),
                      ptr(hf), ptr(out), ptr(saved), ptr(ws), n), "gla_chunk_fwd");
  return {hf, out, saved};
}
variable_list chunk_backward(const Dims& d, const Tensor& g, const Tensor& v, const Tensor& k, const Tensor& q, const Tensor& saved,
                             const Tensor& dhf0, const Tensor& dout0, int64_t chunk, int64_t impl) {
  std::vector<int64_t> hs(v.sizes().begin(), v.sizes().end());        // (B,) H, D, D
  hs[hs.size() - 3] = d.H; hs[hs.size() - 2] = d.D;
  Tensor dh = torch::empty(hs, v.options());
  Tensor dhf = grad_or_zeros(dhf0, dh), dout = grad_or_zeros(dout0, v);
  Tensor dg = torch::empty_like(g), dv = torch::empty_like(v), dk = torch::empty_like(k), dq = torch::empty_like(q);
  const size_t n = gla_chunk_training_workspace_bytes(d.B, d.T, d.H, d.D, chunk, d.dt, (int)impl, 1);
  Tensor ws = bytes(v, n);
  check(gla_chunk_bwd(stream_of(v), d.B, d.T, d.H, d.D, chunk, d.dt, (int)impl, (const float*)ptr(g), ptr(v), ptr(k), ptr(q), ptr(saved),
                      ptr(dhf), ptr(dout), ptr(dh), (float*)ptr(dg), ptr(dv), ptr(dk), ptr(dq), ptr(ws), n), "gla_chunk_bwd");
  return {dh, dg, dv, dk, dq};
}
struct ChunkFn : torch::autograd::Function<ChunkFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& h0, const Tensor& g0, const Tensor& v0, const Tensor& k0,
                               const Tensor& q0, int64_t B, int64_t T, int64_t H, int64_t D, int64_t dt, int64_t chunk, int64_t impl) {
    const Dims d{B, T, H, D, (int)dt};
    Tensor h = h0.contiguous(), g = f32(g0), v = v0.contiguous(), k = k0.contiguous(), q = q0.contiguous();
    variable_list r = chunk_forward(d, h, g, v, k, q, chunk, impl, true);
    ctx->save_for_backward({g, v, k, q, r[2]});
    ctx->set_materialize_grads(false);
    ctx->saved_data["d"] = std::vector<int64_t>{B, T, H, D, dt, chunk, impl, (int64_t)g0.scalar_type()};
    return {r[0], r[1]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto a = ctx->saved_data["d"].toIntVector();
    const variable_list s = ctx->get_saved_variables();
    const Tensor &g = s[0], &v = s[1], &k = s[2], &q = s[3];
    const int dt = (int)a[4], impl = (int)a[6];
    variable_list r = chunk_backward(Dims{a[0], a[1], a[2], a[3], dt}, g, v, k, q, s[4], grads[0], grads[1], a[5], impl);
    const auto gt = (torch::ScalarType)a[7];
    if (gt != torch::kFloat32) r[1] = r[1].to(gt);
    r.resize(12);
    return r;
  }
};
std::optional<std::tuple<Tensor, Tensor>> chunk_gla(const Tensor& h, const Tensor& g, const Tensor& v, const Tensor& k, const Tensor& q,
                                                    int64_t chunk, int64_t impl) {
  Dims d;
  if (!dims_of(h, g, v, k, q, d) || chunk <= 0 || (chunk & (chunk - 1)) || d.T % chunk) return std::nullopt;
  no_forward_mode("chunk_gla", {&h, &g, &v, &k, &q});
  if (wants_grad({&h, &g, &v, &k, &q})) {
    variable_list r = ChunkFn::apply(h, g, v, k, q, d.B, d.T, d.H, d.D, d.dt, chunk, impl);
    return std::make_tuple(r[0], r[1]);
  }
  variable_list r = chunk_forward(d, h.contiguous(), f32(g), v.contiguous(), k.contiguous(), q.contiguous(), chunk, impl, false);
  return std::make_tuple(r[0], r[1]);
}

// ---- recurrent_gla -------------------------------------------------------------------------------------------------
variable_list recurrent_forward(const Dims& d, const Tensor& h, const Tensor& g, const Tensor& v, const Tensor& k, const Tensor& q,
                                bool reverse, bool out_f32) {
  Tensor hf = torch::empty_like(h), out = torch::empty(v.sizes(), v.options().dtype(out_f32 ? torch::kFloat32 : v.scalar_type()));
  Tensor ws = bytes_or(v, gla_recurrent_fwd_workspace_bytes(d.B, d.T, d.H, d.D, d.dt), 0);
  check(gla_recurrent_fwd_ws(stream_of(v), d.B, d.T, d.H, d.D, d.dt, ptr(h), (const float*)ptr(g), ptr(v), ptr(k), ptr(q), ptr(hf),
                             ptr(out), dt_of(out), reverse, ptr(ws), size_of(ws)), "gla_recurrent_fwd_ws");
  return {hf, out};
}
struct RecurrentFn : torch::autograd::Function<RecurrentFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& h0, const Tensor& g0, const Tensor& v0, const Tensor& k0,
                               const Tensor& q0, int64_t B, int64_t T, int64_t H, int64_t D, int64_t dt, bool reverse, bool out_f32) {
    const Dims d{B, T, H, D, (int)dt};
    Tensor h = h0.contiguous(), g = f32(g0), v = v0.contiguous(), k = k0.contiguous(), q = q0.contiguous();
    variable_list r = recurrent_forward(d, h, g, v, k, q, reverse, out_f32);
    ctx->save_for_backward({h, g, v, k, q});
    ctx->set_materialize_grads(false);
    ctx->saved_data["d"] = std::vector<int64_t>{B, T, H, D, dt, reverse, (int64_t)g0.scalar_type(), (int64_t)r[1].scalar_type()};
    return r;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto a = ctx->saved_data["d"].toIntVector();
    const variable_list s = ctx->get_saved_variables();
    const Tensor &h = s[0], &g = s[1], &v = s[2], &k = s[3], &q = s[4];
    Tensor dhf = grad_or_zeros(grads[0], h);
    Tensor dout = grads[1].defined() ? grads[1].contiguous() : torch::zeros(v.sizes(), v.options().dtype((torch::ScalarType)a[7]));
    if (dt_of(dout) < 0) dout = dout.to(torch::kFloat32);
    Tensor dh = torch::empty_like(h), dg = torch::empty_like(g), dv = torch::empty_like(v), dk = torch::empty_like(k), dq = torch::empty_like(q);
    const auto n = [&](int least) { return gla_recurrent_bwd_workspace_bytes_dout(a[0], a[1], a[2], a[3], (int)a[4], dt_of(dout), least); };
    Tensor ws = bytes_or(v, n(0), n(1));
    check(gla_recurrent_bwd(stream_of(v), a[0], a[1], a[2], a[3], (int)a[4], ptr(h), (const float*)ptr(g), ptr(v), ptr(k), ptr(q), ptr(dhf),
                            ptr(dout), dt_of(dout), ptr(dh), (float*)ptr(dg), ptr(dv), ptr(dk), ptr(dq), (int)a[5], ptr(ws), size_of(ws)),
          "gla_recurrent_bwd");
    const auto gt = (torch::ScalarType)a[6];
    variable_list r{dh, gt == torch::kFloat32 ? dg : dg.to(gt), dv, dk, dq};
    r.resize(12);
    return r;
  }
};
std::optional<std::tuple<Tensor, Tensor>> recurrent_gla(const Tensor& h, const Tensor& g, const Tensor& v, const Tensor& k,
                                                        const Tensor& q, bool reverse, bool out_f32) {
  Dims d;
  if (!dims_of(h, g, v, k, q, d)) return std::nullopt;
  no_forward_mode("recurrent_gla", {&h, &g, &v, &k, &q});
  variable_list r = wants_grad({&h, &g, &v, &k, &q})
                        ? RecurrentFn::apply(h, g, v, k, q, d.B, d.T, d.H, d.D, d.dt, reverse, out_f32)
                        : recurrent_forward(d, h.contiguous(), f32(g), v.contiguous(), k.contiguous(), q.contiguous(), reverse, out_f32);
  return std::make_tuple(r[0], r[1]);
}

// ---- chunk_gla over packed sequences ---------------------------------------------------------------------------------
// Offsets either in host memory (any rising sequence) or as a CUDA int32 tensor (multiples of the chunk).
struct PackedFn : torch::autograd::Function<PackedFn> {
  static variable_list run(const Dims& d, int64_t nseq, const Tensor& h, const Tensor& g, const Tensor& v, const Tensor& k, const Tensor& q,
                           const Tensor& offsets, int64_t chunk, bool residuals) {
    Tensor hf = torch::empty_like(h), out = torch::empty_like(v);
    void* st = stream_of(v);
    if (!offsets.is_cuda()) {
      const int32_t* cu = offsets.data_ptr<int32_t>();
      const size_t n = gla_chunk_ragged_workspace_bytes(d.H, d.D, d.dt, nseq, cu, 0);
      if (n == 0) raise("chunk_gla_packed: unsupported configuration " + shape_text(d, chunk, v));
      Tensor saved = residuals ? bytes(v, gla_chunk_ragged_saved_bytes(d.H, d.D, d.dt, nseq, cu)) : Tensor(), ws = bytes(v, n);
      check(gla_chunk_fwd_ragged(st, d.T, d.H, d.D, d.dt, nseq, cu, ptr(h), (const float*)ptr(g), ptr(v), ptr(k), ptr(q), ptr(hf), ptr(out),
                                 ptr(saved), ptr(ws), n), "gla_chunk_fwd_ragged");
      return {hf, out, saved};
    }
    const size_t n = gla_chunk_fwd_workspace_bytes(1, d.T, d.H, d.D, chunk, d.dt, GLA_IMPL_TCGEN05);
    if (n == 0) raise("chunk_gla_packed: unsupported configuration " + shape_text(d, chunk, v));
    Tensor saved = residuals ? bytes(v, gla_chunk_saved_bytes(1, d.T, d.H, d.D, chunk, d.dt, GLA_IMPL_TCGEN05)) : Tensor(), ws = bytes(v, n);
    check(gla_chunk_fwd_packed(st, d.T, d.H, d.D, chunk, d.dt, nseq, offsets.data_ptr<int32_t>(), ptr(h), (const float*)ptr(g), ptr(v), ptr(k),
                               ptr(q), ptr(hf), ptr(out), ptr(saved), ptr(ws), n), "gla_chunk_fwd_packed");
    return {hf, out, saved};
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& h0, const Tensor& g0, const Tensor& v0, const Tensor& k0,
                               const Tensor& q0, const Tensor& cu, int64_t chunk, int64_t dt) {
    const Dims d{1, v0.size(0), v0.size(1), v0.size(2), (int)dt};
    Tensor h = h0.contiguous(), g = f32(g0), v = v0.contiguous(), k = k0.contiguous(), q = q0.contiguous();
    variable_list r = run(d, h.size(0), h, g, v, k, q, cu, chunk, true);
    // (a copy of offsets in host memory: the caller may fill its array with the next batch's before the backward)
    ctx->save_for_backward({g, v, k, q, r[2], cu.is_cuda() ? cu : cu.clone()});
    ctx->set_materialize_grads(false);
    ctx->saved_data["d"] = std::vector<int64_t>{h.size(0), chunk, dt, !cu.is_cuda(), (int64_t)g0.scalar_type()};
    return {r[0], r[1]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto a = ctx->saved_data["d"].toIntVector();
    const variable_list s = ctx->get_saved_variables();
    const Tensor &g = s[0], &v = s[1], &k = s[2], &q = s[3];
    const int64_t nseq = a[0], T = v.size(0), H = v.size(1), D = v.size(2);
    const int dt = (int)a[2];
    Tensor dh = torch::empty({nseq, H, D, D}, v.options());
    Tensor dhf = grad_or_zeros(grads[0], dh), dout = grad_or_zeros(grads[1], v);
    Tensor dg = torch::empty_like(g), dv = torch::empty_like(v), dk = torch::empty_like(k), dq = torch::empty_like(q);
    const int32_t* cu = s[5].data_ptr<int32_t>();
    if (a[3]) {
      const size_t n = gla_chunk_ragged_workspace_bytes(H, D, dt, nseq, cu, 1);
      Tensor ws = bytes(v, n);
      check(gla_chunk_bwd_ragged(stream_of(v), T, H, D, dt, nseq, cu, (const float*)ptr(g), ptr(v), ptr(k), ptr(q), ptr(s[4]), ptr(dhf),
                                 ptr(dout), ptr(dh), (float*)ptr(dg), ptr(dv), ptr(dk), ptr(dq), ptr(ws), n), "gla_chunk_bwd_ragged");
    } else {
      const size_t n = gla_chunk_bwd_workspace_bytes(1, T, H, D, a[1], dt, GLA_IMPL_TCGEN05);
      Tensor ws = bytes(v, n);
      check(gla_chunk_bwd_packed(stream_of(v), T, H, D, a[1], dt, nseq, cu, (const float*)ptr(g), ptr(v), ptr(k), ptr(q), ptr(s[4]), ptr(dhf),
                                 ptr(dout), ptr(dh), (float*)ptr(dg), ptr(dv), ptr(dk), ptr(dq), ptr(ws), n), "gla_chunk_bwd_packed");
    }
    const auto gt = (torch::ScalarType)a[4];
    variable_list r{dh, gt == torch::kFloat32 ? dg : dg.to(gt), dv, dk, dq};
    r.resize(8);
    return r;
  }
};
std::optional<std::tuple<Tensor, Tensor>> chunk_gla_packed(const Tensor& h, const Tensor& g, const Tensor& v, const Tensor& k,
                                                           const Tensor& q, const Tensor& cu, int64_t chunk) {
  if (!v.defined() || !here(v) || v.dim() != 3 || h.dim() != 4 || cu.dim() != 1 || cu.numel() != h.size(0) + 1) return std::nullopt;
  Dims d{1, v.size(0), v.size(1), v.size(2), dt_of(v)};
  for (const Tensor* t : {&h, &g, &k, &q}) if (t->device() != v.device()) return std::nullopt;
  if (g.sizes() != v.sizes() || k.sizes() != v.sizes() || q.sizes() != v.sizes()) return std::nullopt;
  if (h.size(1) != d.H || h.size(2) != d.D || h.size(3) != d.D || d.dt < 0 || cu.scalar_type() != torch::kInt32) return std::nullopt;
  for (const Tensor* t : {&h, &k, &q}) if (t->scalar_type() != v.scalar_type()) return std::nullopt;
  if (chunk <= 0 || (chunk & (chunk - 1)) || chunk % 128) return std::nullopt;
  Tensor c = cu.contiguous();
  if (!c.is_cuda()) {
    const int32_t* p = c.data_ptr<int32_t>();
    if (p[0] != 0 || p[h.size(0)] != d.T) return std::nullopt;
    int64_t padded = 0;          // sequences in whole chunks of 128, which `chunk` has to divide
    for (int64_t s = 0; s < h.size(0); ++s) {
      if (p[s + 1] <= p[s]) return std::nullopt;
      padded += (p[s + 1] - p[s] + 127) / 128 * 128;
    }
    if (chunk > 256 || padded % chunk)
      raise("chunk_gla_packed: unsupported configuration " + shape_text({1, padded, d.H, d.D, d.dt}, chunk, v));
  } else if (c.device() != v.device()) {
    return std::nullopt;
  }
  no_forward_mode("chunk_gla_packed", {&h, &g, &v, &k, &q});
  variable_list r = wants_grad({&h, &g, &v, &k, &q})
                        ? PackedFn::apply(h, g, v, k, q, c, chunk, (int64_t)d.dt)
                        : PackedFn::run(d, h.size(0), h.contiguous(), f32(g), v.contiguous(), k.contiguous(), q.contiguous(), c, chunk, false);
  return std::make_tuple(r[0], r[1]);
}

// ---- decode step ---------------------------------------------------------------------------------------------------
std::optional<Tensor> decode_step(Tensor state, const Tensor& g, const Tensor& v, const Tensor& k, const Tensor& q,
                                  std::optional<torch::ScalarType> out_dtype) {
  if (!state.defined() || !here(state) || state.dim() != 4 || state.scalar_type() != torch::kFloat32 || !state.is_contiguous()) return std::nullopt;
  const int64_t B = state.size(0), H = state.size(1), D = state.size(2);
  if (state.size(3) != D || v.dim() != 3 || v.size(0) != B || v.size(1) != H || v.size(2) != D) return std::nullopt;
  for (const Tensor* t : {&g, &k, &q}) if (t->sizes() != v.sizes()) return std::nullopt;
  for (const Tensor* t : {&g, &v, &k, &q}) if (t->device() != state.device()) return std::nullopt;
  if (dt_of(v) < 0 || k.scalar_type() != v.scalar_type() || q.scalar_type() != v.scalar_type()) return std::nullopt;
  const auto od = out_dtype.value_or(v.scalar_type());
  if (od != torch::kFloat32 && od != torch::kBFloat16) return std::nullopt;
  torch::NoGradGuard no_grad;
  Tensor g32 = f32(g), vc = v.contiguous(), kc = k.contiguous(), qc = q.contiguous(), out = torch::empty({B, H, D}, v.options().dtype(od));
  check(gla_decode_step(stream_of(v), B, H, D, dt_of(v), (float*)ptr(state), (const float*)ptr(g32), ptr(vc), ptr(kc), ptr(qc), ptr(out),
                        dt_of(out)), "gla_decode_step");
  return out;
}

// ---- the GLA layer as one node -------------------------------------------------------------------------------------------
// Projections (library GEMMs), gate, chunk_gla, head norm with output gate, output projection.  As separate autograd
// nodes the layer is bound by the host (about twenty nodes, 1.1 ms at 16384 tokens against 0.8 ms of kernels) and the
// gradient of x is five products plus four additions; here the products accumulate into one array, the scale of k
// rides on the products that make and consume it, and the bias gradient comes out of the gate's own backward pass.
struct LayerFn : torch::autograd::Function<LayerFn> {
  enum { X, HID, WQ, WK, WV, WGD, WGU, BGU, WOG, WO, NW, NIN };
  static variable_list run(const Dims& d, const Tensor& x, const Tensor& hidden, const variable_list& w, int64_t chunk, double tau_inv,
                           double eps, bool residuals) {
    const int64_t rows = d.B * d.T, inner = d.H * d.D;
    const auto heads = [&](const Tensor& t) { return t.view({d.B, d.T, d.H, d.D}); };
    Tensor x2 = x.view({rows, x.size(2)});
    Tensor q = at::mm(x2, w[WQ].t()), v = at::mm(x2, w[WV].t()), og = at::mm(x2, w[WOG].t());
    Tensor k = torch::empty({rows, inner}, x.options());
    at::addmm_out(k, k, x2, w[WK].t(), 0, 1.0 / std::sqrt((double)d.D));
    Tensor z1 = at::mm(x2, w[WGD].t()), z = at::addmm(w[BGU], z1, w[WGU].t());
    Tensor g = torch::empty({d.B, d.T, d.H, d.D}, x.options().dtype(torch::kFloat32));
    void* st = stream_of(x);
    check(gla_layer_gate_fwd(st, rows * inner, d.dt, ptr(z), (float)tau_inv, (float*)ptr(g)), "gla_layer_gate_fwd");
    variable_list c = chunk_forward(d, hidden, g, heads(v), heads(k), heads(q), chunk, GLA_IMPL_AUTO, residuals);
    Tensor y0 = torch::empty({rows, inner}, x.options()), rstd = torch::empty({rows * d.H}, g.options());
    check(gla_layer_headnorm_gate_fwd(st, rows * d.H, d.D, d.dt, ptr(c[1]), ptr(og), (const float*)ptr(w[NW]), (float)eps, ptr(y0),
                                      (float*)ptr(rstd)), "gla_layer_headnorm_gate_fwd");
    Tensor y = at::mm(y0, w[WO].t()).view({d.B, d.T, w[WO].size(0)});
    if (!residuals) return {y, c[0]};
    return {y, c[0], q, k, v, g, og, z1, z, c[1], rstd, y0, c[2]};
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& x0, const Tensor& hidden0, const Tensor& wq, const Tensor& wk, const Tensor& wv,
                               const Tensor& wgd, const Tensor& wgu, const Tensor& bgu, const Tensor& wog, const Tensor& wo,
                               const Tensor& nw, int64_t H, int64_t D, int64_t dt, int64_t chunk, double tau_inv, double eps) {
    const Dims d{x0.size(0), x0.size(1), H, D, (int)dt};
    const Tensor x = x0.contiguous(), hidden = hidden0.contiguous();
    variable_list w{Tensor(), Tensor(), wq, wk, wv, wgd, wgu, bgu, wog, wo, nw};
    variable_list r = run(d, x, hidden, w, chunk, tau_inv, eps, true);
    variable_list keep{x, wq, wk, wv, wgd, wgu, wog, wo, nw};
    keep.insert(keep.end(), r.begin() + 2, r.end());
    ctx->save_for_backward(keep);
    ctx->set_materialize_grads(false);
    ctx->saved_data["i"] = std::vector<int64_t>{d.B, d.T, H, D, dt, chunk};
    ctx->saved_data["t"] = tau_inv;
    if (!wants_any({&x0, &hidden0, &wq, &wk, &wv, &wgd, &wgu, &bgu})) ctx->mark_non_differentiable({r[1]});
    return {r[0], r[1]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto a = ctx->saved_data["i"].toIntVector();
    const double tau_inv = ctx->saved_data["t"].toDouble();
    torch::NoGradGuard no_grad;       // (under create_graph: no second derivative of parts of the layer)
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x = s[0], &wq = s[1], &wk = s[2], &wv = s[3], &wgd = s[4], &wgu = s[5], &wog = s[6], &wo = s[7], &nw = s[8];
    const Tensor &q = s[9], &k = s[10], &v = s[11], &g = s[12], &og = s[13], &z1 = s[14], &z = s[15], &out = s[16], &rstd = s[17], &y0 = s[18];
    const Dims d{a[0], a[1], a[2], a[3], (int)a[4]};
    const int64_t rows = d.B * d.T, inner = d.H * d.D;
    void* st = stream_of(x);
    const auto heads = [&](const Tensor& t) { return t.view({d.B, d.T, d.H, d.D}); };
    const auto flat = [&](const Tensor& t) { return t.view({rows, inner}); };
    Tensor x2 = x.view({rows, x.size(2)});
    const auto need = [&](size_t i) { return ctx->needs_input_grad(i); };
    const bool need_gate = need(WGD) || need(WGU) || need(BGU) || need(X);      // of the gate projection's output
    const bool need_core = need_gate || need(HID) || need(WQ) || need(WK) || need(WV);
    Tensor dout, dog, dnw, dwo;
    if (grads[0].defined()) {
      Tensor dy = grads[0].to(x.scalar_type()).contiguous().view({rows, wo.size(0)});
      if (need(WO)) dwo = at::mm(dy.t(), y0);
      if (need_core || need(WOG) || need(NW)) {
        Tensor dy0 = at::mm(dy, wo);
        dout = torch::empty_like(out);
        dog = torch::empty_like(og);
        if (need(NW)) dnw = torch::empty_like(nw);
        const size_t n = need(NW) ? gla_layer_headnorm_gate_bwd_workspace_bytes(rows * d.H, d.D) : 0;
        Tensor ws = bytes(x, n);
        check(gla_layer_headnorm_gate_bwd(st, rows * d.H, d.D, d.dt, ptr(out), ptr(og), (const float*)ptr(nw), (const float*)ptr(rstd), ptr(dy0),
                                          ptr(dout), ptr(dog), (float*)ptr(dnw), ptr(ws), n), "gla_layer_headnorm_gate_bwd");
      }
    }
    variable_list r(NIN + 6);
    if (need_core) {
      variable_list c = chunk_backward(d, g, heads(v), heads(k), heads(q), s[19], grads[1], dout, a[5], GLA_IMPL_AUTO);
      const double ks = 1.0 / std::sqrt((double)d.D);
      Tensor dv = flat(c[2]), dk = flat(c[3]), dq = flat(c[4]), dz1;
      r[HID] = c[0];
      if (need_gate) {
        Tensor dz = torch::empty_like(z), dbgu = torch::empty({inner}, x.options());
        const size_t n = gla_layer_gate_bwd_bias_workspace_bytes(rows, inner);
        Tensor ws = bytes(x, n);
        check(gla_layer_gate_bwd_bias(st, rows, inner, d.dt, ptr(z), (const float*)ptr(c[1]), (float)tau_inv, ptr(dz), ptr(dbgu), ptr(ws), n),
              "gla_layer_gate_bwd_bias");
        r[BGU] = dbgu;
        if (need(WGU)) r[WGU] = at::mm(dz.t(), z1);
        if (need(WGD) || need(X)) dz1 = at::mm(dz, wgu);
        if (need(WGD)) r[WGD] = at::mm(dz1.t(), x2);
      }
      if (need(WQ)) r[WQ] = at::mm(dq.t(), x2);
      if (need(WV)) r[WV] = at::mm(dv.t(), x2);
      if (need(WK)) {
        r[WK] = torch::empty(wk.sizes(), x.options());
        at::addmm_out(r[WK], r[WK], dk.t(), x2, 0, ks);
      }
      if (need(X)) {
        Tensor dx = at::mm(dq, wq);
        dx.addmm_(dk, wk, 1, ks).addmm_(dv, wv).addmm_(dz1, wgd);
        if (dog.defined()) dx.addmm_(dog, wog);
        r[X] = dx.view(x.sizes());
      }
    }
    if (dog.defined() && need(WOG)) r[WOG] = at::mm(dog.t(), x2);
    r[WO] = dwo;
    r[NW] = dnw;
    return r;
  }
};
// w: q, k, v, gate_down, gate_up, gate_up bias, out_gate, o projections and the head norm's weight, each as its module
// holds it
std::optional<std::tuple<Tensor, Tensor>> gla_layer(const Tensor& x, const std::optional<Tensor>& hidden0, const variable_list& w,
                                                    int64_t H, int64_t D, int64_t chunk, double tau_inv, double eps) {
  if (!x.defined() || !here(x) || x.dim() != 3 || w.size() != 9 || dt_of(x) < 0 || x.numel() == 0) return std::nullopt;
  const int64_t dm = x.size(2), inner = H * D, lr = w[3].dim() == 2 ? w[3].size(0) : -1;
  const auto is = [&](const Tensor& t, int64_t r, int64_t c) {
    return t.device() == x.device() && t.scalar_type() == x.scalar_type() && t.dim() == 2 && t.size(0) == r && t.size(1) == c && t.is_contiguous();
  };
  if (!is(w[0], inner, dm) || !is(w[1], inner, dm) || !is(w[2], inner, dm) || !is(w[3], lr, dm) || !is(w[4], inner, lr) || !is(w[6], inner, dm) ||
      !is(w[7], dm, inner))
    return std::nullopt;
  if (w[5].dim() != 1 || w[5].size(0) != inner || w[5].scalar_type() != x.scalar_type() || w[5].device() != x.device()) return std::nullopt;
  if (w[8].dim() != 1 || w[8].size(0) != D || w[8].scalar_type() != torch::kFloat32 || w[8].device() != x.device() || !w[8].is_contiguous()) return std::nullopt;
  if ((D != 32 && D != 64 && D != 128 && D != 256) || chunk <= 0 || (chunk & (chunk - 1)) || x.size(1) % chunk) return std::nullopt;
  const Dims d{x.size(0), x.size(1), H, D, dt_of(x)};
  Tensor hidden = hidden0.has_value() ? *hidden0 : torch::zeros({d.B, H, D, D}, x.options().requires_grad(false));
  if (hidden.dim() != 4 || hidden.size(0) != d.B || hidden.size(1) != H || hidden.size(2) != D || hidden.size(3) != D ||
      hidden.scalar_type() != x.scalar_type() || hidden.device() != x.device())
    return std::nullopt;
  no_forward_mode("GLALayer", {&x, &hidden, &w[0], &w[1], &w[2], &w[3], &w[4], &w[5], &w[6], &w[7], &w[8]});
  if (wants_grad({&x, &hidden, &w[0], &w[1], &w[2], &w[3], &w[4], &w[5], &w[6], &w[7], &w[8]})) {
    variable_list r = LayerFn::apply(x, hidden, w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], H, D, (int64_t)d.dt, chunk, tau_inv, eps);
    return std::make_tuple(r[0], r[1]);
  }
  variable_list in{Tensor(), Tensor()};
  in.insert(in.end(), w.begin(), w.end());
  variable_list r = LayerFn::run(d, x.contiguous(), hidden.contiguous(), in, chunk, tau_inv, eps, false);
  return std::make_tuple(r[0], r[1]);
}

// ---- scans ---------------------------------------------------------------------------------------------------------
std::optional<Tensor> scan(int64_t op, const Tensor& src, int64_t axis, const std::optional<Tensor>& init, bool reverse,
                           std::optional<torch::ScalarType> out_dtype) {
  const int64_t nd = src.dim();
  if (axis < 0) axis += nd;
  if (!here(src) || dt_of(src) < 0 || axis < 0 || axis >= nd) return std::nullopt;
  const auto od = out_dtype.value_or(src.scalar_type());
  if (od != torch::kFloat32 && od != torch::kBFloat16) return std::nullopt;
  int64_t N = 1, D = 1;
  for (int64_t i = 0; i < axis; ++i) N *= src.size(i);
  for (int64_t i = axis + 1; i < nd; ++i) D *= src.size(i);
  torch::NoGradGuard no_grad;
  Tensor i0;
  if (init.has_value()) {
    if (init->dim() != nd - 1 || init->device() != src.device()) return std::nullopt;
    for (int64_t i = 0; i < nd - 1; ++i) if (init->size(i) != src.size(i < axis ? i : i + 1)) return std::nullopt;
    i0 = init->to(src.scalar_type()).contiguous();
  }
  Tensor x = src.contiguous(), dst = torch::empty(src.sizes(), src.options().dtype(od));
  check(gla_scan(stream_of(src), (int)op, N, src.size(axis), D, ptr(x), ptr(i0), ptr(dst), reverse, dt_of(src), dt_of(dst)), "gla_scan");
  return dst;
}
std::optional<std::tuple<Tensor, Tensor>> rnn(const Tensor& g, const Tensor& kv, const std::optional<Tensor>& ig,
                                              const std::optional<Tensor>& ikv, bool reverse, bool last_only) {
  if (!here(kv) || (kv.dim() != 3 && kv.dim() != 4) || dt_of(kv) < 0 || ig.has_value() != ikv.has_value()) return std::nullopt;
  const int b = kv.dim() == 4;
  const int64_t N = b ? kv.size(0) : 1, T = kv.size(b), K = kv.size(b + 1), V = kv.size(b + 2);
  if (g.dim() != 2 + b || (b && g.size(0) != N) || g.size(b) != T || g.size(b + 1) != K || g.device() != kv.device()) return std::nullopt;
  torch::NoGradGuard no_grad;
  Tensor g32 = f32(g), x = kv.contiguous(), ig32, ikvc;
  if (ig.has_value()) {
    if (ig->device() != kv.device() || ikv->device() != kv.device() || ig->numel() != N * K || ikv->numel() != N * K * V) return std::nullopt;
    ig32 = f32(*ig);
    ikvc = ikv->to(kv.scalar_type()).contiguous();
  }
  // every row is written, except with last_only, where the rows in between are documented as undefined but were zero
  Tensor out_log = last_only ? torch::zeros_like(g32) : torch::empty_like(g32), out_state = last_only ? torch::zeros_like(x) : torch::empty_like(x);
  const size_t n = last_only ? 0 : gla_rnn_scan_workspace_bytes(N, T, K, V);
  Tensor ws = bytes(kv, n);
  check(gla_rnn_scan_ws(stream_of(kv), N, T, K, V, (const float*)ptr(g32), ptr(x), (const float*)ptr(ig32), ptr(ikvc), (float*)ptr(out_log),
                        ptr(out_state), reverse, last_only, dt_of(kv), ptr(ws), n), "gla_rnn_scan_ws");
  return std::make_tuple(g.scalar_type() == torch::kFloat32 ? out_log : out_log.to(g.scalar_type()), out_state);
}

}  // namespace

PYBIND11_MODULE(gla_b200_host, m) {
  using release = py::call_guard<py::gil_scoped_release>;
  m.def("set_error_class", [](py::object c) { g_error = c.release().ptr(); });
  m.def("chunk_gla", &chunk_gla, release());
  m.def("recurrent_gla", &recurrent_gla, release());
  m.def("chunk_gla_packed", &chunk_gla_packed, release());
  m.def("gla_layer", &gla_layer, release());
  m.def("decode_step", &decode_step, release());
  m.def("scan", &scan, release());
  m.def("rnn", &rnn, release());
}
