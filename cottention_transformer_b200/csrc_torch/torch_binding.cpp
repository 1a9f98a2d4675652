// Compiled torch binding over the C ABI of libcottention_b200.so (include/cottention_b200.h).
//
// 1. The reference's extension module: four functions with the signature its pybind block registers
//    (Cuda_Kernel/combined_kernel_general.cu:353,444-454),
//        float32 / float64 / float16 / bfloat16 (Tensor Q, Tensor K, Tensor V, int block_size,
//                                                bool inplace = false, bool reversed = false) -> Tensor
//    with the checks, messages, autocast dtype rule and in-place behaviour of forward_<dtype> (:355-407).
// 2. The fused operators as torch.library ops (namespace cottention_b200), so that the autograd functions of the
//    package make one dispatcher call per direction instead of a dozen Python-level tensor calls -- at BERT shapes
//    the step is otherwise bound by the host, not by its kernels.
//
// 3. The autograd functions around them, and the decode and prefill calls.
//
// Nothing here computes: every function validates, allocates its outputs and calls one extern "C" entry point on
// torch's current stream.  The ctypes route (cottention_transformer_b200/_lib.py) stays for non-torch hosts.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>
#include <torch/library.h>

#include "../../include/cottention_b200.h"

namespace {

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return COTT_F32;
    case at::kDouble: return COTT_F64;
    case at::kHalf: return COTT_F16;
    case at::kBFloat16: return COTT_BF16;
    default: TORCH_CHECK(false, "Only float32, float64, float16, and bfloat16 are supported");
  }
}

void check(int status, const char* what) {
  TORCH_CHECK(status == COTT_OK, what, ": ", cott_status_string(status), " (", status, "): ", cott_last_error());
}

void* stream_of(const at::Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

const void* ptr_or_null(const c10::optional<at::Tensor>& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }

// ---- 1. FastAttention2.kernel.<dtype> ------------------------------------------------------------------------
// AUTOCAST: the dtype the entry point runs in when autocast is on and Q is float32 (:377-389)
template <at::ScalarType AUTOCAST>
at::Tensor forward_(at::Tensor& Q, at::Tensor& K, at::Tensor& V, const int8_t block_size, bool inplace, bool reversed) {
  (void)block_size;  // accepted and ignored, as in the reference (:353)
  TORCH_CHECK(Q.device().is_cuda(), "Q must be a CUDA tensor");
  TORCH_CHECK(K.device().is_cuda(), "K must be a CUDA tensor");
  TORCH_CHECK(V.device().is_cuda(), "V must be a CUDA tensor");
  TORCH_CHECK(Q.dim() == 4 && K.dim() == 4 && V.dim() == 4, "Q, K and V must be 4-dimensional [N, H, S, D]");
  TORCH_CHECK(Q.size(3) == K.size(3), "Q and K must have the same dimension");
  const int64_t D_attn = Q.size(3);
  TORCH_CHECK(D_attn % 16 == 0, "D_attn must be divisible by 16");
  TORCH_CHECK(D_attn >= 16 * 2, "D_attn must be greater than or equal to 16*2");
  for (int i = 0; i < 3; ++i)
    TORCH_CHECK(K.size(i) == Q.size(i) && V.size(i) == Q.size(i), "Q, K and V must agree in their first three dimensions");
  const at::ScalarType data_type =
      (at::autocast::is_autocast_enabled(at::kCUDA) && Q.scalar_type() == at::kFloat) ? AUTOCAST : Q.scalar_type();
  const int code = dtype_code(data_type);
  Q = Q.contiguous().to(data_type);  // :397-399 (rebinding the caller's handles, like the reference's Tensor&)
  K = K.contiguous().to(data_type);
  V = V.contiguous().to(data_type);
  at::Tensor out = inplace ? V : at::empty({Q.size(0), Q.size(1), Q.size(2), V.size(3)}, Q.options());  // :402-407
  const c10::cuda::CUDAGuard guard(Q.device());  // :412
  check(cott_scan(Q.data_ptr(), K.data_ptr(), V.data_ptr(), out.data_ptr(), (int)Q.size(0), (int)Q.size(1), (int)Q.size(2),
                  (int)D_attn, (int)V.size(3), code, reversed ? 1 : 0, stream_of(Q)),
        "cott_scan");
  return out;
}

// ---- 2. fused operators ---------------------------------------------------------------------------------------
// norm_const as the floats the C side reads: no copy when it already is a dense fp32 tensor on this device
at::Tensor nc_floats(const at::Tensor& norm_const, const at::Tensor& like) {
  at::Tensor nc = norm_const.detach();
  if (nc.scalar_type() != at::kFloat || nc.device() != like.device()) nc = nc.to(like.device(), at::kFloat);
  return nc.contiguous();
}
at::Tensor nc_f32(const at::Tensor& norm_const, const at::Tensor& like, int64_t H) {
  TORCH_CHECK(norm_const.numel() == H, "norm_const must have one entry per head (", H, "), got ", norm_const.numel());
  return nc_floats(norm_const, like);
}
// (the packed and decode entry points take a longer parameter, as they always have; a shorter one would be read past its end)
at::Tensor nc_at_least(const at::Tensor& norm_const, const at::Tensor& like, int64_t H) {
  TORCH_CHECK(norm_const.numel() >= H, "norm_const must have one entry per head (", H, "), got ", norm_const.numel());
  return nc_floats(norm_const, like);
}

// causal forward: returns (out, workspace, saved); workspace / saved are empty tensors when not needed
std::tuple<at::Tensor, at::Tensor, at::Tensor> causal_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                                          const at::Tensor& norm_const, const c10::optional<at::Tensor>& keep,
                                                          int64_t nseg, bool save_states) {
  TORCH_CHECK(q.is_cuda() && q.is_contiguous() && k.is_contiguous() && v.is_contiguous(), "contiguous CUDA tensors expected");
  const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), D = (int)q.size(3);
  const int code = dtype_code(q.scalar_type());
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor nc = nc_f32(norm_const, q, H);
  at::Tensor out = at::empty_like(v);
  const auto bytes = q.options().dtype(at::kByte);
  if (nseg <= 0) nseg = cott_cos_attn_seg_choice(B, H, N);
  const bool general = nseg > 1 || (keep.has_value() && keep->defined());
  at::Tensor ws = at::empty({general ? (int64_t)std::max<size_t>(cott_cos_attn_seg_workspace_bytes(B, H, N, (int)nseg), 16) : 0}, bytes);
  at::Tensor saved = at::empty({save_states ? (int64_t)std::max<size_t>(cott_cos_attn_saved_bytes(B, H, N), 16) : 0}, bytes);
  const unsigned char* kp = static_cast<const unsigned char*>(ptr_or_null(keep));
  if (save_states)
    check(cott_cos_attn_fwd_train(q.data_ptr(), k.data_ptr(), v.data_ptr(), kp, nc.data_ptr<float>(), out.data_ptr(), saved.data_ptr(),
                                  general ? ws.data_ptr() : nullptr, (int)nseg, nullptr, B, H, N, D, D, code, stream_of(q)),
          "cott_cos_attn_fwd_train");
  else if (general)
    check(cott_cos_attn_fwd_seg(q.data_ptr(), k.data_ptr(), v.data_ptr(), kp, nc.data_ptr<float>(), out.data_ptr(), ws.data_ptr(),
                                (int)nseg, nullptr, B, H, N, D, D, code, stream_of(q)),
          "cott_cos_attn_fwd_seg");
  else
    check(cott_cos_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), nc.data_ptr<float>(), out.data_ptr(), B, H, N, D, D, code,
                            stream_of(q)),
          "cott_cos_attn_fwd");
  return {out, ws, saved};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> causal_bwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                                                      const at::Tensor& norm_const,
                                                                      const c10::optional<at::Tensor>& keep, const at::Tensor& dout_,
                                                                      const at::Tensor& ws, const at::Tensor& saved, int64_t nseg) {
  const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), D = (int)q.size(3);
  const int code = dtype_code(q.scalar_type());
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor nc = nc_f32(norm_const, q, H);
  at::Tensor dout = dout_.contiguous().to(q.scalar_type());
  at::Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  at::Tensor dnc = at::empty({H}, q.options().dtype(at::kFloat));
  const unsigned char* kp = static_cast<const unsigned char*>(ptr_or_null(keep));
  void* wsp = ws.numel() ? ws.data_ptr() : nullptr;
  if (nseg <= 0) nseg = cott_cos_attn_seg_choice(B, H, N);  // the forward's choice for the same sizes on the same device
  if (saved.numel())
    check(cott_cos_attn_bwd_train(q.data_ptr(), k.data_ptr(), v.data_ptr(), kp, nc.data_ptr<float>(), dout.data_ptr(), saved.data_ptr(), wsp,
                                  (int)nseg, nullptr, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dnc.data_ptr<float>(), B, H, N, D, D,
                                  code, stream_of(q)),
          "cott_cos_attn_bwd_train");
  else if (ws.numel())
    check(cott_cos_attn_bwd_seg(q.data_ptr(), k.data_ptr(), v.data_ptr(), kp, nc.data_ptr<float>(), dout.data_ptr(), wsp, (int)nseg, nullptr,
                                dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dnc.data_ptr<float>(), B, H, N, D, D, code, stream_of(q)),
          "cott_cos_attn_bwd_seg");
  else
    check(cott_cos_attn_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), nc.data_ptr<float>(), dout.data_ptr(), dq.data_ptr(), dk.data_ptr(),
                            dv.data_ptr(), dnc.data_ptr<float>(), B, H, N, D, D, code, stream_of(q)),
          "cott_cos_attn_bwd");
  return {dq, dk, dv, dnc};
}

// bidirectional forward: returns (out, scratch)
std::tuple<at::Tensor, at::Tensor> bidir_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& norm_const,
                                             const c10::optional<at::Tensor>& keep) {
  TORCH_CHECK(q.is_cuda() && q.is_contiguous() && k.is_contiguous() && v.is_contiguous(), "contiguous CUDA tensors expected");
  const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), Dk = (int)q.size(3), Dv = (int)v.size(3);
  const int code = dtype_code(q.scalar_type());
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor nc = nc_f32(norm_const, q, H);
  at::Tensor out = at::empty({B, H, N, Dv}, q.options());
  at::Tensor scratch = at::empty({(int64_t)std::max<size_t>(cott_bidir_scratch_bytes(B, H, N, Dk, Dv, code), 1)}, q.options().dtype(at::kByte));
  check(cott_bidir_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), static_cast<const unsigned char*>(ptr_or_null(keep)), nc.data_ptr<float>(),
                       out.data_ptr(), scratch.data_ptr(), B, H, N, Dk, Dv, code, stream_of(q)),
        "cott_bidir_fwd");
  return {out, scratch};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> bidir_bwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                                                     const at::Tensor& norm_const, const c10::optional<at::Tensor>& keep,
                                                                     const at::Tensor& dout_, const at::Tensor& scratch) {
  const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), Dk = (int)q.size(3), Dv = (int)v.size(3);
  const int code = dtype_code(q.scalar_type());
  const c10::cuda::CUDAGuard guard(q.device());
  at::Tensor nc = nc_f32(norm_const, q, H);
  at::Tensor dout = dout_.contiguous().to(q.scalar_type());
  at::Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  at::Tensor dnc = at::empty({H}, q.options().dtype(at::kFloat));
  at::Tensor scratch2 = at::empty_like(scratch);
  check(cott_bidir_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), static_cast<const unsigned char*>(ptr_or_null(keep)), nc.data_ptr<float>(),
                       dout.data_ptr(), scratch.data_ptr(), scratch2.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                       dnc.data_ptr<float>(), B, H, N, Dk, Dv, code, stream_of(q)),
        "cott_bidir_bwd");
  return {dq, dk, dv, dnc};
}

// ---- 3. autograd functions --------------------------------------------------------------------------------------
// One call from Python per direction: validation, allocation, launches and the autograd node in C++.  (A step of a small
// model is bound by the host: two Python-level autograd functions, ctypes conversions and dispatcher calls cost more
// than the kernels of a 200-token sequence.)  The Python autograd functions of cos_attention.py stay for hosts without
// this module and for the cases that need them (tracing, functorch transforms); both end in the same C calls.
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;
using OptTensor = c10::optional<at::Tensor>;

bool has(const OptTensor& t) { return t.has_value() && t->defined(); }
OptTensor keep_u8(const OptTensor& keep, const at::Tensor& like) {
  if (!has(keep)) return c10::nullopt;
  // always a tensor of our own: the backward reads it again, whatever the caller has done to the mask by then.  (A bool
  // mask is read as the bytes it is, which a plain copy gives.)
  if (keep->scalar_type() == at::kBool && keep->device() == like.device()) return keep->clone(at::MemoryFormat::Contiguous);
  at::Tensor k = keep->to(like.device(), at::kByte).contiguous();
  return k.is_alias_of(*keep) ? k.clone() : k;
}
// the gradient of norm_const in the shape and dtype of the parameter
at::Tensor nc_grad(const at::Tensor& dnc, at::IntArrayRef shape, at::ScalarType dtype) {
  at::Tensor g = dnc.reshape(shape);
  return g.scalar_type() == dtype ? g : g.to(dtype);
}
// [B, H, N, D] tensors of one shape: the C side takes the sizes from q alone
void check_bhnd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
  if (q.dim() != 4) throw py::value_error("[B, H, N, D] tensors expected, got " + std::to_string(q.dim()) + " dimensions");
  TORCH_CHECK(k.sizes() == q.sizes() && v.sizes() == q.sizes(), "q, k and v must have the same shape, got ", q.sizes(), ", ", k.sizes(), " and ",
              v.sizes());
}
at::Tensor bytes_like(const at::Tensor& t, size_t n) { return at::empty({(int64_t)std::max<size_t>(n, 16)}, t.options().dtype(at::kByte)); }
const unsigned char* u8(const OptTensor& t) { return static_cast<const unsigned char*>(ptr_or_null(t)); }
at::Tensor dense_as(const at::Tensor& t, at::ScalarType dtype) {
  at::Tensor c = t.contiguous();
  return c.scalar_type() == dtype ? c : c.to(dtype);
}
void save_nc(AutogradContext* ctx, const at::Tensor& norm_const) {
  ctx->saved_data["nc_shape"] = norm_const.sizes().vec();
  ctx->saved_data["nc_dtype"] = (int64_t)norm_const.scalar_type();
}
at::Tensor nc_grad(AutogradContext* ctx, const at::Tensor& dnc) {
  return nc_grad(dnc, ctx->saved_data["nc_shape"].toIntVector(), (at::ScalarType)ctx->saved_data["nc_dtype"].toInt());
}
void save_opt(AutogradContext* ctx, const char* key, const OptTensor& t) {
  if (has(t)) ctx->saved_data[key] = *t;
}
OptTensor load_opt(AutogradContext* ctx, const char* key) {
  const auto it = ctx->saved_data.find(key);
  return it == ctx->saved_data.end() ? OptTensor() : OptTensor(it->second.toTensor());
}

// 16-bit, head dim 64
struct CausalFn : torch::autograd::Function<CausalFn> {
  static Variable forward(AutogradContext* ctx, const at::Tensor& q_, const at::Tensor& k_, const at::Tensor& v_, const at::Tensor& norm_const,
                          const OptTensor& keep, int64_t nseg, bool one_pass) {
    check_bhnd(q_, k_, v_);
    const at::Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
    const OptTensor kp = keep_u8(keep, q);
    auto [out, ws, saved] = causal_fwd(q, k, v, norm_const, kp, nseg, one_pass);
    ctx->save_for_backward({q, k, v, norm_const.detach()});
    ctx->saved_data["ws"] = ws;
    ctx->saved_data["saved"] = saved;
    ctx->saved_data["nseg"] = nseg;
    save_opt(ctx, "keep", kp);
    save_nc(ctx, norm_const);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const at::Tensor ws = ctx->saved_data["ws"].toTensor(), saved = ctx->saved_data["saved"].toTensor();
    const int64_t nseg = ctx->saved_data["nseg"].toInt();
    at::Tensor dq, dk, dv, dnc;
    if (at::GradMode::is_enabled()) {  // create_graph: through the dispatcher, which says that there is no second derivative
      static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("cottention_b200::causal_bwd", "").typed<decltype(causal_bwd)>();
      std::tie(dq, dk, dv, dnc) = op.call(s[0], s[1], s[2], s[3], load_opt(ctx, "keep"), grads[0], ws, saved, nseg);
    } else {
      std::tie(dq, dk, dv, dnc) = causal_bwd(s[0], s[1], s[2], s[3], load_opt(ctx, "keep"), grads[0], ws, saved, nseg);
    }
    return {dq, dk, dv, nc_grad(ctx, dnc), Variable(), Variable(), Variable()};
  }
};

// the packed [B, N, 3, H, 64] forms
struct Packed {
  at::Tensor qkv;
  int64_t B, N, H, D, e;
  cott_layout lay;
  explicit Packed(const at::Tensor& t)
      : qkv(t), B(t.size(0)), N(t.size(1)), H(t.size(3)), D(t.size(4)), e(t.element_size()),
        lay{N * 3 * H * D, D, 3 * H * D, N * H * D, D, H * D} {}
  char* part(int i) const { return static_cast<char*>(qkv.data_ptr()) + i * H * D * e; }  // q, k, v of the first token
};
struct CausalPackedFn : torch::autograd::Function<CausalPackedFn> {
  static Variable forward(AutogradContext* ctx, const at::Tensor& qkv_, const at::Tensor& norm_const, const OptTensor& keep,
                          const OptTensor& sin, const OptTensor& cos, bool keep_rotated) {
    const Packed p(qkv_.contiguous());
    const c10::cuda::CUDAGuard guard(p.qkv.device());
    const at::Tensor nc = nc_at_least(norm_const, p.qkv, p.H);
    const OptTensor kp = keep_u8(keep, p.qkv);
    at::Tensor out = at::empty({p.B, p.N, p.H, p.D}, p.qkv.options());
    const int code = dtype_code(p.qkv.scalar_type()), B = (int)p.B, H = (int)p.H, N = (int)p.N, D = (int)p.D;
    const bool rot = has(sin);
    const int nseg = cott_cos_attn_seg_choice(B, H, N);
    at::Tensor ws = bytes_like(p.qkv, cott_cos_attn_seg_workspace_bytes(B, H, N, nseg));
    const at::Tensor rqk = rot ? rotated(p, *sin, *cos) : at::Tensor();
    const cott_layout ql = qk_layout(p);
    check(cott_cos_attn_fwd_split(rot ? rqk.data_ptr() : p.part(0), rot ? k_of(rqk, p) : p.part(1), p.part(2), u8(kp), nc.data_ptr<float>(),
                                  out.data_ptr(), ws.data_ptr(), nseg, &p.lay, rot ? &ql : nullptr, B, H, N, D, D, code, stream_of(p.qkv)),
          "cott_cos_attn_fwd_split");
    ctx->save_for_backward({p.qkv, nc, rot ? *sin : at::Tensor(), rot ? *cos : at::Tensor(), keep_rotated ? rqk : at::Tensor()});
    ctx->saved_data["ws"] = ws;
    ctx->saved_data["nseg"] = (int64_t)nseg;
    save_opt(ctx, "keep", kp);
    save_nc(ctx, norm_const);
    return out;
  }
  static cott_layout qk_layout(const Packed& p) { return cott_layout{p.N * 2 * p.H * p.D, p.D, 2 * p.H * p.D, 0, 0, 0}; }
  static void* k_of(const at::Tensor& rqk, const Packed& p) { return static_cast<char*>(rqk.data_ptr()) + p.H * p.D * p.e; }
  static long long table_stride(const Packed& p, const at::Tensor& sin) { return sin.dim() == 3 && sin.size(0) > 1 ? (long long)(p.N * sin.size(-1)) : 0; }
  // q and k of `p`, rotated: [B, N, 2, H, D]
  static at::Tensor rotated(const Packed& p, const at::Tensor& sin, const at::Tensor& cos) {
    at::Tensor rqk = at::empty({p.B, p.N, 2, p.H, p.D}, p.qkv.options());
    const cott_layout ql = qk_layout(p);
    check(cott_rotary_copy(p.part(0), p.part(1), rqk.data_ptr(), k_of(rqk, p), sin.data_ptr<float>(), cos.data_ptr<float>(), &p.lay, &ql, (int)p.B,
                           (int)p.H, (int)p.N, (int)p.D, (int)(2 * sin.size(-1)), table_stride(p, sin), dtype_code(p.qkv.scalar_type()),
                           stream_of(p.qkv)),
          "cott_rotary_copy");
    return rqk;
  }
  // the gradients of the rotated q and k in `p`, back through the rotation in place
  static void rotate_back(const Packed& p, const at::Tensor& sin, const at::Tensor& cos) {
    check(cott_rotary(p.part(0), p.part(1), sin.data_ptr<float>(), cos.data_ptr<float>(), &p.lay, (int)p.B, (int)p.H, (int)p.N, (int)p.D,
                      (int)(2 * sin.size(-1)), table_stride(p, sin), 1, dtype_code(p.qkv.scalar_type()), stream_of(p.qkv)),
          "cott_rotary");
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Packed p(s[0]), d(at::empty_like(s[0]));
    const c10::cuda::CUDAGuard guard(p.qkv.device());
    const at::Tensor &nc = s[1], dout = dense_as(grads[0], p.qkv.scalar_type()), ws = ctx->saved_data["ws"].toTensor();
    const OptTensor kp = load_opt(ctx, "keep");
    at::Tensor dnc = at::empty({p.H}, p.qkv.options().dtype(at::kFloat));
    const int code = dtype_code(p.qkv.scalar_type()), B = (int)p.B, H = (int)p.H, N = (int)p.N, D = (int)p.D;
    const bool rot = s[2].defined();
    const at::Tensor rqk = !rot || s[4].defined() ? s[4] : rotated(p, s[2], s[3]);
    const cott_layout ql = qk_layout(p);
    check(cott_cos_attn_bwd_split(rot ? rqk.data_ptr() : p.part(0), rot ? k_of(rqk, p) : p.part(1), p.part(2), u8(kp), nc.data_ptr<float>(),
                                  dout.data_ptr(), ws.data_ptr(), (int)ctx->saved_data["nseg"].toInt(), &p.lay, rot ? &ql : nullptr, d.part(0),
                                  d.part(1), d.part(2), dnc.data_ptr<float>(), B, H, N, D, D, code, stream_of(p.qkv)),
          "cott_cos_attn_bwd_split");
    if (rot) rotate_back(d, s[2], s[3]);
    return {d.qkv, nc_grad(ctx, dnc), Variable(), Variable(), Variable(), Variable()};
  }
};
struct BidirPackedFn : torch::autograd::Function<BidirPackedFn> {
  static Variable forward(AutogradContext* ctx, const at::Tensor& qkv_, const at::Tensor& norm_const, const OptTensor& keep) {
    const Packed p(qkv_.contiguous());
    const c10::cuda::CUDAGuard guard(p.qkv.device());
    const at::Tensor nc = nc_at_least(norm_const, p.qkv, p.H);
    const OptTensor kp = keep_u8(keep, p.qkv);
    at::Tensor out = at::empty({p.B, p.N, p.H, p.D}, p.qkv.options());
    check(cott_bidir_fwd_strided(p.part(0), p.part(1), p.part(2), u8(kp), nc.data_ptr<float>(), out.data_ptr(), &p.lay, (int)p.B, (int)p.H,
                                 (int)p.N, (int)p.D, (int)p.D, dtype_code(p.qkv.scalar_type()), stream_of(p.qkv)),
          "cott_bidir_fwd_strided");
    ctx->save_for_backward({p.qkv, nc});
    save_opt(ctx, "keep", kp);
    save_nc(ctx, norm_const);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Packed p(s[0]), d(at::empty_like(s[0]));
    const c10::cuda::CUDAGuard guard(p.qkv.device());
    const at::Tensor dout = dense_as(grads[0], p.qkv.scalar_type());
    at::Tensor dnc = at::empty({p.H}, p.qkv.options().dtype(at::kFloat));
    check(cott_bidir_bwd_strided(p.part(0), p.part(1), p.part(2), u8(load_opt(ctx, "keep")), s[1].data_ptr<float>(), dout.data_ptr(), &p.lay,
                                 d.part(0), d.part(1), d.part(2), dnc.data_ptr<float>(), (int)p.B, (int)p.H, (int)p.N, (int)p.D, (int)p.D,
                                 dtype_code(p.qkv.scalar_type()), stream_of(p.qkv)),
          "cott_bidir_bwd_strided");
    return {d.qkv, nc_grad(ctx, dnc), Variable()};
  }
};

// 16-bit, head dim 128
struct WideFn : torch::autograd::Function<WideFn> {
  static Variable forward(AutogradContext* ctx, const at::Tensor& q_, const at::Tensor& k_, const at::Tensor& v_, const at::Tensor& norm_const,
                          const OptTensor& keep) {
    check_bhnd(q_, k_, v_);
    const at::Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
    const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), D = (int)q.size(3);
    const c10::cuda::CUDAGuard guard(q.device());
    const at::Tensor nc = nc_f32(norm_const, q, H);
    const OptTensor kp = keep_u8(keep, q);
    at::Tensor out = at::empty_like(v), ws = bytes_like(q, cott_cos_attn_wide_workspace_bytes(B, H, N));
    check(cott_cos_attn_wide_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), u8(kp), nc.data_ptr<float>(), out.data_ptr(), ws.data_ptr(), B, H, N, D,
                                 D, dtype_code(q.scalar_type()), stream_of(q)),
          "cott_cos_attn_wide_fwd");
    ctx->save_for_backward({q, k, v, nc, ws});
    save_opt(ctx, "keep", kp);
    save_nc(ctx, norm_const);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const at::Tensor &q = s[0], dout = dense_as(grads[0], q.scalar_type());
    const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), D = (int)q.size(3);
    const c10::cuda::CUDAGuard guard(q.device());
    at::Tensor dq = at::empty_like(q), dk = at::empty_like(s[1]), dv = at::empty_like(s[2]), dnc = at::empty({H}, q.options().dtype(at::kFloat));
    check(cott_cos_attn_wide_bwd(q.data_ptr(), s[1].data_ptr(), s[2].data_ptr(), u8(load_opt(ctx, "keep")), s[3].data_ptr<float>(), nullptr,
                                 dout.data_ptr(), s[4].data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dnc.data_ptr<float>(), B, H, N, D,
                                 D, dtype_code(q.scalar_type()), stream_of(q)),
          "cott_cos_attn_wide_bwd");
    return {dq, dk, dv, nc_grad(ctx, dnc), Variable()};
  }
};

// Custom_Kernel.py's CustomAttention: forward and the three permuted scans through the entry point of Q's dtype
at::Tensor scan_by_dtype(at::ScalarType t, at::Tensor Q, at::Tensor K, at::Tensor V, bool reversed) {
  return t == at::kHalf ? forward_<at::kHalf>(Q, K, V, 1, false, reversed) : forward_<at::kBFloat16>(Q, K, V, 1, false, reversed);
}
struct ScanFn : torch::autograd::Function<ScanFn> {
  // `entry`: the dtype whose entry point the scans go through
  static Variable forward(AutogradContext* ctx, const at::Tensor& Q, const at::Tensor& K, const at::Tensor& V, int64_t entry, bool reversed) {
    ctx->save_for_backward({Q, K, V});
    ctx->saved_data["scan"] = 2 * entry + (reversed ? 1 : 0);
    return scan_by_dtype((at::ScalarType)entry, Q, K, V, reversed);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const at::Tensor &Q = s[0], &K = s[1], &V = s[2], g = grads[0].contiguous();
    const int64_t scan = ctx->saved_data["scan"].toInt(), entry = scan / 2;
    const at::ScalarType t = (at::ScalarType)entry;
    const bool rev = scan % 2;
    if (at::GradMode::is_enabled())  // create_graph: the gradients are scans themselves, with nodes of their own
      return {apply(g, V, K, entry, rev), apply(V, g, Q, entry, !rev), apply(K, Q, g, entry, !rev), Variable(), Variable()};
    // one dtype and one shape in 16 bits: the three scans in one C call (autocast only ever concerns fp32 tensors)
    if (!rev && (t == at::kHalf || t == at::kBFloat16) && Q.scalar_type() == t && K.scalar_type() == t && V.scalar_type() == t && g.scalar_type() == t &&
        Q.dim() == 4 && Q.sizes() == K.sizes() && Q.sizes() == V.sizes() && Q.sizes() == g.sizes() && Q.size(3) == 64) {
      const c10::cuda::CUDAGuard guard(Q.device());
      at::Tensor dq = at::empty_like(Q), dk = at::empty_like(K), dv = at::empty_like(V);
      check(cott_scan_bwd(Q.data_ptr(), K.data_ptr(), V.data_ptr(), g.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), (int)Q.size(0),
                          (int)Q.size(1), (int)Q.size(2), 64, 64, dtype_code(t), stream_of(Q)),
            "cott_scan_bwd");
      return {dq, dk, dv, Variable(), Variable()};
    }
    return {scan_by_dtype(t, g, V, K, rev), scan_by_dtype(t, V, g, Q, !rev), scan_by_dtype(t, K, Q, g, !rev), Variable(), Variable()};
  }
};
// (dense before the node, so that what it saves is still connected to the caller's tensors)
at::Tensor custom_attention(const at::Tensor& Q, const at::Tensor& K, const at::Tensor& V) {
  return ScanFn::apply(Q.contiguous(), K.contiguous(), V.contiguous(), (int64_t)Q.scalar_type(), false);
}

// one decode call on a [B, H, Dv, Dk] state
at::Tensor decode_steps(const at::Tensor& state, const at::Tensor& q_, const at::Tensor& k_, const at::Tensor& v_, const at::Tensor& norm_const,
                        int64_t pos) {
  const at::Tensor q = q_.contiguous(), k = dense_as(k_.scalar_type() == q.scalar_type() ? k_ : k_.to(q.scalar_type()), q.scalar_type()),
                   v = dense_as(v_.scalar_type() == q.scalar_type() ? v_ : v_.to(q.scalar_type()), q.scalar_type());
  TORCH_CHECK(k.numel() == q.numel() && v.numel() == q.size(0) * q.size(1) * q.size(2) * v.size(3) &&
                  state.numel() >= q.size(0) * q.size(1) * v.size(3) * q.size(3),
              "q, k, v and the state do not fit each other: ", q.sizes(), ", ", k.sizes(), ", ", v.sizes(), ", ", state.sizes());
  const c10::cuda::CUDAGuard guard(q.device());
  const at::Tensor nc = nc_at_least(norm_const, q, q.size(1));
  at::Tensor out = at::empty({q.size(0), q.size(1), q.size(2), v.size(3)}, q.options());
  check(cott_decode_steps(state.data_ptr<float>(), q.data_ptr(), k.data_ptr(), v.data_ptr(), nc.data_ptr<float>(), out.data_ptr(), (int)q.size(0),
                          (int)q.size(1), (int)q.size(2), (int)q.size(3), (int)v.size(3), dtype_code(q.scalar_type()), pos, nullptr, stream_of(q)),
        "cott_decode_steps");
  return out;
}

// a whole prompt: outputs and the decode state it leaves (head dim 64 or 128)
at::Tensor prefill(const at::Tensor& state, const at::Tensor& q_, const at::Tensor& k_, const at::Tensor& v_, const at::Tensor& norm_const) {
  check_bhnd(q_, k_, v_);
  const at::Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
  const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), D = (int)q.size(3);
  TORCH_CHECK(state.numel() >= q.size(0) * q.size(1) * D * D, "the state is smaller than the prompt's ", B, " x ", H, " sequences need");
  const c10::cuda::CUDAGuard guard(q.device());
  const at::Tensor nc = nc_f32(norm_const, q, H);
  const int nseg = D == 128 ? 1 : cott_cos_attn_seg_choice(B, H, N);
  at::Tensor out = at::empty_like(v);
  const at::Tensor ws = bytes_like(q, D == 128 ? cott_cos_attn_wide_workspace_bytes(B, H, N) : cott_cos_attn_seg_workspace_bytes(B, H, N, nseg));
  check(cott_cos_attn_prefill(q.data_ptr(), k.data_ptr(), v.data_ptr(), nc.data_ptr<float>(), out.data_ptr(), state.data_ptr<float>(),
                              ws.data_ptr(), nseg, B, H, N, D, D, dtype_code(q.scalar_type()), stream_of(q)),
        "cott_cos_attn_prefill");
  return out;
}

// fp32, head dims 32 and 64
at::Tensor dense16(const at::Tensor& t) {
  at::Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 ? c.clone() : c;
}
// the module math in differentiable torch operators around the scan, for gradients that are differentiated again
at::Tensor exact_causal(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& norm_const, const OptTensor& keep) {
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2);
  at::Tensor qh = q / q.norm(2, -1, true).clamp_min(1e-12), kh = k / k.norm(2, -1, true).clamp_min(1e-12);
  const at::Tensor n = has(keep) ? keep->to(at::kLong).cumsum(-1).to(q.scalar_type()).view({B, 1, N, 1})
                                 : at::arange(1, N + 1, q.options()).view({1, 1, N, 1});
  at::Tensor vp = v / n.pow(norm_const.sigmoid().reshape({1, H, 1, 1})).clamp_min(1);
  if (has(keep)) {
    const at::Tensor m = keep->view({B, 1, N, 1}).to(q.scalar_type());
    qh = qh * m, kh = kh * m, vp = vp * m;
  }
  return custom_attention(qh, kh, vp);
}
struct F32Fn : torch::autograd::Function<F32Fn> {
  static Variable forward(AutogradContext* ctx, const at::Tensor& q_, const at::Tensor& k_, const at::Tensor& v_, const at::Tensor& norm_const,
                          const OptTensor& keep) {
    const at::Tensor q = dense16(q_), k = dense16(k_), v = dense16(v_), nc = norm_const.contiguous();
    const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), D = (int)q.size(3);
    const c10::cuda::CUDAGuard guard(q.device());
    at::Tensor out = at::empty(q.sizes(), q.options()), ws = bytes_like(q, cott_cos_attn_f32_workspace_bytes(B, H, N, D));
    check(cott_cos_attn_f32_fwd(q.data_ptr<float>(), k.data_ptr<float>(), v.data_ptr<float>(), u8(keep), nc.data_ptr<float>(), out.data_ptr<float>(),
                                ws.data_ptr(), B, H, N, D, stream_of(q)),
          "cott_cos_attn_f32_fwd");
    ctx->save_for_backward({q_, k_, v_, norm_const});
    ctx->saved_data["ws"] = ws;
    save_opt(ctx, "keep", keep);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const OptTensor keep = load_opt(ctx, "keep");
    if (at::GradMode::is_enabled()) {  // create_graph
      variable_list x, wanted;
      for (const at::Tensor& t : s) x.push_back(t.view_as(t));  // (one name per argument: the same tensor may be several of them)
      for (const at::Tensor& t : x)
        if (t.requires_grad()) wanted.push_back(t);
      variable_list g = torch::autograd::grad({exact_causal(x[0], x[1], x[2], x[3], keep)}, wanted, {grads[0]}, true, true, true);
      variable_list r(5);
      for (size_t i = 0, j = 0; i < 4; ++i)
        if (x[i].requires_grad()) r[i] = g[j++];
      return r;
    }
    const at::Tensor q = dense16(s[0]), k = dense16(s[1]), v = dense16(s[2]), nc = s[3].contiguous(), dout = dense16(grads[0]);
    const int B = (int)q.size(0), H = (int)q.size(1), N = (int)q.size(2), D = (int)q.size(3);
    const c10::cuda::CUDAGuard guard(q.device());
    at::Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v), dnc = at::empty_like(nc);
    const at::Tensor ws = bytes_like(q, cott_cos_attn_f32_workspace_bytes(B, H, N, D));
    check(cott_cos_attn_f32_bwd(q.data_ptr<float>(), k.data_ptr<float>(), v.data_ptr<float>(), u8(keep), nc.data_ptr<float>(),
                                dout.data_ptr<float>(), ctx->saved_data["ws"].toTensor().data_ptr(), ws.data_ptr(), dq.data_ptr<float>(),
                                dk.data_ptr<float>(), dv.data_ptr<float>(), dnc.data_ptr<float>(), B, H, N, D, stream_of(q)),
          "cott_cos_attn_f32_bwd");
    return {dq, dk, dv, dnc, Variable()};
  }
};

// what Python calls
at::Tensor cos_attn_causal(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& norm_const, const OptTensor& keep,
                           int64_t nseg, bool one_pass) {
  return CausalFn::apply(q, k, v, norm_const, keep, nseg, one_pass);
}
at::Tensor cos_attn_wide(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& norm_const, const OptTensor& keep) {
  return WideFn::apply(q, k, v, norm_const, keep);
}
// (private copies of the parameter and of the mask: neither is read at its own address again after this call)
at::Tensor cos_attn_f32(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& norm_const, const OptTensor& keep) {
  return F32Fn::apply(q, k, v, norm_const.clone(), has(keep) ? OptTensor(keep->clone(at::MemoryFormat::Contiguous)) : OptTensor());
}
at::Tensor causal_packed(const at::Tensor& qkv, const at::Tensor& norm_const, const OptTensor& keep, const OptTensor& sin, const OptTensor& cos,
                         bool keep_rotated) {
  return CausalPackedFn::apply(qkv, norm_const, keep, sin, cos, keep_rotated);
}
at::Tensor bidir_packed(const at::Tensor& qkv, const at::Tensor& norm_const, const OptTensor& keep) {
  return BidirPackedFn::apply(qkv, norm_const, keep);
}

}  // namespace

TORCH_LIBRARY(cottention_b200, m) {
  m.def("causal_fwd(Tensor q, Tensor k, Tensor v, Tensor norm_const, Tensor? keep, int nseg, bool save_states) -> (Tensor, Tensor, Tensor)");
  m.def("causal_bwd(Tensor q, Tensor k, Tensor v, Tensor norm_const, Tensor? keep, Tensor dout, Tensor ws, Tensor saved, int nseg) -> (Tensor, Tensor, Tensor, Tensor)");
  m.def("bidir_fwd(Tensor q, Tensor k, Tensor v, Tensor norm_const, Tensor? keep) -> (Tensor, Tensor)");
  m.def("bidir_bwd(Tensor q, Tensor k, Tensor v, Tensor norm_const, Tensor? keep, Tensor dout, Tensor scratch) -> (Tensor, Tensor, Tensor, Tensor)");
}
TORCH_LIBRARY_IMPL(cottention_b200, CUDA, m) {
  m.impl("causal_fwd", &causal_fwd);
  m.impl("causal_bwd", &causal_bwd);
  m.impl("bidir_fwd", &bidir_fwd);
  m.impl("bidir_bwd", &bidir_bwd);
}

// The reference registers its four functions with pybind (combined_kernel_general.cu:444-454); the argument names and
// defaults are its own.
PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  // how a non-zero status of the C ABI surfaces in Python: RuntimeError carrying the status text and the library's message
  m.def("_raise_for_status", [](int status) { check(status, "cottention_b200"); }, py::arg("status"));
  // Without the interpreter lock, as calls through ctypes and torch.ops run: a launch may wait for room in the stream's
  // queue, and what the queue waits for may be another Python thread.
  using Unlocked = py::call_guard<py::gil_scoped_release>;
  m.def("cos_attn_causal", &cos_attn_causal, Unlocked());
  m.def("cos_attn_wide", &cos_attn_wide, Unlocked());
  m.def("cos_attn_f32", &cos_attn_f32, Unlocked());
  m.def("causal_packed", &causal_packed, Unlocked());
  m.def("bidir_packed", &bidir_packed, Unlocked());
  m.def("custom_attention", &custom_attention, Unlocked());
  m.def("decode_steps", &decode_steps, Unlocked());
  m.def("prefill", &prefill, Unlocked());
  m.def("float32", &forward_<at::kBFloat16>, "FastAttention forward (float32 entry point)", py::arg("Q"), py::arg("K"), py::arg("V"),
        py::arg("block_size"), py::arg("inplace") = false, py::arg("reversed") = false);
  m.def("float64", &forward_<at::kBFloat16>, "FastAttention forward (float64 entry point)", py::arg("Q"), py::arg("K"), py::arg("V"),
        py::arg("block_size"), py::arg("inplace") = false, py::arg("reversed") = false);
  m.def("float16", &forward_<at::kHalf>, "FastAttention forward (float16 entry point)", py::arg("Q"), py::arg("K"), py::arg("V"),
        py::arg("block_size"), py::arg("inplace") = false, py::arg("reversed") = false);
  m.def("bfloat16", &forward_<at::kBFloat16>, "FastAttention forward (bfloat16 entry point)", py::arg("Q"), py::arg("K"), py::arg("V"),
        py::arg("block_size"), py::arg("inplace") = false, py::arg("reversed") = false);
}
