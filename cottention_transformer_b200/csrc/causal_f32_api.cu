// C ABI of the fused fp32 causal cosine attention (CUDA cores).
#include "causal_f32.cuh"

using namespace cott;

namespace {

int check_f32_args(int B, int H, int N, int D) {
  if (B < 0 || H < 0 || N < 0) return fail(COTT_ERR_SHAPE, "negative size B=%d H=%d N=%d", B, H, N);
  if (D != 32 && D != 64) return fail(COTT_ERR_UNSUPPORTED, "the fused fp32 path is built for head dims 32 and 64 (got %d)", D);
  if ((long)B * H * ((N + kF32Chunk - 1) / kF32Chunk) > 0x7fffffffL) return fail(COTT_ERR_SHAPE, "B*H*N too large");
  return COTT_OK;
}
int check_f32_ptrs(std::initializer_list<const void*> ps) {
  for (const void* p : ps) {
    if (!p) return fail(COTT_ERR_NULL, "null tensor pointer");
    if (reinterpret_cast<uintptr_t>(p) & 15) return fail(COTT_ERR_ALIGN, "tensors must be 16-byte aligned");
  }
  return COTT_OK;
}
int f32_chunks(int N) { return (N + kF32Chunk - 1) / kF32Chunk; }
size_t f32_state_floats(int B, int H, int N, int D) { return (size_t)B * H * f32_chunks(N) * D * D; }

template <int D, bool REV>
int launch_f32_states(const float* y, const float* z, const unsigned char* keep, const float* nc, float* state, int B, int H, int N,
                      cudaStream_t stream) {
  const int nch = f32_chunks(N);
  const unsigned grid = (unsigned)((long)B * H * nch);
  COTT_CUDA_TRY(launch_pdl(f32_state_kernel<D, REV>, dim3(grid), kF32Threads, 2 * kF32Chunk * (D + 4) * sizeof(float), stream, y, z, keep, nc,
                           state, H, N, nch));
  COTT_CUDA_TRY(launch_pdl(f32_prefix_kernel<REV>, dim3((unsigned)((long)B * H), D * D / kF32Threads), kF32Threads, 0, stream, state, nch, D * D));
  return COTT_OK;
}

template <int D, bool FWD>
int launch_f32_chunks(const F32Args& g, int B, cudaStream_t stream) {
  const size_t smem = (3 * kF32Chunk * (D + 4) + kF32Chunk * (kF32Chunk + 4)) * sizeof(float);
  auto kern = f32_chunk_kernel<D, FWD>;
  COTT_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  COTT_CUDA_TRY(launch_pdl(kern, dim3((unsigned)((long)B * g.H * g.nchunks), FWD ? 1 : 3), kF32Threads, smem, stream, g));
  return COTT_OK;
}

template <int D>
int run_f32_fwd(F32Args g, float* ws, int B, cudaStream_t stream) {
  int st = launch_f32_states<D, false>(g.k, g.v, g.keep, g.norm_const, ws, B, g.H, g.N, stream);
  if (st) return st;
  g.prefix = ws;
  return launch_f32_chunks<D, true>(g, B, stream);
}

template <int D>
int run_f32_bwd(F32Args g, const float* fwd_ws, float* ws, float* dnorm, int B, cudaStream_t stream) {
  const size_t A = f32_state_floats(B, g.H, g.N, D);
  int st = launch_f32_states<D, true>(g.q, g.dout, g.keep, g.norm_const, ws, B, g.H, g.N, stream);
  if (st) return st;
  g.prefix = fwd_ws;
  g.suffix = ws;
  g.gpart = reinterpret_cast<double*>(ws + A);
  if ((st = launch_f32_chunks<D, false>(g, B, stream))) return st;
  COTT_CUDA_TRY(launch_pdl(f32_dnorm_kernel, dim3((unsigned)g.H), kF32Threads, 0, stream, static_cast<const double*>(g.gpart), g.norm_const, dnorm, B,
                           g.H, g.nchunks));
  return COTT_OK;
}

}  // namespace

extern "C" {

size_t cott_cos_attn_f32_workspace_bytes(int B, int H, int N, int D) {
  if (B <= 0 || H <= 0 || N <= 0 || D <= 0) return 0;
  return f32_state_floats(B, H, N, D) * sizeof(float) + (size_t)B * H * f32_chunks(N) * sizeof(double);
}

int cott_cos_attn_f32_fwd(const float* q, const float* k, const float* v, const unsigned char* keep, const float* norm_const, float* out,
                          void* workspace, int B, int H, int N, int D, void* stream) {
  int st = check_f32_args(B, H, N, D);
  if (st) return st;
  if ((long)B * H * N == 0) return COTT_OK;
  if ((st = check_f32_ptrs({q, k, v, out, workspace}))) return st;
  if (!norm_const) return fail(COTT_ERR_NULL, "null pointer: norm_const");
  DeviceScope scope(q);
  COTT_CUDA_TRY(scope.status());
  F32Args g = {};
  g.q = q, g.k = k, g.v = v, g.keep = keep, g.norm_const = norm_const, g.out = out, g.H = H, g.N = N, g.nchunks = f32_chunks(N);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float* ws = static_cast<float*>(workspace);
  return D == 64 ? run_f32_fwd<64>(g, ws, B, s) : run_f32_fwd<32>(g, ws, B, s);
}

int cott_cos_attn_f32_bwd(const float* q, const float* k, const float* v, const unsigned char* keep, const float* norm_const,
                          const float* dout, const void* fwd_workspace, void* workspace, float* dq, float* dk, float* dv,
                          float* dnorm_const, int B, int H, int N, int D, void* stream) {
  int st = check_f32_args(B, H, N, D);
  if (st) return st;
  if (!dnorm_const && H > 0) return fail(COTT_ERR_NULL, "null pointer: dnorm_const");
  if ((long)B * H * N == 0) {
    if (H > 0) COTT_CUDA_TRY(cudaMemsetAsync(dnorm_const, 0, sizeof(float) * H, static_cast<cudaStream_t>(stream)));
    return COTT_OK;
  }
  if ((st = check_f32_ptrs({q, k, v, dout, fwd_workspace, workspace, dq, dk, dv}))) return st;
  if (!norm_const) return fail(COTT_ERR_NULL, "null pointer: norm_const");
  DeviceScope scope(q);
  COTT_CUDA_TRY(scope.status());
  F32Args g = {};
  g.q = q, g.k = k, g.v = v, g.dout = dout, g.keep = keep, g.norm_const = norm_const, g.dq = dq, g.dk = dk, g.dv = dv;
  g.H = H, g.N = N, g.nchunks = f32_chunks(N);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float* fws = static_cast<const float*>(fwd_workspace);
  float* ws = static_cast<float*>(workspace);
  return D == 64 ? run_f32_bwd<64>(g, fws, ws, dnorm_const, B, s) : run_f32_bwd<32>(g, fws, ws, dnorm_const, B, s);
}

}  // extern "C"
