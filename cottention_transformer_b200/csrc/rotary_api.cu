// Rotary position embedding of the reference's GPT module (GPT_Trainer/GPTCosAttention.py:458-476, the GPT-J
// "rotate every two" form of transformers' apply_rotary_pos_emb), applied in place to q and k wherever they
// lie -- e.g. the q and k slices of a packed [B, N, 3, H, d] projection output -- in one pass:
//   x'[2i]   = x[2i] cos_i - x[2i+1] sin_i
//   x'[2i+1] = x[2i+1] cos_i + x[2i] sin_i          i < rot_dim / 2, the other elements pass through
// `inverse` applies the transposed rotation (sin -> -sin), which is the backward of the op.
// HBM-bound elementwise work: one 16-byte piece (four pairs) per thread, fp32 arithmetic, one read and one write
// of q and k; the tables are [N, rot_dim/2] fp32 (per batch entry when `table_batch_stride` is not 0).
#include "common.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

using namespace cott;

namespace {

template <typename T> struct Pair16;
template <> struct Pair16<__nv_bfloat16> {
  static __device__ __forceinline__ float2 unpack(uint32_t u) { return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};
template <> struct Pair16<__half> {
  static __device__ __forceinline__ float2 unpack(uint32_t u) { return __half22float2(*reinterpret_cast<__half2*>(&u)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};

// One thread per 16-byte piece of a row, for q and k both (same sin / cos); blockIdx.y walks the batch.  `all` pieces of
// a row are moved from (q, k) to (oq, ok), the first `pieces` of them rotated; in place (the same pointers and strides)
// only the rotated ones are touched.  Index arithmetic in 32 bits where a batch entry has fewer than 2^32 pieces: with
// 64-bit divisions the kernel was bound by them (B 8, H 16, N 1024, rotary dim 64: 12.9 -> 10.8 us, in place or copying).
struct RotStrides {
  long long b, h, n;
};
template <typename T, typename I>
__global__ void __launch_bounds__(256)
rotary_kernel(const T* q, const T* k, T* oq, T* ok, const float* __restrict__ sin_t, const float* __restrict__ cos_t, RotStrides si,
              RotStrides so, int B, I H, I N, I pieces, I all, long long table_batch_stride, float sign, bool h_inner) {
  pdl_allow_next();  // (the causal kernels that follow set themselves up meanwhile)
  pdl_wait_prior();
  const I idx = static_cast<I>(blockIdx.x) * 256 + threadIdx.x;
  if (idx >= H * N * all) return;
  const I row = idx / all, p = idx - row * all;
  // consecutive threads walk the dimension with the smaller stride (heads in a packed [B, N, 3, H, d] tensor)
  const I inner = h_inner ? H : N, hi = row / inner, lo = row - hi * inner;
  const I n = h_inner ? hi : lo, h = h_inner ? lo : hi;
  for (int b = blockIdx.y; b < B; b += gridDim.y) {
    const long long in = b * si.b + h * si.h + n * si.n + p * 8, out = b * so.b + h * so.h + n * so.n + p * 8;
    uint4 u[2] = {*reinterpret_cast<const uint4*>(q + in), *reinterpret_cast<const uint4*>(k + in)};
    if (p < pieces) {
      const long long t = b * table_batch_stride + static_cast<long long>(n) * (pieces * 4) + p * 4;
      const float4 s4 = *reinterpret_cast<const float4*>(sin_t + t), c4 = *reinterpret_cast<const float4*>(cos_t + t);
      const float s[4] = {sign * s4.x, sign * s4.y, sign * s4.z, sign * s4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
      for (int t2 = 0; t2 < 2; ++t2) {
        uint32_t* w = reinterpret_cast<uint32_t*>(&u[t2]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = Pair16<T>::unpack(w[e]);
          float xo, yo;
          rot_pair(f.x, f.y, c[e], s[e], xo, yo);
          w[e] = Pair16<T>::pack(xo, yo);
        }
      }
    }
    *reinterpret_cast<uint4*>(oq + out) = u[0];
    *reinterpret_cast<uint4*>(ok + out) = u[1];
  }
}

template <typename T>
int launch_rotary(const void* q, const void* k, void* oq, void* ok, const float* sin_t, const float* cos_t, RotStrides si, RotStrides so,
                  int B, int H, int N, int pieces, int all, long long table_batch_stride, float sign, cudaStream_t stream) {
  const unsigned long long per = static_cast<unsigned long long>(H) * N * all;
  if (per > 256ull * 0x7fffffffull) return fail(COTT_ERR_SHAPE, "H*N too large");
  const dim3 grid(static_cast<unsigned>((per + 255) / 256), B < 65535 ? B : 65535);
  const bool h_inner = si.h < si.n;
  const T *qt = static_cast<const T*>(q), *kt = static_cast<const T*>(k);
  T *oqt = static_cast<T*>(oq), *okt = static_cast<T*>(ok);
  if (per + 256 < (1ull << 32))
    COTT_CUDA_TRY(launch_pdl(rotary_kernel<T, unsigned>, grid, 256, 0, stream, qt, kt, oqt, okt, sin_t, cos_t, si, so, B, (unsigned)H, (unsigned)N,
                             (unsigned)pieces, (unsigned)all, table_batch_stride, sign, h_inner));
  else
    COTT_CUDA_TRY(launch_pdl(rotary_kernel<T, unsigned long long>, grid, 256, 0, stream, qt, kt, oqt, okt, sin_t, cos_t, si, so, B,
                             (unsigned long long)H, (unsigned long long)N, (unsigned long long)pieces, (unsigned long long)all,
                             table_batch_stride, sign, h_inner));
  return COTT_OK;
}

int check_rotary_args(std::initializer_list<const void*> ptrs, int B, int H, int N, int D, int rot_dim, long long table_batch_stride, int dtype,
                      std::initializer_list<RotStrides> strides) {
  if (dtype != COTT_BF16 && dtype != COTT_F16)
    return fail(COTT_ERR_DTYPE, "cott_rotary takes float16 / bfloat16 (dtype code %d)", dtype);
  if (B < 0 || H < 0 || N < 0) return fail(COTT_ERR_SHAPE, "negative size B=%d H=%d N=%d", B, H, N);
  if (D < 8 || D % 8 || rot_dim < 8 || rot_dim % 8 || rot_dim > D)
    return fail(COTT_ERR_SHAPE, "head dim and rotary dim must be multiples of 8 with rot_dim <= D (got %d, %d)", D, rot_dim);
  if ((long)B * H * N == 0) return COTT_OK;
  for (const void* p : ptrs)
    if (!p) return fail(COTT_ERR_NULL, "null pointer");
  for (const RotStrides& st : strides)
    if ((st.b | st.h | st.n) & 7) return fail(COTT_ERR_ALIGN, "strides must be multiples of 8 elements");
  if (table_batch_stride & 3) return fail(COTT_ERR_ALIGN, "strides must be multiples of 8 elements");
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) return fail(COTT_ERR_ALIGN, "tensors must be 16-byte aligned");
  return COTT_OK;
}
RotStrides rot_strides(const cott_layout* l, int H, int N, int D) {
  return l ? RotStrides{l->in_b, l->in_h, l->in_n} : RotStrides{(long long)H * N * D, (long long)N * D, D};
}

}  // namespace

extern "C" {

int cott_rotary(void* q, void* k, const float* sin_table, const float* cos_table, const cott_layout* layout, int B, int H, int N, int D,
                int rot_dim, long long table_batch_stride, int inverse, int dtype, void* stream) {
  const RotStrides st = rot_strides(layout, H, N, D);
  int r = check_rotary_args({q, k, sin_table, cos_table}, B, H, N, D, rot_dim, table_batch_stride, dtype, {st});
  if (r || (long)B * H * N == 0) return r;
  DeviceScope scope(q);
  COTT_CUDA_TRY(scope.status());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float sign = inverse ? -1.f : 1.f;
  return dtype == COTT_BF16 ? launch_rotary<__nv_bfloat16>(q, k, q, k, sin_table, cos_table, st, st, B, H, N, rot_dim / 8, rot_dim / 8,
                                                          table_batch_stride, sign, s)
                            : launch_rotary<__half>(q, k, q, k, sin_table, cos_table, st, st, B, H, N, rot_dim / 8, rot_dim / 8,
                                                    table_batch_stride, sign, s);
}

int cott_rotary_copy(const void* q, const void* k, void* q_out, void* k_out, const float* sin_table, const float* cos_table,
                     const cott_layout* layout, const cott_layout* out_layout, int B, int H, int N, int D, int rot_dim,
                     long long table_batch_stride, int dtype, void* stream) {
  const RotStrides si = rot_strides(layout, H, N, D), so = rot_strides(out_layout, H, N, D);
  int r = check_rotary_args({q, k, q_out, k_out, sin_table, cos_table}, B, H, N, D, rot_dim, table_batch_stride, dtype, {si, so});
  if (r || (long)B * H * N == 0) return r;
  DeviceScope scope(q);
  COTT_CUDA_TRY(scope.status());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return dtype == COTT_BF16 ? launch_rotary<__nv_bfloat16>(q, k, q_out, k_out, sin_table, cos_table, si, so, B, H, N, rot_dim / 8, D / 8,
                                                          table_batch_stride, 1.f, s)
                            : launch_rotary<__half>(q, k, q_out, k_out, sin_table, cos_table, si, so, B, H, N, rot_dim / 8, D / 8,
                                                    table_batch_stride, 1.f, s);
}

}  // extern "C"
