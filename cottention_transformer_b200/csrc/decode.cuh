// Recurrent decode step of cosine attention (HBM-bound, CUDA cores).
//
// Per (batch, head) the reference keeps a d_v x d_k state and, per generated token
// (GPT_Trainer/GPTCosAttention.py:229-230,236,253-272):
//     q^ = q/|q|,  k^ = k/|k|,  v' = v / max(pos^sigmoid(c_h), 1)          pos = 1-based position
//     state[j][i] += v'[j] * k^[i]                                          (:264, layout [d_v, d_k])
//     out[j]       = sum_i q^[i] * state[j][i]                              (:267)
// The reference runs this on the CPU in float64 for batch 1; here the state is fp32 in HBM,
// [B, H, d_v, d_k], updated in place.  A CTA owns some rows of a (b,h) state (they are independent of each other); a row of the state is spread over d_k/4 lanes that each own one float4, so
// every state access is a coalesced 128-bit access and the row dot product is a shuffle reduction.
//
// cott_decode_steps runs T consecutive positions in one launch with the state held in registers
// between steps (it is read from and written to HBM once), which is also how a prompt is absorbed.
#pragma once

#include "common.cuh"

namespace cott {

// How a state is spread: state rows (held in registers) and threads of a CTA, CTAs per SM (the register budget), and whether a
// state may be more than one CTA.  Bound by HBM for one token a call, by the token loop's latency for several.
// Measured, us a call (device time, launches back to back, state in fp32):
//   d = 64, 64 rows x 128 threads.  Eight CTAs per SM leave 64 registers and spill in the token loop, seven do not, and the 1024
//     states of a batch-64, 16-head step are still one wave: one token 7.2 -> 6.2, 16 tokens 49.9 -> 40.8 (fp32 tokens 48.2 ->
//     40.2).  The first row and the row count of a split state, as run-time values, cost the same loop 3-8 % (52.3, 52.1).
//   d = 128, 32 rows x 128 threads x 7, a state in four CTAs: their loads, products and stores are at different points and the
//     last wave is short.  A whole state per CTA (256 threads x 2): one token 27.6 -> 26.5 for 1024 states, 5.0 -> 3.6 for 32; 16
//     tokens 202 -> 171, 47.0 -> 32.9 for 128.  (With eight per SM 128 states took 48.7.)
//   d = 128, one token and 1024 states or more: 64 rows x 128 threads x 4, which load q and k half as often.  1024 states 26.5 ->
//     25.8, 4096 states 96.3 -> 88.8, 8192 with fp32 tokens 190.5 -> 172.4; below, and for more tokens, it is the slower one
//     (512 states 14.9 -> 15.3, 1024 states with four tokens 52.6 -> 58.1).
template <int ROWS, int THREADS, int CTAS, bool SPLIT> struct DecodeCfg {
  static constexpr int kRows = ROWS, kThreads = THREADS, kCtas = CTAS;
  static constexpr bool kSplit = SPLIT;
};

template <typename T>
__device__ __forceinline__ float ld_as_float(const T* p) { return to_acc(*p); }

// q, k: [B,H,T,Dk]  v, out: [B,H,T,Dv] (T = 1 for a single step); state: [B,H,Dv,Dk] fp32.
// positions: optional [B] int64 array of the 1-based position of the FIRST token of this call for
// each batch entry; if null, `pos0` is used for all.  LPR = lanes per state row = Dk/4.
// (the kernel is latency-bound on its state loads, so resident CTAs are what hides the HBM latency)
template <typename T, int DK, typename CFG>
__global__ void __launch_bounds__(CFG::kThreads, CFG::kCtas)
decode_kernel(float* __restrict__ state, const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
              const float* __restrict__ norm_const, T* __restrict__ out, int H, int Dv, int Tsteps, long long pos0,
              const long long* __restrict__ positions) {
  constexpr int ROWS = CFG::kRows;
  constexpr int LPR = DK / 4;                    // lanes per row (4, 8, 16 or 32)
  constexpr int ROWS_PER_PASS = CFG::kThreads / LPR;
  constexpr int MAXR = (ROWS + ROWS_PER_PASS - 1) / ROWS_PER_PASS;  // state rows held per thread
  __shared__ float sq[DK], sk[DK], sv[ROWS];
  __shared__ float red[2][CFG::kThreads / 32];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long bh = blockIdx.x;
  const int b = static_cast<int>(bh / H), h = static_cast<int>(bh % H);
  // Programmatic dependent launch: a token-by-token loop is a chain of these launches, each waiting for the state the
  // one before wrote.  The launch is allowed to begin while its predecessor in the stream is still draining (its CTAs
  // are placed as slots free up, instead of after the whole grid has retired and a launch gap has passed); nothing
  // that another kernel may have produced -- state, q, k, v, norm_const -- is read before the wait below.
  pdl_allow_next();
  pdl_wait_prior();
  const float sigma = 1.0f / (1.0f + __expf(-norm_const[h]));
  const long long p0 = positions ? positions[b] : pos0;
  const int piece = tid % LPR;        // which float4 of the row
  const int j0 = CFG::kSplit ? static_cast<int>(blockIdx.y) * ROWS : 0;  // first row of this CTA
  const int rows = CFG::kSplit ? min(ROWS, Dv - j0) : Dv;
  const int row0 = tid / LPR;         // first row of this thread, in the CTA; then += ROWS_PER_PASS

  float* st = state + (bh * static_cast<long>(Dv) + j0) * DK;
  float4 s[MAXR];
#pragma unroll
  for (int r = 0; r < MAXR; ++r) {
    const int j = row0 + r * ROWS_PER_PASS;
    s[r] = (j < rows) ? *reinterpret_cast<const float4*>(st + static_cast<long>(j) * DK + 4 * piece)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
  }

  for (int t = 0; t < Tsteps; ++t) {
    const T* qt = q + (bh * Tsteps + t) * static_cast<long>(DK);
    const T* kt = k + (bh * Tsteps + t) * static_cast<long>(DK);
    const T* vt = v + (bh * Tsteps + t) * static_cast<long>(Dv) + j0;
    // stage q, k, v and their norms
    float x = 0.f, y = 0.f;
    if (tid < DK) {
      x = ld_as_float(qt + tid);
      y = ld_as_float(kt + tid);
      sq[tid] = x;
      sk[tid] = y;
    }
    if (tid < rows) sv[tid] = ld_as_float(vt + tid);
    float xx = x * x, yy = y * y;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      xx += __shfl_xor_sync(0xffffffffu, xx, off);
      yy += __shfl_xor_sync(0xffffffffu, yy, off);
    }
    if (lane == 0) {
      red[0][warp] = xx;
      red[1][warp] = yy;
    }
    __syncthreads();
    float nq = 0.f, nk = 0.f;
#pragma unroll
    for (int w = 0; w < CFG::kThreads / 32; ++w) {
      nq += red[0][w];
      nk += red[1][w];
    }
    const float rq = 1.0f / fmaxf(sqrtf(nq), 1e-12f);
    const float rk = 1.0f / fmaxf(sqrtf(nk), 1e-12f);
    const float a = 1.0f / fmaxf(exp2f(sigma * log2f(static_cast<float>(p0 + t))), 1.0f);
    const float4 k4 = *reinterpret_cast<const float4*>(sk + 4 * piece);
    const float4 q4 = *reinterpret_cast<const float4*>(sq + 4 * piece);
    const float ws = rk * a;
#pragma unroll
    for (int r = 0; r < MAXR; ++r) {
      const int j = row0 + r * ROWS_PER_PASS;
      const bool valid = j < rows;  // the same for all LPR lanes of a row; rows of one warp may differ
      const float vj = valid ? sv[j] * ws : 0.f;
      s[r].x += vj * k4.x;
      s[r].y += vj * k4.y;
      s[r].z += vj * k4.z;
      s[r].w += vj * k4.w;
      float dot = q4.x * s[r].x + q4.y * s[r].y + q4.z * s[r].z + q4.w * s[r].w;
#pragma unroll
      for (int off = LPR / 2; off > 0; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off, LPR);
      if (valid && piece == 0) out[(bh * Tsteps + t) * static_cast<long>(Dv) + j0 + j] = from_acc<T>(dot * rq);
    }
    __syncthreads();  // sq/sk/sv/red are rewritten by the next step
  }

#pragma unroll
  for (int r = 0; r < MAXR; ++r) {
    const int j = row0 + r * ROWS_PER_PASS;
    if (j < rows) *reinterpret_cast<float4*>(st + static_cast<long>(j) * DK + 4 * piece) = s[r];
  }
}

inline int decode_sms() {
  int sm = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
  return sm;
}
template <typename T> struct DecodeCall {
  float* state;
  const T *q, *k, *v;
  const float* nc;
  T* out;
  unsigned states;
  int H, Dv, T_steps;
  long long pos0;
  const long long* positions;
  cudaStream_t stream;
};
template <typename T, int DK, typename CFG>
int launch_decode_as(const DecodeCall<T>& c) {
  COTT_CUDA_TRY(launch_pdl(decode_kernel<T, DK, CFG>, dim3(c.states, (c.Dv + CFG::kRows - 1) / CFG::kRows), CFG::kThreads, 0, c.stream, c.state, c.q,
                           c.k, c.v, c.nc, c.out, c.H, c.Dv, c.T_steps, c.pos0, c.positions));
  return COTT_OK;
}
// Seven CTAs per SM or eight, for the splits that have the choice: a CTA takes about 8/7 as long with eight, but where they save a
// wave they are the better ones (d = 64, eight tokens: 1036 states 22.2 us in one wave of seven, 1040 26.6 in one of eight, 1200 31.2 in two).
template <typename T, int DK, int ROWS, bool SPLIT>
int launch_decode_waves(const DecodeCall<T>& c) {
  const long n = static_cast<long>(c.states) * ((c.Dv + ROWS - 1) / ROWS), s7 = 7l * decode_sms(), s8 = 8l * decode_sms();
  return 8 * ((n + s8 - 1) / s8) < 7 * ((n + s7 - 1) / s7) ? launch_decode_as<T, DK, DecodeCfg<ROWS, 128, 8, SPLIT>>(c)
                                                          : launch_decode_as<T, DK, DecodeCfg<ROWS, 128, 7, SPLIT>>(c);
}
// `whole`: every state by one CTA
template <typename T, int DK>
int launch_decode_dk(const DecodeCall<T>& c, bool whole) {
  if constexpr (DK == 128) {
    // (several tokens, and states that are one wave by themselves but not in four CTAs of seven per SM: 272 states, eight fp32
    // tokens 25.6 us against 27.0 in four CTAs of eight)
    if (c.T_steps > 1 && c.states <= 2u * decode_sms() && 4l * c.states > 7l * decode_sms()) whole = true;
    if (whole) return launch_decode_as<T, DK, DecodeCfg<128, 256, 2, false>>(c);
    if (c.T_steps == 1 && c.states >= 1024) return launch_decode_as<T, DK, DecodeCfg<64, 128, 4, true>>(c);
    return launch_decode_waves<T, DK, 32, true>(c);
  } else {
    if (whole && c.Dv > 64) return launch_decode_as<T, DK, DecodeCfg<128, 256, 4, false>>(c);
    if constexpr (DK == 64) return c.Dv <= 64 ? launch_decode_waves<T, DK, 64, false>(c) : launch_decode_waves<T, DK, 64, true>(c);
    return c.Dv <= 64 ? launch_decode_as<T, DK, DecodeCfg<64, 128, 8, false>>(c) : launch_decode_as<T, DK, DecodeCfg<64, 128, 8, true>>(c);
  }
}

template <typename T>
int launch_decode(float* state, const void* q, const void* k, const void* v, const float* nc, void* out, int B, int H,
                  int Dk, int Dv, int T_steps, long long pos0, const long long* positions, cudaStream_t stream) {
  const unsigned states = static_cast<unsigned>(static_cast<long>(B) * H);
  // Every CTA of a state reads the whole of q and k (and its own part of v), at its own time.  Tokens that `out` is written
  // over are therefore read by one CTA per state, which has read a token when it stores the output of it.
  const size_t tokens = static_cast<size_t>(states) * T_steps * sizeof(T);
  auto overlaps = [&](const void* p, int d) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), o = reinterpret_cast<uintptr_t>(out);
    return a < o + tokens * Dv && o < a + tokens * d;
  };
  const bool whole = overlaps(q, Dk) || overlaps(k, Dk) || (out != v && overlaps(v, Dv));
  const DecodeCall<T> c = {state, static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), nc, static_cast<T*>(out), states, H,
                           Dv, T_steps, pos0, positions, stream};
  int st = COTT_OK;
  switch (Dk) {
    case 16: st = launch_decode_dk<T, 16>(c, whole); break;
    case 32: st = launch_decode_dk<T, 32>(c, whole); break;
    case 64: st = launch_decode_dk<T, 64>(c, whole); break;
    case 128: st = launch_decode_dk<T, 128>(c, whole); break;
    default: return fail(COTT_ERR_SHAPE, "decode supports D_attn in {16, 32, 64, 128} (got %d)", Dk);
  }
  if (st) return st;
  COTT_CUDA_TRY(cudaGetLastError());
  return COTT_OK;
}

}  // namespace cott
