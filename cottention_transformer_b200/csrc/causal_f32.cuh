// Fused causal cosine attention in fp32 on CUDA cores, head dims 32 and 64: the mode that is used to check a model.
//
// Math (GPT_Trainer/GPTCosAttention.py:229-248,282 and its backward, see causal_tc.cuh), with every product and sum in
// fp32 and the module's own roundings: q^ = q / max(|q|, 1e-12), k^ likewise, v' = v / max(n_s^sigma, 1), masked rows zero.
//
// The sequence is cut into chunks of 64 positions, from its start for the passes that run forward and from its end for those that
// run backward (a sum that starts with a whole chunk needs the state for fewer rows: the error of dk and dv against 64 bits over
// sequences of 64 to 1024 is 2.2e-7, with one grid for both directions it was 2.3e-7), and EVERY chunk of EVERY (batch, head)
// is a CTA of its own:
//   1. f32_state_kernel    the chunk's own state  sum_s y_s (x) z_s   (forward: k^, v'; reverse: q^, dO)
//   2. f32_prefix_kernel   exclusive prefix (suffix) over the chunks of a sequence, in place
//   3. f32_chunk_kernel    the rows of the chunk: mask(A B^T) C + A M with M the state before (after) the chunk
// The backward runs step 3 for dq, dk and dv as three independent CTAs per chunk; all four passes are the same product
// chain with other operands:
//   out: A = q^  B = k^  C = v'  M = S       dq: A = dO  B = v'  C = k^  M = S^T
//   dk:  A = v'  B = dO  C = q^  M = R^T     dv: A = k^  B = q^  C = dO  M = R
// All of them are launched with programmatic dependent launch (common.cuh): seven short kernels in a row (113 -> 108 us a step
// at the sizes below).
// Bound by the fp32 FMA rate and the staging before it (256 CTAs at B 2, H 8, N 1024: 3 x 64^3 multiply-adds each).
// Measured there, forward + backward: 104 us a step (11 + 7 + 20 | 10 + 6 + 52 + 3 one by one); B 8, H 16, N 1024 521 us;
// four exact scans with one CTA per sequence (16 of 148 SMs busy, 236 us each) between fifty elementwise passes took 1206 us.
#pragma once

#include "common.cuh"

namespace cott {

constexpr int kF32Chunk = 64;
constexpr int kF32Threads = 256;
constexpr float kF32Eps = 1e-12f;  // F.normalize

enum { kF32Out = 0, kF32Dq = 1, kF32Dk = 2, kF32Dv = 3 };
enum { kF32Raw = 0, kF32Norm = 1, kF32Value = 2 };  // how the rows of a tile are scaled when it is staged

template <int N> struct F32Vec;
template <> struct F32Vec<4> { using type = float4; };
template <> struct F32Vec<2> { using type = float2; };
template <int N>
__device__ __forceinline__ void f32_load(float (&x)[N], const float* p) {
  const typename F32Vec<N>::type v = *reinterpret_cast<const typename F32Vec<N>::type*>(p);
#pragma unroll
  for (int e = 0; e < N; ++e) x[e] = reinterpret_cast<const float*>(&v)[e];
}
template <int N>
__device__ __forceinline__ void f32_store(float* p, const float (&x)[N]) {
  typename F32Vec<N>::type v;
#pragma unroll
  for (int e = 0; e < N; ++e) reinterpret_cast<float*>(&v)[e] = x[e];
  *reinterpret_cast<typename F32Vec<N>::type*>(p) = v;
}
// sum over the 16 threads that share a row (tx = the low four bits of the lane)
__device__ __forceinline__ float f32_row_sum(float x) {
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}
// max(x, lo) that lets a NaN through, as torch.clamp does
__device__ __forceinline__ float f32_clamp_min(float x, float lo) { return x < lo ? lo : x; }

// first position of a chunk; cut from the end, the first chunk of a sequence may begin before it
template <bool REV>
__device__ __forceinline__ int f32_chunk_start(int chunk, int nchunks, int N) {
  return REV ? N - kF32Chunk * (nchunks - chunk) : kF32Chunk * chunk;
}
__device__ __forceinline__ bool f32_inside(int pos, int N) { return static_cast<unsigned>(pos) < static_cast<unsigned>(N); }

// The row factors of a chunk: div[r] = max(n^sigma, 1), n[r] = the running count n_s, take[r] = un-masked.
struct F32Rows {
  float div[kF32Chunk], n[kF32Chunk], take[kF32Chunk];
  int part[kF32Threads / 32];
};
// (Counts the kept positions before the chunk itself: the flags of a sequence are few bytes, and a launch less.)
__device__ __forceinline__ void f32_rows(F32Rows& rows, const unsigned char* keep_b, int c0, int N, float sigma) {
  const int tid = threadIdx.x;
  int before = c0;
  if (keep_b) {
    int cnt = 0;
    for (int s = tid; s < c0; s += kF32Threads) cnt += keep_b[s] ? 1 : 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
    if ((tid & 31) == 0) rows.part[tid >> 5] = cnt;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int w = 0; w < kF32Threads / 32; ++w) before += rows.part[w];
  }
  if (tid < kF32Chunk) {
    int n = max(before + tid + 1, 0);
    float take = f32_inside(c0 + tid, N) ? 1.f : 0.f;
    if (keep_b) {
      // inclusive count inside the chunk: the flags before this thread's 32-row half, then the ballot of its own half
      const bool kp = f32_inside(c0 + tid, N) && keep_b[c0 + tid];
      const unsigned mine = __ballot_sync(0xffffffffu, kp);
      n = before + __popc(mine & (0xffffffffu >> (31 - (tid & 31))));
      if (tid >= 32)
        for (int s = 0; s < 32; ++s) n += (f32_inside(c0 + s, N) && keep_b[c0 + s]) ? 1 : 0;
      take = kp ? 1.f : 0.f;
    }
    rows.n[tid] = static_cast<float>(n);
    rows.div[tid] = f32_clamp_min(powf(static_cast<float>(n), sigma), 1.0f);
    rows.take[tid] = take;
  }
  __syncthreads();
}

// one [64 x D] tile of a tensor -> shared memory (row stride D + 4), its rows scaled by KIND; thread (ty, tx) stages
// columns NB tx .. of rows ty + 16 a
template <int D, int KIND>
__device__ __forceinline__ void f32_stage(float* dst, const float* __restrict__ src, const F32Rows& rows, int c0, int N, int tx, int ty) {
  constexpr int NB = D / 16, LD = D + 4;
  float x[4][NB];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = ty + 16 * a;
#pragma unroll
    for (int e = 0; e < NB; ++e) x[a][e] = 0.f;
    if (f32_inside(c0 + r, N)) f32_load<NB>(x[a], src + static_cast<long>(c0 + r) * D + NB * tx);
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = ty + 16 * a;
    if constexpr (KIND == kF32Norm) {
      float s = 0.f;
#pragma unroll
      for (int e = 0; e < NB; ++e) s = fmaf(x[a][e], x[a][e], s);
      const float d = f32_clamp_min(sqrtf(f32_row_sum(s)), kF32Eps), m = rows.take[r];
#pragma unroll
      for (int e = 0; e < NB; ++e) x[a][e] = (x[a][e] / d) * m;
    } else if constexpr (KIND == kF32Value) {
      const float d = rows.div[r], m = rows.take[r];
#pragma unroll
      for (int e = 0; e < NB; ++e) x[a][e] = (x[a][e] / d) * m;
    }
    f32_store<NB>(dst + r * LD + NB * tx, x[a]);
  }
}

// state[bh][chunk][i][j] = sum over the chunk of y_s[i] z_s[j].  grid = B*H * chunks, block = 256.
template <int D, bool REV>
__global__ void __launch_bounds__(kF32Threads)
f32_state_kernel(const float* __restrict__ y, const float* __restrict__ z, const unsigned char* __restrict__ keep,
                 const float* __restrict__ norm_const, float* __restrict__ state, int H, int N, int nchunks) {
  constexpr int NB = D / 16, LD = D + 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sY = reinterpret_cast<float*>(smem_raw);
  float* sZ = sY + kF32Chunk * LD;
  __shared__ F32Rows rows;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long bh = blockIdx.x / nchunks;
  const int c0 = f32_chunk_start<REV>(static_cast<int>(blockIdx.x % nchunks), nchunks, N), h = static_cast<int>(bh % H);
  pdl_allow_next();
  pdl_wait_prior();
  const float sigma = 1.0f / (1.0f + expf(-norm_const[h]));
  f32_rows(rows, keep ? keep + (bh / H) * N : nullptr, c0, N, sigma);
  f32_stage<D, kF32Norm>(sY, y + bh * N * D, rows, c0, N, tx, ty);
  f32_stage<D, REV ? kF32Raw : kF32Value>(sZ, z + bh * N * D, rows, c0, N, tx, ty);
  __syncthreads();
  float acc[NB][NB] = {};
#pragma unroll 8
  for (int s = 0; s < kF32Chunk; ++s) {
    float a[NB], b[NB];
    f32_load<NB>(a, sY + s * LD + NB * ty);
    f32_load<NB>(b, sZ + s * LD + NB * tx);
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  }
  float* dst = state + static_cast<long>(blockIdx.x) * (D * D);
#pragma unroll
  for (int i = 0; i < NB; ++i) f32_store<NB>(dst + (NB * ty + i) * D + NB * tx, acc[i]);
}

// Exclusive prefix (REV: suffix) over the chunks of a sequence, in place.  grid = (B*H, D*D / 256), block = 256: a
// thread owns one element; eight chunks are loaded at a time so that the chain is additions, not memory round trips.
template <bool REV>
__global__ void __launch_bounds__(kF32Threads) f32_prefix_kernel(float* __restrict__ state, int nchunks, int elems) {
  float* p = state + static_cast<long>(blockIdx.x) * nchunks * elems + blockIdx.y * kF32Threads + threadIdx.x;
  pdl_allow_next();
  pdl_wait_prior();
  float run = 0.f;
  for (int c = 0; c < nchunks; c += 8) {
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = c + u < nchunks ? p[static_cast<long>(REV ? nchunks - 1 - c - u : c + u) * elems] : 0.f;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (c + u < nchunks) p[static_cast<long>(REV ? nchunks - 1 - c - u : c + u) * elems] = run;
      run += x[u];
    }
  }
}

struct F32Args {
  const float *q, *k, *v, *dout;
  const unsigned char* keep;
  const float* norm_const;
  const float *prefix, *suffix;  // [B*H][chunks][D][D]
  float *out, *dq, *dk, *dv;
  double* gpart;                 // [B*H][chunks]: sum_s ln(n_s) (v'_s . dv'_s) of the chunk
  int H, N, nchunks;
};

// The 4 x NB block of a thread: rows ty + 16 a, columns NB tx + e -- or tx + 16 e when M enters transposed, so that
// the rows of M a half-warp reads are consecutive (no bank conflicts).
template <int D, int PASS>
__device__ __forceinline__ void f32_chunk(const F32Args& g, float* sA, float* sB, float* sC, float* sP, F32Rows& rows) {
  constexpr int NB = D / 16, LD = D + 4, LP = kF32Chunk + 4;
  constexpr bool LOWER = PASS == kF32Out || PASS == kF32Dq;  // column <= row survives, else column >= row
  constexpr bool MT = PASS == kF32Dq || PASS == kF32Dk;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long bh = blockIdx.x / g.nchunks;
  const int N = g.N, chunk = static_cast<int>(blockIdx.x % g.nchunks), c0 = f32_chunk_start<!LOWER>(chunk, g.nchunks, N), h = static_cast<int>(bh % g.H);
  const long base = bh * N * D;
  const float sigma = 1.0f / (1.0f + expf(-g.norm_const[h]));
  const bool with_state = LOWER ? chunk > 0 : chunk + 1 < g.nchunks;  // the first (last) chunk has nothing before (after) it

  // the state rows of this thread, fetched now and put over the B tile once the scores have been taken
  float m[NB][NB];
  if (with_state) {
    const float* src = (LOWER ? g.prefix : g.suffix) + static_cast<long>(blockIdx.x) * (D * D);
#pragma unroll
    for (int i = 0; i < NB; ++i) f32_load<NB>(m[i], src + (ty + 16 * i) * D + NB * tx);
  }
  f32_rows(rows, g.keep ? g.keep + (bh / g.H) * N : nullptr, c0, N, sigma);
  if constexpr (PASS == kF32Out) {
    f32_stage<D, kF32Norm>(sA, g.q + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Norm>(sB, g.k + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Value>(sC, g.v + base, rows, c0, N, tx, ty);
  } else if constexpr (PASS == kF32Dq) {
    f32_stage<D, kF32Raw>(sA, g.dout + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Value>(sB, g.v + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Norm>(sC, g.k + base, rows, c0, N, tx, ty);
  } else if constexpr (PASS == kF32Dk) {
    f32_stage<D, kF32Value>(sA, g.v + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Raw>(sB, g.dout + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Norm>(sC, g.q + base, rows, c0, N, tx, ty);
  } else {
    f32_stage<D, kF32Norm>(sA, g.k + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Norm>(sB, g.q + base, rows, c0, N, tx, ty);
    f32_stage<D, kF32Raw>(sC, g.dout + base, rows, c0, N, tx, ty);
  }
  __syncthreads();

  {  // P = mask(A B^T): rows ty + 16 a, columns tx + 16 b
    float p[4][4] = {};
#pragma unroll 4
    for (int i = 0; i < D; i += 4) {
      float a[4][4], b[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) f32_load<4>(a[r], sA + (ty + 16 * r) * LD + i);
#pragma unroll
      for (int r = 0; r < 4; ++r) f32_load<4>(b[r], sB + (tx + 16 * r) * LD + i);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) p[r][c] = fmaf(a[r][e], b[c][e], p[r][c]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int t = ty + 16 * r, s = tx + 16 * c;
        sP[t * LP + s] = (LOWER ? s <= t : s >= t) ? p[r][c] : 0.f;
      }
  }
  __syncthreads();
  if (with_state) {
#pragma unroll
    for (int i = 0; i < NB; ++i) f32_store<NB>(sB + (ty + 16 * i) * LD + NB * tx, m[i]);
  }

  float acc[4][NB] = {};
  {  // acc = P C by blocks of 16 columns.  A row takes the columns on its side of the diagonal and no other: a masked score
     // times an infinity is a NaN, so what a row may not see is not multiplied by zero but left out.  Row ty + 16 r has the
     // blocks before (after) block r whole, block r up to (from) itself.
#pragma unroll
    for (int blk = 0; blk < 4; ++blk) {
#pragma unroll 2
      for (int s = 16 * blk; s < 16 * blk + 16; s += 4) {
        float p[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (LOWER ? r >= blk : r <= blk) f32_load<4>(p[r], sP + (ty + 16 * r) * LP + s);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float b[NB];
          if constexpr (MT) {
#pragma unroll
            for (int j = 0; j < NB; ++j) b[j] = sC[(s + e) * LD + tx + 16 * j];
          } else {
            f32_load<NB>(b, sC + (s + e) * LD + NB * tx);
          }
          const bool own = LOWER ? s + e <= ty + 16 * blk : s + e >= ty + 16 * blk;
#pragma unroll
          for (int r = 0; r < 4; ++r)
            if ((LOWER ? r > blk : r < blk) || (r == blk && own)) {
#pragma unroll
              for (int j = 0; j < NB; ++j) acc[r][j] = fmaf(p[r][e], b[j], acc[r][j]);
            }
        }
      }
    }
  }
  if (with_state) {  // acc += A M (or A M^T)
    __syncthreads();
#pragma unroll 2
    for (int i = 0; i < D; i += 4) {
      float a[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) f32_load<4>(a[r], sA + (ty + 16 * r) * LD + i);
      if constexpr (MT) {
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          float b[4];
          f32_load<4>(b, sB + (tx + 16 * j) * LD + i);
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][j] = fmaf(a[r][e], b[e], acc[r][j]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float b[NB];
          f32_load<NB>(b, sB + (i + e) * LD + NB * tx);
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int j = 0; j < NB; ++j) acc[r][j] = fmaf(a[r][e], b[j], acc[r][j]);
        }
      }
    }
  }

  // ---- epilogue: rows ty + 16 r
  if constexpr (PASS == kF32Out) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (f32_inside(c0 + ty + 16 * r, N)) f32_store<NB>(g.out + base + static_cast<long>(c0 + ty + 16 * r) * D + NB * tx, acc[r]);
  } else if constexpr (MT) {
    // through the normalisation: dx = (g - x^ (x^ . g)) / max(|x|, eps) with g the masked row and x^ = x / max(|x|, eps);
    // a row shorter than eps is divided by eps alone (its norm was clamped: no gradient through it)
    const float* x_all = (PASS == kF32Dq ? g.q : g.k) + base;
    float* dx_all = (PASS == kF32Dq ? g.dq : g.dk) + base;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = ty + 16 * r;
      const bool in = f32_inside(c0 + t, N);
      const long o = static_cast<long>(c0 + t) * D + tx;
      float x[NB], s = 0.f;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        x[j] = in ? x_all[o + 16 * j] : 0.f;
        s = fmaf(x[j], x[j], s);
      }
      const float norm = sqrtf(f32_row_sum(s)), d = f32_clamp_min(norm, kF32Eps), take = rows.take[t];
      float dot = 0.f;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        x[j] /= d;
        acc[r][j] *= take;
        dot = fmaf(x[j], acc[r][j], dot);
      }
      dot = f32_row_sum(dot);
      if (norm < kF32Eps) dot = 0.f;
      if (in) {
#pragma unroll
        for (int j = 0; j < NB; ++j) dx_all[o + 16 * j] = (acc[r][j] - x[j] * dot) / d;
      }
    }
  } else {
    // dv = dv' / div;  the gradient of norm_const collects ln(n) (v' . dv').  A sum of terms of both signs: its rows are
    // added up in fp64.
    double gsum = 0.0;
    double* ln = reinterpret_cast<double*>(sP);  // (the scores have been read)
    __syncthreads();
    if (tid < kF32Chunk) ln[tid] = rows.n[tid] > 1.f ? log(static_cast<double>(rows.n[tid])) : 0.0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = ty + 16 * r;
      const bool in = f32_inside(c0 + t, N);
      const long o = base + static_cast<long>(c0 + t) * D + NB * tx;
      const float d = rows.div[t], n = rows.n[t], take = rows.take[t];
      float v[NB] = {};
      double dot = 0.0;
      if (in) f32_load<NB>(v, g.v + o);
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        acc[r][j] *= take;
        dot = fma(static_cast<double>(v[j] / d), static_cast<double>(acc[r][j]), dot);
        acc[r][j] /= d;
      }
      if (in && n >= 1.f) gsum += ln[t] * dot;  // (ln 1 = 0 times an infinity is a NaN, here as in the module math)
      if (in) f32_store<NB>(g.dv + o, acc[r]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) gsum += __shfl_xor_sync(0xffffffffu, gsum, off);
    double* part = ln + kF32Chunk;
    if ((tid & 31) == 0) part[tid >> 5] = gsum;
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
      for (int w = 0; w < kF32Threads / 32; ++w) s += part[w];
      g.gpart[blockIdx.x] = s;
    }
  }
}

// Three CTAs of 70 KB per SM (D = 64): they cover each other's staging.
// FWD: grid = B*H * chunks.  Backward: grid = (B*H * chunks, 3), y = dq, dk, dv.
template <int D, bool FWD>
__global__ void __launch_bounds__(kF32Threads, 3) f32_chunk_kernel(const F32Args g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sA = reinterpret_cast<float*>(smem_raw);
  float* sB = sA + kF32Chunk * (D + 4);
  float* sC = sB + kF32Chunk * (D + 4);
  float* sP = sC + kF32Chunk * (D + 4);
  __shared__ F32Rows rows;
  pdl_allow_next();
  pdl_wait_prior();
  if constexpr (FWD) {
    f32_chunk<D, kF32Out>(g, sA, sB, sC, sP, rows);
  } else {
    if (blockIdx.y == 0)
      f32_chunk<D, kF32Dq>(g, sA, sB, sC, sP, rows);
    else if (blockIdx.y == 1)
      f32_chunk<D, kF32Dk>(g, sA, sB, sC, sP, rows);
    else
      f32_chunk<D, kF32Dv>(g, sA, sB, sC, sP, rows);
  }
}

// dnorm[h] = -sigma (1 - sigma) sum over the batch and the chunks of gpart, in a fixed order.  grid = H, block = 256.
__global__ void __launch_bounds__(kF32Threads)
f32_dnorm_kernel(const double* __restrict__ gpart, const float* __restrict__ norm_const, float* __restrict__ dnorm, int B, int H, int nchunks) {
  const int h = blockIdx.x;
  __shared__ double part[kF32Threads / 32];
  pdl_allow_next();
  pdl_wait_prior();
  double s = 0.0;
  for (int i = threadIdx.x; i < B * nchunks; i += kF32Threads) s += gpart[(static_cast<long>(i / nchunks) * H + h) * nchunks + i % nchunks];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kF32Threads / 32; ++w) t += part[w];
    const double sigma = 1.0 / (1.0 + exp(-static_cast<double>(norm_const[h])));
    dnorm[h] = static_cast<float>(-sigma * (1.0 - sigma) * t);
  }
}

}  // namespace cott
