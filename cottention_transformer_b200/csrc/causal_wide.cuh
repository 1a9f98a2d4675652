// Causal scan with head dim 128 on the 5th-generation tensor cores (tcgen05 + TMEM + TMA): the kernel behind
// cott_scan and the fused cosine attention for D_attn = 128.
//
// The reference runs kernel_mod_4<T, 32> for D_attn >= 128 (Cuda_Kernel/combined_kernel_general.cu:173-251, selected at
// :281-284): one warp per output column, four state elements per lane, N serial steps.  Here a CTA owns one
// (batch, head) sequence and one W-column slice of the value / output dimension, walks the sequence in chunks of
// 128 positions, and the whole head dimension of Q and K goes into the SAME score and state accumulators:
//   P   = mask(X Y^T)            128 x 128, contraction over 128 = two 64-column panels, 8 k-steps   (tcgen05, TMEM)
//   Acc = P Zs + X S             128 x W                                                             (A = P from TMEM)
//   S  += Y^T Zs                 128 x W with M = 128: the natural tcgen05 shape, every TMEM lane holds a state row
// X, Y are [128 x 128] tiles (two swizzled 64-column panels each), Zs the [128 x W] slice of Z with its rows scaled.
// Nothing goes through a scratch buffer and the products are rounded to 16 bits once.
//
// W = 128 wherever the value dimension is a multiple of 128, else 64.  A chunk is a chain of hand-offs (load -> row pass
// -> scores -> mask -> products -> output rows) of 3-4.5 us whatever W is, so the width sets the rate: with W = 64 two
// CTAs computed the same scores and re-read the same X and Y.  Measured at B 1, H 16, N 16384 (bf16): a pass 104 -> 65-75 us,
// a state-only pass 45 -> 31 us, forward + backward 563 -> 392 us (a row-dot pass, two transposes and the eps pass went too).
//
// The module math around the scan (GPT_Trainer/GPTCosAttention.py:229-248 and its backward) is row scalings, which
// enter through hooks rather than through extra passes over the tensors (the hooks that use a whole row need W = 128 =
// the head dim):
//   NORMS   (forward): 1/|x_t|, 1/|y_s| from the tiles themselves, Zs = diag(keep a_s / |y_s|) Z, out rows / |x_t|;
//           the three row vectors are also written out for the backward
//   yscale, zscale, oscale: per-position fp32 vectors that scale the rows of Y (in shared memory), of Z (likewise)
//           and of the output
//   C: a fourth tensor whose rows enter the output rows, o = oscale:
//           kWdRowAdd   out = o acc + ccoef[pos] C                       (dk: ccoef = -eps / |k|^2)
//           kWdRowNorm  out = o acc - o^3 (C . acc) C                    (dq through the normalisation of q)
//           kWdRowEps   out = o acc, and with eps = o (C . acc) = v' . dv': ck_out = -rk^2 eps and the gradient of
//                       norm_const, -sigma (1 - sigma) sum ln(n) eps     (dv)
// REV walks the sequence backwards with the mask flipped (the reversed scans of Custom_Kernel.py:107-108).
// STATE_ONLY keeps only the state chain and writes the segment's own S to global memory (segment-parallel launches).
//
// Shared memory (all dynamic, W = 128): two stages of (X 32 KB, Y 32 KB, Z 32 KB) and the 16-bit state operand 32 KB =
// 224 KB, then the barriers.  Output rows are staged over the X tile, whose readers are done when the accumulator is
// complete; Y and Z of a stage are refilled at that moment (they have a barrier of their own, so the row pass of the next
// use runs while X is still being stored and reloaded), X once its store has read it.
// TMEM: P 2 x 128 | Acc W | S W.
#pragma once

#include "causal_tc.cuh"

namespace cott {

constexpr int kWdThreads = 768;  // 3 issuing warps, 1 TMA warp, 5 groups of 4 warps
constexpr int kWdStages = 2;
template <int W, bool STATE_ONLY> struct WdCfg {
  static constexpr int kPanels = W / 64;                                        // 64-column panels of Z, S and the output
  static constexpr int kStages = STATE_ONLY ? 3 : kWdStages;                    // (the state chain has no X tile)
  static constexpr int kStageBytes = ((STATE_ONLY ? 2 : 4) + kPanels) * kTileBytes;
  static constexpr int kStateBytes = STATE_ONLY ? 0 : kPanels * kTileBytes;     // the 16-bit [128 x W] state operand
  static constexpr size_t kSmemBytes = kStages * kStageBytes + kStateBytes + 2 * 2 * kTcChunk * sizeof(float) + 40 * sizeof(uint64_t);
};
enum { kWdRowPlain = 0, kWdRowAdd = 1, kWdRowNorm = 2, kWdRowEps = 3 };

struct WideArgs {
  const float* yscale;  // [B*H*N] or null
  const float* zscale;
  const float* oscale;
  const float* ccoef;       // kWdRowAdd
  const float* norm_const;  // NORMS and kWdRowEps: [H]
  float* rq_out;        // NORMS only (may be null): 1/|x_t|, 1/|y_s|, keep a_s/|y_s|
  float* rk_out;
  float* w_out;
  const float* rk;      // kWdRowEps: 1/|k|
  float* ck_out;        // kWdRowEps
  float* dnorm;         // kWdRowEps: [H], accumulated by atomics (zero it first)
  const float* init_state;  // [B*H][slices][nseg][128 x W] fp32, the state before each segment in scan order, or null
  int init_transposed;      // W = 128: the matrices of init_state are the transposes of this pass's states
  float* state_out;         // STATE_ONLY: [B*H][slices][nseg][128 x W]
  float* decode_state;      // NORMS: the state after the whole sequence, [B*H][128][128] with the value index first, or null
  const unsigned char* keep;  // NORMS only: padding ([B, N]) or null; with it `count`, its inclusive running count (also kWdRowEps)
  const int* count;
  const void* c;        // the C tensor [B,H,N,dz] (dense), or null
  int row_mode;
  int dz;               // row length of Z / C / out in elements
  int chunks_per_seg;
  int H, N;
};

// a 128-column row of a two-panel tile.  (Rolled two-piece routines on purpose: versions with eight pieces in flight
// are faster in isolation and slowed the whole kernel down -- every role runs on every scheduler and competes for
// one instruction cache.)
template <typename T>
__device__ __forceinline__ float row_sumsq2(unsigned char* tile, int row) {
  return row_sumsq_rolled<T>(tile, row) + row_sumsq_rolled<T>(tile + kTileBytes, row);
}

template <typename T, int W, bool REV, bool NORMS, bool STATE_ONLY>
__global__ void __launch_bounds__(kWdThreads, 1)
wide_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapY,
            const __grid_constant__ CUtensorMap mapZ, const __grid_constant__ CUtensorMap mapOut, const WideArgs a) {
  using namespace ptx;
  using Cfg = WdCfg<W, STATE_ONLY>;
  constexpr int NS = Cfg::kStages, NP = Cfg::kPanels;
  constexpr bool BF = Pack2<T>::kBf16;
  static_assert(!NORMS || W == 128, "the row norm of x is shared by the two output groups: head dim = W = 128");

  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* sS = smem + NS * Cfg::kStageBytes;  // [128 x W] 16-bit state operand (rows = columns of Y)
  float* s_x = reinterpret_cast<float*>(sS + Cfg::kStateBytes);  // [2 chunk parities][2 panels][128]: half-row sums the output groups exchange
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_x + 2 * 2 * kTcChunk);
  uint64_t *bar_full_x = bars, *bar_full = bars + 3, *bar_free_in = bars + 6, *bar_out = bars + 9, *bar_prep = bars + 12,
           *bar_p_full = bars + 15, *bar_p_ready = bars + 17, *bar_acc_full = bars + 19;
  uint64_t &bar_acc_free = bars[21], &bar_xs = bars[22], &bar_state = bars[23], &bar_s_full = bars[24], &bar_state2 = bars[25],
           &bar_init = bars[26];
  uint64_t* bar_pair = bars + 28;  // [4]: the two output warps that share rows 32 wq .. exchange their half-row sums
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 27);
  int& abort_flag_s = *(reinterpret_cast<int*>(bars + 27) + 1);
  volatile int* abort_flag = &abort_flag_s;

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int bh = blockIdx.x, slice = blockIdx.y, seg = blockIdx.z;
  const int h = bh % a.H, bb = bh / a.H;
  const int N = a.N;
  const int total_chunks = (N + kTcChunk - 1) / kTcChunk;
  const int chunk0 = seg * a.chunks_per_seg;
  const int nchunks = min(a.chunks_per_seg, total_chunks - chunk0);
  const bool has_init = !STATE_ONLY && a.init_state != nullptr && seg > 0;
  // state updates of this CTA: the one after its last chunk is only needed by STATE_ONLY and as the decode state
  const bool final_state = NORMS && !STATE_ONLY && a.decode_state != nullptr && seg + 1 == static_cast<int>(gridDim.z);
  const int nstates = STATE_ONLY || final_state ? nchunks : nchunks - 1;
  const size_t state_index = (static_cast<size_t>(bh) * gridDim.y + slice) * gridDim.z + seg;
  const size_t row_base = static_cast<size_t>(bh) * N;  // the per-position vectors are [B*H, N]
  const unsigned char* keep_b = (NORMS && a.keep) ? a.keep + static_cast<size_t>(bb) * N : nullptr;
  const int* count_b = a.count ? a.count + static_cast<size_t>(bb) * N : nullptr;
  // first row of local chunk c (the reversed scan numbers chunks and segments from the end of the sequence)
  auto row0_of = [&](int c) { return (REV ? total_chunks - 1 - (chunk0 + c) : chunk0 + c) * kTcChunk; };
  // tiles of a stage: Y (2 panels), Z (NP panels), X (2 panels, the first NP of which receive the output rows)
  auto st_y = [&](int c) { return smem + (c % NS) * Cfg::kStageBytes; };
  auto st_z = [&](int c) { return st_y(c) + 2 * kTileBytes; };
  auto st_x = [&](int c) { return st_z(c) + NP * kTileBytes; };

  if (smem_u32(smem) & 1023u) {  // the swizzle atoms need the 1024-byte alignment the declaration asks for
    if (tid == 0) atomicCAS(&g_cott_status, 0, (15 << 16));
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < 3; ++s) {
      mbar_init(&bar_full_x[s], 1);
      mbar_init(&bar_full[s], 1);
      // state group (STATE_ONLY: the MMA commit itself): state MMAs done; the TMA thread waits for the accumulator MMAs
      mbar_init(&bar_free_in[s], STATE_ONLY ? 1 : 4);
      mbar_init(&bar_out[s], 4 * NP);
      mbar_init(&bar_prep[s], 4);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bar_p_full[b], 1);
      mbar_init(&bar_p_ready[b], 4);
      mbar_init(&bar_acc_full[b], 1);
    }
    mbar_init(&bar_acc_free, 4 * NP);
    mbar_init(&bar_xs, 1);
    mbar_init(&bar_state, 4);
    mbar_init(&bar_s_full, 1);
    mbar_init(&bar_state2, 4);
    mbar_init(&bar_init, 4);
    for (int w = 0; w < 4; ++w) mbar_init(&bar_pair[w], 2);
    mbar_fence_init();
    abort_flag_s = 0;
    tma_prefetch_desc(&mapX);
    tma_prefetch_desc(&mapY);
    tma_prefetch_desc(&mapZ);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t tP0 = tmem, tAcc = tmem + 256, tS = tmem + 384;  // P 2 x 128 | Acc W | S W

  // Roles:
  //   warp 0, one thread:  scores P(c+1) = X Y^T
  //   warp 1, one thread:  accumulators Acc(c) = X S + P Zs
  //   warp 19, one thread: state S += Y^T Zs (c)
  //   warps 2-5:        mask group: mask + convert P in TMEM
  //   warps 6-9, 20-23: output groups (panel 0 / panel 1 of the slice): accumulator -> output rows
  //   warps 10-13:      state group: fp32 state -> 16-bit operand
  //   warp 14, one thread: TMA loads and stores
  //   warps 15-18:      operand group: row norms / row scalings of Y and Z in place
  constexpr uint32_t kIdescP = make_idesc(128, 128, BF, false, false);
  constexpr uint32_t kIdescAcc = make_idesc(128, W, BF, false, true);
  constexpr uint32_t kIdescS = make_idesc(128, W, BF, true, true);
  constexpr uint64_t kPanel = kTileBytes >> 4;
  // an MN-major operand of one or two 64-column panels, kTileBytes apart
  auto pdesc = [](unsigned char* p) { return make_smem_desc(smem_u32(p), kTileBytes, 1024); };
  if (warp == 14) {
    // ---------------------------------------------------------------- TMA loads and stores
    if (elect_one()) {
      const int xz = W * slice;  // column offset of the Z / C / output slice
      auto load_yz = [&](int c) {
        const int s = c % NS, y = row0_of(c);
        mbar_expect_tx(&bar_full[s], (2 + NP) * kTileBytes);
        tma_load_tile_x(st_y(c), &mapY, &bar_full[s], 0, y, h, bb);
        tma_load_tile_x(st_y(c) + kTileBytes, &mapY, &bar_full[s], 64, y, h, bb);
        for (int p = 0; p < NP; ++p) tma_load_tile_x(st_z(c) + p * kTileBytes, &mapZ, &bar_full[s], xz + 64 * p, y, h, bb);
      };
      auto load_x = [&](int c) {
        const int s = c % NS, y = row0_of(c);
        mbar_expect_tx(&bar_full_x[s], 2 * kTileBytes);
        tma_load_tile_x(st_x(c), &mapX, &bar_full_x[s], 0, y, h, bb);
        tma_load_tile_x(st_x(c) + kTileBytes, &mapX, &bar_full_x[s], 64, y, h, bb);
      };
      auto prefetch = [&](int c) {  // pull a chunk further ahead into L2: with two stages a refill should be an L2 hit
        if (c >= nchunks) return;
        const int y = row0_of(c);
        if (!STATE_ONLY) {
          tma_prefetch_tile_x(&mapX, 0, y, h, bb);
          tma_prefetch_tile_x(&mapX, 64, y, h, bb);
        }
        tma_prefetch_tile_x(&mapY, 0, y, h, bb);
        tma_prefetch_tile_x(&mapY, 64, y, h, bb);
        for (int p = 0; p < NP; ++p) tma_prefetch_tile_x(&mapZ, xz + 64 * p, y, h, bb);
      };
      for (int c = 0; c < NS && c < nchunks; ++c) {
        load_yz(c);
        if (!STATE_ONLY) load_x(c);
      }
      prefetch(NS);
      for (int c = 0; c < nchunks; ++c) {
        const int s = c % NS;
        const bool refill = c + NS < nchunks;
        if (refill) {
          // every MMA of chunk c has completed: Y and Z have no reader left
          if (!STATE_ONLY && !wait_bar(&bar_acc_full[c & 1], (c >> 1) & 1, abort_flag, kWaitAcc, c)) break;
          if (!wait_bar(&bar_free_in[s], (c / NS) & 1, abort_flag, kWaitStageFree, c)) break;
          load_yz(c + NS);
          prefetch(c + NS + 1);
        }
        if (STATE_ONLY) continue;
        if (!wait_bar(&bar_out[s], (c / NS) & 1, abort_flag, kWaitStageFree, c)) break;
        for (int p = 0; p < NP; ++p) tma_store_tile_x(&mapOut, st_x(c) + p * kTileBytes, xz + 64 * p, row0_of(c), h, bb);
        tma_store_commit();
        if (refill) {
          tma_store_wait_read<0>();
          load_x(c + NS);
        }
      }
      tma_store_wait<0>();
    }
  } else if (warp == 0) {
    // ---------------------------------------------------------------- scores
    if (!STATE_ONLY && elect_one()) {
      auto issue_scores = [&](int c) {  // caller has waited for the prepared tiles of chunk c and for the buffer
        const uint64_t dX = kdesc(smem_u32(st_x(c))), dY = kdesc(smem_u32(st_y(c)));
        const uint32_t tP = tP0 + 128 * (c & 1);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          mma_ss(tP, dX + (k >> 2) * kPanel + 2 * (k & 3), dY + (k >> 2) * kPanel + 2 * (k & 3), kIdescP, k > 0);
        mma_commit(&bar_p_full[c & 1]);
      };
      // The scores read X and Y only: they can go as soon as the TMA has landed, without waiting for the row pass
      // of the operand group -- unless that pass rewrites Y (yscale).
      uint64_t* gate = a.yscale ? bar_prep : bar_full;
      bool ok = wait_bar2(&gate[0], 0, &bar_full_x[0], 0, abort_flag, kWaitPrepped, 0);
      if (ok) {
        tc_fence_after_sync();
        issue_scores(0);
      }
      for (int c = 0; ok && c + 1 < nchunks; ++c) {
        // scores of chunk c+1: its tiles, and (buffer reuse) the accumulator MMAs of chunk c-1 done
        const int s1 = (c + 1) % NS;
        ok = wait_bar4(&gate[s1], ((c + 1) / NS) & 1, &bar_full_x[s1], ((c + 1) / NS) & 1, c >= 1 ? &bar_acc_full[(c + 1) & 1] : nullptr,
                       ((c - 1) >> 1) & 1, nullptr, 0, abort_flag, kWaitTma, c);
        if (!ok) break;
        tc_fence_after_sync();
        issue_scores(c + 1);
      }
    }
  } else if (warp == 19) {
    // ---------------------------------------------------------------- state
    if (elect_one()) {
      for (int c = 0; c < nstates; ++c) {
        // state update of chunk c: its prepared tiles, and the conversion of S after chunk c-1 (it reads the fp32 state)
        if (!wait_bar4(&bar_prep[c % NS], (c / NS) & 1, (!STATE_ONLY && c > 0) ? &bar_state2 : (has_init ? &bar_init : nullptr),
                       c > 0 ? ((c - 1) & 1) : 0, nullptr, 0, nullptr, 0, abort_flag, kWaitPrepped, c))
          break;
        tc_fence_after_sync();
        // A = Y^T: MN-major, M = 128 = the two panels of Y, K = the 128 positions
        const uint64_t dYm = pdesc(st_y(c)), dZm = pdesc(st_z(c));
        mma_ss(tS, dYm, dZm, kIdescS, (c > 0 || has_init) ? 1u : 0u);
#pragma unroll
        for (int k = 1; k < 8; ++k) mma_ss(tS, dYm + 128 * k, dZm + 128 * k, kIdescS, 1u);
        if (STATE_ONLY) mma_commit(&bar_free_in[c % NS]);
        if (!STATE_ONLY || c + 1 == nstates) mma_commit(&bar_s_full);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- accumulators
    if (!STATE_ONLY && elect_one()) {
      const uint64_t dS = pdesc(sS);
      for (int c = 0; c < nchunks; ++c) {
        const int s = c % NS, b = c & 1;
        const uint64_t dX = kdesc(smem_u32(st_x(c))), dZm = pdesc(st_z(c));
        const uint32_t tP = tP0 + 128 * b;
        const bool with_s = c > 0 || has_init;
        // the state term: the 16-bit state after chunk c-1 and the accumulator read out
        if (!wait_bar4(&bar_full_x[s], (c / NS) & 1, c > 0 ? &bar_state : (has_init ? &bar_init : nullptr), c > 0 ? ((c - 1) & 1) : 0,
                       c > 0 ? &bar_acc_free : nullptr, (c - 1) & 1, nullptr, 0, abort_flag, kWaitState, c))
          break;
        tc_fence_after_sync();
        if (with_s) {
          // Acc = X S: A = X K-major over both panels, B = the 16-bit state [K = 128 rows, N = W], MN-major
#pragma unroll
          for (int k = 0; k < 8; ++k) mma_ss(tAcc, dX + (k >> 2) * kPanel + 2 * (k & 3), dS + 128 * k, kIdescAcc, k > 0);
        }
        mma_commit(&bar_xs);  // the 16-bit state has been read: it may be rewritten
        // masked scores of chunk c, the prepared Z
        if (!wait_bar2(&bar_p_ready[b], (c >> 1) & 1, &bar_prep[s], (c / NS) & 1, abort_flag, kWaitScoreReady, c)) break;
        tc_fence_after_sync();
        mma_ts(tAcc, tP, dZm, kIdescAcc, with_s ? 1u : 0u);  // Acc += P Zs   (P from TMEM, Zs MN-major)
#pragma unroll
        for (int k = 1; k < 8; ++k) mma_ts(tAcc, tP + 8 * k, dZm + 128 * k, kIdescAcc, 1u);
        mma_commit(&bar_acc_full[b]);
      }
    }
  } else if (warp < 6) {
    // ---------------------------------------------------------------- mask group
    if (!STATE_ONLY) {
      const int wq = warp & 3;
      const uint32_t lane_base = static_cast<uint32_t>(32 * wq) << 16;
      for (int c = 0; c < nchunks; ++c) {
        const int b = c & 1;
        if (!wait_bar_warp(&bar_p_full[b], (c >> 1) & 1, abort_flag, kWaitScore, c)) break;
        tc_fence_after_sync();
        mask_pack_inplace<T, !REV>(tP0 + 128 * b + lane_base, lane, wq);
        tc_fence_before_sync();
        warp_arrive(&bar_p_ready[b], lane);
      }
    }
  } else if (warp >= 10 && warp < 14) {
    // ---------------------------------------------------------------- state group (thread = state row = TMEM lane)
    const int wq = warp & 3, row = 32 * wq + lane;
    const uint32_t lane_base = static_cast<uint32_t>(32 * wq) << 16;
    // 32 fp32 columns 32 blk .. of this thread's row -> the 16-bit operand
    auto to_operand = [&](const uint32_t* r, int blk) {
      unsigned char* dst = sS + (blk >> 1) * kTileBytes;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *tile_piece(dst, row, 4 * (blk & 1) + j) =
            make_uint4(Pack2<T>::pack(__uint_as_float(r[8 * j]), __uint_as_float(r[8 * j + 1])),
                       Pack2<T>::pack(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3])),
                       Pack2<T>::pack(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5])),
                       Pack2<T>::pack(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7])));
    };
    if (has_init) {
      // the state before this segment: fp32 into TMEM, 16-bit into the operand buffer.  (Transposed: this thread's row
      // is a column of the stored matrix, and consecutive threads read consecutive elements.)
      const float* src = a.init_state + state_index * (kTcChunk * W);
#pragma unroll 1
      for (int blk = 0; blk < 2 * NP; ++blk) {
        uint32_t r[32];
        if (a.init_transposed) {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(src[(32 * blk + j) * W + row]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 f = *reinterpret_cast<const float4*>(src + row * W + 32 * blk + 4 * j);
            r[4 * j] = __float_as_uint(f.x), r[4 * j + 1] = __float_as_uint(f.y);
            r[4 * j + 2] = __float_as_uint(f.z), r[4 * j + 3] = __float_as_uint(f.w);
          }
        }
        tmem_st_x32(tS + lane_base + 32 * blk, r);
        to_operand(r, blk);
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      warp_arrive(&bar_init, lane);
    }
    if (STATE_ONLY) {
      // after the last state MMA the segment's own state goes to global memory
      if (wait_bar_warp(&bar_s_full, 0, abort_flag, kWaitState, 0)) {
        tc_fence_after_sync();
        float* dst = a.state_out + state_index * (kTcChunk * W) + row * W;
#pragma unroll 1
        for (int blk = 0; blk < 4 * NP; ++blk) {
          uint32_t r[16];
          tmem_ld_x16(tS + lane_base + 16 * blk, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(dst + 16 * blk + 4 * j) =
                make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                            __uint_as_float(r[4 * j + 3]));
        }
      }
    } else {
      for (int c = 0; c < nstates; ++c) {
        // S after chunk c -> 16-bit operand for chunk c+1, once the state term of chunk c has read the operand
        if (!wait_bar_warp(&bar_s_full, c & 1, abort_flag, kWaitState, c)) break;
        if (NORMS && c + 1 == nchunks) {  // the last one: to the decode state [value][key], row = key index
          tc_fence_after_sync();
          float* dst = a.decode_state + static_cast<size_t>(bh) * (128 * 128) + row;
#pragma unroll 1
          for (int blk = 0; blk < 8; ++blk) {
            uint32_t r[16];
            tmem_ld_x16(tS + lane_base + 16 * blk, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) dst[(16 * blk + j) * 128] = __uint_as_float(r[j]);
          }
          break;
        }
        if (lane == 0) mbar_arrive(&bar_free_in[c % NS]);  // the state MMAs of chunk c have read its tiles
        if (!wait_bar_warp(&bar_xs, c & 1, abort_flag, kWaitAccFree, c)) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int blk = 0; blk < 2 * NP; ++blk) {
          uint32_t r[32];
          tmem_ld_x32(tS + lane_base + 32 * blk, r);
          tmem_ld_wait();
          to_operand(r, blk);
        }
        tc_fence_before_sync();
        fence_proxy_async_smem();
        warp_arrive(&bar_state2, lane);  // the fp32 state has been read: the next state MMAs may run
        if (lane == 0) mbar_arrive(&bar_state);
      }
    }
  } else if (warp >= 15 && warp < 19) {
    // ---------------------------------------------------------------- operand group: rows of Y and Z in place
    const int row = 32 * (warp & 3) + lane;
    const float sigma = NORMS ? 1.0f / (1.0f + __expf(-a.norm_const[h])) : 0.f;
    for (int c = 0; c < nchunks; ++c) {
      const int s = c % NS;
      const int pos = row0_of(c) + row;
      float ys = 1.f, zs = 1.f;
      if constexpr (!NORMS) {  // (read before the wait: they travel with the tiles)
        if (a.yscale) ys = pos < N ? a.yscale[row_base + pos] : 0.f;
        if (a.zscale) zs = pos < N ? a.zscale[row_base + pos] : 0.f;
      }
      if (!wait_bar_warp(&bar_full[s], (c / NS) & 1, abort_flag, kWaitTma, c)) break;
      if constexpr (NORMS) {
        const RowMask m = row_mask(keep_b, count_b, pos, N);
        const float rk = m.kp ? inv_norm(row_sumsq2<T>(st_y(c), row)) : 0.f;
        const float w = rk * length_factor(m.n, sigma);
        for (int p = 0; p < NP; ++p) scale_row_rolled<T>(st_z(c) + p * kTileBytes, row, w);
        if (!STATE_ONLY && slice == 0 && pos < N && a.rk_out) {
          a.rk_out[row_base + pos] = rk;
          a.w_out[row_base + pos] = w;
        }
      } else {
        if (a.yscale) {
          scale_row_rolled<T>(st_y(c), row, ys);
          scale_row_rolled<T>(st_y(c) + kTileBytes, row, ys);
        }
        if (a.zscale)
          for (int p = 0; p < NP; ++p) scale_row_rolled<T>(st_z(c) + p * kTileBytes, row, zs);
      }
      fence_proxy_async_smem();
      warp_arrive(&bar_prep[s], lane);
    }
  } else if ((warp >= 6 && warp < 10) || warp >= 20) {
    // ---------------------------------------------------------------- output groups (panel 0, panel 1)
    const int panel = warp >= 20 ? 1 : 0;
    if (!STATE_ONLY && panel < NP) {
      const int wq = warp & 3, row = 32 * wq + lane;
      const uint32_t lane_base = static_cast<uint32_t>(32 * wq) << 16;
      const bool has_c = a.c != nullptr;
      // sum of this thread's half-row value and its partner's (the warp of the other panel that owns the same rows).
      // Two buffers by chunk parity: a buffer is written again two chunks later, past the pair's next barrier.
      // (One exchange per chunk, so the barrier's phase is the chunk's parity.)
      auto pair_sum = [&](float& x, int c) -> bool {
        if constexpr (NP == 2) {
          float* buf = s_x + (c & 1) * 2 * kTcChunk;
          buf[panel * kTcChunk + row] = x;
          warp_arrive(&bar_pair[wq], lane);
          if (!wait_bar_warp(&bar_pair[wq], c & 1, abort_flag, kWaitPrepped, c)) return false;
          x += buf[(panel ^ 1) * kTcChunk + row];
        }
        return true;
      };
      const float sigma = a.row_mode == kWdRowEps ? 1.0f / (1.0f + __expf(-a.norm_const[h])) : 0.f;
      float gsum = 0.f;  // sum of ln(n_s) eps_s over this thread's rows
      for (int c = 0; c < nchunks; ++c) {
        const int s = c % NS, b = c & 1;
        const int pos = row0_of(c) + row;
        unsigned char* dst = st_x(c) + panel * kTileBytes;
        float beta = 1.f, alpha = 0.f, rk = 0.f;
        if constexpr (NORMS) {
          // the row norm of x only needs the TMA data: taken while the MMAs run
          if (!wait_bar_warp(&bar_full_x[s], (c / NS) & 1, abort_flag, kWaitTma, c)) break;
          float ss = row_sumsq_rolled<T>(dst, row);
          if (!pair_sum(ss, c)) break;
          beta = row_mask(keep_b, count_b, pos, N).kp ? inv_norm(ss) : 0.f;
          if (panel == 0 && pos < N && a.rq_out) a.rq_out[row_base + pos] = beta;
        } else {
          if (a.oscale) beta = pos < N ? a.oscale[row_base + pos] : 0.f;
          if (a.row_mode == kWdRowAdd) alpha = pos < N ? a.ccoef[row_base + pos] : 0.f;
          if (a.row_mode == kWdRowEps) rk = pos < N ? a.rk[row_base + pos] : 0.f;
        }
        // the warp's C rows, straight from global memory and issued now, so that the loads have the wait below to land:
        // lane l takes piece l % 8 of rows 4 j + l / 8 (four whole 128-byte rows per instruction)
        uint4 u[8];
        if (has_c) {
          const int r0 = row0_of(c) + 32 * wq + (lane >> 3);
          const T* src = static_cast<const T*>(a.c) + 64 * (NP * slice + panel) + 8 * (lane & 7);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            u[j] = r0 + 4 * j < N ? *reinterpret_cast<const uint4*>(src + (row_base + r0 + 4 * j) * a.dz) : make_uint4(0, 0, 0, 0);
        }
        if (!wait_bar_warp(&bar_acc_full[b], (c >> 1) & 1, abort_flag, kWaitAcc, c)) break;
        tc_fence_after_sync();
        const uint32_t t = tAcc + 64 * panel + lane_base;
        if (has_c) {  // the X tile has no reader left: the C rows go there, and are replaced by the output rows
#pragma unroll
          for (int j = 0; j < 8; ++j) *tile_piece(dst, 32 * wq + 4 * j + (lane >> 3), lane & 7) = u[j];
          __syncwarp();
          if (a.row_mode == kWdRowEps) {
            float eps = beta * row_from_acc_dot<T>(dst, row, t, beta);
            if (!pair_sum(eps, c)) break;
            if (panel == 0 && pos < N) {
              a.ck_out[row_base + pos] = -rk * rk * eps;
              const float n = count_b ? fmaxf(static_cast<float>(count_b[pos]), 1.f) : static_cast<float>(pos + 1);
              if (n > 1.f) gsum += logf(n) * eps;
            }
          } else {
            if (a.row_mode == kWdRowNorm) {
              float dot = row_dot_acc<T>(dst, row, t);
              if (!pair_sum(dot, c)) break;
              alpha = -beta * beta * (beta * dot);  // (x^ . g first: the cube of 1/|x| underflows from |x| = 5e12 on)
            }
            row_from_acc<T, true>(dst, row, t, beta, alpha);
          }
        } else {
          row_from_acc<T, false>(dst, row, t, beta, 0.f);
        }
        tc_fence_before_sync();
        warp_arrive(&bar_acc_free, lane);
        fence_proxy_async_smem();
        warp_arrive(&bar_out[s], lane);
      }
      if (a.row_mode == kWdRowEps && panel == 0) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) gsum += __shfl_down_sync(0xffffffffu, gsum, off);
        if (lane == 0) atomicAdd(a.dnorm + h, -sigma * (1.0f - sigma) * gsum);
      }
    }
  }

  // ---- leave: make sure no TMA of this CTA is still in flight (bounded), release TMEM ------------
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag) {
    for (int c = (nchunks > NS ? nchunks - NS : 0); c < nchunks; ++c) {
      mbar_wait(&bar_full[c % NS], (c / NS) & 1, 64);
      if (!STATE_ONLY) mbar_wait(&bar_full_x[c % NS], (c / NS) & 1, 64);
    }
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// Decode state of a whole prompt from the segment states of a head-dim-128 state pass:
// state[bh][j][i] (+)= sum_seg seg_state[bh][seg][i][j]   (the decode kernel keeps the value index first,
// GPTCosAttention.py:264).  grid = (B*H, any), block 256: a block takes 32 x 32 tiles through shared memory, so that
// both sides are read and written in whole lines.
__global__ void __launch_bounds__(256)
wide_seg_to_decode_state_kernel(const float* __restrict__ seg_state, float* __restrict__ state, int nseg, int accumulate) {
  __shared__ float tile[32][33];
  const size_t base = static_cast<size_t>(blockIdx.x) * nseg * (128 * 128);
  float* dst = state + static_cast<size_t>(blockIdx.x) * (128 * 128);
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for (int tl = blockIdx.y; tl < 16; tl += gridDim.y) {
    const int i0 = 32 * (tl >> 2), j0 = 32 * (tl & 3);
#pragma unroll
    for (int r = 0; r < 32; r += 8) {
      float sum = 0.f;
      for (int s = 0; s < nseg; ++s) sum += seg_state[base + static_cast<size_t>(s) * (128 * 128) + (i0 + y + r) * 128 + j0 + x];
      tile[y + r][x] = sum;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 32; r += 8) {
      float* d = dst + (j0 + y + r) * 128 + i0 + x;
      *d = (accumulate ? *d : 0.f) + tile[x][y + r];
    }
    __syncthreads();
  }
}

}  // namespace cott
