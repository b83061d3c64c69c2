// fmha_fwd_fast_sm100.cu — the production forward kernel: compact masks only (none, valid
// lengths, additive [B,S_k] row, or a packed variable-length batch), optional Philox dropout,
// writes O and the row logsumexp.
//
// CTA organisation as in the general kernel in fmha_fwd_sm100.cu (TMA producer, tcgen05.mma
// issuer, four softmax warps with one thread per query row; S in tensor memory, P written back
// over it, O beside it).  Head dimension 64 walks the keys in 64-key steps (S 64 + O 64 = 128
// tensor-memory columns); there the producer and the MMA issuer are ONE warp, so a CTA has five
// warps and four CTAs share an SM at 96 registers per thread.  Head dimension 128 uses 128-key
// steps, separate producer and MMA warps and two CTAs per SM.  The softmax is written for instruction count and
// latency, because at head dimension 64 the softmax warps, not the tensor core, set the pace:
//   * mask kind, dropout and the packed-batch bookkeeping are template parameters: no
//     per-chunk branches and no registers spent on modes that are off;
//   * the row maximum is taken over the raw accumulators with 3-input max (the scale is
//     positive), the exponent argument is one packed fma.rn.f32x2 per two elements, the row
//     sum one packed add;
//   * without dropout the scores of a step are read from tensor memory once and held in registers between the maximum and
//     the exponentials; with dropout, whose keep words need registers as well, they are read twice, the load of the next 32
//     columns in flight while the current 32 are processed (exceptions with an additive mask: softmax_step);
//   * with an additive key mask a step whose mask is zero throughout is done like one without a mask, and one whose keys are all
//     masked away, and would add exact zeros, writes zeros for P (B=64 H=16 S=384, lengths U[S/3, S] as a mask: 76.3 -> 65.2 us together with the early loads
//     below);
//     each softmax warp reads the mask for itself, under the wait for the scores;
//   * few CTAs against many keys: the key steps of a query tile are dealt out over a cluster (fwd_key_split); many CTAs of
//     unequal length: the longest sequences first (length_class_shift);
//   * Philox uses one 32x32->64 multiply per product, its keep words for a key step are
//     computed before the step's scores are awaited (they do not depend on them), and the
//     keep decision is applied to the packed 16-bit pairs with two byte permutes and two ANDs
//     per four elements;
//   * the MMA warp issues in bursts from a converged warp (see umma_ss_x4 in sm100_ptx.cuh).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "../../include/fmha_sm100.h"
#include "fmha_device_utils.cuh"
#include "fmha_fwd_softmax.cuh"
#include "fmha_kernel_args.h"
#include "philox.cuh"
#include "sm100_ptx.cuh"

namespace fmha {

namespace {

// D = 128: 192 threads (TMA producer warp, MMA warp, four softmax warps).  D = 64: 160 threads, one warp issues both
// the TMA loads and the MMAs.  Registers are allocated per SM sub-partition (16 384 each, warps dealt round-robin):
// four CTAs of six warps put six warps on a sub-partition (80 registers per thread), four CTAs of five warps put
// five (96), where the plain variant and dropout stay out of local memory (4 bytes with a cluster), the additive mask spills 32 to 36
// bytes and both 24 to 28 (spill stores; D = 128 at 168 registers: plain 36 to 44, dropout 20 to 24, additive 112 to 116, both 140 to 144).
constexpr int kThreadsSplit = 192, kThreadsMerged = 160;
template <int D> constexpr int fast_threads() { return D == 64 ? kThreadsMerged : kThreadsSplit; }
constexpr int kMaxKeySplit = 8;   // portable cluster size

enum FastWaitSite {
  kFQFull = 111, kFKEmpty = 112, kFVEmpty = 113, kFKFull = 114, kFVFull = 115, kFPFull = 116, kFSFull = 117,
  kFOFull = 118, kFQkDone = 119
};

// TN = keys per step.  D = 64 uses 64-key steps: S (64 columns) + O (64 columns) = 128 tensor-memory
// columns and 48 KB of shared memory per CTA, so FOUR CTAs share an SM and their softmax and
// tensor-core phases interleave; D = 128 uses 128-key steps and two CTAs per SM.
template <int D, bool DROP = false>
struct FastSmem {
  static constexpr int TN = (D == 64) ? 64 : 128;
  // Four CTAs per SM at D = 64 (five warps each: 96 registers per thread), two at D = 128.
  static constexpr int kCtasPerSm = (D == 64) ? 4 : 2;
  static constexpr int kStages = (D == 64) ? 2 : 1;
  static constexpr int kQBytes = kTileM * D * 2;
  static constexpr int kTileBytes = TN * D * 2;    // one K or V tile
  static constexpr int kSubTile = TN * 128;        // one 64-column sub-tile of a K/V tile
  static constexpr int kOffQ = 0;
  static constexpr int kOffK = kOffQ + kQBytes;
  static constexpr int kOffV = kOffK + kStages * kTileBytes;
  static constexpr int kOffMask = kOffV + kStages * kTileBytes;  // TN floats per softmax warp
  static constexpr int kOffBar = kOffMask + 4 * TN * 4;
  static constexpr int kNumBars = 4 + (D == 64 ? 2 : 4) * kStages;   // at D = 64 no buffer has a barrier for being empty
  static constexpr int kOffMisc = kOffBar + kNumBars * 8;
  static constexpr int kBytes = kOffMisc + 16;
  static constexpr int kDynBytes = kBytes + 1024;
};

}  // namespace

// PACKED: the batch is one [total_rows, H, D] tensor per operand with row offsets (FMHA_MASK_CU_SEQLENS); a
// template parameter so that the padded kernels carry none of its bookkeeping in registers.
// SPLIT: the keys of a query tile are dealt out over the CTAs of a cluster (see fwd_key_split); each runs its share of
// the key steps and leaves its unnormalised O, row maximum and row sum in its own shared memory, and the cluster
// combines them through distributed shared memory.
template <int D, bool BF16, bool KEYADD, bool DROP, bool PACKED = false, bool SPLIT = false>
__global__ void __launch_bounds__(fast_threads<D>(), FastSmem<D, DROP>::kCtasPerSm) fmha_fwd_fast_kernel(const __grid_constant__ FwdArgs a) {
  griddep_wait();
  constexpr bool MERGED = (D == 64);          // one warp issues the loads and the MMAs
  constexpr int kAllocWarp = 1;               // owns the tensor-memory allocation
  constexpr int kFirstSoftmaxThread = MERGED ? 32 : 64;
  using L = FastSmem<D>;
  constexpr int ST = L::kStages;
  constexpr int TN = L::TN;
  constexpr int kTmemCols = (TN + D <= 128) ? 128 : 256;
  constexpr uint32_t kColS = 0, kColO = TN;
  constexpr int kFmt = BF16 ? 1 : 0;
  constexpr uint32_t kIdescQK = make_idesc_f16(128, TN, kFmt, false, false);
  constexpr uint32_t kIdescPV = make_idesc_f16(128, D, kFmt, false, true);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + L::kOffQ;
  uint8_t* sK = smem + L::kOffK;
  uint8_t* sV = smem + L::kOffV;
  float* sMask = reinterpret_cast<float*>(smem + L::kOffMask);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* q_full = bars + 0;
  uint64_t* s_full = bars + 1;
  uint64_t* p_full = bars + 2;
  uint64_t* o_full = bars + 3;
  uint64_t* k_full = bars + 4;
  uint64_t* v_full = k_full + ST;
  uint64_t* k_empty = v_full + ST;   // D = 128 only
  uint64_t* v_empty = k_empty + ST;
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 4);
  // Philox offset of this launch: the launch parameter plus the optional device-resident value.  Kept in shared
  // memory and read where a draw starts, so that it holds no register in between.
  volatile uint32_t* philox_off = reinterpret_cast<volatile uint32_t*>(smem + L::kOffMisc + 8);
  volatile int* uncovered = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 12);   // packed: rows may be left to zero

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int h = blockIdx.y;
  int b = blockIdx.z;
  int ordered_len = 0;   // the valid length, where it is known already
  if constexpr (D == 64 && !KEYADD && !SPLIT) {
    if (a.length_class_shift >= 0) {
      const int* len = reinterpret_cast<const int*>(a.mask);
      int n = 0;
      if (lane < a.B) n = PACKED ? len[lane + 1] - len[lane] : len[lane];
      if (n > a.S_k || (!PACKED && n <= 0)) n = a.S_k;
      b = batch_of_rank(b, a.B, static_cast<uint32_t>(max(n - 1, 0)) >> a.length_class_shift);
      ordered_len = __shfl_sync(0xffffffffu, n, b);
    }
  }
  const int n_split = SPLIT ? static_cast<int>(cluster_size()) : 1;
  const int split = SPLIT ? static_cast<int>(cluster_rank()) : 0;
  const int q0 = (SPLIT ? blockIdx.x / n_split : blockIdx.x) * kTileM;
  const int bh = b * a.H + h;

  int k_limit = a.S_k;
  int q_limit = a.S_q;     // query rows [0, q_limit) of this (b, h) exist
  int row_base = 0;        // packed batch: first row of sequence b in the [total_rows, H, D] tensors
  int tb = b;              // batch coordinate of the tensor maps (0 for a packed batch)
  constexpr bool packed = PACKED;
  if (!packed && a.mask_kind == FMHA_MASK_SEQLEN) {
    const int len = ordered_len > 0 ? ordered_len : reinterpret_cast<const int*>(a.mask)[b];
    if (len > 0 && len < a.S_k) k_limit = len;
  } else if (packed) {
    const int* cu = reinterpret_cast<const int*>(a.mask);
    row_base = cu[b];
    const int all = cu[b + 1] - row_base;
    const int len = row_base < 0 ? 0 : min(all, a.S_q);   // a sequence longer than the stated maximum is cut there
    k_limit = len;
    q_limit = min(len, a.total_rows - row_base);   // offsets past the tensor, which the host cannot see: no row behind it is written
    tb = 0;
    if (q0 >= len) {   // this sequence has no such query tile (whole CTA, before any barrier)
      if (a.zero_uncovered)
        zero_uncovered_rows(a.o_ptr, a.o_ss, a.o_sh, h, b, a.B, cu, a.S_q, a.total_rows, D, q0, q0 + kTileM,
                            a.zero_uncovered == kUncoveredAll, threadIdx.x, blockDim.x);
      return;
    }
    if (threadIdx.x == 0) *uncovered = a.zero_uncovered && (q0 + kTileM > len || all > len);
  }
  const int n_kv_all = (k_limit + TN - 1) / TN;
  // key steps of this CTA: [j0, j0 + n_kv); with SPLIT possibly none
  const int j0 = SPLIT ? n_kv_all * split / n_split : 0;
  const int n_kv = SPLIT ? n_kv_all * (split + 1) / n_split - j0 : n_kv_all;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *philox_off = a.philox_offset + (a.philox_offset_dev != nullptr ? static_cast<uint32_t>(*a.philox_offset_dev) : 0u);
    mbar_init(q_full, 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 4);
    mbar_init(o_full, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(v_full + s, 1);
      if constexpr (!MERGED) {
        mbar_init(k_empty + s, 1);
        mbar_init(v_empty + s, 1);
      }
    }
    mbar_fence_init();
    fence_proxy_async_smem();
    // The first product's operands, by the thread that has set up their barriers: the rest of the set-up, tensor memory above all,
    // takes as long as they do (some 1 000 of a CTA's first 3 500 cycles; back to back in a graph, B=13 H=12 S=197 10.1 -> 9.2 us, B=64 H=16 S=128 12.6 ->
    // 11.9, B=32 H=12 S=512 with dropout 51.4 -> 50.4).
    mbar_arrive_expect_tx(q_full, L::kQBytes);
#pragma unroll
    for (int c = 0; c < D / 64; ++c) tma_load_4d(sQ + c * 16384, &a.tm_q, q_full, c * 64, row_base + q0, h, tb);
    if (n_kv > 0) {
      mbar_arrive_expect_tx(k_full, L::kTileBytes);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) tma_load_4d(sK + c * L::kSubTile, &a.tm_k, k_full, c * 64, row_base + j0 * TN, h, tb);
    }
    tma_prefetch_desc(&a.tm_v);
    tma_prefetch_desc(&a.tm_o);
  }
  if (warp == kAllocWarp) {
    tmem_alloc(tmem_base_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_base_slot;
  const WaitCtx wctx{abort_flag, a.status};

  if (warp == 0 && !MERGED) {
    // ============================ TMA producer ======================================
    if (lane == 0) {
      for (int j = 0; j < n_kv; ++j) {
        const int s = j % ST;
        if (j >= ST) mbar_wait(k_empty + s, ((j / ST) - 1) & 1, wctx, kFKEmpty);
        if (j > 0) {
          mbar_arrive_expect_tx(k_full + s, L::kTileBytes);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(sK + s * L::kTileBytes + c * L::kSubTile, &a.tm_k, k_full + s, c * 64, row_base + (j0 + j) * TN, h, tb);
        }
        if (j >= ST) mbar_wait(v_empty + s, ((j / ST) - 1) & 1, wctx, kFVEmpty);
        mbar_arrive_expect_tx(v_full + s, L::kTileBytes);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_4d(sV + s * L::kTileBytes + c * L::kSubTile, &a.tm_v, v_full + s, c * 64, row_base + (j0 + j) * TN, h, tb);
      }
    }
  } else if (warp == 0 && MERGED) {
    // ============================ TMA producer + MMA issuer in one warp (D = 64) =====
    // The warp runs convergently; one elected lane issues the loads, MMA bursts go out as in the split version.
    // Under the softmax of step j it waits for Q K^T(j) (P V(j-1), issued before it, has completed by then too), refills what
    // these have released, K of step j+ST and V of step j-1+ST, and makes sure that V(j) and K(j+1) are there.  When P(j) comes,
    // P V(j) and Q K^T(j+1) go out back to back: a poll between them (some 300 cycles while MMAs with both operands in shared
    // memory run) or a second one after P(j) would stand in the chain the step time hangs on.
    // (Polls in between, and 128 arrivals on p_full instead of one per warp: B=4 H=16 S=2048 115.9 us against 101.3, B=64 H=16
    // S=512 104.8 against 100.5; the split version B=16 H=8 S=512 D=128 with an additive mask 31.3 against 27.7.)
    if constexpr (MERGED) {
      constexpr int KQ = D / 16;     // k-steps of S = Q K^T
      constexpr int KP = TN / 16;    // k-steps of O += P V
      static_assert(KQ == 4 && KP == 4, "merged warp: D = 64 with 64-key steps");
      const uint32_t tS = tmem_base + kColS;
      const uint32_t tO = tmem_base + kColO;
      auto load_k = [&](int j) {
        const int s = j % ST;
        mbar_arrive_expect_tx(k_full + s, L::kTileBytes);
        tma_load_4d(sK + s * L::kTileBytes, &a.tm_k, k_full + s, 0, row_base + (j0 + j) * TN, h, tb);
      };
      auto load_v = [&](int j) {
        const int s = j % ST;
        mbar_arrive_expect_tx(v_full + s, L::kTileBytes);
        tma_load_4d(sV + s * L::kTileBytes, &a.tm_v, v_full + s, 0, row_base + (j0 + j) * TN, h, tb);
      };
      const uint64_t dq = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
      uint64_t aq[KQ];
#pragma unroll
      for (int kk = 0; kk < KQ; ++kk) aq[kk] = dq + kmajor_step(kk, 16384);
      auto issue_qk = [&](int j) {
        const uint64_t dk = make_smem_desc_sw128(smem_u32(sK + (j % ST) * L::kTileBytes), 16, 1024);
        uint64_t bk[KQ];
#pragma unroll
        for (int kk = 0; kk < KQ; ++kk) bk[kk] = dk + kmajor_step(kk, L::kSubTile);
        umma_ss_x4(tS, aq, bk, kIdescQK, 0u);
        umma_commit_elect(s_full);
      };
      mbar_wait(q_full, 0, wctx, kFQFull);
      if (n_kv > 0) {
        mbar_wait(k_full, 0, wctx, kFKFull);
        tc_fence_after_sync();
        issue_qk(0);
        if (elect_one()) {   // after Q and K(0): the first product waits for these alone
          load_v(0);
          if (n_kv > 1) {
            load_k(1);
            load_v(1);
          }
        }
        __syncwarp();
      }
      for (int j = 0; j < n_kv; ++j) {
        const int s = j % ST;
        const uint64_t dv = make_smem_desc_sw128(smem_u32(sV + s * L::kTileBytes), L::kSubTile, 1024);
        uint64_t bv[KP];
#pragma unroll
        for (int kk = 0; kk < KP; ++kk) bv[kk] = dv + mnmajor_step(kk);
        const bool more_k = j + ST < n_kv, more_v = j >= 1 && j - 1 + ST < n_kv, more = j + 1 < n_kv;
        if (more_k || more_v) {
          mbar_wait(s_full, j & 1, wctx, kFQkDone);
          if (elect_one()) {
            if (more_k) load_k(j + ST);
            if (more_v) load_v(j - 1 + ST);
          }
          __syncwarp();
        }
        mbar_wait(v_full + s, (j / ST) & 1, wctx, kFVFull);
        if (more) mbar_wait(k_full + (j + 1) % ST, ((j + 1) / ST) & 1, wctx, kFKFull);
        mbar_wait(p_full, j & 1, wctx, kFPFull);
        tc_fence_after_sync();
        umma_ts_x4(tO, tS, 8u, bv, kIdescPV, (j > 0) ? 1u : 0u);
        if (more) issue_qk(j + 1);
      }
      umma_commit_elect(o_full);
    }
  } else if (warp == 1 && !MERGED) {
    // ============================ MMA issuer ========================================
    // The warp runs the loop convergently and issues the MMAs in bursts from one elected lane
    // with descriptors prepared beforehand (see umma_ss_x4): a single lane that computes each
    // descriptor and then issues is starved of issue slots by the softmax warps.
    {
      constexpr int KQ = D / 16;     // k-steps of S = Q K^T
      constexpr int KP = TN / 16;    // k-steps of O += P V
      const uint32_t tS = tmem_base + kColS;
      const uint32_t tO = tmem_base + kColO;
      const uint64_t dq = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
      uint64_t aq[KQ];
#pragma unroll
      for (int kk = 0; kk < KQ; ++kk) aq[kk] = dq + kmajor_step(kk, 16384);
      auto issue_qk = [&](int j) {
        const int s = j % ST;
        const uint64_t dk = make_smem_desc_sw128(smem_u32(sK + s * L::kTileBytes), 16, 1024);
        uint64_t bk[KQ];
#pragma unroll
        for (int kk = 0; kk < KQ; ++kk) bk[kk] = dk + kmajor_step(kk, L::kSubTile);
        if constexpr (KQ == 4) umma_ss_x4(tS, aq, bk, kIdescQK, 0u);
        else umma_ss_x8(tS, aq, bk, kIdescQK, 0u);
        umma_commit_elect(s_full);
        umma_commit_elect(k_empty + s);
      };
      mbar_wait(q_full, 0, wctx, kFQFull);
      if (n_kv > 0) {
        mbar_wait(k_full, 0, wctx, kFKFull);
        tc_fence_after_sync();
        issue_qk(0);
      }
      for (int j = 0; j < n_kv; ++j) {
        const int s = j % ST;
        const uint64_t dv = make_smem_desc_sw128(smem_u32(sV + s * L::kTileBytes), L::kSubTile, 1024);
        uint64_t bv[KP];
#pragma unroll
        for (int kk = 0; kk < KP; ++kk) bv[kk] = dv + mnmajor_step(kk);
        const bool more = j + 1 < n_kv;
        // what P V(j) and Q K^T(j+1) need is waited for under the softmax of step j, see the merged version
        mbar_wait(v_full + s, (j / ST) & 1, wctx, kFVFull);
        if (more) mbar_wait(k_full + (j + 1) % ST, ((j + 1) / ST) & 1, wctx, kFKFull);
        mbar_wait(p_full, j & 1, wctx, kFPFull);
        tc_fence_after_sync();
        const uint32_t acc0 = (j > 0) ? 1u : 0u;
        {
          const uint64_t (&b0)[4] = *reinterpret_cast<const uint64_t (*)[4]>(&bv[0]);
          umma_ts_x4(tO, tS, 8u, b0, kIdescPV, acc0);
        }
        if constexpr (KP == 8) {
          const uint64_t (&b1)[4] = *reinterpret_cast<const uint64_t (*)[4]>(&bv[4]);
          umma_ts_x4(tO, tS + 32u, 8u, b1, kIdescPV, 1u);
        }
        umma_commit_elect(v_empty + s);
        if (more) issue_qk(j + 1);
      }
      umma_commit_elect(o_full);
    }
  } else {
    // ============================ softmax / epilogue ================================
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int tid = threadIdx.x - kFirstSoftmaxThread;
    const int q_row = q0 + row;
    const bool row_ok = q_row < q_limit;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr + kColS;
    const uint32_t tO = tmem_base + lane_addr + kColO;
    const float sl2 = a.scale_log2;
    const DropRow drop_row = {a.philox_keys, philox_off, static_cast<uint32_t>(a.philox_bh_offset + bh), static_cast<uint32_t>(q_row), a.philox_thr};

    // Rows past the end are never stored, so with a handful of query rows against long keys a warp that has no row
    // leaves P and O undefined instead of competing with the others.  (No gain at a ragged last tile of a full grid.)
    const bool warp_idle = SPLIT && q0 + quad * 32 >= q_limit;

    auto arrive_p = [&]() {   // one arrival per warp
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    };

    float m_ref = -INFINITY;
    float2 sum2 = make_float2(0.f, 0.f);  // running sum of exp2(t - m_ref), two interleaved partial sums

    [[maybe_unused]] float* mask_stage = sMask + quad * TN;   // the warp's own copy of the step's mask in the log2 domain

    for (int j = 0; j < n_kv; ++j) {
      const int col0 = (j0 + j) * TN;
      const int n_cols = min(TN, k_limit - col0);
      int kind = kMaskZero;
      if constexpr (KEYADD) {   // under the wait for the scores (each warp for itself: the warps of a CTA need no barrier for it)
        float mk[TN / 32];
        bool exists[TN / 32];
#pragma unroll
        for (int i = 0; i < TN / 32; ++i) {
          const int c = col0 + i * 32 + lane;
          exists[i] = c < a.S_k;
          mk[i] = exists[i] ? reinterpret_cast<const float*>(a.mask)[static_cast<size_t>(b) * a.S_k + c] * kLog2eF : 0.f;
        }
        kind = mask_step_kind(mk, exists);
        if (kind != kMaskZero) {
          __syncwarp();   // the step before has been read
#pragma unroll
          for (int i = 0; i < TN / 32; ++i) mask_stage[i * 32 + lane] = mk[i];
          __syncwarp();
        }
      }
      if (warp_idle) {   // no query row of this warp exists: only keep the step's barriers in phase
        mbar_wait(s_full, j & 1, wctx, kFSFull, 32);
        arrive_p();
        continue;
      }
      auto wait_s = [&]() { mbar_wait(s_full, j & 1, wctx, kFSFull, 32); };
      auto arrive = [&](int) { arrive_p(); };
      if constexpr (D == 64)
        softmax_step_64<BF16, KEYADD, DROP>(tS, tO, col0, n_cols, sl2, mask_stage, kind, drop_row, m_ref, sum2, wait_s, arrive);
      else
        softmax_step_128<BF16, KEYADD, DROP, 0>(tS, tO, col0, n_cols, sl2, mask_stage, kind, drop_row, m_ref, sum2, wait_s, arrive, [] {}, [] {});
    }

    // ---- epilogue ------------------------------------------------------------------------
    mbar_wait(o_full, 0, wctx, kFOFull, 32);
    tc_fence_after_sync();
    const float l_sum = sum2.x + sum2.y;
    if constexpr (SPLIT) {
      // this CTA's share of the row: [128][D] fp32 over the K and V buffers (every load has been consumed) with the
      // 16-byte chunks of a row XORed by the row, so that the 32 rows of a warp spread over the banks; statistics
      // where Q was
      float2* stats = reinterpret_cast<float2*>(sQ);
      stats[row] = make_float2(m_ref, l_sum);
      uint8_t* part = sK + row * (D * 4);
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        if (n_kv > 0) {   // with no key step nothing has been accumulated
          tmem_ld32(tO + c * 32, r);
          tmem_wait_ld_dep(r);
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k) r[k] = 0u;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(part + (((c * 8 + q) ^ (row & 7)) << 4)) =
              make_uint4(r[q * 4], r[q * 4 + 1], r[q * 4 + 2], r[q * 4 + 3]);
      }
    } else {
    const float out_scale = (DROP ? a.dropout_scale : 1.0f) / l_sum;
    if (a.lse != nullptr && row_ok) {
      const size_t li = packed ? static_cast<size_t>(h) * a.total_rows + row_base + q_row   // [H, total_rows]
                               : static_cast<size_t>(bh) * a.S_q + q_row;                   // [B*H, S_q]
      a.lse[li] = (m_ref + fast_log2(l_sum)) * kLn2F;
    }
    // A packed batch's last query tile of a sequence holds rows of the NEXT sequence past q_limit: its rows
    // are written one by one from registers instead of through the tile store.
    const bool partial_rows = packed && (q0 + kTileM > q_limit);
    // (Q is no longer needed: every Q K^T has completed.)
    o_tile_out<D, BF16>(tO, out_scale, sQ, row, partial_rows, row_ok,
                        reinterpret_cast<unsigned short*>(a.o_ptr) + static_cast<int64_t>(row_base + q_row) * a.o_ss + static_cast<int64_t>(h) * a.o_sh);
    fence_proxy_async_smem();
    named_bar_sync(1, 128);
    if (tid == 0) {
      if (*abort_flag == 0 && !partial_rows) {
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_store_4d(&a.tm_o, sQ + c * 16384, c * 64, row_base + q0, h, tb);
        tma_store_commit();
      }
      tma_store_wait_read();  // the shared-memory source must outlive the copy; the writes finish on their own
    }
    }
  }

  if constexpr (PACKED) {   // last, so that no start of a CTA waits for the offsets
    if (*uncovered)
      zero_uncovered_rows(a.o_ptr, a.o_ss, a.o_sh, h, b, a.B, reinterpret_cast<const int*>(a.mask), a.S_q, a.total_rows, D, q0,
                          q0 + kTileM, a.zero_uncovered == kUncoveredAll, threadIdx.x, blockDim.x);
  }
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (SPLIT) {
    // ============================ combine the cluster's shares ======================
    // Work: (query row, 8 columns) pairs, dealt out over all threads of the cluster; every thread reads the row's
    // statistics and its 8 columns of every share.  No wait precedes the cluster barriers that is not bounded, so
    // every CTA arrives, also after a wait was given up.
    cluster_sync();
    const int rows = min(kTileM, q_limit - q0);
    const int items = *abort_flag ? 0 : rows * (D / 8);
    const uint32_t stats_addr = smem_u32(sQ), part_addr = smem_u32(sK);
    for (int i = split * blockDim.x + threadIdx.x; i < items; i += n_split * blockDim.x) {
      const int row = i / (D / 8), ch = i % (D / 8);
      float m[kMaxKeySplit], l[kMaxKeySplit];
      float m_all = -INFINITY, l_all = 0.f;
#pragma unroll
      for (int k = 0; k < kMaxKeySplit; ++k) {
        const float2 st = k < n_split ? dsmem_ld2(dsmem_map(stats_addr + row * 8, k)) : make_float2(-INFINITY, 0.f);
        m[k] = st.x;
        l[k] = st.y;
        m_all = fmaxf(m_all, m[k]);
      }
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < kMaxKeySplit; ++k) {
        if (k >= n_split) break;
        const float w = fast_exp2(m[k] - m_all);   // 0 for a share without key steps, or with keys masked by -inf only
        l_all = fmaf(w, l[k], l_all);
        const uint32_t src = dsmem_map(part_addr + row * (D * 4), k);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float4 x = dsmem_ld4(src + (((ch * 2 + q) ^ (row & 7)) << 4));
          acc[q * 4 + 0] = fmaf(w, x.x, acc[q * 4 + 0]);
          acc[q * 4 + 1] = fmaf(w, x.y, acc[q * 4 + 1]);
          acc[q * 4 + 2] = fmaf(w, x.z, acc[q * 4 + 2]);
          acc[q * 4 + 3] = fmaf(w, x.w, acc[q * 4 + 3]);
        }
      }
      const float out_scale = (DROP ? a.dropout_scale : 1.0f) / l_all;
      uint4 w4;
      w4.x = pack2<BF16>(acc[0] * out_scale, acc[1] * out_scale);
      w4.y = pack2<BF16>(acc[2] * out_scale, acc[3] * out_scale);
      w4.z = pack2<BF16>(acc[4] * out_scale, acc[5] * out_scale);
      w4.w = pack2<BF16>(acc[6] * out_scale, acc[7] * out_scale);
      *reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(a.o_ptr) + b * a.o_sb + h * a.o_sh +
                                static_cast<int64_t>(q0 + row) * a.o_ss + ch * 8) = w4;
      if (ch == 0 && a.lse != nullptr)
        a.lse[static_cast<size_t>(bh) * a.S_q + q0 + row] = (m_all + fast_log2(l_all)) * kLn2F;
    }
    cluster_sync();   // no CTA leaves while another one reads its shared memory
  }
  if (*abort_flag) {
    for (int k = 0; k < 20; ++k) __nanosleep(1000000);
    __syncthreads();
  }
  if (warp == kAllocWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Over how many CTAs of a cluster the keys of a query tile are split: the candidate (1, 2, 4, 8) of least modelled time, in units
// of one key step of a CTA that has its SM to itself (0.97 us at D = 64, 1.7 us at D = 128, measured: there a step is a chain of
// latencies, as long for one query row as for 128; 1.2 units with an additive mask or dropout).  A split adds the cluster
// launch, its barriers and the combination (`overhead`, from the times of 4 to 96 tiles over 128 to 2048 keys).  With more CTAs
// than SMs a step takes 1.2 times as long and the start of a cluster longer, the more the larger it is; more than two CTAs per
// SM never paid.  Measured, one share / the split chosen: 24 tiles of 20 rows, 1024 keys D=64 18.6 / 9.6 us (4), D=128 17.2 / 10.0
// (4); 12 tiles of 128 rows 18.6 / 10.1 (8) and 17.6 / 13.2 (4); 48 tiles, 1024 keys 19.0 / 14.0 (4) and 17.6 / 15.8 (2), 512 keys
// 11.2 / 11.0 (2) and 10.9 (1; 15.4 as 4 shares); 32 tiles, 384 keys D=64 9.1 (1; 14.6 as 8 shares).
static int fwd_key_split(int64_t ctas, int steps, int S_q, int D, bool long_step, int sms) {
  static constexpr float kOverhead[2][2][3] = {{{1.9f, 2.4f, 3.2f}, {3.7f, 4.0f, 4.8f}},     // D = 64: up to 32 rows, more
                                               {{1.05f, 1.5f, 2.2f}, {2.75f, 3.4f, 4.7f}}};  // D = 128
  const bool few_rows = S_q <= 32;
  const float step = long_step ? 1.2f : 1.0f;
  int best = 1;
  float best_cost = static_cast<float>(steps) * step;
  for (int s = 2, i = 0; s <= kMaxKeySplit && ctas * s <= 2 * static_cast<int64_t>(sms) && s < 2 * steps; s *= 2, ++i) {
    const bool crowded = ctas * s > sms;
    const float cost = static_cast<float>((steps + s - 1) / s) * step * (crowded ? 1.2f : 1.0f) + kOverhead[D == 64 ? 0 : 1][few_rows ? 0 : 1][i] +
                       (crowded ? (few_rows ? 0.1f : 0.6f) * s : 0.f);
    if (cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

// Longest sequences first: with valid lengths the CTAs of a batch differ in their number of key steps, and they start in grid
// order.  The shift that puts the lengths into eight classes, or -1 for the order of the batch.  Each CTA finds its batch
// element by itself (a load and some 200 cycles at its start), which pays at D = 64 up to four rounds of resident CTAs, where
// the last ones to finish leave SMs idle (lengths U[S/2, S]: B=8 H=12 S=512 16.2 -> 14.9 us, B=16 H=8 S=640 with dropout
// 35.2 -> 33.3, B=32 H=12 S=512 with dropout 57.0 -> 54.2); beyond it does not (B=64 H=16 S=384 62.3 -> 64.9 us, with two
// elements per lane), nor at D = 128, where a CTA's start is the longer chain (B=16 H=12 S=512 37.1 -> 38.4 us), and with no
// more CTAs than SMs the order does not matter.  These figures are of a CTA per tile.  The kernel that goes from tile to tile keeps the rule, and gains
// as much: B=32 S=512 with dropout, lengths U[256, 512] 12 heads 48.3 -> 45.1 us, 16 heads 64.7 -> 58.8, U[128, 512] 45.3 -> 39.2 and 57.1 -> 51.2, B=32
// H=16 S=256 without 16.8 -> 15.8.
int fwd_length_class_shift(const FwdArgs& a, int D, int64_t ctas, bool no_lengths) {
  if (no_lengths || D != 64 || (a.mask_kind != FMHA_MASK_SEQLEN && a.mask_kind != FMHA_MASK_CU_SEQLENS) || a.B < 2 || a.B > kMaxOrdered)
    return -1;
  const int64_t sms = sm_count();
  if (ctas <= sms || ctas > 4 * FastSmem<64>::kCtasPerSm * sms) return -1;
  int shift = 0;
  while ((a.S_k - 1) >> shift > 7) ++shift;
  return shift;
}

template <int D, bool BF16, bool KEYADD, bool DROP, bool PACKED = false, bool SPLIT = false>
static int launch_fast_impl(const FwdArgs& a, cudaStream_t stream, int n_split = 1) {
  using L = FastSmem<D>;
  if constexpr (!PACKED && !SPLIT) {
    const int s = fwd_key_split(static_cast<int64_t>((a.S_q + kTileM - 1) / kTileM) * a.H * a.B, (a.S_k + L::TN - 1) / L::TN, a.S_q, D,
                                KEYADD || DROP, sm_count());
    if (s > 1) return launch_fast_impl<D, BF16, KEYADD, DROP, false, true>(a, stream, s);
  }
  auto kfn = fmha_fwd_fast_kernel<D, BF16, KEYADD, DROP, PACKED, SPLIT>;
  static std::atomic<bool> configured[64] = {};   // per device; set after the attribute call succeeded
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  dim3 grid((a.S_q + kTileM - 1) / kTileM * n_split, a.H, a.B);
  FwdArgs args = a;
  args.length_class_shift = fwd_length_class_shift(a, D, static_cast<int64_t>(grid.x) * grid.y * grid.z, KEYADD || SPLIT);
  const cudaError_t e = launch_overlapped(kfn, grid, dim3(fast_threads<D>()), L::kDynBytes, stream, args, SPLIT ? n_split : 0);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_fwd_fast(const FwdArgs& a, int D, int dtype, cudaStream_t stream) {
  if (fwd_pair_applies(a, D)) return launch_fwd_pair(a, dtype, stream);
  if (fwd_chain_applies(a, D)) return launch_fwd_chain(a, dtype, stream);
  const bool bf = dtype == FMHA_DTYPE_BF16;
  const bool keyadd = a.mask_kind == FMHA_MASK_KEY_ADDITIVE;
  const bool drop = a.dropout_kind == FMHA_DROPOUT_PHILOX;
  if (a.mask_kind == FMHA_MASK_CU_SEQLENS) {
#define FMHA_FAST_PACKED(DD, BF, DR) \
  if (D == DD && bf == BF && drop == DR) return launch_fast_impl<DD, BF, false, DR, true>(a, stream);
    FMHA_FAST_PACKED(64, false, false)
    FMHA_FAST_PACKED(64, false, true)
    FMHA_FAST_PACKED(64, true, false)
    FMHA_FAST_PACKED(64, true, true)
    FMHA_FAST_PACKED(128, false, false)
    FMHA_FAST_PACKED(128, false, true)
    FMHA_FAST_PACKED(128, true, false)
    FMHA_FAST_PACKED(128, true, true)
#undef FMHA_FAST_PACKED
    return static_cast<int>(cudaErrorInvalidValue);
  }
#define FMHA_FAST_CASE(DD, BF, KA, DR) \
  if (D == DD && bf == BF && keyadd == KA && drop == DR) return launch_fast_impl<DD, BF, KA, DR>(a, stream);
  FMHA_FAST_CASE(64, false, false, false)
  FMHA_FAST_CASE(64, false, false, true)
  FMHA_FAST_CASE(64, false, true, false)
  FMHA_FAST_CASE(64, false, true, true)
  FMHA_FAST_CASE(64, true, false, false)
  FMHA_FAST_CASE(64, true, false, true)
  FMHA_FAST_CASE(64, true, true, false)
  FMHA_FAST_CASE(64, true, true, true)
  FMHA_FAST_CASE(128, false, false, false)
  FMHA_FAST_CASE(128, false, false, true)
  FMHA_FAST_CASE(128, false, true, false)
  FMHA_FAST_CASE(128, false, true, true)
  FMHA_FAST_CASE(128, true, false, false)
  FMHA_FAST_CASE(128, true, false, true)
  FMHA_FAST_CASE(128, true, true, false)
  FMHA_FAST_CASE(128, true, true, true)
#undef FMHA_FAST_CASE
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // namespace fmha
