// fmha_fwd_chain_sm100.cu — forward kernel of head dimension 64 for grids of more query tiles than the chip holds at a time and few key
// steps (fwd_chain_pays): compact masks (none, valid lengths, additive [B,S_k] row), optional Philox dropout, O and the row logsumexp.
//
// The CTA of fmha_fwd_fast_sm100.cu (one 128-row query tile, 64-key steps, five warps, four CTAs per SM), which goes on to further
// tiles handed out by cluster launch control, without a gap between them: under the softmax of a tile's last step the next
// tile's Q and first two K tiles are loaded, its first Q K^T goes out right behind the last P V, and its V tiles are loaded while
// the softmax warps do its first step.  O leaves through the V buffers, by a tile store of the warp that issues loads and MMAs.
//
// What bounds it: a key step takes a softmax warp 2 200 to 2 900 cycles (draws 750, wait for the scores 120, maximum and exponentials 1 300, with
// dropout 1 650), four of which run at a time per scheduler against 512 of exponentials each; a CTA per tile added its start (launch, tensor
// memory, first loads, first product: 3 500 cycles) and its end (2 500), here a tile ends in 1 800 (P V 500, O 800, the next item 400).
// Four CTAs per SM hide part of either: B=64 H=16 S=384 with an additive mask 65.8 -> 62.9 us, B=32 H=12 S=512 with dropout 49.4 -> 47.7,
// B=228 H=12 S=64 with a mask 23.1 -> 17.8 (kernel times).  With an additive mask it spills 68 bytes where the other kernel spills 32 (with dropout as well 8, 24
// there; without either 4, none there).  The additive mask of a step brought into shared memory a step ahead took its 600 cycles
// out of the chain and left the time as it was (62.9 / 64.3).  A packed batch is left to the other kernel: each tile past the end of its
// sequence costs a question and an answer here (the tracked unpadded batch 62.2 -> 68.3).
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

constexpr int kChThreads = 160;
constexpr int kChCtasPerSm = 4;

enum ChainWaitSite {
  kChQFull = 121, kChKFull = 122, kChVFull = 123, kChPFull = 124, kChSFull = 125, kChQkDone = 126, kChOFull = 127, kChOStaged = 128,
  kChItem = 129, kChItemEmpty = 130, kChClc = 131, kChSmemBase = 132
};

constexpr int D = 64;
struct ChainSmem {
  static constexpr int TN = 64;                    // keys per step
  static constexpr int kQBytes = kTileM * D * 2;
  static constexpr int kTile = TN * D * 2;         // a K or V tile
  static constexpr int kOffQ = 0;
  static constexpr int kOffK = kOffQ + kQBytes;    // 2 tiles
  static constexpr int kOffV = kOffK + 2 * kTile;  // 2 tiles; between two query tiles the O tile
  static constexpr int kOffMask = kOffV + 2 * kTile;   // TN floats per softmax warp
  static constexpr int kOffItems = kOffMask + 4 * TN * 4;   // 2 x 16 bytes
  static constexpr int kOffClc = kOffItems + 32;
  static constexpr int kOffBar = kOffClc + 16;
  static constexpr int kNumBars = 14;
  static constexpr int kOffMisc = kOffBar + kNumBars * 8;   // tensor-memory base, abort flag, Philox offset
  static constexpr int kDynBytes = kOffMisc + 16;           // 1024-byte aligned base: checked by the kernel
  static_assert(2 * kTile == kTileM * D * 2, "the O tile fits over V");
};

struct ChainItem {
  int b, h, q0;
  int k_limit;   // keys [0, k_limit) of this (b, h)
};

}  // namespace

template <bool BF16, bool KEYADD, bool DROP>
__global__ void __launch_bounds__(kChThreads, kChCtasPerSm) fmha_fwd_chain_kernel(const __grid_constant__ FwdArgs a) {
  griddep_wait();
  using L = ChainSmem;
  constexpr int TN = L::TN;
  constexpr int kTmemCols = 128;
  constexpr uint32_t kColS = 0, kColO = TN;
  constexpr int kFmt = BF16 ? 1 : 0;
  constexpr uint32_t kIdescQK = make_idesc_f16(128, TN, kFmt, false, false);
  constexpr uint32_t kIdescPV = make_idesc_f16(128, D, kFmt, false, true);

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem + L::kOffQ;
  uint8_t* sK = smem + L::kOffK;
  uint8_t* sV = smem + L::kOffV;
  uint4* clc_answer = reinterpret_cast<uint4*>(smem + L::kOffClc);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* q_full = bars + 0;
  uint64_t* s_full = bars + 1;
  uint64_t* p_full = bars + 2;       // one arrival per softmax warp
  uint64_t* o_full = bars + 3;
  uint64_t* o_staged = bars + 4;     // O has been read, and is in shared memory (one arrival per softmax warp)
  uint64_t* clc_full = bars + 5;
  uint64_t* k_full = bars + 6;       // [2]
  uint64_t* v_full = bars + 8;       // [2]
  uint64_t* item_full = bars + 10;   // [2]
  uint64_t* item_empty = bars + 12;  // [2] one arrival per softmax warp
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 4);
  volatile uint32_t* philox_off = reinterpret_cast<volatile uint32_t*>(smem + L::kOffMisc + 8);   // launch parameter plus device-resident value

  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0 && a.status != nullptr) atomicCAS(a.status, 0, kChSmemBase);
    return;
  }
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitCtx wctx{abort_flag, a.status};
  const uint32_t ring = smem_u32(smem + L::kOffItems);

  // Whole warp.
  auto decode = [&](int x, int y, int z) {
    ChainItem it;
    int b = z;
    it.h = y;
    it.q0 = x * kTileM;
    it.k_limit = a.S_k;
    if constexpr (!KEYADD) {
      if (a.length_class_shift >= 0) {
        const int* len = reinterpret_cast<const int*>(a.mask);
        int n = 0;
        if (lane < a.B) n = len[lane];
        if (n > a.S_k || n <= 0) n = a.S_k;
        b = batch_of_rank(z, a.B, static_cast<uint32_t>(max(n - 1, 0)) >> a.length_class_shift);
      }
    }
    it.b = b;
    if (a.mask_kind == FMHA_MASK_SEQLEN) {
      const int len = reinterpret_cast<const int*>(a.mask)[b];
      if (len > 0 && len < a.S_k) it.k_limit = len;
    }
    return it;
  };

  auto load_q = [&](const ChainItem& it) {   // one lane
    mbar_arrive_expect_tx(q_full, L::kQBytes);
    tma_load_4d(sQ, &a.tm_q, q_full, 0, it.q0, it.h, it.b);
  };
  auto load_k = [&](const ChainItem& it, int j, uint32_t g) {   // key step j of the item, step g of the CTA
    mbar_arrive_expect_tx(k_full + (g & 1), L::kTile);
    tma_load_4d(sK + (g & 1) * L::kTile, &a.tm_k, k_full + (g & 1), 0, j * TN, it.h, it.b);
  };
  auto load_v = [&](const ChainItem& it, int j, uint32_t g) {
    mbar_arrive_expect_tx(v_full + (g & 1), L::kTile);
    tma_load_4d(sV + (g & 1) * L::kTile, &a.tm_v, v_full + (g & 1), 0, j * TN, it.h, it.b);
  };
  auto steps_of = [&](const ChainItem& it) { return (it.k_limit + TN - 1) / TN; };

  ChainItem it;
  if (warp == 0) {
    if (lane == 0) {
      *abort_flag = 0;
      *philox_off = a.philox_offset + (a.philox_offset_dev != nullptr ? static_cast<uint32_t>(*a.philox_offset_dev) : 0u);
      mbar_init(q_full, 1);
      mbar_init(s_full, 1);
      mbar_init(p_full, 4);
      mbar_init(o_full, 1);
      mbar_init(o_staged, 4);
      mbar_init(clc_full, 1);
      for (int s = 0; s < 2; ++s) {
        mbar_init(k_full + s, 1);
        mbar_init(v_full + s, 1);
        mbar_init(item_full + s, 1);
        mbar_init(item_empty + s, 4);
      }
      mbar_fence_init();
      fence_proxy_async_smem();
    }
    __syncwarp();
    it = decode(blockIdx.x, blockIdx.y, blockIdx.z);
    if (elect_one()) {   // before tensor memory is there, as in the other kernel
      load_q(it);
      load_k(it, 0, 0);
    }
    __syncwarp();
  }
  if (warp == 1) {
    tmem_alloc(tmem_base_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_base_slot;

  if (warp == 0) {
    // ============================ loads, MMAs, O stores, work items ====================
    // The whole warp runs this convergently; one elected lane issues loads and stores, MMAs go out in bursts (see umma_ss_x4).  No
    // buffer has a barrier for being empty: K(g) has been read when S(g) is there, V(g) when S(g+1) is, V of an item's last step
    // when O is.  Key steps are counted through all items (g); what needs no wait under the softmax of a step is waited for there.
    const uint32_t tS = tmem_base + kColS, tO = tmem_base + kColO;
    const uint64_t dq = make_smem_desc_sw128(smem_u32(sQ), 16, 1024);
    auto issue_qk = [&](uint32_t g) {
      const uint64_t dk = make_smem_desc_sw128(smem_u32(sK + (g & 1) * L::kTile), 16, 1024);
      uint64_t x[4], y[4];
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        x[kk] = dq + kmajor_step(kk, 16384);
        y[kk] = dk + kmajor_step(kk, L::kTile);
      }
      umma_ss_x4(tS, x, y, kIdescQK, 0u);
      umma_commit_elect(s_full);
    };
    int n = 0;          // items published
    uint32_t g0 = 0;    // the item's first key step
    uint32_t w = 0;     // its number
    uint32_t clc_phase = 0;
    bool more_items = true, asked = false;   // of the grid: CTAs that have not been launched
    auto publish = [&](const ChainItem& x, bool end) {
      const int slot = n & 1;
      if (n >= 2) mbar_wait(item_empty + slot, ((n >> 1) - 1) & 1, wctx, kChItemEmpty);
      if (lane == 0) {
        sts128(ring + slot * 16, end ? 0xffffffffu : static_cast<uint32_t>(x.b), static_cast<uint32_t>(x.h), static_cast<uint32_t>(x.q0),
               static_cast<uint32_t>(x.k_limit));
        mbar_arrive(item_full + slot);
      }
      __syncwarp();
      ++n;
    };
    auto ask = [&]() {   // for the index of a CTA that has not been launched
      if (!more_items) return;
      if (elect_one()) {
        mbar_arrive_expect_tx(clc_full, 16);
        clc_try_cancel(clc_answer, clc_full);
      }
      __syncwarp();
      asked = true;
    };
    auto answer = [&](ChainItem& x) -> bool {   // whether there was one
      if (!asked) return false;
      asked = false;
      mbar_wait(clc_full, clc_phase, wctx, kChClc);
      clc_phase ^= 1u;
      int cx, cy, cz;
      const bool have = clc_query(clc_answer, cx, cy, cz) && *abort_flag == 0;
      fence_proxy_async_smem();   // the answer's place is written by the async proxy again
      more_items = __all_sync(0xffffffffu, have);
      if (more_items) x = decode(cx, cy, cz);
      return more_items;
    };
    auto store_o = [&](const ChainItem& x, uint32_t phase) {   // O of a finished item, staged by the softmax warps
      mbar_wait(o_staged, phase, wctx, kChOStaged);
      tc_fence_after_sync();
      if (elect_one()) {
        if (*abort_flag == 0) {
          tma_store_4d(&a.tm_o, sV, 0, x.q0, x.h, x.b);
          tma_store_commit();
        }
        tma_store_wait_read();
      }
      __syncwarp();
    };

    publish(it, false);
    ChainItem prev = it;
    int k_loaded = 1;     // K tiles of `it` on their way, and its Q
    for (bool run = true; run;) {
      const int n_kv = steps_of(it);
      mbar_wait(q_full, w & 1, wctx, kChQFull);
      mbar_wait(k_full + (g0 & 1), (g0 >> 1) & 1, wctx, kChKFull);
      tc_fence_after_sync();
      issue_qk(g0);
      if (w > 0) store_o(prev, (w - 1) & 1);
      if (elect_one()) {
        load_v(it, 0, g0);
        if (n_kv > 1) {
          if (k_loaded < 2) load_k(it, 1, g0 + 1);
          load_v(it, 1, g0 + 1);
        }
      }
      __syncwarp();
      ask();
      ChainItem nxt = it;
      run = false;
      int nxt_k = 0;
      for (int j = 0; j < n_kv; ++j) {
        const uint32_t g = g0 + j;
        const uint64_t dv = make_smem_desc_sw128(smem_u32(sV + (g & 1) * L::kTile), L::kTile, 1024);
        uint64_t bv[4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) bv[kk] = dv + mnmajor_step(kk);
        const bool last = j + 1 == n_kv, more_k = j + 2 < n_kv, more_v = j >= 1 && !last;
        if (more_k || more_v || (last && asked)) {
          mbar_wait(s_full, g & 1, wctx, kChQkDone);
          if (elect_one()) {
            if (more_k) load_k(it, j + 2, g + 2);
            if (more_v) load_v(it, j + 1, g + 1);
          }
          __syncwarp();
          if (last) {   // Q and both K buffers have been read
            run = answer(nxt);
            if (run) {
              const int nk = steps_of(nxt);
              nxt_k = nk > 1 ? 2 : 1;
              if (elect_one()) {
                load_q(nxt);
                load_k(nxt, 0, g + 1);
                if (nk > 1) load_k(nxt, 1, g + 2);
              }
              __syncwarp();
              publish(nxt, false);
            }
          }
        }
        mbar_wait(v_full + (g & 1), (g >> 1) & 1, wctx, kChVFull);
        if (!last) mbar_wait(k_full + ((g + 1) & 1), ((g + 1) >> 1) & 1, wctx, kChKFull);
        mbar_wait(p_full, g & 1, wctx, kChPFull);
        tc_fence_after_sync();
        umma_ts_x4(tO, tS, 8u, bv, kIdescPV, (j > 0) ? 1u : 0u);
        if (!last) issue_qk(g + 1);
      }
      umma_commit_elect(o_full);
      g0 += n_kv;
      ++w;
      prev = it;
      k_loaded = nxt_k;
      it = nxt;
    }
    publish(it, true);
    store_o(prev, (w - 1) & 1);
  } else {
    // ============================ softmax / epilogue ================================
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr + kColS;
    const uint32_t tO = tmem_base + lane_addr + kColO;
    const float sl2 = a.scale_log2;
    float* mask_stage = reinterpret_cast<float*>(smem + L::kOffMask) + quad * TN;   // the warp's own copy of the step's mask in the log2 domain
    uint32_t g = 0, w = 0;
    int b, h, q0, k_limit;   // the item; b < 0: no more work
    auto fetch_item = [&](uint32_t n) {
      mbar_wait(item_full + (n & 1), (n >> 1) & 1, wctx, kChItem, 32);
      const uint4 x = lds128(ring + (n & 1) * 16);
      b = __shfl_sync(0xffffffffu, *abort_flag ? -1 : static_cast<int>(x.x), 0);
      h = static_cast<int>(x.y);
      q0 = static_cast<int>(x.z);
      k_limit = static_cast<int>(x.w);
    };
    fetch_item(0);
    while (b >= 0) {
      const DropRow drop_row = {a.philox_keys, philox_off, static_cast<uint32_t>(a.philox_bh_offset + b * a.H + h), static_cast<uint32_t>(q0 + row),
                                a.philox_thr};
      float m_ref = -INFINITY;
      float2 sum2 = make_float2(0.f, 0.f);   // running sum of exp2(t - m_ref), two interleaved partial sums
      for (int col0 = 0; col0 < k_limit; col0 += TN, ++g) {
        int kind = kMaskZero;
        if constexpr (KEYADD) {   // under the wait for the scores (each warp for itself)
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
        auto wait_s = [&]() { mbar_wait(s_full, g & 1, wctx, kChSFull, 32); };
        auto arrive = [&](int) {   // one arrival per warp
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full);
        };
        softmax_step_64<BF16, KEYADD, DROP>(tS, tO, col0, min(TN, k_limit - col0), sl2, mask_stage, kind, drop_row, m_ref, sum2, wait_s, arrive);
      }
      // ---- write-out ---------------------------------------------------------------------
      const uint4 y = lds128(ring + (w & 1) * 16);   // the item again, instead of in registers through the key steps
      mbar_wait(o_full, w & 1, wctx, kChOFull, 32);
      tc_fence_after_sync();
      const int q_row = static_cast<int>(y.z) + row;
      const float l_sum = sum2.x + sum2.y;
      if (a.lse != nullptr && q_row < a.S_q && *abort_flag == 0)
        a.lse[static_cast<size_t>(y.x * a.H + y.y) * a.S_q + q_row] = (m_ref + fast_log2(l_sum)) * kLn2F;
      o_tile_out<D, BF16>(tO, (DROP ? a.dropout_scale : 1.0f) / l_sum, sV, row, false, true, nullptr);
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(o_staged);
        mbar_arrive(item_empty + (w & 1));
      }
      ++w;
      fetch_item(w);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int k = 0; k < 20; ++k) __nanosleep(1000000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Where going on to a next tile is worth more than what it costs (state carried through the key steps, the next tile settled on
// before this one ends): few key steps, and enough rounds of resident CTAs that one badly placed tile does not decide.  Measured,
// this kernel / a CTA per tile: without dropout or mask S=48 0.80 to 0.94, 128 0.90 to 0.96, 256 0.93 to 1.00, 384 0.96 to 0.99 from three
// rounds on and 1.03 at 1.8, 449 1.01 to 1.05, 849 and 2048 1.02 to 1.06; additive mask S=64 0.77, 128 0.88 to 0.97, 384 0.96, 449 0.93 to
// 1.05; dropout S=128 0.90 to 0.98 from 2.3 rounds on and up to 1.04 below, 197 1.07 at 1.2 rounds and 0.94 at 5.5, 512 0.97 to 1.00, 849 and
// more 0.98 to 1.06; both, S=197 1.03 at 1.6 rounds and 0.94 to 0.99 from three on.  Between one and two rounds of five and six key steps with a mask
// it depends on the padding and on how the last tiles fall (300 and 384 keys, 1.0 to 2.0 rounds: 0.96 to 1.04 with lengths U[0.4 S, S], 0.96 to 1.07 with a mask that
// masks nothing, 0.95 to 1.00 with one that is nowhere zero).
bool fwd_chain_pays(int64_t sms, int64_t tiles, int64_t S_k, bool keyadd, bool dropout) {
  const int64_t round = kChCtasPerSm * sms;
  if (tiles <= round) return false;
  if (dropout) return S_k <= 640 && 2 * tiles >= (keyadd ? 6 : 5) * round;
  return S_k <= 384 && (keyadd || S_k <= 256 || tiles >= 3 * round);
}
// The same where it is known whether sequences may differ in length.  Without lengths, dropout or mask a second round that is nearly full of four whole key
// steps does not pay (S_k=256, 1.6 and 1.7 rounds 0.98 to 0.99, 1.8 to 2.0 rounds 1.03 to 1.045, 2.05 0.97; 1.8 to 2.0 rounds with lengths 0.95 to 0.98,
// S_k=240 0.98 to 1.00, 224 and 208 0.95 to 0.97, 192 1.00 to 1.01).
bool fwd_chain_pays(int64_t sms, int64_t tiles, int64_t S_k, bool keyadd, bool dropout, bool lengths) {
  const int64_t round = kChCtasPerSm * sms;
  if (!keyadd && !dropout && !lengths && S_k > 240 && 10 * tiles > 17 * round && tiles <= 2 * round) return false;
  return fwd_chain_pays(sms, tiles, S_k, keyadd, dropout);
}
bool fwd_chain_applies(const FwdArgs& a, int head_dim) {
  const int64_t tiles = static_cast<int64_t>((a.S_q + kTileM - 1) / kTileM) * a.H * a.B;
  return head_dim == D && a.mask_kind != FMHA_MASK_CU_SEQLENS &&
         fwd_chain_pays(sm_count(), tiles, a.S_k, a.mask_kind == FMHA_MASK_KEY_ADDITIVE, a.dropout_kind == FMHA_DROPOUT_PHILOX,
                        a.mask_kind == FMHA_MASK_SEQLEN);
}

template <bool BF16, bool KEYADD, bool DROP>
static int launch_chain_impl(const FwdArgs& a, cudaStream_t stream) {
  using L = ChainSmem;
  auto kfn = fmha_fwd_chain_kernel<BF16, KEYADD, DROP>;
  static std::atomic<bool> configured[64] = {};   // per device; set after the attribute call succeeded
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const dim3 grid((a.S_q + kTileM - 1) / kTileM, a.H, a.B);
  FwdArgs args = a;
  args.length_class_shift = fwd_length_class_shift(a, D, static_cast<int64_t>(grid.x) * grid.y * grid.z, KEYADD);
  const cudaError_t e = launch_overlapped(kfn, grid, dim3(kChThreads), L::kDynBytes, stream, args);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_fwd_chain(const FwdArgs& a, int dtype, cudaStream_t stream) {
  const bool bf = dtype == FMHA_DTYPE_BF16;
  const bool keyadd = a.mask_kind == FMHA_MASK_KEY_ADDITIVE;
  const bool drop = a.dropout_kind == FMHA_DROPOUT_PHILOX;
#define FMHA_CHAIN_CASE(BF, KA, DR) \
  if (bf == BF && keyadd == KA && drop == DR) return launch_chain_impl<BF, KA, DR>(a, stream);
  FMHA_CHAIN_CASE(false, false, false)
  FMHA_CHAIN_CASE(false, false, true)
  FMHA_CHAIN_CASE(false, true, false)
  FMHA_CHAIN_CASE(false, true, true)
  FMHA_CHAIN_CASE(true, false, false)
  FMHA_CHAIN_CASE(true, false, true)
  FMHA_CHAIN_CASE(true, true, false)
  FMHA_CHAIN_CASE(true, true, true)
#undef FMHA_CHAIN_CASE
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // namespace fmha
