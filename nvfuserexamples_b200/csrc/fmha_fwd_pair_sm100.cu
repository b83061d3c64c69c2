// fmha_fwd_pair_sm100.cu — forward kernel of head dimension 128 for grids that fill the chip (fwd_pair_pays): compact masks (none, valid lengths,
// additive [B,S_k] row, packed batch), no dropout, O and the row logsumexp.
//
// A CTA, one per SM, works on TWO 128-row query tiles of a head at once, which share the K and V tiles it loads, and goes on to the
// next pair (handed out by cluster launch control) without a gap: the producer loads the next pair's Q, K and V under this pair's
// last steps.  Twelve warps: TMA producer, an MMA issuer per tile, a warp for the additive mask, four softmax warps (thread = query
// row) per tile.  Tensor memory: S 2 x 128 columns (P over S), O 2 x 128.
//
// What bounds it: per key step and tile the tensor core needs 1 024 cycles and the exponentials another 1 024 (16 results per clock
// and SM), one after the other within a tile, so the two tiles have to take turns at both.  Left alone they fall into step, both at
// the exponentials and then both at the tensor core: two tiles in step take 5 200 cycles per key step, two independent CTAs per SM
// with a tile each (fmha_fwd_fast_sm100.cu) 4 400, and with the turns enforced by barriers (`turn`) 3 300 (B=16 H=16 S=2048 without
// a mask: 605 us, 519, 475).  What is left of a step is a chain of 1 350 cycles of exponentials, 1 000 for P V and Q K^T of the tile,
// 480 for the row maximum; at that rate the clock gives way to power (1.7 GHz): a quarter of the exponentials as a polynomial on the
// FMA pipe shortened the chain by 5 %, and the time not at all.
//
// Measured, two tiles / one tile per CTA: B=16 H=16 S=1024 additive mask 137 / 174 us, lengths U[S/2,S] 109 / 125, S=512 42.6 / 49.3,
// B=32 H=16 S=2048 lengths 735 / 832, B=4 102 / 116.  With dropout the draws of one tile would have to fit beside the other's
// exponentials on the same pipes: B=4 H=16 S=2048 195 / 173 with turns, 225 / 173 without: left to the other kernel.
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

constexpr int kPairThreads = 384;
constexpr int kItemSlots = 4;

enum PairWaitSite {
  kPrQFull = 171, kPrQEmpty = 172, kPrKvFull = 173, kPrKvEmpty = 174, kPrSFull = 175, kPrPFull = 176, kPrOFull = 177,
  kPrMaskFull = 178, kPrMaskEmpty = 179, kPrItem = 180, kPrItemEmpty = 181, kPrClc = 182, kPrSmemBase = 183, kPrTurn = 184
};

constexpr int D = 128;
struct PairSmem {
  static constexpr int TN = 128;         // keys per step
  static constexpr int kSlots = 4;       // K and V tiles take turns in one ring
  static constexpr int kPFirst = 3;      // 32-column chunks of P that go to the tensor core ahead of the rest
  // Registers per thread: at launch (65 536 over 384 threads), then of the control and of the softmax warps.
  static constexpr int kRegsLaunch = 168, kRegsControl = 72, kRegsSoftmax = 216;
  static_assert(128 * kRegsControl + 256 * kRegsSoftmax <= kPairThreads * kRegsLaunch, "a larger sum would wait forever");
  static constexpr int kTile = 128 * D * 2;            // a Q, K or V tile
  static constexpr int kSub = 128 * 128;               // one 64-column sub-tile of it
  static constexpr int kOffQ = 0;                      // 2 tiles
  static constexpr int kOffO = kOffQ + 2 * kTile;      // staging of O on its way out: 32 rows x 64 columns per softmax warp
  static constexpr int kOffKv = kOffO + 8 * 4096;
  static constexpr int kOffMask = kOffKv + kSlots * kTile;     // 2 x TN floats
  static constexpr int kOffItems = kOffMask + 2 * TN * 4;      // kItemSlots x 32 bytes
  static constexpr int kOffClc = kOffItems + kItemSlots * 32;
  static constexpr int kOffBar = kOffClc + 16;
  static constexpr int kNumBars = 2 * kSlots + 2 + 2 + 2 + 4 + 2 + 2 + 2 + 2 * kItemSlots + 1 + 8;
  static constexpr int kOffMisc = kOffBar + kNumBars * 8;      // tensor-memory base, abort flag, 2 mask kinds
  static constexpr int kDynBytes = kOffMisc + 16;              // 1024-byte aligned base: checked by the kernel
  static_assert(kDynBytes <= 232448, "shared memory budget exceeded");
};

struct PairItem {
  int tiles;   // < 0: no more work; 0: no query row (packed batch); else 1 or 2 query tiles
  int b, h, q0;
  int k_limit, q_limit;   // keys [0, k_limit) and query rows [0, q_limit) of this (b, h)
  int row_base;           // packed batch: first row of the sequence in the [total_rows, H, D] tensors
};

// Position in a ring of N slots.
template <int N>
struct RingPos {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++slot == N) {
      slot = 0;
      phase ^= 1u;
    }
  }
};

}  // namespace

// O of a warp's 32 query rows out of tensor memory, scaled and rounded, to global memory in whole 128-byte pieces of rows, by
// way of 4 KB of shared memory of the warp's own: 2 330 cycles beside the other tile's steps.  (A tile store per 64 columns, with
// the group barriers and the wait for its source that it needs, took 2 630; 16-byte stores of each lane's own row 3 700.)
template <bool BF16>
__device__ __forceinline__ void o_warp_out(uint32_t tO, float out_scale, uint32_t stage, unsigned short* rows, int64_t stride, int n_rows,
                                           int lane) {
#pragma unroll
  for (int c = 0; c < D / 64; ++c) {
    uint32_t r[2][32];
    tmem_ld32(tO + c * 64, r[0]);
    tmem_ld32(tO + c * 64 + 32, r[1]);
    tmem_wait_ld_dep(r[0]);
    tmem_wait_ld_dep(r[1]);
    auto v = [&](int k) { return __uint_as_float(r[k / 32][k % 32]) * out_scale; };
    if (c > 0) __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q)
      sts128(stage + sw128_offset(lane, q), pack2<BF16>(v(q * 8), v(q * 8 + 1)), pack2<BF16>(v(q * 8 + 2), v(q * 8 + 3)),
             pack2<BF16>(v(q * 8 + 4), v(q * 8 + 5)), pack2<BF16>(v(q * 8 + 6), v(q * 8 + 7)));
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = i * 4 + (lane >> 3), ch = lane & 7;
      const uint4 w = lds128(stage + sw128_offset(row, ch));
      if (row < n_rows) *reinterpret_cast<uint4*>(rows + row * stride + c * 64 + ch * 8) = w;
    }
  }
}

template <bool BF16, bool KEYADD, bool PACKED>
__global__ void __launch_bounds__(kPairThreads, 1) fmha_fwd_pair_kernel(const __grid_constant__ FwdArgs a) {
  griddep_wait();
  using L = PairSmem;
  constexpr int TN = L::TN, NS = L::kSlots, PF = L::kPFirst;
  constexpr int kTmemCols = 2 * (TN + D);
  constexpr uint32_t kColS = 0, kColO = 2 * TN;   // + tile * TN, + tile * D
  constexpr int kFmt = BF16 ? 1 : 0;
  constexpr uint32_t kIdescQK = make_idesc_f16(128, TN, kFmt, false, false);
  constexpr uint32_t kIdescPV = make_idesc_f16(128, D, kFmt, false, true);

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem + L::kOffQ;
  uint8_t* sO = smem + L::kOffO;
  uint8_t* sKv = smem + L::kOffKv;
  float* sMask = reinterpret_cast<float*>(smem + L::kOffMask);
  uint4* clc_answer = reinterpret_cast<uint4*>(smem + L::kOffClc);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* kv_full = bars;                // [NS]
  uint64_t* kv_empty = kv_full + NS;       // [NS] one arrival per tile
  uint64_t* q_full = kv_empty + NS;        // [2] by tile, as all below
  uint64_t* q_empty = q_full + 2;          // [2] the item's last Q K^T has completed
  uint64_t* s_full = q_empty + 2;          // [2]
  uint64_t* p_full = s_full + 2;           // [2][2] a part of P is in tensor memory, S has been read (one arrival per warp)
  uint64_t* o_full = p_full + 4;      // [2]
  uint64_t* mask_full = o_full + 2;        // [2] by parity of the key step
  uint64_t* mask_empty = mask_full + 2;    // [2]
  uint64_t* item_full = mask_empty + 2;    // [kItemSlots]
  uint64_t* item_empty = item_full + kItemSlots;
  uint64_t* clc_full = item_empty + kItemSlots;
  uint64_t* turn = clc_full + 1;           // [2][4] by tile and quarter: the other tile's warp has done its exponentials
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 4);
  volatile int* mask_kind = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 8);    // [2]

  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0 && a.status != nullptr) atomicCAS(a.status, 0, kPrSmemBase);
    return;
  }
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitCtx wctx{abort_flag, a.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full + i, 1);
      mbar_init(q_empty + i, 1);
      mbar_init(s_full + i, 1);
      mbar_init(p_full + i * 2, 4);
      mbar_init(p_full + i * 2 + 1, 4);
      mbar_init(o_full + i, 1);
      mbar_init(mask_full + i, 1);
      mbar_init(mask_empty + i, 8);
    }
    for (int i = 0; i < NS; ++i) {
      mbar_init(kv_full + i, 1);
      mbar_init(kv_empty + i, 2);
    }
    for (int i = 0; i < kItemSlots; ++i) {
      mbar_init(item_full + i, 1);
      mbar_init(item_empty + i, KEYADD ? 11 : 10);   // MMA warps, mask warp, softmax warps
    }
    mbar_init(clc_full, 1);
    for (int i = 0; i < 8; ++i) mbar_init(turn + i, 1);
    mbar_fence_init();
    tma_prefetch_desc(&a.tm_q);
    tma_prefetch_desc(&a.tm_k);
    tma_prefetch_desc(&a.tm_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_base_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_base_slot;

  // Item number n from the ring (whole warp); the slot is given back by item_done.
  const uint32_t ring = smem_u32(smem + L::kOffItems);
  auto read_item = [&](int n) {
    const int slot = n % kItemSlots;
    const uint4 x = lds128(ring + slot * 32), y = lds128(ring + slot * 32 + 16);
    PairItem it;
    it.tiles = static_cast<int>(x.x);
    it.b = static_cast<int>(x.y);
    it.h = static_cast<int>(x.z);
    it.q0 = static_cast<int>(x.w);
    it.k_limit = static_cast<int>(y.x);
    it.q_limit = static_cast<int>(y.y);
    it.row_base = static_cast<int>(y.z);
    return it;
  };
  auto fetch_item = [&](int n, uint32_t sleep_ns) {
    mbar_wait(item_full + n % kItemSlots, (n / kItemSlots) & 1, wctx, kPrItem, sleep_ns);
    PairItem it = read_item(n);
    it.tiles = __shfl_sync(0xffffffffu, *abort_flag ? -1 : it.tiles, 0);
    return it;
  };
  auto item_done = [&](int n) {
    __syncwarp();
    if (lane == 0) mbar_arrive(item_empty + n % kItemSlots);
  };

  if (warp < 4) {
  regs_release<L::kRegsControl>();
  if (warp == 0) {
    // ============================ TMA producer (whole warp, lane 0 issues) ===========
    auto decode = [&](int x, int y, int z) {
      PairItem it;
      int b = z;
      if constexpr (!KEYADD) {
        if (a.length_class_shift >= 0) {
          const int* len = reinterpret_cast<const int*>(a.mask);
          int n = 0;
          if (lane < a.B) n = PACKED ? len[lane + 1] - len[lane] : len[lane];
          if (n > a.S_k || (!PACKED && n <= 0)) n = a.S_k;
          b = batch_of_rank(z, a.B, static_cast<uint32_t>(max(n - 1, 0)) >> a.length_class_shift);
        }
      }
      it.b = b;
      it.h = y;
      it.q0 = x * 2 * kTileM;
      it.k_limit = a.S_k;
      it.q_limit = a.S_q;
      it.row_base = 0;
      if (!PACKED && a.mask_kind == FMHA_MASK_SEQLEN) {
        const int len = reinterpret_cast<const int*>(a.mask)[b];
        if (len > 0 && len < a.S_k) it.k_limit = len;
      } else if (PACKED) {
        const int* cu = reinterpret_cast<const int*>(a.mask);
        it.row_base = cu[b];
        it.k_limit = it.row_base < 0 ? 0 : min(cu[b + 1] - it.row_base, a.S_q);   // a sequence longer than the stated maximum is cut there
        it.q_limit = min(it.k_limit, a.total_rows - it.row_base);   // offsets past the tensor, which the host cannot see: no row behind it
      }
      const int rows = it.q_limit - it.q0;
      it.tiles = rows <= 0 ? 0 : rows <= kTileM ? 1 : 2;
      return it;
    };
    RingPos<NS> kv;
    uint32_t kv_used = 0;     // slots filled so far, up to NS
    int n = 0, w = 0, w1 = 0;   // items, items with work, with two tiles so far
    uint32_t clc_phase = 0;
    PairItem it = decode(blockIdx.x, blockIdx.y, blockIdx.z);
    auto load_tile = [&](const void* tmap, int row, int h, int tb) {   // lane 0
      if (kv_used >= NS) mbar_wait(kv_empty + kv.slot, kv.phase ^ 1u, wctx, kPrKvEmpty);
      mbar_arrive_expect_tx(kv_full + kv.slot, L::kTile);
#pragma unroll
      for (int c = 0; c < D / 64; ++c)
        tma_load_4d(sKv + kv.slot * L::kTile + c * L::kSub, tmap, kv_full + kv.slot, c * 64, row, h, tb);
      kv.next();
      ++kv_used;
    };
    while (true) {
      const int slot = n % kItemSlots;
      if (lane == 0) {
        if (n >= kItemSlots) mbar_wait(item_empty + slot, (n / kItemSlots - 1) & 1, wctx, kPrItemEmpty);
        sts128(ring + slot * 32, static_cast<uint32_t>(it.tiles), static_cast<uint32_t>(it.b), static_cast<uint32_t>(it.h),
               static_cast<uint32_t>(it.q0));
        sts128(ring + slot * 32 + 16, static_cast<uint32_t>(it.k_limit), static_cast<uint32_t>(it.q_limit),
               static_cast<uint32_t>(it.row_base), 0u);
        mbar_arrive(item_full + slot);
      }
      __syncwarp();
      if (it.tiles < 0) break;
      ++n;
      if (it.tiles > 0) {
        const int tb = PACKED ? 0 : it.b;
        const int n_kv = (it.k_limit + TN - 1) / TN;
        for (int j = 0; j < n_kv && lane == 0; ++j) {
          load_tile(&a.tm_k, it.row_base + j * TN, it.h, tb);
          load_tile(&a.tm_v, it.row_base + j * TN, it.h, tb);
          if (j == 0) {   // the buffers come free with the last Q K^T of the item before
            for (int g = 0; g < it.tiles; ++g) {
              const int wg = g == 0 ? w : w1;
              if (wg > 0) mbar_wait(q_empty + g, (wg - 1) & 1, wctx, kPrQEmpty);
              mbar_arrive_expect_tx(q_full + g, L::kTile);
#pragma unroll
              for (int c = 0; c < D / 64; ++c)
                tma_load_4d(sQ + g * L::kTile + c * 16384, &a.tm_q, q_full + g, c * 64, it.row_base + it.q0 + g * kTileM, it.h, tb);
            }
          }
        }
        __syncwarp();
        w1 += it.tiles - 1;
        ++w;
      }
      // The next item.  Not asked for before this CTA's first product has been formed: on a chip that is still filling up, the
      // CTA that would be taken over may be about to start on an idle SM.
      it.tiles = -1;
      if (a.persist) {
        if (lane == 0) {
          if (w == 1 && kv_used <= NS) mbar_wait(kv_empty, 0, wctx, kPrKvEmpty);   // (else a slot has been waited for)
          mbar_arrive_expect_tx(clc_full, 16);
          clc_try_cancel(clc_answer, clc_full);
        }
        __syncwarp();
        mbar_wait(clc_full, clc_phase, wctx, kPrClc);
        clc_phase ^= 1u;
        int x, y, z;
        const bool have = clc_query(clc_answer, x, y, z) && *abort_flag == 0;
        fence_proxy_async_smem();   // the answer's place is written by the async proxy again
        if (__all_sync(0xffffffffu, have)) it = decode(x, y, z);
      }
    }
  } else if (warp <= 2) {
    // ============================ MMA issuers, one warp per tile ======================
    // Whole warp, bursts from one elected lane (see umma_ss_x4).  When P(j) is there, P V(j) and Q K^T(j+1) go out back to back;
    // what they need is waited for before P is.  The tensor core works in order, so Q K^T(j+1) may overwrite P(j), and the first
    // P V of an item the O of the one before, which has been read when the first P arrives.
    constexpr int KQ = D / 16, KP = TN / 16;   // k-steps of S = Q K^T and of O += P V
    const int g = warp - 1;
    const uint32_t tS = tmem_base + kColS + g * TN, tO = tmem_base + kColO + g * D;
    const uint64_t dq = make_smem_desc_sw128(smem_u32(sQ + g * L::kTile), 16, 1024);
    auto issue_qk = [&](int slot, bool last) {
      const uint64_t dk = make_smem_desc_sw128(smem_u32(sKv + slot * L::kTile), 16, 1024);
      uint64_t x[KQ], y[KQ];
#pragma unroll
      for (int kk = 0; kk < KQ; ++kk) {
        x[kk] = dq + kmajor_step(kk, 16384);
        y[kk] = dk + kmajor_step(kk, L::kSub);
      }
      umma_ss_x8(tS, x, y, kIdescQK, 0u);
      umma_commit_elect(s_full + g);
      if (last) umma_commit_elect(q_empty + g);
      umma_commit_elect(kv_empty + slot);
    };
    RingPos<NS> kv;
    uint32_t p_par = 0u;
    int w = 0;
    for (int n = 0;; ++n) {
      const PairItem it = fetch_item(n, 0);
      item_done(n);
      if (it.tiles < 0) break;
      if (it.tiles == 0) continue;
      const int n_kv = (it.k_limit + TN - 1) / TN;
      if (g >= it.tiles) {   // no such tile: only keep the ring going
        for (int i = 0; i < 2 * n_kv; ++i, kv.next()) {
          mbar_wait(kv_full + kv.slot, kv.phase, wctx, kPrKvFull, 200);
          __syncwarp();
          if (lane == 0) mbar_arrive(kv_empty + kv.slot);
        }
        continue;
      }
      mbar_wait(kv_full + kv.slot, kv.phase, wctx, kPrKvFull);
      mbar_wait(q_full + g, w & 1, wctx, kPrQFull);
      tc_fence_after_sync();
      issue_qk(kv.slot, n_kv == 1);
      for (int j = 0; j < n_kv; ++j) {
        kv.next();   // V(j)
        RingPos<NS> nk = kv;
        nk.next();   // K(j+1)
        const bool more = j + 1 < n_kv;
        const uint64_t dv = make_smem_desc_sw128(smem_u32(sKv + kv.slot * L::kTile), L::kSub, 1024);
        mbar_wait(kv_full + kv.slot, kv.phase, wctx, kPrKvFull);
        if (more) mbar_wait(kv_full + nk.slot, nk.phase, wctx, kPrKvFull);
        uint64_t y[KP];
#pragma unroll
        for (int kk = 0; kk < KP; ++kk) y[kk] = dv + mnmajor_step(kk);
        mbar_wait(p_full + g * 2, p_par, wctx, kPrPFull);
        tc_fence_after_sync();
        umma_ts<0, PF * 2>(tO, tS, y, kIdescPV, (j > 0) ? 1u : 0u);
        mbar_wait(p_full + g * 2 + 1, p_par, wctx, kPrPFull);
        tc_fence_after_sync();
        umma_ts<PF * 2, KP>(tO, tS, y, kIdescPV, 1u);
        p_par ^= 1u;
        if (more) issue_qk(nk.slot, j + 2 == n_kv);
        else umma_commit_elect(o_full + g);
        umma_commit_elect(kv_empty + kv.slot);
        kv = nk;
      }
      ++w;
    }
  } else if constexpr (KEYADD) {
    // ============================ additive mask, in the log2 domain ====================
    int t = 0;
    for (int n = 0;; ++n) {
      const PairItem it = fetch_item(n, 0);
      item_done(n);
      if (it.tiles < 0) break;
      const float* mask = reinterpret_cast<const float*>(a.mask) + static_cast<size_t>(it.b) * a.S_k;
      for (int k0 = 0; k0 < it.k_limit; k0 += TN, ++t) {
        const int s = t & 1;
        float mk[TN / 32];
        bool exists[TN / 32];
#pragma unroll
        for (int i = 0; i < TN / 32; ++i) {
          const int c = k0 + i * 32 + lane;
          exists[i] = c < a.S_k;
          mk[i] = exists[i] ? mask[c] * kLog2eF : 0.f;
        }
        const int kind = mask_step_kind(mk, exists);
        if (t >= 2) mbar_wait(mask_empty + s, ((t >> 1) - 1) & 1, wctx, kPrMaskEmpty);
#pragma unroll
        for (int i = 0; i < TN / 32; ++i) sMask[s * TN + i * 32 + lane] = mk[i];
        if (lane == 0) mask_kind[s] = kind;
        __syncwarp();
        if (lane == 0) mbar_arrive(mask_full + s);
      }
    }
  }
  } else {
    // ============================ softmax / epilogue ================================
    regs_take<L::kRegsSoftmax>();
    const int g = (warp - 4) >> 2;       // which tile of the pair
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr + kColS + g * TN;
    const uint32_t tO = tmem_base + lane_addr + kColO + g * D;
    const float sl2 = a.scale_log2;
    uint32_t s_par = 0, o_par = 0, turn_par = g == 0 ? 1u : 0u;   // tile 0 begins
    const DropRow no_drop = {a.philox_keys, nullptr, 0u, 0u, 0u};
    [[maybe_unused]] int t = 0;   // key steps (of both tiles' items) so far
    for (int n = 0;; ++n) {
      PairItem it = fetch_item(n, 32);
      if (it.tiles < 0) break;
      int q_row = it.q0 + g * kTileM + row;
      if (g < it.tiles) {
        const int n_kv = (it.k_limit + TN - 1) / TN;
        float m_ref = -INFINITY;
        float2 sum2 = make_float2(0.f, 0.f);   // running sum of exp2(t - m_ref), two interleaved partial sums
        auto wait_s = [&]() { mbar_wait(s_full + g, s_par, wctx, kPrSFull, 32); };
        auto arrive_p = [&](int part) {
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full + g * 2 + part);
        };
        // Turns at the exponentials: warp `quad` of the one tile and of the other, which share a scheduler and its special-function
        // unit.
        const bool turns = it.tiles == 2;
        auto turn_begin = [&]() {
          if (turns) {
            mbar_wait(turn + g * 4 + quad, turn_par, wctx, kPrTurn);
            turn_par ^= 1u;
          }
        };
        auto turn_end = [&]() {
          if (turns && lane == 0) mbar_arrive(turn + (g ^ 1) * 4 + quad);
        };
        for (int j = 0; j < n_kv; ++j) {
          const float* mask_stage = sMask + (t & 1) * TN;
          int kind = kMaskZero;
          if constexpr (KEYADD) {
            mbar_wait(mask_full + (t & 1), (t >> 1) & 1, wctx, kPrMaskFull, 32);
            kind = __shfl_sync(0xffffffffu, mask_kind[t & 1], 0);
          }
          softmax_step_128<BF16, KEYADD, false, PF>(tS, tO, j * TN, min(TN, it.k_limit - j * TN), sl2, mask_stage, kind, no_drop, m_ref,
                                                      sum2, wait_s, arrive_p, turn_begin, turn_end);
          s_par ^= 1u;
          if constexpr (KEYADD) {
            if (lane == 0) mbar_arrive(mask_empty + (t & 1));
            ++t;
          }
        }
        // ---- write-out ---------------------------------------------------------------------
        mbar_wait(o_full + g, o_par, wctx, kPrOFull, 32);
        o_par ^= 1u;
        tc_fence_after_sync();
        it = read_item(n);   // again, instead of in registers through the key steps
        q_row = it.q0 + g * kTileM + row;
        // After a given-up wait tensor memory holds anything; and the item is this one only if none had been given up when it was read.
        if (!__any_sync(0xffffffffu, *abort_flag != 0)) {
          const bool row_ok = q_row < it.q_limit;
          const float l_sum = sum2.x + sum2.y;
          if (a.lse != nullptr && row_ok) {
            const size_t li = PACKED ? static_cast<size_t>(it.h) * a.total_rows + it.row_base + q_row   // [H, total_rows]
                                     : static_cast<size_t>(it.b * a.H + it.h) * a.S_q + q_row;          // [B*H, S_q]
            a.lse[li] = (m_ref + fast_log2(l_sum)) * kLn2F;
          }
          unsigned short* o_rows = reinterpret_cast<unsigned short*>(a.o_ptr) + static_cast<int64_t>(it.h) * a.o_sh +
                                   (PACKED ? 0 : it.b * a.o_sb) + static_cast<int64_t>(it.row_base + it.q0 + g * kTileM + quad * 32) * a.o_ss;
          o_warp_out<BF16>(tO, 1.0f / l_sum, smem_u32(sO) + (warp - 4) * 4096, o_rows, a.o_ss,
                           it.q_limit - (it.q0 + g * kTileM + quad * 32), lane);
        }
        tc_fence_before_sync();
      } else if constexpr (KEYADD) {   // the other tile has work, this one does not exist: only keep the mask ring going
        for (int k0 = 0; k0 < it.k_limit; k0 += TN, ++t) {
          mbar_wait(mask_full + (t & 1), (t >> 1) & 1, wctx, kPrMaskFull, 1000);
          __syncwarp();
          if (lane == 0) mbar_arrive(mask_empty + (t & 1));
        }
      }
      if constexpr (PACKED) {
        if (a.zero_uncovered) {
          const int* cu = reinterpret_cast<const int*>(a.mask);
          const int q0 = it.q0 + g * kTileM;
          if (q0 < a.S_q && (q0 + kTileM > it.q_limit || cu[it.b + 1] - it.row_base > it.q_limit))
            zero_uncovered_rows(a.o_ptr, a.o_ss, a.o_sh, it.h, it.b, a.B, cu, a.S_q, a.total_rows, D, q0, q0 + kTileM,
                                a.zero_uncovered == kUncoveredAll, row, 128);
        }
      }
      item_done(n);
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

// No dropout, three or more key steps, and grids of at least two query tiles per SM, one round of the other kernel's capacity:
// at one or two steps a CTA's life is its start and its end (S_q=256: S_k=128 12.8 / 12.2 us, S_k=256 16.2 / 16.0, S_k=1024 39.0 /
// 40.2).  A head with an odd number of tiles leaves half a CTA idle for one item, which takes nearly as long as a whole one: the
// rounds of pairs over the SMs may be at most 8/7 of the rounds of tiles (H=16: S=384 B=16 34.4 / 33.0 us at 4/3, S=640 68.2 / 69.3 at
// 6/5, B=8 S=1152 94.1 / 90.1 at 5/4).  Of three tiles a third is lost, more than the rounds show: one tile per CTA (S=384 H=4
// B=50 1.06, with lengths U[S/2, S] 1.20, H=12 B=9 1.11 times its time in pairs).
// One round: where each pair has an SM of its own and single tiles would have to share some, and all are of one length of 1 024 keys or more
// (S=1024 H=12 B=2 20.9 us one tile per CTA / 20.3, S=2048 36.8 / 34.6, S=2565 46.7 / 44.2; an additive mask, S=1536 H=16 37.3 / 32.2; with
// lengths U[0.3 S, S] S=1024 19.3 / 20.3).
// Packed batch: only total_rows tells how full it is.  A sequence below the maximum leaves the other kernel with CTAs that start for
// nothing (B=64 H=16, maximum 512, 102 rows each: 36.4 us in pairs / 48.9), so two tiles per CTA stay the choice for most of them, except on
// small grids: with no more than 1.2 tiles of the average length per SM, pairing takes from the tiles the SM of their own (H=8
// B=10, maximum 512, 153 rows each: 10.7 / 9.7; H=4 B=6, 2048, 165 rows: 10.2 / 9.2), and just above two tiles per SM by the maximum the rounds count
// that the average length makes (H=8 B=10, 512, 307 rows: 160 pairs take two rounds, 240 tiles one, 18.0 / 11.9).
bool fwd_pair_pays(int64_t sms, int64_t B, int64_t H, int64_t S_q, int64_t S_k, bool lengths, int64_t packed_rows) {
  if (sms <= 0 || S_k <= 256) return false;   // no multiprocessors: the query for their number has failed
  const int64_t heads = B * H;
  auto tiles = [](int64_t rows) { return (rows + kTileM - 1) / kTileM; };
  auto even_rounds = [&](int64_t n) {
    const int64_t pair_rounds = (heads * ((n + 1) / 2) + sms - 1) / sms, tile_rounds = (heads * n + 2 * sms - 1) / (2 * sms);
    return 7 * pair_rounds <= 8 * tile_rounds;
  };
  const int64_t n = tiles(S_q);
  if (n == 3) return false;
  if (!lengths && S_k >= 1024 && heads * n > sms && heads * ((n + 1) / 2) <= sms) return true;
  if (heads * n < 2 * sms || !even_rounds(n)) return false;
  if (packed_rows > 0) {
    const int64_t n_avg = tiles(std::min(S_q, (packed_rows + B - 1) / B));
    if (heads * n <= 3 * sms && 5 * heads * n_avg <= 6 * sms) return false;
    if (10 * heads * n <= 23 * sms && !even_rounds(n_avg)) return false;
  }
  return true;
}
bool fwd_pair_applies(const FwdArgs& a, int head_dim) {
  if (head_dim != D || a.dropout_kind == FMHA_DROPOUT_PHILOX) return false;
  const bool packed = a.mask_kind == FMHA_MASK_CU_SEQLENS;
  return fwd_pair_pays(sm_count(), a.B, a.H, a.S_q, a.S_k, packed || a.mask_kind == FMHA_MASK_SEQLEN, packed ? a.total_rows : 0);
}

template <bool BF16, bool KEYADD, bool PACKED>
static int launch_pair_impl(const FwdArgs& a, cudaStream_t stream) {
  using L = PairSmem;
  auto kfn = fmha_fwd_pair_kernel<BF16, KEYADD, PACKED>;
  static std::atomic<bool> configured[64] = {};   // per device; set after the attribute call succeeded
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaFuncAttributes attr;   // the register split waits for what the launch does not bring along
    if ((e = cudaFuncGetAttributes(&attr, kfn)) != cudaSuccess) return static_cast<int>(e);
    if (attr.numRegs < L::kRegsLaunch) return static_cast<int>(cudaErrorInvalidConfiguration);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const dim3 grid((a.S_q + 2 * kTileM - 1) / (2 * kTileM), a.H, a.B);
  const int64_t items = static_cast<int64_t>(grid.x) * grid.y * grid.z;
  FwdArgs args = a;
  args.persist = items > sm_count();
  args.length_class_shift = -1;
  if (args.persist && (a.mask_kind == FMHA_MASK_SEQLEN || a.mask_kind == FMHA_MASK_CU_SEQLENS) && a.B >= 2 && a.B <= kMaxOrdered) {
    args.length_class_shift = 0;
    while ((a.S_k - 1) >> args.length_class_shift > 7) ++args.length_class_shift;
  }
  const cudaError_t e = launch_overlapped(kfn, grid, dim3(kPairThreads), L::kDynBytes, stream, args);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_fwd_pair(const FwdArgs& a, int dtype, cudaStream_t stream) {
  const bool bf = dtype == FMHA_DTYPE_BF16;
  const bool packed = a.mask_kind == FMHA_MASK_CU_SEQLENS;
  const bool keyadd = a.mask_kind == FMHA_MASK_KEY_ADDITIVE;
#define FMHA_PAIR_CASE(BF, KA, PK) \
  if (bf == BF && keyadd == KA && packed == PK) return launch_pair_impl<BF, KA, PK>(a, stream);
  FMHA_PAIR_CASE(false, false, false)
  FMHA_PAIR_CASE(false, true, false)
  FMHA_PAIR_CASE(false, false, true)
  FMHA_PAIR_CASE(true, false, false)
  FMHA_PAIR_CASE(true, true, false)
  FMHA_PAIR_CASE(true, false, true)
#undef FMHA_PAIR_CASE
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // namespace fmha
