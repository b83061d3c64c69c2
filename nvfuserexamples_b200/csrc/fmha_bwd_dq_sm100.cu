// fmha_bwd_dq_sm100.cu — dQ of the backward pass at head dimension 128, and the row term delta = rowsum(dO * O) that the
// dK / dV kernel (fmha_bwd_sm100.cu) reads afterwards.
//
// Why two kernels at D = 128.  One pass over the (key tile, query tile) pairs has to add every fp32 dQ tile (64 KB) to an
// accumulator in global memory: at the 5.4 TB/s this GPU's L2 takes reductions that alone is 3 400 cycles per tile and
// SM (measured), beside 2 560 cycles of MMAs, plus an accumulator to clear and to convert.  Forming S and dP twice (seven
// 128 x 128 x 128 products instead of five, 3 584 MMA cycles) needs no reduction at all, leaves each kernel room in
// tensor memory to run ahead, and makes dQ reproducible.  At D = 64 the exponentials, which would double, are the larger
// share and the single pass stays.
//
// One CTA per SM walks (128-row query tile, head, batch) items handed out by cluster launch control (a running CTA takes
// over the index of a CTA that has not been launched yet).  Per key tile: S = Q K^T, dP = dO V^T, dS = P (keep dP -
// delta/c) -> tensor memory over dP, dQ += dS K.  Tensor memory: S 128 | dP 128 | dQ 128 | Q 64 | dO 64 columns.  S of the
// next key tile (also of the next item) is formed while the current one is exponentiated, dP of it behind dQ of this one.
// Q and dO, the A operands of every S and dP of an item, are copied to tensor memory once: with both operands in shared
// memory a 128-column MMA takes all of its bandwidth, the loads of K and V (64 KB per tile) then cost S and dP half as much
// again, and a shared-memory read of another warp - a barrier poll, say - takes 330 cycles instead of 65 (measured).
//   warp 0: TMA producer (and the additive mask row)   warp 1: MMA issuer   warps 2-17: thread = query row x 32 keys
//   warps 18, 19: lse and delta of the item's rows, one item ahead
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <type_traits>

#include "../../include/fmha_sm100.h"
#include "fmha_device_utils.cuh"
#include "fmha_kernel_args.h"
#include "philox.cuh"
#include "sm100_ptx.cuh"

namespace fmha {

namespace {

constexpr int kDqCompute = 512;
constexpr int kDqStatWarp = 2 + kDqCompute / 32;      // the first of two
constexpr int kDqThreads = 64 + kDqCompute + 64;
constexpr uint32_t kDqSleepNs = 32;
constexpr int kDeltaPassKeys = 1024;   // up to here (in a grid larger than the chip) delta has a pass of its own, see launch_dq_impl
constexpr float kDqLog2e = 1.4426950408889634f;

enum DqWaitSite {
  kDqsQ = 231, kDqsQEmpty = 232, kDqsDo = 233, kDqsDoEmpty = 234, kDqsK = 235, kDqsKEmpty = 236, kDqsV = 237, kDqsVEmpty = 238,
  kDqsS = 239, kDqsSFree = 240, kDqsDp = 241, kDqsDs = 242, kDqsOut = 243, kDqsStat = 244, kDqsStatEmpty = 245, kDqsMask = 246,
  kDqsItem = 247, kDqsItemEmpty = 248
};

struct DqSmem {
  static constexpr int D = 128;
  static constexpr int kTile = kTileM * D * 2;        // 32 KB
  static constexpr int kKStages = 3;                  // K is read by S (a tile ahead) and by dQ, V by dP only
  static constexpr int kOffQ = 0;
  static constexpr int kOffdO = kOffQ + kTile;
  static constexpr int kOffK = kOffdO + kTile;
  static constexpr int kOffV = kOffK + kKStages * kTile;
  static constexpr int kOffStage = kOffV + kTile;     // dQ on its way out: 1 KB per compute warp
  static constexpr int kOffStats = kOffStage + 16384; // 2 slots x (128 of -lse*log2e, 128 of delta/c)
  static constexpr int kOffMask = kOffStats + 2 * 2 * kTileM * 4;   // additive mask (log2 domain) of a K stage
  static constexpr int kOffItems = kOffMask + kKStages * kTileN * 4;
  static constexpr int kOffBar = kOffItems + 32;
  static constexpr int kNumBars = 4 + 3 * kKStages + 2 + 2 + 1 + 1 + 1 + 4 + 4;
  static constexpr int kOffMisc = kOffBar + kNumBars * 8;
  static constexpr int kDynBytes = kOffMisc + 16;   // 1024-byte aligned base: checked by the kernel
  static_assert(kDynBytes <= 232448, "shared memory budget of one CTA exceeded");
};

// The product of two rows of 128 values that 16 lanes hold, 16 bytes each; in every one of the lanes.
template <bool BF16>
__device__ __forceinline__ float row_dot16(const uint4& o, const uint4& d) {
  const uint32_t xo[4] = {o.x, o.y, o.z, o.w}, xd[4] = {d.x, d.y, d.z, d.w};
  float sum = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    sum = fmaf(unpack_lo<BF16>(xo[e]), unpack_lo<BF16>(xd[e]), sum);
    sum = fmaf(unpack_hi<BF16>(xo[e]), unpack_hi<BF16>(xd[e]), sum);
  }
#pragma unroll
  for (int m = 1; m < 16; m *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, m);
  return sum;
}

enum DqItemState { kDqEnd, kDqEmpty, kDqWork };
struct DqItem {
  int state;
  int b, h, bh, q0;
  int n_kv, k_limit, q_limit;   // key tiles, keys [0, k_limit) and query rows [0, q_limit) of this (b, h)
  int row_base, tb;             // packed batch: first row of the sequence; batch coordinate of the tensor maps
};

}  // namespace

template <bool BF16, bool KEYADD, bool DROP, bool PACKED>
__global__ void __launch_bounds__(kDqThreads, 1) fmha_bwd_dq_kernel(const __grid_constant__ BwdArgs a) {
  griddep_wait();
  using L = DqSmem;
  constexpr int D = 128;
  constexpr int KS = L::kKStages;
  constexpr int kTmemCols = 512;
  constexpr uint32_t kColS = 0, kColdP = 128, kColdQ = 256, kColQ = 384, kColdO = 448;
  constexpr int kFmt = BF16 ? 1 : 0;
  constexpr uint32_t kIdescKK = make_idesc_f16(128, 128, kFmt, false, false);
  constexpr uint32_t kIdescKN = make_idesc_f16(128, D, kFmt, false, true);

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem + L::kOffQ;
  uint8_t* sdO = smem + L::kOffdO;
  uint8_t* sK = smem + L::kOffK;
  uint8_t* sV = smem + L::kOffV;
  float* sStats = reinterpret_cast<float*>(smem + L::kOffStats);
  float* sMask = reinterpret_cast<float*>(smem + L::kOffMask);
  uint4* items = reinterpret_cast<uint4*>(smem + L::kOffItems);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* q_full = bars + 0;
  uint64_t* q_empty = bars + 1;     // Q has been copied to tensor memory
  uint64_t* do_full = bars + 2;
  uint64_t* do_empty = bars + 3;    // dO has been copied to tensor memory
  uint64_t* k_full = bars + 4;      // [KS]
  uint64_t* k_empty = k_full + KS;  // [KS] dQ += dS K of the tile has completed
  uint64_t* mask_full = k_empty + KS;   // [KS]
  uint64_t* v_full = mask_full + KS;
  uint64_t* v_empty = v_full + 1;   // dP of the tile has completed
  uint64_t* s_full = v_empty + 1;
  uint64_t* s_free = s_full + 1;    // S has been read (all compute threads)
  uint64_t* dp_full = s_free + 1;
  uint64_t* ds_full = dp_full + 1;  // dS is in tensor memory, dP has been read (all compute threads)
  uint64_t* dq_full = ds_full + 1;  // dQ of an item is complete
  uint64_t* stat_full = dq_full + 1;    // [2] by item parity
  uint64_t* stat_empty = stat_full + 2; // [2]
  uint64_t* item_full = stat_empty + 2; // [2]
  uint64_t* item_empty = item_full + 2; // [2]
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 4);
  volatile uint32_t* philox_off = reinterpret_cast<volatile uint32_t*>(smem + L::kOffMisc + 8);

  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0 && a.status != nullptr) atomicCAS(a.status, 0, kDqsItem);
    return;
  }
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitCtx wctx{abort_flag, a.status};
  constexpr bool packed = PACKED;
  const bool persist = a.persist != 0;   // the grid is larger than the number of SMs

  auto decode = [&](int x, int y, int z) {
    DqItem it;
    it.h = y;
    it.b = z;
    it.bh = z * a.H + y;
    it.q0 = x * kTileM;
    it.k_limit = a.S_k;
    it.q_limit = a.S_q;
    it.row_base = 0;
    it.tb = z;
    if (!packed && a.mask_kind == FMHA_MASK_SEQLEN) {
      const int len = reinterpret_cast<const int*>(a.mask)[z];
      if (len > 0 && len < a.S_k) it.k_limit = len;
    } else if (packed) {
      const int* cu = reinterpret_cast<const int*>(a.mask);
      it.row_base = cu[z];
      it.k_limit = it.q_limit = packed_rows(it.row_base, cu[z + 1], a.S_q, a.total_rows);
      it.tb = 0;
    }
    it.n_kv = (it.k_limit + kTileN - 1) / kTileN;
    it.state = it.q0 < it.q_limit ? kDqWork : kDqEmpty;
    return it;
  };
  // Asks for the index of one more CTA of the grid (item number n of this CTA), written to slot n & 1.
  auto request_item = [&](int n) {
    const int slot = n & 1;
    if (n >= 3) mbar_wait(item_empty + slot, ((n - 3) >> 1) & 1, wctx, kDqsItemEmpty);
    mbar_arrive_expect_tx(item_full + slot, 16);
    clc_try_cancel(items + slot, item_full + slot);
  };
  // Item number n (whole warp; n >= 1).  Only the producer asks, the others tell it that they have read the slot.
  auto fetch_item = [&](int n, bool producer) {
    const int slot = n & 1;
    mbar_wait(item_full + slot, ((n - 1) >> 1) & 1, wctx, kDqsItem, producer ? 0 : kDqSleepNs);
    int x, y, z;
    const bool have = clc_query(items + slot, x, y, z) && *abort_flag == 0;
    fence_proxy_async_smem();   // the slot's next content is written by the async proxy
    __syncwarp();
    if (!producer && lane == 0) mbar_arrive(item_empty + slot);
    DqItem it;
    it.state = kDqEnd;
    if (have) it = decode(x, y, z);
    return it;
  };
  // The next item with work after item number n (which is advanced).
  auto next_work = [&](int& n, bool producer) {
    DqItem it;
    it.state = kDqEnd;
    if (!persist) return it;
    while (true) {
      it = fetch_item(++n, producer);
      if (it.state != kDqEmpty) return it;
      if (producer) {
        if (lane == 0) request_item(n + 1);
        __syncwarp();
      }
    }
  };
  auto first_work = [&](int& n, bool producer) {
    DqItem it = decode(blockIdx.x, blockIdx.y, blockIdx.z);
    if (packed && it.state == kDqEmpty) {
      if (producer && persist) {
        if (lane == 0) request_item(1);
        __syncwarp();
      }
      it = next_work(n, producer);
    }
    return it;
  };

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *philox_off = a.philox_offset + (a.philox_offset_dev != nullptr ? static_cast<uint32_t>(*a.philox_offset_dev) : 0u);
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    for (int s = 0; s < KS; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(k_empty + s, 1);
      mbar_init(mask_full + s, 1);
    }
    mbar_init(v_full, 1);
    mbar_init(v_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(s_free, kDqCompute);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, kDqCompute);
    mbar_init(dq_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(stat_full + s, 2);
      mbar_init(stat_empty + s, kDqCompute / 32);
      mbar_init(item_full + s, 1);
      mbar_init(item_empty + s, 1 + kDqCompute / 32 + 2);   // MMA warp, compute warps, statistics warps
    }
    mbar_fence_init();
    tma_prefetch_desc(&a.tm_q);
    tma_prefetch_desc(&a.tm_k);
    tma_prefetch_desc(&a.tm_v);
    tma_prefetch_desc(&a.tm_do);
    tma_prefetch_desc(&a.tm_dq);
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
    // ============================ TMA producer ======================================
    int n = 0, w = 0, g = 0;   // item number, items with work and key tiles so far
    for (DqItem it = first_work(n, true); it.state == kDqWork; it = next_work(n, true), ++w) {
      for (int j = 0; j < it.n_kv; ++j, ++g) {
        const int s = g % KS;
        if (lane == 0) {
          if (j == 0) {
            if (w > 0) mbar_wait(q_empty, (w - 1) & 1, wctx, kDqsQEmpty);
            mbar_arrive_expect_tx(q_full, L::kTile);
            for (int c = 0; c < 2; ++c) tma_load_4d(sQ + c * 16384, &a.tm_q, q_full, c * 64, it.row_base + it.q0, it.h, it.tb);
          }
          if (g >= KS) mbar_wait(k_empty + s, (g / KS - 1) & 1, wctx, kDqsKEmpty);
          mbar_arrive_expect_tx(k_full + s, L::kTile);
          for (int c = 0; c < 2; ++c)
            tma_load_4d(sK + s * L::kTile + c * 16384, &a.tm_k, k_full + s, c * 64, it.row_base + j * kTileN, it.h, it.tb);
          if (j == 0) {
            if (w > 0) mbar_wait(do_empty, (w - 1) & 1, wctx, kDqsDoEmpty);
            mbar_arrive_expect_tx(do_full, L::kTile);
            for (int c = 0; c < 2; ++c) tma_load_4d(sdO + c * 16384, &a.tm_do, do_full, c * 64, it.row_base + it.q0, it.h, it.tb);
          }
          if (g >= 1) mbar_wait(v_empty, (g - 1) & 1, wctx, kDqsVEmpty);
          mbar_arrive_expect_tx(v_full, L::kTile);
          for (int c = 0; c < 2; ++c) tma_load_4d(sV + c * 16384, &a.tm_v, v_full, c * 64, it.row_base + j * kTileN, it.h, it.tb);
          // Early, for the statistics warps need the next item's rows in time; but the first time not at once: on a chip
          // that is still filling up, the CTA asked for may be about to start on an idle SM.
          if (persist && j == (w == 0 ? min(2, it.n_kv - 1) : 0)) request_item(n + 1);
        }
        __syncwarp();
        if constexpr (KEYADD) {   // the slot is free: its K stage was
          const float* mask = reinterpret_cast<const float*>(a.mask) + static_cast<size_t>(it.b) * a.S_k;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int c = j * kTileN + k * 32 + lane;
            sMask[s * kTileN + k * 32 + lane] = c < a.S_k ? mask[c] * kDqLog2e : 0.f;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(mask_full + s);
        }
      }
    }
  } else if (warp == 1) {
    // ============================ MMA issuer ========================================
    // Convergent warp, bursts from one elected lane (see umma_ss_x4).  Per tile t: S(t+1) as soon as S(t) has been read; then,
    // with dS(t) there, dQ(t) and dP(t+1), which overwrites dS(t): the tensor core works in order.  Every wait is for
    // something that needs an MMA issued after the previous wait on the same barrier, so no barrier can be a phase ahead
    // of this warp.
    const uint32_t tS = tmem_base + kColS, tdP = tmem_base + kColdP, tdQ = tmem_base + kColdQ, tQ = tmem_base + kColQ,
                   tdO = tmem_base + kColdO;
    // Q or dO of an item to tensor memory; the copy is ordered behind the previous item's last use of these columns and
    // before the MMAs issued after it.
    auto copy_a = [&](uint32_t dst, const uint8_t* tile, uint64_t* full, uint64_t* empty, int w, int site) {
      mbar_wait(full, w & 1, wctx, site);
      tc_fence_after_sync();
      const uint64_t d = make_smem_desc_sw128(smem_u32(tile), 16, 1024);
      uint64_t x[8];
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) x[kk] = d + kmajor_step(kk, 16384);
      tmem_cp_128x256b_x8(dst, x);
      umma_commit_elect(empty);
    };
    // [128 x 128] = A (tensor memory) * (rows of a K or V tile)^T
    auto issue_kk = [&](uint32_t d, uint32_t a_tmem, const uint8_t* b_tile) {
      const uint64_t db = make_smem_desc_sw128(smem_u32(b_tile), 16, 1024);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint64_t y[4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) y[kk] = db + kmajor_step(hf * 4 + kk, 16384);
        umma_ts_x4(d, a_tmem + hf * 32, 8u, y, kIdescKK, hf);
      }
    };
    // S and dP of key tile number t of this CTA; `first` of its item number w (with work)
    auto issue_s = [&](int t, int w, bool first) {
      if (first) copy_a(tQ, sQ, q_full, q_empty, w, kDqsQ);
      mbar_wait(k_full + t % KS, (t / KS) & 1, wctx, kDqsK);
      tc_fence_after_sync();
      issue_kk(tS, tQ, sK + (t % KS) * L::kTile);
      umma_commit_elect(s_full);
    };
    auto issue_dp = [&](int t, int w, bool first) {
      if (first) copy_a(tdO, sdO, do_full, do_empty, w, kDqsDo);
      mbar_wait(v_full, t & 1, wctx, kDqsV);
      tc_fence_after_sync();
      issue_kk(tdP, tdO, sV);
      umma_commit_elect(dp_full);
      umma_commit_elect(v_empty);
    };
    int n = 0, w = 0, t = 0;
    DqItem it = first_work(n, false);
    if (it.state == kDqWork) {
      issue_s(0, 0, true);
      issue_dp(0, 0, true);
    }
    while (it.state == kDqWork) {
      DqItem nxt = it;
      for (int j = 0; j < it.n_kv; ++j, ++t) {
        const bool last = j + 1 == it.n_kv;
        if (last) nxt = next_work(n, false);
        const bool more = !last || nxt.state == kDqWork;
        if (more) {
          mbar_wait(s_free, t & 1, wctx, kDqsSFree);
          issue_s(t + 1, w + 1, last);
        }
        mbar_wait(ds_full, t & 1, wctx, kDqsDs);
        tc_fence_after_sync();
        const uint64_t dk = make_smem_desc_sw128(smem_u32(sK + (t % KS) * L::kTile), 16384, 1024);   // K as MN-major B
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint64_t y[4];
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) y[kk] = dk + mnmajor_step(hf * 4 + kk);
          umma_ts_2x2(tdQ, tdP + hf * 64, tdP + hf * 64 + 32, 8u, y, kIdescKN, (j > 0 || hf > 0) ? 1u : 0u);
        }
        umma_commit_elect(k_empty + t % KS);
        if (last) umma_commit_elect(dq_full);
        if (more) issue_dp(t + 1, w + 1, last);
      }
      ++w;
      it = nxt;
    }
  } else if (warp >= kDqStatWarp) {
    // ============================ row statistics =====================================
    // lse and delta of the item's rows [64*half, +64), one item ahead; delta is also written for the dK / dV kernel.
    const int half = warp - kDqStatWarp;
    const float inv_c = DROP ? 1.0f / a.dropout_scale : 1.0f;
    const int part = lane & 15;       // 16-byte piece of a row; a warp instruction covers two rows
    auto side_jobs = [&](const DqItem& x) {   // for every item of the grid, whether it has work or not
      if (x.state == kDqEnd) return;
      if (x.bh == 0 && x.q0 == 0 && half == 0 && lane == 0) *a.work_counter = 0;   // the dK / dV kernel draws its items from it
      if (packed && a.zero.grad[0].ptr != nullptr && (x.q0 + kTileM > x.q_limit || x.q_limit == a.S_q)) {
        for (int k = 0; k < 3; ++k)
          zero_uncovered_rows(a.zero.grad[k].ptr, a.zero.grad[k].stride_s, a.zero.grad[k].stride_h, x.h, x.b, a.B,
                              reinterpret_cast<const int*>(a.mask), a.S_q, a.total_rows, D, x.q0, x.q0 + kTileM,
                              a.zero.mode == kUncoveredAll, half * 32 + lane, 64);
      }
    };
    int n = 0, w = 0;
    DqItem it = decode(blockIdx.x, blockIdx.y, blockIdx.z);
    while (it.state != kDqEnd) {
      side_jobs(it);
      if (it.state == kDqWork) {
        const int slot = w & 1;
        float* st = sStats + slot * 2 * kTileM;
        const float* lse = a.lse + (packed ? static_cast<int64_t>(it.h) * a.total_rows + it.row_base : static_cast<int64_t>(it.bh) * a.S_q);
        float* delta = a.delta + static_cast<int64_t>(it.bh) * a.S_q;
        const int64_t b_o = packed ? static_cast<int64_t>(it.row_base) * a.o_ss : static_cast<int64_t>(it.b) * a.o_sb;
        const int64_t b_do = packed ? static_cast<int64_t>(it.row_base) * a.do_ss : static_cast<int64_t>(it.b) * a.do_sb;
        const unsigned short* po = static_cast<const unsigned short*>(a.o_ptr) + b_o + it.h * a.o_sh + part * 8;
        const unsigned short* pd = static_cast<const unsigned short*>(a.do_ptr) + b_do + it.h * a.do_sh + part * 8;
        if (w >= 2) mbar_wait(stat_empty + slot, ((w >> 1) - 1) & 1, wctx, kDqsStatEmpty);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int r = half * 64 + k * 32 + lane, q = it.q0 + r;
          st[r] = q < it.q_limit ? -lse[q] * kDqLog2e : -INFINITY;   // rows past the end: their probabilities are zero
        }
        if (!persist) {
          // the compute warps form delta
        } else if (a.o_ptr == nullptr) {   // delta is there already (bwd_delta_kernel)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int r = half * 64 + k * 32 + lane, q = it.q0 + r;
            st[kTileM + r] = q < it.q_limit ? delta[q] * inv_c : 0.f;
          }
        } else
        for (int r0 = half * 64; r0 < half * 64 + 64; r0 += 16) {
          uint4 wo[8], wd[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int64_t q = it.q0 + r0 + 2 * k + (lane >> 4);
            wo[k] = wd[k] = make_uint4(0u, 0u, 0u, 0u);
            if (q < it.q_limit) {
              wo[k] = __ldg(reinterpret_cast<const uint4*>(po + q * a.o_ss));
              wd[k] = __ldg(reinterpret_cast<const uint4*>(pd + q * a.do_ss));
            }
          }
          float v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint32_t xo[4] = {wo[k].x, wo[k].y, wo[k].z, wo[k].w}, xd[4] = {wd[k].x, wd[k].y, wd[k].z, wd[k].w};
            v[k] = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              v[k] = fmaf(unpack_lo<BF16>(xo[e]), unpack_lo<BF16>(xd[e]), v[k]);
              v[k] = fmaf(unpack_hi<BF16>(xo[e]), unpack_hi<BF16>(xd[e]), v[k]);
            }
          }
          // Eight sums over 16 lanes: in each of three steps a lane keeps half of its values and gets the partner's other
          // half; `idx` ends as the value it has kept.  (One sum after the other, four shuffles deep each, took 2 000
          // cycles per batch and made items of few key tiles wait for their statistics.)
          int idx = 0;
#pragma unroll
          for (int m = 8, cnt = 4; m >= 2; m /= 2, cnt /= 2) {
            const bool up = part & m;
            idx = idx * 2 + (up ? 1 : 0);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (k < cnt) {
                const float send = up ? v[k] : v[k + cnt], own = up ? v[k + cnt] : v[k];
                v[k] = own + __shfl_xor_sync(0xffffffffu, send, m);
              }
          }
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
          const int r = r0 + 2 * idx + (lane >> 4);
          if ((part & 1) == 0) {
            st[kTileM + r] = v[0] * inv_c;
            if (it.q0 + r < it.q_limit) delta[it.q0 + r] = v[0];
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(stat_full + slot);
        ++w;
      }
      if (!persist) break;
      it = fetch_item(++n, false);
    }
  } else {
    // ============================ compute warps =====================================
    const int cw = warp - 2;             // 0..15
    const int quad = warp & 3;           // tensor-memory lane quarter of this warp
    const int cq = cw >> 2;              // its 32 keys of every tile
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const float sl2 = a.scale_log2;
    const float out_mul = a.scale * (DROP ? a.dropout_scale : 1.0f);   // dS carries no dropout factor, dQ gets it here
    uint8_t* stage = smem + L::kOffStage + cw * 1024;

    // dQ of a finished item: tensor memory -> registers -> staging tile (32 rows x 16 columns) -> TMA store, twice.
    auto store_dq = [&](int wi, const DqItem& x) {
      mbar_wait(dq_full, wi & 1, wctx, kDqsOut, kDqSleepNs);
      tc_fence_after_sync();
      // packed batch: rows of a slice that reaches past the end of the sequence are written one by one
      const bool edge = packed && (x.q0 + quad * 32 + 32 > x.q_limit);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[16];
        tmem_ld16(tmem_base + lane_addr + kColdQ + cq * 32 + c * 16, r);
        tmem_wait_ld();
        if (lane == 0) tma_store_wait_read();
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint4 v;
          v.x = pack2<BF16>(__uint_as_float(r[q * 8 + 0]) * out_mul, __uint_as_float(r[q * 8 + 1]) * out_mul);
          v.y = pack2<BF16>(__uint_as_float(r[q * 8 + 2]) * out_mul, __uint_as_float(r[q * 8 + 3]) * out_mul);
          v.z = pack2<BF16>(__uint_as_float(r[q * 8 + 4]) * out_mul, __uint_as_float(r[q * 8 + 5]) * out_mul);
          v.w = pack2<BF16>(__uint_as_float(r[q * 8 + 6]) * out_mul, __uint_as_float(r[q * 8 + 7]) * out_mul);
          if (edge) {
            unsigned short* out = static_cast<unsigned short*>(a.dq_ptr) + static_cast<int64_t>(x.row_base + x.q0 + row) * a.dq_ss +
                                  static_cast<int64_t>(x.h) * a.dq_sh + cq * 32 + c * 16 + q * 8;
            if (x.q0 + row < x.q_limit) *reinterpret_cast<uint4*>(out) = v;
          } else {
            sts128(smem_u32(stage) + lane * 32 + q * 16, v.x, v.y, v.z, v.w);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && *abort_flag == 0 && !edge) {
          tma_store_4d(&a.tm_dq, stage, cq * 32 + c * 16, x.row_base + x.q0 + quad * 32, x.h, x.tb);
          tma_store_commit();
        }
      }
      tc_fence_before_sync();
    };

    int n = 0, w = 0, t = 0;
    DqItem prev;
    prev.state = kDqEnd;
    DqItem it = first_work(n, false);
    if (!persist && it.state == kDqWork) {
      // The CTA's only item: its delta while Q, K, dO and V are on their way, eight rows per warp, 16 lanes per row.  A pass of its
      // own is on the critical path of so small a grid, and so are the two statistics warps (B=1 H=12 S=128, forward and backward,
      // 22.0 -> 20.7 us; B=1 H=8 S=2048 95.7 -> 87.5).
      const int64_t b_o = packed ? static_cast<int64_t>(it.row_base) * a.o_ss : static_cast<int64_t>(it.b) * a.o_sb;
      const int64_t b_do = packed ? static_cast<int64_t>(it.row_base) * a.do_ss : static_cast<int64_t>(it.b) * a.do_sb;
      const unsigned short* po = static_cast<const unsigned short*>(a.o_ptr) + b_o + it.h * a.o_sh + (lane & 15) * 8;
      const unsigned short* pd = static_cast<const unsigned short*>(a.do_ptr) + b_do + it.h * a.do_sh + (lane & 15) * 8;
      uint4 wo[4], wd[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t q = it.q0 + cw * 8 + 2 * k + (lane >> 4);
        wo[k] = wd[k] = make_uint4(0u, 0u, 0u, 0u);
        if (q < it.q_limit) {
          wo[k] = __ldg(reinterpret_cast<const uint4*>(po + q * a.o_ss));
          wd[k] = __ldg(reinterpret_cast<const uint4*>(pd + q * a.do_ss));
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float sum = row_dot16<BF16>(wo[k], wd[k]);
        const int r = cw * 8 + 2 * k + (lane >> 4);
        if ((lane & 15) == 0) {
          sStats[kTileM + r] = sum * (DROP ? 1.0f / a.dropout_scale : 1.0f);
          if (it.q0 + r < it.q_limit) a.delta[static_cast<int64_t>(it.bh) * a.S_q + it.q0 + r] = sum;
        }
      }
      named_bar_sync(1, kDqCompute);
    }
    while (it.state == kDqWork) {
      const uint32_t gbh = static_cast<uint32_t>(a.philox_bh_offset + it.bh);
      mbar_wait(stat_full + (w & 1), (w >> 1) & 1, wctx, kDqsStat, kDqSleepNs);
      const float neg_lse2 = sStats[(w & 1) * 2 * kTileM + row];
      const float neg_delta = -sStats[(w & 1) * 2 * kTileM + kTileM + row];
      __syncwarp();
      if (lane == 0) mbar_arrive(stat_empty + (w & 1));
      for (int j = 0; j < it.n_kv; ++j, ++t) {
        const int n_cols = min(32, it.k_limit - j * kTileN - cq * 32);   // valid keys among this thread's 32
        [[maybe_unused]] uint32_t kw[8];
        if constexpr (DROP) {
          const uint32_t poff = *philox_off;
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            const U4 u = dropout_draw_keys(a.philox_keys, poff, gbh, static_cast<uint32_t>(it.q0 + row),
                                           static_cast<uint32_t>((j * kTileN + cq * 32) / 16 + d));
            kw[d * 4 + 0] = (u.x & 0x7F7F7F7Fu) + (0x80u - a.philox_thr) * 0x01010101u;
            kw[d * 4 + 1] = (u.y & 0x7F7F7F7Fu) + (0x80u - a.philox_thr) * 0x01010101u;
            kw[d * 4 + 2] = (u.z & 0x7F7F7F7Fu) + (0x80u - a.philox_thr) * 0x01010101u;
            kw[d * 4 + 3] = (u.w & 0x7F7F7F7Fu) + (0x80u - a.philox_thr) * 0x01010101u;
          }
        }
        const int ks = t % KS;
        if constexpr (KEYADD) mbar_wait(mask_full + ks, (t / KS) & 1, wctx, kDqsMask, kDqSleepNs);
        mbar_wait(s_full, t & 1, wctx, kDqsS, kDqSleepNs);
        tc_fence_after_sync();
        uint32_t p[32];
        tmem_ld32(tmem_base + lane_addr + kColS + cq * 32, p);
        tmem_wait_ld_dep(p);
        tc_fence_before_sync();
        mbar_arrive(s_free);
        const float2 sl22 = make_float2(sl2, sl2);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          float2 x = make_float2(neg_lse2, neg_lse2);
          if constexpr (KEYADD) x = __fadd2_rn(x, *reinterpret_cast<const float2*>(sMask + ks * kTileN + cq * 32 + 2 * k));
          x = __ffma2_rn(make_float2(__uint_as_float(p[2 * k]), __uint_as_float(p[2 * k + 1])), sl22, x);
          p[2 * k] = __float_as_uint(fast_exp2(x.x));
          p[2 * k + 1] = __float_as_uint(fast_exp2(x.y));
        }
        if (n_cols < 32) {
#pragma unroll
          for (int k = 0; k < 32; ++k)
            if (k >= n_cols) p[k] = 0u;
        }
        if (j == 0 && prev.state == kDqWork) {   // before this thread's dS lets the tensor core overwrite the previous dQ
          store_dq(w - 1, prev);
          prev.state = kDqEnd;
        }
        mbar_wait(dp_full, t & 1, wctx, kDqsDp, kDqSleepNs);
        tc_fence_after_sync();
        const float2 nd2 = make_float2(neg_delta, neg_delta);
        uint32_t pk[16];
        uint32_t dp[32];
        tmem_ld32(tmem_base + lane_addr + kColdP + cq * 32, dp);
        tmem_wait_ld_dep(dp);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          if constexpr (DROP) {
            const uint32_t word = kw[k >> 1];
            dp[2 * k] &= prmt(word, 0u, (k & 1) ? 0xAAAAu : 0x8888u);
            dp[2 * k + 1] &= prmt(word, 0u, (k & 1) ? 0xBBBBu : 0x9999u);
          }
          const float2 d = __fadd2_rn(make_float2(__uint_as_float(dp[2 * k]), __uint_as_float(dp[2 * k + 1])), nd2);
          const float2 ds = __fmul2_rn(make_float2(__uint_as_float(p[2 * k]), __uint_as_float(p[2 * k + 1])), d);
          pk[k] = pack2<BF16>(ds.x, ds.y);
        }
        tmem_st16(tmem_base + lane_addr + kColdP + cq * 32, pk);   // over this thread's own columns of dP
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(ds_full);
      }
      prev = it;
      ++w;
      it = next_work(n, false);
    }
    if (prev.state == kDqWork) store_dq(w - 1, prev);
    if (lane == 0) tma_store_wait_read();   // shared memory stays valid until the TMA unit has read it
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

// delta alone, in a pass of its own: 16 lanes per row, four rows per lane.
template <bool BF16>
__global__ void __launch_bounds__(256) bwd_delta_kernel(const __grid_constant__ BwdArgs a) {
  griddep_wait();
  const int bh = blockIdx.x, h = bh % a.H, b = bh / a.H;
  const int part = threadIdx.x & 15;
  int q_limit = a.S_q;
  int64_t base_o = static_cast<int64_t>(b) * a.o_sb, base_do = static_cast<int64_t>(b) * a.do_sb;
  if (a.mask_kind == FMHA_MASK_CU_SEQLENS) {
    const int* cu = static_cast<const int*>(a.mask);
    q_limit = packed_rows(cu[b], cu[b + 1], a.S_q, a.total_rows);
    base_o = static_cast<int64_t>(cu[b]) * a.o_ss;
    base_do = static_cast<int64_t>(cu[b]) * a.do_ss;
  }
  const unsigned short* po = static_cast<const unsigned short*>(a.o_ptr) + base_o + h * a.o_sh + part * 8;
  const unsigned short* pd = static_cast<const unsigned short*>(a.do_ptr) + base_do + h * a.do_sh + part * 8;
  uint4 wo[4], wd[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t q = blockIdx.y * 64 + k * 16 + (threadIdx.x >> 4);
    wo[k] = wd[k] = make_uint4(0u, 0u, 0u, 0u);
    if (q < q_limit) {
      wo[k] = __ldg(reinterpret_cast<const uint4*>(po + q * a.o_ss));
      wd[k] = __ldg(reinterpret_cast<const uint4*>(pd + q * a.do_ss));
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float sum = row_dot16<BF16>(wo[k], wd[k]);
    const int q = blockIdx.y * 64 + k * 16 + (threadIdx.x >> 4);
    if (part == 0 && q < q_limit) a.delta[static_cast<int64_t>(bh) * a.S_q + q] = sum;
  }
}

template <bool BF16, bool KEYADD, bool DROP, bool PACKED>
static int launch_dq_impl(const BwdArgs& a, cudaStream_t stream) {
  auto kfn = fmha_bwd_dq_kernel<BF16, KEYADD, DROP, PACKED>;
  static std::atomic<bool> configured[64] = {};   // per device; set after the attribute call succeeded
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, DqSmem::kDynBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const dim3 grid((a.S_q + kTileM - 1) / kTileM, a.H, a.B);
  BwdArgs args = a;
  // The two statistics warps need 12 000 cycles for an item's delta, five key tiles' worth: with fewer tiles the compute
  // warps wait (9 600 cycles per item at four), and a separate pass over O and dO is the cheaper way (B=16 H=16 S=512 with
  // dropout: 162 us for the whole backward fused, 158 separate; from S_k = 2048 on it is hidden).  In between the line hardly
  // matters: forward and backward fused / separate, 768 keys 276.6 / 280.1, with lengths 247.6 / 249.3, 1024 keys 310 / 315, with
  // dropout 364.5 / 368.6, 1280 keys 404.8 / 409.6, 487.7 / 495.0 with dropout, where runs of one side differ by up to 4 %.
  args.persist = static_cast<int64_t>(grid.x) * grid.y * grid.z > sm_count();
  if (args.persist && a.S_k <= kDeltaPassKeys) {
    const cudaError_t e = launch_overlapped(bwd_delta_kernel<BF16>, dim3(static_cast<unsigned>(a.B) * a.H, (a.S_q + 63) / 64), dim3(256), 0,
                                            stream, a);
    if (e != cudaSuccess) return static_cast<int>(e);
    args.o_ptr = nullptr;
  }
  const cudaError_t e = launch_overlapped(kfn, grid, dim3(kDqThreads), DqSmem::kDynBytes, stream, args);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_bwd_dq(const BwdArgs& a, int dtype, cudaStream_t stream) {
  const bool bf = dtype == FMHA_DTYPE_BF16;
  const bool keyadd = a.mask_kind == FMHA_MASK_KEY_ADDITIVE;
  const bool drop = a.dropout_kind == FMHA_DROPOUT_PHILOX;
  const bool packed = a.mask_kind == FMHA_MASK_CU_SEQLENS;
#define FMHA_DQ_CASE(BF, KA, DR, PK) \
  if (bf == BF && keyadd == KA && drop == DR && packed == PK) return launch_dq_impl<BF, KA, DR, PK>(a, stream);
#define FMHA_DQ_CASES(BF, DR) FMHA_DQ_CASE(BF, false, DR, false) FMHA_DQ_CASE(BF, true, DR, false) FMHA_DQ_CASE(BF, false, DR, true)
  FMHA_DQ_CASES(false, false)
  FMHA_DQ_CASES(false, true)
  FMHA_DQ_CASES(true, false)
  FMHA_DQ_CASES(true, true)
#undef FMHA_DQ_CASES
#undef FMHA_DQ_CASE
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // namespace fmha
