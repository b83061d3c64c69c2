// fmha_bwd_sm100.cu — fused multi-head-attention backward for B200 (sm_100a).
//
// The reference project has no backward pass (shmsong/NvFuserExamples README.md:1); its
// provision for one is the pair of S x S tensors saved by FMHATrainKernelSaveIntermediate
// (fmha/fmha_manual.cpp:891-897).  This backward needs neither: it recomputes the
// probabilities from Q, K and the per-row logsumexp the forward kernel wrote.
//
// Head dimension 64, three kernels per call (one where there is a single key tile, see ONE_KV):
//   1. bwd_prepare : delta[row] = sum_d dO[row,d] * O[row,d], and zero the fp32 dQ accumulator
//   2. bwd_main    : persistent CTAs (one per SM) draw (128-key tile, head, batch) work items from a
//                    counter and loop over the 128-row query tiles of each
//                      S^T = K Q^T           dP^T = V dO^T            (tcgen05.mma, fp32 in TMEM)
//                      P  = exp2(S*scale*log2e + mask - lse*log2e)   (16 warps, thread = key, a quarter of the queries)
//                      dS = P * (keep*dP - delta/c)                   c = 1/(1-p_drop)
//                      dV += (keep*P)^T dO     dK += dS^T Q     dQ_tile = dS K
//                    P^T goes to tensor memory as the A operand of dV, dS^T there as that of dK and to shared memory (16-bit,
//                    128-byte swizzle) as the MN-major operand of dQ; dQ tiles are added to
//                    the fp32 accumulator from registers; dK and dV leave through per-warp staging tiles and TMA stores
//                    when the next item is already under way.
//   3. bwd_finish  : dQ = (scale * accumulator) rounded to the 16-bit dtype
// Head dimension 128: the kernel in fmha_bwd_dq_sm100.cu writes dQ and delta, then bwd_main as above without dQ (dS^T stays
// in tensor memory).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include <cstring>
#include <type_traits>

#include "../../include/fmha_sm100.h"
#include "fmha_device_utils.cuh"
#include "fmha_kernel_args.h"
#include "philox.cuh"
#include "sm100_ptx.cuh"

namespace fmha {

namespace {

#ifndef FMHA_BWD_POLL_SLEEP_NS
#define FMHA_BWD_POLL_SLEEP_NS 48
#endif
constexpr uint32_t kComputeSleepNs = FMHA_BWD_POLL_SLEEP_NS;  // pause between barrier polls of the compute warps
constexpr int kComputeThreads = 512;               // 16 compute warps
constexpr int kBwdStatWarp = 2 + kComputeThreads / 32;   // the warp that fetches lse and delta (ONE_KV: lse)
constexpr int kBwdThreads = 64 + kComputeThreads + 32;   // + producer warp + MMA warp + statistics warp
constexpr float kLog2eB = 1.4426950408889634f;

enum BwdWaitSite {
  kSiteKFull = 201, kSiteQFull = 202, kSiteQEmpty = 203, kSiteSFull = 204, kSitePFull = 205, kSiteDqFull = 206,
  kSiteDqFree = 207, kSiteAccFull = 208, kSiteDpFull = 209, kSiteKEmpty = 210, kSiteItemFull = 211, kSiteItemEmpty = 212,
  kSiteDoFull = 213, kSiteDoEmpty = 214, kSiteDsFull = 215, kSiteStatFull = 216, kSiteStatEmpty = 217, kSiteSmemBase = 218,
  kSiteVFull = 219, kSiteVEmpty = 220
};

template <int D>
struct BwdSmem {
  // Two stages of Q and of dO.  D = 64: two K/V buffers (the next work item's K and V arrive while this one finishes) and
  // two dS buffers.  D = 128: one K/V buffer, read for the last time a tile before the item ends, and no dS buffers.
  static constexpr int kKvBufs = (D == 64) ? 2 : 1;
  static constexpr int kQStages = 2;
  static constexpr int kDoStages = 2;
  static constexpr int kDsBufs = (D == 64) ? 2 : 0;
  static constexpr int kTileBytes = kTileM * D * 2;
  static constexpr int kDsBytes = kTileM * kTileN * 2;
  static constexpr int kOffK = 0;
  static constexpr int kOffV = kOffK + kKvBufs * kTileBytes;
  static constexpr int kOffQ = kOffV + kKvBufs * kTileBytes;
  static constexpr int kOffdO = kOffQ + kQStages * kTileBytes;
  static constexpr int kOffdS = kOffdO + kDoStages * kTileBytes;
  // Staging of dK and dV on their way out, 2 KB per compute warp.
  static constexpr int kOffStage = kOffdS + kDsBufs * kDsBytes;
  static constexpr int kOffStats = kOffStage + 32768;         // 2 slots x (128 of -lse*log2e, 128 of delta/c)
  static constexpr int kOffBar = kOffStats + 2 * 2 * kTileM * 4;
  static constexpr int kNumBars = 7 + 4 * kKvBufs + 2 * kQStages + 2 * kDoStages + 8;
  static constexpr int kOffRing = (kOffBar + kNumBars * 8 + 15) / 16 * 16;   // 2 work items of 32 bytes
  static constexpr int kOffRec = kOffRing + 64;   // two 16-byte item records per compute warp
  static constexpr int kOffMisc = kOffRec + 512;
  static constexpr int kBytes = kOffMisc + 16;
  // The tiles need a 1024-byte aligned base.  Dynamic shared memory of a kernel without static shared memory begins at
  // such an address; the kernel checks it and gives up if that should ever not hold.
  static constexpr int kDynBytes = kBytes;
  static_assert(kDynBytes <= 232448, "shared memory budget of one CTA exceeded");
};

}  // namespace

// ---------------------------------------------------------------------------------------
// 1. delta and accumulator clearing
// ---------------------------------------------------------------------------------------
constexpr int kAccumD = 64;   // the head dimension whose dQ goes through the fp32 accumulator
struct PrepArgs {
  const void* o;
  const void* d_o;
  int64_t o_sb, o_sh, o_ss, do_sb, do_sh, do_ss;
  BwdArgs m;   // the main kernel's arguments
};

// Transposes the 32 x 32 bit matrix a warp holds as one row per lane: afterwards bit L of lane p is what bit p of lane L
// was.  Five exchanges of half-blocks: 16 and 8 bits as byte permutes, 4, 2 and 1 as a rotation and a bit select.
__device__ __forceinline__ uint32_t warp_bit_transpose(uint32_t x, int lane) {
  uint32_t y = __shfl_xor_sync(0xffffffffu, x, 16);
  x = prmt(x, y, (lane & 16) ? 0x3276u : 0x5410u);
  y = __shfl_xor_sync(0xffffffffu, x, 8);
  x = prmt(x, y, (lane & 8) ? 0x3715u : 0x6240u);
#pragma unroll
  for (int s = 4; s >= 1; s >>= 1) {
    const uint32_t low = s == 4 ? 0x0F0F0F0Fu : s == 2 ? 0x33333333u : 0x55555555u;
    const bool up = lane & s;
    y = __shfl_xor_sync(0xffffffffu, x, s);
    y = __funnelshift_l(y, y, up ? 32 - s : s);
    const uint32_t own = up ? ~low : low;
    x = (x & own) | (y & ~own);
  }
  return x;
}
// Keep decisions of 32 query rows (from q0) x 32 keys (from 16*kb), by a whole warp: every lane makes the two Philox draws of
// one row, the bits are transposed, and lane l gets key l's: those of rows 4j..4j+3 are the top bits of the four bytes of
// (word << j).
__device__ __forceinline__ uint32_t keep_word_32x32(const PhiloxKeys& keys, uint32_t offset, uint32_t bh, uint32_t q0, uint32_t kb,
                                                    uint32_t thr, int lane) {
  const uint32_t q_row = q0 + 4 * (7 - (lane & 7)) + (lane >> 3);
  uint32_t keep = 0u;
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const U4 u = dropout_draw_keys(keys, offset, bh, q_row, kb + d);
    const uint32_t ws[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)   // the keep bit of key 16d + 4k + e ends as bit 8e + 4d + k
      keep = (keep >> 1) | (((ws[k] & 0x7F7F7F7Fu) + (0x80u - thr) * 0x01010101u) & 0x80808080u);
  }
  keep = warp_bit_transpose(keep, lane);
  return __shfl_sync(0xffffffffu, keep, 8 * (lane & 3) + (lane >> 2));
}

// A row's 64 products, eight lanes with eight each: the sum in all of them.
template <bool BF16>
__device__ __forceinline__ float row_dot(const uint4& x, const uint4& y) {
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
  float sum = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    sum = fmaf(unpack_lo<BF16>(xs[k]), unpack_lo<BF16>(ys[k]), sum);
    sum = fmaf(unpack_hi<BF16>(xs[k]), unpack_hi<BF16>(ys[k]), sum);
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  sum += __shfl_xor_sync(0xffffffffu, sum, 4);
  return sum;
}

// Bound by memory: O and dO in, the accumulator out (B=32 H=16 S=512: 134 MB in 18.4 us, 7.3 TB/s, above the card's copy rate, because a part
// of the accumulator stays in the L2 cache; with each thread clearing the 32 bytes of its own eight columns, half a sector an instruction, 19.8).  PACKED: a block waits for the row offsets before it can load, so on large grids it
// takes four times the rows (R), their loads in flight together, and four blocks an SM leave the rare zeroing of uncovered rows its registers
// (12 288 rows, 16 heads 20.6 -> 15.3 us; twice the rows 15.9, in 32 registers 17.4).  Where that leaves less than 1.5 blocks per multiprocessor there is
// nothing to hide the wait behind, and blocks of 32 rows are done sooner (whole backward with four / one times 32 rows: 4 blocks of 128 rows
// 14.2 / 13.9 us, 48 18.4 / 17.9, 96 17.3 / 16.8, 192 21.7 / 21.3 and with short sequences 16.4 / 16.7, 288 24.3 / 24.7 and 17.4 / 18.5).
template <bool BF16, bool PACKED, int R>
__global__ void __launch_bounds__(256, PACKED ? 4 : 8) bwd_prepare_kernel(const __grid_constant__ PrepArgs a) {
  griddep_wait();
  // grid = (B*H, blocks of 32 R rows); 8 threads per row, 8 elements each.
  // The head index comes from the grid, so no thread divides 64-bit indices.
  constexpr int D = kAccumD, per = D / 8;
  const BwdArgs& m = a.m;
  const int part = threadIdx.x & 7;
  const int bh = blockIdx.x;
  const int h = bh % m.H;
  const int b = bh / m.H;
  const int r0 = blockIdx.y * (32 * R);
  const int r = r0 + (threadIdx.x >> 3);   // and 32 k further on; < S_q_pad
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *m.work_counter = 0;
  // packed batch: row r of sequence b is row cu[b] + r of the tensors, and exists for r < cu[b+1] - cu[b]
  int64_t row_o = static_cast<int64_t>(b) * a.o_sb + static_cast<int64_t>(r) * a.o_ss;
  int64_t row_do = static_cast<int64_t>(b) * a.do_sb + static_cast<int64_t>(r) * a.do_ss;
  int q_limit = m.S_q;
  if constexpr (PACKED) {
    const int* cu = static_cast<const int*>(m.mask);
    const int base = cu[b];
    const int len = cu[b + 1] - base;
    q_limit = packed_rows(base, cu[b + 1], m.S_q, m.total_rows);
    if (m.zero.grad[0].ptr != nullptr && (r0 + 32 * R > q_limit || len > q_limit)) {
      for (int t = 0; t < 3; ++t)
        zero_uncovered_rows(m.zero.grad[t].ptr, m.zero.grad[t].stride_s, m.zero.grad[t].stride_h, h, b, m.B, cu, m.S_q, m.total_rows, D,
                            r0, r0 + 32 * R, m.zero.mode == kUncoveredAll, threadIdx.x, blockDim.x);
    }
    if (r0 >= q_limit || m.dq_accum == nullptr) return;   // nothing of the accumulator there is added to or read; or rows to zero are all there is to do
    row_o = static_cast<int64_t>(base + r) * a.o_ss;
    row_do = static_cast<int64_t>(base + r) * a.do_ss;
  }
  uint4 wo[R], wd[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    wo[k] = wd[k] = make_uint4(0u, 0u, 0u, 0u);
    if (r + 32 * k < q_limit) {
      wo[k] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(a.o) + row_o + 32 * k * a.o_ss + h * a.o_sh + part * per));
      wd[k] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(a.d_o) + row_do + 32 * k * a.do_ss + h * a.do_sh + part * per));
    }
  }
  // the accumulator's rows, a warp's store to 512 consecutive bytes (S_q_pad is a multiple of 128 rows)
  float4* acc = reinterpret_cast<float4*>(m.dq_accum + (static_cast<int64_t>(bh) * m.S_q_pad + r0) * D) + threadIdx.x;
#pragma unroll
  for (int i = 0; i < 2 * R; ++i) acc[i * 256] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const float sum = row_dot<BF16>(wo[k], wd[k]);
    if (part == 0 && r + 32 * k < q_limit) m.delta[static_cast<int64_t>(bh) * m.S_q + r + 32 * k] = sum;
  }
}

// ---------------------------------------------------------------------------------------
// 3. dQ = scale * accumulator
// ---------------------------------------------------------------------------------------
struct FinishArgs {
  const float* dq_accum;
  void* dq;
  int64_t sb, sh, ss;
  int B, H, S_q, S_q_pad;
  float scale;
  const int* cu_seqlens;  // packed batch: row offsets into the [total_rows, H, D] dQ (sb unused), else null
  int total_rows;
};

// A block converts 128 rows of a head: coalesced 16-byte reads of the accumulator (eight in flight per thread),
// through shared memory to coalesced 16-byte writes of the rows.
constexpr int kFinishRows = 128;
template <bool BF16>
__global__ void __launch_bounds__(256) bwd_finish_kernel(const FinishArgs a) {
  griddep_wait();
  constexpr int D = kAccumD, R = kFinishRows;
  constexpr int kStride = D * 2 + 8;    // bytes; 8-byte accesses of consecutive rows hit different banks
  __shared__ __align__(16) uint8_t tile[R * kStride];
  const int bh = blockIdx.x;
  const int h = bh % a.H;
  const int b = bh / a.H;
  const int r0 = blockIdx.y * R;
  int64_t base = static_cast<int64_t>(b) * a.sb;
  int q_limit = a.S_q;
  if (a.cu_seqlens != nullptr) {
    const int first = a.cu_seqlens[b];
    q_limit = packed_rows(first, a.cu_seqlens[b + 1], a.S_q, a.total_rows);
    base = static_cast<int64_t>(first) * a.ss;
  }
  if (r0 >= q_limit) return;
  const float4* src = reinterpret_cast<const float4*>(a.dq_accum + (static_cast<int64_t>(bh) * a.S_q_pad + r0) * D);
  float4 x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = src[k * 256 + threadIdx.x];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int i = k * 256 + threadIdx.x;   // see dq_accum_index
    const int row = (i / (8 * D)) * 32 + (i & 31), c4 = (i / 32) % (D / 4);
    *reinterpret_cast<uint2*>(tile + row * kStride + c4 * 8) =
        make_uint2(pack2<BF16>(x[k].x * a.scale, x[k].y * a.scale), pack2<BF16>(x[k].z * a.scale, x[k].w * a.scale));
  }
  __syncthreads();
  unsigned short* dst = reinterpret_cast<unsigned short*>(a.dq) + base + h * a.sh;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = k * 256 + threadIdx.x;
    const int row = i / (D / 8), ch = i % (D / 8);
    const uint2 lo = *reinterpret_cast<const uint2*>(tile + row * kStride + ch * 16);
    const uint2 hi = *reinterpret_cast<const uint2*>(tile + row * kStride + ch * 16 + 8);
    if (r0 + row < q_limit) *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(r0 + row) * a.ss + ch * 8) = make_uint4(lo.x, lo.y, hi.x, hi.y);
  }
}

// ---------------------------------------------------------------------------------------
// 2. main kernel
// ---------------------------------------------------------------------------------------
// Work.  An item is one (128-key tile, head, batch); kv tile is the fastest index.  One CTA per SM
// draws items from a global counter (the first item is blockIdx.x), so the fixed cost of an item --
// loading K and V, the first S/dP, the last tile's dV/dK/dQ, the dQ reduce and the dK/dV write-out --
// overlaps the neighbouring items instead of leaving the SM idle (it was ~30 % of a CTA's life when
// every item was its own CTA).  Items whose key tile lies wholly past the valid length write zeros.
//
// Layout.  Scores are formed transposed, S^T = K Q^T and dP^T = V dO^T with keys along the tensor-memory lanes, so that
// P^T, written back to tensor memory by the thread that computed it, is the A operand of dV += P^T dO: it is neither
// written to shared memory nor read from it, and dS^T likewise that of dK += dS^T Q.  At D = 128 dQ is another kernel's
// (fmha_bwd_dq_sm100.cu); at D = 64 dS also feeds dQ = dS K and goes to shared memory as well, and K and V, the A operands of
// S^T and dP^T, lie in tensor memory.  What is saved is shared-memory bandwidth: a 128 x 128 x 16 MMA with both operands in
// shared memory takes all of it (64 cycles, 8 KB; with 64 columns 48 cycles instead of 32), and while such MMAs run a
// shared-memory access of another warp - a barrier poll, a read of lse - takes 330 cycles instead of 65 (measured).
// In this layout a thread is a key: lse and delta vary along its columns and come from shared memory (broadcast reads;
// a helper warp fetches them one to two tiles ahead), the additive key mask is one value per thread, and the dropout
// draws, which give 16 keys of one query row each, are made by the thread of that row and transposed in the warp.
//
// Schedule inside the stream of (item, query tile) pairs, numbered t = 0, 1, ...:
//   compute warps:  S(t) -> P(t) -> tensor memory (p_full) -> dP(t) -> dS(t) -> shared / tensor memory (ds_full) ->
//                   [D = 64: dQ(t-1) out]; dK and dV of an item leave when the next item's first P is ready.
//   MMA warp:       on p_full(t): dV(t), S(t+1), which overwrites P(t); on ds_full(t): dK(t), dP(t+1), which overwrites dS(t),
//                   and (D = 64) dQ(t).  S(t+1) and dP(t+1) may belong to the next item.
// Position of element (row, col) of a 128-row tile of the fp32 dQ accumulator: 32-row groups, in them groups of four
// columns, in them the 32 rows with their four values each.
template <int D>
__device__ __forceinline__ int dq_accum_index(int row, int col) {
  return (((row >> 5) * (D / 4) + (col >> 2)) * 32 + (row & 31)) * 4 + (col & 3);
}

struct BwdItem {
  int id;      // < 0: no more work
  int b, h, k0, n_cols;   // n_cols <= 0: key tile wholly masked out
  int n_q;     // query tiles of this item
  int q_limit; // query rows [0, q_limit) exist
  int row_base;  // packed batch: first row of the sequence in the [total_rows, H, D] tensors (else 0)
};

// PACKED: FMHA_MASK_CU_SEQLENS; a template parameter so that the padded kernels carry none of its bookkeeping.
// ONE_KV: D = 64 and a single key tile (bwd_one_kv).  Nothing is added up for dQ then, so its tiles are written as they come; delta is formed
// here, by the compute warps, 8 rows each, with the loads under the draws and the wait for S; and work items are equal and need no
// counter.  A packed batch has the pass before it, to zero rows.  The accumulator, its clearing and conversion and the launches around
// this one took 14 to 30 % of the time (whole backward, without / with dropout: B=2 H=4 S=128 10.6 -> 7.8 / 10.9 -> 8.4 us, B=13 H=12 S=100 15.1 -> 11.2 /
// 16.6 -> 13.0, B=32 H=16 S=128 27.8 -> 19.5 / 29.1 -> 23.0, B=128 H=16 94.4 -> 68.3 / 97.8 -> 75.7; packed, B=32 H=16 of 64 to 128 rows 34.2 -> 27.7 / 36.1 -> 31.2).
template <int D, bool BF16, bool KEYADD, bool DROP, bool PACKED = false, bool ONE_KV = false>
__global__ void __launch_bounds__(kBwdThreads, 1) fmha_bwd_kernel(const __grid_constant__ BwdArgs a) {
  griddep_wait();
  using L = BwdSmem<D>;
  constexpr int QS = L::kQStages, OS = L::kDoStages, DS = L::kDsBufs > 0 ? L::kDsBufs : 1, KV = L::kKvBufs;
  constexpr int kTmemCols = 512;
  constexpr uint32_t kColS = 0, kColdP = 128, kColdV = 256, kColdK = 256 + D;
  constexpr uint32_t kColdQ = 384;   // D = 64
  // P^T and dS^T lie over S and dP, a thread's 16 packed columns at the start of its own 32.  D = 64: K and V of an item, the
  // A operands of S^T and dP^T, are copied to tensor memory once.
  constexpr uint32_t kColP = kColS, kColdS = kColdP, kPStride = 32, kColK = 448, kColV = 480;
  constexpr int kFmt = BF16 ? 1 : 0;
  constexpr uint32_t kIdescS = make_idesc_f16(128, 128, kFmt, false, false);
  constexpr uint32_t kIdescMN = make_idesc_f16(128, D, kFmt, true, true);    // dQ: A and B MN-major
  constexpr uint32_t kIdescKN = make_idesc_f16(128, D, kFmt, false, true);   // dV, dK: A K-major (dV: tensor memory), B MN-major

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem + L::kOffK;
  uint8_t* sV = smem + L::kOffV;
  uint8_t* sQ = smem + L::kOffQ;
  uint8_t* sdO = smem + L::kOffdO;
  uint8_t* sdS = smem + L::kOffdS;
  uint8_t* sStage = smem + L::kOffStage;
  float* sStats = reinterpret_cast<float*>(smem + L::kOffStats);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* s_full = bars + 0;     // S of a tile is in tensor memory
  uint64_t* p_full = bars + 1;     // ... and P of it as well; S has been read (all compute threads arrive)
  uint64_t* dp_full = bars + 2;    // dP of a tile is in tensor memory
  uint64_t* ds_full = bars + 3;    // dS is in shared memory; dP has been read (all compute threads arrive)
  uint64_t* dq_full = bars + 4;    // dQ tile is in tensor memory; dV/dK/dQ of that tile are complete
  uint64_t* dq_free = bars + 5;    // dQ tile has been read out (all compute threads arrive)
  uint64_t* acc_full = bars + 6;   // dK / dV of a work item are complete
  uint64_t* k_full = bars + 7;
  uint64_t* k_empty = k_full + KV;   // D = 64: the item's last dQ has completed; D = 128: its last S
  uint64_t* v_full = k_empty + KV;
  uint64_t* v_empty = v_full + KV;   // D = 64: V is in tensor memory; D = 128: the item's last dP has completed
  uint64_t* q_full = v_empty + KV;
  uint64_t* q_empty = q_full + QS;
  uint64_t* do_full = q_empty + QS;
  uint64_t* do_empty = do_full + OS;      // dV of the tile has completed (so P may be overwritten, too)
  uint64_t* stat_full = do_empty + OS;    // [2] lse and delta of a tile's rows are in shared memory
  uint64_t* stat_empty = stat_full + 2;   // [2] ... and have been read (every compute warp arrives)
  uint64_t* item_full = stat_empty + 2;   // [2] ring of work items
  uint64_t* item_empty = item_full + 2;
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 4);
  // Philox offset of this launch (launch parameter + optional device-resident value), read where a draw starts
  volatile uint32_t* philox_off = reinterpret_cast<volatile uint32_t*>(smem + L::kOffMisc + 8);

  if (smem_u32(smem) & 1023) {   // see kDynBytes
    if (threadIdx.x == 0 && a.status != nullptr) atomicCAS(a.status, 0, kSiteSmemBase);
    return;
  }
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int kv_tiles = (a.S_k + kTileN - 1) / kTileN;
  const int n_q_all = (a.S_q + kTileM - 1) / kTileM;
  const int num_items = kv_tiles * a.H * a.B;
  constexpr bool packed = PACKED;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *philox_off = a.philox_offset + (a.philox_offset_dev != nullptr ? static_cast<uint32_t>(*a.philox_offset_dev) : 0u);
    mbar_init(s_full, 1);
    mbar_init(p_full, kComputeThreads);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, kComputeThreads);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, kComputeThreads);
    mbar_init(acc_full, 1);
    for (int s = 0; s < KV; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(k_empty + s, 1);
      mbar_init(v_full + s, 1);
      mbar_init(v_empty + s, 1);
    }
    for (int s = 0; s < QS; ++s) {
      mbar_init(q_full + s, 1);
      mbar_init(q_empty + s, 1);
    }
    for (int s = 0; s < OS; ++s) {
      mbar_init(do_full + s, 1);
      mbar_init(do_empty + s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(stat_full + s, ONE_KV ? 1 + kComputeThreads / 32 : 1);
      mbar_init(stat_empty + s, kComputeThreads / 32);
      mbar_init(item_full + s, 1);
      mbar_init(item_empty + s, 2 + kComputeThreads / 32);   // MMA warp, statistics warp, every compute warp
    }
    mbar_fence_init();
    tma_prefetch_desc(&a.tm_q);
    tma_prefetch_desc(&a.tm_k);
    tma_prefetch_desc(&a.tm_v);
    tma_prefetch_desc(&a.tm_do);
    tma_prefetch_desc(&a.tm_dk);
    tma_prefetch_desc(&a.tm_dv);
  }
  if (warp == 1) {
    tmem_alloc(tmem_base_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_base_slot;
  const WaitCtx wctx{abort_flag, a.status};

  // By the producer alone: the others get the result through shared memory (divisions and a read of the mask per item and
  // warp stood in the way of every item's first tile).
  auto decode = [&](int id) {
    BwdItem it;
    it.id = id;
    it.b = it.h = it.k0 = 0;
    it.n_cols = 0;
    it.n_q = n_q_all;
    it.q_limit = a.S_q;
    it.row_base = 0;
    if (id >= 0) {
      const int kv_tile = id % kv_tiles;
      const int bh = id / kv_tiles;
      it.h = bh % a.H;
      it.b = bh / a.H;
      it.k0 = kv_tile * kTileN;
      int k_limit = a.S_k;
      if (!packed && a.mask_kind == FMHA_MASK_SEQLEN) {
        const int len = reinterpret_cast<const int*>(a.mask)[it.b];
        if (len > 0 && len < a.S_k) k_limit = len;
      } else if (packed) {
        const int* cu = reinterpret_cast<const int*>(a.mask);
        it.row_base = cu[it.b];
        // a sequence longer than the stated maximum is cut there: its tiles would otherwise run into the next
        // head's rows of the dQ accumulator and of delta
        k_limit = it.q_limit = packed_rows(it.row_base, cu[it.b + 1], a.S_q, a.total_rows);
        it.n_q = (it.q_limit + kTileM - 1) / kTileM;
      }
      it.n_cols = min(kTileN, k_limit - it.k0);
    }
    return it;
  };
  const uint32_t ring = smem_u32(smem + L::kOffRing);
  // Consumer side of the work-item ring (whole warp): item number `n` of this CTA.
  auto fetch_item = [&](int n, uint32_t sleep_ns) {
    const int slot = n & 1;
    mbar_wait(item_full + slot, (n >> 1) & 1, wctx, kSiteItemFull, sleep_ns);
    const uint4 x = lds128(ring + slot * 32), y = lds128(ring + slot * 32 + 16);
    BwdItem it;
    it.id = *abort_flag ? -1 : static_cast<int>(x.x);
    it.b = static_cast<int>(x.y);
    it.h = static_cast<int>(x.z);
    it.k0 = static_cast<int>(x.w);
    it.n_cols = static_cast<int>(y.x);
    it.n_q = static_cast<int>(y.y);
    it.q_limit = static_cast<int>(y.z);
    it.row_base = static_cast<int>(y.w);
    __syncwarp();
    if (lane == 0) mbar_arrive(item_empty + slot);
    return it;
  };

  if (warp == 0) {
    // ============================ TMA producer ======================================
    if (lane == 0) {
      int w = 0, g = 0;   // work items with keys / query tiles loaded so far
      int next = static_cast<int>(blockIdx.x);
      for (int n = 0;; ++n) {
        const int slot = n & 1;
        const BwdItem it = decode(next < num_items && !*abort_flag ? next : -1);
        if (n >= 2) mbar_wait(item_empty + slot, ((n >> 1) - 1) & 1, wctx, kSiteItemEmpty);
        sts128(ring + slot * 32, static_cast<uint32_t>(it.id), static_cast<uint32_t>(it.b), static_cast<uint32_t>(it.h),
               static_cast<uint32_t>(it.k0));
        sts128(ring + slot * 32 + 16, static_cast<uint32_t>(it.n_cols), static_cast<uint32_t>(it.n_q), static_cast<uint32_t>(it.q_limit),
               static_cast<uint32_t>(it.row_base));
        mbar_arrive(item_full + slot);
        if (it.id < 0) break;
        if constexpr (ONE_KV) next += static_cast<int>(gridDim.x);
        else next = atomicAdd(a.work_counter, 1) + static_cast<int>(gridDim.x);   // not looked at before this item's loads are out
        const int tb = packed ? 0 : it.b;
        if (it.n_cols <= 0) continue;
        const int kvb = w % KV;
        const uint32_t kvp = (w / KV - 1) & 1;
        if (w >= KV) mbar_wait(k_empty + kvb, kvp, wctx, kSiteKEmpty);
        mbar_arrive_expect_tx(k_full + kvb, L::kTileBytes);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_4d(sK + kvb * L::kTileBytes + c * 16384, &a.tm_k, k_full + kvb, c * 64, it.row_base + it.k0, it.h, tb);
        for (int i = 0; i < it.n_q; ++i, ++g) {
          const int qs = g % QS, os = g % OS;
          if (g >= QS) mbar_wait(q_empty + qs, ((g / QS) - 1) & 1, wctx, kSiteQEmpty);
          mbar_arrive_expect_tx(q_full + qs, L::kTileBytes);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(sQ + qs * L::kTileBytes + c * 16384, &a.tm_q, q_full + qs, c * 64, it.row_base + i * kTileM, it.h, tb);
          if (i == 0) {   // V after the first Q: with one K/V buffer it comes free after K
            if (w >= KV) mbar_wait(v_empty + kvb, kvp, wctx, kSiteVEmpty);
            mbar_arrive_expect_tx(v_full + kvb, L::kTileBytes);
#pragma unroll
            for (int c = 0; c < D / 64; ++c)
              tma_load_4d(sV + kvb * L::kTileBytes + c * 16384, &a.tm_v, v_full + kvb, c * 64, it.row_base + it.k0, it.h, tb);
          }
          if (g >= OS) mbar_wait(do_empty + os, ((g / OS) - 1) & 1, wctx, kSiteDoEmpty);
          mbar_arrive_expect_tx(do_full + os, L::kTileBytes);
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_load_4d(sdO + os * L::kTileBytes + c * 16384, &a.tm_do, do_full + os, c * 64, it.row_base + i * kTileM, it.h, tb);
        }
        ++w;
      }
    }
  } else if (warp == 1) {
    // ============================ MMA issuer ========================================
    // The whole warp runs this loop convergently; the MMAs go out in bursts of 4 or 8 from one
    // elected lane with descriptors prepared beforehand as warp-uniform values (see umma_ss_x4).
    // A loop in which a single lane computes each descriptor and then issues was starved by the
    // compute warps' arithmetic: ~150 cycles per MMA during their exp/Philox phase.
    constexpr int KS = D / 16;      // k-steps of S and dP
    const uint32_t tS = tmem_base + kColS, tdP = tmem_base + kColdP, tdV = tmem_base + kColdV,
                   tdK = tmem_base + kColdK, tdQ = tmem_base + kColdQ, tP = tmem_base + kColP;
    // [128 x 128] = A (rows of D values, K-major) * B (likewise)^T
    auto issue_kk = [&](uint32_t d, const uint8_t* a_tile, const uint8_t* b_tile) {
      const uint64_t da = make_smem_desc_sw128(smem_u32(a_tile), 16, 1024), db = make_smem_desc_sw128(smem_u32(b_tile), 16, 1024);
      uint64_t x[KS], y[KS];
#pragma unroll
      for (int kk = 0; kk < KS; ++kk) {
        x[kk] = da + kmajor_step(kk, 16384);
        y[kk] = db + kmajor_step(kk, 16384);
      }
      if constexpr (KS == 4) umma_ss_x4(d, x, y, kIdescS, 0u);
      else umma_ss_x8(d, x, y, kIdescS, 0u);
    };
    // D = 64: K or V tile to 32 tensor-memory columns (in the tensor core's pipe, in order with the MMAs), and
    // [128 x 128] = A (there) * B (rows of 64 values, K-major)^T
    auto copy_a = [&](uint32_t dst, const uint8_t* tile) {
      const uint64_t d = make_smem_desc_sw128(smem_u32(tile), 16, 1024);
      uint64_t x[4];
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) x[kk] = d + kmajor_step(kk, 16384);
      tmem_cp_128x256b_x4(dst, x);
    };
    auto issue_tk = [&](uint32_t d, uint32_t a_tmem, const uint8_t* b_tile) {
      const uint64_t db = make_smem_desc_sw128(smem_u32(b_tile), 16, 1024);
      uint64_t y[4];
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) y[kk] = db + kmajor_step(kk, 16384);
      umma_ts_x4(d, a_tmem, 8u, y, kIdescS, 0u);
    };
    // S^T and dP^T of tile tt, which belongs to item number wi (with work) and is its first / last one
    auto issue_s = [&](int tt, int wi, bool first, bool last) {
      if (first) {
        mbar_wait(k_full + wi % KV, (wi / KV) & 1, wctx, kSiteKFull);
        if constexpr (D == 64) copy_a(tmem_base + kColK, sK + (wi % KV) * L::kTileBytes);
      }
      if (first) mbar_wait(q_full + tt % QS, (tt / QS) & 1, wctx, kSiteQFull);   // else waited for already
      tc_fence_after_sync();
      if constexpr (D == 64) issue_tk(tS, tmem_base + kColK, sQ + (tt % QS) * L::kTileBytes);
      else issue_kk(tS, sK + (wi % KV) * L::kTileBytes, sQ + (tt % QS) * L::kTileBytes);
      umma_commit_elect(s_full);
      if (D == 128 && last) umma_commit_elect(k_empty + wi % KV);
    };
    auto issue_dp = [&](int tt, int wi, bool first, bool last) {
      if (first) {
        mbar_wait(v_full + wi % KV, (wi / KV) & 1, wctx, kSiteVFull);
        if constexpr (D == 64) {
          copy_a(tmem_base + kColV, sV + (wi % KV) * L::kTileBytes);
          umma_commit_elect(v_empty + wi % KV);
        }
      }
      if (first) mbar_wait(do_full + tt % OS, (tt / OS) & 1, wctx, kSiteDoFull);
      tc_fence_after_sync();
      if constexpr (D == 64) issue_tk(tdP, tmem_base + kColV, sdO + (tt % OS) * L::kTileBytes);
      else issue_kk(tdP, sV + (wi % KV) * L::kTileBytes, sdO + (tt % OS) * L::kTileBytes);
      umma_commit_elect(dp_full);
      if (D == 128 && last) umma_commit_elect(v_empty + wi % KV);
    };

    int n = 0, w = 0, t = 0;   // items fetched, items with work, query tiles so far
    auto next_work = [&]() {   // the next item with keys
      BwdItem it = fetch_item(n++, 0);
      while (it.id >= 0 && it.n_cols <= 0) it = fetch_item(n++, 0);
      return it;
    };
    BwdItem cur = next_work();
    if (cur.id >= 0) {
      issue_s(0, 0, true, cur.n_q == 1);
      issue_dp(0, 0, true, cur.n_q == 1);
    }
    while (cur.id >= 0) {
      const int kvb = w % KV;
      const int n_q = cur.n_q;
      BwdItem nxt = cur;
      for (int i = 0; i < n_q; ++i, ++t) {
        const bool last = i + 1 == n_q;
        const int qs = t % QS, os = t % OS;
        const uint32_t acc0 = (i > 0) ? 1u : 0u;
        // (the next tile's Q and, below, dO are usually there: polled here, the answer does not hold up S and dP)
        if (!last) mbar_wait(q_full + (t + 1) % QS, ((t + 1) / QS) & 1, wctx, kSiteQFull);
        // ---- dV += P^T dO: A from tensor memory, dO read MN-major (16 query rows = 2048 B per k-step) ----------------
        const uint64_t ddO_m = make_smem_desc_sw128(smem_u32(sdO + os * L::kTileBytes), 16384, 1024);
        mbar_wait(p_full, t & 1, wctx, kSitePFull);
        tc_fence_after_sync();
        {
          uint64_t y[4];
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) y[kk] = ddO_m + mnmajor_step(hf * 4 + kk);
            const uint32_t p0 = tP + 2 * hf * kPStride;
            umma_ts_2x2(tdV, p0, p0 + kPStride, 8u, y, kIdescKN, hf == 0 ? acc0 : 1u);
          }
        }
        umma_commit_elect(do_empty + os);   // dP(t) came before, so dO(t) is not read again
        // ---- S of the next tile ------------------------------------------------------------------------------------------------
        if (last) nxt = next_work();   // the compute warps finish tile t, and any items without keys, without another MMA
        const bool more = !last || nxt.id >= 0;
        const int wn = last ? w + 1 : w;                                  // item of tile t+1, and whether t+1 is its last tile
        const bool next_last = last ? nxt.n_q == 1 : i + 2 == n_q;
        if (more) issue_s(t + 1, wn, last, next_last);
        // ---- dK += dS^T Q (A from tensor memory), dP of the next tile over dS(t), dQ tile = dS K ------------------------------
        const uint64_t dQ_m = make_smem_desc_sw128(smem_u32(sQ + qs * L::kTileBytes), 16384, 1024);
        if (!last) mbar_wait(do_full + (t + 1) % OS, ((t + 1) / OS) & 1, wctx, kSiteDoFull);
        mbar_wait(ds_full, t & 1, wctx, kSiteDsFull);
        tc_fence_after_sync();
        {
          const uint32_t tdS = tmem_base + kColdS;
          uint64_t y[4];
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) y[kk] = dQ_m + mnmajor_step(hf * 4 + kk);
            umma_ts_2x2(tdK, tdS + 2 * hf * kPStride, tdS + (2 * hf + 1) * kPStride, 8u, y, kIdescKN, hf == 0 ? acc0 : 1u);
          }
        }
        umma_commit_elect(q_empty + qs);
        if (last) umma_commit_elect(acc_full);
        if (more) issue_dp(t + 1, wn, last, next_last);
        if constexpr (D == 64) {
          const uint64_t ddS_m = make_smem_desc_sw128(smem_u32(sdS + (t % DS) * L::kDsBytes), 16384, 1024);   // MN-major A (queries x keys)
          const uint64_t dK_m = make_smem_desc_sw128(smem_u32(sK + kvb * L::kTileBytes), 16384, 1024);        // MN-major B
          if (t > 0) {
            mbar_wait(dq_free, (t - 1) & 1, wctx, kSiteDqFree);
            tc_fence_after_sync();
          }
          uint64_t x[8], y[8];
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            x[kk] = ddS_m + mnmajor_step(kk);
            y[kk] = dK_m + mnmajor_step(kk);
          }
          umma_ss_x8(tdQ, x, y, kIdescMN, 0u);
          umma_commit_elect(dq_full);
          if (last) umma_commit_elect(k_empty + kvb);   // K of this item is not read again
        }
      }
      ++w;
      cur = nxt;
    }
  } else if (warp == kBwdStatWarp) {
    // ============================ row statistics =====================================
    // lse and delta of a tile's 128 query rows (ONE_KV: lse alone), in the form the compute warps use them, one to two tiles ahead.
    const float inv_c = DROP ? 1.0f / a.dropout_scale : 1.0f;
    int n = 0, t = 0;
    while (true) {
      const BwdItem cur = fetch_item(n++, 0);
      if (cur.id < 0) break;
      if (cur.n_cols <= 0) continue;
      // logsumexp rows: [B*H, S_q], or [H, total_rows] for a packed batch; delta is always [B*H, S_q]
      const float* lse = a.lse + (packed ? static_cast<int64_t>(cur.h) * a.total_rows + cur.row_base : static_cast<int64_t>(cur.b * a.H + cur.h) * a.S_q);
      const float* delta = a.delta + static_cast<int64_t>(cur.b * a.H + cur.h) * a.S_q;
      for (int i = 0; i < cur.n_q; ++i, ++t) {
        float x[4], d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = i * kTileM + k * 32 + lane;
          x[k] = INFINITY;   // rows past the end: their probabilities are zero
          d[k] = 0.f;
          if (r < cur.q_limit) {
            x[k] = lse[r];
            if (!ONE_KV) d[k] = delta[r];
          }
        }
        const int slot = t & 1;
        if (t >= 2) mbar_wait(stat_empty + slot, ((t >> 1) - 1) & 1, wctx, kSiteStatEmpty);
        float* st = sStats + slot * 2 * kTileM;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          st[k * 32 + lane] = -x[k] * kLog2eB;
          if (!ONE_KV) st[kTileM + k * 32 + lane] = d[k] * inv_c;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(stat_full + slot);
      }
    }
  } else {
    // ============================ compute warps =====================================
    // 16 warps: warp (quad, cq) owns keys [32*quad, +32) (its tensor-memory lane quarter, one key per thread) and the
    // query columns [32*cq, +32) of every 128 x 128 tile.
    const int cw = warp - 2;             // 0..15
    const int quad = warp & 3;           // tensor-memory lane quarter of this warp
    const int cq = cw >> 2;              // which 32 columns of the tile
    const int row = quad * 32 + lane;    // key within the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const float sl2 = a.scale_log2;
    // With dropout dS is formed as P*(keep*dP - delta/c) and the factor c = 1/(1-p) moves into the
    // final scaling of dQ and dK (and of dV, whose P operand is unscaled as well).
    const float dscale = DROP ? a.dropout_scale : 1.0f;
    constexpr int DQ = D / 4;            // columns of a [128 x D] accumulator handled by one thread
    uint8_t* stage = sStage + cw * 2048;   // this warp's staging tile for dK and dV

    // Every warp polls the mbarrier itself: funnelling the wait through one warp and a named barrier
    // was measured 8 % slower (it removes the skew between warps that lets their phases overlap).
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int site) {
      mbar_wait(bar, parity, wctx, site, kComputeSleepNs);
      tc_fence_after_sync();
    };
    // What the write-outs of an item done during the next one (dK and dV, ONE_KV: its last dQ tile) need to know of it waits in shared memory.
    const uint32_t rec = smem_u32(smem + L::kOffRec) + cw * 32;
    // Frees the warp's staging tile (its previous TMA copies have been read).
    auto stage_free = [&]() {
      if (lane == 0) tma_store_wait_read();
      __syncwarp();
    };
    // dQ tile `tt` (rows = queries): tensor memory -> registers -> fp32 accumulator, 16 bytes per reduction.  The
    // accumulator is laid out so that a warp's instruction covers 512 consecutive bytes (dq_accum_index), which keeps the
    // tile out of shared memory: staged there for TMA reduce-adds it cost 32 (D = 64) or 64 KB written and read again per
    // tile, a fifth of all shared-memory traffic.
    // `tile` is its place there; ONE_KV: twice its number within the item, and the parity of the item's.
    [[maybe_unused]] auto dq_readout = [&](int tt, int tile) {   // D = 64
      wait_all(dq_full, tt & 1, kSiteDqFull);
      uint32_t r[DQ];
#pragma unroll
      for (int c = 0; c < DQ / 16; ++c)
        tmem_ld16(tmem_base + lane_addr + kColdQ + cq * DQ + c * 16, *reinterpret_cast<uint32_t(*)[16]>(r + c * 16));
      tmem_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(dq_free);                          // the dQ columns may be overwritten
      if constexpr (ONE_KV) {
        const uint4 x = lds128(rec + (tile & 1) * 16);
        const int64_t h = x.x & 0xffffu, b = packed ? 0u : x.x >> 16;
        const int q = (tile >> 1) * kTileM + row;
        if (q < static_cast<int>(x.w) && *abort_flag == 0) {
          const float mul = a.scale * dscale;
          uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(a.dq_ptr) + b * a.dq_sb + h * a.dq_sh +
                                                static_cast<int64_t>(static_cast<int>(x.z) + q) * a.dq_ss + cq * DQ);
          auto pair = [&](int k) { return pack2<BF16>(__uint_as_float(r[k]) * mul, __uint_as_float(r[k + 1]) * mul); };
#pragma unroll
          for (int k = 0; k < DQ / 8; ++k) dst[k] = make_uint4(pair(8 * k), pair(8 * k + 2), pair(8 * k + 4), pair(8 * k + 6));
        }
        return;
      }
      float* dst = a.dq_accum + static_cast<int64_t>(tile) * (kTileM * D) + dq_accum_index<D>(row, cq * DQ);
#pragma unroll
      for (int q = 0; q < DQ / 4; ++q)
        red_add_v4(dst + q * 128, __uint_as_float(r[q * 4]), __uint_as_float(r[q * 4 + 1]), __uint_as_float(r[q * 4 + 2]),
                   __uint_as_float(r[q * 4 + 3]));
    };
    // dK and dV of a finished item: tensor memory -> registers -> this warp's staging tile -> two TMA
    // stores issued by its lane 0.  Warp (quad, cq) holds key rows [32*quad, +32) x columns [cq*DQ, +DQ)
    // of both accumulators: 32 rows of DQ*2 bytes each.  The staging tile holds one of them at D = 128, both at D = 64
    // (dV first).  Rows past S_k are clipped by the TMA unit.
    constexpr int kDkvRowBytes = DQ * 2;
    auto store_dkdv = [&](int h, int b, int k0, int row_base, int q_limit, bool from_tmem) {
      // Packed batch: a slice that reaches past the end of the sequence would overwrite the next sequence's
      // rows, so its rows are written one by one from registers.
      const int key = k0 + quad * 32 + lane;
      const bool edge = packed && (k0 + quad * 32 + 32 > q_limit);
      stage_free();
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const float mul = (which == 0) ? dscale : a.scale * dscale;
        uint8_t* tile = stage + (D == 64 ? which * 32 * kDkvRowBytes : 0);
        const uint32_t rowaddr = smem_u32(tile) + lane * kDkvRowBytes;
        if (D == 128 && which == 1) stage_free();
        unsigned short* grow = reinterpret_cast<unsigned short*>(which == 0 ? a.dv_ptr : a.dk_ptr) +
                               static_cast<int64_t>(row_base + key) * (which == 0 ? a.dv_ss : a.dk_ss) +
                               static_cast<int64_t>(h) * (which == 0 ? a.dv_sh : a.dk_sh) + cq * DQ;
#pragma unroll
        for (int c = 0; c < DQ / 16; ++c) {
          uint32_t r[16];
          if (from_tmem) {
            tmem_ld16(tmem_base + lane_addr + (which == 0 ? kColdV : kColdK) + cq * DQ + c * 16, r);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) r[k] = 0u;
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint4 w;
            w.x = pack2<BF16>(__uint_as_float(r[q * 8 + 0]) * mul, __uint_as_float(r[q * 8 + 1]) * mul);
            w.y = pack2<BF16>(__uint_as_float(r[q * 8 + 2]) * mul, __uint_as_float(r[q * 8 + 3]) * mul);
            w.z = pack2<BF16>(__uint_as_float(r[q * 8 + 4]) * mul, __uint_as_float(r[q * 8 + 5]) * mul);
            w.w = pack2<BF16>(__uint_as_float(r[q * 8 + 6]) * mul, __uint_as_float(r[q * 8 + 7]) * mul);
            if (edge) {
              if (key < q_limit) *reinterpret_cast<uint4*>(grow + c * 16 + q * 8) = w;
            } else {
              sts128(rowaddr + c * 32 + q * 16, w.x, w.y, w.z, w.w);
            }
          }
        }
        if (D == 64 && which == 0) continue;   // one fence and one commit for both
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && *abort_flag == 0 && !edge) {
          const int row0 = row_base + k0 + quad * 32, tb = packed ? 0 : b;
          if (D == 64 || which == 0) tma_store_4d(&a.tm_dv, stage, cq * DQ, row0, h, tb);
          if (which == 1) tma_store_4d(&a.tm_dk, tile, cq * DQ, row0, h, tb);
          tma_store_commit();
        }
      }
    };

    int n = 0, w = 0, t = 0;      // items fetched, items with work, query tiles so far
    bool pending = false;         // dK and dV of item number w-1 (with work) are still in tensor memory
    auto store_pending = [&]() {
      const uint4 r = lds128(rec + ((w - 1) & 1) * 16);
      store_dkdv(static_cast<int>(r.x & 0xffffu), static_cast<int>(r.x >> 16), static_cast<int>(r.y), static_cast<int>(r.z),
                 static_cast<int>(r.w), true);
      pending = false;
    };
    [[maybe_unused]] int prev_tile = 0;       // D = 64: tile t-1 as dq_readout wants it,
    [[maybe_unused]] bool dq_out = true;      // and whether its dQ has been read out

    while (true) {
      const BwdItem cur = fetch_item(n++, kComputeSleepNs);
      if (cur.id < 0) break;
      if (cur.n_cols <= 0) {
        if (packed) continue;   // a packed sequence has no rows past its length
        store_dkdv(cur.h, cur.b, cur.k0, cur.row_base, cur.q_limit, false);   // key tile wholly past the valid length: its gradients are zero
        continue;
      }
      if (lane == 0)   // h, b <= 65535
        sts128(rec + (w & 1) * 16, static_cast<uint32_t>(cur.h) | static_cast<uint32_t>(cur.b) << 16, static_cast<uint32_t>(cur.k0),
               static_cast<uint32_t>(cur.row_base), static_cast<uint32_t>(cur.q_limit));
      const int n_cols = cur.n_cols, bh = cur.b * a.H + cur.h, n_q = cur.n_q;
      const uint32_t gbh = static_cast<uint32_t>(a.philox_bh_offset + bh);
      const bool key_ok = row < n_cols;     // keys past the valid length / tensor edge
      float key_add = 0.f;
      if constexpr (KEYADD) {
        const int c = cur.k0 + row;
        if (c < a.S_k) key_add = reinterpret_cast<const float*>(a.mask)[static_cast<size_t>(cur.b) * a.S_k + c] * kLog2eB;
      }

      for (int i = 0; i < n_q; ++i, ++t) {
        // ONE_KV: O and dO for delta of rows [8 cw, +8) of the tile, eight lanes a row, four rows an instruction.  (Its place among the
        // statistics is free: every warp has passed the barriers of the tile before.)
        [[maybe_unused]] uint4 wo[2], wd[2];
        if constexpr (ONE_KV) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int64_t r = i * kTileM + cw * 8 + k * 4 + (lane >> 3);
            wo[k] = wd[k] = make_uint4(0u, 0u, 0u, 0u);
            if (r < (packed ? cur.q_limit : a.S_q)) {
              const int64_t at = packed ? cur.row_base + r : r, b = packed ? 0 : cur.b;
              wo[k] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(a.o_ptr) + b * a.o_sb + cur.h * a.o_sh + at * a.o_ss) + (lane & 7));
              wd[k] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(a.do_ptr) + b * a.do_sb + cur.h * a.do_sh + at * a.do_ss) + (lane & 7));
            }
          }
        }
        // Keep decisions of this thread's key and 32 query columns, drawn before S is needed.  (Measured and not better: after P
        // or dS has been handed on, a tile ahead; among the exponentials; half of the warps ahead of the others; one bit per score
        // from the pass before, whose draws cost there what they save here - B=16 H=16 S=1024 320 us for the backward against 319 -
        // and take memory.)
        [[maybe_unused]] uint32_t keep = 0u;
        if constexpr (DROP) {
          keep = keep_word_32x32(a.philox_keys, *philox_off, gbh, static_cast<uint32_t>(i * kTileM + cq * 32),
                                 static_cast<uint32_t>((cur.k0 + quad * 32) / 16), a.philox_thr, lane);
        }
        if constexpr (ONE_KV) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float sum = row_dot<BF16>(wo[k], wd[k]);
            if ((lane & 7) == 0) sStats[(t & 1) * 2 * kTileM + kTileM + cw * 8 + k * 4 + (lane >> 3)] = sum * (DROP ? 1.0f / a.dropout_scale : 1.0f);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(stat_full + (t & 1));
        }
        const uint32_t stats = smem_u32(sStats + (t & 1) * 2 * kTileM + cq * 32);
        {   // both polls go out before either answer is looked at
          const bool st_ok = mbar_try_wait(stat_full + (t & 1), (t >> 1) & 1), s_ok = mbar_try_wait(s_full, t & 1);
          if (!st_ok) mbar_wait(stat_full + (t & 1), (t >> 1) & 1, wctx, kSiteStatFull, kComputeSleepNs);
          if (!s_ok) mbar_wait(s_full, t & 1, wctx, kSiteSFull, kComputeSleepNs);
          tc_fence_after_sync();
        }
        // ---- P ----------------------------------------------------------------------------------------------------------
        uint32_t p[32];
        tmem_ld32(tmem_base + lane_addr + kColS + cq * 32, p);
        tmem_wait_ld_dep(p);
        const float2 sl22 = make_float2(sl2, sl2);
        const float2 add2 = make_float2(key_add, key_add);
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {   // four columns at a time
          const uint4 nl = lds128(stats + j * 16);
          float2 l0 = make_float2(__uint_as_float(nl.x), __uint_as_float(nl.y)), l1 = make_float2(__uint_as_float(nl.z), __uint_as_float(nl.w));
          if constexpr (KEYADD) {
            l0 = __fadd2_rn(l0, add2);
            l1 = __fadd2_rn(l1, add2);
          }
          const float2 x0 = __ffma2_rn(make_float2(__uint_as_float(p[4 * j]), __uint_as_float(p[4 * j + 1])), sl22, l0);
          const float2 x1 = __ffma2_rn(make_float2(__uint_as_float(p[4 * j + 2]), __uint_as_float(p[4 * j + 3])), sl22, l1);
          const float e0 = fast_exp2(x0.x), e1 = fast_exp2(x0.y), e2 = fast_exp2(x1.x), e3 = fast_exp2(x1.y);
          p[4 * j] = __float_as_uint(e0);
          p[4 * j + 1] = __float_as_uint(e1);
          p[4 * j + 2] = __float_as_uint(e2);
          p[4 * j + 3] = __float_as_uint(e3);
          pk[2 * j] = pack2<BF16>(e0, e1);
          pk[2 * j + 1] = pack2<BF16>(e2, e3);
          if constexpr (DROP) {
            pk[2 * j] &= prmt(keep << j, 0u, 0x9988u);
            pk[2 * j + 1] &= prmt(keep << j, 0u, 0xBBAAu);
          }
        }
        if (n_cols < kTileN && !key_ok) {
#pragma unroll
          for (int k = 0; k < 16; ++k) pk[k] = 0u;
        }
        if (pending) {
          // dK and dV of the previous item must be out of tensor memory before this tile's P lets the tensor core
          // overwrite dV.
          wait_all(acc_full, (w - 1) & 1, kSiteAccFull);
          store_pending();
        }
        tmem_st16(tmem_base + lane_addr + kColP + cq * kPStride, pk);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(p_full);
        // ---- dS -----------------------------------------------------------------------------------------------------------
        wait_all(dp_full, t & 1, kSiteDpFull);
        uint32_t dp[32];
        tmem_ld32(tmem_base + lane_addr + kColdP + cq * 32, dp);
        tmem_wait_ld_dep(dp);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint4 de = lds128(stats + kTileM * 4 + j * 16);
          if constexpr (DROP) {
            const uint32_t y = keep << j;
            dp[4 * j] &= prmt(y, 0u, 0x8888u);
            dp[4 * j + 1] &= prmt(y, 0u, 0x9999u);
            dp[4 * j + 2] &= prmt(y, 0u, 0xAAAAu);
            dp[4 * j + 3] &= prmt(y, 0u, 0xBBBBu);
          }
          const float2 d0 = __fadd2_rn(make_float2(__uint_as_float(dp[4 * j]), __uint_as_float(dp[4 * j + 1])),
                                       make_float2(-__uint_as_float(de.x), -__uint_as_float(de.y)));
          const float2 d1 = __fadd2_rn(make_float2(__uint_as_float(dp[4 * j + 2]), __uint_as_float(dp[4 * j + 3])),
                                       make_float2(-__uint_as_float(de.z), -__uint_as_float(de.w)));
          const float2 s0 = __fmul2_rn(make_float2(__uint_as_float(p[4 * j]), __uint_as_float(p[4 * j + 1])), d0);
          const float2 s1 = __fmul2_rn(make_float2(__uint_as_float(p[4 * j + 2]), __uint_as_float(p[4 * j + 3])), d1);
          pk[2 * j] = pack2<BF16>(s0.x, s0.y);
          pk[2 * j + 1] = pack2<BF16>(s1.x, s1.y);
        }
        if (n_cols < kTileN && !key_ok) {
#pragma unroll
          for (int k = 0; k < 16; ++k) pk[k] = 0u;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(stat_empty + (t & 1));
        if constexpr (D == 64) {
          // query columns [32*cq, +32) of key `row`: 64 bytes = 16-byte chunks (cq%2)*4 .. +3 of sub-tile cq/2
          const uint32_t buf = smem_u32(sdS + (t % DS) * L::kDsBytes + (cq >> 1) * 16384);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            sts128(buf + sw128_offset(row, (cq & 1) * 4 + q), pk[q * 4], pk[q * 4 + 1], pk[q * 4 + 2], pk[q * 4 + 3]);
          fence_proxy_async_smem();
        }
        tmem_st16(tmem_base + lane_addr + kColdS + cq * kPStride, pk);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(ds_full);
        if constexpr (D == 64) {
          if (!dq_out) dq_readout(t - 1, prev_tile);
          dq_out = false;
          prev_tile = ONE_KV ? 2 * i + (w & 1) : bh * n_q_all + i;
        }
      }
      pending = true;
      ++w;
    }
    // ---- drain: the last tile's dQ and the last item's dK, dV ------------------------------
    if constexpr (D == 64) {
      if (!dq_out) dq_readout(t - 1, prev_tile);
    }
    if (pending) {
      wait_all(acc_full, (w - 1) & 1, kSiteAccFull);
      store_pending();
    }
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

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------
// Head dimension 64, one key tile: whether the main kernel is all there is (ONE_KV), in a packed batch after the pass before it has zeroed rows, and nothing
// else.  Not for a few heads of many query tiles: delta formed within an item costs each of its tiles 0.6 us, in a pass of its own it has the whole chip
// (8 heads, S_k=50, alone / with the passes: S_q=256 10.7 / 12.3 us, 384 13.7 / 13.9, 512 17.0 / 15.4).  Where it is taken, S_k=100: 1 to 1024 heads,
// S_q=128 0.67 to 0.84 of the passes' time, 384 0.69 to 1.00, 48 heads and more S_q=512 0.71 to 0.98, 96 and more 1024 0.69 to 1.00 (1.02 at 160 heads).
bool bwd_one_kv(int D, int64_t heads, int S_q, int S_k) {
  return D == 64 && S_k <= kTileN && (S_q <= 3 * kTileM || heads >= 12 * ((S_q + kTileM - 1) / kTileM));
}

template <int D, bool BF16, bool KEYADD, bool DROP, bool PACKED = false, bool ONE_KV = false>
static int launch_bwd_impl(const BwdArgs& a, cudaStream_t stream) {
  using L = BwdSmem<D>;
  auto kfn = fmha_bwd_kernel<D, BF16, KEYADD, DROP, PACKED, ONE_KV>;
  static std::atomic<bool> configured[64] = {};   // per device; set after the attribute call succeeded
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const int64_t items = static_cast<int64_t>((a.S_k + kTileN - 1) / kTileN) * a.H * a.B;
  const int grid = static_cast<int>(std::min<int64_t>(items, sm_count()));   // one persistent CTA per SM
  const cudaError_t e = launch_overlapped(kfn, dim3(grid), dim3(kBwdThreads), L::kDynBytes, stream, a);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_bwd(const BwdArgs& a, int D, int dtype, cudaStream_t stream) {
  const bool bf = dtype == FMHA_DTYPE_BF16;
  const bool keyadd = a.mask_kind == FMHA_MASK_KEY_ADDITIVE;
  const bool drop = a.dropout_kind == FMHA_DROPOUT_PHILOX;
  const bool one_kv = bwd_one_kv(D, static_cast<int64_t>(a.B) * a.H, a.S_q, a.S_k);
  if (a.mask_kind == FMHA_MASK_CU_SEQLENS) {
#define FMHA_BWD_ONE_PACKED(BF, DR) \
  if (one_kv && bf == BF && drop == DR) return launch_bwd_impl<64, BF, false, DR, true, true>(a, stream);
    FMHA_BWD_ONE_PACKED(false, false)
    FMHA_BWD_ONE_PACKED(false, true)
    FMHA_BWD_ONE_PACKED(true, false)
    FMHA_BWD_ONE_PACKED(true, true)
#undef FMHA_BWD_ONE_PACKED
#define FMHA_BWD_PACKED(DD, BF, DR) \
  if (D == DD && bf == BF && drop == DR) return launch_bwd_impl<DD, BF, false, DR, true>(a, stream);
    FMHA_BWD_PACKED(64, false, false)
    FMHA_BWD_PACKED(64, false, true)
    FMHA_BWD_PACKED(64, true, false)
    FMHA_BWD_PACKED(64, true, true)
    FMHA_BWD_PACKED(128, false, false)
    FMHA_BWD_PACKED(128, false, true)
    FMHA_BWD_PACKED(128, true, false)
    FMHA_BWD_PACKED(128, true, true)
#undef FMHA_BWD_PACKED
    return static_cast<int>(cudaErrorInvalidValue);
  }
  if (one_kv) {
#define FMHA_BWD_ONE(BF, KA, DR) \
  if (bf == BF && keyadd == KA && drop == DR) return launch_bwd_impl<64, BF, KA, DR, false, true>(a, stream);
    FMHA_BWD_ONE(false, false, false)
    FMHA_BWD_ONE(false, false, true)
    FMHA_BWD_ONE(false, true, false)
    FMHA_BWD_ONE(false, true, true)
    FMHA_BWD_ONE(true, false, false)
    FMHA_BWD_ONE(true, false, true)
    FMHA_BWD_ONE(true, true, false)
    FMHA_BWD_ONE(true, true, true)
#undef FMHA_BWD_ONE
  }
#define FMHA_BWD_CASE(DD, BF, KA, DR) \
  if (D == DD && bf == BF && keyadd == KA && drop == DR) return launch_bwd_impl<DD, BF, KA, DR>(a, stream);
  FMHA_BWD_CASE(64, false, false, false)
  FMHA_BWD_CASE(64, false, false, true)
  FMHA_BWD_CASE(64, false, true, false)
  FMHA_BWD_CASE(64, false, true, true)
  FMHA_BWD_CASE(64, true, false, false)
  FMHA_BWD_CASE(64, true, false, true)
  FMHA_BWD_CASE(64, true, true, false)
  FMHA_BWD_CASE(64, true, true, true)
  FMHA_BWD_CASE(128, false, false, false)
  FMHA_BWD_CASE(128, false, false, true)
  FMHA_BWD_CASE(128, false, true, false)
  FMHA_BWD_CASE(128, false, true, true)
  FMHA_BWD_CASE(128, true, false, false)
  FMHA_BWD_CASE(128, true, false, true)
  FMHA_BWD_CASE(128, true, true, false)
  FMHA_BWD_CASE(128, true, true, true)
#undef FMHA_BWD_CASE
  return static_cast<int>(cudaErrorInvalidValue);
}

int launch_bwd_prepare(const fmha_tensor4& ot, const fmha_tensor4& dot, const BwdArgs& m, int dtype, cudaStream_t stream) {
  PrepArgs p;
  p.o = ot.ptr; p.d_o = dot.ptr;
  p.o_sb = ot.stride_b; p.o_sh = ot.stride_h; p.o_ss = ot.stride_s;
  p.do_sb = dot.stride_b; p.do_sh = dot.stride_h; p.do_ss = dot.stride_s;
  p.m = m;
  const bool packed = m.mask_kind == FMHA_MASK_CU_SEQLENS, bf = dtype == FMHA_DTYPE_BF16;
  const bool four = packed && static_cast<int64_t>(m.B) * m.H * (m.S_q_pad / 128) * 2 >= 3 * static_cast<int64_t>(sm_count());
  const dim3 grid(static_cast<unsigned>(m.B) * m.H, static_cast<unsigned>(m.S_q_pad / (four ? 128 : 32)));
  auto kfn = four     ? (bf ? bwd_prepare_kernel<true, true, 4> : bwd_prepare_kernel<false, true, 4>)
             : packed ? (bf ? bwd_prepare_kernel<true, true, 1> : bwd_prepare_kernel<false, true, 1>)
                      : (bf ? bwd_prepare_kernel<true, false, 1> : bwd_prepare_kernel<false, false, 1>);
  const cudaError_t e = launch_overlapped(kfn, grid, dim3(256), 0, stream, p);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_bwd_finish(const float* dq_accum, const fmha_tensor4& dq, int B, int H, int S_q, int S_q_pad, int dtype, float scale,
                      const int* cu_seqlens, int total_rows, cudaStream_t stream) {
  FinishArgs f;
  f.dq_accum = dq_accum; f.dq = dq.ptr;
  f.sb = dq.stride_b; f.sh = dq.stride_h; f.ss = dq.stride_s;
  f.B = B; f.H = H; f.S_q = S_q; f.S_q_pad = S_q_pad; f.scale = scale;
  f.cu_seqlens = cu_seqlens; f.total_rows = total_rows;
  const dim3 grid(static_cast<unsigned>(B) * H, static_cast<unsigned>((S_q + kFinishRows - 1) / kFinishRows));
  auto kfn = dtype == FMHA_DTYPE_BF16 ? bwd_finish_kernel<true> : bwd_finish_kernel<false>;
  const cudaError_t e = launch_overlapped(kfn, grid, dim3(256), 0, stream, f);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

}  // namespace fmha
