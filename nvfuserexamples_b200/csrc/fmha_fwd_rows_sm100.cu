// fmha_fwd_rows_sm100.cu — forward kernel for at most 16 query rows per head: new rows against keys and values computed
// before ("decode"), cross-attention of a short query.  Same inputs, masks, dropout bits and outputs as the production
// kernel in fmha_fwd_fast_sm100.cu.
//
// Bound: every key and value is used by at most 16 query rows, 16 flops per byte at S_q = 16, so the time is what it
// takes to bring K and V in; a 128-row tcgen05 tile would spend 7/8 of its exponentials and most of a key step's
// latency chain on rows that do not exist (1.9 us per 128 keys, measured).  Hence: m16n8k16 MMAs from registers, which
// fit the row count exactly and need no tensor-memory round trip; each of the four consumer warps takes 16 of every 64
// keys and runs its own online softmax, so no warp waits for another one inside the key loop; a producer warp keeps
// three (D = 64: six) 64-key stages of K and V in flight through TMA, about 190 KB per SM with two CTAs; the key steps of
// a head are dealt out over a cluster of up to eight CTAs, whose shares meet through distributed shared memory.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "../../include/fmha_sm100.h"
#include "fmha_device_utils.cuh"
#include "fmha_kernel_args.h"
#include "philox.cuh"
#include "sm100_ptx.cuh"

namespace fmha {

namespace {

constexpr int kRwRows = 16;                 // query rows of one MMA tile
constexpr int kRwWarps = 4;                 // consumer warps, 16 keys of a step each
constexpr int kRwThreads = 32 * (kRwWarps + 1);
constexpr int kRwMaxSplit = 8;              // portable cluster size
constexpr float kRwLog2e = 1.4426950408889634f;
constexpr float kRwLn2 = 0.6931471805599453f;

enum RwWaitSite { kRwFull = 161, kRwEmpty = 162 };

template <int D>
struct RwSmem {
  static constexpr int kTile = kRowsKeyStep * D * 2;      // K or V of a step
  static constexpr int kSub = kRowsKeyStep * 128;         // its 64-column sub-tile (128-byte swizzle)
  static constexpr int kStages = D == 64 ? 6 : 3;
  static constexpr int kOffBar = kStages * 2 * kTile;
  static constexpr int kOffMisc = kOffBar + 2 * kStages * 8;
  static constexpr int kBytes = kOffMisc + 16;
  static constexpr int kDynBytes = kBytes + 1024;
  // after the key loop, over the stages: O shares of the four warps and of the CTA, [16][D + 8] fp32 each (the padding
  // spreads the rows over the banks), and their row statistics
  static constexpr int kRowFloats = D + 8;
  static constexpr int kShare = kRwRows * kRowFloats * 4;
  static constexpr int kOffStats = (kRwWarps + 1) * kShare;
  static_assert(kOffStats + (kRwWarps + 1) * kRwRows * 8 <= kOffBar, "the shares fit over the stages");
};

template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(saddr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(saddr)
               : "memory");
}

}  // namespace

template <int D, bool BF16, bool KEYADD, bool DROP>
__global__ void __launch_bounds__(kRwThreads, 2) fmha_fwd_rows_kernel(const __grid_constant__ FwdArgs a) {
  griddep_wait();
  using L = RwSmem<D>;
  constexpr int ST = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kOffBar);   // [ST] K and V of a step have landed
  uint64_t* empty = full + ST;                                       // [ST] ... and the four consumer warps are done with them
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc);
  const WaitCtx wctx{abort_flag, a.status};

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int h = blockIdx.y, b = blockIdx.z;
  const int bh = b * a.H + h;
  const int n_split = static_cast<int>(gridDim.x);   // the cluster spans the grid's x axis
  const int split = static_cast<int>(blockIdx.x);
  int k_limit = a.S_k;
  if (a.mask_kind == FMHA_MASK_SEQLEN) {
    const int len = reinterpret_cast<const int*>(a.mask)[b];
    if (len > 0 && len < a.S_k) k_limit = len;
  }
  // this CTA's key steps; possibly none
  const int n_all = (k_limit + kRowsKeyStep - 1) / kRowsKeyStep;
  const int j0 = n_all * split / n_split, j1 = n_all * (split + 1) / n_split;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < ST; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, kRwWarps);
    }
    mbar_fence_init();
  }
  __syncthreads();

  const int g = lane >> 2, t = lane & 3;   // this thread's MMA rows are g and g + 8, its columns 2t and 2t + 1 of every 8
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

  if (warp == kRwWarps) {
    // ============================ TMA producer ======================================
    if (lane == 0) {
      for (int j = j0; j < j1; ++j) {
        const int i = j - j0, s = i % ST;
        if (i >= ST) mbar_wait(empty + s, (i / ST - 1) & 1, wctx, kRwEmpty);
        mbar_arrive_expect_tx(full + s, 2 * L::kTile);
        uint8_t* k = smem + s * 2 * L::kTile;
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_4d(k + c * L::kSub, &a.tm_k, full + s, c * 64, j * kRowsKeyStep, h, b);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_4d(k + L::kTile + c * L::kSub, &a.tm_v, full + s, c * 64, j * kRowsKeyStep, h, b);
      }
    }
  } else {
    // ============================ consumers =========================================
    // Q fragments of the 16 rows (rows past S_q are zeros)
    uint32_t qf[D / 16][4];
    {
      const unsigned short* q = reinterpret_cast<const unsigned short*>(a.q_ptr) + b * a.q_sb + h * a.q_sh;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = g + (e & 1) * 8, col = ks * 16 + (e >> 1) * 8 + 2 * t;
          qf[ks][e] = row < a.S_q ? __ldg(reinterpret_cast<const unsigned int*>(q + row * a.q_ss + col)) : 0u;
        }
    }
    const uint32_t poff = DROP ? a.philox_offset + (a.philox_offset_dev != nullptr ? static_cast<uint32_t>(*a.philox_offset_dev) : 0u) : 0u;
    const uint32_t gbh = static_cast<uint32_t>(a.philox_bh_offset + bh);
    const float sl2 = a.scale_log2;
    // ldmatrix: lane (mi, r) addresses row r of 8x8 block mi
    const int mi = lane >> 3, r = lane & 7;
    const int k_row = warp * 16 + (mi >> 1) * 8 + r, k_ch = mi & 1;   // K blocks: (keys lo, dims lo), (lo, hi), (hi, lo), (hi, hi)
    const int v_row = warp * 16 + (mi & 1) * 8 + r, v_ch = mi >> 1;   // V blocks, transposed: (keys lo, dims lo), (hi, lo), ...

    for (int j = j0; j < j1; ++j) {
      const int i = j - j0, s = i % ST;
      const int key0 = j * kRowsKeyStep + warp * 16;   // this warp's 16 keys
      float madd[2][2];
      if constexpr (KEYADD) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int key = key0 + nt * 8 + 2 * t + e;
            madd[nt][e] = key < a.S_k ? __ldg(reinterpret_cast<const float*>(a.mask) + static_cast<size_t>(b) * a.S_k + key) * kRwLog2e : 0.f;
          }
      }
      uint32_t keep[2][2];   // dropout: 16-bit lane masks of the packed pairs, [row half][n tile]
      if constexpr (DROP) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const U4 d = dropout_draw_keys(a.philox_keys, poff, gbh, static_cast<uint32_t>(g + hf * 8), static_cast<uint32_t>(key0 / 16));
          // keys 2t, 2t+1 and 8 + 2t, 9 + 2t of the 16: bytes 2(t&1), +1 of words t/2 and 2 + t/2
          const uint32_t w0 = dropout_keep_bits(t < 2 ? d.x : d.y, a.philox_thr), w1 = dropout_keep_bits(t < 2 ? d.z : d.w, a.philox_thr);
          const uint32_t sel = (t & 1) ? 0xBBAAu : 0x9988u;
          keep[hf][0] = prmt(w0, 0u, sel);
          keep[hf][1] = prmt(w1, 0u, sel);
        }
      }
      mbar_wait(full + s, (i / ST) & 1, wctx, kRwFull);
      if (key0 < k_limit) {
        const uint32_t sk = smem_u32(smem + s * 2 * L::kTile), sv = sk + L::kTile;
        float sc[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          uint32_t kf[4];
          ldmatrix_x4(kf, sk + (ks / 4) * L::kSub + sw128_offset(k_row, (ks % 4) * 2 + k_ch));
          mma_16816<BF16>(sc[0], qf[ks], kf[0], kf[1]);
          mma_16816<BF16>(sc[1], qf[ks], kf[2], kf[3]);
        }
        // scaled and masked scores in the log2 domain
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float x = sc[nt][e] * sl2;
            if constexpr (KEYADD) x = fmaf(sc[nt][e], sl2, madd[nt][e & 1]);
            if (key0 + nt * 8 + 2 * t + (e & 1) >= k_limit) x = -INFINITY;
            sc[nt][e] = x;
          }
        uint32_t p[4];
        float alpha[2];
        bool moved = false;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          float mx = fmaxf(fmaxf(sc[0][2 * hf], sc[0][2 * hf + 1]), fmaxf(sc[1][2 * hf], sc[1][2 * hf + 1]));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
          float m_new = fmaxf(m[hf], mx);
          if (m[hf] != -INFINITY && m_new - m[hf] <= 8.0f) m_new = m[hf];   // lazy: exponentials stay below 2^8
          alpha[hf] = m_new == m[hf] ? 1.0f : fast_exp2(m[hf] - m_new);
          moved |= m_new != m[hf];
          m[hf] = m_new;
          const float neg_m = m_new == -INFINITY ? 0.f : -m_new;   // only keys masked with -inf so far
          float e[2][2];
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int c = 0; c < 2; ++c) e[nt][c] = fast_exp2(sc[nt][2 * hf + c] + neg_m);
          l[hf] = l[hf] * alpha[hf] + ((e[0][0] + e[0][1]) + (e[1][0] + e[1][1]));
          p[hf] = pack2<BF16>(e[0][0], e[0][1]);
          p[2 + hf] = pack2<BF16>(e[1][0], e[1][1]);
          if constexpr (DROP) {
            p[hf] &= keep[hf][0];
            p[2 + hf] &= keep[hf][1];
          }
        }
        if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
          for (int nt = 0; nt < D / 8; ++nt) {
            o[nt][0] *= alpha[0];
            o[nt][1] *= alpha[0];
            o[nt][2] *= alpha[1];
            o[nt][3] *= alpha[1];
          }
        }
#pragma unroll
        for (int np = 0; np < D / 16; ++np) {
          uint32_t vf[4];
          ldmatrix_x4_trans(vf, sv + (np / 4) * L::kSub + sw128_offset(v_row, (np % 4) * 2 + v_ch));
          mma_16816<BF16>(o[2 * np], p, vf[0], vf[1]);
          mma_16816<BF16>(o[2 * np + 1], p, vf[2], vf[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty + s);
    }
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      l[hf] += __shfl_xor_sync(0xffffffffu, l[hf], 1);
      l[hf] += __shfl_xor_sync(0xffffffffu, l[hf], 2);
    }
  }
  __syncthreads();   // every stage has been read: the shares may overwrite them

  // ============================ combine ===============================================
  float2* stats = reinterpret_cast<float2*>(smem + L::kOffStats);   // [5][16] (maximum, sum)
  if (warp < kRwWarps) {
    float* share = reinterpret_cast<float*>(smem + warp * L::kShare);
#pragma unroll
    for (int nt = 0; nt < D / 8; ++nt) {
      *reinterpret_cast<float2*>(share + g * L::kRowFloats + nt * 8 + 2 * t) = make_float2(o[nt][0], o[nt][1]);
      *reinterpret_cast<float2*>(share + (g + 8) * L::kRowFloats + nt * 8 + 2 * t) = make_float2(o[nt][2], o[nt][3]);
    }
    if (t == 0) {
      stats[warp * kRwRows + g] = make_float2(m[0], l[0]);
      stats[warp * kRwRows + g + 8] = make_float2(m[1], l[1]);
    }
  }
  __syncthreads();
  // Work: (row, 8 columns).  `read` gives share k's statistics of the row or its 8 columns.
  auto finish = [&](int row, int ch, float m_all, float l_all, const float (&acc)[8]) {
    const float out_scale = (DROP ? a.dropout_scale : 1.0f) / l_all;
    uint4 w;
    w.x = pack2<BF16>(acc[0] * out_scale, acc[1] * out_scale);
    w.y = pack2<BF16>(acc[2] * out_scale, acc[3] * out_scale);
    w.z = pack2<BF16>(acc[4] * out_scale, acc[5] * out_scale);
    w.w = pack2<BF16>(acc[6] * out_scale, acc[7] * out_scale);
    *reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(a.o_ptr) + b * a.o_sb + h * a.o_sh + row * a.o_ss + ch * 8) = w;
    if (ch == 0 && a.lse != nullptr) a.lse[static_cast<size_t>(bh) * a.S_q + row] = (m_all + fast_log2(l_all)) * kRwLn2;
  };
  const int items = *abort_flag ? 0 : a.S_q * (D / 8);
  for (int i = threadIdx.x; i < items; i += kRwThreads) {   // over the four warps
    const int row = i / (D / 8), ch = i % (D / 8);
    float m_all = -INFINITY, l_all = 0.f, acc[8] = {};
#pragma unroll
    for (int k = 0; k < kRwWarps; ++k) m_all = fmaxf(m_all, stats[k * kRwRows + row].x);
#pragma unroll
    for (int k = 0; k < kRwWarps; ++k) {
      const float2 st = stats[k * kRwRows + row];
      const float w = st.x == -INFINITY ? 0.f : fast_exp2(st.x - m_all);   // a warp without keys
      l_all = fmaf(w, st.y, l_all);
      const float4* src = reinterpret_cast<const float4*>(smem + k * L::kShare + (row * L::kRowFloats + ch * 8) * 4);
      const float4 x = src[0], y = src[1];
      acc[0] = fmaf(w, x.x, acc[0]); acc[1] = fmaf(w, x.y, acc[1]); acc[2] = fmaf(w, x.z, acc[2]); acc[3] = fmaf(w, x.w, acc[3]);
      acc[4] = fmaf(w, y.x, acc[4]); acc[5] = fmaf(w, y.y, acc[5]); acc[6] = fmaf(w, y.z, acc[6]); acc[7] = fmaf(w, y.w, acc[7]);
    }
    if (n_split == 1) {
      finish(row, ch, m_all, l_all, acc);
    } else {
      float4* dst = reinterpret_cast<float4*>(smem + kRwWarps * L::kShare + (row * L::kRowFloats + ch * 8) * 4);
      dst[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      dst[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
      if (ch == 0) stats[kRwWarps * kRwRows + row] = make_float2(m_all, l_all);
    }
  }
  if (n_split > 1) {
    cluster_sync();
    const uint32_t share0 = smem_u32(smem + kRwWarps * L::kShare), stats0 = smem_u32(stats + kRwWarps * kRwRows);
    for (int i = split * kRwThreads + threadIdx.x; i < items; i += n_split * kRwThreads) {   // over the cluster's CTAs
      const int row = i / (D / 8), ch = i % (D / 8);
      float mk[kRwMaxSplit], lk[kRwMaxSplit];
      float m_all = -INFINITY, l_all = 0.f, acc[8] = {};
#pragma unroll
      for (int k = 0; k < kRwMaxSplit; ++k) {
        const float2 st = k < n_split ? dsmem_ld2(dsmem_map(stats0 + row * 8, k)) : make_float2(-INFINITY, 0.f);
        mk[k] = st.x;
        lk[k] = st.y;
        m_all = fmaxf(m_all, mk[k]);
      }
#pragma unroll
      for (int k = 0; k < kRwMaxSplit; ++k) {
        if (k >= n_split) break;
        const float w = mk[k] == -INFINITY ? 0.f : fast_exp2(mk[k] - m_all);   // a CTA without key steps
        l_all = fmaf(w, lk[k], l_all);
        const uint32_t src = dsmem_map(share0 + (row * L::kRowFloats + ch * 8) * 4, k);
        const float4 x = dsmem_ld4(src), y = dsmem_ld4(src + 16);
        acc[0] = fmaf(w, x.x, acc[0]); acc[1] = fmaf(w, x.y, acc[1]); acc[2] = fmaf(w, x.z, acc[2]); acc[3] = fmaf(w, x.w, acc[3]);
        acc[4] = fmaf(w, y.x, acc[4]); acc[5] = fmaf(w, y.y, acc[5]); acc[6] = fmaf(w, y.z, acc[6]); acc[7] = fmaf(w, y.w, acc[7]);
      }
      finish(row, ch, m_all, l_all, acc);
    }
    cluster_sync();   // no CTA leaves while another one reads its shared memory
  }
  if (*abort_flag) {
    for (int k = 0; k < 20; ++k) __nanosleep(1000000);   // copies in flight end before the CTA does
    __syncthreads();
  }
}

// Up to 16 rows, but not where so many heads have so few keys that a CTA here is mostly start and end: at D = 64 four CTAs of the
// tile kernel share an SM, two of this one.  The lines lie where the two cross (this kernel / the tile kernel, us): 16 rows, 64
// keys 1024 heads 10.8 / 9.9, 2048 18.8 / 16.3, 8192 76.8 / 57.3; 128 keys 2048 heads 21.9 / 21.8, 4096 47.2 / 41.6; 256 keys 4096
// heads 61.2 / 62.2; 8 rows, 64 keys 2048 heads 16.8 / 16.2; 4 rows 15.8 / 16.2, 8192 heads (more than the L2 cache) 68.1 / 57.8.
// With dropout the tile kernel draws for 128 rows: 8 rows, 64 keys, 4096 heads 0.97 times its time, 16 rows 1.11 times.
bool fwd_rows_applies(int S_q, int S_k, int D, int64_t heads, bool dropout) {
  if (S_q > kRwRows) return false;
  const int steps = (S_k + kRowsKeyStep - 1) / kRowsKeyStep;
  const int64_t per_sm = heads / std::max(sm_count(), 1);
  if (D != 64 || steps > (dropout ? 1 : 3)) return true;
  return S_q <= (dropout ? 8 : 4) ? S_k <= 32 || per_sm < 32 || steps > 1 : per_sm < 8 * steps;
}

template <int D, bool BF16, bool KEYADD, bool DROP>
static int launch_rows_impl(const FwdArgs& a, cudaStream_t stream) {
  using L = RwSmem<D>;
  auto kfn = fmha_fwd_rows_kernel<D, BF16, KEYADD, DROP>;
  static std::atomic<bool> configured[64] = {};   // per device; set after the attribute call succeeded
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  // Shares per head: enough CTAs for two on every SM (their stages together keep the memory busy), but at least two key
  // steps each, below which a share's start-up and the combination outweigh its loads.
  const int64_t heads = static_cast<int64_t>(a.B) * a.H;
  const int steps = (a.S_k + kRowsKeyStep - 1) / kRowsKeyStep;
  int n_split = 1;
  while (n_split < kRwMaxSplit && heads * n_split * 2 <= 2 * static_cast<int64_t>(sm_count()) && steps >= 4 * n_split) n_split *= 2;
  const cudaError_t e = launch_overlapped(kfn, dim3(n_split, a.H, a.B), dim3(kRwThreads), L::kDynBytes, stream, a, n_split > 1 ? n_split : 0);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

int launch_fwd_rows(const FwdArgs& a, int D, int dtype, cudaStream_t stream) {
  const bool bf = dtype == FMHA_DTYPE_BF16;
  const bool keyadd = a.mask_kind == FMHA_MASK_KEY_ADDITIVE;
  const bool drop = a.dropout_kind == FMHA_DROPOUT_PHILOX;
#define FMHA_ROWS_CASE(DD, BF, KA, DR) \
  if (D == DD && bf == BF && keyadd == KA && drop == DR) return launch_rows_impl<DD, BF, KA, DR>(a, stream);
#define FMHA_ROWS_CASES(DD, BF) \
  FMHA_ROWS_CASE(DD, BF, false, false) FMHA_ROWS_CASE(DD, BF, false, true) FMHA_ROWS_CASE(DD, BF, true, false) FMHA_ROWS_CASE(DD, BF, true, true)
  FMHA_ROWS_CASES(64, false)
  FMHA_ROWS_CASES(64, true)
  FMHA_ROWS_CASES(128, false)
  FMHA_ROWS_CASES(128, true)
#undef FMHA_ROWS_CASES
#undef FMHA_ROWS_CASE
  return static_cast<int>(cudaErrorInvalidValue);
}

}  // namespace fmha
