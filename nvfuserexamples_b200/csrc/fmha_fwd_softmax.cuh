// fmha_fwd_softmax.cuh — what one softmax thread (one query row) does per key step and at the end of a query tile: shared by
// the three forward kernels for compact masks and any number of rows (fmha_fwd_fast_sm100.cu, fmha_fwd_pair_sm100.cu, fmha_fwd_chain_sm100.cu).
#pragma once
#include "fmha_device_utils.cuh"
#include "philox.cuh"
#include "sm100_ptx.cuh"

namespace fmha {

constexpr float kLog2eF = 1.4426950408889634f;
constexpr float kLn2F = 0.6931471805599453f;

// Additive key mask, in the log2 domain: a key at or above kDeadMask may matter (scores of N(0,1) rows are a few units,
// a padding mask is -10000 * log2e), a step with only keys below it is looked at for a shortcut; exp2(x) is zero in fp32,
// flushed subnormals included, for x < -126: kZeroExp leaves a margin for the rounding of the difference.  A step whose mask is
// zero throughout is treated like one without a mask.
enum MaskStep { kMaskZero = 0, kMaskAny = 1, kMaskDead = 2 };
constexpr float kDeadMask = -1000.0f;
constexpr float kZeroExp = -200.0f;
// Floor of a step's row maximum: the lowest float, not -inf, so that a step or a share whose scores are all -inf (an additive
// mask of -inf, or of the lowest float, which becomes -inf times log2 e) gives exponentials of zero, not of -inf - (-inf).  No
// finite score is below it.  (As the start of the running maximum it does the same, but the additive variant at D = 128 then
// spills more: B=32 H=16 S=512 103.7 -> 107.8 us.)
constexpr float kNoScore = -3.402823466e+38f;
// The kind of a step from its mask values, a whole warp holding them (`exists`: the key does).
template <int N>
__device__ __forceinline__ int mask_step_kind(const float (&mk)[N], const bool (&exists)[N]) {
  bool zero = true, dead = true;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    zero &= !exists[i] || mk[i] == 0.f;
    dead &= !exists[i] || mk[i] < kDeadMask;
  }
  return __all_sync(0xffffffffu, zero) ? kMaskZero : __all_sync(0xffffffffu, dead) ? kMaskDead : kMaskAny;
}

// 32 columns of a row: t holds their scores; produces 16 packed 16-bit pairs of exp2(t * sl2 - m_ref) (dropout applied) and
// adds the undropped values to sum2.
template <bool BF16, bool DROP>
__device__ __forceinline__ void softmax_chunk(const uint32_t (&t)[32], float sl2, float neg_m, float2& sum2,
                                              uint32_t (&packed)[16], const uint32_t* keepw) {
  const float2 sl22 = make_float2(sl2, sl2);
  const float2 negm2 = make_float2(neg_m, neg_m);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    float2 x = make_float2(__uint_as_float(t[2 * k]), __uint_as_float(t[2 * k + 1]));
    x = __ffma2_rn(x, sl22, negm2);
    float2 p;
    p.x = fast_exp2(x.x);
    p.y = fast_exp2(x.y);
    sum2 = __fadd2_rn(sum2, p);
    packed[k] = pack2<BF16>(p.x, p.y);
  }
  if constexpr (DROP) {
    // keepw[i]: bit 7 of byte e = keep decision of column 4*i + e; the permutes replicate it over a 16-bit lane
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      packed[2 * i] &= prmt(keepw[i], 0u, 0x9988u);
      packed[2 * i + 1] &= prmt(keepw[i], 0u, 0xBBAAu);
    }
  }
}

// What the keep decisions of a row depend on besides the key.
struct DropRow {
  const PhiloxKeys& keys;
  volatile const uint32_t* offset;   // shared memory: read where a draw starts, so that it holds no register in between
  uint32_t bh, row, thr;
};

// One key step of TN keys: scores from tS, the running maximum and sum, P over the scores, O rescaled where the maximum has
// moved by more than 2^8.  n_cols < TN: the others lie past the end.  KEYADD: `kind` of the step's mask, which mask_stage
// holds in the log2 domain unless it is zero.  wait_s returns when the scores are there; arrive_p(1) hands P to the
// tensor core, or, with P_FIRST > 0, arrive_p(0) its first P_FIRST chunks of 32 columns and arrive_p(1) the rest.  The exponentials
// lie between turn_begin and turn_end.
// FROM: at least so many columns exist.  PAD: P of as many further columns is zero.
template <int D, int TN, bool BF16, bool KEYADD, bool DROP, int P_FIRST, int FROM, int PAD, class WaitS, class ArriveP, class TurnBegin, class TurnEnd>
__device__ __forceinline__ void softmax_step(uint32_t tS, uint32_t tO, int key0, int n_cols, float sl2, const float* mask_stage, int kind,
                                             const DropRow& dr, float& m_ref, float2& sum2, const WaitS& wait_s, const ArriveP& arrive_p,
                                             const TurnBegin& turn_begin, const TurnEnd& turn_end) {
  // The look at a dead step can only succeed where every row's maximum so far is that of a live key; before the first of them (left
  // padding) the step is done like any other at once, without a second reading and maximum (lengths U[0.05 S, 0.1 S], padding on the
  // left: B=64 H=16 S=384 D = 64 89.7 -> 82.7 us, with dropout 130.6 -> 117.2; B=1 H=12 S=2048 D = 128 52.4 -> 47.8).
  if constexpr (KEYADD) {
    if (kind == kMaskDead && __any_sync(0xffffffffu, !(m_ref > kDeadMask))) kind = kMaskAny;
  }
  // Keep decisions of this step's TN columns: Philox does not depend on the scores, so it runs
  // before they are awaited, while the tensor core is still busy with Q K^T.
  [[maybe_unused]] uint32_t keepw[DROP ? TN / 4 : 1];
  auto draw_keep_words = [&]() {
    const uint32_t kb0 = static_cast<uint32_t>(key0 / 16);
    const uint32_t poff = *dr.offset;
#pragma unroll
    for (int d = 0; d < TN / 16; ++d) {
      const U4 draw = dropout_draw_keys(dr.keys, poff, dr.bh, dr.row, kb0 + d);
      keepw[d * 4 + 0] = (draw.x & 0x7F7F7F7Fu) + (0x80u - dr.thr) * 0x01010101u;
      keepw[d * 4 + 1] = (draw.y & 0x7F7F7F7Fu) + (0x80u - dr.thr) * 0x01010101u;
      keepw[d * 4 + 2] = (draw.z & 0x7F7F7F7Fu) + (0x80u - dr.thr) * 0x01010101u;
      keepw[d * 4 + 3] = (draw.w & 0x7F7F7F7Fu) + (0x80u - dr.thr) * 0x01010101u;
    }
  };
[[maybe_unused]] draw_and_look:
  if constexpr (DROP) {
    if (!KEYADD || kind != kMaskDead) draw_keep_words();
  }
  wait_s();
  tc_fence_after_sync();

  // ---- scores into registers (raw, or scaled and masked with an additive mask), row maximum --------------------
  // Without dropout they stay there until they are exponentiated.  With dropout the step's keep words are live as well:
  // the scores are read a second time, 32 columns at a time (held, they spilled more and cost 57.2 against 55.7 us at B=32
  // H=12 S=512).
  constexpr bool HOLD = !DROP;
  // Mask and dropout, D = 128: the scores with the mask added go back to tensor memory for the second reading, which needs neither the mask
  // nor the choice then (a mask that is nowhere zero, B=32 H=16 S=512 145.7 -> 137.0 us, S_q=102 S_k=449 18.5 -> 15.3; right padding 126.5 ->
  // 121.3; at D = 64, four CTAs per SM, the stores cost more than they spare: S=1024 188.8 -> 191.0).
  constexpr bool REWRITE = KEYADD && DROP && D == 128;
  const float mul = KEYADD && kind == kMaskAny ? 1.0f : sl2;   // what takes a score as held to the log2 domain
  auto finish_scores = [&](int c, uint32_t (&v)[32]) {   // mask added, keys past the end to -inf (exp2 makes them zero)
    if (KEYADD && kind == kMaskAny) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float4 mk = *reinterpret_cast<const float4*>(mask_stage + c * 32 + 4 * k);
        const float2 sl22 = make_float2(sl2, sl2);
        const float2 t0 = __ffma2_rn(make_float2(__uint_as_float(v[4 * k]), __uint_as_float(v[4 * k + 1])), sl22, make_float2(mk.x, mk.y));
        const float2 t1 = __ffma2_rn(make_float2(__uint_as_float(v[4 * k + 2]), __uint_as_float(v[4 * k + 3])), sl22, make_float2(mk.z, mk.w));
        v[4 * k] = __float_as_uint(t0.x);
        v[4 * k + 1] = __float_as_uint(t0.y);
        v[4 * k + 2] = __float_as_uint(t1.x);
        v[4 * k + 3] = __float_as_uint(t1.y);
      }
    }
    if (c * 32 + 32 > FROM && n_cols < TN) {
#pragma unroll
      for (int k = 0; k < 32; ++k)
        if (c * 32 + k >= n_cols) v[k] = __float_as_uint(-INFINITY);
    }
  };
  uint32_t sv[TN / 32][32];
  // The maximum of 32 columns is taken while the next 32 are on their way (D = 128: B=16 H=16 S=1024 163.1 -> 161.6 us, S=512
  // with dropout 57.5 -> 56.1; with an additive mask B=64 H=16 S=384 D = 64 67.6 -> 66.7).  Not with mask and dropout at D = 64, where the
  // 96 registers hold one 32 columns beside the keep words (76 -> 24 bytes of spill stores; lengths U[0.4 S, S], B=16 H=16 S=1024 143 -> 130 us,
  // a mask that is nowhere zero 188.6 -> 170.6).
  constexpr bool AHEAD = !(KEYADD && DROP && D == 64);
  // All at once with a mask and the scores held at D = 128 in 168 registers (a mask that is nowhere zero, B=5 H=8 S=528 18.9 -> 18.1 us, B=2 H=12
  // S=1331 35.4 -> 34.1); the kernel of two tiles per CTA has 216 and is faster without (B=16 H=16 S=2048 475 / 493).
  constexpr bool ALL = KEYADD && HOLD && D == 128 && P_FIRST == 0;
#pragma unroll
  for (int c = 0; c < (ALL ? TN / 32 : 1); ++c) tmem_ld32(tS + c * 32, sv[c]);
#pragma unroll
  for (int c = 0; c < (ALL ? TN / 32 : 1); ++c) tmem_wait_ld_dep(sv[c]);
  float tile_max = kNoScore;
#pragma unroll
  for (int c = 0; c < TN / 32; ++c) {
    if (AHEAD && !ALL && c + 1 < TN / 32) tmem_ld32(tS + (c + 1) * 32, sv[c + 1]);
    finish_scores(c, sv[c]);
    if constexpr (REWRITE) {
      if (kind == kMaskAny || n_cols < TN) tmem_st32(tS + c * 32, sv[c]);
    }
    auto v = [&](int k) { return __uint_as_float(sv[c][k]); };
    // with an additive mask a NaN has to show in the maximum, or the shortcut below would step over it
    auto max3 = [](float x, float y, float z) { return fmax3<KEYADD>(x, y, z); };
    float m0 = max3(v(0), v(1), v(2));
    float m1 = max3(v(3), v(4), v(5));
#pragma unroll
    for (int k = 6; k + 3 < 32; k += 4) {
      m0 = max3(m0, v(k), v(k + 1));
      m1 = max3(m1, v(k + 2), v(k + 3));
    }
    tile_max = max3(tile_max, max3(m0, m1, v(30)), v(31));
    if (!ALL && c + 1 < TN / 32) {
      if (!AHEAD) tmem_ld32(tS + (c + 1) * 32, sv[c + 1]);
      tmem_wait_ld_dep(sv[c + 1]);
    }
  }
  tile_max = fmax3<KEYADD>(tile_max * mul, kNoScore, kNoScore);   // scale > 0: the maximum commutes with it; the floor may have passed the range
  // A step whose keys are all masked away (the padded end of a sequence): when every score of it lies so far below
  // the reference maximum that its exponential is zero in fp32, P is zero and nothing else changes.  Decided on the
  // scores themselves, so the result is the same bits; a third of the steps of a batch with lengths in [S/3, S].
  if constexpr (KEYADD) {
    if (kind == kMaskDead && __all_sync(0xffffffffu, tile_max + kDeadMask - m_ref < kZeroExp)) {   // every mask value is below kDeadMask
      turn_begin();
      turn_end();
      const uint32_t zero[16] = {};
#pragma unroll
      for (int c = 0; c < (TN + PAD) / 32; ++c) tmem_st16(tS + c * 16, zero);
      tmem_wait_st();
      tc_fence_before_sync();
      if (P_FIRST > 0) arrive_p(0);
      arrive_p(1);
      return;
    }
    if (kind == kMaskDead) {   // rare, and a second copy of what came before costs every step
      kind = kMaskAny;
      goto draw_and_look;
    }
  }
  // ---- running reference maximum, lazy rescale of O ------------------------------------
  {
    float m_new = fmaxf(m_ref, tile_max);
    if (m_ref != -INFINITY && m_new - m_ref <= 8.0f) m_new = m_ref;  // exponentials stay below 2^8
    const bool moved = (m_new != m_ref) && (m_ref != -INFINITY);
    const float alpha = (m_ref == -INFINITY) ? 0.f : fast_exp2(m_ref - m_new);
    if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
      for (int c = 0; c < D / 8; ++c) {   // eight columns at a time: the scores of the step stay in registers meanwhile
        uint32_t r[8];
        tmem_ld8(tO + c * 8, r);
        tmem_wait_ld_dep8(r);
#pragma unroll
        for (int k = 0; k < 8; ++k) r[k] = __float_as_uint(__uint_as_float(r[k]) * alpha);
        tmem_st8(tO + c * 8, r);
      }
    }
    sum2.x *= alpha;
    sum2.y *= alpha;
    m_ref = m_new;
  }
  turn_begin();
  // ---- exponentials, dropout, P over S ---------------------------------------------------------------------
  auto hand_over = [&](int c) {   // after 32-column chunk c
    if (PAD == 0 && c + 1 == P_FIRST) {
      tmem_wait_st();
      tc_fence_before_sync();
      arrive_p(0);
    }
  };
  if constexpr (HOLD) {
#pragma unroll
    for (int c = 0; c < TN / 32; ++c) {
      uint32_t packed[16];
      softmax_chunk<BF16, DROP>(sv[c], mul, -m_ref, sum2, packed, keepw);
      tmem_st16(tS + c * 16, packed);
      hand_over(c);
    }
  } else if constexpr (TN == 32) {
    uint32_t packed[16];
    softmax_chunk<BF16, DROP>(sv[0], mul, -m_ref, sum2, packed, keepw);
    tmem_st16(tS, packed);
  } else {
    uint32_t ra[32], rb[32], packed[16];   // chunk c+1 (then c+2) is in flight while chunk c (c+1) is processed
    if constexpr (REWRITE) tmem_wait_st();
    tmem_ld32(tS, ra);
#pragma unroll
    for (int c = 0; c < TN / 32; c += 2) {
      tmem_wait_ld_dep(ra);
      if constexpr (!REWRITE) finish_scores(c, ra);
      tmem_ld32(tS + (c + 1) * 32, rb);
      softmax_chunk<BF16, DROP>(ra, mul, -m_ref, sum2, packed, keepw + (DROP ? c * 8 : 0));
      tmem_st16(tS + c * 16, packed);
      hand_over(c);
      tmem_wait_ld_dep(rb);
      if constexpr (!REWRITE) finish_scores(c + 1, rb);
      if (c + 2 < TN / 32) tmem_ld32(tS + (c + 2) * 32, ra);
      softmax_chunk<BF16, DROP>(rb, mul, -m_ref, sum2, packed, keepw + (DROP ? c * 8 + 8 : 0));
      tmem_st16(tS + c * 16 + 16, packed);
      hand_over(c + 1);
    }
  }
  if constexpr (PAD > 0) {
    const uint32_t zero[16] = {};
#pragma unroll
    for (int c = TN / 32; c < (TN + PAD) / 32; ++c) tmem_st16(tS + c * 16, zero);
  }
  turn_end();
  tmem_wait_st();
  tc_fence_before_sync();
  if (PAD > 0 && P_FIRST > 0) arrive_p(0);
  arrive_p(1);
}

// A 64-key step at head dimension 64.  The last one of a tile may have 32 keys or fewer (one in two, where lengths are spread): then
// only its first half is read, drawn for and exponentiated, and a longer one looks for keys past the end in its second half alone
// (kernel times, a CTA per tile: B=32 S=512 with dropout, lengths U[256, 512] 12 heads 50.1 -> 46.9 us, 16 heads 64.0 -> 59.8, B=16 H=8 S=160 8.3 -> 7.1,
// B=13 H=12 S=197 without 8.6 -> 8.3; few keys split over a cluster, 449 with lengths 7.20 -> 7.34).  Not with an
// additive mask, which has such a step only where S_k is no multiple of 64, and registers to spare for a second copy nowhere (B=64 H=16 S=384
// 65.8 -> 67.7).
template <bool BF16, bool KEYADD, bool DROP, class WaitS, class ArriveP>
__device__ __forceinline__ void softmax_step_64(uint32_t tS, uint32_t tO, int key0, int n_cols, float sl2, const float* mask_stage, int kind,
                                                const DropRow& dr, float& m_ref, float2& sum2, const WaitS& wait_s, const ArriveP& arrive_p) {
  auto none = [] {};
  if constexpr (KEYADD) softmax_step<64, 64, BF16, KEYADD, DROP, 0, 0, 0>(tS, tO, key0, n_cols, sl2, mask_stage, kind, dr, m_ref, sum2, wait_s, arrive_p, none, none);
  else if (n_cols > 32) softmax_step<64, 64, BF16, KEYADD, DROP, 0, 32, 0>(tS, tO, key0, n_cols, sl2, mask_stage, kind, dr, m_ref, sum2, wait_s, arrive_p, none, none);
  else softmax_step<64, 32, BF16, KEYADD, DROP, 0, 0, 32>(tS, tO, key0, n_cols, sl2, mask_stage, kind, dr, m_ref, sum2, wait_s, arrive_p, none, none);
}

// The same at head dimension 128, 128 keys a step and 64 to the half (kernel times: S=64 without a mask B=8 H=12 5.3 -> 4.5 us, with dropout
// B=36 H=16 14.1 -> 10.2; lengths with dropout B=16 H=8 S=640 packed 37.5 -> 33.8, B=10 H=8 S=2048 140 -> 134; without, two tiles per CTA,
// B=16 H=16 S=300 25.8 -> 24.0, B=12 H=12 S=2048 212 -> 210; of 90 sizes none slower).  With an additive mask as well, which gains here even
// where no last step is short: B=98 H=16 S=256 108 -> 104, B=64 H=16 S=384 133 -> 127, S=160 B=34 H=8 18.0 -> 15.8.  With mask and dropout, whose spills
// it raises from 116 to 140 bytes: B=36 H=16 S=64 15.7 -> 11.6, S=160 B=34 H=8 21.2 -> 18.1, S=300 B=12 H=12 25.6 -> 23.9, S=384 and more 0.94 to 1.00 of the time,
// one whole step on a small grid 6.03 -> 6.15, keys split over a cluster 0.91 to 1.04.
template <bool BF16, bool KEYADD, bool DROP, int P_FIRST, class WaitS, class ArriveP, class TurnBegin, class TurnEnd>
__device__ __forceinline__ void softmax_step_128(uint32_t tS, uint32_t tO, int key0, int n_cols, float sl2, const float* mask_stage, int kind,
                                                 const DropRow& dr, float& m_ref, float2& sum2, const WaitS& wait_s, const ArriveP& arrive_p,
                                                 const TurnBegin& turn_begin, const TurnEnd& turn_end) {
  if (n_cols > 64)
    softmax_step<128, 128, BF16, KEYADD, DROP, P_FIRST, 64, 0>(tS, tO, key0, n_cols, sl2, mask_stage, kind, dr, m_ref, sum2, wait_s, arrive_p, turn_begin, turn_end);
  else
    softmax_step<128, 64, BF16, KEYADD, DROP, P_FIRST, 0, 64>(tS, tO, key0, n_cols, sl2, mask_stage, kind, dr, m_ref, sum2, wait_s, arrive_p, turn_begin, turn_end);
}

// O of a finished query tile out of tensor memory, scaled and rounded: into `tile` (shared memory, 128 rows in the swizzled
// layout of the O tensor map), or, where the tile reaches into rows that are not its own, the valid rows straight to `grow`.
template <int D, bool BF16>
__device__ __forceinline__ void o_tile_out(uint32_t tO, float out_scale, uint8_t* tile, int row, bool by_rows, bool row_ok,
                                           unsigned short* grow) {
#pragma unroll
  for (int c = 0; c < D / 32; ++c) {
    uint32_t r[32];
    tmem_ld32(tO + c * 32, r);
    tmem_wait_ld_dep(r);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint4 w;
      w.x = pack2<BF16>(__uint_as_float(r[q * 8 + 0]) * out_scale, __uint_as_float(r[q * 8 + 1]) * out_scale);
      w.y = pack2<BF16>(__uint_as_float(r[q * 8 + 2]) * out_scale, __uint_as_float(r[q * 8 + 3]) * out_scale);
      w.z = pack2<BF16>(__uint_as_float(r[q * 8 + 4]) * out_scale, __uint_as_float(r[q * 8 + 5]) * out_scale);
      w.w = pack2<BF16>(__uint_as_float(r[q * 8 + 6]) * out_scale, __uint_as_float(r[q * 8 + 7]) * out_scale);
      if (by_rows) {
        if (row_ok) *reinterpret_cast<uint4*>(grow + c * 32 + q * 8) = w;
      } else {
        *reinterpret_cast<uint4*>(tile + (c / 2) * 16384 + sw128_offset(row, (c % 2) * 4 + q)) = w;
      }
    }
  }
}

}  // namespace fmha
