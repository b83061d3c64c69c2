// fmha_device_utils.cuh — small device helpers shared by the forward and backward kernels:
// 16-bit packing for fp16 / bf16, byte permutes, and row-segment loads/stores of the dense
// [B*H, S_q, S_k] tensors the legacy operators use.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace fmha {

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}
template <bool BF16>
__device__ __forceinline__ float unpack_lo(uint32_t v) {
  if constexpr (BF16) return __uint_as_float(v << 16);
  else return __half2float(__ushort_as_half(static_cast<unsigned short>(v & 0xffff)));
}
template <bool BF16>
__device__ __forceinline__ float unpack_hi(uint32_t v) {
  if constexpr (BF16) return __uint_as_float(v & 0xffff0000u);
  else return __half2float(__ushort_as_half(static_cast<unsigned short>(v >> 16)));
}
template <bool BF16>
__device__ __forceinline__ float load_elem(const void* base, size_t idx) {
  const unsigned short raw = reinterpret_cast<const unsigned short*>(base)[idx];
  if constexpr (BF16) return __uint_as_float(static_cast<uint32_t>(raw) << 16);
  else return __half2float(__ushort_as_half(raw));
}
template <bool BF16>
__device__ __forceinline__ unsigned short to_elem(float x) {
  if constexpr (BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(x));
  else return __half_as_ushort(__float2half_rn(x));
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// Loads 32 consecutive elements of a dense [.., S_k] row (16-bit dtype) as floats; entries
// past `n_valid` read as `fill`.  Uses 16-byte loads when the row segment is aligned.
template <bool BF16>
__device__ __forceinline__ void load_row32(const void* base, size_t elem_off, int n_valid, float fill,
                                           float (&out)[32]) {
  const unsigned short* p = reinterpret_cast<const unsigned short*>(base) + elem_off;
  if (n_valid >= 32 && ((reinterpret_cast<uintptr_t>(p) & 15) == 0)) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(p) + v);
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        out[v * 8 + 2 * k] = unpack_lo<BF16>(ws[k]);
        out[v * 8 + 2 * k + 1] = unpack_hi<BF16>(ws[k]);
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < 32; ++k) out[k] = (k < n_valid) ? load_elem<BF16>(p, k) : fill;
  }
}

template <bool BF16>
__device__ __forceinline__ void store_row32(void* base, size_t elem_off, int n_valid, const float (&v)[32]) {
  unsigned short* p = reinterpret_cast<unsigned short*>(base) + elem_off;
  if (n_valid >= 32 && ((reinterpret_cast<uintptr_t>(p) & 15) == 0)) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint4 w;
      w.x = pack2<BF16>(v[q * 8 + 0], v[q * 8 + 1]);
      w.y = pack2<BF16>(v[q * 8 + 2], v[q * 8 + 3]);
      w.z = pack2<BF16>(v[q * 8 + 4], v[q * 8 + 5]);
      w.w = pack2<BF16>(v[q * 8 + 6], v[q * 8 + 7]);
      reinterpret_cast<uint4*>(p)[q] = w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 32; ++k)
      if (k < n_valid) p[k] = to_elem<BF16>(v[k]);
  }
}

// The batch element of a given rank when they are sorted by a class (0..7) each, highest first, ties in batch order; evaluated
// by a whole warp, the same result in every lane.  Lane b holds the class of element b < B <= kMaxOrdered.  A descent over
// the three bits: of the elements still in question, those with the bit set come first.
constexpr int kMaxOrdered = 32;
__device__ __forceinline__ int batch_of_rank(int rank, int B, uint32_t cls) {
  const int lane = threadIdx.x & 31;
  uint32_t in = 0xffffffffu >> (32 - B);
#pragma unroll
  for (int bit = 2; bit >= 0; --bit) {
    const uint32_t set = in & __ballot_sync(0xffffffffu, (cls >> bit) & 1u);
    const int n = __popc(set);
    const bool among = rank < n;
    rank -= among ? 0 : n;
    in = among ? set : in & ~set;
  }
  return __ffs(__ballot_sync(0xffffffffu, (in >> lane & 1u) && __popc(in & ((1u << lane) - 1u)) == rank)) - 1;
}

// Packed batch, backward: the rows of the sequence whose offsets are `first` and `next`.  It is cut at the stated maximum length, and at the end of
// the tensor where its offset reaches past that, which the host cannot see; one that begins before the tensor has none.  (The forward counts keys
// behind the tensor as zeros, which are in the logsumexp and add nothing to any gradient.)  No branch on `first`, behind which the compiler
// moves the load of `next`: a second wait for memory in front of everything a block does (0.1 to 0.3 us a call of short kernels).
__device__ __forceinline__ int packed_rows(int first, int next, int max_len, int total_rows) {
  return min(min(next - first, max_len), total_rows - first) & ~(first >> 31);
}

// Packed batch, FMHA_FLAG_ZERO_UNCOVERED: zeroes, in head h of a [total_rows, H, D] tensor, the caller's share of the rows that no
// tile covers.  The caller stands for rows [r0, r1) of sequence b, as if every sequence had max_len rows; all callers together
// stand for all of them.  A sequence past max_len: its callers share the rows it is cut by.  Rows outside all sequences (`outside`;
// at most as many as the batch has rows of padding in this sense, else zero_outside_rows_kernel): the k-th row of padding, counted
// through the batch, stands for the k-th such row, so that callers without padding have nothing to look up and no caller has more
// rows than its own.  (One caller per head for all of them took three to four times as long as the fill of whole tensors that this
// replaces where a buffer was far from full.)  Offsets outside the tensor, which the host cannot see, are cut to its rows.
// Only callers with r1 > len or len > max_len can have a share.
__device__ __forceinline__ void zero_uncovered_rows(void* base, int64_t stride_s, int64_t stride_h, int h, int b, int B,
                                                    const int* cu, int max_len, int total_rows, int D, int r0, int r1, bool outside,
                                                    int tid, int nthreads) {
  const int lo = cu[b], hi = cu[b + 1], len = hi - lo;
  r1 = min(r1, max_len);
  auto zero = [&](int64_t from, int64_t to) {
    from = max(from, static_cast<int64_t>(0));
    to = min(to, static_cast<int64_t>(total_rows));
    const int per_row = D / 8;   // 16-byte pieces
    for (int64_t i = tid; i < (to - from) * per_row; i += nthreads)
      *reinterpret_cast<uint4*>(static_cast<unsigned short*>(base) + (from + i / per_row) * stride_s + h * stride_h +
                                (i % per_row) * 8) = make_uint4(0u, 0u, 0u, 0u);
  };
  if (len > max_len) {
    const int64_t cut = len - max_len, at = static_cast<int64_t>(lo) + max_len;
    zero(at + cut * r0 / max_len, at + cut * r1 / max_len);
  } else if (outside && r1 > len) {
    const int64_t first = cu[0], last = cu[B], n = first + total_rows - last;
    const int64_t pad0 = max(r0, len);
    const int64_t k0 = static_cast<int64_t>(b) * max_len - (lo - first) + (pad0 - len), k1 = min(k0 + (r1 - pad0), n);
    if (k0 < first) zero(k0, min(k1, first));
    if (k1 > first) zero(last + max(k0, first) - first, last + k1 - first);
  }
}

}  // namespace fmha
