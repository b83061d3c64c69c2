// fmha_kernel_args.h — parameter blocks passed (by value, __grid_constant__) to the kernels,
// and the launch functions the C ABI layer calls.  Internal to the library.
#pragma once
#include <cuda.h>  // CUtensorMap (type only; the encode entry point is looked up at run time)
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/fmha_sm100.h"
#include "philox.cuh"

namespace fmha {

constexpr int kTileM = 128;  // query rows per CTA tile
constexpr int kTileN = 128;  // keys per step (general forward kernel, backward kernel)
// Keys per step of the forward kernel that will run: the production kernel walks the keys in
// 64-key steps at head dimension 64 (see fmha_fwd_fast_sm100.cu); the TMA box of K and V follows.
constexpr int kRowsKeyStep = 64;   // keys per step of the kernel for a handful of query rows
constexpr int fwd_key_tile(int D, bool legacy) { return (!legacy && D == 64) ? 64 : 128; }

struct FwdArgs {
  alignas(64) CUtensorMap tm_q;
  alignas(64) CUtensorMap tm_k;
  alignas(64) CUtensorMap tm_v;
  alignas(64) CUtensorMap tm_o;
  // general kernel only: the dense [B*H*S_q, S_k] 16-bit padding mask as a 2-D map with {64 x 128} boxes
  alignas(64) CUtensorMap tm_mask;
  // dense-mask kernel only: the dense dropout mask, same shape and boxes as tm_mask (valid when dmask_tiles is 1)
  alignas(64) CUtensorMap tm_dmask;
  int dmask_tiles;
  // dense-mask kernel only: the two saved [B*H, S_q, S_k] tensors as 3-D maps {S_k, S_q, B*H} with {64 x 128 x 1}
  // boxes, so that a tile stored at the end of a head's rows is clipped there (valid when save_tiles is 1)
  alignas(64) CUtensorMap tm_save_sm;
  alignas(64) CUtensorMap tm_save_dr;
  int save_tiles;
  int mask_tiles;   // 0: the mask is read with plain loads; 1: staged tile by tile through TMA
  // FMHA_MASK_CU_SEQLENS (production kernel): mask = int32 [B+1] row offsets into the packed [total_rows, H, D]
  // tensors; o_ptr / strides serve the row-wise stores of a sequence's last, partial query tile
  int total_rows;
  int zero_uncovered;         // FMHA_FLAG_ZERO_UNCOVERED: 0, or an UncoveredMode
  int persist;                // pair kernel: a CTA takes further items of the grid when it has done its own
  int length_class_shift;     // production kernels: -1, or the grid's last axis counts batch elements by (length - 1) >> shift
  const void* q_ptr;          // the kernel for a handful of query rows reads Q with plain loads
  int64_t q_ss, q_sh, q_sb;
  void* o_ptr;
  int64_t o_ss, o_sh, o_sb;   // strides in elements (o_sb: dense-mask kernel, which stores O row by row)
  int B, H, S_q, S_k;
  float scale_log2;  // softmax scale * log2(e)
  float scale;       // softmax scale
  float* lse;
  int mask_kind;
  const void* mask;
  int dropout_kind;
  const void* dropout_mask;
  float dropout_scale;   // multiplier applied to kept probabilities
  uint32_t philox_thr;   // 7-bit threshold
  uint64_t philox_seed;
  PhiloxKeys philox_keys;  // round keys of philox_seed
  uint32_t philox_offset;
  const long long* philox_offset_dev;   // optional device value added to philox_offset (production kernel)
  int philox_bh_offset;
  void* save_softmax;
  void* save_dropout;
  uint8_t* keep_mask_out;
  float* debug_scores;
  int* status;
};

// FMHA_FLAG_ZERO_UNCOVERED: the kernels zero the rows sequences are cut by, and those outside all sequences unless
// zero_outside_rows_kernel has (there are more of them than rows of padding, see zero_uncovered_rows).
enum UncoveredMode { kUncoveredAll = 1, kUncoveredCut = 2 };
// The backward pass: the three gradients (ptr null: none).
struct UncoveredRows {
  fmha_tensor4 grad[3];
  int total_rows;
  int mode;
};

struct BwdArgs {
  alignas(64) CUtensorMap tm_q;
  alignas(64) CUtensorMap tm_k;
  alignas(64) CUtensorMap tm_v;
  alignas(64) CUtensorMap tm_do;
  alignas(64) CUtensorMap tm_dk;  // 16-bit outputs, {D/4 x 32} boxes (one per compute warp), no swizzle
  alignas(64) CUtensorMap tm_dv;
  alignas(64) CUtensorMap tm_dq;   // head dimension 128, dQ kernel (fmha_bwd_dq_sm100.cu): 16-bit dQ in {16 x 32} boxes
  // O and dO for the row term delta, in the kernel that forms it, and dQ where it is written row by row: the dQ kernel, and the main kernel
  // with a single key tile at head dimension 64 (ONE_KV)
  const void* o_ptr;
  const void* do_ptr;
  int64_t o_sb, o_sh, o_ss, do_sb, do_sh, do_ss;
  void* dq_ptr;
  int64_t dq_ss, dq_sh, dq_sb;
  UncoveredRows zero;
  int persist;   // a CTA takes further work items of the grid when it has done its own
  int B, H, S_q, S_k;
  float scale;       // softmax scale
  float scale_log2;  // softmax scale * log2(e)
  const float* lse;  // [B*H, S_q] natural log
  float* delta;        // [B*H, S_q] rowsum(dO * O); not used with ONE_KV
  float* dq_accum;     // head dimension 64: [B*H, S_q_pad, D] fp32 in the blocked order of dq_accum_index, zero on entry; null: not used
  int* work_counter;   // zero on entry; the persistent CTAs draw their work items from it (not with ONE_KV: every grid-th item)
  // FMHA_MASK_CU_SEQLENS: mask = int32 [B+1] row offsets into the packed [total_rows, H, D] tensors; the raw
  // dK / dV pointers serve the row-wise stores of a sequence's last, partial key tile
  int total_rows;
  void* dk_ptr;
  void* dv_ptr;
  int64_t dk_ss, dk_sh, dv_ss, dv_sh;
  int S_q_pad;         // S_q rounded up to the tile
  int mask_kind;
  const void* mask;
  int dropout_kind;
  float dropout_scale;
  uint32_t philox_thr;
  uint64_t philox_seed;
  PhiloxKeys philox_keys;  // round keys of philox_seed
  uint32_t philox_offset;
  const long long* philox_offset_dev;   // optional device value added to philox_offset
  int philox_bh_offset;
  int* status;
};

// Launchers (defined in the .cu files).  Return a cudaError_t as int.
int launch_fwd(const FwdArgs& a, int D, int dtype, bool legacy, bool p_via_smem, cudaStream_t stream);
int launch_fwd_fast(const FwdArgs& a, int D, int dtype, cudaStream_t stream);
// the same for grids that fill the chip: two query tiles per CTA, persistent (fmha_fwd_pair_sm100.cu)
bool fwd_pair_applies(const FwdArgs& a, int D);
// its rule on sizes, on a device of `sms` multiprocessors (lengths: sequences may differ; packed_rows: rows of a packed batch, else 0)
bool fwd_pair_pays(int64_t sms, int64_t B, int64_t H, int64_t S_q, int64_t S_k, bool lengths, int64_t packed_rows);
int launch_fwd_pair(const FwdArgs& a, int dtype, cudaStream_t stream);
// the one-tile kernel's choice of order: a shift that puts the lengths into classes, or -1
int fwd_length_class_shift(const FwdArgs& a, int D, int64_t ctas, bool no_lengths);
// the same at head dimension 64 for grids of more tiles than the chip holds: a CTA takes one tile after the other (fmha_fwd_chain_sm100.cu)
bool fwd_chain_applies(const FwdArgs& a, int D);
// its rule on sizes, on a device of `sms` multiprocessors
bool fwd_chain_pays(int64_t sms, int64_t tiles, int64_t S_k, bool keyadd, bool dropout);
bool fwd_chain_pays(int64_t sms, int64_t tiles, int64_t S_k, bool keyadd, bool dropout, bool lengths);   // lengths: sequences may differ
int launch_fwd_chain(const FwdArgs& a, int dtype, cudaStream_t stream);
// the kernel for a handful of query rows per head (fmha_fwd_rows_sm100.cu): compact masks, not packed
bool fwd_rows_applies(int S_q, int S_k, int D, int64_t heads, bool dropout);
int launch_fwd_rows(const FwdArgs& a, int D, int dtype, cudaStream_t stream);
// the persistent kernel of the dense-mask operators at head dimension 64 (fmha_fwd_dense_sm100.cu)
bool fwd_dense_applies(const FwdArgs& a, int D);
int launch_fwd_dense(const FwdArgs& a, int dtype, cudaStream_t stream);
int launch_bwd_dq(const BwdArgs& a, int dtype, cudaStream_t stream);   // head dimension 128: dQ, delta, work counter
int launch_bwd(const BwdArgs& a, int D, int dtype, cudaStream_t stream);
// head dimension 64, one key tile: whether the main kernel is all there is (ONE_KV in fmha_bwd_sm100.cu)
bool bwd_one_kv(int D, int64_t heads, int S_q, int S_k);
// head dimension 64: the passes before and after the main kernel
// `m`: the main kernel's arguments (sizes, mask, Philox, workspace)
int launch_bwd_prepare(const fmha_tensor4& ot, const fmha_tensor4& dot, const BwdArgs& m, int dtype, cudaStream_t stream);
int launch_bwd_finish(const float* dq_accum, const fmha_tensor4& dq, int B, int H, int S_q, int S_q_pad, int dtype, float scale,
                      const int* cu_seqlens, int total_rows, cudaStream_t stream);

// Multiprocessors of the current device, asked for once per device.
inline int sm_count() {
  static std::atomic<int> count[64] = {};
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && (n = count[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (dev >= 0 && dev < 64) count[dev].store(n, std::memory_order_relaxed);
  return n;
}

// Launches `kernel` with programmatic stream serialization: its CTAs may be scheduled while the previous
// kernel of the stream drains (which hides the launch latency between the kernels of a training step); the
// kernel itself calls griddep_wait() before it touches global memory, so stream order is preserved.
template <typename Arg>
inline cudaError_t launch_overlapped(void (*kernel)(Arg), dim3 grid, dim3 block, size_t smem_bytes, cudaStream_t stream,
                                     const Arg& arg, int cluster_x = 0) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster_x > 0) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(cluster_x);
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kernel, arg);
}

}  // namespace fmha
