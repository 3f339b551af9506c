// Launchers shared between the MLP translation units.
#pragma once
#include <cuda.h>  // CUtensorMap (the encoder is reached through the runtime's entry-point query)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "nerfgb.h"

namespace nerfgb {

// Optional indirection of an MLP launch's rows. Logical row k in [0, n) is
// physical row map[k] of xyz, of the outputs and (divided by rows_per_dir)
// of dirs; with n_dev the row count is read on the device as
// min(*n_dev, n), so a compaction kernel can feed the MLP without a host
// round trip. Both NULL: the identity and the host count.
struct RowMap {
  const int *map = nullptr;
  const int *n_dev = nullptr;
};

// A tensor map of 16-bit elements over `base` (mlp_tc.cu): rank dims
// (innermost first), the byte strides of dims 1.. (multiples of 16), box
// sizes; no interleave, zero fill outside the dims; no swizzle, or with
// swizzle128 the 128-byte swizzle (box rows of 128 bytes land with their
// 16-byte chunks permuted by the row within each 8-row, 1024-byte block).
int encode_tensor_map_u16(CUtensorMap *map, const void *base, int rank, const unsigned long long *dims,
                          const unsigned long long *strides, const unsigned *box, bool swizzle128 = false);

// FP32 SIMT forward (mlp.cu).
int launch_mlp_fp32(const void *packed, const float *xyz, const float *dirs, long long n, int rows_per_dir,
                    float *rgb, float *sigma, cudaStream_t stream, const RowMap &rm = RowMap());

// FP32 SIMT forward that also stores every layer's activations (mlp.cu).
int launch_mlp_fp32_store(const void *packed, const float *xyz, const float *dirs, long long n, int rows_per_dir,
                          float *rgb, float *sigma, float *acts, cudaStream_t stream);

// BF16 tcgen05 forward (mlp_tc.cu).
int launch_mlp_bf16(const void *packed, const float *xyz, const float *dirs, long long n, int rows_per_dir,
                    float *rgb, float *sigma, int *err_word, cudaStream_t stream, const RowMap &rm = RowMap());

// BF16 tcgen05 forward that also writes the BF16 activation tape (kActsLd
// values per row, the FP32 tape's columns) for the BF16 backward (mlp_tc.cu).
int launch_mlp_bf16_train(const void *packed, const float *xyz, const float *dirs, long long n, int rows_per_dir,
                          float *rgb, float *sigma, uint16_t *tape, int *err_word, cudaStream_t stream);

// The failure path's test hook of a tensor-core kernel of the backward: a limit
// on its bounded waits (ns; 0: its own) and, withheld, one of the copies or
// arrivals that they wait for.
struct WaitTest {
  unsigned long long wait_ns = 0;
  int withhold = 0;
};

// Backward of the sigma and rgb heads (mlp_train.cu) from an FP32 or a BF16
// activation tape: dz9 = dL/d(dense_9 pre-activation), row stride 256 (128
// used), FP32 or BF16; dsp [n] = dL/d(sigma pre-activation). sums
// [kHeadMaxBlocks][kHeadSums]: each block's sums for the gradients of the heads
// and (BF16) of dense_9's bias, of *blocks blocks; add_head_sums adds one element
// up, by a warp: the gradient then takes one addition per call, whatever the
// number of rows and blocks.
constexpr int kHeadMaxBlocks = 512;
// the rgb head's kernel [128][3] and bias, the sigma head's kernel [256] and bias
// (as in the flat blob), dense_9's bias [128]
constexpr int kHeadSumsFp32 = 644, kHeadSums = 772;
int launch_head_bwd(const float *table, const float *tape, long long n, const float *d_rgb, const float *d_sigma,
                    float *dz9, float *dsp, float *sums, int *blocks, cudaStream_t stream);
int launch_head_bwd(const float *table, const uint16_t *tape, long long n, const float *d_rgb,
                    const float *d_sigma, __nv_bfloat16 *dz9, float *dsp, float *sums, int *blocks,
                    cudaStream_t stream);
__device__ __forceinline__ void add_head_sums(const float *__restrict__ sums, int blocks, int e, int lane,
                                              float *__restrict__ grads) {
  Sum sum;
  for (int b = lane; b < blocks; b += 32) sum.add(sums[(long long)b * kHeadSums + e]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float s = __shfl_xor_sync(0xffffffffu, sum.s, o), rest = __shfl_xor_sync(0xffffffffu, sum.rest, o);
    sum.add(s);
    sum.rest = fadd(sum.rest, rest);
  }
  const long long at = e < 387   ? flat_offset(11) + e
                       : e < 644 ? flat_offset(8) + (e - 387)
                                 : flat_offset(10) + (long long)flat_in(10) * flat_out(10) + (e - 644);
  // (atomic: what marks the gradient after a timeout may be on its way)
  if (lane == 0) atomicAdd(grads + at, sum.total());
}

// The dX products of the BF16 backward (mlp_bwd_tc.cu): dz [10][n][256] BF16,
// dz[9] in, dz[8] .. dz[0] out. bias [kChainMaxPairs * 2][kChainBias]: each
// CTA's sums of the dZ of dense_0 .. dense_8 (256 columns each), of *ctas CTAs.
// wpack (mlp_chain_pack_bytes, 16-byte aligned) from the FP32 pack's weights by
// launch_mlp_chain_pack; sigma_w: the sigma head's weights.
constexpr int kChainMaxPairs = 76, kChainBias = 9 * 256;
long long mlp_chain_pack_bytes();
int launch_mlp_chain_pack(const float *packed_fp32, void *wpack, cudaStream_t stream);
int launch_mlp_chain(const void *wpack, const float *sigma_w, const uint16_t *tape, const float *dsp, long long n,
                     __nv_bfloat16 *dz, float *bias, int *ctas, int *err, cudaStream_t stream,
                     const WaitTest &wt = WaitTest());

// The dX products of the FP32 backward (gemm_fp32_tc.cu): dz [10][n][256],
// dz[9] in (128 columns), dz[8] .. dz[0] out. wpack (fp32_chain_pack_bytes,
// 16-byte aligned) from the FP32 pack's weights by launch_fp32_chain_pack;
// sigma_w: the sigma head's weights. After a timeout all of grads is not a
// number and, unless NULL, *err_word the status; launch_fp32_dw likewise.
long long fp32_chain_pack_bytes();
int launch_fp32_chain_pack(const float *packed, void *wpack, cudaStream_t stream);
int launch_fp32_chain(const void *wpack, const float *sigma_w, const float *acts, const float *dsp, long long n,
                      float *dz, float *grads, int *err_word, cudaStream_t stream,
                      const WaitTest &wt = WaitTest());

// Weight and bias gradients of dense_0 .. dense_9 in the FP32 backward
// (gemm_fp32_tc.cu): every layer's In^T dZ and column sums of dZ over n rows
// added to the flat gradient blob, In from the FP32 tape, dz [10][n][256]. With
// them the heads' sums of `head_blocks` blocks.
int launch_fp32_dw(const float *acts, const float *dz, const float *heads, int head_blocks, long long n, float *grads,
                   int *err_word, cudaStream_t stream, const WaitTest &wt = WaitTest());

// Tensor-core weight gradients of the BF16 backward (gemm_tc.cu): every
// layer's In^T dZ over n rows added to the flat gradient blob, In from the
// BF16 tape, dz [10][n][256] BF16; part: gemm_dw_partial_floats() floats. With
// them the chain's bias sums (of `ctas` CTAs) and the heads' (of `head_blocks`
// blocks).
int launch_gemm_dw(const uint16_t *tape, const __nv_bfloat16 *dz, long long n, float *grads, float *part,
                   const float *bias, int ctas, const float *heads, int head_blocks, int *err, cudaStream_t stream,
                   const WaitTest &wt = WaitTest());
long long gemm_dw_partial_floats();
// The BF16 (pair) or FP8 tensor-core forward with a chosen limit on every
// bounded wait (ns) and the weight chunk at position `withhold` of the load
// sequence of the (even) CTA left unloaded, so that a wait runs out: the
// failure path's test hook (mlp_tc.cu).
int launch_mlp_wait_test(const void *packed, bool fp8, const float *xyz, const float *dirs, long long n, int rpd,
                         float *rgb, float *sigma, int *err_word, cudaStream_t stream, unsigned long long wait_ns,
                         long long withhold);

// FP8-e4m3 tcgen05 forward (mlp_tc.cu).
int launch_mlp_fp8(const void *packed, const float *xyz, const float *dirs, long long n, int rows_per_dir,
                   float *rgb, float *sigma, int *err_word, cudaStream_t stream, const RowMap &rm = RowMap());

// The BF16 backward (mlp_train_bf16.cu), nerfgb_mlp_backward_bf16 with the test
// hooks of its two tensor-core kernels.
int mlp_backward_bf16(const void *packed_fp32, const void *tape, long long n_rows, const float *d_rgb,
                      const float *d_sigma, float *grad_params, void *workspace, int *err_word, void *stream,
                      const WaitTest &chain, const WaitTest &dw);

// Dispatch on precision (render.cu).
int launch_mlp(const void *packed, int precision, const float *xyz, const float *dirs, long long n, int rpd,
               float *rgb, float *sigma, int *err_word, cudaStream_t stream, const RowMap &rm = RowMap());

// Sample gates (gate.cu). Coarse: sample (r, j) is on where w[r*S + j] > tau;
// writes mask[r*S + j] (0/1), appends the on samples' indices r*S + j to
// row_map (rays in any order, samples of a ray in order) and adds their
// number to *count. Fine: sample (r, j) of the sorted union is on where it is
// a coarse sample whose mask is on, or a fine draw (perm >= Sc); with the
// draws' bins (piece [R, S - Sc], not NULL) only a fine draw whose bin's mask
// is on.
int launch_gate_coarse(const float *w, int R, int S, float tau, unsigned char *mask, int *row_map, int *count,
                       cudaStream_t stream);
int launch_gate_fine(const int *perm, const unsigned char *mask_c, const int *piece, int R, int Sc, int S,
                     int *row_map, int *count, cudaStream_t stream);

// Proposal network forward (proposal.cu).
int launch_proposal_forward(const float *params, const float *xyz, long long n, float *sigma, cudaStream_t stream);
// The same network on tensor cores: BF16 operands, FP32 accumulation (proposal.cu).
int launch_proposal_forward_bf16(const float *params, const float *xyz, long long n, float *sigma,
                                 cudaStream_t stream);

// Compositing with a chosen last interval (ray_ops.cu): last_delta >= 0 is
// used as is (the reference uses 1e10), < 0 means the previous spacing.
// sample_rgb and the map outputs may be NULL.
// Optional gate on the compositor's weights (the coarse gate of the gated
// render): sample j of a ray is on where w > tau (NaN: off); mask [R*S]
// (0/1, may be NULL), the on samples' indices appended to row_map at slots
// taken from *count, sig_zero (may be NULL) zeroed at the off samples.
struct CompositeGate {
  float tau = 0.0f;
  unsigned char *mask = nullptr;
  int *row_map = nullptr, *count = nullptr;
  float *sig_zero = nullptr;
};
int launch_composite(const float *sample_rgb, const float *sigma, const float *t_vals, int n_rays, int n_samples,
                     int white_bg, int trans_mode, float last_delta, float *weights, float *pred_rgb,
                     float *pred_depth, float *acc_map, cudaStream_t stream,
                     const CompositeGate &gate = CompositeGate());

// Stratified coarse sampler (ray_ops.cu); u_vals NULL with perturb: the
// Philox draws of nerfgb_uniform(seed, 0, R*S) are made in the kernel.
int launch_coarse_sample(const float *rays_o, const float *rays_d, const float *near, const float *far,
                         const float *u_vals, unsigned long long seed, int R, int S, int perturb, int lin_inv,
                         float *xyz, float *dirs, float *t_vals, float *edges, float *widths, cudaStream_t stream);

// What the fine sampler (ray_ops.cu) fuses around the sampling, all fields
// optional: the coarse pass's compositing (the bin weights from sigma_c
// [R*Sc] instead of bin_weights; with rgb_c [R*Sc,3] and map_* also the
// coarse maps; w_c receives the weights), the fine gate of the gated render
// (a member of the sorted union is on where it is a fine draw or its coarse
// sample's mask_c entry is on; on members appended to row_map at slots from
// *count, sig_zero / rgb_zero zeroed at the off members), and the Philox
// draws of nerfgb_uniform(seed, R*Sc, R*Sf) when u_vals is NULL.
struct FineFuse {
  const float *sigma_c = nullptr, *rgb_c = nullptr;
  int mode = NERFGB_TRANS_LOGSUM, white_bg = 0;
  float *w_c = nullptr;
  float *map_rgb = nullptr, *map_depth = nullptr, *map_acc = nullptr;
  const unsigned char *mask_c = nullptr;
  int *row_map = nullptr, *count = nullptr;
  float *sig_zero = nullptr, *rgb_zero = nullptr;
  int gate_draws = 0;  // 1: a fine draw is on only where its coarse bin's gate is
  unsigned long long seed = 0;
};
int launch_fine_sample(const float *rays_o, const float *rays_d, const float *bin_weights, const float *left_edges,
                       int ld_left, const float *bin_widths, const float *t_vals_coarse, const float *u_vals,
                       int n_rays, int n_coarse, int n_fine, float *xyz, float *dirs, float *t_vals,
                       int *piece_idxs, int *sort_perm, cudaStream_t stream, const FineFuse &fz);
int launch_composite_bwd(const float *sigma, const float *t, const float *rgb, const float *grad_map,
                         const float *grad_w, int R, int S, int white_bg, float last_delta, float *grad_sigma,
                         float *grad_rgb, cudaStream_t stream);

// The BF16/FP8 proposal paths' front end (proposal.cu), one warp per ray:
// stratified samples (xyz, t_vals, edges [R, S+1], widths), the BF16
// proposal density at them, its weights over the bins (to w_out when not
// NULL) and, with gate.row_map, the coarse gate.
int launch_prop_front(const float *params, const float *rays_o, const float *rays_d, const float *near,
                      const float *far, const float *u, unsigned long long seed, int R, int S, int perturb,
                      int lin_inv, int mode, float *xyz, float *t_vals, float *edges, float *widths, float *w_out,
                      const CompositeGate &gate, cudaStream_t stream);

#ifdef NERF_BOUNDS_CHECK
// Error words of the bounds-check build, one per translation unit (common.cuh).
int bounds_read_ray_ops(int reset);
int bounds_read_gate(int reset);
int bounds_read_mlp(int reset);
int bounds_read_proposal(int reset);
int bounds_read_mlp_tc(int reset);
#endif

}  // namespace nerfgb
