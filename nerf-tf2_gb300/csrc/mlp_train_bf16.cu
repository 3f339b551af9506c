// BF16 backward of the NeRF MLP (nerf/core/model.py:334-394; the gradient
// tf.GradientTape takes at model.py:148-170) with FP32 master weights.
//
// The forward is the tensor-core BF16 kernel with its tape (mlp_tc.cu,
// STORE): each layer's BF16 activations are exactly the operands its
// successor's MMAs read. The backward, in chunks of kChunkRows rows:
//   heads   dZ_9 (BF16), dpre_sigma, sums per block for the gradients of the
//           heads and of dense_9's bias (mlp_train.cu)
//   chain   dZ_8 .. dZ_0 and their column sums per CTA, one kernel (mlp_bwd_tc.cu)
//   dW      every layer's In^T dZ, one kernel and a reduction, which adds up
//           those sums too (gemm_tc.cu)
// every product on the tensor cores from BF16 operands (W the BF16 rounding
// of the FP32 master weights), accumulating in FP32.
#include <cuda_bf16.h>

#include "common.cuh"
#include "mlp_internal.cuh"

namespace nerfgb {
namespace train16 {

// Rows per chunk: bounds the workspace (5 KB of dZ per row, 5.4 GB), far
// enough out that a 4,096-ray batch is one chunk per network.
constexpr long long kChunkRows = 1LL << 20;

struct Ws {
  float *dsp, *part;    // dpre_sigma, the dW kernel's partial sums
  __nv_bfloat16 *dz;    // [10][rows][256]
  void *wpack;          // the chain's BF16 weights
  float *bias, *heads;  // the chain's bias sums, the heads' sums
  long long bytes;
};

static long long a256(long long b) { return (b + 255) / 256 * 256; }

static Ws carve(void *base, long long n) {
  Ws w{};
  const long long rows = n < kChunkRows ? n : kChunkRows;
  long long off = 0;
  auto take = [&](long long bytes) -> char * {
    char *p = base ? static_cast<char *>(base) + off : nullptr;
    off += a256(bytes);
    return p;
  };
  w.dz = reinterpret_cast<__nv_bfloat16 *>(take(kNumGemm * rows * 256 * 2));
  w.dsp = reinterpret_cast<float *>(take(rows * 4));
  w.wpack = take(mlp_chain_pack_bytes());
  w.part = reinterpret_cast<float *>(take(gemm_dw_partial_floats() * 4));
  w.bias = reinterpret_cast<float *>(take(2LL * kChainMaxPairs * kChainBias * 4));
  w.heads = reinterpret_cast<float *>(take((long long)kHeadMaxBlocks * kHeadSums * 4));
  w.bytes = off;
  return w;
}

}  // namespace train16
}  // namespace nerfgb

using namespace nerfgb;

extern "C" long long nerfgb_mlp_backward_bf16_workspace_bytes(long long n_rows) {
  if (n_rows < 0) return -1;
  return train16::carve(nullptr, n_rows).bytes;
}

extern "C" int nerfgb_mlp_forward_train_bf16(const void *packed_bf16, const float *xyz, const float *dirs,
                                             long long n_rows, int rows_per_dir, float *rgb, float *sigma,
                                             void *tape, int *err_word, void *stream) {
  if (n_rows < 0 || rows_per_dir < 1) return NERFGB_E_INVALID_ARG;
  if (n_rows == 0) return NERFGB_OK;
  if (!packed_bf16 || !xyz || !dirs || !rgb || !sigma || !tape || !err_word || !aligned(packed_bf16, 256) ||
      !aligned(tape, 16))
    return NERFGB_E_INVALID_ARG;
  return launch_mlp_bf16_train(packed_bf16, xyz, dirs, n_rows, rows_per_dir, rgb, sigma,
                               reinterpret_cast<uint16_t *>(tape), err_word, as_stream(stream));
}

namespace nerfgb {
int mlp_backward_bf16(const void *packed_fp32, const void *tape, long long n_rows, const float *d_rgb,
                      const float *d_sigma, float *grad_params, void *workspace, int *err_word, void *stream,
                      const WaitTest &chain, const WaitTest &dw) {
  using namespace train16;
  if (n_rows < 0) return NERFGB_E_INVALID_ARG;
  if (n_rows == 0) return NERFGB_OK;
  if (!packed_fp32 || !tape || !d_rgb || !grad_params || !workspace || !err_word || !aligned(packed_fp32, 256) ||
      !aligned(tape, 16) || !aligned(workspace, 256))
    return NERFGB_E_INVALID_ARG;
  cudaStream_t st = as_stream(stream);
  const float *W = reinterpret_cast<const float *>(packed_fp32);  // FP32 pack: [Kp][N] blocks, then the table
  const float *table = W + kFp32TableOff;
  const uint16_t *tp = reinterpret_cast<const uint16_t *>(tape);
  Ws w = carve(workspace, n_rows);
  int rc;
  if ((rc = launch_mlp_chain_pack(W, w.wpack, st)) != NERFGB_OK) return rc;
  for (long long r0 = 0; r0 < n_rows; r0 += kChunkRows) {
    const long long n = n_rows - r0 < kChunkRows ? n_rows - r0 : kChunkRows;
    const uint16_t *t = tp + r0 * kActsLd;
    int head_blocks = 0, ctas = 0;
    if ((rc = launch_head_bwd(table, t, n, d_rgb + 3 * r0, d_sigma ? d_sigma + r0 : nullptr, w.dz + 9 * n * 256, w.dsp,
                              w.heads, &head_blocks, st)) != NERFGB_OK)
      return rc;
    if ((rc = launch_mlp_chain(w.wpack, table + kSigmaWOff, t, w.dsp, n, w.dz, w.bias, &ctas, err_word, st, chain)) !=
        NERFGB_OK)
      return rc;
    if ((rc = launch_gemm_dw(t, w.dz, n, grad_params, w.part, w.bias, ctas, w.heads, head_blocks, err_word, st, dw)) !=
        NERFGB_OK)
      return rc;
  }
  return NERFGB_OK;
}
}  // namespace nerfgb

extern "C" int nerfgb_mlp_backward_bf16(const void *packed_fp32, const void *tape, long long n_rows,
                                        const float *d_rgb, const float *d_sigma, float *grad_params,
                                        void *workspace, int *err_word, void *stream) {
  return mlp_backward_bf16(packed_fp32, tape, n_rows, d_rgb, d_sigma, grad_params, workspace, err_word, stream,
                           WaitTest(), WaitTest());
}
