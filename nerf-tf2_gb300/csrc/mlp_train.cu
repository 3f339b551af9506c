// Backward pass of the NeRF MLP (nerf/core/model.py:334-394), the gradient
// tf.GradientTape takes at model.py:148-170, in FP32 with FP32 master
// weights.
//
// The forward (mlp.cu, STORE variant) writes every layer's post-activation
// rows to `acts` (kActsLd floats per row). The backward takes the rows in
// chunks of kChunkRows; per chunk
//   head kernel   rgb = sigmoid(h9 Wr + br), sigma = ReLU(h7 ws + bs):
//                 dZ9 = (dpre_rgb Wr^T) * [h9 > 0], dpre_sigma, sums per block
//                 for the head gradients
//   chain kernel  for every layer from dense_9 down:
//                 dZ_prev[m][k] = (sum_n dZ[m][n] W[k][n] + dpre_sigma[m] ws[k])
//                                 * [h_prev[m][k] > 0]
//   dW kernel     for every layer: dW[k][n] += sum_m In[m][k] dZ[m][n], db[n]
//                 += sum_m dZ[m][n]
// the last two on the tensor cores in FP32 accuracy (gemm_fp32_tc.cu).
// Gradients land in the flat Keras layout of the parameter blob.
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "mlp_internal.cuh"

namespace nerfgb {
namespace train {

constexpr int kDzLd = 256;  // row stride of the dZ buffers
// Rows per chunk: the workspace holds every layer's dZ of one chunk (four
// 256-row tiles per pair of the chain kernel, 76 pairs).
constexpr long long kChunkRows = 4LL * 76 * 256;

// ---------------------------------------------------------------------------
// Heads
// ---------------------------------------------------------------------------
// A tape row's values of a lane, as loaded: h9 columns 4l .. 4l + 3, h7 columns 8l .. 8l + 7.
template <typename T>
struct HeadRow;
template <>
struct HeadRow<float> {
  float4 a, b, c;
  __device__ __forceinline__ void load(const float *p, int lane) {
    a = *reinterpret_cast<const float4 *>(p + acts_offset(9) + 4 * lane);
    b = *reinterpret_cast<const float4 *>(p + acts_offset(7) + 8 * lane);
    c = *reinterpret_cast<const float4 *>(p + acts_offset(7) + 8 * lane + 4);
  }
  __device__ __forceinline__ void zero() { a = b = c = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void get(float (&h9)[4], float (&h7)[8]) const {
    h9[0] = a.x; h9[1] = a.y; h9[2] = a.z; h9[3] = a.w;
    h7[0] = b.x; h7[1] = b.y; h7[2] = b.z; h7[3] = b.w; h7[4] = c.x; h7[5] = c.y; h7[6] = c.z; h7[7] = c.w;
  }
};
template <>
struct HeadRow<uint16_t> {
  uint2 a;
  uint4 b;
  __device__ __forceinline__ void load(const uint16_t *p, int lane) {
    a = *reinterpret_cast<const uint2 *>(p + acts_offset(9) + 4 * lane);
    b = *reinterpret_cast<const uint4 *>(p + acts_offset(7) + 8 * lane);
  }
  __device__ __forceinline__ void zero() {
    a = make_uint2(0u, 0u);
    b = make_uint4(0u, 0u, 0u, 0u);
  }
  __device__ __forceinline__ void get(float (&h9)[4], float (&h7)[8]) const {
    const uint32_t w[6] = {a.x, a.y, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xffff0000u);
      if (i < 2) {
        h9[(2 * i) % 4] = lo;
        h9[(2 * i + 1) % 4] = hi;
      } else {
        h7[(2 * i - 4) & 7] = lo;
        h7[(2 * i - 3) & 7] = hi;
      }
    }
  }
};

// A warp takes two rows at a time, the next two on their way: lane l owns h9
// columns 4l..4l+3 and h7 columns 8l..8l+7 (coalesced tape loads). The rows'
// eight head dot products (rgb's three and sigma's) are lane partials added
// over the lanes at distances 16, 8, 4, 2, 1; at the first three a lane passes
// on the half of the values that it does not keep, so the lanes l, l ^ 1, l ^ 2,
// l ^ 3 end with value l / 4 and compute what follows from it once, and eight
// shuffles give it to all (every sum the same bits as when each lane kept all
// eight: 40 shuffles and six sigmoids per lane and two rows, 0.50 ms of a
// 4,096-ray BF16 step, 0.23 here). dZ9 is written 16 bytes per lane, and the head
// weights' gradients accumulate in the lanes' registers over all of the warp's
// rows; a block's sums (shared atomics) go to the workspace, where the weight
// gradients' kernels add them up (add_head_sums).
constexpr int kHeadWarps = 8;
constexpr int kHeadRows = 2;

// TZ: dz9's type. BF16 (the tensor-core backward's operand): dense_9's bias
// gradient, the column sums of the FP32 values, is taken here too.
template <typename T, typename TZ>
__global__ void __launch_bounds__(32 * kHeadWarps, 2)
    head_bwd_kernel(const float *__restrict__ table, const T *__restrict__ acts, long long n,
                    const float *__restrict__ d_rgb, const float *__restrict__ d_sigma, TZ *__restrict__ dz9,
                    float *__restrict__ dsp_out, float *__restrict__ sums) {
  constexpr bool kBf16 = !std::is_same<TZ, float>::value;
  constexpr int kAcc = kBf16 ? kHeadSums : kHeadSumsFp32;
  __shared__ float sAcc[kAcc];  // dWr [128][3], dbr [3], dws [256], dbs [1] (BF16: db9 [128])
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < kAcc; e += blockDim.x) sAcc[e] = 0.0f;
  float wr[4][3], wsg[8];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int c = 0; c < 3; ++c) wr[j][c] = table[kRgbWOff + (4 * lane + j) * 3 + c];
#pragma unroll
  for (int j = 0; j < 8; ++j) wsg[j] = table[kSigmaWOff + 8 * lane + j];
  const float bias = ((lane >> 2) & 3) < 3 ? table[kRgbBOff + ((lane >> 2) & 3)] : table[kSigmaBOff];  // of the lane's value
  float gwr[4][3], gws[8], gbias = 0.0f, gb9[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 4; ++j) gwr[j][0] = gwr[j][1] = gwr[j][2] = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) gws[j] = 0.0f;
  __syncthreads();
  const long long wstep = (long long)gridDim.x * kHeadWarps * kHeadRows;
  const int q = lane >> 4, comp = (lane >> 2) & 3;  // the lane's value: row q's rgb[comp] or (3) sigma
  HeadRow<T> next[kHeadRows];
  float next_d;
  auto load = [&](long long r0) {
#pragma unroll
    for (int i = 0; i < kHeadRows; ++i) {
      if (r0 + i < n)
        next[i].load(acts + (r0 + i) * kActsLd, lane);
      else
        next[i].zero();
    }
    next_d = 0.0f;
    if (r0 + q < n && (comp < 3 || d_sigma)) next_d = comp < 3 ? d_rgb[(r0 + q) * 3 + comp] : d_sigma[r0 + q];
  };
  long long r0 = ((long long)blockIdx.x * kHeadWarps + warp) * kHeadRows;
  load(r0);
#pragma unroll 1
  for (; r0 < n; r0 += wstep) {
    float h9[kHeadRows][4], h7[kHeadRows][8];
#pragma unroll
    for (int i = 0; i < kHeadRows; ++i) next[i].get(h9[i], h7[i]);
    const float d = next_d;
    load(r0 + wstep);
    float v[8];
#pragma unroll
    for (int i = 0; i < kHeadRows; ++i) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[4 * i + c] = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[4 * i + c] = fmaf(h9[i][j], wr[j][c], v[4 * i + c]);
      }
      v[4 * i + 3] = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[4 * i + 3] = fmaf(h7[i][j], wsg[j], v[4 * i + 3]);
    }
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) {
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < o / 4; ++i) {
        const float keep = upper ? v[i + o / 4] : v[i], give = upper ? v[i] : v[i + o / 4];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    // rgb = sigmoid(h9 Wr + br), sigma = ReLU(h7 ws + bs) (model.py:374-386)
    const float y = 1.0f / (1.0f + expf(-(bias + v[0])));
    const float mine = r0 + q >= n ? 0.0f : comp < 3 ? d * y * (1.0f - y) : v[0] + bias > 0.0f ? d : 0.0f;
    if (comp == 3 && (lane & 3) == 0 && r0 + q < n) dsp_out[r0 + q] = mine;
#pragma unroll
    for (int i = 0; i < kHeadRows; ++i) {
      float drp[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) drp[c] = __shfl_sync(0xffffffffu, mine, 16 * i + 4 * c);
      const float dsp = __shfl_sync(0xffffffffu, mine, 16 * i + 12);
      const long long r = r0 + i;
      if (r < n) {
        float o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float g = drp[0] * wr[j][0] + drp[1] * wr[j][1] + drp[2] * wr[j][2];
          o[j] = h9[i][j] > 0.0f ? g : 0.0f;
        }
        if constexpr (kBf16) {
          const __nv_bfloat162 p0 = __floats2bfloat162_rn(o[0], o[1]), p1 = __floats2bfloat162_rn(o[2], o[3]);
          *reinterpret_cast<uint2 *>(dz9 + r * kDzLd + 4 * lane) =
              make_uint2(*reinterpret_cast<const uint32_t *>(&p0), *reinterpret_cast<const uint32_t *>(&p1));
#pragma unroll
          for (int j = 0; j < 4; ++j) gb9[j] += o[j];
        } else {
          *reinterpret_cast<float4 *>(dz9 + r * kDzLd + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < 3; ++c) gwr[j][c] = fmaf(h9[i][j], drp[c], gwr[j][c]);
#pragma unroll
      for (int j = 0; j < 8; ++j) gws[j] = fmaf(h7[i][j], dsp, gws[j]);
    }
    gbias += mine;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int c = 0; c < 3; ++c) atomicAdd(&sAcc[(4 * lane + j) * 3 + c], gwr[j][c]);
#pragma unroll
  for (int j = 0; j < 8; ++j) atomicAdd(&sAcc[387 + 8 * lane + j], gws[j]);
  if (kBf16) {
#pragma unroll
    for (int j = 0; j < 4; ++j) atomicAdd(&sAcc[(kBf16 ? 644 : 0) + 4 * lane + j], gb9[j]);
  }
  if ((lane & 3) == 0) atomicAdd(&sAcc[comp < 3 ? 384 + comp : 643], gbias);
  __syncthreads();
  for (int e = threadIdx.x; e < kAcc; e += blockDim.x) sums[(long long)blockIdx.x * kHeadSums + e] = sAcc[e];
}

}  // namespace train

template <typename T, typename TZ>
static int launch_head_bwd_t(const float *table, const T *tape, long long n, const float *d_rgb,
                             const float *d_sigma, TZ *dz9, float *dsp, float *sums, int *used, cudaStream_t st) {
  using namespace train;
  *used = 0;
  if (n == 0) return NERFGB_OK;
  const long long rows_per_block = (long long)kHeadWarps * kHeadRows;
  const long long blocks = (n + rows_per_block - 1) / rows_per_block;
  const int sms = num_sms();
  long long cap = (long long)(sms > 0 ? sms : 148) * 2;  // two blocks per SM (launch bounds)
  if (cap > kHeadMaxBlocks) cap = kHeadMaxBlocks;
  *used = (int)(blocks < cap ? blocks : cap);
  head_bwd_kernel<T, TZ><<<(unsigned)*used, 32 * kHeadWarps, 0, st>>>(table, tape, n, d_rgb, d_sigma, dz9, dsp, sums);
  return launch_status();
}

int launch_head_bwd(const float *table, const float *tape, long long n, const float *d_rgb, const float *d_sigma,
                    float *dz9, float *dsp, float *sums, int *blocks, cudaStream_t st) {
  return launch_head_bwd_t(table, tape, n, d_rgb, d_sigma, dz9, dsp, sums, blocks, st);
}

int launch_head_bwd(const float *table, const uint16_t *tape, long long n, const float *d_rgb,
                    const float *d_sigma, __nv_bfloat16 *dz9, float *dsp, float *sums, int *blocks,
                    cudaStream_t st) {
  return launch_head_bwd_t(table, tape, n, d_rgb, d_sigma, dz9, dsp, sums, blocks, st);
}

namespace train {

struct Ws {
  float *wpack, *heads, *dsp, *dz;
  long long rows, bytes;
};
static Ws carve(void *base, long long n) {
  Ws w{};
  float *p = reinterpret_cast<float *>(base);
  w.rows = n < kChunkRows ? n : kChunkRows;
  const long long pack = fp32_chain_pack_bytes() / (long long)sizeof(float);
  constexpr long long heads = (long long)kHeadMaxBlocks * kHeadSums;
  w.wpack = p;
  w.heads = p + pack;
  w.dz = w.heads + heads;
  w.dsp = w.dz + kNumGemm * w.rows * kDzLd;
  w.bytes = (pack + heads + w.rows * (kNumGemm * kDzLd + 1)) * (long long)sizeof(float);
  return w;
}

}  // namespace train
}  // namespace nerfgb

using namespace nerfgb;

extern "C" long long nerfgb_mlp_acts_floats_per_row(void) { return kActsLd; }

extern "C" long long nerfgb_mlp_backward_workspace_bytes(long long n_rows) {
  if (n_rows < 0) return -1;
  return train::carve(nullptr, n_rows).bytes;
}

extern "C" int nerfgb_mlp_forward_train(const void *packed, const float *xyz, const float *dirs, long long n_rows,
                                        int rows_per_dir, float *rgb, float *sigma, float *acts, void *stream) {
  if (n_rows < 0 || rows_per_dir < 1) return NERFGB_E_INVALID_ARG;
  if (n_rows == 0) return NERFGB_OK;
  if (!packed || !xyz || !dirs || !rgb || !sigma || !acts || !aligned(packed, 256) || !aligned(acts, 16))
    return NERFGB_E_INVALID_ARG;
  return launch_mlp_fp32_store(packed, xyz, dirs, n_rows, rows_per_dir, rgb, sigma, acts, as_stream(stream));
}

static int mlp_backward_fp32(const void *packed, const float *acts, long long n_rows, const float *d_rgb,
                             const float *d_sigma, float *grad_params, void *workspace, int *err_word, void *stream,
                             const WaitTest &chain, const WaitTest &dw) {
  using namespace train;
  if (n_rows < 0) return NERFGB_E_INVALID_ARG;
  if (n_rows == 0) return NERFGB_OK;
  if (!packed || !acts || !d_rgb || !grad_params || !workspace || !aligned(packed, 256) || !aligned(acts, 16) ||
      !aligned(workspace, 16))
    return NERFGB_E_INVALID_ARG;
  cudaStream_t st = as_stream(stream);
  const float *W = reinterpret_cast<const float *>(packed);  // FP32 pack: padded [Kp][N] blocks
  const float *table = W + kFp32TableOff;
  const Ws w = carve(workspace, n_rows);
  int rc;
  if ((rc = launch_fp32_chain_pack(W, w.wpack, st)) != NERFGB_OK) return rc;
  for (long long r0 = 0; r0 < n_rows; r0 += kChunkRows) {
    const long long n = n_rows - r0 < kChunkRows ? n_rows - r0 : kChunkRows;
    const float *a = acts + r0 * kActsLd;
    int head_blocks = 0;
    if ((rc = launch_head_bwd(table, a, n, d_rgb + 3 * r0, d_sigma ? d_sigma + r0 : nullptr, w.dz + 9 * n * kDzLd,
                              w.dsp, w.heads, &head_blocks, st)) != NERFGB_OK)
      return rc;
    if ((rc = launch_fp32_chain(w.wpack, table + kSigmaWOff, a, w.dsp, n, w.dz, grad_params, err_word, st, chain)) !=
        NERFGB_OK)
      return rc;
    if ((rc = launch_fp32_dw(a, w.dz, w.heads, head_blocks, n, grad_params, err_word, st, dw)) != NERFGB_OK) return rc;
  }
  return NERFGB_OK;
}

extern "C" int nerfgb_mlp_backward(const void *packed, const float *acts, long long n_rows, const float *d_rgb,
                                   const float *d_sigma, float *grad_params, void *workspace, void *stream) {
  return mlp_backward_fp32(packed, acts, n_rows, d_rgb, d_sigma, grad_params, workspace, nullptr, stream, WaitTest(),
                           WaitTest());
}

extern "C" int nerfgb_mlp_backward_checked(const void *packed, const float *acts, long long n_rows, const float *d_rgb,
                                           const float *d_sigma, float *grad_params, void *workspace, int *err_word,
                                           void *stream) {
  if (n_rows > 0 && !err_word) return NERFGB_E_INVALID_ARG;
  return mlp_backward_fp32(packed, acts, n_rows, d_rgb, d_sigma, grad_params, workspace, err_word, stream, WaitTest(),
                           WaitTest());
}

extern "C" int nerfgb_mlp_backward_wait_test(const void *packed_fp32, int precision, const void *tape, long long n_rows,
                                             const float *d_rgb, const float *d_sigma, float *grad_params,
                                             void *workspace, int *err_word, unsigned long long wait_ns, int withhold,
                                             void *stream) {
  if (precision != NERFGB_PREC_FP32 && precision != NERFGB_PREC_BF16) return NERFGB_E_UNSUPPORTED;
  if (wait_ns < 1000ull || wait_ns > 10000000000ull || withhold < 0 || withhold > 2) return NERFGB_E_INVALID_ARG;
  if (n_rows > 0 && !err_word) return NERFGB_E_INVALID_ARG;
  const WaitTest chain{wait_ns, withhold == 1}, dw{wait_ns, withhold == 2};
  if (precision == NERFGB_PREC_BF16)
    return mlp_backward_bf16(packed_fp32, tape, n_rows, d_rgb, d_sigma, grad_params, workspace, err_word, stream, chain,
                             dw);
  return mlp_backward_fp32(packed_fp32, reinterpret_cast<const float *>(tape), n_rows, d_rgb, d_sigma, grad_params,
                           workspace, err_word, stream, chain, dw);
}
