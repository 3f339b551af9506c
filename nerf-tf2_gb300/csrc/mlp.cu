// NeRF MLP (nerf/core/model.py:334-394): weight packing, the FP32 SIMT
// forward (the plain path) and the precision dispatcher.
//
// FP32 SIMT forward: one CTA of 256 threads owns a tile of 64 rows (or fewer:
// launch_fp32), two CTAs per SM. The tile's activations stay in shared memory
// for all ten GEMM layers (X[rows][320]: hidden state in columns 0..255, enc_xyz
// in 256..319, later enc_dir in 256..287); the product and its tiling are
// fp32_tile.cuh's. 100,003 rows: 2.12 ms, 56 TFLOP/s (3.18 ms with one CTA per
// SM, scalar FMAs and warps of 8 rows x 256 columns), the same outputs bit for
// bit. (The split products of gemm_fp32_tc.cu would be several times faster. They
// would need a second accumulator and sums in registers like those to be as
// accurate, and not every output then has the bits that it has had: a
// pre-activation near 0 on the other side turns a ReLU, and with it the row's
// gradient.)
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "common.cuh"
#include "fp32_tile.cuh"
#include "mlp_internal.cuh"

namespace nerfgb {

// ---------------------------------------------------------------------------
// Packing
// ---------------------------------------------------------------------------
__global__ void pack_kernel(const float *__restrict__ flat, int precision, unsigned char *__restrict__ out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kGemmWElems) {
    int g = 0;
    while (g + 1 < kNumGemm && i >= gemm_w_offset(g + 1)) ++g;
    long long e = i - gemm_w_offset(g);
    const int N = gemm_n(g);
    int k = (int)(e / N), n = (int)(e - (long long)k * N);
    const int L = flat_idx_of_gemm(g);
    float v = (k < gemm_k(g)) ? flat[flat_offset(L) + (long long)k * N + n] : 0.0f;
    if (precision == NERFGB_PREC_FP32) {
      reinterpret_cast<float *>(out)[i] = v;
    } else if (precision == NERFGB_PREC_FP8) {
      const float sc = reinterpret_cast<const float *>(out + kFp8ScaleOff)[bias_offset(g) + n];
      __nv_fp8_e4m3 q(sc > 0.0f ? v / sc : 0.0f);
      out[pair_w_byte(g, k, fp8_row(g, n), 1)] = *reinterpret_cast<unsigned char *>(&q);
    } else {
      *reinterpret_cast<__nv_bfloat16 *>(out + pair_w_byte(g, k, n, 2)) = __float2bfloat16_rn(v);
    }
    return;
  }
  long long t = i - kGemmWElems;
  if (t >= kTableElems) return;
  float v = 0.0f;
  if (t < kBiasElems) {
    int g = 0;
    while (g + 1 < kNumGemm && t >= bias_offset(g + 1)) ++g;
    int n = (int)t - bias_offset(g);
    const int L = flat_idx_of_gemm(g);
    v = flat[flat_offset(L) + (long long)flat_in(L) * flat_out(L) + n];
  } else if (t < kSigmaBOff) {
    v = flat[flat_offset(8) + (t - kSigmaWOff)];
  } else if (t == kSigmaBOff) {
    v = flat[flat_offset(8) + 256];
  } else if (t >= kRgbWOff && t < kRgbBOff) {
    v = flat[flat_offset(11) + (t - kRgbWOff)];
  } else if (t >= kRgbBOff && t < kRgbBOff + 3) {
    v = flat[flat_offset(11) + 128 * 3 + (t - kRgbBOff)];
  }
  float *table = reinterpret_cast<float *>(
      out + (precision == NERFGB_PREC_FP32 ? kFp32TableOff * 4
                                            : precision == NERFGB_PREC_BF16 ? kBf16TableOff : kFp8TableOff));
  table[t] = v;
}

// FP8 per-output-channel scales: scale[g][n] = max_k |W_g[k][n]| / 448.
__global__ void fp8_scale_kernel(const float *__restrict__ flat, unsigned char *__restrict__ out) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= kBiasElems) return;
  int g = 0;
  while (g + 1 < kNumGemm && e >= bias_offset(g + 1)) ++g;
  const int n = e - bias_offset(g), N = gemm_n(g), L = flat_idx_of_gemm(g);
  float m = 0.0f;
  for (int k = 0; k < gemm_k(g); ++k) m = fmaxf(m, fabsf(flat[flat_offset(L) + (long long)k * N + n]));
  reinterpret_cast<float *>(out + kFp8ScaleOff)[e] = m / kE4M3Max;
}

// ---------------------------------------------------------------------------
// FP32 SIMT forward
// ---------------------------------------------------------------------------
using fp32::kXLD;

// Copies columns [c0, c0 + nc) of the tile's kTM X rows to acts[row][off ..].
template <int kTM>
__device__ __forceinline__ void store_cols(float *__restrict__ acts, long long row0, long long n, const float *X,
                                           int c0, int nc, int off, int tid) {
  const int per_row = nc / 4;
  for (int e = tid; e < kTM * per_row; e += 256) {
    const int r = e / per_row, q = e - r * per_row;
    if (row0 + r < n)
      *reinterpret_cast<float4 *>(acts + (row0 + r) * kActsLd + off + 4 * q) =
          *reinterpret_cast<const float4 *>(X + r * kXLD + c0 + 4 * q);
  }
}

// STORE: also write every layer's post-activation rows to `acts` (training).
// rm: optional row map (logical row k reads and writes physical row
// rm.map[k]) and device row count; not used with STORE.
template <bool STORE, int RI>
__global__ void __launch_bounds__(fp32::kThreads, 2)
    mlp_fp32_kernel(const float *__restrict__ pk, const float *__restrict__ xyz,
                    const float *__restrict__ dirs, long long n_max, int rpd, float *__restrict__ rgb,
                    float *__restrict__ sigma, float *__restrict__ acts, RowMap rm) {
  constexpr int kTM = 8 * RI;  // rows per tile
  extern __shared__ __align__(16) float sm[];
  float *X = sm;
  float *Wb = sm + kTM * kXLD;
  const float *table = pk + kFp32TableOff;
  const int tid = threadIdx.x;
  const fp32::Place<RI> p256(tid, 256), p128(tid, 128);
  const long long n = rm.n_dev ? min((long long)*rm.n_dev, n_max) : n_max;
  const long long ntiles = (n + kTM - 1) / kTM;
  auto phys = [&](long long k) -> long long {
    return rm.map ? (long long)NG_IDX(rm.map[k], n_max, kSiteMlpRowMapFp32) : k;
  };
  int buf = 0;
  if ((long long)blockIdx.x < ntiles) fp32::load_chunk<256>(pk, Wb, tid);  // the first weight chunk

  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long row0 = tile * kTM;
    // enc_xyz -> X[:, 256..319] (model.py:319-331), column 319 = 0.
    for (int e = tid; e < kTM * 33; e += 256) {
      int r = e / 33, j = e - r * 33;
      long long gr = row0 + r;
      bool valid = gr < n;
      const long long pr = valid ? phys(gr) : 0;
      float *xr = X + r * kXLD + 256;
      if (j < 3) {
        xr[j] = valid ? xyz[pr * 3 + j] : 0.0f;
      } else {
        int jj = j - 3, c = jj / 10, l = jj - c * 10;
        float xv = valid ? xyz[pr * 3 + c] : 0.0f;
        float s, co;
        sincosf(fmul(xv, enc_multiplier(l)), &s, &co);
        xr[3 + c * 20 + 2 * l] = s;
        xr[3 + c * 20 + 2 * l + 1] = co;
      }
    }
    if (tid < kTM) X[tid * kXLD + 319] = 0.0f;

    for (int g = 0; g < kNumGemm; ++g) {
      const int N = gemm_n(g);
      const int kin = (g == 0) ? 256 : 0;
      // the chunk that follows this layer's last: the next layer's (the next tile's) first
      const bool more = g + 1 < kNumGemm || tile + gridDim.x < ntiles;
      const int gn = g + 1 < kNumGemm ? g + 1 : 0;
      const float *W = pk + gemm_w_offset(g), *Wn = pk + gemm_w_offset(gn);
      const int next_n = more ? gemm_n(gn) : 0;
      float acc[RI][8];
      if (N == 256)
        fp32::layer<256, RI>(X, Wb, buf, W, gemm_kp(g), kin, Wn, next_n, tid, p256, acc);
      else
        fp32::layer<128, RI>(X, Wb, buf, W, gemm_kp(g), kin, Wn, next_n, tid, p128, acc);
      // Epilogue: bias (+ReLU) into X[:, 0..N).
      const fp32::Place<RI> &pl = N == 256 ? p256 : p128;
      const float *bias = table + bias_offset(g);
      const bool relu = gemm_relu(g);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h == 1 && N != 256) break;
        const int col = pl.col(h);
        float4 bv = *reinterpret_cast<const float4 *>(bias + col);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          float4 v = make_float4(acc[i][4 * h] + bv.x, acc[i][4 * h + 1] + bv.y, acc[i][4 * h + 2] + bv.z,
                                 acc[i][4 * h + 3] + bv.w);
          if (relu) {
            v.x = fmaxf(v.x, 0.f);
            v.y = fmaxf(v.y, 0.f);
            v.z = fmaxf(v.z, 0.f);
            v.w = fmaxf(v.w, 0.f);
          }
          *reinterpret_cast<float4 *>(X + pl.row(i) * kXLD + col) = v;
        }
      }
      if (g == 8) {
        // enc_dir -> X[:, 256..287] (enc_xyz is dead after dense_5).
        for (int e = tid; e < kTM * 15; e += 256) {
          int r = e / 15, j = e - r * 15;
          long long gr = row0 + r;
          long long dr = phys(gr < n ? gr : n - 1) / rpd;
          float *xr = X + r * kXLD + 256;
          if (j < 3) {
            xr[j] = dirs[dr * 3 + j];
          } else {
            int jj = j - 3, c = jj / 4, l = jj - c * 4;
            float s, co;
            sincosf(fmul(dirs[dr * 3 + c], enc_multiplier(l)), &s, &co);
            xr[3 + c * 8 + 2 * l] = s;
            xr[3 + c * 8 + 2 * l + 1] = co;
          }
        }
        for (int e = tid; e < kTM * 5; e += 256) X[(e / 5) * kXLD + 283 + e % 5] = 0.0f;
      }
      __syncthreads();
      if (STORE) {
        store_cols<kTM>(acts, row0, n, X, 0, N, acts_offset(g), tid);
        if (g == 0) store_cols<kTM>(acts, row0, n, X, 256, 64, kActsEncXyz, tid);
        if (g == 8) store_cols<kTM>(acts, row0, n, X, 256, 32, kActsEncDir, tid);
      }
      if (g == 7) {
        // sigma = ReLU(h7 . w + b) (model.py:374-375).
        int r = tid >> 2, part = tid & 3;  // (r < kTM by whole warps)
        const float *sw = table + kSigmaWOff;
        float s = 0.0f;
        for (int k = part * 64; r < kTM && k < part * 64 + 64; ++k) s = fmaf(X[r * kXLD + k], sw[k], s);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (part == 0 && r < kTM && row0 + r < n) sigma[phys(row0 + r)] = fmaxf(s + table[kSigmaBOff], 0.0f);
        __syncthreads();
      }
    }
    // rgb = sigmoid(h9 . W + b) (model.py:386-387).
    for (int e = tid; e < kTM * 3; e += 256) {
      int r = e / 3, c = e - r * 3;
      const float *rw = table + kRgbWOff;
      float s = 0.0f;
      for (int k = 0; k < 128; ++k) s = fmaf(X[r * kXLD + k], rw[k * 3 + c], s);
      s += table[kRgbBOff + c];
      if (row0 + r < n) rgb[phys(row0 + r) * 3 + c] = 1.0f / (1.0f + expf(-s));
    }
    __syncthreads();
  }
}

}  // namespace nerfgb

using namespace nerfgb;

extern "C" long long nerfgb_mlp_param_count(void) { return kParamCount; }

extern "C" long long nerfgb_mlp_packed_bytes(int precision) {
  if (precision == NERFGB_PREC_FP32) return kFp32PackBytes;
  if (precision == NERFGB_PREC_BF16) return kBf16PackBytes;
  if (precision == NERFGB_PREC_FP8) return kFp8PackBytes;
  return -1;
}

extern "C" int nerfgb_mlp_pack(const float *params, int precision, void *packed, void *stream) {
  if (precision != NERFGB_PREC_FP32 && precision != NERFGB_PREC_BF16 && precision != NERFGB_PREC_FP8)
    return NERFGB_E_UNSUPPORTED;
  if (!params || !packed || !aligned(packed, 256) || !aligned(params, 4)) return NERFGB_E_INVALID_ARG;
  if (precision == NERFGB_PREC_FP8) {
    fp8_scale_kernel<<<(kBiasElems + 255) / 256, 256, 0, as_stream(stream)>>>(
        params, reinterpret_cast<unsigned char *>(packed));
    if (launch_status() != NERFGB_OK) return NERFGB_E_CUDA;
  }
  long long total = kGemmWElems + kTableElems;
  pack_kernel<<<(int)((total + 255) / 256), 256, 0, as_stream(stream)>>>(
      params, precision, reinterpret_cast<unsigned char *>(packed));
  return launch_status();
}

namespace nerfgb {
// Rows per tile, 8 RI. A wave of two CTAs per SM takes 406, 355, 317, 234, 195
// us for RI = 8, 7, 6, 4, 2 (about RI + 3 units), and about half where an SM has
// one CTA: up to one tile per SM, or up to half as many tiles left for the last
// wave (the first CTAs; more of them share SMs). The RI with the least half
// waves * (RI + 3) is taken: a last wave that 64-row tiles would leave nearly
// empty then costs less, and a small batch spreads over more SMs (100,003 rows
// 2.21 -> 2.12 ms, 20,000: 0.59 -> 0.52, 1,000: 229 -> 118 us). Every output is
// the same chain of FMAs whatever RI.
static long long half_waves(long long tiles, int sms) {
  const long long rest = tiles % (2 * sms);
  return tiles / (2 * sms) * 2 + (rest == 0 ? 0 : tiles <= sms || rest <= sms / 2 ? 1 : 2);
}

template <bool STORE, int RI>
static int launch_fp32_tiles(int sms, const void *packed, const float *xyz, const float *dirs, long long n, int rpd,
                             float *rgb, float *sigma, float *acts, cudaStream_t stream, const RowMap &rm) {
  constexpr size_t smem = fp32::smem_of(RI);
  if (cudaFuncSetAttribute(mlp_fp32_kernel<STORE, RI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return NERFGB_E_CUDA;
  const long long tiles = (n + 8 * RI - 1) / (8 * RI);
  mlp_fp32_kernel<STORE, RI><<<(int)(tiles < 2 * sms ? tiles : 2 * sms), fp32::kThreads, smem, stream>>>(
      reinterpret_cast<const float *>(packed), xyz, dirs, n, rpd, rgb, sigma, acts, rm);
  return launch_status();
}

template <bool STORE>
static int launch_fp32(const void *packed, const float *xyz, const float *dirs, long long n, int rpd, float *rgb,
                       float *sigma, float *acts, cudaStream_t stream, const RowMap &rm) {
  const int sms = num_sms();
  if (sms <= 0) return NERFGB_E_DEVICE;
  constexpr int sizes[5] = {8, 7, 6, 4, 2};
  int best = 8;
  long long least = 0;
  for (int ri : sizes) {
    const long long cost = half_waves((n + 8 * ri - 1) / (8 * ri), sms) * (ri + 3);
    if (least == 0 || cost < least) {
      least = cost;
      best = ri;
    }
  }
  switch (best) {
    case 7: return launch_fp32_tiles<STORE, 7>(sms, packed, xyz, dirs, n, rpd, rgb, sigma, acts, stream, rm);
    case 6: return launch_fp32_tiles<STORE, 6>(sms, packed, xyz, dirs, n, rpd, rgb, sigma, acts, stream, rm);
    case 4: return launch_fp32_tiles<STORE, 4>(sms, packed, xyz, dirs, n, rpd, rgb, sigma, acts, stream, rm);
    case 2: return launch_fp32_tiles<STORE, 2>(sms, packed, xyz, dirs, n, rpd, rgb, sigma, acts, stream, rm);
    default: return launch_fp32_tiles<STORE, 8>(sms, packed, xyz, dirs, n, rpd, rgb, sigma, acts, stream, rm);
  }
}

int launch_mlp_fp32(const void *packed, const float *xyz, const float *dirs, long long n, int rpd,
                    float *rgb, float *sigma, cudaStream_t stream, const RowMap &rm) {
  return launch_fp32<false>(packed, xyz, dirs, n, rpd, rgb, sigma, nullptr, stream, rm);
}

int launch_mlp_fp32_store(const void *packed, const float *xyz, const float *dirs, long long n, int rpd,
                          float *rgb, float *sigma, float *acts, cudaStream_t stream) {
  return launch_fp32<true>(packed, xyz, dirs, n, rpd, rgb, sigma, acts, stream, RowMap());
}
}  // namespace nerfgb

extern "C" int nerfgb_mlp_forward(const void *packed, int precision, const float *xyz, const float *dirs,
                                  long long n_rows, int rows_per_dir, float *rgb, float *sigma,
                                  int *err_word, void *stream) {
  if (n_rows < 0 || rows_per_dir < 1) return NERFGB_E_INVALID_ARG;
  if (precision != NERFGB_PREC_FP32 && precision != NERFGB_PREC_BF16 && precision != NERFGB_PREC_FP8)
    return NERFGB_E_UNSUPPORTED;
  if (n_rows == 0) return NERFGB_OK;
  if (!packed || !xyz || !dirs || !rgb || !sigma || !aligned(packed, 256)) return NERFGB_E_INVALID_ARG;
  if (precision == NERFGB_PREC_FP32)
    return launch_mlp_fp32(packed, xyz, dirs, n_rows, rows_per_dir, rgb, sigma, as_stream(stream));
  if (!err_word) return NERFGB_E_INVALID_ARG;
  if (precision == NERFGB_PREC_FP8)
    return launch_mlp_fp8(packed, xyz, dirs, n_rows, rows_per_dir, rgb, sigma, err_word, as_stream(stream));
  return launch_mlp_bf16(packed, xyz, dirs, n_rows, rows_per_dir, rgb, sigma, err_word, as_stream(stream));
}

extern "C" int nerfgb_mlp_forward_wait_test(const void *packed, int precision, const float *xyz, const float *dirs,
                                            long long n_rows, int rows_per_dir, float *rgb, float *sigma,
                                            int *err_word, unsigned long long wait_ns, long long withhold_chunk,
                                            void *stream) {
  if (n_rows < 0 || rows_per_dir < 1) return NERFGB_E_INVALID_ARG;
  if (precision != NERFGB_PREC_BF16 && precision != NERFGB_PREC_FP8) return NERFGB_E_UNSUPPORTED;
  if (wait_ns < 1000ull || wait_ns > 10000000000ull) return NERFGB_E_INVALID_ARG;
  if (n_rows == 0) return NERFGB_OK;
  if (!packed || !xyz || !dirs || !rgb || !sigma || !err_word || !aligned(packed, 256)) return NERFGB_E_INVALID_ARG;
  return launch_mlp_wait_test(packed, precision == NERFGB_PREC_FP8, xyz, dirs, n_rows, rows_per_dir, rgb, sigma,
                              err_word, as_stream(stream), wait_ns, withhold_chunk);
}

extern "C" int nerfgb_mlp_forward_mapped(const void *packed, int precision, const float *xyz, const float *dirs,
                                         long long n_rows_max, int rows_per_dir, const int *row_map,
                                         const int *n_rows_dev, float *rgb, float *sigma, int *err_word,
                                         void *stream) {
  if (n_rows_max < 0 || rows_per_dir < 1) return NERFGB_E_INVALID_ARG;
  if (precision != NERFGB_PREC_FP32 && precision != NERFGB_PREC_BF16 && precision != NERFGB_PREC_FP8)
    return NERFGB_E_UNSUPPORTED;
  if (n_rows_max == 0) return NERFGB_OK;
  if (!packed || !xyz || !dirs || !rgb || !sigma || !aligned(packed, 256)) return NERFGB_E_INVALID_ARG;
  if (precision != NERFGB_PREC_FP32 && !err_word) return NERFGB_E_INVALID_ARG;
  RowMap rm;
  rm.map = row_map;
  rm.n_dev = n_rows_dev;
  return launch_mlp(packed, precision, xyz, dirs, n_rows_max, rows_per_dir, rgb, sigma, err_word,
                    as_stream(stream), rm);
}

#ifdef NERF_BOUNDS_CHECK
namespace nerfgb {
NG_BOUNDS_READER(bounds_read_mlp)
}  // namespace nerfgb
#endif
