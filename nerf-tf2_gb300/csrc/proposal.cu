// Learned proposal sampler (not in the reference): a 2x64 ReLU MLP on the
// L=6 positional encoding of xyz (39 inputs, the concatenation convention of
// nerf/core/model.py:323-330) with a softplus density output. Its weights
// are composited over finite bins: the last interval is the previous
// spacing, not the reference's 1e10 (ray_utils.py:465-468). With 1e10, any
// positive density in the last bin takes all remaining transmittance and
// d(alpha_last)/d(sigma) vanishes, so a learned density could neither avoid
// nor be taught to avoid piling every ray's fine samples into that bin. At inference
// its density at the 64 stratified samples, composited exactly as the coarse
// pass is (ray_utils.py:426-482), replaces the coarse MLP's weights as the
// PDF of the inverse-transform fine sampler (ray_utils.py:276-406).
//
// Parameters (flat float32, 6,785 values): W1 [39,64], b1 [64], W2 [64,64],
// b2 [64], W3 [64], b3 [1].
//
// FP32 forward and backward: 128-sample tiles per CTA of 256 threads, every
// step a small matrix product from shared memory (tile_product), vectors of a
// tile stored [component][sample]. The weight gradients are summed in registers
// over two tiles, then in shared memory over the CTA's tiles, and are added to the
// blob at the end, one atomicAdd per parameter per CTA.
#include <cuda_bf16.h>
#include <math.h>

#include "common.cuh"
#include "mlp_internal.cuh"
#include "ray_device.cuh"

namespace nerfgb {
namespace prop {

constexpr int kIn = 39, kH = 64;
constexpr int kW1 = 0, kB1 = kW1 + kIn * kH, kW2 = kB1 + kH, kB2 = kW2 + kH * kH, kW3 = kB2 + kH, kB3 = kW3 + kH;
constexpr int kParams = kB3 + 1;  // 6785
constexpr int kThreads = 256;
constexpr int kTS = 128;          // samples per tile
constexpr int kLdS = kTS + 4;     // row stride of the tile's [component][sample] arrays

__device__ __forceinline__ float softplus(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }

// What bounds these kernels is the FP32 FMA pipe, given enough reuse: a
// thread per sample with the weights broadcast from shared memory spent two
// shared-memory wavefronts per four FMAs (262,144 samples: forward 127 us,
// backward 634 us, against 99 and 256 here). A thread holds 8 samples x 4
// outputs: samples 4*sg .. +3 and 64 + 4*sg .. +3 (sg = 4*(warp/2) + lane/8),
// outputs 4*og .. +3 (og = 8*(warp%2) + lane%8). Tiles of 64 samples (4 x 4 per
// thread, two CTAs per SM in the backward) ran 373 us together against 355.
struct Place {
  int s0, j0;
  __device__ __forceinline__ explicit Place(int tid) {
    const int warp = tid >> 5, lane = tid & 31;
    s0 = 4 * ((warp >> 1) * 4 + (lane >> 3));
    j0 = 4 * ((warp & 1) * 8 + (lane & 7));
  }
  __device__ __forceinline__ int sample(int i) const { return s0 + (i & 3) + (i >> 2) * 64; }
};

// acc[i][j] += sum_k A[k][sample i] B[k][output j], k in order, paired FMAs
// over adjacent outputs (each half rounded as fmaf).
template <int K>
__device__ __forceinline__ void tile_product(const float *A, const float *B, const Place &pl, float (&acc)[8][4]) {
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    float a[8];
    *reinterpret_cast<float4 *>(a) = *reinterpret_cast<const float4 *>(A + k * kLdS + pl.s0);
    *reinterpret_cast<float4 *>(a + 4) = *reinterpret_cast<const float4 *>(A + k * kLdS + 64 + pl.s0);
    const float4 b = *reinterpret_cast<const float4 *>(B + k * kH + pl.j0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      fma_f32x2(acc[i][0], acc[i][1], a[i], a[i], b.x, b.y, acc[i][0], acc[i][1]);
      fma_f32x2(acc[i][2], acc[i][3], a[i], a[i], b.z, b.w, acc[i][2], acc[i][3]);
    }
  }
}
// The thread's 8 x 4 values to dst [output][sample].
__device__ __forceinline__ void store_tile(float *dst, const Place &pl, const float (&v)[8][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float *d = dst + (pl.j0 + j) * kLdS + pl.s0;
    *reinterpret_cast<float4 *>(d) = make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
    *reinterpret_cast<float4 *>(d + 64) = make_float4(v[4][j], v[5][j], v[6][j], v[7][j]);
  }
}

// Tile of samples [i0, i0 + 128): the encodings into enc [39][kLdS], h1 =
// ReLU(enc W1 + b1) into h1 [64][kLdS], and this thread's z2 = h1 W2 + b2 in
// z2. sw: the parameters. All threads; h1 is complete on return (and enc).
__device__ __forceinline__ void hidden_tile(const float *sw, const float *__restrict__ xyz, long long i0, long long n,
                                            float *enc, float *h1, const Place &pl, float (&z2)[8][4]) {
  for (int e = threadIdx.x; e < kTS * 21; e += kThreads) {
    const int q = e / kTS, sidx = e % kTS;
    const int c = q < 3 ? q : (q - 3) / 6, l = (q - 3) % 6;
    const float x = i0 + sidx < n ? xyz[3 * (i0 + sidx) + c] : 0.0f;
    if (q < 3) {
      enc[c * kLdS + sidx] = x;
    } else {
      float sn, cs;
      sincosf(fmul(x, enc_multiplier(l)), &sn, &cs);
      enc[(3 + c * 12 + 2 * l) * kLdS + sidx] = sn;
      enc[(3 + c * 12 + 2 * l + 1) * kLdS + sidx] = cs;
    }
  }
  __syncthreads();
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = sw[kB1 + pl.j0 + j];
  tile_product<kIn>(enc, sw + kW1, pl, acc);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[i][j] = fmaxf(acc[i][j], 0.0f);
      z2[i][j] = sw[kB2 + pl.j0 + j];
    }
  store_tile(h1, pl, acc);
  __syncthreads();
  tile_product<kH>(h1, sw + kW2, pl, z2);
}

// z3 = b3 + relu(z2) . W3 of one sample from h2 = ReLU(z2) [64][kLdS], in order.
__device__ __forceinline__ float head(const float *sw, const float *h2, int sidx) {
  float z3 = sw[kB3];
#pragma unroll 16
  for (int j = 0; j < kH; ++j) z3 = fmaf(h2[j * kLdS + sidx], sw[kW3 + j], z3);
  return z3;
}

__device__ __forceinline__ void load_params(const float *__restrict__ p, float *sw) {
  for (int i = threadIdx.x; i < kParams; i += blockDim.x) sw[i] = p[i];
}

constexpr int kParamsPad = (kParams + 3) / 4 * 4;
constexpr size_t kFwdSmem = (size_t)(kParamsPad + kIn * kLdS + kH * kLdS) * sizeof(float);  // two CTAs per SM

__global__ void __launch_bounds__(kThreads, 2)
    prop_fwd_kernel(const float *__restrict__ params, const float *__restrict__ xyz, long long n,
                    float *__restrict__ sigma) {
  extern __shared__ __align__(16) float sm[];
  float *sw = sm, *enc = sm + kParamsPad, *h1 = enc + kIn * kLdS;
  const Place pl(threadIdx.x);
  load_params(params, sw);
  __syncthreads();
  const long long ntiles = (n + kTS - 1) / kTS;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    float z2[8][4];
    hidden_tile(sw, xyz, tile * kTS, n, enc, h1, pl, z2);
    __syncthreads();  // h1 is used up: h2 takes its place
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) z2[i][j] = fmaxf(z2[i][j], 0.0f);
    store_tile(h1, pl, z2);
    __syncthreads();
    if (threadIdx.x < kTS) {
      const long long i = tile * kTS + threadIdx.x;
      const float z3 = head(sw, h1, threadIdx.x);
      if (i < n) sigma[i] = softplus(z3);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Inference forward on tensor cores: BF16 operands, FP32 accumulation
// (mma.sync m16n8k16; at 6,656 MAC per sample the kernel is bound by the
// encoding and its memory traffic, not by the tensor pipe). One warp per 16
// samples: layer 1's accumulator fragments are layer 2's A fragments (the
// m16n8 C layout of two n-tiles is the m16k16 A layout), so h1 never leaves
// registers. Weights sit in shared memory transposed ([n][k], k contiguous),
// rows padded by 8 BF16 so that a B-fragment load is conflict-free.
// ---------------------------------------------------------------------------
constexpr int kK1 = 48;              // 39 inputs padded to 3 k-steps of 16
constexpr int kLd1 = kK1 + 8, kLd2 = kH + 8;
constexpr int kFwdWarps = 4;
constexpr int kEncLdB = kK1 + 8;     // per-warp encoding rows (BF16), padded

__device__ __forceinline__ uint32_t bf16x2_relu(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The proposal's weights in shared memory for the BF16 forward.
struct PropSmemBf16 {
  __nv_bfloat16 W1[kH * kLd1];
  __nv_bfloat16 W2[kH * kLd2];
  float B1[kH], B2[kH], W3[kH], B3;
};

// All threads of the block; the caller synchronises. Weights transposed into
// [n][k] (reads follow the [k][n] source, coalesced).
__device__ __forceinline__ void stage_weights_bf16(const float *__restrict__ params, PropSmemBf16 &sp) {
  for (int e = threadIdx.x; e < kLd1 * kH; e += blockDim.x) {
    const int k = e / kH, nn = e % kH;
    sp.W1[nn * kLd1 + k] = __float2bfloat16_rn(k < kIn ? params[kW1 + k * kH + nn] : 0.0f);
  }
  for (int e = threadIdx.x; e < kLd2 * kH; e += blockDim.x) {
    const int k = e / kH, nn = e % kH;
    sp.W2[nn * kLd2 + k] = __float2bfloat16_rn(k < kH ? params[kW2 + k * kH + nn] : 0.0f);
  }
  for (int j = threadIdx.x; j < kH; j += blockDim.x) {
    sp.B1[j] = params[kB1 + j];
    sp.B2[j] = params[kB2 + j];
    sp.W3[j] = params[kW3 + j];
  }
  if (threadIdx.x == 0) sp.B3 = params[kB3];
}

// Octaves l0 .. l1-1 of coordinate c of the encoding (sin, cos of
// x * 2^l pi) from one sincosf at octave l0: the angle doubles exactly from
// one octave to the next, and sin 2a = (2 sin a) cos a, cos 2a = cos a cos a
// - sin a sin a, each operation rounded in FP32 (no FMA). Five doublings put
// an absolute error of a few 1e-6 on a value that is then rounded to BF16.
__device__ __forceinline__ void encode_octaves_bf16(__nv_bfloat16 *er, float xc, int c, int l0, int l1) {
  float sn, cs;
  sincosf(fmul(xc, enc_multiplier(l0)), &sn, &cs);
  for (int l = l0; l < l1; ++l) {
    if (l > l0) {
      const float s2 = fmul(fmul(2.0f, sn), cs);
      cs = fsub(fmul(cs, cs), fmul(sn, sn));
      sn = s2;
    }
    er[3 + c * 12 + 2 * l] = __float2bfloat16_rn(sn);
    er[3 + c * 12 + 2 * l + 1] = __float2bfloat16_rn(cs);
  }
}

// One 16-row tile's encodings (BF16) into the warp's buffer: two lanes per
// row (row = lane / 2). Lane h = 0 writes the three coordinates, coordinate
// 0's six octaves and coordinate 2's octaves 0-2; lane h = 1 the zero
// padding, coordinate 1's octaves and coordinate 2's octaves 3-5 (two
// sincosf per lane, encode_octaves_bf16). x: the lane's row's point.
__device__ __forceinline__ void encode_row_bf16(__nv_bfloat16 *enc, int lane, const float (&x)[3]) {
  const int row = lane >> 1, h = lane & 1;
  __nv_bfloat16 *er = enc + row * kEncLdB;
  if (h == 0) {
    er[0] = __float2bfloat16_rn(x[0]);
    er[1] = __float2bfloat16_rn(x[1]);
    er[2] = __float2bfloat16_rn(x[2]);
    encode_octaves_bf16(er, x[0], 0, 0, 6);
    encode_octaves_bf16(er, x[2], 2, 0, 3);
  } else {
#pragma unroll
    for (int k = kIn; k < kK1; ++k) er[k] = __float2bfloat16_rn(0.0f);
    encode_octaves_bf16(er, x[1], 1, 0, 6);
    encode_octaves_bf16(er, x[2], 2, 3, 6);
  }
}

// The densities of the tile's rows g = lane / 4 (s0) and g + 8 (s1), valid
// in the lanes with lane % 4 == 0, from the encodings in the warp's buffer.
__device__ __forceinline__ void tile_sigma_bf16(const PropSmemBf16 &sp, const __nv_bfloat16 *enc, int lane,
                                                float &s0, float &s1) {
  const int g = lane >> 2, t = lane & 3;
  // layer 1: [16 x 48] enc x [48 x 64] W1, accumulators start at b1
  float d1[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    d1[j][0] = d1[j][2] = sp.B1[8 * j + 2 * t];
    d1[j][1] = d1[j][3] = sp.B1[8 * j + 2 * t + 1];
  }
#pragma unroll
  for (int ks = 0; ks < kK1 / 16; ++ks) {
    const int k0 = 16 * ks + 2 * t;
    const uint32_t *e0 = reinterpret_cast<const uint32_t *>(enc + g * kEncLdB + k0);
    const uint32_t *e1 = reinterpret_cast<const uint32_t *>(enc + (g + 8) * kEncLdB + k0);
    const uint32_t a[4] = {e0[0], e1[0], e0[4], e1[4]};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const __nv_bfloat16 *b = sp.W1 + (8 * j + g) * kLd1 + k0;
      mma_bf16(d1[j], a, *reinterpret_cast<const uint32_t *>(b), *reinterpret_cast<const uint32_t *>(b + 8));
    }
  }
  // layer 2: relu(h1) as BF16 A fragments straight from the layer-1 accumulators
  float d2[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    d2[j][0] = d2[j][2] = sp.B2[8 * j + 2 * t];
    d2[j][1] = d2[j][3] = sp.B2[8 * j + 2 * t + 1];
  }
#pragma unroll
  for (int ks = 0; ks < kH / 16; ++ks) {
    const uint32_t a[4] = {bf16x2_relu(d1[2 * ks][0], d1[2 * ks][1]), bf16x2_relu(d1[2 * ks][2], d1[2 * ks][3]),
                           bf16x2_relu(d1[2 * ks + 1][0], d1[2 * ks + 1][1]),
                           bf16x2_relu(d1[2 * ks + 1][2], d1[2 * ks + 1][3])};
    const int k0 = 16 * ks + 2 * t;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const __nv_bfloat16 *b = sp.W2 + (8 * j + g) * kLd2 + k0;
      mma_bf16(d2[j], a, *reinterpret_cast<const uint32_t *>(b), *reinterpret_cast<const uint32_t *>(b + 8));
    }
  }
  // layer 3 (FP32): relu(z2) . w3 over this thread's 16 columns, then the quad
  float p0 = 0.0f, p1 = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float w0 = sp.W3[8 * j + 2 * t], w1 = sp.W3[8 * j + 2 * t + 1];
    p0 = fmaf(fmaxf(d2[j][0], 0.0f), w0, fmaf(fmaxf(d2[j][1], 0.0f), w1, p0));
    p1 = fmaf(fmaxf(d2[j][2], 0.0f), w0, fmaf(fmaxf(d2[j][3], 0.0f), w1, p1));
  }
  p0 += __shfl_xor_sync(0xffffffffu, p0, 1);
  p1 += __shfl_xor_sync(0xffffffffu, p1, 1);
  p0 += __shfl_xor_sync(0xffffffffu, p0, 2);
  p1 += __shfl_xor_sync(0xffffffffu, p1, 2);
  s0 = softplus(sp.B3 + p0);
  s1 = softplus(sp.B3 + p1);
}

__global__ void __launch_bounds__(32 * kFwdWarps)
    prop_fwd_bf16_kernel(const float *__restrict__ params, const float *__restrict__ xyz, long long n,
                         float *__restrict__ sigma) {
  __shared__ __align__(16) PropSmemBf16 sp;
  __shared__ __align__(16) __nv_bfloat16 sEnc[kFwdWarps][16 * kEncLdB];
  stage_weights_bf16(params, sp);
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const long long ntiles = (n + 15) / 16;
  const long long wstride = (long long)gridDim.x * kFwdWarps;
  __nv_bfloat16 *enc = sEnc[threadIdx.x >> 5];
  for (long long tile = (long long)blockIdx.x * kFwdWarps + (threadIdx.x >> 5); tile < ntiles; tile += wstride) {
    const long long r0 = tile * 16 + g, r1 = r0 + 8;
    {
      const long long gr = tile * 16 + (lane >> 1);
      float x[3] = {0.f, 0.f, 0.f};
      if (gr < n) {
        x[0] = xyz[3 * gr];
        x[1] = xyz[3 * gr + 1];
        x[2] = xyz[3 * gr + 2];
      }
      encode_row_bf16(enc, lane, x);
    }
    __syncwarp();
    float s0, s1;
    tile_sigma_bf16(sp, enc, lane, s0, s1);
    if (t == 0) {
      if (r0 < n) sigma[r0] = s0;
      if (r1 < n) sigma[r1] = s1;
    }
    __syncwarp();  // the buffer is rewritten by the next tile
  }
}

// ---------------------------------------------------------------------------
// Front end of the BF16/FP8 proposal paths, one warp per ray: the ray's S
// stratified samples (coarse_sample_kernel's arithmetic: Philox draws
// inside, t, bin edges, widths, points written out), the proposal density
// at them (prop_fwd_bf16_kernel's arithmetic, 16 samples per tile), the
// proposal weights over the bins (composite_ray with the finite last
// interval, nerfgb_proposal_weights' arithmetic) written to w_out when
// given, and with gate_map the coarse gate (sample j on where its weight >
// tau; gate_ray zeroes the coarse sigma at the off samples). Replaces the
// coarse sampler, proposal forward and proposal compositing launches.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(32 * kFwdWarps)
    prop_front_kernel(const float *__restrict__ params, const float *__restrict__ rays_o,
                      const float *__restrict__ rays_d, const float *__restrict__ near,
                      const float *__restrict__ far, const float *__restrict__ u, unsigned long long seed, int R,
                      int S, int perturb, int lin_inv, int mode, float *__restrict__ xyz, float *__restrict__ t_out,
                      float *__restrict__ edges, float *__restrict__ widths, float *__restrict__ w_out, float tau,
                      unsigned char *__restrict__ gate_mask, int *__restrict__ gate_map,
                      int *__restrict__ gate_count, float *__restrict__ gate_sig_zero) {
  __shared__ __align__(16) PropSmemBf16 sp;
  __shared__ __align__(16) __nv_bfloat16 sEnc[kFwdWarps][16 * kEncLdB];
  extern __shared__ float fsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  float *s_t = fsm + warp * 6 * S;  // t [S], sigma [S], weights [S], points [3S]
  float *s_sig = s_t + S;
  float *s_w = s_sig + S;
  float *s_x = s_w + S;
  __nv_bfloat16 *enc = sEnc[warp];
  stage_weights_bf16(params, sp);
  __syncthreads();
  for (int r = blockIdx.x * kFwdWarps + warp; r < R; r += gridDim.x * kFwdWarps) {
    const long long base = (long long)r * S;
    const float nr = near[r], fr = far[r];
    for (int i = lane; i < S; i += 32) {
      const BinSample b = coarse_bin_sample(rays_o, rays_d, nr, fr, u, seed, r, S, i, perturb, lin_inv);
      t_out[base + i] = b.t;
      widths[base + i] = b.w;
      edges[(long long)r * (S + 1) + i] = b.e0;
      if (i == S - 1) edges[(long long)r * (S + 1) + S] = b.e1;
      s_t[i] = b.t;
#pragma unroll
      for (int c = 0; c < 3; ++c) s_x[3 * i + c] = b.x[c];
    }
    __syncwarp();
    for (int j = lane; j < 3 * S; j += 32) xyz[3 * base + j] = s_x[j];
    for (int i0 = 0; i0 < S; i0 += 16) {
      const int i = i0 + (lane >> 1);
      float x[3] = {0.f, 0.f, 0.f};
      if (i < S) {
        x[0] = s_x[3 * i];
        x[1] = s_x[3 * i + 1];
        x[2] = s_x[3 * i + 2];
      }
      encode_row_bf16(enc, lane, x);
      __syncwarp();
      float s0, s1;
      tile_sigma_bf16(sp, enc, lane, s0, s1);
      if (t4 == 0) {
        if (i0 + g < S) s_sig[i0 + g] = s0;
        if (i0 + g + 8 < S) s_sig[i0 + g + 8] = s1;
      }
      __syncwarp();  // the buffer is rewritten by the next tile; s_sig complete
    }
    float m[5];
    composite_ray(lane, s_t, s_sig, nullptr, S, mode, -1.0f, s_w, m);
    __syncwarp();
    if (w_out)
      for (int j = lane; j < S; j += 32) w_out[base + j] = s_w[j];
    if (gate_map)
      gate_ray(lane, base, S, R, [&](int j) { return s_w[j] > tau; }, gate_mask, gate_map, gate_count,
               gate_sig_zero, nullptr, kSiteGateCoarse);
    __syncwarp();
  }
}

constexpr int kSums = 4 * 4 + 3 * 4 + 3 * 4;  // a thread's sums of dW2, dW1 and db1, db2, dW3
constexpr size_t kBwdSmem =
    (size_t)(kParamsPad + kH * kH + 48 * kLdS + 3 * kH * kLdS + kTS + kSums * kThreads) * sizeof(float);

// dW[r][c] of sum_s A[r][s] B[c][s] over the tile's samples: thread (tr, tc)
// holds rows tr + 16 i, columns tc + 16 j, as sums over even and odd samples.
// (Chains of 128 additions, over two tiles, then one addition per two tiles: with
// the chains over all of a CTA's tiles, 1,300 of them for 400,000 samples, and
// the other sums added to the blob by every warp, the gradient was further from
// 64 bits than with one thread per sample and sums per tile: b1 4.5e-7 of its norm
// at 100,000 samples against 2.8e-7, W3 8.8e-7 at 400,000 against 4.7e-7.)
template <int NR>
__device__ __forceinline__ void outer_tile(const float *A, const float *B, int tr, int tc, float (&acc)[NR][4][2]) {
#pragma unroll 4
  for (int q = 0; q < kTS; q += 4) {
    float4 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4 *>(B + (tc + 16 * j) * kLdS + q);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const float4 a = *reinterpret_cast<const float4 *>(A + (tr + 16 * i) * kLdS + q);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float(&c)[2] = acc[i][j];
        fma_f32x2(c[0], c[1], a.x, a.y, b[j].x, b[j].y, c[0], c[1]);
        fma_f32x2(c[0], c[1], a.z, a.w, b[j].z, b[j].w, c[0], c[1]);
      }
    }
  }
}

// grads += d/dparams sum_i dsigma_i * sigma_i.
__global__ void __launch_bounds__(kThreads, 1)
    prop_bwd_kernel(const float *__restrict__ params, const float *__restrict__ xyz, const float *__restrict__ dsig,
                    long long n, float *__restrict__ grads) {
  extern __shared__ __align__(16) float sm[];
  float *sw = sm;
  float *w2t = sw + kParamsPad;      // W2 transposed
  float *enc = w2t + kH * kH;        // 39 rows (48 for the weight gradient's row tiles, the rest 0)
  float *h1 = enc + 48 * kLdS;
  float *dz2 = h1 + kH * kLdS;       // first h2
  float *dz1 = dz2 + kH * kLdS;
  float *dz3 = dz1 + kH * kLdS;
  float *sums = dz3 + kTS + threadIdx.x;  // [kSums][kThreads]
  const int tid = threadIdx.x, tr = tid >> 4, tc = tid & 15;
  const Place pl(tid);
  load_params(params, sw);
  for (int e = tid; e < (48 - kIn) * kLdS; e += kThreads) enc[kIn * kLdS + e] = 0.0f;
  __syncthreads();
  for (int e = tid; e < kH * kH; e += kThreads) w2t[(e % kH) * kH + e / kH] = sw[kW2 + e];
#pragma unroll
  for (int i = 0; i < kSums; ++i) sums[i * kThreads] = 0.0f;
  float gw2[4][4][2] = {}, gw1[3][4][2] = {};
  bool second = false;
  float gb1[4] = {}, gb2[4] = {}, gw3[4] = {}, gb3 = 0.0f;
  const long long ntiles = (n + kTS - 1) / kTS;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long i0 = tile * kTS;
    float z2[8][4], v[8][4];
    hidden_tile(sw, xyz, i0, n, enc, h1, pl, z2);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = fmaxf(z2[i][j], 0.0f);
    store_tile(dz2, pl, v);
    __syncthreads();
    if (tid < kTS) {
      const float z3 = head(sw, dz2, tid);
      const float d = i0 + tid < n ? dsig[i0 + tid] / (1.0f + expf(-z3)) : 0.0f;  // softplus' = sigmoid
      dz3[tid] = d;
      gb3 += d;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float d = dz3[pl.sample(i)];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        gw3[j] = fmaf(v[i][j], d, gw3[j]);
        v[i][j] = z2[i][j] > 0.0f ? sw[kW3 + pl.j0 + j] * d : 0.0f;
        gb2[j] += v[i][j];
        z2[i][j] = 0.0f;
      }
    }
    store_tile(dz2, pl, v);
    __syncthreads();
    // dz1 = (dz2 W2^T) * [h1 > 0]
    tile_product<kH>(dz2, w2t, pl, z2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float *h = h1 + (pl.j0 + j) * kLdS;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (!(h[pl.sample(i)] > 0.0f)) z2[i][j] = 0.0f;
        gb1[j] += z2[i][j];
      }
    }
    store_tile(dz1, pl, z2);
    outer_tile<4>(h1, dz2, tr, tc, gw2);
    __syncthreads();
    outer_tile<3>(enc, dz1, tr, tc, gw1);
    if (second || tile + gridDim.x >= ntiles) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sums[(4 * i + j) * kThreads] += gw2[i][j][0] + gw2[i][j][1];
          gw2[i][j][0] = gw2[i][j][1] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          sums[(16 + 4 * i + j) * kThreads] += gw1[i][j][0] + gw1[i][j][1];
          gw1[i][j][0] = gw1[i][j][1] = 0.0f;
        }
        sums[(28 + j) * kThreads] += gb1[j];
        sums[(32 + j) * kThreads] += gb2[j];
        sums[(36 + j) * kThreads] += gw3[j];
        gb1[j] = gb2[j] = gw3[j] = 0.0f;
      }
    }
    second = !second;
    __syncthreads();  // the tile's arrays are rewritten
  }
  float *of_warp = dz1 + (tid >> 6) * 256;  // [4 sample groups of warps][db1, db2, dW3 [64], db3]
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) atomicAdd(grads + kW2 + (tr + 16 * i) * kH + tc + 16 * j, sums[(4 * i + j) * kThreads]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (tr + 16 * i < kIn) atomicAdd(grads + kW1 + (tr + 16 * i) * kH + tc + 16 * j, sums[(16 + 4 * i + j) * kThreads]);
    float b1 = sums[(28 + j) * kThreads], b2 = sums[(32 + j) * kThreads], w3 = sums[(36 + j) * kThreads];
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {  // over the warp's sample groups
      b1 += __shfl_xor_sync(0xffffffffu, b1, o);
      b2 += __shfl_xor_sync(0xffffffffu, b2, o);
      w3 += __shfl_xor_sync(0xffffffffu, w3, o);
    }
    if ((tid & 31) < 8) {
      of_warp[pl.j0 + j] = b1;
      of_warp[64 + pl.j0 + j] = b2;
      of_warp[128 + pl.j0 + j] = w3;
    }
  }
  if (tid < kTS) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
    if ((tid & 31) == 0) dz1[(tid >> 5) * 256 + 192] = gb3;
  }
  __syncthreads();
  if (tid <= 192) {
    const int at = tid < 64 ? kB1 + tid : tid < 128 ? kB2 + tid - 64 : tid < 192 ? kW3 + tid - 128 : kB3;
    atomicAdd(grads + at, (dz1[tid] + dz1[256 + tid]) + (dz1[512 + tid] + dz1[768 + tid]));
  }
}

}  // namespace prop

int launch_proposal_forward(const float *params, const float *xyz, long long n, float *sigma, cudaStream_t stream) {
  if (cudaFuncSetAttribute(prop::prop_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)prop::kFwdSmem) != cudaSuccess)
    return NERFGB_E_CUDA;
  const long long tiles = (n + prop::kTS - 1) / prop::kTS;
  const int sms = num_sms();
  const long long cap = (long long)(sms > 0 ? sms : 148) * 2;
  prop::prop_fwd_kernel<<<(unsigned)(tiles < cap ? tiles : cap), prop::kThreads, prop::kFwdSmem, stream>>>(params, xyz,
                                                                                                         n, sigma);
  return launch_status();
}

int launch_proposal_forward_bf16(const float *params, const float *xyz, long long n, float *sigma,
                                 cudaStream_t stream) {
  // persistent: two CTAs per SM, so that each converts the weights once for
  // many 16-sample tiles
  const long long tiles = (n + 16 * prop::kFwdWarps - 1) / (16 * prop::kFwdWarps);
  const int sms = num_sms();
  const long long cap = (long long)(sms > 0 ? sms : 148) * 2;
  prop::prop_fwd_bf16_kernel<<<(unsigned)(tiles < cap ? tiles : cap), 32 * prop::kFwdWarps, 0, stream>>>(
      params, xyz, n, sigma);
  return launch_status();
}

int launch_prop_front(const float *params, const float *rays_o, const float *rays_d, const float *near,
                      const float *far, const float *u, unsigned long long seed, int R, int S, int perturb,
                      int lin_inv, int mode, float *xyz, float *t_vals, float *edges, float *widths, float *w_out,
                      const CompositeGate &gate, cudaStream_t stream) {
  if (R == 0) return NERFGB_OK;
  const size_t smem = (size_t)prop::kFwdWarps * 6 * S * sizeof(float);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(prop::prop_front_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return NERFGB_E_CUDA;
  // persistent: each CTA converts the weights once for many rays
  const long long blocks = (R + prop::kFwdWarps - 1) / prop::kFwdWarps;
  const int sms = num_sms();
  const long long cap = (long long)(sms > 0 ? sms : 148) * 4;
  prop::prop_front_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 32 * prop::kFwdWarps, smem, stream>>>(
      params, rays_o, rays_d, near, far, u, seed, R, S, perturb, lin_inv, mode, xyz, t_vals, edges, widths, w_out,
      gate.tau, gate.mask, gate.row_map, gate.count, gate.sig_zero);
  return launch_status();
}

}  // namespace nerfgb

using namespace nerfgb;

extern "C" long long nerfgb_proposal_param_count(void) { return prop::kParams; }

extern "C" int nerfgb_proposal_weights(const float *sigma, const float *t_vals, int n_rays, int n_bins, int trans_mode,
                                       float *weights, void *stream) {
  if (n_rays < 0 || n_bins < 2) return NERFGB_E_INVALID_ARG;
  if (n_bins > 2048) return NERFGB_E_UNSUPPORTED;
  if (trans_mode != NERFGB_TRANS_CUMPROD && trans_mode != NERFGB_TRANS_LOGSUM) return NERFGB_E_UNSUPPORTED;
  if (n_rays == 0) return NERFGB_OK;
  if (!sigma || !t_vals || !weights) return NERFGB_E_INVALID_ARG;
  return launch_composite(nullptr, sigma, t_vals, n_rays, n_bins, 0, trans_mode, -1.0f, weights, nullptr, nullptr,
                          nullptr, as_stream(stream));
}

extern "C" int nerfgb_proposal_weights_backward(const float *sigma, const float *t_vals, const float *grad_weights,
                                                int n_rays, int n_bins, float *grad_sigma, void *stream) {
  if (n_rays < 0 || n_bins < 2) return NERFGB_E_INVALID_ARG;
  if (n_bins > 2048) return NERFGB_E_UNSUPPORTED;
  if (n_rays == 0) return NERFGB_OK;
  if (!sigma || !t_vals || !grad_weights || !grad_sigma) return NERFGB_E_INVALID_ARG;
  return launch_composite_bwd(sigma, t_vals, nullptr, nullptr, grad_weights, n_rays, n_bins, 0, -1.0f, grad_sigma,
                              nullptr, as_stream(stream));
}

extern "C" int nerfgb_proposal_forward_bf16(const float *params, const float *xyz, long long n, float *sigma,
                                            void *stream) {
  if (n < 0) return NERFGB_E_INVALID_ARG;
  if (n == 0) return NERFGB_OK;
  if (!params || !xyz || !sigma) return NERFGB_E_INVALID_ARG;
  return launch_proposal_forward_bf16(params, xyz, n, sigma, as_stream(stream));
}

extern "C" int nerfgb_proposal_forward(const float *params, const float *xyz, long long n, float *sigma,
                                       void *stream) {
  if (n < 0) return NERFGB_E_INVALID_ARG;
  if (n == 0) return NERFGB_OK;
  if (!params || !xyz || !sigma) return NERFGB_E_INVALID_ARG;
  return launch_proposal_forward(params, xyz, n, sigma, as_stream(stream));
}

extern "C" int nerfgb_proposal_backward(const float *params, const float *xyz, const float *grad_sigma, long long n,
                                        float *grad_params, void *stream) {
  if (n < 0) return NERFGB_E_INVALID_ARG;
  if (n == 0) return NERFGB_OK;
  if (!params || !xyz || !grad_sigma || !grad_params) return NERFGB_E_INVALID_ARG;
  if (cudaFuncSetAttribute(prop::prop_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)prop::kBwdSmem) != cudaSuccess)
    return NERFGB_E_CUDA;
  const long long ntiles = (n + prop::kTS - 1) / prop::kTS;
  int sms = num_sms();
  int grid = (int)(ntiles < sms ? ntiles : sms);
  prop::prop_bwd_kernel<<<grid, prop::kThreads, prop::kBwdSmem, as_stream(stream)>>>(params, xyz, grad_sigma, n,
                                                                                      grad_params);
  return launch_status();
}

#ifdef NERF_BOUNDS_CHECK
namespace nerfgb {
NG_BOUNDS_READER(bounds_read_proposal)
}  // namespace nerfgb
#endif
