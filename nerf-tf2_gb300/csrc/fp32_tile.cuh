// The FP32 tile product of the FP32 forward (mlp.cu): a CTA of 256 threads
// holds 8 RI rows (RI <= 8) of activations in shared memory for a whole chain of
// layers and multiplies them by [K][N] weights streamed from L2 in 16-row chunks.
//
// Bound by the FP32 FMA pipe; the rest is shaped so that nothing else is:
// - Paired FMAs (fma.rn.f32x2, each half rounded as fmaf): 2.09 cycles of
//   the pipe for two products against 2 x 1.22 for FFMA, and half the issue
//   slots, which the loads then use. A pair is two adjacent columns, so every
//   output keeps its own chain of FMAs over k in order.
// - A warp owns 4 RI rows x 64 columns, a thread RI x (4 + 4): for RI = 8, 20 shared-memory
//   wavefronts per 4 k instead of 49 for a warp of 8 rows x 256 columns. Rows
//   are dealt 4 apart and the row stride is 324 floats, so the four row
//   groups of a load fall in different banks.
// - 16-row chunks and one barrier per chunk (the next chunk's copy starts
//   right after it) leave room for two CTAs per SM, one's barriers and
//   epilogues under the other's FMAs.
#pragma once
#include "common.cuh"

namespace nerfgb {
namespace fp32 {

constexpr int kKC = 16;    // K rows per weight chunk
constexpr int kXLD = 324;  // X row stride (floats): 256 + 64 columns, padded
constexpr int kThreads = 256;
constexpr size_t smem_of(int ri) { return (size_t)(8 * ri * kXLD + 2 * kKC * 256) * sizeof(float); }
static_assert(2 * (smem_of(8) + 1024) <= 228 * 1024, "two CTAs per SM");

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
// One 16 x N chunk of weights (contiguous) into dst.
template <int N>
__device__ __forceinline__ void load_chunk(const float *__restrict__ src, float *dst, int tid) {
#pragma unroll
  for (int p = 0; p < kKC * N / 4; p += kThreads) cp_async16(dst + 4 * (p + tid), src + 4 * (p + tid));
  asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ void wait_chunk() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// A thread's place in the tile: rows row(i), i < RI, and columns col(h) .. +3,
// h < 2 (h < 1 where N is 128).
template <int RI>
struct Place {
  int wr, lr, c0;
  __device__ __forceinline__ explicit Place(int tid, int N) {
    const int warp = tid >> 5, lane = tid & 31;
    wr = warp & 1;
    lr = lane >> 3;
    c0 = (warp >> 1) * (N / 4) + (lane & 7) * 4;
  }
  __device__ __forceinline__ int row(int i) const { return wr * 4 * RI + 4 * i + lr; }
  __device__ __forceinline__ int col(int h) const { return c0 + 32 * h; }
};

__device__ __forceinline__ float f4c(const float4 &v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

// acc += X[rows][k0 .. k0 + 16) W[16][N]; x: &X[place.row(0)][k0], w: &W[0][place.col(0)].
template <int N, int RI>
__device__ __forceinline__ void chunk(const float *__restrict__ x, const float *__restrict__ w, float (&acc)[RI][8]) {
#pragma unroll
  for (int kk = 0; kk < kKC; kk += 4) {
    float4 a[RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4 *>(x + 4 * i * kXLD + kk);
#pragma unroll
    for (int kq = 0; kq < 4; ++kq) {
#pragma unroll
      for (int h = 0; h < N / 128; ++h) {
        const float4 b = *reinterpret_cast<const float4 *>(w + (kk + kq) * N + 32 * h);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          const float av = f4c(a[i], kq);
          float *c = acc[i] + 4 * h;
          fma_f32x2(c[0], c[1], av, av, b.x, b.y, c[0], c[1]);
          fma_f32x2(c[2], c[3], av, av, b.z, b.w, c[2], c[3]);
        }
      }
    }
  }
}

// One layer: acc = X[:, kin .. kin + K) W, W [K][N] whose first chunk is in
// (or on its way to) wb[buf]; meanwhile the next layer's first chunk, at
// next [.][N2] (N2 = 0: none), is copied as this layer's last is used.
// Ends with every warp done reading X.
template <int N, int RI>
__device__ __forceinline__ void layer(const float *X, float *wb, int &buf, const float *__restrict__ W, int K, int kin,
                                      const float *__restrict__ next, int next_n, int tid, const Place<RI> &pl,
                                      float (&acc)[RI][8]) {
#pragma unroll
  for (int i = 0; i < RI; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += kKC) {
    wait_chunk();
    __syncthreads();  // the chunk (and, at k0 = 0, X) is there; the chunk before is used up
    float *other = wb + (buf ^ 1) * kKC * 256;
    if (k0 + kKC < K)
      load_chunk<N>(W + (long long)(k0 + kKC) * N, other, tid);
    else if (next_n == 256)
      load_chunk<256>(next, other, tid);
    else if (next_n == 128)
      load_chunk<128>(next, other, tid);
    chunk<N, RI>(X + pl.row(0) * kXLD + kin + k0, wb + buf * kKC * 256 + pl.c0, acc);
    buf ^= 1;
  }
  __syncthreads();
}

}  // namespace fp32
}  // namespace nerfgb
