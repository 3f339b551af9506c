// The dX products of the BF16 MLP backward (the gradient tf.GradientTape
// takes at nerf/core/model.py:148-170 through the Dense layers of
// model.py:366-387) as one kernel: for a tile of rows, every layer from
// dense_9 down to dense_1,
//   raw[m][k] = bf16(sum_n dZ_g[m][n] W_g[k][n])            (k < 256)
//   z = raw (+ dpre_sigma[m] ws[k] below dense_8) (* [h_{g-1}[m][k] > 0])
//   dZ_{g-1} = bf16(z),  db_{g-1}[k] = sum_m z[m][k]
// with dZ in shared memory from one layer to the next. dZ of every layer goes
// to HBM for the weight gradients (gemm_tc.cu).
//
// What bounds it is HBM: per row and layer 512 bytes of activations (the ReLU
// mask) in and 512 bytes of dZ out, ~5.7k cycles of an SM's share of the
// copy bandwidth per 128 rows against 2,048 cycles of MMAs. A GEMM kernel and
// a mask kernel per layer moved 2.5 KB per row and layer for the same: 4.4 ms of
// a 4,096-ray step's two networks against 1.63 here (10.1 GB, 6.2 TB/s).
//
// The machinery is the forward's (mlp_tc.cu): cluster pairs on two 256-row
// sub-tiles (128 rows per CTA), 2-SM MMAs (M = 256, N = 256, B = W as [k][n],
// split by k between the CTAs), a five-stage weight ring, eight epilogue warps
// reading the accumulator as 16x256b fragments. Per sub-tile one I/O thread
//   - copies the rows' dZ_9 into the activation region (a tensor copy that
//     completes on the even CTA's barrier, where the issuer waits);
//   - as soon as a layer's MMAs have read the region, copies the layer's
//     activations over it: the epilogue reads them there with ldmatrix (the
//     fragments its accumulator has) and stores the masked result in their
//     place with stmatrix, so the mask needs no room of its own. The copy's
//     latency (~1.5k cycles) hides behind the other sub-tile; what the region
//     takes next was fetched into L2 a layer earlier (1 % of the time);
//   - stores the region to the layer's dZ.
// Bias sums: a thread's rows, then a reduce-scatter over the warp's row groups
// and one atomic per column, warp and sub-tile into the CTA's own sums in the
// workspace, which the weight gradients' reduction adds up (gemm_tc.cu). With the
// gradient itself as their target one number took an addition for every 32 rows:
// of 786,432 rows alike 2e-4 of it was lost, 1e-6 here, and the backward took
// 2.82 ms, 2.77 here.
//
// Every mbarrier wait is bounded; on a timeout the kernel reports, drains and
// returns as mlp_tc.cu's does.
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "mlp_internal.cuh"
#include "pair_tc.cuh"
#include "tcgen05.cuh"

namespace nerfgb {
namespace tcb {

using namespace tc;

constexpr int kSubRows = 256;
constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + kEpiWarps + 2) * 32;
constexpr int kNst = 5;
constexpr uint32_t kActOff = kNst * kPairStage;
constexpr uint32_t kActBytes = 4 * kAtom;
constexpr uint32_t kMisc = kActOff + 2 * kActBytes;
constexpr uint32_t kBarFull = kMisc;          // [kNst]
constexpr uint32_t kBarEmpty = kMisc + 64;    // [kNst]
constexpr uint32_t kBarAccf = kMisc + 128;    // [2] accumulators full
constexpr uint32_t kBarActr = kMisc + 144;    // [2] operand written, accumulator read
constexpr uint32_t kBarLoad = kMisc + 160;    // [2] dZ_9 of both CTAs there (the even CTA's)
constexpr uint32_t kBarMask = kMisc + 176;    // [2] the layer's activations there
constexpr uint32_t kBarRdy = kMisc + 192;     // [2] dZ written, to be stored
constexpr uint32_t kBarDrain = kMisc + 208;
constexpr uint32_t kTmemSlot = kMisc + 216;
constexpr uint32_t kAbort = kMisc + 224;      // int, then the wait limit (u64) at +8
constexpr uint32_t kSmemBytes = kMisc + 256;
static_assert(kSmemBytes <= 227 * 1024 && kAbort % 8 == 0, "shared memory");

// w: the pack below as 2-D 256-byte rows, boxes of 64 rows (a CTA's half of a
// chunk); act: the tape as 3-D (64 elements, rows, atoms), boxes of 128 rows
// by 4 atoms; dz[l]: layer l's dZ, boxes of 128 rows by 4 atoms (dz[9], 128
// columns: 2). All 128-byte swizzled but w.
struct Maps {
  CUtensorMap w, act, dz[kNumGemm];
};

// Weights of the chain, in its order dense_9 .. dense_1: per layer, chunks of
// 64 n; per chunk k-half 0 then 1 (128 rows each), K-major core matrices.
__host__ __device__ constexpr int chain_n(int i) { return gemm_n(9 - i); }  // i-th layer of the chain
constexpr long long kPackBytes = (long long)(128 + 8 * 256) * 256 * 2;

__global__ void pack_kernel(const float *__restrict__ W, uint8_t *__restrict__ out) {
  const int i = blockIdx.y, g = 9 - i, N = gemm_n(g);
  const long long base = i == 0 ? 0 : (long long)(128 + (i - 1) * 256) * 256 * 2;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;  // k * N + n
  if (e >= 256 * N) return;
  const int k = e / N, n = e % N;
  const long long byte = base + (long long)(n / 64) * (2 * kPairStage) + (k / 128) * kPairStage + ((n % 64) / 8) * 2048 +
                         (k % 128) * 16 + (n % 8) * 2;
  *reinterpret_cast<__nv_bfloat16 *>(out + byte) = __float2bfloat16_rn(W[gemm_w_offset(g) + e]);
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&m)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(m[0]), "=r"(m[1]), "=r"(m[2]), "=r"(m[3])
               : "r"(addr)
               : "memory");
}

// The MMAs of one layer (NC chunks of 64 n) for sub-tile S.
template <int NC, int S>
__device__ __forceinline__ void issue_chain(uint32_t sbase, uint32_t tmem, bool release, RingPos &rp,
                                            volatile int *abort_flag, int *err) {
  constexpr int H = 128;
  const uint32_t sw = sbase & 0x3FFFFu;
  issue_run<kNst, NC, 4, H, false, true, S == 0>(sbase + kBarFull, sbase + kBarEmpty, (sw >> 4) | ((uint32_t)H << 16),
                                                 ((sw + kActOff + S * kActBytes) >> 4) | (1u << 16), tmem + S * 256,
                                                 idesc_bf16(256, 256), release, rp, abort_flag, err);
}

// 64 columns x 16 rows of a layer's result: acc (raw) rounded to BF16, the
// sigma head's term, the mask already in the operand at addr (stmatrix/
// ldmatrix addressing of mlp_tc.cu), the result in its place, sums per column.
template <bool MASK, bool SIG>
__device__ __forceinline__ void finish_frag(uint32_t addr, uint32_t cx, const uint32_t (&raw)[32], float ds0, float ds1,
                                            const float *ws, float (&sum)[16]) {
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    const uint32_t a = addr + (((uint32_t)i ^ cx) << 4);
    uint32_t w[4], m[4];
    if (MASK) ldmatrix_x4(a, m);
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // group i + j / 2; rows lane/4 (even j), + 8 (odd)
      const int r = 4 * (i + j / 2) + 2 * (j & 1), c = 2 * (i + j / 2);
      w[j] = pack_bf16(__uint_as_float(raw[r]), __uint_as_float(raw[r + 1]));
      float z0 = __uint_as_float(w[j] << 16), z1 = __uint_as_float(w[j] & 0xffff0000u);
      if (SIG) {
        const float2 s = *reinterpret_cast<const float2 *>(ws + 8 * (i + j / 2));
        z0 = fmaf((j & 1) ? ds1 : ds0, s.x, z0);
        z1 = fmaf((j & 1) ? ds1 : ds0, s.y, z1);
      }
      if (MASK) {
        // ReLU outputs: > 0 unless 0 (or -0)
        if ((int)(m[j] << 16) <= 0) z0 = 0.0f;
        if ((int)(m[j] & 0xffff0000u) <= 0) z1 = 0.0f;
      }
      if (MASK || SIG) w[j] = pack_bf16(z0, z1);
      sum[c] += z0;
      sum[c + 1] += z1;
    }
    stmatrix_x4(a, w[0], w[1], w[2], w[3]);
  }
}

// sum[2i + e]: this thread's rows' sums of columns 8i + 2 (lane % 4) + e. Adds
// the warp's sums of the 64 columns to db.
__device__ __forceinline__ void add_columns(const float (&sum)[16], int lane, float *__restrict__ db) {
  float a[8], b[4], c[2];
  const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float o = __shfl_xor_sync(0xffffffffu, u16 ? sum[j] : sum[j + 8], 16);
    a[j] = (u16 ? sum[j + 8] : sum[j]) + o;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float o = __shfl_xor_sync(0xffffffffu, u8 ? a[j] : a[j + 4], 8);
    b[j] = (u8 ? a[j + 4] : a[j]) + o;
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float o = __shfl_xor_sync(0xffffffffu, u4 ? b[j] : b[j + 2], 4);
    c[j] = (u4 ? b[j + 2] : b[j]) + o;
  }
  // the lane's group of eight columns is its bits 4, 3, 2: lane / 4
  float *d = db + 8 * (lane >> 2) + 2 * (lane & 3);
  atomicAdd(d, c[0]);
  atomicAdd(d + 1, c[1]);
}

__global__ void __launch_bounds__(kThreads, 1)
    chain_kernel(const float *__restrict__ ws, const float *__restrict__ dsp, long long n, float *__restrict__ bias,
                 int *__restrict__ err, WaitTest wt, const __grid_constant__ Maps maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kAbort);
  // this pair's sub-tiles, as in mlp_tc.cu
  const uint32_t crank = cluster_rank();
  int first, count;
  {
    const unsigned subs = (unsigned)((n + kSubRows - 1) / kSubRows), np = cluster_count(), p = cluster_id();
    const unsigned q = subs / np, rest = subs % np;
    first = (int)(p * q + min(p, rest));
    count = (sbase & 1023u) != 0 ? 0 : (int)(q + (p < rest ? 1u : 0u));
  }
  const int ntiles = (count + 1) / 2;
  bias += (long long)blockIdx.x * kChainBias;
  for (int e = threadIdx.x; e < kChainBias; e += kThreads) bias[e] = 0.0f;
  auto row_of = [&](int k, int s) -> long long {
    return (long long)(first + 2 * k + s) * kSubRows + (int)crank * 128;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kNst; ++s) {
      mbar_init(sbase + kBarFull + 8 * s, 1);
      mbar_init(sbase + kBarEmpty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(sbase + kBarAccf + 8 * s, 1);
      mbar_init(sbase + kBarActr + 8 * s, 2 * kEpiWarps);
      mbar_init(sbase + kBarLoad + 8 * s, 1);
      mbar_init(sbase + kBarMask + 8 * s, 1);
      mbar_init(sbase + kBarRdy + 8 * s, kEpiWarps);
    }
    mbar_init(sbase + kBarDrain, 1);
    *abort_flag = 0;
    set_wait_limit(abort_flag, wt.wait_ns != 0 ? wt.wait_ns : kWaitNs);
    if ((sbase & 1023u) != 0) atomicExch(err, NERFGB_E_UNSUPPORTED);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kTmemSlot),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + kTmemSlot);

  if (warp == 0) {
    // ---------------- weight producer (mlp_tc.cu) ----------------
    if (lane == 0) {
      uint32_t used = 0;
      int st = 0;
      bool ok = true;
      for (int tile = 0; tile < ntiles && ok; ++tile)
        for (uint32_t src = 0; src < (uint32_t)kPackBytes; src += 2 * kPairStage) {
          if (!wait_bar(sbase + kBarEmpty + 8 * st, ((used >> st) & 1u) ^ 1u, abort_flag, err)) {
            ok = false;
            break;
          }
          const uint32_t full = sbase + kBarFull + 8 * st;
          // (test hook: the even CTA leaves out the tile's second chunk)
          if (!(wt.withhold != 0 && crank == 0 && src == 2 * kPairStage)) {
            if (crank == 0) mbar_expect_tx(full, 2 * kPairStage);
            tma_2d_pair(sbase + st * kPairStage, &maps.w, 0, (int)((src + crank * kPairStage) >> 8),
                        crank == 0 ? full : peer_addr(full, 0));
          }
          used ^= 1u << st;
          if (++st == kNst) st = 0;
        }
      if (!ok && crank == 0) {
        const uint64_t t0 = globaltimer();
        for (int k = 0; k < kNst; ++k)
          while (!mbar_try(sbase + kBarFull + 8 * k, ((used >> k) & 1u) ^ 1u) && globaltimer() - t0 < 10000000ull) {
          }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the even CTA's) ----------------
    if (lane == 0 && crank == 0) {
      uint32_t peer_tmem;
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_tmem) : "r"(peer_addr(sbase + kTmemSlot, 1))
                   : "memory");
      if (peer_tmem != tmem) {
        atomicExch(err, NERFGB_E_UNSUPPORTED);
        *abort_flag = 1;
      }
      RingPos rp{0, 0u};
      uint32_t actr_phase = 0;  // both sub-tiles' operand barriers, toggled per layer after the first
      for (int tile = 0; tile < ntiles; ++tile) {
        if (*abort_flag) break;
        const int nsub = 2 * tile + 1 < count ? 2 : 1;
#pragma unroll 1
        for (int i = 0; i < 9; ++i) {
          const RingPos start = rp;
          for (int s = 0; s < nsub; ++s) {
            // the first layer's operand is the copied dZ_9; its accumulator was read with dZ_0 of the tile before
            if (i == 0) wait_fast(sbase + kBarLoad + 8 * s, (uint32_t)(tile & 1), abort_flag, err);
            if (i > 0 || tile > 0) wait_fast(sbase + kBarActr + 8 * s, actr_phase, abort_flag, err);
            tc_fence_after();
            if (s == 1) rp = start;
            const bool release = s == nsub - 1;
            if (i == 0) {
              if (s == 0)
                issue_chain<2, 0>(sbase, tmem, release, rp, abort_flag, err);
              else
                issue_chain<2, 1>(sbase, tmem, release, rp, abort_flag, err);
            } else {
              if (s == 0)
                issue_chain<4, 0>(sbase, tmem, release, rp, abort_flag, err);
              else
                issue_chain<4, 1>(sbase, tmem, release, rp, abort_flag, err);
            }
            tc_commit_pair(sbase + kBarAccf + 8 * s);
          }
          if (i > 0 || tile > 0) actr_phase ^= 1u;
        }
      }
      if (ntiles > 0) {
        tc_commit_pair(sbase + kBarDrain);
        uint64_t t0 = globaltimer();
        while (!mbar_try(sbase + kBarDrain, 0) && globaltimer() - t0 < 100000000ull) {
        }
      }
    }
  } else if (warp >= 2 + kEpiWarps) {
    // ---------------- I/O of sub-tile s ----------------
    const int s = warp - 2 - kEpiWarps;
    if (lane == 0) {
      const uint32_t act = sbase + kActOff + s * kActBytes;
      const uint32_t accf = sbase + kBarAccf + 8 * s, rdy = sbase + kBarRdy + 8 * s, mask = sbase + kBarMask + 8 * s;
      uint32_t phase = 0, masks = 0;  // accf and rdy complete once per layer; masks: loads issued
      bool ok = true;
      for (int tile = 0; 2 * tile + s < count && ok; ++tile) {
        const int row = (int)row_of(tile, s);
        // dZ_9 (the region is free: dZ_0 of the tile before has been read by its store)
        const uint32_t load = sbase + kBarLoad + 8 * s;
        if (crank == 0) mbar_expect_tx(load, 2 * 2 * kAtom);
        tma_load_3d_pair(act, &maps.dz[9], row, 0, crank == 0 ? load : peer_addr(load, 0));
        for (int g = 9; g >= 1; --g) {
          if (!wait_bar(accf, phase, abort_flag, err)) {
            ok = false;
            break;
          }
          if (g < 9) {  // the region is free: the layer's activations
            mbar_expect_tx(mask, 4 * kAtom);
            tma_load_3d(act, &maps.act, row, acts_offset(g - 1) / 64, mask);
            ++masks;
          }
          // what the region takes after that, into L2
          if (g > 1)
            tma_prefetch_3d(&maps.act, row, acts_offset(g - 2) / 64);
          else if (2 * (tile + 1) + s < count)
            tma_prefetch_3d(&maps.dz[9], (int)row_of(tile + 1, s), 0);
          if (!wait_bar(rdy, phase, abort_flag, err)) {
            ok = false;
            break;
          }
          phase ^= 1u;
          if (row < n) {  // (a box from row n on would write nothing)
            tma_store_3d(&maps.dz[g - 1], act, 0, row, 0);
            bulk_commit();
            bulk_wait_read();
          }
        }
      }
      bulk_wait_all();
      if (!ok && masks > 0) {
        // Drain: the last mask copy still in flight (bounded).
        const uint64_t t0 = globaltimer();
        while (!mbar_try(mask, (masks - 1) & 1u) && globaltimer() - t0 < 10000000ull) {
        }
      }
    }
  } else {
    // ---------------- epilogue warps ----------------
    const int qd = warp & 3, hf = (warp - 2) >> 2;
    const uint32_t tlane = tmem + ((uint32_t)(32 * qd) << 16) + 128 * hf;
    const uint32_t frag_row =
        (uint32_t)(32 * qd + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128u + (uint32_t)(2 * hf) * kAtom;
    const uint32_t cx = (uint32_t)((lane >> 4) ^ (lane & 7));
    uint32_t accf_phase = 0, mask_phase = 0;
    bool ok = true;
#pragma unroll 1
    for (int tile = 0; tile < ntiles && ok; ++tile) {
      const int nsub = 2 * tile + 1 < count ? 2 : 1;
#pragma unroll 1
      for (int g = 9; g >= 1 && ok; --g) {
        // bias gradient of the layer whose dZ this is, dense_{g-1}
        float *db = bias + (g - 1) * kW + 128 * hf;
#pragma unroll 1
        for (int s = 0; s < nsub; ++s) {
          const uint32_t dst = sbase + kActOff + s * kActBytes + frag_row, ta = tlane + s * 256;
          float ds[4] = {0.f, 0.f, 0.f, 0.f};
          if (g == 8) {
            const long long row = row_of(tile, s) + 32 * qd + (lane >> 2);
#pragma unroll
            for (int i = 0; i < 4; ++i) ds[i] = row + 8 * i < n ? dsp[row + 8 * i] : 0.0f;
          }
          bool got = wait_bar(sbase + kBarAccf + 8 * s, accf_phase, abort_flag, err);
          if (got && g < 9) got = wait_bar(sbase + kBarMask + 8 * s, mask_phase, abort_flag, err);
          if (!__all_sync(0xffffffffu, got)) {
            ok = false;
            break;
          }
          tc_fence_after();
          uint32_t ra[32], rb[32];
          tmem_ld_frag64(ta, ra);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t d = dst + (uint32_t)c * kAtom;
            const float *w = ws + 128 * hf + 64 * c + 2 * (lane & 3);
            float sum[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
            tmem_wait32(ra);
            tmem_ld_frag64(ta + (16u << 16) + 64 * c, rb);
            if (g == 8)
              finish_frag<true, true>(d, cx, ra, ds[0], ds[1], w, sum);
            else if (g == 9)
              finish_frag<false, false>(d, cx, ra, 0.f, 0.f, w, sum);
            else
              finish_frag<true, false>(d, cx, ra, 0.f, 0.f, w, sum);
            tmem_wait32(rb);
            if (c == 0) tmem_ld_frag64(ta + 64, ra);
            if (g == 8)
              finish_frag<true, true>(d + 16 * 128, cx, rb, ds[2], ds[3], w, sum);
            else if (g == 9)
              finish_frag<false, false>(d + 16 * 128, cx, rb, 0.f, 0.f, w, sum);
            else
              finish_frag<true, false>(d + 16 * 128, cx, rb, 0.f, 0.f, w, sum);
            if (c == 1) {
              // the operand is written and the accumulator read
              fence_proxy_async();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) {
                mbar_arrive_remote(peer_addr(sbase + kBarActr + 8 * s, 0));
                mbar_arrive(sbase + kBarRdy + 8 * s);
              }
            }
            add_columns(sum, lane, db + 64 * c);
          }
        }
        accf_phase ^= 1u;
        if (g < 9) mask_phase ^= 1u;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (crank == 1 && warp == 1 && lane == 0 && ntiles > 0) {
    uint64_t t0 = globaltimer();
    while (!mbar_try(sbase + kBarDrain, 0) && globaltimer() - t0 < 100000000ull) {
    }
    // after a timeout (in either CTA) copies that complete on the even CTA's
    // barriers may be in flight: give them 100 us (mlp_tc.cu)
    uint32_t peer_abort;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_abort) : "r"(peer_addr(sbase + kAbort, 0)) : "memory");
    if (*abort_flag || peer_abort) {
      t0 = globaltimer();
      while (globaltimer() - t0 < 100000ull) {
      }
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

}  // namespace tcb

long long mlp_chain_pack_bytes() { return tcb::kPackBytes; }

int launch_mlp_chain_pack(const float *packed_fp32, void *wpack, cudaStream_t stream) {
  tcb::pack_kernel<<<dim3(256, 9), 256, 0, stream>>>(packed_fp32, reinterpret_cast<uint8_t *>(wpack));
  return launch_status();
}

int launch_mlp_chain(const void *wpack, const float *sigma_w, const uint16_t *tape, const float *dsp, long long n,
                     __nv_bfloat16 *dz, float *bias, int *ctas, int *err, cudaStream_t stream, const WaitTest &wt) {
  using namespace tcb;
  *ctas = 0;
  if (n == 0) return NERFGB_OK;
  if (cudaFuncSetAttribute(chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes) != cudaSuccess)
    return NERFGB_E_CUDA;
  const int sms = num_sms();
  if (sms <= 0) return NERFGB_E_DEVICE;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // co-resident pairs, asked once per device (as mlp_tc.cu)
  static std::mutex mu;
  static std::unordered_map<int, int> pairs_of_device;
  int dev = -1, max_pairs;
  if (cudaGetDevice(&dev) != cudaSuccess) return NERFGB_E_DEVICE;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto hit = pairs_of_device.find(dev);
    if (hit == pairs_of_device.end()) {
      cfg.gridDim = dim3((unsigned)(sms / 2 * 2));
      int m = 0;
      if (cudaOccupancyMaxActiveClusters(&m, chain_kernel, &cfg) != cudaSuccess) return NERFGB_E_CUDA;
      hit = pairs_of_device.emplace(dev, m).first;
    }
    max_pairs = hit->second < kChainMaxPairs ? hit->second : kChainMaxPairs;
  }
  if (max_pairs < 1) return NERFGB_E_UNSUPPORTED;
  const long long subs = (n + kSubRows - 1) / kSubRows, pairs = subs < max_pairs ? subs : max_pairs;
  cfg.gridDim = dim3((unsigned)(2 * pairs));
  *ctas = (int)(2 * pairs);
  Maps maps{};
  int rc;
  {
    const unsigned long long dims[2] = {128, (unsigned long long)(kPackBytes / 256)}, strides[1] = {256};
    const unsigned box[2] = {128, 64};
    if ((rc = encode_tensor_map_u16(&maps.w, wpack, 2, dims, strides, box)) != NERFGB_OK) return rc;
  }
  {
    const unsigned long long dims[3] = {64, (unsigned long long)n, kActsEncDir / 64};
    const unsigned long long strides[2] = {(unsigned long long)kActsLd * 2, 128};
    const unsigned box[3] = {64, 128, 4};
    if ((rc = encode_tensor_map_u16(&maps.act, tape, 3, dims, strides, box, true)) != NERFGB_OK) return rc;
  }
  for (int l = 0; l < kNumGemm; ++l) {
    const unsigned long long dims[3] = {64, (unsigned long long)n, 4}, strides[2] = {512, 128};
    const unsigned box[3] = {64, 128, l == 9 ? 2u : 4u};
    if ((rc = encode_tensor_map_u16(&maps.dz[l], dz + (long long)l * n * 256, 3, dims, strides, box, true)) != NERFGB_OK)
      return rc;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, chain_kernel, sigma_w, dsp, n, bias, err, wt, maps);
  rc = launch_status();  // (clears a failed launch's error)
  return e == cudaSuccess ? rc : NERFGB_E_CUDA;
}

}  // namespace nerfgb
