// Tensor-core BF16 weight gradients of the MLP backward (the gradient
// tf.GradientTape takes at nerf/core/model.py:148-170 through the Dense
// layers of model.py:366-387), FP32 accumulation in TMEM: for every layer
//
//   dW[k][n] = sum_m In[m][k] dZ[m][n]        (tcgen05.mma.cta_group::1.kind::f16)
//
// with In the tape's columns of the layer's input and dZ the layer's buffer,
// both read MN-major (the reduction along the rows) straight from row-major
// memory by tensor copies in the 128-byte swizzled layout: 3-D boxes of
// 64-element atoms by kKc rows by the atoms of the tile, atom a at a*8 KB, row
// k at k*128 bytes (smem_desc_mn_sw128, the instruction descriptor's transpose
// bits set), rows and atoms past the bounds zero-filled.
//
// Bound by HBM (every byte of tape and dZ once, dZ_0, dZ_5 and dZ_9 twice).
// All layers are one launch: a work item is a layer's product over a split of
// the rows, one split per SM and layer, so every CTA takes one item of each
// layer and the twelve launch tails are one: 2.0 ms of a 4,096-ray step (11.2
// GB, 5.6 TB/s) and 0.22 for the reduction, against 2.16 and 0.36 with a launch
// per layer.
// Fewer, longer splits would save partial sums (256 KB per item) but the
// tensor core's FP32 accumulation truncates: its error grows with the rows of
// one accumulation (4e-6 relative over 4,096 rows of random signs, 1.8e-5 over
// 16,384; the splits are added in FP32 with rounding). Each item's partial goes
// to a workspace and one reduction kernel adds the splits into the gradient blob.
//
// Warp roles (6 warps): 0-3 epilogue (TMEM lane quadrant = warp), 4 the
// loader (one thread, an NST-stage ring, full/empty mbarriers), 5 TMEM
// allocation and the MMA issuer (one thread). Items are taken persistently:
// item = blockIdx.x + i * gridDim.x.
//
// Every mbarrier wait is bounded (tc::wait_bar): on a timeout the kernel
// writes NERFGB_E_TIMEOUT to *err, every role stops, the loader drains its
// copies, the issuer drains its MMAs, TMEM is freed and the kernel returns.
#include <cuda_bf16.h>
#include <stdint.h>

#include "common.cuh"
#include "mlp_internal.cuh"
#include "tcgen05.cuh"

namespace nerfgb {
namespace gemm {

using namespace tc;

constexpr int kKc = 64;  // rows (K) per stage: 4 MMAs of K = 16
constexpr int kEpiWarps = 4;
constexpr int kLoadWarp = kEpiWarps, kIssuerWarp = kEpiWarps + 1;
constexpr int kThreads = (kIssuerWarp + 1) * 32;
constexpr uint32_t kAtomBytes = 64 * 128;     // 64 columns x kKc rows
constexpr uint32_t kABytes = 4 * kAtomBytes;  // up to 256 columns of In
constexpr uint32_t kStage = 2 * kABytes;
constexpr int kNst = 3;
constexpr uint32_t kBar0 = kNst * kStage;
constexpr uint32_t kBarFull = kBar0;         // [kNst]
constexpr uint32_t kBarEmpty = kBar0 + 32;   // [kNst]
constexpr uint32_t kBarAcc = kBar0 + 64;     // an item's accumulator is complete
constexpr uint32_t kBarTmem = kBar0 + 72;    // ... has been read
constexpr uint32_t kBarDrain = kBar0 + 80;
constexpr uint32_t kTmemSlot = kBar0 + 88;
constexpr uint32_t kAbort = kBar0 + 96;      // int, then the wait limit (u64) at +8
constexpr uint32_t kSmem = kBar0 + 112;
static_assert(kSmem <= 227 * 1024, "ring");

// One layer's product: In = tape atoms [atom, atom + 2 mt) (K of their columns
// are rows of the gradient, the rest is ignored), dZ of layer slot, N columns;
// the gradient of flat layer `flat`, rows k_dst0 ..
struct Job {
  int atom, mt, K, slot, N, flat, k_dst0;
};
constexpr int kJobs = 12;
__host__ __device__ constexpr Job job_of(int j) {
  return j == 0   ? Job{acts_offset(8) / 64, 2, 256, 9, 128, 10, 0}
         : j == 1 ? Job{kActsEncDir / 64, 1, 27, 9, 128, 10, 256}
         : j == 2 ? Job{acts_offset(7) / 64, 2, 256, 8, 256, 9, 0}
         : j == 3 ? Job{kActsEncXyz / 64, 1, 63, 5, 256, 5, 256}
         : j == 4 ? Job{kActsEncXyz / 64, 1, 63, 0, 256, 0, 0}
                  : Job{acts_offset(j - 5) / 64, 2, 256, j - 4, 256, j - 4, 0};  // dense_1 .. dense_7
}
static_assert(kActsEncDir % 64 == 0 && kActsEncXyz == 0 && acts_offset(0) % 64 == 0, "inputs start on tape atoms");
// Items: job j's split i is item j * splits + i, the 64-row chunks [i * chunks
// / splits, (i + 1) * chunks / splits).
struct Split {
  int splits;
  long long chunks, M;
  __host__ __device__ void rows(int i, long long &kb, long long &ke) const {
    kb = i * chunks / splits * kKc;
    ke = (i + 1) * chunks / splits * kKc;
    if (ke > M) ke = M;
  }
};

struct Maps {
  CUtensorMap a[2];          // the tape, boxes of 2 and 4 atoms
  CUtensorMap b[kNumGemm];   // dZ per layer, boxes of its columns
};

// One box of a 3-D tensor map into shared memory at dst, completing on the
// mbarrier bar (coordinates innermost first).
__device__ __forceinline__ void tma_3d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}

// Descriptor of an MN-major operand in the 128-byte swizzled layout: atoms
// of 64 MN-elements (128-byte rows, one per K row), 64 K rows each (8 KB),
// each 1024-byte block of 8 K rows with its 16-byte chunks permuted by the
// row (as the 128-byte-swizzle tensor copy of a box of 64 elements x 64
// rows x atoms writes them; blocks 1024-byte aligned). LBO = 8192 (between
// MN atoms), SBO = 1024 (between 8-row K blocks), swizzle mode 2; a K step
// of 16 rows advances the start address by 2048 bytes.
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(8192u >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

__global__ void __launch_bounds__(kThreads, 1)
    dw_kernel(float *__restrict__ part, int *__restrict__ err, const Split split,
              const __grid_constant__ Maps maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kAbort);
  // (the swizzled stages need 1024-byte alignment: without it nothing runs)
  const int items = (sbase & 1023u) != 0 ? 0 : kJobs * split.splits;
  auto item = [&](int it, Job &job, long long &kb, long long &ke) {
    job = job_of(it / split.splits);
    split.rows(it % split.splits, kb, ke);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kNst; ++s) {
      mbar_init(sbase + kBarFull + 8 * s, 1);
      mbar_init(sbase + kBarEmpty + 8 * s, 1);
    }
    mbar_init(sbase + kBarAcc, 1);
    mbar_init(sbase + kBarTmem, kEpiWarps);
    mbar_init(sbase + kBarDrain, 1);
    *abort_flag = 0;
    set_wait_limit(abort_flag, kWaitNs);
    if ((sbase & 1023u) != 0) atomicExch(err, NERFGB_E_UNSUPPORTED);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssuerWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kTmemSlot),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + kTmemSlot);

  if (warp == kLoadWarp) {
    // ---------------- loader ----------------
    if (lane == 0) {
      long long q = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
        Job job;
        long long kb, ke;
        item(it, job, kb, ke);
        const uint32_t bytes = (uint32_t)(2 * job.mt + job.N / 64) * kAtomBytes;
        for (long long k0 = kb; k0 < ke; k0 += kKc, ++q) {
          const int st = (int)(q % kNst);
          if (!wait_bar(sbase + kBarEmpty + 8 * st, (uint32_t)((q / kNst) & 1) ^ 1u, abort_flag, err) || *abort_flag) {
            ok = false;
            break;
          }
          const uint32_t full = sbase + kBarFull + 8 * st, sa = sbase + st * kStage;
          mbar_expect_tx(full, bytes);
          tma_3d(sa, &maps.a[job.mt - 1], 0, (int)k0, job.atom, full);
          tma_3d(sa + kABytes, &maps.b[job.slot], 0, (int)k0, 0, full);
        }
      }
      if (!ok) {
        // Drain: wait (bounded) for the copies of the stages still in flight.
        const uint64_t t0 = globaltimer();
        for (long long d = q > kNst ? q - kNst : 0; d < q; ++d)
          while (!mbar_try(sbase + kBarFull + 8 * (int)(d % kNst), (uint32_t)((d / kNst) & 1)) &&
                 globaltimer() - t0 < 10000000ull) {
          }
      }
    }
  } else if (warp == kIssuerWarp) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      long long q = 0;
      uint32_t n_items = 0;
      bool issued = false;
      for (int it = blockIdx.x; it < items; it += gridDim.x, ++n_items) {
        if (*abort_flag) break;
        Job job;
        long long kb, ke;
        item(it, job, kb, ke);
        const uint32_t idesc = idesc_bf16(128, 0) | (1u << 15) | (1u << 16) | ((uint32_t)(job.N >> 3) << 17);
        // the epilogue has read the item before's accumulator
        if (n_items > 0) {
          if (!wait_bar(sbase + kBarTmem, (n_items - 1) & 1u, abort_flag, err)) break;
          tc_fence_after();
        }
        uint32_t acc = 0;
        for (long long k0 = kb; k0 < ke; k0 += kKc, ++q) {
          const int st = (int)(q % kNst);
          if (!wait_bar(sbase + kBarFull + 8 * st, (uint32_t)((q / kNst) & 1), abort_flag, err)) break;
          tc_fence_after();
          const uint32_t sa = (sbase + st * kStage) & 0x3FFFFu, sb = sa + kABytes;
#pragma unroll
          for (int s = 0; s < kKc / 16; ++s) {
            const uint64_t bdesc = smem_desc_mn_sw128(sb + 2048u * s);
            tc_mma(tmem, smem_desc_mn_sw128(sa + 2048u * s), bdesc, idesc, acc);
            if (job.mt == 2) tc_mma(tmem + 256, smem_desc_mn_sw128(sa + 2 * kAtomBytes + 2048u * s), bdesc, idesc, acc);
            acc = 1;
          }
          issued = true;
          tc_commit(sbase + kBarEmpty + 8 * st);
        }
        if (*abort_flag) break;
        tc_commit(sbase + kBarAcc);
      }
      if (issued) {
        tc_commit(sbase + kBarDrain);
        const uint64_t t0 = globaltimer();
        while (!mbar_try(sbase + kBarDrain, 0) && globaltimer() - t0 < 100000000ull) {
        }
      }
    }
  } else {
    // ---------------- epilogue: the item's partial sums, [256][256] FP32 ----------------
    uint32_t n_items = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x, ++n_items) {
      Job job;
      long long kb, ke;
      item(it, job, kb, ke);
      if (!__all_sync(0xffffffffu, wait_bar(sbase + kBarAcc, n_items & 1u, abort_flag, err))) break;
      tc_fence_after();
#pragma unroll 1
      for (int h = 0; h < job.mt; ++h) {
        const int r = h * 128 + 32 * warp + lane;  // row of dW (= TMEM lane)
        if (h * 128 + 32 * warp >= job.K) continue;
        const uint32_t tl = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)h * 256u;
#pragma unroll 1
        for (int j = 0; j < job.N / 32; ++j) {
          uint32_t raw[32];
          tmem_ld32(tl + 32u * j, raw);
          tmem_wait32(raw);
          float4 *dst = reinterpret_cast<float4 *>(part + ((long long)it * 256 + r) * 256 + 32 * j);
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            dst[q4] = make_float4(__uint_as_float(raw[4 * q4]), __uint_as_float(raw[4 * q4 + 1]),
                                  __uint_as_float(raw[4 * q4 + 2]), __uint_as_float(raw[4 * q4 + 3]));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(sbase + kBarTmem);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kIssuerWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// grads[k_dst0 + r][c] += sum over the job's splits of part[item][r][c], r < K,
// c < N; blocks [first(j), first(j + 1)) are job j's. A block takes 64
// elements; its four warp pairs sum the splits s = g, g + 4, ... (g = the
// pair) in order, and the four sums are added in order: the same result
// whatever the launch.
constexpr int kRedElems = 64, kRedGroups = 4;
__host__ __device__ constexpr int red_first(int j) {
  int b = 0;
  for (int i = 0; i < j; ++i) b += job_of(i).K * job_of(i).N / kRedElems;
  return b;
}
static_assert(27 * 128 % kRedElems == 0 && 63 * 256 % kRedElems == 0, "whole blocks per job");

__global__ void __launch_bounds__(kRedElems *kRedGroups)
    reduce_splits_kernel(const float *__restrict__ part, const Split split, float *__restrict__ grads) {
  __shared__ float sums[kRedGroups][kRedElems];
  int j = 0;
  while (j + 1 < kJobs && (int)blockIdx.x >= red_first(j + 1)) ++j;
  const Job job = job_of(j);
  const int t = threadIdx.x % kRedElems, grp = threadIdx.x / kRedElems;
  const int e = ((int)blockIdx.x - red_first(j)) * kRedElems + t, r = e / job.N, c = e % job.N;
  float s = 0.0f;
  for (int k = grp; k < split.splits; k += kRedGroups)
    s += part[((long long)(j * split.splits + k) * 256 + r) * 256 + c];
  sums[grp][t] = s;
  __syncthreads();
  if (grp == 0)
    grads[flat_offset(job.flat) + (long long)(job.k_dst0 + r) * job.N + c] +=
        ((sums[0][t] + sums[1][t]) + sums[2][t]) + sums[3][t];
}

}  // namespace gemm

// Splits of a layer: one per SM, at most kDwSplits (the workspace), at most
// one per 64 rows.
constexpr int kDwSplits = 152;
long long gemm_dw_partial_floats(long long M) {
  const long long chunks = (M + gemm::kKc - 1) / gemm::kKc;
  return gemm::kJobs * (chunks < kDwSplits ? chunks : kDwSplits) * 256 * 256;
}

int launch_gemm_dw(const uint16_t *tape, const __nv_bfloat16 *dz, long long M, float *grads, float *part, int *err,
                   cudaStream_t st) {
  using namespace gemm;
  if (M == 0) return NERFGB_OK;
  if (cudaFuncSetAttribute(dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess)
    return NERFGB_E_CUDA;
  const int sms = num_sms();
  if (sms <= 0) return NERFGB_E_DEVICE;
  Split split{};
  split.M = M;
  split.chunks = (M + kKc - 1) / kKc;
  split.splits = sms < kDwSplits ? sms : kDwSplits;
  if (split.chunks < split.splits) split.splits = (int)split.chunks;
  Maps maps{};
  int rc;
  for (int i = 0; i < 2; ++i) {
    // atoms past the row's last whole one belong to the next row: not in the map
    const unsigned long long dims[3] = {64, (unsigned long long)M, kActsLd / 64};
    const unsigned long long strides[2] = {(unsigned long long)kActsLd * 2, 128};
    const unsigned box[3] = {64, kKc, i == 0 ? 2u : 4u};
    if ((rc = encode_tensor_map_u16(&maps.a[i], tape, 3, dims, strides, box, true)) != NERFGB_OK) return rc;
  }
  for (int l = 0; l < kNumGemm; ++l) {
    const unsigned long long dims[3] = {64, (unsigned long long)M, 4}, strides[2] = {512, 128};
    const unsigned box[3] = {64, kKc, l == 9 ? 2u : 4u};
    if ((rc = encode_tensor_map_u16(&maps.b[l], dz + (long long)l * M * 256, 3, dims, strides, box, true)) != NERFGB_OK)
      return rc;
  }
  // a grid of the splits: CTA i takes split i of every layer
  dw_kernel<<<split.splits, kThreads, kSmem, st>>>(part, err, split, maps);
  if ((rc = launch_status()) != NERFGB_OK) return rc;
  reduce_splits_kernel<<<red_first(kJobs), kRedElems * kRedGroups, 0, st>>>(part, split, grads);
  return launch_status();
}

}  // namespace nerfgb
