// Tensor-core BF16 weight gradients of the MLP backward (the gradient
// tf.GradientTape takes at nerf/core/model.py:148-170 through the Dense
// layers of model.py:366-387), FP32 accumulation: for every layer
//
//   dW[k][n] = sum_m In[m][k] dZ[m][n]        (tcgen05.mma.cta_group::2.kind::f16)
//
// with In the tape's columns of the layer's input and dZ the layer's buffer,
// both read MN-major (the reduction along the rows) straight from row-major
// memory by tensor copies in the 128-byte swizzled layout: 3-D boxes of
// 64-element atoms by kRows rows by the atoms of the operand, atom a at a*8 KB,
// row k at k*128 bytes (desc_mn_sw128, the instruction descriptor's transpose
// bits set), rows past the bounds zero-filled.
//
// Bound by HBM (every byte of tape and dZ once, dZ_5, dZ_9 and enc_xyz twice:
// 11.1 GB of a 4,096-ray step). All layers are one launch; the 64-row stages of
// all jobs in order are dealt evenly to the pairs, so a pair has one or two
// layers' sums at a time. The tensor core's FP32 accumulation
// truncates (4e-6 relative over 4,096 rows of random signs), so an accumulator
// takes a window of 1, 2 or 4 stages (launch_gemm_dw) and the windows' sums are
// added in registers with rounding, one accumulator in TMEM being read while the
// other fills. A layer's pairs leave partial sums in a workspace that one
// reduction kernel adds into the gradient, always in the same order, without the
// additions' rounding. With the accumulators themselves as the partial sums a
// layer had to be split 152 times (up to ~5,000 rows each) and their 0.48 GB were
// written and read per network: 2.0 ms of the step, and 0.22 for the reduction;
// 1.73 and 0.04 here (6.5 TB/s). Error of the sums against 64 bits, from the same
// dZ, of their norm (as split 152 times): 1,000 rows 6e-8 (7e-8), 20,000 1.3e-7
// (1.6e-7), 786,432 4e-7 (5e-6).
//
// Warp roles (12 warps): 0-7 the windows' sums (TMEM lane quadrant w % 4, column
// half w / 4; 128 registers each), 8 the loader (one thread, a kNst-stage ring,
// full/empty mbarriers), 9 the MMA issuer (one thread of the even CTA).
//
// Every mbarrier wait is bounded (tc::wait_bar): on a timeout the kernel
// writes NERFGB_E_TIMEOUT to *err, every role stops, the loader drains its
// copies, the issuer drains its MMAs, TMEM is freed and the kernel returns.
#include <cuda_bf16.h>
#include <stdint.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "mlp_internal.cuh"
#include "tcgen05.cuh"

namespace nerfgb {
namespace gemm {

using namespace tc;

constexpr int kRows = 64;   // rows (K) per stage: 4 MMAs of K = 16
constexpr int kSumWarps = 8, kLoadWarp = 8, kIssuerWarp = 9, kThreads = 12 * 32;
constexpr uint32_t kAtomBytes = 64 * 128;  // 64 columns x kRows rows
constexpr uint32_t kOperand = 2 * kAtomBytes;
constexpr uint32_t kStage = 2 * kOperand;  // A, B: up to 128 columns each per CTA
constexpr int kNst = 6;
constexpr int kMaxPairs = 76;  // (the workspace)
constexpr uint32_t kBar0 = kNst * kStage;
constexpr uint32_t kBarFull = kBar0;         // [kNst] (both CTAs' copies, on the even CTA)
constexpr uint32_t kBarEmpty = kBar0 + 48;   // [kNst]
constexpr uint32_t kBarAcc = kBar0 + 96;     // [2] a window's accumulator is complete
constexpr uint32_t kBarRead = kBar0 + 112;   // [2] ... has been read (by both CTAs)
constexpr uint32_t kBarDrain = kBar0 + 128;
constexpr uint32_t kTmemSlot = kBar0 + 136;
constexpr uint32_t kAbort = kBar0 + 144;     // int, then the wait limit (u64) at +8
constexpr uint32_t kSmem = kBar0 + 160;
static_assert(kSmem <= 227 * 1024, "ring");

// One product. Plain: A = 256 columns of the tape from `atom` (64 columns each)
// on, the layer's input, B = the dZ of `slot` (N columns). Flipped (inputs of
// fewer than 64 columns, K): A = the dZ of `slot` (N columns), B = the tape's
// atom, in the even CTA alone, of which K columns count; the result is
// transposed. The gradient of flat layer `flat`, rows k_dst0 ..
struct Job {
  int atom, slot, K, N, flat, k_dst0;
  bool flip;
  // columns of the MMA, and this CTA's atoms of A and B
  __host__ __device__ constexpr int n_mma() const { return flip ? 128 : N; }
  __host__ __device__ constexpr int atoms_a(int rank) const { return flip && N == 128 && rank == 1 ? 0 : 2; }
  __host__ __device__ constexpr int atoms_b(int rank) const { return flip ? 1 - rank : N / 128; }
  __host__ __device__ constexpr int atoms() const { return atoms_a(0) + atoms_a(1) + atoms_b(0) + atoms_b(1); }
};
constexpr int kJobs = 12;
__host__ __device__ constexpr Job job_of(int j) {
  return j == 0   ? Job{acts_offset(8) / 64, 9, 256, 128, 10, 0, false}
         : j == 1 ? Job{kActsEncDir / 64, 9, 27, 128, 10, 256, true}
         : j == 2 ? Job{acts_offset(7) / 64, 8, 256, 256, 9, 0, false}
         : j == 3 ? Job{kActsEncXyz / 64, 5, 63, 256, 5, 256, true}
         : j == 4 ? Job{kActsEncXyz / 64, 0, 63, 256, 0, 0, true}
                  : Job{acts_offset(j - 5) / 64, j - 4, 256, 256, j - 4, 0, false};  // dense_1 .. dense_7
}
static_assert(kActsEncDir % 64 == 0 && kActsEncXyz == 0 && acts_offset(0) % 64 == 0, "inputs start on tape atoms");
// A pair's stages of job j (every job has `stages`): all jobs' stages in order,
// dealt evenly by number (the narrow jobs' take as long: a copy's latency over
// the ring's stages, not its bytes; dealt by bytes dW took 1.3 times as long).
// Its partial sums go to slot pair + j (of two items in order, one of the two
// is greater).
__device__ __forceinline__ void stages_of(int j, long long stages, int pair, int pairs, long long &b, long long &e) {
  const long long lo = pair * (kJobs * stages) / pairs - j * stages, hi = (pair + 1) * (kJobs * stages) / pairs - j * stages;
  b = lo < 0 ? 0 : lo > stages ? stages : lo;
  e = hi < 0 ? 0 : hi > stages ? stages : hi;
}

struct Maps {
  CUtensorMap tape[2];           // boxes of 1 and 2 atoms
  CUtensorMap dz[kNumGemm][2];   // per layer
};

// Descriptor of an MN-major operand in the 128-byte swizzled layout: atoms
// of 64 MN-elements (128-byte rows, one per K row), 64 K rows each (8 KB),
// each 1024-byte block of 8 K rows with its 16-byte chunks permuted by the
// row (as the 128-byte-swizzle tensor copy of a box of 64 elements x 64
// rows x atoms writes them; blocks 1024-byte aligned). LBO = 8192 (between
// MN atoms), SBO = 1024 (between 8-row K blocks), swizzle mode 2; a K step
// of 16 rows advances the start address by 2048 bytes.
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(8192u >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

__global__ void __launch_bounds__(kThreads, 1)
    dw_kernel(float *__restrict__ part, int *__restrict__ err, long long n, int window, WaitTest wt,
              const __grid_constant__ Maps maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_rank();
  const int pair = (int)cluster_id(), pairs = (int)cluster_count();
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kAbort);
  // (the swizzled stages need 1024-byte alignment: without it nothing runs)
  const long long stages = (sbase & 1023u) != 0 ? 0 : (n + kRows - 1) / kRows;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kNst; ++s) {
      mbar_init(sbase + kBarFull + 8 * s, 1);
      mbar_init(sbase + kBarEmpty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(sbase + kBarAcc + 8 * s, 1);
      mbar_init(sbase + kBarRead + 8 * s, 2 * kSumWarps);
    }
    mbar_init(sbase + kBarDrain, 1);
    *abort_flag = 0;
    set_wait_limit(abort_flag, wt.wait_ns != 0 ? wt.wait_ns : kWaitNs);
    if ((sbase & 1023u) != 0) atomicExch(err, NERFGB_E_UNSUPPORTED);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssuerWarp) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kTmemSlot),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + kTmemSlot);

  if (warp == kLoadWarp) {
    // ---------------- loader ----------------
    if (lane == 0) {
      uint32_t used = 0;  // bit st: parity of the copies issued into stage st
      int st = 0;
      bool ok = true, withheld = wt.withhold == 0;
      for (int j = 0; j < kJobs && ok; ++j) {
        const Job job = job_of(j);
        long long sb, se;
        stages_of(j, stages, pair, pairs, sb, se);
        const int na = job.atoms_a(crank), nb = job.atoms_b(crank);
        const CUtensorMap *ma = job.flip ? &maps.dz[job.slot][1] : &maps.tape[1];
        const CUtensorMap *mb = job.flip ? &maps.tape[0] : &maps.dz[job.slot][job.N / 128 - 1];
        // first atoms
        const int a0 = (job.flip ? 0 : job.atom) + 2 * (int)crank, b0 = job.flip ? job.atom : (job.N / 128) * (int)crank;
        for (long long i = sb; i < se; ++i) {
          if (!wait_bar(sbase + kBarEmpty + 8 * st, ((used >> st) & 1u) ^ 1u, abort_flag, err)) {
            ok = false;
            break;
          }
          const uint32_t full = sbase + kBarFull + 8 * st, to = sbase + st * kStage;
          const uint32_t bar = crank == 0 ? full : peer_addr(full, 0);
          if (st == 1 && crank == 0 && !withheld) {
            withheld = true;  // (test hook: this stage's copies are left out)
          } else {
            if (crank == 0) mbar_expect_tx(full, (uint32_t)job.atoms() * kAtomBytes);
            if (na) tma_load_3d_pair(to, ma, (int)(i * kRows), a0, bar);
            if (nb) tma_load_3d_pair(to + kOperand, mb, (int)(i * kRows), b0, bar);
          }
          used ^= 1u << st;
          if (++st == kNst) st = 0;
        }
      }
      if (!ok && crank == 0) {
        // Drain: wait (bounded) for the stages' last copies.
        const uint64_t t0 = globaltimer();
        for (int k = 0; k < kNst; ++k)
          while (!mbar_try(sbase + kBarFull + 8 * k, ((used >> k) & 1u) ^ 1u) && globaltimer() - t0 < 10000000ull) {
          }
      }
    }
  } else if (warp == kIssuerWarp) {
    // ---------------- MMA issuer ----------------
    if (lane == 0 && crank == 0) {
      // both CTAs must hold the same TMEM columns (the collective allocation gives them)
      uint32_t peer_tmem;
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_tmem) : "r"(peer_addr(sbase + kTmemSlot, 1))
                   : "memory");
      if (peer_tmem != tmem) {
        atomicExch(err, NERFGB_E_UNSUPPORTED);
        *abort_flag = 1;
      }
      uint32_t phase = 0, w = 0;  // bit st: parity of the stage's next copies; windows so far
      int st = 0;
      for (int j = 0; j < kJobs && !*abort_flag; ++j) {
        const Job job = job_of(j);
        long long sb, se;
        stages_of(j, stages, pair, pairs, sb, se);
        const uint32_t idesc = idesc_bf16(256, 0) | (1u << 15) | (1u << 16) | ((uint32_t)(job.n_mma() >> 3) << 17);
        for (long long i = sb; i < se && !*abort_flag; i += window, ++w) {
          const int count = (int)(se - i < window ? se - i : window);
          // the sums have read the window before last
          if (!wait_bar(sbase + kBarRead + 8 * (w & 1), ((w >> 1) & 1u) ^ 1u, abort_flag, err)) break;
          tc_fence_after();
          for (int c = 0; c < count; ++c) {
            if (!wait_bar(sbase + kBarFull + 8 * st, (phase >> st) & 1u, abort_flag, err)) break;
            tc_fence_after();
            const uint64_t a = desc_mn_sw128(sbase + st * kStage), b = desc_mn_sw128(sbase + st * kStage + kOperand);
#pragma unroll
            for (int s = 0; s < kRows / 16; ++s)
              tc_mma_pair(tmem + 256u * (w & 1), a + (2048 >> 4) * s, b + (2048 >> 4) * s, idesc, c + s > 0 ? 1u : 0u);
            tc_commit_pair(sbase + kBarEmpty + 8 * st);
            phase ^= 1u << st;
            if (++st == kNst) st = 0;
          }
          tc_commit_pair(sbase + kBarAcc + 8 * (w & 1));
        }
      }
      if (stages > 0) {
        // Drain every MMA issued before TMEM is released (in both CTAs).
        tc_commit_pair(sbase + kBarDrain);
        const uint64_t t0 = globaltimer();
        while (!mbar_try(sbase + kBarDrain, 0) && globaltimer() - t0 < 100000000ull) {
        }
      }
    }
  } else if (warp < kSumWarps) {
    // ---------------- the windows' sums, then the item's partial, [256][256] FP32 ----------------
    const int qd = warp & 3, h = warp >> 2;
    const uint32_t tl = tmem + ((uint32_t)(32 * qd) << 16);
    bool ok = true;
    uint32_t w = 0;
#pragma unroll 1
    for (int j = 0; j < kJobs && ok; ++j) {
      const Job job = job_of(j);
      long long sb, se;
      stages_of(j, stages, pair, pairs, sb, se);
      if (sb >= se) continue;
      const int cols = (job.flip ? 64 : job.N) / 2, c0 = h * cols;  // 128, 64 or 32
      float sum[4][2][16];
#pragma unroll
      for (int f = 0; f < 8; ++f)
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[f / 2][f % 2][i] = 0.0f;
#pragma unroll 1
      for (int left = (int)((se - sb + window - 1) / window); left > 0; --left, ++w) {
        if (!__all_sync(0xffffffffu, wait_bar(sbase + kBarAcc + 8 * (w & 1), (w >> 1) & 1u, abort_flag, err))) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int f = 0; f < 8; ++f) {
          if (32 * (f / 2) < cols) {
            uint32_t raw[16];
            tmem_ld_frag32(tl + ((uint32_t)(16 * (f % 2)) << 16) + 256u * (w & 1) + c0 + 32 * (f / 2), raw);
            tmem_wait16(raw);
            float *s = sum[f / 2][f % 2];
#pragma unroll
            for (int i = 0; i < 16; i += 2)
              add_f32x2(s[i], s[i + 1], s[i], s[i + 1], __uint_as_float(raw[i]), __uint_as_float(raw[i + 1]));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(peer_addr(sbase + kBarRead + 8 * (w & 1), 0));
      }
      if (!ok) break;
      // rows of D: the layer's inputs (flipped: outputs); columns: its outputs (inputs)
      float *dst = part + ((long long)(pair + j) * 256 + crank * 128 + 32 * qd + lane / 4) * 256 + c0 + 2 * (lane % 4);
#pragma unroll
      for (int f = 0; f < 8; ++f) {
        if (32 * (f / 2) >= cols) continue;
#pragma unroll
        for (int i = 0; i < 16; i += 2)
          *reinterpret_cast<float2 *>(dst + (16 * (f % 2) + 8 * ((i >> 1) & 1)) * 256 + 32 * (f / 2) + 8 * (i / 4)) =
              make_float2(sum[f / 2][f % 2][i], sum[f / 2][f % 2][i + 1]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (crank == 1 && threadIdx.x == 0 && stages > 0) {
    // the even CTA's MMAs read this CTA's stages: its last commit
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
  if (warp == kIssuerWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// grads[k_dst0 + k][c] += the job's partial sums, pair after pair; blocks
// [first(j), first(j + 1)) are job j's, kRedElems elements each; those from
// first(kJobs) on add the CTAs' bias sums of dense_0 .. dense_8, then the heads'
// (a warp per element).
constexpr int kRedElems = 64;
__host__ __device__ constexpr int red_first(int j) {
  int b = 0;
  for (int i = 0; i < j; ++i) b += job_of(i).K * job_of(i).N / kRedElems;
  return b;
}
static_assert(27 * 128 % kRedElems == 0 && 63 * 256 % kRedElems == 0, "whole blocks per job");

__global__ void __launch_bounds__(kRedElems)
    reduce_kernel(const float *__restrict__ part, long long stages, int pairs, const float *__restrict__ bias, int ctas,
                  const float *__restrict__ heads, int head_blocks, float *__restrict__ grads) {
  constexpr int kBiasEnd = red_first(kJobs) + kChainBias / kRedElems;
  if ((int)blockIdx.x >= kBiasEnd) {
    const int e = ((int)blockIdx.x - kBiasEnd) * (kRedElems / 32) + threadIdx.x / 32;
    add_head_sums(heads, head_blocks, e, threadIdx.x % 32, grads);
    return;
  }
  if ((int)blockIdx.x >= red_first(kJobs)) {
    const int e = ((int)blockIdx.x - red_first(kJobs)) * kRedElems + threadIdx.x, l = e / kW;
    const int fl = flat_idx_of_gemm(l);
    Sum sum;
#pragma unroll 8
    for (int i = 0; i < ctas; ++i) sum.add(bias[(long long)i * kChainBias + e]);
    grads[flat_offset(fl) + (long long)flat_in(fl) * flat_out(fl) + e % kW] += sum.total();
    return;
  }
  int j = 0;
  while (j + 1 < kJobs && (int)blockIdx.x >= red_first(j + 1)) ++j;
  const Job job = job_of(j);
  const int e = ((int)blockIdx.x - red_first(j)) * kRedElems + threadIdx.x;
  // element k, c of the gradient; flipped: of the partial's row c, column k (lanes along c either way)
  const int k = e / job.N, c = e % job.N;
  const long long at = job.flip ? (long long)c * 256 + k : (long long)k * 256 + c;
  // the pairs whose share meets the job's
  const int first = j * pairs / kJobs, count = min((j + 1) * pairs / kJobs, pairs - 1) - first + 1;
  __shared__ bool any[kMaxPairs];
  for (int p = threadIdx.x; p < count; p += kRedElems) {
    long long b, t;
    stages_of(j, stages, first + p, pairs, b, t);
    any[p] = b < t;
  }
  __syncthreads();
  const float *src = part + (long long)(first + j) * 65536 + at;
  Sum sum;
#pragma unroll 4
  for (int p = 0; p < count; ++p) sum.add(any[p] ? src[p * 65536LL] : 0.0f);
  grads[flat_offset(job.flat) + (long long)(job.k_dst0 + k) * job.N + c] += sum.total();
}

}  // namespace gemm

long long gemm_dw_partial_floats() { return (gemm::kMaxPairs + gemm::kJobs) * 65536LL; }

int launch_gemm_dw(const uint16_t *tape, const __nv_bfloat16 *dz, long long n, float *grads, float *part,
                   const float *bias, int ctas, const float *heads, int head_blocks, int *err, cudaStream_t st,
                   const WaitTest &wt) {
  using namespace gemm;
  if (n == 0) return NERFGB_OK;
  if (cudaFuncSetAttribute(dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess)
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
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // co-resident pairs, asked once per device (as mlp_tc.cu)
  static std::mutex mu;
  static std::unordered_map<int, int> pairs_of_device;
  int dev = -1, most;
  if (cudaGetDevice(&dev) != cudaSuccess) return NERFGB_E_DEVICE;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto hit = pairs_of_device.find(dev);
    if (hit == pairs_of_device.end()) {
      cfg.gridDim = dim3((unsigned)(sms / 2 * 2));
      int m = 0;
      if (cudaOccupancyMaxActiveClusters(&m, dw_kernel, &cfg) != cudaSuccess) return NERFGB_E_CUDA;
      hit = pairs_of_device.emplace(dev, m).first;
    }
    most = hit->second < gemm::kMaxPairs ? hit->second : gemm::kMaxPairs;
  }
  if (most < 1) return NERFGB_E_UNSUPPORTED;
  const long long stages = (n + kRows - 1) / kRows;
  const int pairs = (int)(kJobs * stages < most ? kJobs * stages : most);
  cfg.gridDim = dim3((unsigned)(2 * pairs));
  Maps maps{};
  int rc;
  for (unsigned i = 0; i < 2; ++i) {
    const unsigned box[3] = {64, kRows, i + 1};
    {
      // atoms past the row's last whole one belong to the next row: not in the map
      const unsigned long long dims[3] = {64, (unsigned long long)n, kActsLd / 64};
      const unsigned long long strides[2] = {(unsigned long long)kActsLd * 2, 128};
      if ((rc = encode_tensor_map_u16(&maps.tape[i], tape, 3, dims, strides, box, true)) != NERFGB_OK) return rc;
    }
    for (int l = 0; l < kNumGemm; ++l) {
      const unsigned long long dims[3] = {64, (unsigned long long)n, 4}, strides[2] = {512, 128};
      if ((rc = encode_tensor_map_u16(&maps.dz[l][i], dz + (long long)l * n * 256, 3, dims, strides, box, true)) !=
          NERFGB_OK)
        return rc;
    }
  }
  // Stages per window: short ones for few rows, where what an accumulator cuts
  // off is most of the error (a pair of 2 to 32 stages: 6e-8 - 9e-8 of the sums'
  // norm with windows of one, 9e-8 - 1.2e-7 of two, 1.1e-7 - 1.9e-7 of four), longer
  // ones for many, where it is the additions' rounding (1,940 stages: 7.5e-7 with
  // one, 5.4e-7 with two, 4.1e-7 with four). The times are alike (786,432 rows 2.82, 2.82,
  // 2.81 ms of backward).
  const long long each = kJobs * stages / pairs;
  const int window = each <= 32 ? 1 : each <= 512 ? 2 : 4;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, dw_kernel, part, err, n, window, wt, maps);
  if ((rc = launch_status()) != NERFGB_OK) return rc;  // (clears a failed launch's error)
  if (e != cudaSuccess) return NERFGB_E_CUDA;
  static_assert(kChainBias % kRedElems == 0 && kHeadSums % (kRedElems / 32) == 0, "whole blocks of bias and head sums");
  reduce_kernel<<<red_first(kJobs) + kChainBias / kRedElems + kHeadSums / (kRedElems / 32), kRedElems, 0, st>>>(
      part, stages, pairs, bias, ctas, heads, head_blocks, grads);
  return launch_status();
}

}  // namespace nerfgb
