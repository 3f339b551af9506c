// The products of the FP32 MLP backward on the tensor cores (the gradient
// tf.GradientTape takes at nerf/core/model.py:148-170 through the Dense
// layers of model.py:366-387): for every layer
//
//   dW[k][n] += sum_m In[m][k] dZ[m][n],   db[n] += sum_m dZ[m][n]    (dw_kernel)
//   dZ_prev[m][k] = (sum_n dZ[m][n] W[k][n] + dpre_sigma[m] ws[k])
//                   * [h_prev[m][k] > 0]                             (chain_kernel)
//
// in FP32 accuracy from BF16 products. An FP32 value is exactly the sum of
// three BF16 values (x rounded, what that leaves rounded, and the rest: 24
// significant bits in three groups of eight); of the nine products of two such
// sums the six largest are taken (x0 y0, x0 y1, x1 y0, x1 y1, x0 y2, x2 y0: what
// is left out is below 2^-24 of the product and of either sign).
//
// The tensor core's FP32 accumulation truncates. So x0 y0, a product of 16 bits,
// has an accumulator of its own for the 64 terms of one stage (four
// accumulations): a sum of few such terms is exact, one of 64 loses little, and
// the stages' sums are added in registers with rounding. The five low products,
// smallest first, gather in a second accumulator over a layer of a tile
// (chain_kernel) or kLow stages (dw_kernel); what truncation takes of them is
// 2^-8 of that. With all six in one accumulator per stage every product was cut
// off instead of rounded (a single one off by 5e-8 RMS, mean -4.3e-8) and a
// layer's dZ came out 4e-8 too small. The gradient's error of its norm against
// 64-bit arithmetic (from the chains of FMAs before): 1 row 1.0e-7 (2.5e-7),
// 1,000 rows 1.3e-7 (4.4e-7), 65,536 3.1e-7 (1.3e-6), and for every layer no
// larger; a single product's 2.6e-8 RMS (2.5e-8; x1 y2 and x2 y1 would make that
// 2.5e-8 too, and the kernels 22 % slower). What is not finite, or above 3.39e38
// (BF16's largest), becomes NaN.
//
// Six BF16 products are still four to five times the rate of the FP32 FMA
// pipe, which bound the kernels before: of a 1,024-ray step's two networks
// (262,144 rows) dW took 6.2 ms, 1.45 here, and the chain 5.5, 1.97 here. A stage
// is 3,072 cycles of MMAs, and ~450 KB through an SM's shared memory and L1 (the
// MMAs' operands 288, the parts' stores, the loads), 3.6k cycles at 128 bytes per
// cycle. dw_kernel converts both operands with eight warps, which takes longer
// than a stage's MMAs (with four of them 7k cycles per stage, and 12.7k with the
// MMAs issued by one of them). In
// chain_kernel the sums' warps also write dZ, and a CTA moves ~0.6 MB per layer
// and tile through L2 (half the stores, of 16 bytes, took as long, tensor stores
// through shared memory longer).
//
// CTAs run as cluster pairs (tcgen05.mma.cta_group::2, M = 256): each CTA
// converts its half of either operand's columns, the even CTA issues. Both operands
// are MN-major (the reduction runs along the rows) in the 128-byte swizzled
// layout (gemm_tc.cu): 64-column atoms of 64 rows x 128 bytes.
//
// Warp roles (16 warps): 0-7 add each stage's accumulator to the item's sums,
// 128 registers per thread, and at the item's end add those to the gradient;
// 8-15 convert, with rows fetched into L2 ahead of them. Thread 0 of the even
// CTA issues the MMAs (a 17th warp for that would make the block's registers
// those of 20). The warp groups trade registers (setmaxnreg): 168 for the sums,
// 88 for the conversion.
//
// Every mbarrier wait is bounded (tc::wait_bar): on a timeout every role
// stops, the issuer drains its MMAs, TMEM is freed and the CTA makes the whole
// gradient NaN (what others add to it stays NaN) and reports to the caller's
// error word, if there is one.
#include <stdint.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "mlp_internal.cuh"
#include "pair_tc.cuh"
#include "tcgen05.cuh"

namespace nerfgb {
namespace split {

using namespace tc;

constexpr int kRows = 64;  // rows (K) per stage
constexpr int kLow = 8;    // stages per window of low sums (dw_kernel)
constexpr int kAhead = 4;  // stages fetched into L2 ahead of the one converted
constexpr int kSumWarps = 8, kConvWarps = 8, kThreads = 32 * (kSumWarps + kConvWarps);
// Registers of the two kinds of warp group (the block is launched with 128 a thread).
constexpr int kSumRegs = 168, kConvRegs = 88;
static_assert(kSumRegs * kSumWarps + kConvRegs * kConvWarps <= 128 * (kSumWarps + kConvWarps), "the launch's registers");
constexpr uint32_t kAtomBytes = 64 * 128;        // 64 columns x 64 rows
constexpr uint32_t kPart = 2 * kAtomBytes;       // one BF16 part of 128 columns
constexpr uint32_t kOperand = 3 * kPart;
constexpr uint32_t kStage = 2 * kOperand;        // A, B
constexpr uint32_t kBar0 = 2 * kStage;
constexpr uint32_t kBarFull = kBar0;             // [2] operands of the stage written (both CTAs)
constexpr uint32_t kBarDone = kBar0 + 16;        // [2] its MMAs are complete: stage free, accumulators full
constexpr uint32_t kBarRead = kBar0 + 32;        // they have been read (by both CTAs), once per stage
constexpr uint32_t kBarB = kBar0 + 48;           // [2] chain: its weights have arrived (both CTAs')
constexpr uint32_t kBarZ = kBar0 + 64;           // [2] chain: a tile's dZ of the layer is written
constexpr uint32_t kBarMask = kBar0 + 80;        // [2] chain: a tile's mask of the layer is written
constexpr uint32_t kBarDrain = kBar0 + 96;
constexpr uint32_t kTmemSlot = kBar0 + 104;
constexpr uint32_t kAbort = kBar0 + 112;         // int, then the wait limit (u64) at +8
constexpr uint32_t kErr = kBar0 + 128;           // int
constexpr uint32_t kMask = kBar0 + 144;          // [2][256 threads] chain: mask bits, 16 bytes each
constexpr uint32_t kShare = kMask;               // [12] dw: Share of a job
constexpr uint32_t kSmem = kMask + 2 * 4096;
static_assert(kSmem <= 227 * 1024, "two stages");

// One product. Plain: A = the tape's columns col .. col + 255 (the layer's
// input), B = the dZ of `slot` (N columns). Flipped (inputs of fewer than 64
// columns, K): A = the dZ of `slot` (M columns), B = the tape's columns col ..
// col + 127, of which the first K count; the result is transposed.
struct Job {
  int col, slot, K, N, flat, k_dst0;
  bool flip, bias;
  __host__ __device__ constexpr int n_mma() const { return flip ? 128 : N; }
  // a stage's cost in units of a quarter of 256 columns' (the conversion bounds the narrow ones)
  __host__ __device__ constexpr int cost() const { return n_mma() == 256 ? 4 : 3; }
};
constexpr int kJobs = 12;
__host__ __device__ constexpr Job job_of(int j) {
  return j == 0   ? Job{acts_offset(8), 9, 256, 128, 10, 0, false, true}
         : j == 1 ? Job{kActsEncDir, 9, 27, 128, 10, 256, true, false}
         : j == 2 ? Job{acts_offset(7), 8, 256, 256, 9, 0, false, true}
         : j == 3 ? Job{kActsEncXyz, 5, 63, 256, 5, 256, true, false}
         : j == 4 ? Job{kActsEncXyz, 0, 63, 256, 0, 0, true, true}
                  : Job{acts_offset(j - 5), j - 4, 256, 256, j - 4, 0, false, true};  // dense_1 .. dense_7
}
static_assert(kActsEncDir + 128 <= kActsLd && kActsLd % 4 == 0, "flipped inputs stay inside the row");
constexpr int cost_sum() {
  int c = 0;
  for (int j = 0; j < kJobs; ++j) c += job_of(j).cost();
  return c;
}

// What the sums' warps need of a job, from shared memory when they do.
struct __align__(16) Share {
  int begin, end;         // the pair's stages
  uint32_t idesc;
  int to;                 // D's first element in the gradient
  int rows, cols, rs, cs;  // of D: those that count, their strides in the gradient
  int part;               // columns per half of the sums' warps
};

// A pair's stages of job j (every job has `stages`): all jobs' stages in order,
// each at the sum of the costs before it, are dealt evenly by cost.
__device__ __forceinline__ void stages_of(int j, int stages, int pair, int pairs, int &b, int &e) {
  long long at = 0;
  for (int i = 0; i < j; ++i) at += (long long)job_of(i).cost() * stages;
  const long long all = (long long)cost_sum() * stages, w = job_of(j).cost();
  const long long lo = pair * all / pairs - at, hi = (pair + 1) * all / pairs - at;
  b = lo <= 0 ? 0 : (int)((lo + w - 1) / w < stages ? (lo + w - 1) / w : stages);
  e = hi <= 0 ? 0 : (int)((hi + w - 1) / w < stages ? (hi + w - 1) / w : stages);
}

__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(kAtomBytes >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

// Barriers, TMEM (all 512 columns of both CTAs; its address) and the pair's start.
__device__ __forceinline__ uint32_t begin(uint8_t *smem, uint32_t sbase, volatile int *abort_flag, int *err,
                                          bool aligned, unsigned long long wait_ns) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(sbase + kBarFull + 8 * s, 2 * kConvWarps);
      mbar_init(sbase + kBarDone + 8 * s, 1);
      mbar_init(sbase + kBarB + 8 * s, 1);
      mbar_init(sbase + kBarZ + 8 * s, kSumWarps);
      mbar_init(sbase + kBarMask + 8 * s, kConvWarps);
    }
    mbar_init(sbase + kBarRead, 2 * kSumWarps);
    mbar_init(sbase + kBarDrain, 1);
    *abort_flag = aligned ? 0 : 1;
    *err = 0;
    set_wait_limit(abort_flag, wait_ns != 0 ? wait_ns : kWaitNs);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kTmemSlot),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  return *reinterpret_cast<volatile uint32_t *>(smem + kTmemSlot);
}

// MMAs of a stage, of K-steps `step` descriptor units apart: of the six products
// FROM .. TO - 1, the five low ones first, smallest first, into the second
// accumulator, which `first` starts again, the high one last, into the first.
template <int FROM, int TO>
__device__ __forceinline__ void issue_products(uint32_t tmem, uint64_t a, uint64_t b, uint32_t step, uint32_t idesc,
                                               bool first) {
  constexpr int px[6] = {0, 2, 1, 0, 1, 0}, py[6] = {2, 0, 1, 1, 0, 0};
  asm volatile("" : "+l"(a), "+l"(b));  // (the descriptors made here, not kept in registers from stage to stage)
#pragma unroll
  for (int i = FROM; i < TO; ++i)
#pragma unroll
    for (int s = 0; s < kRows / 16; ++s)
      tc_mma_pair(tmem + (i < 5 ? 256u : 0u), a + px[i] * (kPart >> 4) + s * step, b + py[i] * (kPart >> 4) + s * step,
                  idesc, (i == 5 && s == 0) || (first && i + s == 0) ? 0u : 1u);
}

// A stage is issued in two parts: kEarly of its low products as soon as its
// operands are there, under the reading of the accumulators of the stage before
// (unless that reads the low sums too), then the rest. (65,536 rows' backward:
// 1,055 us without, 955 with 2 in chain_kernel, 936 with 4, 890 in both kernels;
// with all five low products the issuing warp waits for the tensor core's queue
// before it reads: 1,028.)
constexpr int kEarly = 4;

// A warp's part (cols of 128) of an accumulator added to its sums: eight
// fragments of 16 rows x 32 columns, those from column `cols` on left out.
__device__ __forceinline__ void add_accumulator(uint32_t taddr, int cols, float (&sum)[4][2][16]) {
#pragma unroll
  for (int f = 0; f < 8; ++f) {
    if (32 * (f / 2) < cols) {
      uint32_t raw[16];
      tmem_ld_frag32(taddr + ((uint32_t)(16 * (f % 2)) << 16) + 32 * (f / 2), raw);
      tmem_wait16(raw);
      float *s = sum[f / 2][f % 2];
#pragma unroll
      for (int i = 0; i < 16; i += 2)
        add_f32x2(s[i], s[i + 1], s[i], s[i + 1], __uint_as_float(raw[i]), __uint_as_float(raw[i + 1]));
    }
  }
}
// By a sums' warp: stage q's high sums, at the end of a window also its low ones,
// added; `begin` runs before they are read. False after a timeout.
template <typename F>
__device__ __forceinline__ bool add_stage(uint32_t sbase, uint32_t taddr, uint32_t q, bool low, int cols, int lane,
                                          float (&sum)[4][2][16], volatile int *abort_flag, int *err, F begin) {
  if (!__all_sync(0xffffffffu, wait_bar(sbase + kBarDone + 8 * (q & 1u), (q >> 1) & 1u, abort_flag, err))) return false;
  begin();
  __syncwarp();
  tc_fence_after();
#pragma unroll 1
  for (uint32_t at = 0; at <= (low ? 256u : 0u); at += 256u) add_accumulator(taddr + at, cols, sum);
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive_remote(peer_addr(sbase + kBarRead, 0));
  return true;
}

// Both CTAs must hold the same TMEM columns (the collective allocation gives them).
__device__ __forceinline__ void check_tmem(uint32_t sbase, uint32_t tmem, volatile int *abort_flag) {
  uint32_t peer_tmem;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_tmem) : "r"(peer_addr(sbase + kTmemSlot, 1)) : "memory");
  if (peer_tmem != tmem) *abort_flag = 1;
}

// By the issuer: every MMA is complete (in both CTAs).
__device__ __forceinline__ void drain(uint32_t sbase) {
  tc_commit_pair(sbase + kBarDrain);
  const uint64_t t0 = globaltimer();
  while (!mbar_try(sbase + kBarDrain, 0) && globaltimer() - t0 < 100000000ull) {
  }
}

// The pair's end. After a timeout the gradient is not a number. `ran`: the issuer drains.
__device__ __forceinline__ void finish(uint32_t sbase, uint32_t tmem, volatile int *abort_flag, const int *err,
                                       float *grads, int *err_word, bool ran) {
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (long long e = threadIdx.x; e < kParamCount; e += kThreads) grads[e] = __int_as_float(0x7fffffff);
    if (threadIdx.x == 0 && err_word) atomicExch(err_word, *err != 0 ? *err : NERFGB_E_UNSUPPORTED);
  }
  if (cluster_rank() == 1 && threadIdx.x == 0 && ran) {
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
  if (threadIdx.x < 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// The BF16 parts of two values, packed: what the rounding leaves of a 24-bit
// value has at most 16 bits, of those at most 8, each exactly subtracted.
__device__ __forceinline__ uint32_t next_part(float &x, float &y) {
  const uint32_t p = pack_bf16(x, y);
  x -= __uint_as_float(p << 16);
  y -= __uint_as_float(p & 0xffff0000u);
  return p;
}

__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Eight values of a row to the three parts' 16-byte chunks at dst.
__device__ __forceinline__ void split_store(const float4 &u, const float4 &v, uint32_t dst) {
  float x[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    uint32_t p[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = next_part(x[2 * j], x[2 * j + 1]);
    st_shared_v4(dst + i * kPart, p[0], p[1], p[2], p[3]);
  }
}

__global__ void __launch_bounds__(kThreads, 1)
    dw_kernel(const float *__restrict__ acts, const float *__restrict__ dz, const float *__restrict__ heads,
              int head_blocks, long long n, float *grads, int *err_word, WaitTest wt) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_rank();
  const int pair = (int)cluster_id(), pairs = (int)cluster_count();
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kAbort);
  int *err = reinterpret_cast<int *>(smem + kErr);
  // (the swizzled stages need 1024-byte alignment: without it nothing runs)
  const bool aligned = (sbase & 1023u) == 0;
  const int stages = aligned ? (int)((n + kRows - 1) / kRows) : 0;
  if (threadIdx.x < kJobs) {
    const Job job = job_of(threadIdx.x);
    Share sh;
    stages_of(threadIdx.x, stages, pair, pairs, sh.begin, sh.end);
    sh.idesc = idesc_bf16(256, 0) | (1u << 15) | (1u << 16) | ((uint32_t)(job.n_mma() >> 3) << 17);
    sh.to = (int)flat_offset(job.flat) + job.k_dst0 * job.N;
    // D's rows are the layer's inputs (flipped: outputs), its columns the outputs (inputs)
    sh.rows = job.flip ? job.N : job.K;
    sh.cols = job.flip ? job.K : job.N;
    sh.rs = job.flip ? 1 : job.N;
    sh.cs = job.flip ? job.N : 1;
    sh.part = (job.flip ? 64 : job.N) / 2;
    reinterpret_cast<Share *>(smem + kShare)[threadIdx.x] = sh;
  }

  const uint32_t tmem = begin(smem, sbase, abort_flag, err, aligned, wt.wait_ns);

  if (warp >= kSumWarps) {
    // ---------------- conversion ----------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kConvRegs));
    // A lane takes 8 columns (chunk c of an atom) of the rows r + 16u: warps
    // 0-3 the first atom's, 4-7 the second's.
    const int w = warp - kSumWarps, c = lane & 7, r = (w & 3) * 4 + (lane >> 3);
    const int col = (int)crank * 128 + (w >> 2) * 64 + 8 * c;  // within 256 columns
    const uint32_t dst =
        sbase + (uint32_t)(w >> 2) * kAtomBytes + (uint32_t)r * 128u + (uint32_t)((c ^ (r & 7)) << 4);
    bool ok = true;
    uint32_t q = 0;  // stages so far
    float4 v[4][2];  // A's four units, each replaced by B's once stored, B's by the next stage's A
    // The stage's values of operand A and B: this lane's columns start at pa
    // and pb (nullptr: not needed), `rows` rows from there.
    const float *pa = nullptr, *pb = nullptr;
    int rows = 0;
    auto load = [&](const float *p, int ld, int u) {
      v[u][0] = v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p && r + 16 * u < rows) {
        const float4 *s = reinterpret_cast<const float4 *>(p + (long long)u * 16 * ld);
        v[u][0] = __ldg(s);
        v[u][1] = __ldg(s + 1);
      }
    };
    auto place = [&](const Job &job, int st) {
      const long long m = (long long)st * kRows + r;
      const long long left = n - (long long)st * kRows;
      rows = left < kRows ? (int)left : kRows;
      const float *z = dz + ((long long)job.slot * n + m) * 256, *t = acts + m * kActsLd + job.col;
      // B has N / 2 columns in each CTA
      const int half = job.n_mma() / 2, bc = (w >> 2) * 64 + 8 * c;
      if (job.flip) {
        pa = col < job.N ? z + col : nullptr;
        pb = crank == 0 && bc < 64 ? t + bc : nullptr;
      } else {
        pa = t + col;
        pb = bc < half ? z + (int)crank * half + bc : nullptr;
      }
    };
    // A stage's rows into L2: a lane fetches half of this CTA's columns of one
    // row of either operand (lines of 128 bytes; a bulk prefetch per row took
    // its warp 2k cycles a stage).
    auto prefetch = [&](const Job &job, int st) {
      const int i = w * 32 + lane, is_b = i >> 7;
      const bool tape = (is_b != 0) == job.flip;
      const long long m = (long long)st * kRows + ((i >> 1) & 63);
      const int cols = !is_b ? 128 : job.flip ? 64 : job.N / 2;  // of this CTA
      const int first = (int)crank * cols + (i & 1) * (cols / 2);
      if (m >= n || (job.flip && (is_b ? crank == 1 : first >= job.N))) return;
      const float *src = (tape ? acts + m * kActsLd + job.col : dz + ((long long)job.slot * n + m) * 256) + first;
      prefetch_l2(src);
      if (cols == 128) prefetch_l2(src + 32);
    };
#pragma unroll 1
    for (int j = 0; j < kJobs && ok; ++j) {
      const Job job = job_of(j);
      int sb, se;
      stages_of(j, stages, pair, pairs, sb, se);
      if (sb >= se) continue;
#pragma unroll 1
      for (int st = sb + 1; st < se && st < sb + kAhead; ++st) prefetch(job, st);
      const int lda = job.flip ? 256 : kActsLd, ldb = job.flip ? kActsLd : 256;
      place(job, sb);
#pragma unroll
      for (int u = 0; u < 4; ++u) load(pa, lda, u);
      float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int st = sb; st < se; ++st, ++q) {
        const int k = (int)(q & 1);
        if (!__all_sync(0xffffffffu, wait_bar(sbase + kBarDone + 8 * k, (uint32_t)((q >> 1) & 1) ^ 1u, abort_flag, err))) {
          ok = false;
          break;
        }
        const uint32_t at = dst + (uint32_t)k * kStage;
        if (st + kAhead < se) prefetch(job, st + kAhead);
        auto add = [&](int u) {
          const float4 x = v[u][0], y = v[u][1];
          sum[0] += x.x; sum[1] += x.y; sum[2] += x.z; sum[3] += x.w;
          sum[4] += y.x; sum[5] += y.y; sum[6] += y.z; sum[7] += y.w;
        };
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (pa) {
            if (job.bias && job.flip) add(u);
            split_store(v[u][0], v[u][1], at + 2048u * u);
          }
          load(pb, ldb, u);
        }
        const bool use_b = pb != nullptr;
        if (st + 1 < se)
          place(job, st + 1);
        else
          pa = nullptr;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (use_b) {
            if (job.bias && !job.flip) add(u);
            split_store(v[u][0], v[u][1], at + kOperand + 2048u * u);
          }
          load(pa, lda, u);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && !(wt.withhold != 0 && q == 1 && w == 0))
          mbar_arrive_remote(peer_addr(sbase + kBarFull + 8 * k, 0));
      }
      if (job.bias) {
        // the lanes of a chunk, then the warps (and pairs) by atomics
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 8);
          sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 16);
        }
        const int half = job.n_mma() / 2, bc = (w >> 2) * 64 + 8 * c;
        if (lane < 8 && (job.flip || bc < half)) {
          float *db = grads + flat_offset(job.flat) + (long long)flat_in(job.flat) * job.N +
                      (job.flip ? col : (int)crank * half + bc);
#pragma unroll
          for (int i = 0; i < 8; ++i) atomicAdd(db + i, sum[i]);
        }
      }
    }
    // the heads' sums, a warp per element, under the last stages' MMAs
#pragma unroll 1
    for (int e = (int)blockIdx.x * kConvWarps + w; e < kHeadSumsFp32; e += (int)gridDim.x * kConvWarps)
      add_head_sums(heads, head_blocks, e, lane, grads);
  } else {
    // ---------------- the stages' sums (and the issuer) ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSumRegs));
    // Warp w: TMEM lane quadrant w % 4 (rows of D), half w / 4 of the columns
    // that count, as 16 x 32 fragments (tcgen05.cuh).
    const int qd = warp & 3, h = warp >> 2;
    const uint32_t tl = tmem + ((uint32_t)(32 * qd) << 16);
    const bool issuer = crank == 0 && threadIdx.x == 0;
    if (issuer) check_tmem(sbase, tmem, abort_flag);
    const volatile Share *share = reinterpret_cast<const volatile Share *>(smem + kShare);
    auto early = [&](uint32_t q, uint32_t idesc, bool first) {
      const uint32_t sa = sbase + (q & 1u) * kStage;
      tc_fence_after();
      issue_products<0, kEarly>(tmem, desc_mn_sw128(sa), desc_mn_sw128(sa + kOperand), 2048 >> 4, idesc, first);
    };
    auto issue = [&](uint32_t q, uint32_t idesc, bool first, bool begun) {
      const uint32_t k = q & 1u, sa = sbase + k * kStage;
      if ((!begun && !wait_bar(sbase + kBarFull + 8 * k, (q >> 1) & 1u, abort_flag, err)) ||
          !wait_bar(sbase + kBarRead, k ^ 1u, abort_flag, err))
        return;
      if (!begun) early(q, idesc, first);
      tc_fence_after();
      issue_products<kEarly, 6>(tmem, desc_mn_sw128(sa), desc_mn_sw128(sa + kOperand), 2048 >> 4, idesc, false);
      tc_commit_pair(sbase + kBarDone + 8 * k);
    };
    bool ok = true, begun = false;  // (of the next stage the early part is issued)
    uint32_t q = 0;  // stages so far
#pragma unroll 1
    for (int j = 0; j < kJobs && ok; ++j) {
      int left = share[j].end - share[j].begin;
      if (left <= 0) continue;
      const int cols = share[j].part, c0 = h * cols;
      float sum[4][2][16];
#pragma unroll
      for (int f = 0; f < 8; ++f)
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[f / 2][f % 2][i] = 0.0f;
      int window = 0;  // stages in the window of low sums
#pragma unroll 1
      for (; left > 0 && ok; --left, ++q) {
        if (issuer) issue(q, share[j].idesc, window == 0, begun);
        __syncwarp();
        const bool end = left == 1 || ++window == kLow;
        begun = false;
        ok = add_stage(sbase, tl + c0, q, end, cols, lane, sum, abort_flag, err, [&] {
          const uint32_t k = (q + 1) & 1u;
          if (!issuer || end || !mbar_test(sbase + kBarFull + 8 * k, ((q + 1) >> 1) & 1u)) return;
          early(q + 1, share[j].idesc, false);
          begun = true;
        });
        if (end) window = 0;
      }
      if (!ok) break;
      // (addresses from what is read here: kept over the stages they would spill)
      const volatile Share &sh = share[j];
      int l = lane;
      asm volatile("" : "+r"(l));
      const int row0 = (int)crank * 128 + 32 * qd + l / 4, cl0 = c0 + 2 * (l % 4);
      const int rows = sh.rows, cls = sh.cols, rs = sh.rs, cs = sh.cs;
      float *dW = grads + sh.to + row0 * rs + cl0 * cs;
#pragma unroll
      for (int f = 0; f < 8; ++f) {
        if (32 * (f / 2) >= cols) continue;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int row = 16 * (f % 2) + 8 * ((i >> 1) & 1), cl = 32 * (f / 2) + 8 * (i / 4) + (i & 1);
          if (row0 + row < rows && cl0 + cl < cls) atomicAdd(dW + row * rs + cl * cs, sum[f / 2][f % 2][i]);
        }
      }
    }
    if (issuer && stages > 0) drain(sbase);
  }

  finish(sbase, tmem, abort_flag, err, grads, err_word, stages > 0);
}

// ---------------------------------------------------------------------------
// Chain
// ---------------------------------------------------------------------------
// Weights of GEMM layer g as the B operand of dX: 64 n at a time, for either
// CTA (128 k) the three parts, K-major in the 128-byte swizzled layout: row k
// at k * 128 bytes, its 16-byte chunk c at (c ^ (k & 7)) * 16. Layers from
// dense_9 down.
__host__ __device__ constexpr int first_chunk(int g) { return g == 9 ? 0 : 2 + (8 - g) * 4; }
constexpr long long kPackBytes = (long long)first_chunk(0) * 2 * kOperand;

__global__ void pack_kernel(const float *__restrict__ W, uint8_t *__restrict__ out) {
  const int g = 9 - blockIdx.y, N = gemm_n(g), e = blockIdx.x * blockDim.x + threadIdx.x;  // k * N + n
  if (e >= 256 * N) return;
  const int k = e / N, n = e % N;
  float x = W[gemm_w_offset(g) + e], none = 0.0f;
  uint8_t *dst = out + ((long long)(first_chunk(g) + n / 64) * 2 + k / 128) * kOperand + (k % 128) * 128 +
                 ((((n % 64) / 8) ^ (k & 7)) << 4) + (n % 8) * 2;
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint16_t *>(dst + i * kPart) = (uint16_t)next_part(x, none);
}

// dz [10][n][256]: dz[9] (128 columns) in, dz[8] .. dz[0] out. A pair takes
// tiles of 256 rows (128 per CTA) through all layers, two tiles in turn, so
// that one's sums and dZ are finished under the other's MMAs (with a tile
// alone a layer's first stage waits for the layer before); a tile's dZ goes
// through L2 to the conversion of the next layer (the three parts of a tile
// would fill shared memory). K runs in stages of 64 n: the dZ converted as in
// dw_kernel, K-major, the weights split once (pack_kernel) and copied by TMA.
// The ReLU masks are read as bits by the conversion's warps, a layer after
// their rows were fetched into L2: read by the sums' warps at the end of a
// layer, the loads' latencies were four fifths of the time (1,094 us for 65,536
// rows; in their waits for the stages 550; 490 - 526 here).
__global__ void __launch_bounds__(kThreads, 1)
    chain_kernel(const float *__restrict__ sigma_w, const float *__restrict__ acts, const float *__restrict__ dsp,
                 long long n, float *dz, float *__restrict__ grads, int *err_word, WaitTest wt,
                 const __grid_constant__ CUtensorMap weights) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_rank();
  const int pair = (int)cluster_id(), pairs = (int)cluster_count();
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kAbort);
  int *err = reinterpret_cast<int *>(smem + kErr);
  // (the swizzled stages need 1024-byte alignment: without it nothing runs)
  const bool aligned = (sbase & 1023u) == 0;
  const int tiles = aligned ? (int)((n + 255) / 256) : 0;
  // the tiles dealt evenly and contiguously
  const int first = (int)((long long)pair * tiles / pairs), count = (int)((long long)(pair + 1) * tiles / pairs) - first;
  const uint32_t tmem = begin(smem, sbase, abort_flag, err, aligned, wt.wait_ns);

  if (warp >= kSumWarps) {
    // ---------------- conversion, weight copies ----------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kConvRegs));
    // A lane takes 8 of a stage's 64 n (chunk c) of the rows r + 32u.
    const int w = warp - kSumWarps, c = lane & 7, r = w * 4 + (lane >> 3);
    const uint32_t dst = sbase + (uint32_t)r * 128u + (uint32_t)((c ^ (r & 7)) << 4);
    bool ok = true;
    uint32_t q = 0;
#pragma unroll 1
    for (int t = 0; t < count && ok; t += 2) {
      const int subs = min(2, count - t);
#pragma unroll 1
      for (int g = 9; g >= 1 && ok; --g) {
        const int chunks = gemm_n(g) / 64;
#pragma unroll 1
        for (int s = 0; s < subs && ok; ++s) {
          if (g < 9 && !__all_sync(0xffffffffu, wait_bar(sbase + kBarZ + 8 * s, (uint32_t)(g & 1), abort_flag, err))) {
            ok = false;
            break;
          }
          const long long tile0 = (long long)(first + t + s) * 256 + crank * 128, row = tile0 + r;
          // the next layer's mask into L2, half a row per lane
          if (g > 1 && tile0 + w * 16 + lane / 2 < n) {
            const float *next = acts + (tile0 + w * 16 + lane / 2) * kActsLd + acts_offset(g - 2) + 128 * (lane & 1);
#pragma unroll
            for (int i = 0; i < 4; ++i) prefetch_l2(next + 32 * i);
          }
          // This layer's mask for lane `lane` of sum warp w: its columns of the
          // rows mrow + 8 rr (a bit each), one rr per stage.
          const long long mrow = tile0 + 32 * (w & 3) + lane / 4;
          const float *mask = acts + mrow * kActsLd + acts_offset(g - 1) + 128 * (w >> 2) + 2 * (lane % 4);
          uint32_t bits[4] = {0u, 0u, 0u, 0u};
          float2 m[8];
          auto load_mask = [&](int rr, int half) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              m[i] = make_float2(0.f, 0.f);
              if (g != 9 && mrow + 8 * rr < n)
                m[i] = __ldcs(reinterpret_cast<const float2 *>(mask + (long long)8 * rr * kActsLd + 8 * (8 * half + i)));
            }
          };
          auto mask_bits = [&](int half) {
            uint32_t v = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i)
              v |= (m[i].x > 0.0f ? 1u : 0u) << (2 * (8 * half + i)) | (m[i].y > 0.0f ? 2u : 0u) << (2 * (8 * half + i));
            return v;
          };
          const float *src = dz + ((long long)g * n + row) * 256 + 8 * c;
          float4 v[4][2];
          auto load = [&](int ch, int u) {
            v[u][0] = v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ch < chunks && row + 32 * u < n) {
              // (written in this launch: not through the read-only path)
              const float4 *p = reinterpret_cast<const float4 *>(src + 32 * 256 * u + 64 * ch);
              v[u][0] = __ldcg(p);
              v[u][1] = __ldcg(p + 1);
            }
          };
#pragma unroll
          for (int u = 0; u < 4; ++u) load(0, u);
#pragma unroll 1
          for (int ch = 0; ch < chunks; ++ch, ++q) {
            const uint32_t k = q & 1u;
            load_mask(ch, 0);
            if (!__all_sync(0xffffffffu, wait_bar(sbase + kBarDone + 8 * k, ((q >> 1) & 1u) ^ 1u, abort_flag, err))) {
              ok = false;
              break;
            }
            if (w == 0 && lane == 0 && !(wt.withhold != 0 && q == 1)) {
              const uint32_t bar = sbase + kBarB + 8 * k, to = sbase + k * kStage + kOperand;
              if (crank == 0) mbar_expect_tx(bar, 2 * kOperand);
              const int y = ((first_chunk(g) + ch) * 2 + (int)crank) * (int)(kOperand / 256);
#pragma unroll
              for (int i = 0; i < 3; ++i)
                tma_2d_pair(to + i * kPart, &weights, 0, y + i * (int)(kPart / 256), crank == 0 ? bar : peer_addr(bar, 0));
            }
            __syncwarp();
            uint32_t mb = mask_bits(0);
            load_mask(ch, 1);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              split_store(v[u][0], v[u][1], dst + k * kStage + 4096u * u);
              load(ch + 1, u);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(peer_addr(sbase + kBarFull + 8 * k, 0));
            mb |= mask_bits(1);
#pragma unroll
            for (int i = 0; i < 4; ++i) bits[i] = ch == i ? mb : bits[i];
          }
          if (g != 9) {
            st_shared_v4(sbase + kMask + s * 4096 + (w * 32 + lane) * 16, bits[0], bits[1], bits[2], bits[3]);
            __syncwarp();
            if (lane == 0) mbar_arrive(sbase + kBarMask + 8 * s);
          }
        }
      }
    }
  } else {
    // ---------------- the stages' sums, dZ (and the issuer) ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSumRegs));
    const int qd = warp & 3, h = warp >> 2;
    const uint32_t tl = tmem + ((uint32_t)(32 * qd) << 16) + 128u * h;
    const bool issuer = crank == 0 && threadIdx.x == 0;
    const uint32_t total = (uint32_t)count * first_chunk(0);
    if (issuer) check_tmem(sbase, tmem, abort_flag);
    auto desc = [&](uint32_t addr) { return (uint64_t)kDescHiA << 32 | ((addr & 0x3FFFFu) >> 4) | (1u << 16); };
    auto early = [&](uint32_t q, bool first) {
      const uint32_t sa = sbase + (q & 1u) * kStage;
      tc_fence_after();
      issue_products<0, kEarly>(tmem, desc(sa), desc(sa + kOperand), 32 >> 4, idesc_bf16(256, 256), first);
    };
    auto issue = [&](uint32_t q, bool first, bool begun) {
      const uint32_t k = q & 1u, ph = (q >> 1) & 1u, sa = sbase + k * kStage;
      if ((!begun && (!wait_bar(sbase + kBarFull + 8 * k, ph, abort_flag, err) ||
                      !wait_bar(sbase + kBarB + 8 * k, ph, abort_flag, err))) ||
          !wait_bar(sbase + kBarRead, k ^ 1u, abort_flag, err))
        return;
      if (!begun) early(q, first);
      tc_fence_after();
      issue_products<kEarly, 6>(tmem, desc(sa), desc(sa + kOperand), 32 >> 4, idesc_bf16(256, 256), false);
      tc_commit_pair(sbase + kBarDone + 8 * k);
    };
    bool ok = true;
    uint32_t q = 0, iq = 0;  // stages so far, stages issued
    bool begun = false;      // of stage iq the early part is
#pragma unroll 1
    for (int t = 0; t < count && ok; t += 2) {
      const int subs = min(2, count - t);
#pragma unroll 1
      for (int g = 9; g >= 1 && ok; --g) {
        const int chunks = gemm_n(g) / 64;
#pragma unroll 1
        for (int s = 0; s < subs; ++s) {
          const long long row0 = (long long)(first + t + s) * 256 + crank * 128 + 32 * qd + lane / 4;
          const int col0 = 128 * h + 2 * (lane % 4);
          float sum[4][2][16];
#pragma unroll
          for (int f = 0; f < 8; ++f)
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[f / 2][f % 2][i] = 0.0f;
#pragma unroll 1
          for (int ch = 0; ch < chunks; ++ch, ++q) {
            const bool last = ch + 1 == chunks;
            if (issuer) {
              if (iq == q) issue(iq++, ch == 0, begun);
              begun = false;
            }
            // (tried as the stage before is issued and, if its operands are not there yet, as that is complete)
            auto try_early = [&]() {
              const uint32_t k = iq & 1u, ph = (iq >> 1) & 1u;
              if (!issuer || last || begun || !mbar_test(sbase + kBarFull + 8 * k, ph) ||
                  !mbar_test(sbase + kBarB + 8 * k, ph))
                return;
              early(iq, false);
              begun = true;
            };
            try_early();
            __syncwarp();
            if (!(ok = add_stage(sbase, tl, q, last, 128, lane, sum, abort_flag, err, try_early))) break;
            // the next layer's (the other tile's) first stage under the writing of
            // dZ, unless it waits for that (a tile alone)
            if (issuer && last && subs == 2 && iq < total) issue(iq++, true, false);
            __syncwarp();
          }
          if (!ok) break;
          // dense_9's input, the bottleneck, is linear: no mask
          uint32_t bits[4] = {~0u, ~0u, ~0u, ~0u};
          if (g != 9) {
            if (!__all_sync(0xffffffffu, wait_bar(sbase + kBarMask + 8 * s, (uint32_t)(g & 1), abort_flag, err))) {
              ok = false;
              break;
            }
            ld_shared_v4(sbase + kMask + s * 4096 + threadIdx.x * 16, bits[0], bits[1], bits[2], bits[3]);
          }
          float *out = dz + ((long long)(g - 1) * n + row0) * 256 + col0;
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) {  // rows row0 + 8 rr
            if (row0 + 8 * rr >= n) continue;
            const float ds = g == 8 ? dsp[row0 + 8 * rr] : 0.0f;
#pragma unroll
            for (int j = 0; j < 16; ++j) {  // columns col0 + 8 j, + 1
              const float *a = sum[j / 4][rr / 2] + 4 * (j % 4) + 2 * (rr % 2);
              float2 z = make_float2(a[0], a[1]);
              if (g == 8) {  // dense_8's input h7 also feeds the sigma head
                const float2 ws = *reinterpret_cast<const float2 *>(sigma_w + col0 + 8 * j);
                z.x = fmaf(ds, ws.x, z.x);
                z.y = fmaf(ds, ws.y, z.y);
              }
              z.x = bits[rr] >> (2 * j) & 1u ? z.x : 0.0f;
              z.y = bits[rr] >> (2 * j) & 2u ? z.y : 0.0f;
              *reinterpret_cast<float2 *>(out + 8 * rr * 256 + 8 * j) = z;
            }
          }
          __syncwarp();
          if (g > 1 && lane == 0) mbar_arrive(sbase + kBarZ + 8 * s);
        }
      }
    }
    if (issuer && tiles > 0) drain(sbase);
  }

  finish(sbase, tmem, abort_flag, err, grads, err_word, tiles > 0);
}

}  // namespace split

// Launches a pair kernel on at most `work` pairs, as many as are co-resident
// (asked once per device, as mlp_tc.cu).
namespace split {
struct Pairs {
  std::mutex mu;
  std::unordered_map<int, int> of_device;
};
template <typename... P, typename... A>
static int launch_pairs(void (*kernel)(P...), Pairs &pairs, long long work, cudaStream_t st, const A &...args) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess)
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
  int dev = -1, most;
  if (cudaGetDevice(&dev) != cudaSuccess) return NERFGB_E_DEVICE;
  {
    std::lock_guard<std::mutex> lock(pairs.mu);
    auto hit = pairs.of_device.find(dev);
    if (hit == pairs.of_device.end()) {
      cfg.gridDim = dim3((unsigned)(sms / 2 * 2));
      int m = 0;
      if (cudaOccupancyMaxActiveClusters(&m, kernel, &cfg) != cudaSuccess) return NERFGB_E_CUDA;
      hit = pairs.of_device.emplace(dev, m).first;
    }
    most = hit->second;
  }
  if (most < 1) return NERFGB_E_UNSUPPORTED;
  cfg.gridDim = dim3((unsigned)(2 * (work < most ? work : most)));
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  const int rc = launch_status();  // (clears a failed launch's error)
  return e == cudaSuccess ? rc : NERFGB_E_CUDA;
}
}  // namespace split

int launch_fp32_dw(const float *acts, const float *dz, const float *heads, int head_blocks, long long n, float *grads,
                   int *err_word, cudaStream_t st, const WaitTest &wt) {
  using namespace split;
  if (n == 0) return NERFGB_OK;
  static Pairs pairs;
  return launch_pairs(dw_kernel, pairs, kJobs * ((n + kRows - 1) / kRows), st, acts, dz, heads, head_blocks, n, grads,
                      err_word, wt);
}

long long fp32_chain_pack_bytes() { return split::kPackBytes; }

int launch_fp32_chain_pack(const float *packed, void *wpack, cudaStream_t st) {
  split::pack_kernel<<<dim3(256, 9), 256, 0, st>>>(packed, reinterpret_cast<uint8_t *>(wpack));
  return launch_status();
}

int launch_fp32_chain(const void *wpack, const float *sigma_w, const float *acts, const float *dsp, long long n,
                      float *dz, float *grads, int *err_word, cudaStream_t st, const WaitTest &wt) {
  using namespace split;
  if (n == 0) return NERFGB_OK;
  static Pairs pairs;
  CUtensorMap weights;
  const unsigned long long dims[2] = {128, (unsigned long long)(kPackBytes / 256)}, strides[1] = {256};
  const unsigned box[2] = {128, kPart / 256};
  const int rc = encode_tensor_map_u16(&weights, wpack, 2, dims, strides, box);
  if (rc != NERFGB_OK) return rc;
  return launch_pairs(chain_kernel, pairs, (n + 255) / 256, st, sigma_w, acts, dsp, n, dz, grads, err_word, wt,
                      weights);
}

}  // namespace nerfgb
