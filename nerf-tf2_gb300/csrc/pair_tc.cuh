// MMA issue of the 2-SM pair kernels (mlp_tc.cu, mlp_bwd_tc.cu): A operands in
// 128-byte swizzled atoms (128 rows x 128 bytes of K, 16 KB), B in a ring of
// kPairStage-byte stages filled by the weight producers.
#pragma once
#include "common.cuh"
#include "tcgen05.cuh"

namespace nerfgb {
namespace tc {

constexpr uint32_t kAtom = 16384;  // 128 rows x 128 bytes of K

// tcgen05.mma is issued by one thread, and the tensor pipe runs ahead of it
// by little: every instruction the issuing thread executes between two MMAs
// is latency on the pipe (measured: a 128x256x16 MMA takes 128 cycles; with
// run-time layer shapes, operand selects and 64-bit descriptor assembly per
// MMA the issue loop took ~164 cycles per MMA). So the issue code is shaped
// at compile time per layer: descriptors are two 32-bit words, the high word
// a constant and the low word a base plus immediates (start address >> 4 in
// bits 0-13, LBO >> 4 in bits 16-29). Both precisions take 32 bytes of K per
// MMA (16 BF16 or 32 E4M3), a quarter of a swizzled atom's row.
constexpr uint32_t kDescHiB = (128u >> 4) | (1u << 14);                // no swizzle: SBO = 128
constexpr uint32_t kDescHiA = (1024u >> 4) | (1u << 14) | (2u << 29);  // 128-byte swizzle: SBO = 1024

// Out-of-line slow path of a full-barrier wait: spins until the phase
// completes, the CTA aborts, or the wait limit passes (then raises the abort).
static __device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *err) {
  const uint64_t t0 = globaltimer();
  while (!mbar_try(bar, parity)) {
    if (*abort_flag) return;
    if (globaltimer() - t0 > wait_limit(abort_flag)) {
      atomicExch(err, NERFGB_E_TIMEOUT);
      *abort_flag = 1;
      return;
    }
  }
}

__device__ __forceinline__ void wait_fast(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *err) {
  if (!mbar_try(bar, parity)) wait_slow(bar, parity, abort_flag, err);
}

template <bool F8>
__device__ __forceinline__ void mma_any(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  const uint64_t a = ((uint64_t)kDescHiA << 32) | a_lo, b = ((uint64_t)kDescHiB << 32) | b_lo;
  if (F8)
    tc_mma_pair_f8(d, a, b, idesc, acc);
  else
    tc_mma_pair(d, a, b, idesc, acc);
}

// Ring position of the MMA issuer.
struct RingPos {
  int stage;
  uint32_t phase;
};

// NC stages of ST MMAs (32 bytes of K each) into the accumulators at tmem: A
// from a_lo on (four steps per atom), B from successive ring stages of H rows.
// NST: the ring's stages. FIRST: the run starts the layer (its first MMA overwrites the accumulator).
// WAIT: wait for each stage's weights (sub-tile B's runs follow A's over the
// same stages and skip it). release: free each stage once its MMAs complete.
template <int NST, int NC, int ST, int H, bool F8, bool FIRST, bool WAIT>
__device__ __forceinline__ void issue_run(uint32_t bar_full, uint32_t bar_empty, uint32_t ring_lo, uint32_t a_lo,
                                          uint32_t tmem, uint32_t idesc, bool release, RingPos &rp,
                                          volatile int *abort_flag, int *err) {
#pragma unroll 1
  for (int c = 0; c < NC; ++c) {
    if (WAIT) {
      wait_fast(bar_full + 8 * rp.stage, rp.phase, abort_flag, err);
      tc_fence_after();
    }
    const uint32_t b_lo = ring_lo + (uint32_t)rp.stage * (kPairStage >> 4);
    const uint32_t a = a_lo + (uint32_t)c * (uint32_t)(ST / 4) * (kAtom >> 4);
#pragma unroll
    for (int k = 0; k < ST; ++k)
      mma_any<F8>(tmem, a + (uint32_t)(k / 4) * (kAtom >> 4) + (uint32_t)(k % 4) * 2u, b_lo + (uint32_t)(2 * k * H),
                  idesc, FIRST && k == 0 ? (c > 0 ? 1u : 0u) : 1u);
    if (release) tc_commit_pair(bar_empty + 8 * rp.stage);
    if (++rp.stage == NST) {
      rp.stage = 0;
      rp.phase ^= 1;
    }
  }
}

}  // namespace tc
}  // namespace nerfgb
