// Tensor-core forward of the NeRF MLP (nerf/core/model.py:334-394) on
// sm_103a, BF16 and FP8-e4m3: tcgen05.mma with FP32 accumulators in TMEM,
// operands in shared memory, weights streamed by the tensor-copy (TMA)
// engine. The whole 10-GEMM chain runs on chip: activations never leave
// shared memory and only xyz/dirs (in) and rgb/sigma (out) touch HBM.
//
// CTAs run as cluster pairs. A tile is two sub-tiles (A, B) of 256 rows, 128
// from each CTA; the even CTA issues 2-SM MMAs (tcgen05.mma.cta_group::2,
// M = 256: a sub-tile's rows of both CTAs, B split by N between them), so
// each SM streams only half of every weight chunk. The tensor core runs layer
// g of A, then of B (ping-pong), so that one sub-tile's epilogue overlaps the
// other's MMAs. The rows are dealt to the pairs in 256-row sub-tiles, evenly
// and contiguously; a pair with an odd count runs its last tile with A alone,
// so a small batch (one sub-tile per pair) has half the latency of a whole
// tile and the last wave of a large one is half as coarse.
//
// Warp roles (14 warps; 15 with the tape):
//   warp 0       weight producer: one thread copying weight chunks in ring
//                order (full/empty mbarriers) with 2-SM tensor copies that
//                complete on the even CTA's barrier
//   warp 1       TMEM allocator and, in the even CTA, MMA issuer (one thread;
//                its issue code is generated per kind of layer at compile time)
//   warps 2-9    epilogue of layers 0-8, all on one sub-tile at a time: the
//                accumulator (tcgen05.ld), bias, ReLU, rounding to BF16 (or
//                E4M3) and the next layer's A operand; the sigma head in FP32
//   warps 10-13  beside it, a row per lane: the positional encodings, dense_9
//                and the rgb head in FP32
//   warp 14      (training tape only) one thread storing each written operand
//                region to the tape by a tensor store
//
// What bounds it and why it is laid out so (a 256-wide layer of a sub-tile is
// 2,048 cycles of MMAs in BF16, half that in E4M3; the L1/shared data pipe
// that feeds them also serves the epilogue):
// - The ring's five 16 KB stages hold every layer whole (dense_5's five
//   64-K chunks included), so each weight byte is streamed once per tile and
//   a stage's refill has a whole stage more time. With four stages dense_5
//   and dense_9 were streamed twice and each refill's latency (commit,
//   producer, copy: 1.3-1.9k cycles) was exposed: 13.8k of a BF16 tile's 68.7k
//   cycles were waits for weights.
// - The room for the fifth stage comes from the encodings: one 16 KB region
//   instead of two. dense_0 reads its encoding from the (idle) first 64
//   columns of the sub-tile's activation region; the region E holds A's
//   encoding for dense_5, then (once A's dense_5 MMAs are done) B's, then
//   both sub-tiles' direction encodings for dense_9. The encodings are
//   computed again for each write (by one copy of the code).
// - The epilogue of a plain layer reads the accumulator in the 16x256b
//   fragment layout and stores it with stmatrix: a thread then adds 2 biases
//   per 8 columns instead of 8 (a broadcast LDG.128 costs four wavefronts of
//   the data pipe whatever it fetches), loaded before the accumulator is
//   ready. dense_7 does the same and writes its FP32 ReLU back to TMEM, from
//   where the sigma head reads it a row per lane: the heads' sums run along a
//   row in a fixed order. The head weights sit in shared memory (a broadcast
//   LDS.128 costs two wavefronts).
// - Eight epilogue warps and four side warps with 128 registers, of which a
//   thread spills at most two words: the 28 KB of L1 beside this much shared
//   memory do not hold spills, and a reload is a trip to L2 (sixteen epilogue
//   warps with 96: 648 us, and 1,190 with 200 bytes of spills, against 610).
// - The encodings and dense_9 are the side warps': with the epilogue's eight
//   warps doing them the tensor core waited ~7k cycles per tile for the heads
//   at the tile's end and ~2k more behind the sigma head (BF16 607 us, FP8
//   620, with the tape 930). The rgb head takes a side warp ~2.7k cycles per
//   sub-tile (its broadcast loads alone ~1.3k of the data pipe); shared with
//   the epilogue's warps, which then start dense_0 later, it was 554 and 459.
// - dense_0's operand is written as soon as dense_9 is done, before the rgb
//   head, and its MMAs wait only for the head's reads of the accumulator.
// - E4M3's ReLU runs on the packed words (relu_e4m3x4): 484 -> 452 us.
// - Even deals of 256-row sub-tiles: see above. A tile of one sub-tile has no
//   other one to hide its epilogue under: in BF16 (without the tape, whose
//   stores bound it) a layer's MMAs start on the first half of its K while the
//   epilogue writes the second, from the other accumulator (issue_solo: 1,000
//   rows 31.2 -> 29.3 us).
// Measured against the kernels before (a 4-stage pair kernel in BF16, one CTA
// per tile in FP8): 786,432 rows BF16 783 -> 546 us, with the tape 1,613 ->
// 805, FP8 904 -> 452; 1,000 rows BF16 43 -> 27 us, FP8 41 -> 23.5
// (2 us of either by after_previous, common.cuh). A BF16 tile
// takes ~51k cycles, 37k of them MMAs; the largest waits left are the rgb
// heads at the tile boundary (~5k).
//
// Shared memory: ring [0,80K) | E [80K,96K) | actA, actB | barriers and head
// weights (in the 3 KB left). Operands are K-major in the
// 128-byte swizzled layout: atoms of 128 bytes of K (64 BF16 or 128 E4M3) by
// 128 rows, 16 KB each; row r at r*128, its 16-byte chunk c at (c ^ (r&7))*16,
// so that a region goes to the row-major tape as whole 128-byte rows. Weights:
// no swizzle, 8x16-byte core matrices, (k/KW)*(H*16) + n*16 for the H = N/2
// rows of this CTA (the pack's layout, common.cuh).
//
// Every mbarrier wait is bounded (globaltimer). On a timeout the kernel sets
// *err_word = NERFGB_E_TIMEOUT, raises an abort flag that every role polls,
// drains its own bulk copies and MMAs (bounded), frees TMEM and returns (the
// pair meets at a cluster barrier first, so that neither CTA leaves while
// the other's MMAs or arrivals may still touch it).
#include <cuda.h>  // CUtensorMap (the encoder is reached through the runtime's entry-point query)
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "mlp_internal.cuh"
#include "pair_tc.cuh"
#include "tcgen05.cuh"

namespace nerfgb {
namespace tc {

constexpr int kSubRows = 256;  // rows of a sub-tile: 128 per CTA of the pair
// Warps: producer, issuer, the epilogue's (one per column part and TMEM lane
// quadrant), the side warps (one per quadrant: encodings and the rgb head) and,
// in the kernel that writes the activation tape, one whose first lane stores
// each written operand region to the tape.
constexpr int kParts = 2, kEpiWarps = 4 * kParts;
constexpr int kSideWarp = 2 + kEpiWarps, kTapeWarp = kSideWarp + 4;
__host__ __device__ constexpr int threads_of(bool tape) { return (kTapeWarp + (tape ? 1 : 0)) * 32; }

// Tensor maps of the pack's weights (2-D, 256-byte rows), one per size of a
// CTA's half of a chunk: 16 KB, 8 KB and dense_9's last chunk (4 KB BF16, 2 KB
// E4M3). With the tape: the tape (kActsLd BF16 per row) as 3-D (64 elements,
// rows, 64-element atoms; strides 2 B, the row stride, 128 B; 128-byte
// swizzle), whose boxes of 128 rows have the operand regions' image: tape[0]
// 4 atoms (a 256-wide activation), tape[1] one (enc_xyz), tape[2] two
// (enc_dir and h9's first 96 columns).
struct PairMaps {
  CUtensorMap map[3];
  CUtensorMap tape[3];
};
__host__ __device__ constexpr int pair_map_of(uint32_t bytes) { return bytes == 16384u ? 0 : bytes == 8192u ? 1 : 2; }

template <bool F8>
struct Layout {
  static constexpr uint32_t kE = F8 ? 1 : 2;
  static constexpr int kNst = 5;
  static constexpr uint32_t kEncOff = kNst * kPairStage;
  static constexpr uint32_t kActOff = kEncOff + kAtom;     // + s * kActBytes
  static constexpr uint32_t kActBytes = 128 * 256 * kE;    // per sub-tile
  static constexpr uint32_t kMisc = kActOff + 2 * kActBytes;
  static constexpr uint32_t kBarFull = kMisc;              // [kNst]
  static constexpr uint32_t kBarEmpty = kMisc + 64;        // [kNst]
  static constexpr uint32_t kBarAccf = kMisc + 128;        // [2] accumulator full (layers 0-8)
  static constexpr uint32_t kBarAcc5 = kMisc + 144;        // [2] ... of dense_5, for the side warps
  static constexpr uint32_t kBarAcc9 = kMisc + 160;        // [2] ... of dense_9
  static constexpr uint32_t kBarActr = kMisc + 176;        // [2] operand ready (layers 1-9)
  static constexpr uint32_t kBarAct0 = kMisc + 192;        // [2] dense_0's operand, dense_9's accumulator read
  static constexpr uint32_t kBarEncA = kMisc + 208;        // A's encoding in E
  static constexpr uint32_t kBarEncB = kMisc + 216;        // B's
  static constexpr uint32_t kBarDir = kMisc + 224;         // the direction encodings
  static constexpr uint32_t kBarRead8 = kMisc + 232;       // [2] the second part has read dense_8's accumulator
  static constexpr uint32_t kBarSig = kMisc + 248;         // [2] sigma's sums in TMEM
  static constexpr uint32_t kBarDrain = kMisc + 264;
  static constexpr uint32_t kBarTapeRdy = kMisc + 272;     // [2] h0 .. h8
  static constexpr uint32_t kBarTapeEnc = kMisc + 288;     // [2] enc_xyz
  static constexpr uint32_t kBarTapeTail = kMisc + 304;    // [2] enc_dir and h9
  static constexpr uint32_t kBarTapeDone = kMisc + 320;    // [2]
  static constexpr uint32_t kTmemSlot = kMisc + 336;
  static constexpr uint32_t kAbort = kMisc + 344;          // int, then the wait limit (u64) at +8
  static constexpr uint32_t kHeadW = kMisc + 368;          // the sigma head's weights [256], the rgb head's [128][3]
  static constexpr uint32_t kHeadB = kHeadW + (256 + 384) * 4;  // FP8: dense_9's biases and scales [2][128]
  static constexpr uint32_t kSmemBytes = kHeadB + (F8 ? 1024 : 0);
  static_assert(kSmemBytes <= 227 * 1024 && kAbort % 8 == 0 && kHeadW % 16 == 0, "shared memory");
};

// ---------------------------------------------------------------------------
// Positional encodings as packed A-operand columns.
// ---------------------------------------------------------------------------
// The tensor-core kernels' positional encoding (model.py:319-331): octave
// l of a coordinate from one sincosf at octave 4*floor(l/4) and l % 4 angle
// doublings (the FP32 angle doubles exactly from one octave to the next;
// sin 2a = (2 sin a) cos a, cos 2a = cos a cos a - sin a sin a, each
// operation rounded in FP32): at most three doublings, ~5e-7 from sincosf at
// every octave, below the BF16 (or E4M3) rounding the value then gets. The
// value of an octave does not depend on which warp computes it.
template <int NP, int L, int W, int Q>
__device__ __forceinline__ void encode_pairs_q(const float (&x)[3], float (&v)[W]) {
  float sn = 0.0f, cs = 1.0f;
  int cur_c = -1, cur_l = -1;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int ks = 3 + 2 * p;  // sin at ks, cos at ks + 1
    if (ks + 1 < W * Q || ks >= W * Q + W) continue;
    const int c = p / L, l = p % L;
    if (c != cur_c || (l & 3) == 0 || cur_l != l - 1) {
      // a chain starts at octave 4*floor(l/4)
      const int l0 = l & ~3;
      // (the chains one after another: side by side they take the registers of the epilogue around them)
      float xc = x[c];
      asm volatile("" : "+f"(xc) : "f"(sn), "f"(cs));
      sincosf(fmul(xc, enc_multiplier(l0)), &sn, &cs);
      for (int d = l0; d < l; ++d) {
        const float s2 = fmul(fmul(2.0f, sn), cs);
        cs = fsub(fmul(cs, cs), fmul(sn, sn));
        sn = s2;
      }
    } else {
      const float s2 = fmul(fmul(2.0f, sn), cs);
      cs = fsub(fmul(cs, cs), fmul(sn, sn));
      sn = s2;
    }
    cur_c = c;
    cur_l = l;
    if (ks >= W * Q && ks < W * Q + W) v[ks - W * Q] = sn;
    if (ks + 1 >= W * Q && ks + 1 < W * Q + W) v[ks + 1 - W * Q] = cs;
  }
}

// N values to the K-major operand's bytes.
template <int N, bool F8>
__device__ __forceinline__ void pack_cols(const float (&v)[N], uint32_t (&pk)[F8 ? N / 4 : N / 2]) {
#pragma unroll
  for (int i = 0; i < (F8 ? N / 4 : N / 2); ++i)
    pk[i] = F8 ? pack_e4m3x4(v[(4 * i) % N], v[(4 * i + 1) % N], v[(4 * i + 2) % N], v[(4 * i + 3) % N])
               : pack_bf16(v[2 * i], v[2 * i + 1]);
}
// Packed columns as row r's 16-byte chunks c0 .. of the atom at `atom`.
template <int N>
__device__ __forceinline__ void store_chunks(uint32_t atom, int r, uint32_t c0, const uint32_t (&pk)[N]) {
  const uint32_t row = atom + (uint32_t)r * 128u, x = (uint32_t)r & 7u;
#pragma unroll
  for (int i = 0; i < N / 4; ++i)
    st_shared_v4(row + (((c0 + i) ^ x) << 4), pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
}

// A row's encoding, packed: enc_xyz's 64 columns (63 values, column 63 = 0) or
// enc_dir's 32 (27 values, 5 zero pad).
template <bool F8, bool DIR>
__device__ __forceinline__ void encode_row(const float (&x)[3], uint32_t (&pk)[(DIR ? 32 : 64) / (F8 ? 4 : 2)]) {
  constexpr int W = DIR ? 32 : 64;
  float v[W];
#pragma unroll
  for (int i = 0; i < W; ++i) v[i] = i < 3 ? x[i % 3] : 0.0f;
  encode_pairs_q<DIR ? 12 : 30, DIR ? 4 : 10, W, 0>(x, v);
  pack_cols<W, F8>(v, pk);
}

// ---------------------------------------------------------------------------
// Epilogue of a plain layer: fragments.
// ---------------------------------------------------------------------------
// This thread's biases (FP8: and weight scales) of 32 of the warp's columns
// in the 16x256b layout: group i of eight accumulator columns holds the
// thread's pair at 2*(lane%4). In BF16 they are channels 8i + 2q, +1 (q = lane
// % 4); the FP8 pack orders the channels of each 16 so that the pairs of
// groups 2j and 2j + 1 are channels 16j + 4q .. + 3 (one word of E4M3).
template <bool F8>
struct FragBias {
  float b[8], s[F8 ? 8 : 1];
  __device__ __forceinline__ void load(const float *bias, const float *scale, int q) {
    if (F8) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        *reinterpret_cast<float4 *>(b + 4 * j) = *reinterpret_cast<const float4 *>(bias + 16 * j + 4 * q);
        *reinterpret_cast<float4 *>(s + (F8 ? 4 * j : 0)) = *reinterpret_cast<const float4 *>(scale + 16 * j + 4 * q);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float2 *>(b + 2 * i) = *reinterpret_cast<const float2 *>(bias + 8 * i + 2 * q);
    }
  }
  // accumulator pair of group i to the layer's output
  __device__ __forceinline__ void apply(int i, uint32_t r0, uint32_t r1, float &v0, float &v1) const {
    if (F8)
      fma_f32x2(v0, v1, __uint_as_float(r0), __uint_as_float(r1), s[F8 ? 2 * i : 0], s[F8 ? 2 * i + 1 : 0], b[2 * i],
                b[2 * i + 1]);
    else
      add_f32x2(v0, v1, __uint_as_float(r0), __uint_as_float(r1), b[2 * i], b[2 * i + 1]);
  }
};

// max(x, 0) of four E4M3 values as fmaxf would have it before the rounding:
// zero where the byte's sign is set, and for NaN (0x7F). Three operations on
// the word instead of four FP32 maxima (two cycles each).
__device__ __forceinline__ uint32_t relu_e4m3x4(uint32_t w) {
  // bit 7 of a byte + 1: negative (0x80 .. 0xFE) or 0x7F; no byte is 0xFF, so none carries
  uint32_t m;
  asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(m) : "r"(w + 0x01010101u));  // each byte its sign
  return w & ~m;
}

// 16 rows x 32 columns of fragments (raw: group i's four registers: the pair
// of row lane/4, then of row lane/4 + 8) to the operand: `addr` this lane's
// stmatrix row (row 8*((lane>>3)&1) + lane%8 of the 16, chunk 0), cx = (lane>>4) ^
// (lane & 7) its swizzled chunk in units of 16 bytes, c0 the columns' first
// chunk in the atom (even).
// KEEP: raw becomes the ReLU of the FP32 values (fmaxf: 0 for NaN, as the sigma
// head has it; the BF16 operand keeps NaN, as in every other layer).
template <bool F8, bool KEEP>
__device__ __forceinline__ void store_frag(uint32_t addr, uint32_t cx, uint32_t c0, uint32_t (&raw)[16],
                                           const FragBias<F8> &fb, bool relu) {
  float v[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) fb.apply(i / 2, raw[2 * i], raw[2 * i + 1], v[2 * i], v[2 * i + 1]);
  if (KEEP) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float m = fmaxf(v[i], 0.0f);
      raw[i] = __float_as_uint(m);
      if (F8) v[i] = m;
    }
  }
  uint32_t w[F8 ? 4 : 8];
  if (F8) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {  // chunk j: rows lane/4 (2j), lane/4 + 8 (2j + 1)
      w[2 * j] = pack_e4m3x4(v[8 * j], v[8 * j + 1], v[8 * j + 4], v[8 * j + 5]);
      w[2 * j + 1] = pack_e4m3x4(v[8 * j + 2], v[8 * j + 3], v[8 * j + 6], v[8 * j + 7]);
      if (!KEEP && relu) {
        w[2 * j] = relu_e4m3x4(w[2 * j]);
        w[2 * j + 1] = relu_e4m3x4(w[2 * j + 1]);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)  // chunk i / 2: rows lane/4 (even i), lane/4 + 8
      w[F8 ? 0 : i] = relu ? pack_bf16_relu(v[2 * i], v[2 * i + 1]) : pack_bf16(v[2 * i], v[2 * i + 1]);
  }
#pragma unroll
  for (int m = 0; m < (F8 ? 4 : 8); m += 4)
    stmatrix_x4(addr + (((c0 + m / 2) ^ cx) << 4), w[m], w[m + 1], w[m + 2], w[m + 3]);
}

// 64 columns as two times 32.
template <bool F8>
__device__ __forceinline__ void store_frag64(uint32_t addr, uint32_t cx, uint32_t c0, const uint32_t (&raw)[32],
                                             const FragBias<F8> (&fb)[2], bool relu) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t r[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = raw[16 * h + i];
    store_frag<F8, false>(addr, cx, c0 + (F8 ? 2u : 4u) * h, r, fb[h], relu);
  }
}

// ---------------------------------------------------------------------------
// Epilogue of the head layers: a row per lane, 32 columns at a time.
// ---------------------------------------------------------------------------
// A load that stays where it is written: hoisted and batched by the compiler,
// the head weights' loads would take the registers of everything else (and
// spill).
__device__ __forceinline__ float4 ld_here(const float *p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 lds_here(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
// ---------------------------------------------------------------------------
// MMA issue (pair_tc.cuh): per layer, generated at compile time
// ---------------------------------------------------------------------------
// The MMAs of GEMM layer G for sub-tile S: its K rows are [activation (256) |
// encoding (the rest)] for dense_5 and dense_9, the encoding (in the
// activation region) for dense_0 and the activation alone otherwise.
template <int G, int S, bool F8>
__device__ __forceinline__ void issue_gemm(uint32_t sbase, uint32_t tmem, bool release, uint32_t tile_phase,
                                           RingPos &rp, volatile int *abort_flag, int *err) {
  using L = Layout<F8>;
  constexpr int N = gemm_n(G), H = N / 2;
  constexpr int kSteps = gemm_kp(G) * (int)L::kE / 32;
  constexpr int kPer = (int)kPairStage / (H * 32);  // MMAs per stage
  constexpr int kAct = G == 0 ? kSteps : 256 * (int)L::kE / 32, kEnc = kSteps - kAct;
  constexpr uint32_t idesc = F8 ? idesc_e4m3(256, N) : idesc_bf16(256, N);
  static_assert(G == 0 || kAct % kPer == 0, "stages must not straddle the activation/encoding split");
  static_assert(kEnc <= kPer && (kSteps + kPer - 1) / kPer <= L::kNst, "a layer fits the ring");
  const uint32_t bar_full = sbase + L::kBarFull, bar_empty = sbase + L::kBarEmpty;
  // Descriptor start addresses are 18-bit shared-window offsets (a CTA's
  // window address may carry bits above them, as in a cluster launch).
  const uint32_t sw = sbase & 0x3FFFFu;
  const uint32_t ring_lo = (sw >> 4) | ((uint32_t)H << 16);
  const uint32_t act_lo = ((sw + L::kActOff + S * L::kActBytes) >> 4) | (1u << 16);
  const uint32_t acc = tmem + S * 256;
  if constexpr (kAct >= kPer)
    issue_run<L::kNst, kAct / kPer, kPer, H, F8, true, S == 0>(bar_full, bar_empty, ring_lo, act_lo, acc, idesc, release, rp,
                                                      abort_flag, err);
  else
    issue_run<L::kNst, 1, kAct, H, F8, true, S == 0>(bar_full, bar_empty, ring_lo, act_lo, acc, idesc, release, rp, abort_flag,
                                            err);
  if constexpr (kEnc > 0) {
    if (G == 5 || S == 0) {
      // E holds A's encoding, then B's, then the direction encodings
      wait_fast(sbase + (G == 9 ? L::kBarDir : S == 0 ? L::kBarEncA : L::kBarEncB), tile_phase, abort_flag, err);
      tc_fence_after();
    }
    const uint32_t enc_lo = ((sw + L::kEncOff + (G == 9 ? S * 64u : 0u)) >> 4) | (1u << 16);
    issue_run<L::kNst, 1, kEnc, H, F8, false, S == 0>(bar_full, bar_empty, ring_lo, enc_lo, acc, idesc, release, rp, abort_flag,
                                             err);
  }
}

// One layer: per sub-tile, wait until its A operand is written (and its
// accumulator read), issue, then signal the accumulator full. The last
// sub-tile's MMAs release the layer's stages. actr_phase: the parity of the
// epilogue's operand barriers, toggled per layer from dense_1 on; tile_phase:
// of the barriers that complete once per tile.
template <int G, int S, bool F8>
__device__ __forceinline__ void issue_sub(uint32_t sbase, uint32_t tmem, bool release, RingPos &rp, uint32_t actr_phase,
                                          uint32_t tile_phase, volatile int *abort_flag, int *err) {
  using L = Layout<F8>;
  if (G == 0)
    wait_fast(sbase + L::kBarAct0 + 8 * S, tile_phase, abort_flag, err);
  else
    wait_fast(sbase + L::kBarActr + 8 * S, actr_phase, abort_flag, err);
  tc_fence_after();
  issue_gemm<G, S, F8>(sbase, tmem, release, tile_phase, rp, abort_flag, err);
  if (G == 5) tc_commit_pair(sbase + L::kBarAcc5 + 8 * S);
  tc_commit_pair(sbase + (G == 9 ? L::kBarAcc9 : L::kBarAccf) + 8 * S);
}
template <int G, bool F8>
__device__ __forceinline__ void issue_layer(uint32_t sbase, uint32_t tmem, int nsub, RingPos &rp, uint32_t &actr_phase,
                                            uint32_t tile_phase, volatile int *abort_flag, int *err) {
  const RingPos start = rp;
  issue_sub<G, 0, F8>(sbase, tmem, nsub == 1, rp, actr_phase, tile_phase, abort_flag, err);
  if (nsub == 2) {
    rp = start;
    issue_sub<G, 1, F8>(sbase, tmem, true, rp, actr_phase, tile_phase, abort_flag, err);
  }
  if (G > 0) actr_phase ^= 1u;
}

// BF16, a tile of sub-tile A alone (a pair's odd last one, or a small batch's
// only one): layer G into accumulator G % 2, so that its MMAs can start on the
// first 128 K, which the epilogue signals on A's barrier, while the epilogue
// still reads the accumulator before; the rest follows on B's barrier.
template <int G>
__device__ __forceinline__ void issue_solo(uint32_t sbase, uint32_t acc, RingPos &rp, uint32_t &actr_phase,
                                           uint32_t tile_phase, volatile int *abort_flag, int *err) {
  using L = Layout<false>;
  constexpr int N = gemm_n(G), H = N / 2, kPer = (int)kPairStage / (H * 32), kHalf = 8 / kPer;
  constexpr int kEnc = gemm_kp(G) * 2 / 32 - 16;
  const uint32_t bar_full = sbase + L::kBarFull, bar_empty = sbase + L::kBarEmpty, sw = sbase & 0x3FFFFu;
  const uint32_t ring_lo = (sw >> 4) | ((uint32_t)H << 16), act_lo = ((sw + L::kActOff) >> 4) | (1u << 16);
  wait_fast(sbase + L::kBarActr, actr_phase, abort_flag, err);
  tc_fence_after();
  issue_run<L::kNst, kHalf, kPer, H, false, true, true>(bar_full, bar_empty, ring_lo, act_lo, acc, idesc_bf16(256, N), true,
                                                        rp, abort_flag, err);
  wait_fast(sbase + L::kBarActr + 8, actr_phase, abort_flag, err);
  tc_fence_after();
  issue_run<L::kNst, kHalf, kPer, H, false, false, true>(bar_full, bar_empty, ring_lo, act_lo + 2 * (kAtom >> 4), acc,
                                                         idesc_bf16(256, N), true, rp, abort_flag, err);
  if constexpr (kEnc > 0) {
    wait_fast(sbase + (G == 9 ? L::kBarDir : L::kBarEncA), tile_phase, abort_flag, err);
    tc_fence_after();
    issue_run<L::kNst, 1, kEnc, H, false, false, true>(bar_full, bar_empty, ring_lo,
                                                       ((sw + L::kEncOff) >> 4) | (1u << 16), acc, idesc_bf16(256, N),
                                                       true, rp, abort_flag, err);
  }
  if (G == 5) tc_commit_pair(sbase + L::kBarAcc5);
  tc_commit_pair(sbase + (G == 9 ? L::kBarAcc9 : L::kBarAccf));
  actr_phase ^= 1u;
}

// ---------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------
// F8: E4M3 operands (kind::f8f6f4, K = 32 per MMA) with per-output-channel
// weight scales applied in the epilogue; else BF16 (kind::f16, K = 16).
// STORE (BF16 only, training): every layer's BF16 activations (the operands
// the next layer's MMAs read) and the encodings also go to `tape`, kActsLd
// BF16 values per row at the columns of the FP32 tape (acts_offset).
template <bool F8, bool STORE>
__global__ void __launch_bounds__(threads_of(STORE), 1)
    mlp_tc_kernel(const uint8_t *packed, const float *xyz,
                    const float *dirs, long long n_max, int rpd, float *__restrict__ rgb_out,
                    float *__restrict__ sigma_out, int *__restrict__ err, RowMap rm, uint16_t *__restrict__ tape,
                    unsigned long long wait_ns, long long withhold, const __grid_constant__ PairMaps maps) {
  static_assert(!(STORE && F8), "the activation tape is BF16");
  static_assert(kActsLd % 8 == 0 && kActsEncXyz == 0 && acts_offset(0) == 64 && kActsEncDir % 8 == 0,
                "tape columns in swizzle atoms");
  using L = Layout<F8>;
  extern __shared__ __align__(1024) uint8_t smem[];
  after_previous();
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L::kAbort);
  const float *table = reinterpret_cast<const float *>(packed + (F8 ? kFp8TableOff : kBf16TableOff));
  const float *scales = reinterpret_cast<const float *>(packed + kFp8ScaleOff);  // FP8 only
  // Row count (device-side with a row map from a compaction kernel), and this
  // pair's sub-tiles: [first, first + count) of ceil(n / 256), dealt evenly.
  // Tile k holds sub-tiles first + 2k and, unless it is the odd last one,
  // first + 2k + 1; crank = the CTA's place in its pair.
  const uint32_t crank = cluster_rank();
  const long long n = rm.n_dev ? min((long long)*rm.n_dev, n_max) : n_max;
  int first, count;
  {
    const unsigned subs = (unsigned)((n + kSubRows - 1) / kSubRows), np = cluster_count(), p = cluster_id();
    const unsigned q = subs / np, rest = subs % np;
    first = (int)(p * q + min(p, rest));
    // (the swizzled operands need 1024-byte alignment: without it nothing runs)
    count = (sbase & 1023u) != 0 ? 0 : (int)(q + (p < rest ? 1u : 0u));
  }
  const int ntiles = (count + 1) / 2;
  // logical row r of this CTA's part of sub-tile s of tile k
  auto row_of = [&](int k, int s, int r) -> long long {
    return (long long)(first + 2 * k + s) * kSubRows + (int)crank * 128 + r;
  };

  // head weights: table[kSigmaWOff ..] (256 floats), table[kRgbWOff ..] (384)
  static_assert(kSigmaWOff % 4 == 0 && kRgbWOff % 4 == 0, "float4 copies");
  if (F8 && threadIdx.x < 64)
    reinterpret_cast<float4 *>(smem + L::kHeadB)[threadIdx.x] = reinterpret_cast<const float4 *>(
        (threadIdx.x < 32 ? table : scales - 128) + bias_offset(9))[threadIdx.x];
  if (threadIdx.x < 64 + 96)
    reinterpret_cast<float4 *>(smem + L::kHeadW)[threadIdx.x] = reinterpret_cast<const float4 *>(
        table + (threadIdx.x < 64 ? kSigmaWOff : kRgbWOff - 256))[threadIdx.x];
  if (threadIdx.x == 0) {
    for (int s = 0; s < L::kNst; ++s) {
      // a stage completes on the even CTA's producer's arrival and the bytes
      // of both CTAs' copies (the odd CTA's signal it directly)
      mbar_init(sbase + L::kBarFull + 8 * s, 1);
      mbar_init(sbase + L::kBarEmpty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(sbase + L::kBarAccf + 8 * s, 1);
      mbar_init(sbase + L::kBarAcc5 + 8 * s, 1);
      mbar_init(sbase + L::kBarAcc9 + 8 * s, 1);
      mbar_init(sbase + L::kBarActr + 8 * s, 2 * kEpiWarps);  // one arrival per epilogue warp of both CTAs
      mbar_init(sbase + L::kBarAct0 + 8 * s, 2 * 4);          // ... per side warp of both CTAs
      mbar_init(sbase + L::kBarRead8 + 8 * s, 4);
      mbar_init(sbase + L::kBarSig + 8 * s, 4);
      mbar_init(sbase + L::kBarTapeRdy + 8 * s, kEpiWarps);
      mbar_init(sbase + L::kBarTapeEnc + 8 * s, 4);
      mbar_init(sbase + L::kBarTapeTail + 8 * s, 4);
      mbar_init(sbase + L::kBarTapeDone + 8 * s, 1);
    }
    mbar_init(sbase + L::kBarEncA, 2 * 4);
    mbar_init(sbase + L::kBarEncB, 2 * 4);
    mbar_init(sbase + L::kBarDir, 2 * 4);
    mbar_init(sbase + L::kBarDrain, 1);
    *abort_flag = 0;
    set_wait_limit(abort_flag, wait_ns);
    if ((sbase & 1023u) != 0) atomicExch(err, NERFGB_E_UNSUPPORTED);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    // one warp of each CTA allocates collectively (same address in both)
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + L::kTmemSlot),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before any arrival reaches them
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + L::kTmemSlot);

  if (warp == 0) {
    // ---------------- weight producer ----------------
    // One thread issues the loads in ring order: a stage frees once per
    // chunk of MMAs, and the copies of one thread complete at a few hundred
    // cycles' spacing, so one thread keeps pace. Each CTA copies its N-half
    // with a 2-SM tensor copy that completes on the even CTA's full barrier,
    // whose producer expects both halves' bytes.
    if (lane == 0) {
      uint32_t used = 0;  // bit st: parity of the copies issued into stage st
      int st = 0;
      bool ok = true;
      long long nq = 0;  // chunks of this CTA's load sequence
      for (int tile = 0; tile < ntiles && ok; ++tile)
        for (int g = 0; g < kNumGemm && ok; ++g) {
          const uint32_t H = (uint32_t)gemm_n(g) / 2, per = kPairStage / H;  // bytes of K per full chunk
          uint32_t left = (uint32_t)gemm_kp(g) * L::kE;
          uint32_t src = (uint32_t)(gemm_w_offset(g) * L::kE);
          for (; left > 0; left -= min(left, per), src += 2 * kPairStage) {
            if (!wait_bar(sbase + L::kBarEmpty + 8 * st, ((used >> st) & 1u) ^ 1u, abort_flag, err)) {
              ok = false;
              break;
            }
            // test hook of the failure path: the even CTA leaves chunk `withhold` unloaded
            if (!(nq++ == withhold && crank == 0)) {
              const uint32_t bytes = H * min(left, per);
              const uint32_t full = sbase + L::kBarFull + 8 * st;
              if (crank == 0) mbar_expect_tx(full, 2 * bytes);
              tma_2d_pair(sbase + st * kPairStage, &maps.map[pair_map_of(bytes)], 0,
                          (int)((src + crank * bytes) >> 8), crank == 0 ? full : peer_addr(full, 0));
            }
            used ^= 1u << st;
            if (++st == L::kNst) st = 0;
          }
        }
      if (!ok && crank == 0) {
        // Drain: wait (bounded) for the stages' last copies (both CTAs';
        // the odd CTA's own drain is at the kernel's end).
        const uint64_t t0 = globaltimer();
        for (int k = 0; k < L::kNst; ++k)
          while (!mbar_try(sbase + L::kBarFull + 8 * k, ((used >> k) & 1u) ^ 1u) && globaltimer() - t0 < 10000000ull) {
          }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the even CTA's issues for both) ----------------
    if (lane == 0 && crank == 0) {
      // both CTAs must hold the same TMEM columns (the collective
      // allocation gives them); otherwise issue nothing
      uint32_t peer_tmem;
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_tmem) : "r"(peer_addr(sbase + L::kTmemSlot, 1))
                   : "memory");
      if (peer_tmem != tmem) {
        atomicExch(err, NERFGB_E_UNSUPPORTED);
        *abort_flag = 1;
      }
      // After an abort every wait returns at once: the remaining MMAs of the
      // tile read stale (in-bounds) shared memory and the tile loop ends.
      RingPos rp{0, 0u};
      uint32_t actr_phase = 0;
      for (int tile = 0; tile < ntiles; ++tile) {
        if (*abort_flag) break;
        const int nsub = 2 * tile + 1 < count ? 2 : 1;
        const uint32_t ph = (uint32_t)(tile & 1);
        issue_layer<0, F8>(sbase, tmem, nsub, rp, actr_phase, ph, abort_flag, err);
        if (!F8 && !STORE && nsub == 1) {
          if (tile > 0) {  // the tile before's B has been read
            wait_fast(sbase + L::kBarAct0 + 8, ph, abort_flag, err);
            tc_fence_after();
          }
#pragma unroll 1
          for (int g = 1; g <= 4; ++g) issue_solo<1>(sbase, tmem + 256 * (g & 1), rp, actr_phase, ph, abort_flag, err);
          issue_solo<5>(sbase, tmem + 256, rp, actr_phase, ph, abort_flag, err);
#pragma unroll 1
          for (int g = 6; g <= 8; ++g) issue_solo<6>(sbase, tmem + 256 * (g & 1), rp, actr_phase, ph, abort_flag, err);
          issue_solo<9>(sbase, tmem + 256, rp, actr_phase, ph, abort_flag, err);
          break;  // (the last tile)
        }
        // (one copy of the issue code for the layers of one shape: the
        // kernel's code is several times the instruction cache's first levels)
#pragma unroll 1
        for (int g = 1; g <= 4; ++g) issue_layer<1, F8>(sbase, tmem, nsub, rp, actr_phase, ph, abort_flag, err);
        issue_layer<5, F8>(sbase, tmem, nsub, rp, actr_phase, ph, abort_flag, err);
#pragma unroll 1
        for (int g = 6; g <= 8; ++g) issue_layer<6, F8>(sbase, tmem, nsub, rp, actr_phase, ph, abort_flag, err);
        issue_layer<9, F8>(sbase, tmem, nsub, rp, actr_phase, ph, abort_flag, err);
        static_assert(kNumGemm == 10, "layers 1-4 and 6-8 are alike");
      }
      if (ntiles > 0) {
        // Drain every MMA issued by this thread before TMEM is released (in
        // both CTAs).
        tc_commit_pair(sbase + L::kBarDrain);
        uint64_t t0 = globaltimer();
        while (!mbar_try(sbase + L::kBarDrain, 0) && globaltimer() - t0 < 100000000ull) {
        }
      }
    }
  } else if (STORE && warp == kTapeWarp) {
    // ---------------- tape writer ----------------
    // Per tile and sub-tile ten regions are signalled in order: enc_xyz
    // (dense_0's operand, by the side warps), then h0 .. h8 (each layer's
    // output, the next layer's operand, by the epilogue). Each goes to its
    // tape columns of the sub-tile's 128 rows as one tensor store of 128-byte
    // rows (rows past n are not written); once the store has read shared
    // memory, tape_done tells that the region may be rewritten. The row's last
    // columns, enc_dir and h9, follow in the region's second and third atom
    // on a barrier of their own (before the next tile's enc_xyz, whose
    // tape_done covers them), but for h9's last 32 columns, half an atom,
    // which the side warps store themselves.
    if (lane == 0) {
      uint32_t rdy_phase[2] = {0u, 0u};
      bool ok = true;
      // one region: sub-tile s of tile k, from atom A of the operand to column group z of the tape
      auto store = [&](uint32_t bar, uint32_t parity, const CUtensorMap *map, int k, int s, uint32_t atom, int z) {
        if (!wait_bar(sbase + bar + 8 * s, parity, abort_flag, err)) return false;
        const long long row = row_of(k, s, 0);
        if (row < n) {  // (a box from row n on would write nothing)
          tma_store_3d(map, sbase + L::kActOff + s * L::kActBytes + atom * kAtom, 0, (int)row, z);
          bulk_commit();
          bulk_wait_read();
        }
        return true;
      };
      for (int tile = -1; tile < ntiles && ok; ++tile) {
        const int next_subs = min(2, count - 2 * (tile + 1));
        const int nsub = tile < 0 ? next_subs : 2 * tile + 1 < count ? 2 : 1;
        for (int e = 0; e < 9 && tile >= 0 && ok; ++e)
          for (int s = 0; s < nsub && ok; ++s) {
            ok = store(L::kBarTapeRdy, rdy_phase[s], &maps.tape[0], tile, s, 0, acts_offset(e) / 64);
            rdy_phase[s] ^= 1u;
            if (ok) mbar_arrive(sbase + L::kBarTapeDone + 8 * s);
          }
        for (int s = 0; s < nsub && ok; ++s) {
          if (tile >= 0)
            ok = store(L::kBarTapeTail, (uint32_t)(tile & 1), &maps.tape[2], tile, s, 1, kActsEncDir / 64);
          if (ok && s < next_subs) {
            ok = store(L::kBarTapeEnc, (uint32_t)((tile + 1) & 1), &maps.tape[1], tile + 1, s, 0, 0);
            if (ok) mbar_arrive(sbase + L::kBarTapeDone + 8 * s);
          }
        }
      }
      bulk_wait_all();  // no store still reads this CTA's shared memory or writes the tape
    }
  } else if (warp >= kSideWarp && warp < kTapeWarp) {
    // ---------------- side warps ----------------
    // One warp per TMEM lane quadrant, a row per lane: the encodings and
    // dense_9 with the rgb head (model.py:385-386).
    const int qd = warp & 3, r = 32 * qd + lane;  // row within a sub-tile (= TMEM lane)
    const uint32_t tlane = tmem + ((uint32_t)(32 * qd) << 16);
    const uint32_t enc = sbase + L::kEncOff;
    auto arrive_local = [&](uint32_t bar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    // One arrival per warp on the even CTA's barrier: what the warp wrote to
    // shared memory is visible to the MMAs that wait for it (and what it read
    // from TMEM may be overwritten).
    auto arrive_even = [&](uint32_t bar) {
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(peer_addr(bar, 0));
    };
    auto wait_all = [&](uint32_t bar, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, wait_bar(bar, parity, abort_flag, err));
    };
    // Physical row of a logical row: the row map's entry (without a map the row
    // itself; the last one for rows past n).
    auto phys = [&](long long grow) -> long long {
      const long long g = grow < n ? grow : n - 1;
      return rm.map ? (long long)NG_IDX(rm.map[g], n_max, kSiteMlpRowMap) : g;
    };
    constexpr int kPk = 64 / (F8 ? 4 : 2);
    const float4 bias9 = ld_here(table + bias_offset(9) + 4 * lane);  // dense_9's of columns 4 lane .. + 3 (BF16)
    auto from_lane = [](const float4 &v, int src) {
      return float4{__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                    __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src)};
    };
    // dense_0's operand of sub-tile s is written and its accumulator read
    auto start_layer0 = [&](int s) {
      arrive_even(sbase + L::kBarAct0 + 8 * s);
      if (STORE && lane == 0) mbar_arrive(sbase + L::kBarTapeEnc + 8 * s);
    };
    bool ok = true;
    // (tile -1 is the first tile's start: the end of its dense_9 alone, so that
    // there is one copy of the encoding's code)
#pragma unroll 1
    for (int tile = -1; tile < ntiles && ok; ++tile) {
      const uint32_t ph = (uint32_t)(tile & 1);
      const int next_subs = max(0, min(2, count - 2 * (tile + 1)));  // of the next tile
      const int nsub = 2 * tile + 1 < count ? 2 : 1;
      // The encodings in the order that they are due (one copy of the code):
      // this tile's into E (A's now, as the tile before's dense_9 is done, B's
      // once A's dense_5 is, then the direction encodings once B's is), then
      // the next tile's, kept packed until its operand regions are free.
      uint32_t cur[kPk] = {}, nxt[kPk] = {};
#pragma unroll 1
      for (int q = tile < 0 ? 2 : 0; q < 2 + next_subs; ++q) {
        const int s = q & 1;
        if (q < nsub || q >= 2) {
          const long long grow = row_of(tile + (q >> 1), s, r), p = phys(grow);
          float x[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) x[c] = grow < n ? xyz[p * 3 + c] : 0.0f;
#pragma unroll
          for (int i = 0; i < kPk; ++i) cur[i] = nxt[i];
          encode_row<F8, false>(x, nxt);
        }
        if (q < 2) {
          if (q < nsub) {
            if (q == 1 && !wait_all(sbase + L::kBarAcc5, ph)) {
              ok = false;
              break;
            }
            store_chunks(enc, r, 0u, nxt);
            arrive_even(sbase + (q == 0 ? L::kBarEncA : L::kBarEncB));
          }
          if (q == 1) {
            if (!wait_all(sbase + L::kBarAcc5 + 8 * (nsub - 1), ph)) {
              ok = false;
              break;
            }
#pragma unroll 1
            for (int d = 0; d < nsub; ++d) {
              const long long dr = phys(row_of(tile, d, r)) / rpd;
              float dir[3];
#pragma unroll
              for (int c = 0; c < 3; ++c) dir[c] = dirs[dr * 3 + c];
              uint32_t pd[kPk / 2];
              encode_row<F8, true>(dir, pd);
              store_chunks(enc, r, (uint32_t)(4 * d), pd);
            }
            arrive_even(sbase + L::kBarDir);
          }
        } else if (tile < 0) {
          store_chunks(sbase + L::kActOff + s * L::kActBytes, r, 0u, nxt);
          start_layer0(s);
        }
      }
      if (tile < 0) continue;
      if (!ok) break;
      if (next_subs == 1) {
#pragma unroll
        for (int i = 0; i < kPk; ++i) cur[i] = nxt[i];
      }
#pragma unroll 1
      for (int s = 0; s < nsub; ++s) {
        const uint32_t act = sbase + L::kActOff + s * L::kActBytes;
        // dense_9 is done (with the tape: and h8 stored, the last of the tile's ten regions)
        if (!wait_all(sbase + L::kBarAcc9 + 8 * s, ph) || (STORE && !wait_all(sbase + L::kBarTapeDone + 8 * s, 1u)) ||
            !wait_all(sbase + L::kBarSig + 8 * s, ph)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (s < next_subs) store_chunks(act, r, 0u, cur);
#pragma unroll
        for (int i = 0; i < kPk; ++i) cur[i] = nxt[i];
        const long long grow = row_of(tile, s, r);
        const long long p = phys(grow);
        if (F8) {
          const float a = tmem_ld1(tlane + s * 256 + 254), b = tmem_ld1(tlane + s * 256 + 255);
          if (grow < n) sigma_out[p] = fmaxf((a + b) + table[kSigmaBOff], 0.0f);
        } else {
          float q[4];
          tmem_ld4(tlane + s * 256 + 252, q);
          if (grow < n) sigma_out[p] = fmaxf(((q[0] + q[1]) + (q[2] + q[3])) + table[kSigmaBOff], 0.0f);
        }
        const uint32_t acc9 = tlane + (!F8 && !STORE && nsub == 1 ? 256 : s * 256);  // dense_9's accumulator
        // rgb = sigmoid(h9 . W + b) in FP32. BF16: ((q0 + q1) + (q2 + q3)) of the
        // quarters' sums of 32 columns; FP8: the 128 columns in order.
        float rgb[3] = {0.f, 0.f, 0.f}, half[3] = {0.f, 0.f, 0.f};
        uint32_t ra[16], rb[16];
        tmem_ld16(acc9, ra);
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          float acc[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[c] = F8 ? rgb[c] : 0.0f;
          uint32_t h9[16];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            // 16 columns, the next 16 on their way
            uint32_t(&raw)[16] = k == 0 ? ra : rb;
            const int col = 32 * j + 16 * k;
            tmem_wait16(raw);
            if (k == 0)
              tmem_ld16(acc9 + col + 16, rb);
            else if (j < 3)
              tmem_ld16(acc9 + col + 16, ra);
            else if (s < next_subs)
              start_layer0(s);  // the accumulator is read
            else if (!F8 && !STORE && next_subs == 1)
              arrive_even(sbase + L::kBarAct0 + 8);  // B's, which a tile alone uses too
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 b4 = F8 ? lds_here(sbase + L::kHeadB + 4 * (col + i)) : from_lane(bias9, (col + i) / 4);
              float v[4];
              if (F8) {
                const float4 s4 = lds_here(sbase + L::kHeadB + 512 + 4 * (col + i));
                fma_f32x2(v[0], v[1], __uint_as_float(raw[i]), __uint_as_float(raw[i + 1]), s4.x, s4.y, b4.x, b4.y);
                fma_f32x2(v[2], v[3], __uint_as_float(raw[i + 2]), __uint_as_float(raw[i + 3]), s4.z, s4.w, b4.z, b4.w);
              } else {
                add_f32x2(v[0], v[1], __uint_as_float(raw[i]), __uint_as_float(raw[i + 1]), b4.x, b4.y);
                add_f32x2(v[2], v[3], __uint_as_float(raw[i + 2]), __uint_as_float(raw[i + 3]), b4.z, b4.w);
              }
              // rows col + i .. + 3 of the [128][3] rgb kernel: 12 floats
              const uint32_t wr = sbase + L::kHeadW + 1024 + (col + i) * 12;
              const float4 a4 = lds_here(wr), c4 = lds_here(wr + 16), e4 = lds_here(wr + 32);
              const float w12[12] = {a4.x, a4.y, a4.z, a4.w, c4.x, c4.y, c4.z, c4.w, e4.x, e4.y, e4.z, e4.w};
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const float h = fmaxf(v[q], 0.0f);
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[c] = fmaf(h, w12[3 * q + c], acc[c]);
              }
              if (STORE) {
                h9[8 * k + i / 2] = pack_bf16_relu(v[0], v[1]);
                h9[8 * k + i / 2 + 1] = pack_bf16_relu(v[2], v[3]);
              }
            }
          }
          if (F8) {
#pragma unroll
            for (int c = 0; c < 3; ++c) rgb[c] = acc[c];
          } else if (j & 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              half[c] += acc[c];
              rgb[c] = j == 1 ? half[c] : rgb[c] + half[c];
            }
          } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) half[c] = acc[c];
          }
          if (STORE) {
            // h9's columns as columns 32 + 32j .. of [enc_dir | h9] in the region's atoms 1, 2
            if (j < 3)
              store_chunks(act + kAtom * (1u + (uint32_t)(j + 1) / 2), r, (uint32_t)(((j + 1) & 1) * 4), h9);
            else if (grow < n)
              tape_store32(tape + grow * kActsLd + acts_offset(9) + 96, h9);
          }
        }
        if (STORE) {
          // enc_dir beside h9, then the tail goes to the tape
          uint32_t u[16];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            ld_shared_v4(enc + (uint32_t)r * 128u + (((uint32_t)(4 * s + i) ^ ((uint32_t)r & 7u)) << 4), u[4 * i],
                         u[4 * i + 1], u[4 * i + 2], u[4 * i + 3]);
          store_chunks(act + kAtom, r, 0u, u);
          fence_proxy_async();
          arrive_local(sbase + L::kBarTapeTail + 8 * s);
        }
        if (grow < n) {
#pragma unroll
          for (int c = 0; c < 3; ++c) rgb_out[p * 3 + c] = 1.0f / (1.0f + expf(-(rgb[c] + table[kRgbBOff + c])));
        }
      }
    }
  } else {
    // ---------------- epilogue warps ----------------
    // All eight warps serve whichever sub-tile's accumulator is ready (A, then
    // B, every layer but dense_9). Warp w reads TMEM lane quadrant qd = w % 4
    // (rows 32*qd ..) and column part cq: kCols columns, in BF16 as 64 in either
    // half of the layer, so that its first half is written first. (Spilled registers
    // would not stay in the 28 KB of L1 beside this much shared memory: each reload
    // is a trip to L2.)
    constexpr int kCols = 256 / kParts;
    const int qd = warp & 3, cq = (warp - 2) >> 2;
    const uint32_t tlane = tmem + ((uint32_t)(32 * qd) << 16);
    // stmatrix row of this lane in the part's first atom, and its swizzle (store_frag)
    const uint32_t frag_row = (uint32_t)(32 * qd + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128u +
                              (uint32_t)cq * kAtom;  // (either way the part's first 128 bytes of K)
    const uint32_t cx = (uint32_t)((lane >> 4) ^ (lane & 7));
    auto arrive_local = [&](uint32_t bar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    // first of the part's columns, and from its first half's to its second's
    const int pcol = F8 ? kCols * cq : 64 * cq;
    float sig[2][2] = {};  // the sigma head's sums, of the part (FP8) or of its halves
    uint32_t accf_phase = 0;         // both sub-tiles' accumulator barriers, per layer
    bool ok = true;
#pragma unroll 1
    for (int tile = 0; tile < ntiles && ok; ++tile) {
      const int nsub = 2 * tile + 1 < count ? 2 : 1;
      const bool solo = !F8 && !STORE && nsub == 1;  // (issue_solo)
#pragma unroll 1
      for (int g = 0; g < 9 && ok; ++g) {
#pragma unroll 1
        for (int s = 0; s < nsub; ++s) {
          // the first biases, while the accumulator is computed
          FragBias<F8> fb[2];
          const float *fbias = table + bias_offset(g) + pcol, *fscale = scales + bias_offset(g) + pcol;
          fb[0].load(fbias, fscale, lane & 3);
          fb[1].load(fbias + 32, fscale + 32, lane & 3);
          bool got = wait_bar(sbase + L::kBarAccf + 8 * s, accf_phase, abort_flag, err);
          if (STORE && got) {
            // the tape has what the region held: enc_xyz for g = 0 (of the ten
            // regions of a tile, the side warps wait for the last, h8)
            got = wait_bar(sbase + L::kBarTapeDone + 8 * s, (uint32_t)(g & 1), abort_flag, err);
          }
          // warp-uniform outcome, so that the warp leaves together
          if (!__all_sync(0xffffffffu, got)) {
            ok = false;
            break;
          }
          tc_fence_after();
          // 16 rows x 64 (or 32) columns at a time, each loaded while the one
          // before is stored (dense_8 is linear, model.py:377-378)
          const uint32_t fr = sbase + L::kActOff + s * L::kActBytes + frag_row, ta = tlane + (solo ? 256 * (g & 1) : s * 256) + pcol;
          // the operand of the sub-tile's next layer is written (and its
          // accumulator read): one arrival per warp on the even CTA's barrier
          auto operand_done = [&]() {
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive_remote(peer_addr(sbase + L::kBarActr + (solo ? 8 : 8 * s), 0));
              if (STORE) mbar_arrive(sbase + L::kBarTapeRdy + 8 * s);
            }
          };
          // the operand's first half is written (a tile alone)
          auto first_half = [&]() {
            if (solo) {
              fence_proxy_async();
              tc_fence_before();  // (the accumulator of the layer before, that the MMAs will overwrite, is read)
              __syncwarp();
              if (lane == 0) mbar_arrive_remote(peer_addr(sbase + L::kBarActr, 0));
            }
          };
          if (!F8 && g != 7) {
            uint32_t ra[32], rb[32];
            tmem_ld_frag64(ta, ra);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const uint32_t dst = fr + (uint32_t)(2 * c) * kAtom;
              tmem_wait32(ra);
              tmem_ld_frag64(ta + (16u << 16) + 128 * c, rb);
              store_frag64<F8>(dst, cx, 0u, ra, fb, g != 8);
              tmem_wait32(rb);
              if (c == 0) tmem_ld_frag64(ta + 128, ra);
              store_frag64<F8>(dst + 16 * 128, cx, 0u, rb, fb, g != 8);
              if (c == 0) {
                fb[0].load(fbias + 128, fscale + 128, lane & 3);
                fb[1].load(fbias + 160, fscale + 160, lane & 3);
                first_half();
              }
            }
          } else if (g != 7) {  // (E4M3)
            uint32_t ra[16], rb[16];
            tmem_ld_frag32(ta, ra);
#pragma unroll
            for (int c = 0; c < kCols / 32; ++c) {
              tmem_wait16(ra);
              tmem_ld_frag32(ta + (16u << 16) + 32 * c, rb);
              store_frag<F8, false>(fr, cx, 2u * c, ra, fb[c % 2], g != 8);
              tmem_wait16(rb);
              if (c + 1 < kCols / 32) tmem_ld_frag32(ta + 32 * (c + 1), ra);
              store_frag<F8, false>(fr + 16 * 128, cx, 2u * c, rb, fb[c % 2], g != 8);
              if (c + 2 < kCols / 32) fb[c].load(fbias + 32 * (c + 2), fscale + 32 * (c + 2), lane & 3);
            }
          } else {
            // dense_7: the same, and its FP32 ReLU goes back to the
            // accumulator, from where the sigma head (model.py:374-375)
            // reads it a row per lane
            uint32_t ra[16], rb[16];
            tmem_ld_frag32(ta, ra);
#pragma unroll
            for (int c = 0; c < kCols / 32; ++c) {
              auto at = [](int piece) { return F8 ? 32 * piece : 32 * (piece % 2) + 128 * (piece / 2); };
              const uint32_t dst = fr + (F8 ? 0u : (uint32_t)(c / 2) * (2 * kAtom)), ch = F8 ? 2u * c : 4u * (c % 2);
              tmem_wait16(ra);
              tmem_ld_frag32(ta + (16u << 16) + at(c), rb);
              store_frag<F8, true>(dst, cx, ch, ra, fb[c % 2], true);
              tmem_st_frag32(ta + at(c), ra);
              tmem_wait16(rb);
              if (c + 1 < kCols / 32) tmem_ld_frag32(ta + at(c + 1), ra);
              store_frag<F8, true>(dst + 16 * 128, cx, ch, rb, fb[c % 2], true);
              tmem_st_frag32(ta + (16u << 16) + at(c), rb);
              if (c + 2 < kCols / 32) fb[c].load(fbias + at(c + 2), fscale + at(c + 2), lane & 3);
              if (c == 1) first_half();
            }
            if (solo) operand_done();  // before the sums: dense_8 has the other accumulator
            tmem_wait_st();
            // the head's FP32 sums: BF16 of either half's 64 columns, side by side,
            // FP8 one over the part's columns in order
            const uint32_t sw = sbase + L::kHeadW + 4 * pcol;
            float part_sum = 0.0f, second = 0.0f;
            // channel i of the 32 at accumulator column fp8_row (BF16: in place)
            auto add4 = [&](float &sum, const uint32_t(&v)[32], int i, uint32_t w) {
              const float4 w4 = lds_here(w);
              sum = fmaf(__uint_as_float(v[F8 ? fp8_row(7, i) : i]), w4.x, sum);
              sum = fmaf(__uint_as_float(v[F8 ? fp8_row(7, i + 1) : i + 1]), w4.y, sum);
              sum = fmaf(__uint_as_float(v[F8 ? fp8_row(7, i + 2) : i + 2]), w4.z, sum);
              sum = fmaf(__uint_as_float(v[F8 ? fp8_row(7, i + 3) : i + 3]), w4.w, sum);
            };
#pragma unroll 1
            for (int c = 0; c < kCols / 2; c += 32) {
              const int c0 = F8 ? 2 * c : c, c1 = F8 ? 2 * c + 32 : c + 128;
              uint32_t raw[2][32];
              tmem_ld32(ta + c0, raw[0]);
              tmem_ld32(ta + c1, raw[1]);
              tmem_wait32(raw[0]);
              tmem_wait32(raw[1]);
              if (F8) {
#pragma unroll
                for (int i = 0; i < 32; i += 4) add4(part_sum, raw[0], i, sw + 4 * (c0 + i));
#pragma unroll
                for (int i = 0; i < 32; i += 4) add4(part_sum, raw[1], i, sw + 4 * (c1 + i));
              } else {
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                  add4(part_sum, raw[0], i, sw + 4 * (c0 + i));
                  add4(second, raw[1], i, sw + 4 * (c1 + i));
                }
              }
            }
            if (s == 0) {
              sig[0][0] = part_sum;
              sig[0][1] = second;
            } else {
              sig[1][0] = part_sum;
              sig[1][1] = second;
            }
          }
          if (!solo || g != 7) operand_done();
          if (g == 8) {
            // sigma's sums to the side warps, in the last columns of the
            // accumulator, which dense_9 does not write: the second part's own,
            // so the first part's warp waits until they have been read
            if (cq == 0 && !__all_sync(0xffffffffu, wait_bar(sbase + L::kBarRead8 + 8 * s, (uint32_t)(tile & 1),
                                                             abort_flag, err))) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sums = tlane + s * 256 + (F8 ? 254 : 252) + cq;
            tmem_st1(sums, s == 0 ? sig[0][0] : sig[1][0]);
            if (!F8) tmem_st1(sums + 2, s == 0 ? sig[0][1] : sig[1][1]);
            tmem_wait_st();
            tc_fence_before();
            arrive_local(sbase + (cq == 0 ? L::kBarSig : L::kBarRead8) + 8 * s);
          }
        }
        accf_phase ^= 1;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (crank == 1 && warp == 1 && lane == 0 && ntiles > 0) {
    // the even CTA's last commit (after every MMA on this CTA's data) has
    // reached this CTA
    uint64_t t0 = globaltimer();
    while (!mbar_try(sbase + L::kBarDrain, 0) && globaltimer() - t0 < 100000000ull) {
    }
    // Without a timeout every copy of this CTA was waited for by the even
    // CTA's issuer. After one (in either CTA) copies may still be in
    // flight, and they complete on the even CTA's barriers, which this CTA
    // cannot wait on: give them 100 us (copies from L2 take microseconds).
    uint32_t peer_abort;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_abort) : "r"(peer_addr(sbase + L::kAbort, 0))
                 : "memory");
    if (*abort_flag || peer_abort) {
      t0 = globaltimer();
      while (globaltimer() - t0 < 100000ull) {
      }
    }
  }
  __syncwarp();
  cluster_sync_all();  // no MMA or arrival of the pair touches either CTA any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

}  // namespace tc

// cuTensorMapEncodeTiled, looked up once through the runtime (the library
// does not link the driver library).
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(f);
  });
  return fn;
}

int encode_tensor_map_u16(CUtensorMap *map, const void *base, int rank, const unsigned long long *dims,
                          const unsigned long long *strides, const unsigned *box, bool swizzle128) {
  const EncodeTiledFn enc = encode_tiled();
  if (!enc || rank < 1 || rank > 5) return NERFGB_E_CUDA;
  cuuint64_t d[5], st[4];
  cuuint32_t b[5], e[5];
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    b[i] = box[i];
    e[i] = 1;
    if (i > 0) st[i - 1] = strides[i - 1];
  }
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, (cuuint32_t)rank, const_cast<void *>(base), d, st, b, e,
             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? NERFGB_OK
             : NERFGB_E_CUDA;
}

// The pack's weights as a 2-D tensor of 256-byte rows (128 16-bit elements):
// every CTA's half of a chunk starts on a row and is one box.
static int pair_maps(const uint8_t *packed, bool f8, tc::PairMaps &m) {
  const long long bytes = f8 ? kFp8WBytes : kBf16WBytes;
  if (reinterpret_cast<uintptr_t>(packed) % 256 != 0) return NERFGB_E_INVALID_ARG;
  const unsigned long long dims[2] = {128, (unsigned long long)(bytes / 256)};
  const unsigned long long strides[1] = {256};
  const unsigned rows[3] = {64, 32, f8 ? 8u : 16u};
  for (int i = 0; i < 3; ++i) {
    const unsigned box[2] = {128, rows[i]};
    const int rc = encode_tensor_map_u16(&m.map[i], packed, 2, dims, strides, box);
    if (rc != NERFGB_OK) return rc;
  }
  return NERFGB_OK;
}

template <bool F8, bool STORE>
static int launch_variant(const void *packed, const float *xyz, const float *dirs, long long n, int rpd,
                          float *rgb, float *sigma, int *err_word, cudaStream_t stream, const RowMap &rm,
                          uint16_t *tape = nullptr, unsigned long long wait_ns = tc::kWaitNs,
                          long long withhold = -1) {
  constexpr uint32_t smem = tc::Layout<F8>::kSmemBytes;
  static_assert(kBf16WBytes % 256 == 0 && kFp8WBytes % 256 == 0, "pack rows");
  auto kern = tc::mlp_tc_kernel<F8, STORE>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return NERFGB_E_CUDA;
  const int sms = num_sms();
  if (sms <= 0) return NERFGB_E_DEVICE;
  const uint8_t *pk = reinterpret_cast<const uint8_t *>(packed);
  // Cluster pairs; as many as the device co-schedules (one CTA per SM), at
  // most one per 256-row sub-tile.
  const long long subs = (n + tc::kSubRows - 1) / tc::kSubRows;
  if (subs > 0x7fffffffLL) return NERFGB_E_UNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3((unsigned)tc::threads_of(STORE));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // Co-resident pairs of this kernel, per device (asked once per device;
  // concurrent first calls are serialised).
  static std::mutex mu;
  static std::unordered_map<int, int> pairs_of_device;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return NERFGB_E_DEVICE;
  int max_pairs;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto hit = pairs_of_device.find(dev);
    if (hit == pairs_of_device.end()) {
      cfg.gridDim = dim3((unsigned)(sms / 2 * 2));
      int m = 0;
      if (cudaOccupancyMaxActiveClusters(&m, kern, &cfg) != cudaSuccess) return NERFGB_E_CUDA;
      hit = pairs_of_device.emplace(dev, m).first;
    }
    max_pairs = hit->second;
  }
  if (max_pairs < 1) return NERFGB_E_UNSUPPORTED;
  const long long pairs = subs < max_pairs ? (subs > 0 ? subs : 1) : max_pairs;
  cfg.gridDim = dim3((unsigned)(2 * pairs));
  if (pairs < max_pairs && may_overlap(stream, attr[1])) cfg.numAttrs = 2;
  tc::PairMaps maps{};
  int rc = pair_maps(pk, F8, maps);
  if (rc != NERFGB_OK) return rc;
  if constexpr (STORE) {
    // the tape [n][kActsLd] BF16 as 3-D (64 elements, rows, 64-element atoms
    // but for the last half), boxes of 128 rows by 4, 1 and 2 atoms (tc::PairMaps)
    if (reinterpret_cast<uintptr_t>(tape) % 16 != 0) return NERFGB_E_INVALID_ARG;
    static_assert(kActsEncDir % 64 == 0 && kActsLd * 2 % 16 == 0, "tape atoms");
    const unsigned long long dims[3] = {64, (unsigned long long)(n > 0 ? n : 1), kActsLd / 64};
    const unsigned long long strides[2] = {(unsigned long long)kActsLd * 2, 128};
    const unsigned atoms[3] = {4, 1, 2};
    for (int i = 0; i < 3; ++i) {
      const unsigned box[3] = {64, 128, atoms[i]};
      if ((rc = encode_tensor_map_u16(&maps.tape[i], tape, 3, dims, strides, box, true)) != NERFGB_OK) return rc;
    }
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, pk, xyz, dirs, n, rpd, rgb, sigma, err_word, rm, tape, wait_ns,
                                           withhold, maps);
  rc = launch_status();  // (clears a failed launch's error)
  return e == cudaSuccess ? rc : NERFGB_E_CUDA;
}

int launch_mlp_bf16(const void *packed, const float *xyz, const float *dirs, long long n, int rpd, float *rgb,
                    float *sigma, int *err_word, cudaStream_t stream, const RowMap &rm) {
  return launch_variant<false, false>(packed, xyz, dirs, n, rpd, rgb, sigma, err_word, stream, rm);
}

int launch_mlp_bf16_train(const void *packed, const float *xyz, const float *dirs, long long n, int rpd, float *rgb,
                          float *sigma, uint16_t *tape, int *err_word, cudaStream_t stream) {
  // The inference kernel plus the tape stores (the same outputs bit for bit).
  return launch_variant<false, true>(packed, xyz, dirs, n, rpd, rgb, sigma, err_word, stream, RowMap(), tape);
}

int launch_mlp_fp8(const void *packed, const float *xyz, const float *dirs, long long n, int rpd, float *rgb,
                   float *sigma, int *err_word, cudaStream_t stream, const RowMap &rm) {
  return launch_variant<true, false>(packed, xyz, dirs, n, rpd, rgb, sigma, err_word, stream, rm);
}

int launch_mlp_wait_test(const void *packed, bool fp8, const float *xyz, const float *dirs, long long n, int rpd,
                         float *rgb, float *sigma, int *err_word, cudaStream_t stream, unsigned long long wait_ns,
                         long long withhold) {
  // the kernels of launch_mlp_bf16 / launch_mlp_fp8 with the given wait limit and withheld chunk
  if (fp8)
    return launch_variant<true, false>(packed, xyz, dirs, n, rpd, rgb, sigma, err_word, stream, RowMap(), nullptr,
                                       wait_ns, withhold);
  return launch_variant<false, false>(packed, xyz, dirs, n, rpd, rgb, sigma, err_word, stream, RowMap(), nullptr,
                                      wait_ns, withhold);
}

}  // namespace nerfgb

#ifdef NERF_BOUNDS_CHECK
namespace nerfgb {
NG_BOUNDS_READER(bounds_read_mlp_tc)
}  // namespace nerfgb
#endif
