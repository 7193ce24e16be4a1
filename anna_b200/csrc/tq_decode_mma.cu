// Tensor-core split pass of single-token GQA decode over packed TurboQuant pages (16-bit cache dtypes).
//
// A CTA (4 warps) owns one (row, kv head, chunk).  Chunks that cover the un-quantized window ring run the dense
// tensor-core body (dense_mma_body.cuh); chunks over the packed prefix run the path below.  Per warp and 16-token tile:
//
//   packed bytes of the tile --bulk copy (cp.async.bulk, mbarrier)--> shared (2 stages per warp); a tile of a 16-token
//              page is one linear copy issued by one lane, larger pages take six
//   K codes -> 8-bit A fragments in registers, two tokens x D/4 coordinates per lane, no shared-memory round trip:
//              centroids of 4-bit codes through byte-permute (PRMT) table lookups; signs, and the indices of 2- and 3-bit
//              codes, as the bit planes they are made of (a mask leaves one bit in each of four bytes)
//   S1[16 tok x 8 heads] = centroid(K) . Q1^T      S2 = sign(K) . Q2^T        (mma.sync m16n8k32, 8-bit integers)
//   score = norm * (S1 + rnorm * S2)   with Q1 = fwht(s1*q) * scaling / D
//                                           Q2 = fwht(s2*fwht(s1*q)) * scaling * sqrt(pi/2) / D^1.5
//   online softmax in fp32 on the C fragments; P packed to fp16 and transposed with movmatrix
//   V codes -> fp16 (magic-number trick) -> (code * scale + zero) in fp16 pairs -> A fragments of V^T
//   O^T[D x 8 heads] += V^T . P^T                                              (D/16 mma.sync)
//
// The K-dimension slots of the two score products are free to permute, so each lane takes the coordinates whose
// codes it can unpack with the fewest instructions; Q1 / Q2 fragments are gathered with the same permutation.
#include "balanced_schedule.cuh"
#include "dense_mma_body.cuh"
#include "mbarrier_utils.cuh"
#include "tq_common.cuh"
#include "prefill_params.cuh"
#include "tq_decode_params.cuh"

#include <cstdlib>

namespace anna {

__device__ int32_t g_tq_mma_faults;  // bumped when a bounded wait on a tile copy expires

// Byte permute and logic helpers are plain intrinsics / C so that the compiler can fold the constant selectors and
// masks into immediates; the packed fp16 arithmetic goes through PTX on raw registers.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) { return __byte_perm(a, b, sel); }
// Packed fp16 fused multiply-add on raw registers.  (Going through __half2 objects costs a logic operation per call to
// put the two halves back together.)
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;\n" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// A value the compiler cannot see through: `lane` rides along as an unused operand so that the result counts as
// different in every lane and stays in an ordinary register.  (A value known to be the same in all lanes is moved to a
// uniform register when registers are short and copied back, one instruction each time, in front of every use that
// cannot read it from there.)
__device__ __forceinline__ uint32_t pinned_u32(uint32_t value, int lane) {
  uint32_t r;
  asm volatile("{\n .reg .b32 t;\n mov.b32 t, %2;\n mov.b32 %0, %1;\n}\n" : "=r"(r) : "r"(value), "r"(lane));
  return r;
}
// (x & mask) | bits as one three-input logic operation on registers (written out in C with two register constants it
// becomes two instructions).
__device__ __forceinline__ uint32_t and_or_regs(uint32_t x, uint32_t mask, uint32_t bits) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;\n" : "=r"(r) : "r"(x), "r"(mask), "r"(bits));
  return r;
}

// mma.sync m16n8k16 (fp16 in, fp32 accumulate) without the volatile qualifier: a pure function of its operands, so
// the compiler may interleave the independent accumulation chains of this kernel
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// mma.sync m16n8k32 (signed 8-bit in, 32-bit integer accumulate); same C fragment layout as the fp16 shape above
__device__ __forceinline__ void mma_s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same with unsigned A bytes (one bit of a code plane each)
__device__ __forceinline__ void mma_u8s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Byte permute in PTX's default mode: result byte i is the byte of {a (0-3), b (4-7)} that bits 0-2 of nibble i of
// the low half of `sel` name, or, when bit 3 of that nibble is set, eight copies of that byte's top bit.
__device__ __forceinline__ uint32_t prmt_ptx(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;\n" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// N consecutive 32-bit words from shared memory with the widest aligned load (the address is N*4-byte aligned).
template <int N>
__device__ __forceinline__ void lds_words(const uint8_t* ptr, uint32_t (&dst)[N]) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      const uint4 v = reinterpret_cast<const uint4*>(ptr)[i];
      dst[4 * i] = v.x; dst[4 * i + 1] = v.y; dst[4 * i + 2] = v.z; dst[4 * i + 3] = v.w;
    }
  } else if constexpr (N == 2) {
    const uint2 v = *reinterpret_cast<const uint2*>(ptr);
    dst[0] = v.x; dst[1] = v.y;
  } else {
    static_assert(N == 1, "unsupported word count");
    dst[0] = *reinterpret_cast<const uint32_t*>(ptr);
  }
}

// Blocks until the grids this one was launched behind (programmatic stream serialization) have completed and their
// writes are visible; returns at once for a normal launch.  Every CTA of the packed kernel passes through it before
// it exits, so "the packed kernel is done" implies "the window kernel is done" for whatever comes next in the stream.
__device__ __forceinline__ void wait_for_prior_grids() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Larger of two values, NaN if either is: a NaN query must reach the scores although its bytes cannot hold it.
__device__ __forceinline__ float fmax_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;\n" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

#ifndef ANNA_TQ_CTAS128
#define ANNA_TQ_CTAS128 4
#endif
#ifndef ANNA_TQ_CTAS256
#define ANNA_TQ_CTAS256 3
#endif
#ifndef ANNA_TQ_TILES_PER_STEP
#define ANNA_TQ_TILES_PER_STEP 2
#endif
#ifndef ANNA_TQ_RING_TILES
#define ANNA_TQ_RING_TILES 4
#endif
constexpr float kLazyRescale = 8.0f;  // log2 units: probabilities stay below 2^8, well inside fp16

// Ring stage that is still free once the copies of `stages` - 1 steps have been started from stage `first` on.
constexpr __host__ __device__ int ring_free_stage(int first, int stages) { return (first + stages - 1) % stages; }
constexpr bool ring_free_stage_is_free(int stages) {
  for (int first = 0; first < stages; ++first)
    for (int i = 0; i < stages - 1; ++i)
      if ((first + i) % stages == ring_free_stage(first, stages)) return false;
  return true;
}
static_assert(ring_free_stage_is_free(2) && ring_free_stage_is_free(3) && ring_free_stage_is_free(4),
              "the rotated queries may not lie where copies are in flight");

template <typename T, int D, int BITS>
struct TqMmaCfg {
  static constexpr int kSteps = D / 16;
  // Keys are scored as 8-bit integers against rotated queries that are split into a coarse and a fine byte.  4-bit
  // codes: one byte permute turns four codes into four centroid bytes, a mask leaves four signs.  2- and 3-bit
  // codes: their centroids are linear in the code's bits (+-c0; +-c0 and +-c1 by symmetry), so each bit plane is
  // multiplied by the query bytes as it is -- a mask leaves one bit in each of four bytes, which is four coordinates of
  // a fragment for one logic operation -- and the planes are weighted with the exact centroids afterwards.  Against the
  // fp16 fragments of +-1 (a shift and a logic operation per two coordinates) and 11-bit queries this was: 64 ragged rows
  // of 4-32 K tokens, 2 bits, head_dim 256: 247 -> 212 us; 128 rows of 0.5-16 K, 3 bits, head_dim 128: 261 -> 253 us.
  static constexpr bool kPlanes = BITS != 4;
  static constexpr int kSteps8 = D / 32;                       // k-steps of the 8-bit score products
  // query fragments of one unit, then a second array: the fine bytes of Q1 (4-bit codes) or all of Q2 (planes)
  static constexpr int kFragBytes = 32 * kSteps8 * 16;
  static constexpr int kFrag2Bytes = 32 * kSteps8 * (kPlanes ? 16 : 8);
  static constexpr int kConstOffset = kFragBytes + kFrag2Bytes;  // per-head factors behind them: [6][8] floats
  static constexpr int kGroups = D / 32;                       // value group size is 32 on this path
  static constexpr int kKeyBytes = D * BITS / 8;               // packed key bytes per token
  static constexpr int kIdxBytes = BITS == 3 ? D / 4 : kKeyBytes;  // first plane (all of it unless BITS == 3)
  static constexpr int kSignBytes = BITS == 3 ? D / 8 : 0;     // separate sign plane of the 3-bit format
  static constexpr int kValBytes = D / (BITS == 2 ? 4 : 2);
  // stage layout (bytes): the layout of a 16-token chunk, so a tile of a 16-token page is one linear copy
  static constexpr int kOffKey = 0;
  static constexpr int kOffNorm = 16 * kKeyBytes;
  static constexpr int kOffRnorm = kOffNorm + 64;
  static constexpr int kOffVal = kOffRnorm + 64;
  static constexpr int kOffScale = kOffVal + 16 * kValBytes;
  static constexpr int kOffZero = kOffScale + 16 * kGroups * 2;
  static constexpr int kStageBytes = (kOffZero + 16 * kGroups * 2 + 127) / 128 * 128;
  static constexpr int kTilesPerStep = ANNA_TQ_TILES_PER_STEP;  // 16-token tiles a warp scores together (one softmax update)
  static constexpr int kStages = ANNA_TQ_RING_TILES / kTilesPerStep;  // steps per warp ring; kStages - 1 are in flight
  static constexpr int kMinBlocks = D >= 256 ? ANNA_TQ_CTAS256 : ANNA_TQ_CTAS128;
  static constexpr int kWarpSmem = kStages * kTilesPerStep * kStageBytes;
  static constexpr int kPackedSmem = kMmaWarps * kWarpSmem;
  static constexpr int kMergeSmem = (2 * kMmaWarps * 8 + kMmaWarps * 8 * (D + 4)) * 4;
  static constexpr int kTailSmem = 8 * kFusedMaxChunks * 4;
  static constexpr int kSmemBytes0 = kPackedSmem > kMergeSmem ? kPackedSmem : kMergeSmem;
  static constexpr int kWorkSmem = ((kSmemBytes0 > kTailSmem ? kSmemBytes0 : kTailSmem) + 15) / 16 * 16;
  // behind the working area (which the epilogue reuses): one mbarrier per warp and stage, one valid-token count per tile
  static constexpr int kBarrierBytes = kMmaWarps * kStages * 8;
  static constexpr int kQueryOffset = (kWorkSmem + kBarrierBytes + kMmaWarps * kStages * kTilesPerStep * 4 + 15) / 16 * 16;
  // the query fragments of the CTA live in shared memory (two loads per k-step and step) instead of registers
  static constexpr int kSmemBytes = kQueryOffset + kConstOffset + 6 * 8 * 4;
  // While they are made, the rotated queries (two vectors of two heads per warp) lie in the ring stage that the warp's
  // first copies leave free: with room of their own, four CTAs fill the shared memory and leave the L1 cache nothing.
  // A vector's quarters are 4 floats further apart than their length and odd heads start 16 floats in, so that the eight
  // lanes that load together (two heads x four quarters) find their 16 bytes in different banks.
  static constexpr int kRotFloats = D + 32;
  static_assert(kStages >= 2 && kTilesPerStep * kStageBytes >= 2 * 2 * kRotFloats * 4, "the rotated queries need a free stage");
  // bytes of one 16-token tile in the stage (= in a 16-token page chunk, padding excluded)
  static constexpr int kTileDataBytes = kOffZero + 16 * kGroups * 2;
  // per-lane key code words per token (this lane's D/4 coordinates)
  static constexpr int kIdxWords = BITS == 4 ? D / 32 : D / 64;
  static constexpr int kSignWords = BITS == 3 ? D / 128 : 0;
  static constexpr int kValWords = BITS == 2 ? D / 128 : D / 64;  // per token, this lane's D/8 dims
  static_assert(D == 128 || D == 256, "tensor-core TurboQuant decode is built for head_dim 128 and 256");
};

// Bit planes of 2- and 3-bit codes.  A lane holds the codes of its D/4 coordinates (tig * D/4 ...) of a token as words:
// 16 two-bit fields (2-bit codes; the indices of 3-bit codes) or 32 sign bits (3-bit codes).  Shifted left so that the
// wanted bits sit at the top of each byte, one mask leaves the bits of the four fields / signs that share a position
// inside their byte: byte i of register r (0: k 4tig.., 1: k 16 + 4tig..) of k-step s is
//   fields: coordinate 16 * (2 * (s % kPairs) + r) + 4i + s / kPairs of the lane's run, kPairs = D/128 word pairs
//   signs:  coordinate 32 * (s / 4) + 8i + 2 * (s % 4) + r

// What the query preparation needs besides the queries: the same for every segment of a CTA.
struct TqQueryConsts {
  bool loaded;
  uint32_t flips;    // bit j: coordinate lane * E + j is negated by the first rotation (low byte) / by the second
  uint32_t lut[2];   // 4-bit: the centroids as signed bytes
  float cent_step;   // 4-bit: the value of one step of those bytes
};

// The constants as they are in memory, so that a kernel can read them beside what else it starts with.
template <int D, int BITS>
struct TqRawConsts {
  float s1[D / 32], s2[D / 32], cent[BITS == 4 ? 8 : 1];
  __device__ __forceinline__ void load(const TqDecodeParams& p) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < D / 32; ++j) {
      s1[j] = __ldg(p.signs1 + lane * (D / 32) + j);
      s2[j] = __ldg(p.signs2 + lane * (D / 32) + j);
    }
    if constexpr (BITS == 4) {
#pragma unroll
      for (int e = 0; e < 8; ++e) cent[e] = __ldg(p.centroids + e);
    }
  }
};

template <int D, int BITS>
__device__ __forceinline__ TqQueryConsts load_query_consts(const TqRawConsts<D, BITS>& raw) {
  constexpr int E = D / 32;
  constexpr int kEntries = 1 << (BITS - 1);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  TqQueryConsts qc{true, 0u, {0u, 0u}, 0.0f};
#pragma unroll
  for (int j = 0; j < E; ++j) {
    qc.flips |= (raw.s1[j] < 0.0f ? 1u : 0u) << j;
    qc.flips |= (raw.s2[j] < 0.0f ? 1u : 0u) << (8 + j);
  }
  if constexpr (BITS == 4) {
    // The byte scale of the centroids is the one, among 256 candidates from 127 down to 63 steps for the largest
    // centroid, that leaves the smallest squared rounding error over the codebook.
    __shared__ float best_err_of[kMmaWarps], best_k_of[kMmaWarps];
    float cent[kEntries], cmax = 0.0f;
#pragma unroll
    for (int e = 0; e < kEntries; ++e) {
      cent[e] = raw.cent[e];
      cmax = fmaxf(cmax, fabsf(cent[e]));
    }
    float best_err = INFINITY, best_k = 0.0f;
    if (cmax > 0.0f) {
      for (int j = threadIdx.x; j < 256; j += kMmaThreads) {
        const float k = (127.0f - 0.25f * (float)j) / cmax;
        float err = 0.0f;
#pragma unroll
        for (int e = 0; e < kEntries; ++e) {
          const float d = cent[e] * k - rintf(cent[e] * k);
          err = fmaf(d, d, err);
        }
        err /= k * k;
        if (err < best_err) { best_err = err; best_k = k; }
      }
    }
    auto take = [&](float other_err, float other_k) {
      if (other_err < best_err || (other_err == best_err && other_k > best_k)) { best_err = other_err; best_k = other_k; }
    };
#pragma unroll
    for (int dl = 1; dl < 32; dl <<= 1) {
      const float other_err = __shfl_xor_sync(0xffffffffu, best_err, dl);
      const float other_k = __shfl_xor_sync(0xffffffffu, best_k, dl);
      take(other_err, other_k);
    }
    if (lane == 0) { best_err_of[warp] = best_err; best_k_of[warp] = best_k; }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kMmaWarps; ++w) take(best_err_of[w], best_k_of[w]);
#pragma unroll
    for (int e = 0; e < kEntries; ++e)
      qc.lut[e / 4] |= ((uint32_t)__float2int_rn(cent[e] * best_k) & 0xffu) << (8 * (e % 4));
    qc.lut[0] = pinned_u32(qc.lut[0], lane);
    qc.lut[1] = pinned_u32(qc.lut[1], lane);
    qc.cent_step = best_k > 0.0f ? 1.0f / best_k : 0.0f;
  }
  return qc;
}

template <typename T>
__device__ __forceinline__ T elem_of_bits(unsigned short bits);
template <>
__device__ __forceinline__ __half elem_of_bits<__half>(unsigned short bits) { return __ushort_as_half(bits); }
template <>
__device__ __forceinline__ __nv_bfloat16 elem_of_bits<__nv_bfloat16>(unsigned short bits) { return __ushort_as_bfloat16(bits); }

// This lane's elements (lane * D/32 ...) of the query heads warp and warp + 4, as loaded (rows start on 4-byte boundaries).
template <typename T, int D>
struct TqRawQueries {
  uint32_t w[2][D / 64];
  __device__ __forceinline__ void load(const TqDecodeParams& p, int b, int hq0, int g_count) {
    const T* q = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride_b + (threadIdx.x & 31) * (D / 32);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int g = (int)(threadIdx.x >> 5) + k * kMmaWarps;
      const uint32_t* row = reinterpret_cast<const uint32_t*>(q + (int64_t)(hq0 + g) * p.q_stride_h);
#pragma unroll
      for (int j = 0; j < D / 64; ++j) w[k][j] = g < g_count ? row[j] : 0u;
    }
  }
};

// Rotates the queries of one (row, kv-head group), rounds them to a coarse and a fine byte and leaves them at `query` in
// shared memory as the B fragments of m16n8k32 in the register order of the score products, with the per-head factors
// behind them (offsets of TqMmaCfg).  Every CTA does this for itself, once per segment, while its first tiles are on
// their way: 2-3 us of a CTA, against 5-14 us of a kernel in front of the whole call (which read the rotated vectors with
// 32 lanes in one bank): one row of 4 K tokens 35 -> 27 us, 16 rows of 0.4-4 K at head_dim 256 74 -> 60 us, 128 rows of
// 0.5-16 K 253 -> 247 us, 64 rows of 32 K 630 -> 636 us.  The caller synchronises afterwards.
template <typename T, int D, int BITS>
__device__ __forceinline__ void prepare_query_fragments(const TqDecodeParams& p, uint8_t* smem_raw, uint8_t* query,
                                                        int free_stage, const TqRawQueries<T, D>& raw, int g_count,
                                                        const TqQueryConsts& qc) {
  using Cfg = TqMmaCfg<T, D, BITS>;
  constexpr int E = D / 32;
  constexpr int kSteps8 = Cfg::kSteps8;
  __shared__ float q_scale[2][8];    // 127 / largest coordinate
  __shared__ int rot_at[kMmaWarps];  // where the heads g, g + 4 of warp g are: the free stage differs from warp to warp
  float* consts = reinterpret_cast<float*>(query + Cfg::kConstOffset);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (lane == 0) rot_at[warp] = warp * Cfg::kWarpSmem + free_stage * Cfg::kTilesPerStep * Cfg::kStageBytes;
  __syncwarp();
  // quarter `tig` of rotation `which` of head g
  auto rotated = [&](int which, int g, int tig) {
    return reinterpret_cast<float*>(smem_raw + rot_at[g % kMmaWarps]) + (2 * (g / kMmaWarps) + which) * Cfg::kRotFloats +
           16 * (g & 1) + tig * (D / 4 + 4);
  };
  // heads that do not exist: scale and factors zero, which makes bytes of zero of whatever their vectors hold
  if (threadIdx.x < 8 && (int)threadIdx.x >= g_count) {
    q_scale[0][threadIdx.x] = q_scale[1][threadIdx.x] = 0.0f;
#pragma unroll
    for (int i = 0; i < 6; ++i) consts[8 * i + threadIdx.x] = 0.0f;
  }
  auto coarse = [](float v, float k) { return max(-127, min(127, __float2int_rn(v * k))); };
  auto fine = [](float v, float k, int c) { return max(-127, min(127, __float2int_rn((v * k - (float)c) * 254.0f))); };
  const uint32_t flips = qc.flips;
  // score (log2 units) = norm * (S1 + rnorm * S2) with every constant folded into the factors:
  //   q.k_hat = norm/D * [Q1.c + sqrt(pi/2)/sqrt(D) * rnorm * Q2.sign],  Q1 = fwht(s1*q), Q2 = fwht(s2*Q1)
  const float inv_sqrt_d = rsqrt_dim_const<D>();
  const float log2e = 1.4426950408889634f;
  const float f1 = p.scaling * log2e * inv_sqrt_d * inv_sqrt_d;
  const float f2 = p.scaling * log2e * 1.2533141373155001f * inv_sqrt_d * inv_sqrt_d * inv_sqrt_d;
  for (int k = 0; k < 2; ++k) {
    const int g = warp + k * kMmaWarps;
    if (g >= g_count) break;
    float w[E], w1[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const uint32_t word = k == 0 ? raw.w[0][j / 2] : raw.w[1][j / 2];
      w[j] = ElemTraits<T>::to_float(elem_of_bits<T>((unsigned short)(j % 2 == 0 ? word : word >> 16)));
      if ((flips >> j) & 1u) w[j] = -w[j];
    }
    warp_fwht<E>(w, lane);
    float amax1 = 0.0f, amax2 = 0.0f;
#pragma unroll
    for (int j = 0; j < E; ++j) {
      w1[j] = w[j];
      rotated(0, g, lane / 8)[lane % 8 * E + j] = w[j];
      amax1 = fmax_nan(amax1, fabsf(w[j]));
      if ((flips >> (8 + j)) & 1u) w[j] = -w[j];
    }
    warp_fwht<E>(w, lane);
#pragma unroll
    for (int j = 0; j < E; ++j) {
      rotated(1, g, lane / 8)[lane % 8 * E + j] = w[j];
      amax2 = fmax_nan(amax2, fabsf(w[j]));
    }
    // as integers, non-negative floats keep their order and a NaN is above all of them
    amax1 = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax1)));
    amax2 = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax2)));
    const float k1 = amax1 > 0.0f ? 127.0f / amax1 : 0.0f, k2 = amax2 > 0.0f ? 127.0f / amax2 : 0.0f;
    int total1 = 0, total2 = 0;
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const int c2 = coarse(w[j], k2);
      if constexpr (Cfg::kPlanes) {
        const int c1 = coarse(w1[j], k1);
        total1 += 254 * c1 + fine(w1[j], k1, c1);
        total2 += 254 * c2 + fine(w[j], k2, c2);
      } else {
        total2 += c2;
      }
    }
    if constexpr (Cfg::kPlanes) total1 = __reduce_add_sync(0xffffffffu, total1);
    total2 = __reduce_add_sync(0xffffffffu, total2);
    if (lane == 0) {
      q_scale[0][g] = k1;
      q_scale[1][g] = k2;
      if constexpr (Cfg::kPlanes) {
        // With u = the value of one step of the fine byte and Q the 254 * coarse + fine integers: a plane with its bits
        // at weight 2^j of a byte gives T = 2^j * sum over set bits of Q.
        //   sign plane (+1 set, -1 clear, weight 128):  S2 = T * 2u / 128 - u * sum(Q)
        //   index planes: centroid = z0 + z1 * bit0 + z2 * bit1 (+ z3 * bit0 * bit1, zero for the symmetric codebooks):
        //   S1 = T0 * z1 * u / 64 (+ T1 * z2 * u / 128 + T01 * z3 * u / 64) + z0 * u * sum(Q)
        // [0] factor of bit plane 0, [1] of bit plane 1, [2] of both, [3] constant of S1, [4] factor, [5] constant of S2
        const float u1 = amax1 * f1 / (127.0f * 254.0f), u2 = amax2 * f2 / (127.0f * 254.0f);
        const float* cent = p.centroids;
        const float z1 = __ldg(cent + 1) - __ldg(cent);
        consts[g] = z1 * u1 / 64.0f;
        if constexpr (BITS == 3) {
          consts[8 + g] = (__ldg(cent + 2) - __ldg(cent)) * u1 / 128.0f;
          consts[16 + g] = ((__ldg(cent + 3) - __ldg(cent + 2)) - z1) * u1 / 64.0f;
        }
        consts[24 + g] = __ldg(cent) * u1 * (float)total1;
        consts[32 + g] = u2 / 64.0f;
        consts[40 + g] = -u2 * (float)total2;
      } else {
        // factor of the centroid product; factor and constant of the sign product: the sign plane has its bits at weight
        // 128, and twice the sum over set bits minus the sum over all coordinates is the +-1 product
        consts[g] = amax1 * f1 / (127.0f * 254.0f) * qc.cent_step;
        consts[32 + g] = amax2 * f2 / (127.0f * 64.0f);
        consts[40 + g] = -(amax2 * f2 / 127.0f) * (float)total2;
      }
    }
  }
  __syncthreads();
  const int gid = lane >> 2, tig = lane & 3;
  if constexpr (Cfg::kPlanes) {
    // [s][lane][Q1 coarse b0, b1, Q1 fine b0, b1]   then   [s][lane][Q2 coarse b0, b1, Q2 fine b0, b1]: a warp makes one
    // register of one rotation
    const int which = warp >> 1, r = warp & 1;
    const float k = q_scale[which][gid];
    const float* v = rotated(which, gid, tig);
    uint32_t* out = reinterpret_cast<uint32_t*>(query) + which * 32 * kSteps8 * 4 + lane * 4 + r;
    auto put = [&](int s, float v0, float v1, float v2, float v3) {
      const float x[4] = {v0, v1, v2, v3};
      uint32_t hi = 0u, lo = 0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = coarse(x[i], k);
        hi |= ((uint32_t)c & 0xffu) << (8 * i);
        lo |= ((uint32_t)fine(x[i], k, c) & 0xffu) << (8 * i);
      }
      out[s * 128] = hi;
      out[s * 128 + 2] = lo;
    };
    auto four = [&](int d) { return *reinterpret_cast<const float4*>(v + d); };
    if (BITS == 3 && which == 1) {
      // sign plane: k-step s takes, of each group of 8 coordinates of word s / 4, number 2 * (s % 4) + r
#pragma unroll
      for (int w = 0; w < D / 128; ++w) {
        float4 a[4], b4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          a[i] = four(32 * w + 8 * i);
          b4[i] = four(32 * w + 8 * i + 4);
        }
        if (r == 0) {
          put(4 * w + 0, a[0].x, a[1].x, a[2].x, a[3].x);
          put(4 * w + 1, a[0].z, a[1].z, a[2].z, a[3].z);
          put(4 * w + 2, b4[0].x, b4[1].x, b4[2].x, b4[3].x);
          put(4 * w + 3, b4[0].z, b4[1].z, b4[2].z, b4[3].z);
        } else {
          put(4 * w + 0, a[0].y, a[1].y, a[2].y, a[3].y);
          put(4 * w + 1, a[0].w, a[1].w, a[2].w, a[3].w);
          put(4 * w + 2, b4[0].y, b4[1].y, b4[2].y, b4[3].y);
          put(4 * w + 3, b4[0].w, b4[1].w, b4[2].w, b4[3].w);
        }
      }
    } else {
      // fields: k-step s takes, of each group of 4 coordinates of word 2 * (s % kPairs) + r, number s / kPairs
      constexpr int kPairs = D / 128;
#pragma unroll
      for (int pair = 0; pair < kPairs; ++pair) {
        float4 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = four(16 * (2 * pair + r) + 4 * i);
        put(0 * kPairs + pair, a[0].x, a[1].x, a[2].x, a[3].x);
        put(1 * kPairs + pair, a[0].y, a[1].y, a[2].y, a[3].y);
        put(2 * kPairs + pair, a[0].z, a[1].z, a[2].z, a[3].z);
        put(3 * kPairs + pair, a[0].w, a[1].w, a[2].w, a[3].w);
      }
    }
  } else {
    // lane (gid, tig) feeds head gid with the coordinates of its code word s, tig * D/4 + 8s + {0..3} in the first
    // register and + {4..7} in the second; for the sign product, which uses a coarse byte only, + {0, 2, 4, 6} and
    // + {1, 3, 5, 7} (the low and the high nibbles of the word's bytes)
    //   [s][lane][Q1 coarse b0, b1, Q2 coarse b0, b1]   then   [s][lane][Q1 fine b0, b1]
    const float k1 = q_scale[0][gid], k2 = q_scale[1][gid];
#pragma unroll
    for (int s = warp; s < kSteps8; s += kMmaWarps) {
      float r1[8], r2[8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        *reinterpret_cast<float4*>(r1 + 4 * h) = *reinterpret_cast<const float4*>(rotated(0, gid, tig) + 8 * s + 4 * h);
        *reinterpret_cast<float4*>(r2 + 4 * h) = *reinterpret_cast<const float4*>(rotated(1, gid, tig) + 8 * s + 4 * h);
      }
      uint32_t w[4] = {0u, 0u, 0u, 0u}, wl[2] = {0u, 0u};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c0 = coarse(r1[i], k1), c1 = coarse(r1[4 + i], k1);
        w[0] |= ((uint32_t)c0 & 0xffu) << (8 * i);
        w[1] |= ((uint32_t)c1 & 0xffu) << (8 * i);
        wl[0] |= ((uint32_t)fine(r1[i], k1, c0) & 0xffu) << (8 * i);
        wl[1] |= ((uint32_t)fine(r1[4 + i], k1, c1) & 0xffu) << (8 * i);
        w[2] |= ((uint32_t)coarse(r2[2 * i], k2) & 0xffu) << (8 * i);
        w[3] |= ((uint32_t)coarse(r2[2 * i + 1], k2) & 0xffu) << (8 * i);
      }
      reinterpret_cast<uint4*>(query)[s * 32 + lane] = make_uint4(w[0], w[1], w[2], w[3]);
      reinterpret_cast<uint2*>(query + Cfg::kFragBytes)[s * 32 + lane] = make_uint2(wl[0], wl[1]);
    }
  }
}

// Lengths of one row: keys, quantized ones among them, and the chunks of the fixed-chunk division that hold any.
struct RowChunks {
  int len, quantized, window, packed;
};
__device__ __forceinline__ RowChunks row_chunks(const TqDecodeParams& p, int b) {
  RowChunks r;
  r.len = (int)max((int64_t)0, min(p.lengths[b], p.max_len));
  r.quantized = r.len > p.residual_len ? r.len - p.residual_len : 0;
  r.window = (r.len - r.quantized + p.chunk_tokens - 1) / p.chunk_tokens;
  r.packed = (r.quantized + p.chunk_tokens - 1) / p.chunk_tokens;
  return r;
}

// Chunk `slot` of the un-quantized window ring of a row: the dense tensor-core body with ring addressing.  Also writes the
// zero output of empty rows.  `arrives`: the chunk counts on the merge counter, as one of all active chunks.
template <typename T, int D, int STAGES, int HEADS, bool AHEAD>
__device__ __forceinline__ void tq_window_chunk(const TqDecodeParams& p, uint8_t* smem_raw, const RowChunks& row, int b,
                                                int unit, int units, int slot, bool arrives) {
  const int group_tiles = (p.groups + 7) / 8;
  const int kvh = unit / group_tiles;
  const int g0 = (unit % group_tiles) * 8;
  const int g_count = min(8, p.groups - g0);
  if (row.len == 0) {
    if (p.fused.counters != nullptr && slot == 0)
      fused_write_zero_row<T, D, kMmaThreads>(p.fused, b, kvh * p.groups + g0, g_count);
    return;
  }
  if (slot >= row.window) return;
  const int R = p.residual_len;
  DenseDecodeParams dp{};
  dp.q = p.q; dp.q_stride_b = p.q_stride_b; dp.q_stride_h = p.q_stride_h;
  const int64_t ring_elems = (int64_t)R * D;
  const int64_t slot_base = p.window_slots[b] * 2 * p.kv_heads * ring_elems;
  dp.key = reinterpret_cast<const T*>(p.window) + slot_base;
  dp.value = reinterpret_cast<const T*>(p.window) + slot_base + (int64_t)p.kv_heads * ring_elems;
  dp.page_table = nullptr;
  dp.kv_stride_b = 0; dp.kv_stride_h = ring_elems; dp.kv_stride_t = D;
  dp.ring_len = R;
  dp.block_size = 1; dp.block_shift = 0;
  dp.stats = p.stats; dp.values = p.values;
  dp.q_heads = p.q_heads; dp.kv_heads = p.kv_heads; dp.groups = p.groups;
  dp.chunk_tokens = p.chunk_tokens; dp.num_chunks = p.num_chunks; dp.chunk_capacity = p.chunk_capacity;
  dp.scaling = p.scaling;
  dp.fused = p.fused;
  if (!arrives) dp.fused.counters = nullptr;
  const int t0 = row.quantized + slot * p.chunk_tokens;
  const int t1 = min(row.len, t0 + p.chunk_tokens);
  dense_split_mma_body<T, D, STAGES, HEADS, MergeLoads::kAllColumns, AHEAD>(dp, smem_raw, b, kvh, g0, g_count, t0, t1, slot, row.window + row.packed,
                                     (int64_t)b * units + unit);
}

// Window chunks of every row, grid (num_window_chunks, kv_heads * group tiles, batch).
template <typename T, int D>
__global__ void __launch_bounds__(kMmaThreads, MmaCfg<D>::kMinBlocks) tq_window_split_mma_kernel(const TqDecodeParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // The packed-chunk kernel that follows in the stream reads nothing this kernel writes before the arrival counters
  // say so, and each of its CTAs waits for this grid to complete before it counts itself in or exits, so it may start
  // as soon as every CTA here has been scheduled.
  asm volatile("griddepcontrol.launch_dependents;\n" ::);
  const RowChunks row = row_chunks(p, blockIdx.z);
  // the packed CTAs wait for this grid before they count
  tq_window_chunk<T, D, 2, 8, false>(p, smem_raw, row, blockIdx.z, blockIdx.y, gridDim.y, blockIdx.x,
                           p.window_arrives || row.quantized == 0);
}

// Copy ring of one warp of a packed-prefix CTA; it runs on from one segment to the next.
struct PackedRing {
  int stage;       // stage of the next step
  uint32_t phase;  // parity of the mbarrier phase that step completes
  bool dead;       // a bounded wait expired: this warp consumes nothing any more
};

// Query heads that the merge provides for.  (At head_dim 128 four heads have one column per thread, and the loop for two, which
// they never reach, stays: without it the 4-bit even-share kernel took 1.6 to 3.4 % longer.)
template <int D, bool kPair>
constexpr int kMergeHeads = kPair && D == 256 ? 4 : 8;

// EARLY: what a segment starts with (pages, queries, constants) is read side by side, and the constants are worked out while the first
// copies are on their way.  Kernels of many CTAs per SM, whose latencies others fill, keep the registers instead (64 rows of 32 K,
// 32/8 heads, in chunks: 583 us, 587 with it).  AHEAD: see fused_combine_ahead.  In the other two launches the longer code and its
// registers cost some instances more than the order gains, so each has what measured best: GPU times against neither of the two, means
// over 160-170 shapes per instance (1 to 128 rows of 30 tokens to 32 K, 1 to 12 query heads per KV head).
template <int D, int BITS, bool kPair>
struct TqSmallOrder {
  // AHEAD alone and both.  Head_dim 128, 4 bits: pairs 0.945 and 0.942 (one row of 4000 tokens, 32/8 heads, 11.5 us and 11.7, neither
  // 11.8), eight heads 0.896 and 0.913; 2 bits: pairs 0.946 and 0.951, eight heads 0.907 and 0.906; 3 bits: 0.945 and 0.927, 0.924 and
  // 0.926.  Head_dim 256, by bits: pairs 1.007, 1.020, 0.967 and 0.993, 0.995, 0.971 (four heads in 2 and 3 bits 1.004 and 1.014 with
  // both; neither there was no faster than that over other shapes), eight heads 0.963, 0.973, 0.976 and 0.967, 0.954, 0.980.
  static constexpr bool kEarly = D == 256 || BITS == 3 || (BITS == 2 && !kPair);
};
// Even shares have both (0.94-0.98) but for 4-bit pairs, which are the slower for it in short shares.
template <int D, int BITS, bool kPair>
constexpr bool kShareOrders = BITS == 4 && kPair;
template <int D, int BITS, bool kPair, bool kShort>
struct TqShareOrder {
  // head_dim 128: EARLY has no registers for AHEAD
  static constexpr bool kEarly = !(kShareOrders<D, BITS, kPair> && kShort);
  static constexpr bool kAhead = !kShareOrders<D, BITS, kPair> || kShort == (D == 128);
};

constexpr int32_t kPageNotAsked = INT32_MIN;

// Page of the tile that this lane copies in a warp's first step of a segment that starts at token t0, for kernels that know t0 before
// the row's length: the block table is read beside the length instead of behind it.  Lanes without a tile do not ask.
template <typename T, int D, int BITS>
__device__ __forceinline__ int32_t first_page_of(const TqDecodeParams& p, int b, int t0) {
  constexpr int U = TqMmaCfg<T, D, BITS>::kTilesPerStep;
  const int lane = threadIdx.x & 31;
  if (lane >= U) return kPageNotAsked;
  const uint32_t ts = (uint32_t)(t0 + ((int)(threadIdx.x >> 5) * U + lane) * kTileTokens);
  const uint32_t blk = p.block_shift >= 0 ? ts >> p.block_shift : ts / (uint32_t)p.block_size;
  return (int64_t)blk < p.max_blocks ? p.block_table[(int64_t)b * p.table_stride + blk] : kPageNotAsked;
}

// One packed segment: tokens [t0, t1) of the quantized prefix of (row b, unit = kv head and group of 8 query heads).  The
// partial goes to split-K slot `out_slot` and counts as one of `arrivals`; the CTA that counts last merges `slots` partials.
// All threads of the CTA call it; it ends with the CTA synchronised against reuse of the ring.
//
// kPair (at most 4 query heads): the eight columns of the products are 4 heads x the two tiles of a step.  The query
// operand of a tile is zero in the other tile's columns, so both tiles add into one set of accumulators, and the score
// arithmetic, the softmax and the registers behind it are spent once per two tiles instead of once per tile with half of
// the columns empty; columns j and j + 4 are two partials of head j, merged with those of the other warps.  64 rows of
// 32 K tokens, 4 bits: 636 -> 614 us; 128 rows of 0.5-16 K, 3 bits: 247 -> 239 us.
template <typename T, int D, int BITS, bool kPair, MergeLoads MERGE = MergeLoads::kAllColumns, bool EARLY = false, bool AHEAD = EARLY>
__device__ __forceinline__ void tq_packed_segment(const TqDecodeParams& p, uint8_t* smem_raw,
                                                  TqQueryConsts& qc, PackedRing& ring, int b, int unit,
                                                  int units, int t0, int t1, int out_slot, int slots, int arrivals,
                                                  int32_t first_page = kPageNotAsked,
                                                  TqRawConsts<D, BITS>* consts = nullptr) {
  using Cfg = TqMmaCfg<T, D, BITS>;
  constexpr int U = Cfg::kTilesPerStep;
  constexpr int A = kPair ? 1 : U;  // sets of score accumulators
  static_assert(!kPair || U == 2, "a pair is the two tiles of a step");
  const int group_tiles = (p.groups + 7) / 8;
  const int kvh = unit / group_tiles;
  const int g0 = (unit % group_tiles) * 8;
  const int g_count = min(8, p.groups - g0);
  const int hq0 = kvh * p.groups + g0;
  const int num_tiles = (t1 - t0 + kTileTokens - 1) / kTileTokens;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int gid = lane >> 2;
  const int tig = lane & 3;
  // loop constants held in registers
  // (only the ones this instantiation uses are created)
  const uint32_t nib_mask = BITS != 2 ? pinned_u32(0x03C003C0u, lane) : 0u;    // 4-bit value codes
  const uint32_t magic16 = BITS != 2 ? pinned_u32(0x4C004C00u, lane) : 0u;
  const uint32_t kIdxMask = BITS == 4 ? pinned_u32(0x77777777u, lane) : 0u;    // 4-bit key codes
  const uint32_t kTop = pinned_u32(0x80808080u, lane);                         // bit planes of key codes
  const uint32_t kNext = BITS != 4 ? pinned_u32(0x40404040u, lane) : 0u;
  const uint32_t kTwoBitMask = BITS == 2 ? pinned_u32(0x03000300u, lane) : 0u;  // 2-bit value codes
  const uint32_t kMagic4 = BITS == 2 ? pinned_u32(0x44004400u, lane) : 0u;
  (void)nib_mask; (void)magic16; (void)kIdxMask; (void)kTop; (void)kNext; (void)kTwoBitMask;
  (void)kMagic4;

  const uint32_t warp_smem_u32 = smem_u32(smem_raw + warp * Cfg::kWarpSmem);
  const uint8_t* warp_smem = smem_raw + warp * Cfg::kWarpSmem;
  const int32_t* table_row = p.block_table + (int64_t)b * p.table_stride;
  const uint32_t block_size = (uint32_t)p.block_size;
  const int block_shift = p.block_shift;
  const uint32_t bars_u32 = smem_u32(smem_raw + Cfg::kWorkSmem) + warp * Cfg::kStages * 8;
  volatile int* stage_valid = reinterpret_cast<volatile int*>(smem_raw + Cfg::kWorkSmem + Cfg::kBarrierBytes) +
                              warp * Cfg::kStages * U;
  // Start the copies of one step (U consecutive 16-token tiles) into a stage.  Each tile slot of the stage has the
  // layout of a 16-token page chunk, so with 16-token pages a tile is one linear run; with larger pages it is six runs
  // (codes, norms, residual norms, value codes, scales, zeros).  Lanes 0 .. U-1 look up and copy one tile each; lane 0
  // arms the stage's mbarrier with the bytes of all of them first.  Called by the whole warp.
  auto issue_step = [&](int step, int stage, int32_t page = kPageNotAsked) {
    int valid = 0;
    const uint8_t* chunk_ptr = nullptr;
    int s0 = 0;
    if (lane < U) {
      const int tile = (warp + step * kMmaWarps) * U + lane;
      if (tile < num_tiles) {
        const int ts = t0 + tile * kTileTokens;
        const uint32_t blk = block_shift >= 0 ? ((uint32_t)ts >> block_shift) : ((uint32_t)ts / block_size);
        s0 = ts - (int)(blk * block_size);  // first slot of the tile inside its page
        const int32_t pid = page != kPageNotAsked ? page : table_row[blk];
        if (pid >= 0 && pid < p.num_pages) {  // else a hole in the block table: nothing to copy
          valid = min(kTileTokens, t1 - ts);
          chunk_ptr = p.pages + ((int64_t)pid * p.kv_heads + kvh) * p.layout.chunk_bytes;
        }
      }
      stage_valid[stage * U + lane] = valid;
    }
    const uint32_t bar = bars_u32 + stage * 8;
    const unsigned have = __ballot_sync(0xffffffffu, valid > 0);
    if (lane == 0) {
      if (have != 0u) mbar_expect_tx(bar, (uint32_t)__popc(have) * Cfg::kTileDataBytes);
      else mbar_arrive(bar);  // the phase completes at once
    }
    __syncwarp();
    if (valid > 0) {
      const uint32_t dst = warp_smem_u32 + (stage * U + lane) * Cfg::kStageBytes;
      if (block_size == (uint32_t)kTileTokens) {
        bulk_copy_g2s(dst, chunk_ptr, Cfg::kTileDataBytes, bar);
      } else {
        bulk_copy_g2s(dst + Cfg::kOffKey, chunk_ptr + p.layout.off_kcodes + s0 * Cfg::kKeyBytes, 16 * Cfg::kKeyBytes, bar);
        bulk_copy_g2s(dst + Cfg::kOffNorm, chunk_ptr + p.layout.off_knorm + 4 * s0, 64, bar);
        bulk_copy_g2s(dst + Cfg::kOffRnorm, chunk_ptr + p.layout.off_krnorm + 4 * s0, 64, bar);
        bulk_copy_g2s(dst + Cfg::kOffVal, chunk_ptr + p.layout.off_vdata + s0 * Cfg::kValBytes, 16 * Cfg::kValBytes, bar);
        bulk_copy_g2s(dst + Cfg::kOffScale, chunk_ptr + p.layout.off_vscale + s0 * Cfg::kGroups * 2, 16 * Cfg::kGroups * 2,
                      bar);
        bulk_copy_g2s(dst + Cfg::kOffZero, chunk_ptr + p.layout.off_vzero + s0 * Cfg::kGroups * 2, 16 * Cfg::kGroups * 2,
                      bar);
      }
    }
  };

  // this warp's query rows (heads warp, warp + 4) are on their way, too, before anything waits
  TqRawQueries<T, D> raw;
  if constexpr (EARLY) raw.load(p, b, hq0, g_count);

  const int num_steps = (num_tiles + U - 1) / U;
  const int my_steps = num_steps > warp && !ring.dead ? (num_steps - warp + kMmaWarps - 1) / kMmaWarps : 0;
#pragma unroll
  for (int i = 0; i < Cfg::kStages - 1; ++i)
    if (i < my_steps) issue_step(i, (ring.stage + i) % Cfg::kStages, i == 0 ? first_page : kPageNotAsked);
  if constexpr (!EARLY) raw.load(p, b, hq0, g_count);
  if (EARLY && !qc.loaded) {  // the same in all segments; behind the first copies
    TqRawConsts<D, BITS> mine;
    if (consts == nullptr) mine.load(p);
    qc = load_query_consts(consts != nullptr ? *consts : mine);
  }

  // Q fragments and their factors for this lane's two heads (columns 2tig, 2tig + 1); the softmax scale and log2(e) are
  // folded into the factors
  uint8_t* query = smem_raw + Cfg::kQueryOffset;
  const uint32_t lut[2] = {qc.lut[0], qc.lut[1]};
  prepare_query_fragments<T, D, BITS>(p, smem_raw, query, ring_free_stage(ring.stage, Cfg::kStages), raw, g_count, qc);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the loop's first copy lands where the rotations were
  __syncthreads();
  float m_run[2] = {-INFINITY, -INFINITY};
  float l_run[2] = {0.0f, 0.0f};
  float o_acc[Cfg::kSteps][4];
#pragma unroll
  for (int j = 0; j < Cfg::kSteps; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) o_acc[j][r] = 0.0f;
  const uint4* q_frag = reinterpret_cast<const uint4*>(query) + lane;                     // [s][lane]
  const uint2* q_fine = reinterpret_cast<const uint2*>(query + Cfg::kFragBytes) + lane;   // 4-bit
  const uint4* q_frag2 = reinterpret_cast<const uint4*>(query + Cfg::kFragBytes) + lane;  // planes
  // the fragments of the second tile of a pair: heads 0-3 in columns 4-7 and (from the empty heads 4-7) zeros in 0-3
  const int flip = (lane ^ 16) - lane;
  const int my_tile = kPair ? tig >> 1 : 0;  // tile whose scores this lane's two columns hold
  const int my_head = kPair ? (2 * tig) & 3 : 2 * tig;
  float beta1[2], beta2[2];                                              // factors of the two products
  float k_bit1[2] = {0.0f, 0.0f}, k_both[2] = {0.0f, 0.0f}, c_idx[2] = {0.0f, 0.0f}, c_sign[2] = {0.0f, 0.0f};  // planes
  {
    const float* consts = reinterpret_cast<const float*>(query + Cfg::kConstOffset) + my_head;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      beta1[c] = consts[c];
      if constexpr (Cfg::kPlanes) {
        if constexpr (BITS == 3) {
          k_bit1[c] = consts[8 + c];
          k_both[c] = consts[16 + c];
        }
        c_idx[c] = consts[24 + c];
      }
      beta2[c] = consts[32 + c];
      c_sign[c] = consts[40 + c];
    }
  }
  const bool skewed = BITS == 3 && __any_sync(0xffffffffu, k_both[0] != 0.0f || k_both[1] != 0.0f);
  (void)q_fine; (void)q_frag2; (void)k_bit1; (void)k_both; (void)c_idx; (void)c_sign; (void)lut; (void)skewed; (void)flip;

  // MMA row r of a tile holds token r ^ ((r >> 1) & 1): neighbouring token rows sit in different halves of the
  // shared-memory banks, and with this order the four token rows one value load touches fall into both halves.
  const int tok_lo = gid ^ ((gid >> 1) & 1);  // rows gid and gid + 8 of the score product
  const int tok_hi = tok_lo + 8;
  // k-slots 2tig, 2tig+1 (and +8) of the value product = the same rows
  const int tok_a0 = (2 * tig) ^ (tig & 1), tok_a1 = (2 * tig + 1) ^ (tig & 1);
  // this lane's value dims: D/8 consecutive dims starting at gid * D/8, all inside value group (gid * D/8) / 32
  const int v_group = (gid * (D / 8)) / 32;

  int stage = ring.stage;
  uint32_t phase = ring.phase;
  for (int n = 0; n < my_steps; ++n) {
    __syncwarp();  // every lane is done with the stage that is re-armed next (the one step n - 1 used)
    {
      const int ahead = n + Cfg::kStages - 1;
      if (ahead < my_steps) issue_step(ahead, stage == 0 ? Cfg::kStages - 1 : stage - 1);
    }
    if (!mbar_wait(bars_u32 + stage * 8, phase)) {
      if (lane == 0) atomicAdd(&g_tq_mma_faults, 1);
      // wait (bounded) for the copies still in flight before the epilogue reuses the stages
      for (int k = 1; k < Cfg::kStages && n + k < my_steps; ++k) {
        const int st_k = (stage + k) % Cfg::kStages;
        (void)mbar_wait(bars_u32 + st_k * 8, stage + k >= Cfg::kStages ? phase ^ 1u : phase);
      }
      ring.dead = true;
      break;  // give up on this chunk: the fault counter tells the host that the output is not valid
    }
    const int cur = stage;
    if (++stage == Cfg::kStages) { stage = 0; phase ^= 1u; }
    int valid[U];
    int valid_sum = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      valid[u] = stage_valid[cur * U + u];
      valid_sum += valid[u];
    }
    if (valid_sum == 0) continue;  // holes only: no token of this step exists
    const bool full = valid_sum == U * kTileTokens;
    const uint8_t* st0 = warp_smem + cur * U * Cfg::kStageBytes;

    // ---- scores: U independent pairs of accumulation chains ------------------------------------------------------------
    float s1[A][4], s2[A][4];
    {
      uint32_t iw_lo[U][Cfg::kIdxWords], iw_hi[U][Cfg::kIdxWords];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint8_t* keys = st0 + u * Cfg::kStageBytes + Cfg::kOffKey + tig * (Cfg::kIdxWords * 4);
        lds_words<Cfg::kIdxWords>(keys + tok_lo * Cfg::kKeyBytes, iw_lo[u]);
        lds_words<Cfg::kIdxWords>(keys + tok_hi * Cfg::kKeyBytes, iw_hi[u]);
      }
      if constexpr (BITS == 4) {
        // one code word = 8 coordinates of a token = one k-step: its low half-word selects four centroid bytes, its high
        // half-word the next four; the sign bits of its low and of its high nibbles are a plane each (one logic operation
        // per four coordinates instead of a permute and half a shift: 64 rows of 32 K tokens 612 -> 596 us)
        int i1[A][4], i1l[A][4], i2[A][4];
#pragma unroll
        for (int u = 0; u < A; ++u) {
          i1[u][0] = i1[u][1] = i1[u][2] = i1[u][3] = 0;
          i1l[u][0] = i1l[u][1] = i1l[u][2] = i1l[u][3] = 0;
          i2[u][0] = i2[u][1] = i2[u][2] = i2[u][3] = 0;
        }
#pragma unroll
        for (int s = 0; s < Cfg::kSteps8; ++s) {
          uint4 qc[U];  // q1 b0, q1 b1, q2 b0, q2 b1
          uint2 qf[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            qc[u] = u == 0 || !kPair ? q_frag[s * 32] : q_frag[s * 32 + flip];
            qf[u] = u == 0 || !kPair ? q_fine[s * 32] : q_fine[s * 32 + flip];
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint32_t xl = iw_lo[u][s], xh = iw_hi[u][s];
            const uint32_t ml = xl & kIdxMask, mh = xh & kIdxMask;
            const uint32_t a[4] = {prmt_ptx(lut[0], lut[1], ml), prmt_ptx(lut[0], lut[1], mh),
                                   prmt_ptx(lut[0], lut[1], ml >> 16),
                                   prmt_ptx(lut[0], lut[1], mh >> 16)};
            mma_s8(i1[u % A], a, qc[u].x, qc[u].y);
            mma_s8(i1l[u % A], a, qf[u].x, qf[u].y);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint32_t xl = iw_lo[u][s], xh = iw_hi[u][s];
            const uint32_t a[4] = {(xl << 4) & kTop, (xh << 4) & kTop, xl & kTop, xh & kTop};
            mma_u8s8(i2[u % A], a, qc[u].z, qc[u].w);
          }
        }
#pragma unroll
        for (int u = 0; u < A; ++u)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            // 254 * coarse + fine stays below 2^31 (|coarse| <= 127 * 127 * D); beta1 carries the 1 / 254
            s1[u][r] = (float)(i1[u][r] * 254 + i1l[u][r]) * beta1[r & 1];
            s2[u][r] = fmaf((float)i2[u][r], beta2[r & 1], c_sign[r & 1]);
          }
      } else {
        // fields: bit 1 of a 2-bit field (the sign, or the index's upper bit) at the top of its byte, bit 0 next to it
        constexpr int kPairs = Cfg::kIdxWords / 2;
        int lo_c[A][4], lo_f[A][4], hi_c[A][4], hi_f[A][4];
#pragma unroll
        for (int u = 0; u < A; ++u)
#pragma unroll
          for (int r = 0; r < 4; ++r) lo_c[u][r] = lo_f[u][r] = hi_c[u][r] = hi_f[u][r] = 0;
#pragma unroll
        for (int s = 0; s < Cfg::kSteps8; ++s) {
          const int up = 6 - 2 * (s / kPairs), w = 2 * (s % kPairs);
          uint4 q1[U], qh[U];  // coarse b0, b1, fine b0, b1
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int at = s * 32 + (u == 0 || !kPair ? 0 : flip);
            q1[u] = q_frag[at];
            qh[u] = BITS == 2 ? q_frag2[at] : q1[u];
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint32_t x[4] = {iw_lo[u][w] << up, iw_hi[u][w] << up, iw_lo[u][w + 1] << up, iw_hi[u][w + 1] << up};
            const uint32_t a_lo[4] = {x[0] & kNext, x[1] & kNext, x[2] & kNext, x[3] & kNext};
            mma_u8s8(lo_c[u % A], a_lo, q1[u].x, q1[u].y);
            mma_u8s8(lo_f[u % A], a_lo, q1[u].z, q1[u].w);
            const uint32_t a_hi[4] = {x[0] & kTop, x[1] & kTop, x[2] & kTop, x[3] & kTop};
            mma_u8s8(hi_c[u % A], a_hi, qh[u].x, qh[u].y);
            mma_u8s8(hi_f[u % A], a_hi, qh[u].z, qh[u].w);
          }
        }
        // 254 * coarse + fine stays below 2^31: |T| <= 128 * 127 * D * 255
#pragma unroll
        for (int u = 0; u < A; ++u)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            s1[u][r] = fmaf((float)(lo_c[u][r] * 254 + lo_f[u][r]), beta1[r & 1], c_idx[r & 1]);
            const float t = (float)(hi_c[u][r] * 254 + hi_f[u][r]);
            if constexpr (BITS == 2) s2[u][r] = fmaf(t, beta2[r & 1], c_sign[r & 1]);
            else s1[u][r] = fmaf(t, k_bit1[r & 1], s1[u][r]);
          }
        if constexpr (BITS == 3) {
          if (skewed) {  // the codebook is not symmetric: a third plane, where both bits are set
            asm volatile("" ::: "memory");
#pragma unroll
            for (int u = 0; u < A; ++u)
#pragma unroll
              for (int r = 0; r < 4; ++r) lo_c[u][r] = lo_f[u][r] = 0;
#pragma unroll
            for (int s = 0; s < Cfg::kSteps8; ++s) {
              const int up = 6 - 2 * (s / kPairs), w = 2 * (s % kPairs);
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const uint4 q1 = q_frag[s * 32 + (u == 0 || !kPair ? 0 : flip)];
                const uint32_t x[4] = {iw_lo[u][w] << up, iw_hi[u][w] << up, iw_lo[u][w + 1] << up, iw_hi[u][w + 1] << up};
                uint32_t a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = x[i] & (x[i] >> 1) & kNext;
                mma_u8s8(lo_c[u % A], a, q1.x, q1.y);
                mma_u8s8(lo_f[u % A], a, q1.z, q1.w);
              }
            }
#pragma unroll
            for (int u = 0; u < A; ++u)
#pragma unroll
              for (int r = 0; r < 4; ++r)
                s1[u][r] = fmaf((float)(lo_c[u][r] * 254 + lo_f[u][r]), k_both[r & 1], s1[u][r]);
          }
          uint32_t sw_lo[U][Cfg::kSignWords], sw_hi[U][Cfg::kSignWords];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint8_t* signs = st0 + u * Cfg::kStageBytes + Cfg::kOffKey + Cfg::kIdxBytes + tig * (Cfg::kSignWords * 4);
            lds_words<Cfg::kSignWords>(signs + tok_lo * Cfg::kKeyBytes, sw_lo[u]);
            lds_words<Cfg::kSignWords>(signs + tok_hi * Cfg::kKeyBytes, sw_hi[u]);
#pragma unroll
            for (int r = 0; r < 4; ++r) hi_c[u % A][r] = hi_f[u % A][r] = 0;
          }
#pragma unroll
          for (int s = 0; s < Cfg::kSteps8; ++s) {
            const int up = 7 - 2 * (s % 4), w = s / 4;
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const uint4 q2 = q_frag2[s * 32 + (u == 0 || !kPair ? 0 : flip)];
              const uint32_t a[4] = {(sw_lo[u][w] << up) & kTop, (sw_hi[u][w] << up) & kTop,
                                     (sw_lo[u][w] << (up - 1)) & kTop, (sw_hi[u][w] << (up - 1)) & kTop};
              mma_u8s8(hi_c[u % A], a, q2.x, q2.y);
              mma_u8s8(hi_f[u % A], a, q2.z, q2.w);
            }
          }
#pragma unroll
          for (int u = 0; u < A; ++u)
#pragma unroll
            for (int r = 0; r < 4; ++r)
              s2[u][r] = fmaf((float)(hi_c[u][r] * 254 + hi_f[u][r]), beta2[r & 1], c_sign[r & 1]);
        }
      }
    }
    // score (log2 units) = norm * (S1 + rnorm * S2); the constant factors are folded into the query fragments
    float sc[A][4];
#pragma unroll
    for (int u = 0; u < A; ++u) {
      const uint8_t* st = st0 + (kPair ? my_tile : u) * Cfg::kStageBytes;
      const float* norms = reinterpret_cast<const float*>(st + Cfg::kOffNorm);
      const float* rnorms = reinterpret_cast<const float*>(st + Cfg::kOffRnorm);
      const float n_lo = norms[tok_lo], r_lo = rnorms[tok_lo], n_hi = norms[tok_hi], r_hi = rnorms[tok_hi];
      sc[u][0] = n_lo * fmaf(r_lo, s2[u][0], s1[u][0]);
      sc[u][1] = n_lo * fmaf(r_lo, s2[u][1], s1[u][1]);
      sc[u][2] = n_hi * fmaf(r_hi, s2[u][2], s1[u][2]);
      sc[u][3] = n_hi * fmaf(r_hi, s2[u][3], s1[u][3]);
      if (!full) {  // rows past the end of the prefix (their bytes may be anything)
        asm volatile("" ::: "memory");  // a real (warp-uniform) branch: full steps pay nothing for the masking
        const int tokens = kPair && my_tile != 0 ? valid[U - 1] : valid[u];
        if (tok_lo >= tokens) sc[u][0] = sc[u][1] = -INFINITY;
        if (tok_hi >= tokens) sc[u][2] = sc[u][3] = -INFINITY;
      }
    }

    // ---- online softmax over the U * 16 tokens; the running maximum moves only when it would grow by more than 2^8 ----
    float mx[2] = {fmaxf(sc[0][0], sc[0][2]), fmaxf(sc[0][1], sc[0][3])};
#pragma unroll
    for (int u = 1; u < A; ++u) {
      mx[0] = fmaxf(mx[0], fmaxf(sc[u][0], sc[u][2]));
      mx[1] = fmaxf(mx[1], fmaxf(sc[u][1], sc[u][3]));
    }
#pragma unroll
    for (int d = 4; d <= 16; d <<= 1) {
      mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], d));
      mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], d));
    }
    const bool grew = (mx[0] > m_run[0] + kLazyRescale) || (mx[1] > m_run[1] + kLazyRescale);
    if (__any_sync(0xffffffffu, grew)) {
      const float m_new[2] = {fmaxf(m_run[0], mx[0]), fmaxf(m_run[1], mx[1])};
      const float a0 = fast_exp2(m_run[0] - (m_new[0] == -INFINITY ? 0.0f : m_new[0]));
      const float a1 = fast_exp2(m_run[1] - (m_new[1] == -INFINITY ? 0.0f : m_new[1]));
      l_run[0] *= a0;
      l_run[1] *= a1;
#pragma unroll
      for (int j = 0; j < Cfg::kSteps; ++j) {
        o_acc[j][0] *= a0;
        o_acc[j][1] *= a1;
        o_acc[j][2] *= a0;
        o_acc[j][3] *= a1;
      }
      m_run[0] = m_new[0];
      m_run[1] = m_new[1];
    }
    const float m_ref[2] = {m_run[0] == -INFINITY ? 0.0f : m_run[0], m_run[1] == -INFINITY ? 0.0f : m_run[1]};
    uint32_t pb[U][2];
#pragma unroll
    for (int u = 0; u < A; ++u) {
      const float p0 = fast_exp2(sc[u][0] - m_ref[0]);
      const float p1 = fast_exp2(sc[u][1] - m_ref[1]);
      const float p2 = fast_exp2(sc[u][2] - m_ref[0]);
      const float p3 = fast_exp2(sc[u][3] - m_ref[1]);
      l_run[0] += p0 + p2;
      l_run[1] += p1 + p3;
      pb[u][0] = movmatrix_trans(pack2<__half>(p0, p1));  // rows 2tig, 2tig+1 of head gid
      pb[u][1] = movmatrix_trans(pack2<__half>(p2, p3));  // rows 2tig+8, 2tig+9
    }

    if constexpr (kPair) {  // each tile's probabilities in its own columns, zeros in the other's
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        pb[1][i] = gid >= 4 ? pb[0][i] : 0u;
        pb[0][i] = gid >= 4 ? 0u : pb[0][i];
      }
    }

    // ---- values: lane holds rows {2tig, 2tig+1} and {2tig+8, 2tig+9}, dims gid*D/8 .. +D/8 -----------------------------------
    uint32_t sc_pair[U][2], zp_pair[U][2];
    uint32_t vw[U][4][Cfg::kValWords];  // rows 2tig, 2tig+1, 2tig+8, 2tig+9
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint8_t* st = st0 + u * Cfg::kStageBytes;
      const T* scales = reinterpret_cast<const T*>(st + Cfg::kOffScale) + v_group;
      const T* zeros = reinterpret_cast<const T*>(st + Cfg::kOffZero) + v_group;
      float sv[4], zv[4];
      const int toks[4] = {tok_a0, tok_a1, tok_a0 + 8, tok_a1 + 8};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sv[i] = ElemTraits<T>::to_float(scales[toks[i] * Cfg::kGroups]);
        zv[i] = ElemTraits<T>::to_float(zeros[toks[i] * Cfg::kGroups]);
      }
      if (!full) {
        asm volatile("" ::: "memory");  // a real (warp-uniform) branch, as above
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (toks[i] >= valid[u]) sv[i] = zv[i] = 0.0f;
      }
      sc_pair[u][0] = pack2<__half>(sv[0], sv[1]);
      sc_pair[u][1] = pack2<__half>(sv[2], sv[3]);
      zp_pair[u][0] = pack2<__half>(zv[0], zv[1]);
      zp_pair[u][1] = pack2<__half>(zv[2], zv[3]);
      const uint8_t* vbase = st + Cfg::kOffVal + gid * (Cfg::kValWords * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) lds_words<Cfg::kValWords>(vbase + toks[i] * Cfg::kValBytes, vw[u][i]);
    }
    if constexpr (BITS != 2) {
      // 4-bit codes: one 16-bit half-word = 4 dims; x packs the same 4 dims of two tokens (low / high half).  A code
      // moved to bits 6..9 under the exponent of 16 reads as the fp16 number 16 + code, so one fused multiply-add
      // de-quantises a pair: (16 + code) * scale + (zero - 16 * scale).  The shifted zero point is rounded to fp16 once
      // per token and group; it is no larger than the values themselves, so this costs what their own rounding costs.
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) zp_pair[u][pr] = hfma2_u32(sc_pair[u][pr], 0xCC00CC00u, zp_pair[u][pr]);
#pragma unroll
      for (int hw = 0; hw < Cfg::kValWords * 2; ++hw) {
        const uint32_t sel = (hw % 2) ? 0x7632u : 0x5410u;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          uint32_t r[2][4];
#pragma unroll
          for (int pr = 0; pr < 2; ++pr) {
            const uint32_t x = prmt(vw[u][2 * pr][hw / 2], vw[u][2 * pr + 1][hw / 2], sel);
            const uint32_t scl = sc_pair[u][pr], zpt = zp_pair[u][pr];
            r[pr][0] = hfma2_u32(and_or_regs(x << 6, nib_mask, magic16), scl, zpt);
            r[pr][1] = hfma2_u32(and_or_regs(x << 2, nib_mask, magic16), scl, zpt);
            r[pr][2] = hfma2_u32(and_or_regs(x >> 2, nib_mask, magic16), scl, zpt);
            r[pr][3] = hfma2_u32(and_or_regs(x >> 6, nib_mask, magic16), scl, zpt);
          }
          // dims 4hw + {0,1} -> m-tile 2hw (rows gid, gid+8); dims 4hw + {2,3} -> m-tile 2hw + 1
          const uint32_t a_even[4] = {r[0][0], r[0][1], r[1][0], r[1][1]};
          const uint32_t a_odd[4] = {r[0][2], r[0][3], r[1][2], r[1][3]};
          mma_f16(o_acc[2 * hw], a_even, pb[u][0], pb[u][1]);
          mma_f16(o_acc[2 * hw + 1], a_odd, pb[u][0], pb[u][1]);
        }
      }
    } else {
      // 2-bit codes: one 16-bit half-word = 8 dims.  A code moved to bits 8..9 under the exponent of 4 reads as the fp16
      // number 4 + code, so one fused multiply-add de-quantises a pair: (4 + code) * scale + (zero - 4 * scale); the
      // left shifts run on the multiply pipe.
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) zp_pair[u][pr] = hfma2_u32(sc_pair[u][pr], 0xC400C400u, zp_pair[u][pr]);
#pragma unroll
      for (int hw = 0; hw < Cfg::kValWords * 2; ++hw) {
        const uint32_t sel = (hw % 2) ? 0x7632u : 0x5410u;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          uint32_t r[2][8];
#pragma unroll
          for (int pr = 0; pr < 2; ++pr) {
            const uint32_t x = prmt(vw[u][2 * pr][hw / 2], vw[u][2 * pr + 1][hw / 2], sel);
            const uint32_t scl = sc_pair[u][pr], zpt = zp_pair[u][pr];
            r[pr][0] = hfma2_u32(and_or_regs(x << 8, kTwoBitMask, kMagic4), scl, zpt);
            r[pr][1] = hfma2_u32(and_or_regs(x << 6, kTwoBitMask, kMagic4), scl, zpt);
            r[pr][2] = hfma2_u32(and_or_regs(x << 4, kTwoBitMask, kMagic4), scl, zpt);
            r[pr][3] = hfma2_u32(and_or_regs(x << 2, kTwoBitMask, kMagic4), scl, zpt);
            r[pr][4] = hfma2_u32(and_or_regs(x, kTwoBitMask, kMagic4), scl, zpt);
            r[pr][5] = hfma2_u32(and_or_regs(x >> 2, kTwoBitMask, kMagic4), scl, zpt);
            r[pr][6] = hfma2_u32(and_or_regs(x >> 4, kTwoBitMask, kMagic4), scl, zpt);
            r[pr][7] = hfma2_u32(and_or_regs(x >> 6, kTwoBitMask, kMagic4), scl, zpt);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {  // dims 8hw + {2q, 2q+1} -> m-tile 4hw + q
            const uint32_t a[4] = {r[0][2 * q], r[0][2 * q + 1], r[1][2 * q], r[1][2 * q + 1]};
            mma_f16(o_acc[4 * hw + q], a, pb[u][0], pb[u][1]);
          }
        }
      }
    }
  }
  ring.stage = stage;
  ring.phase = phase;
  // ---- merge the four warps; m-tile j holds dims gid*D/8 + 2j (row gid) and + 2j + 1 (row gid + 8) --------------------------
#pragma unroll
  for (int d = 4; d <= 16; d <<= 1) {
    l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], d);
    l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], d);
  }
  __syncthreads();
  float* sm_m = reinterpret_cast<float*>(smem_raw);
  float* sm_l = sm_m + kMmaWarps * 8;
  float* sm_o = sm_l + kMmaWarps * 8;
  constexpr int kPad = D + 4;
  if (gid == 0) {
    sm_m[warp * 8 + 2 * tig] = m_run[0];
    sm_m[warp * 8 + 2 * tig + 1] = m_run[1];
    sm_l[warp * 8 + 2 * tig] = l_run[0];
    sm_l[warp * 8 + 2 * tig + 1] = l_run[1];
  }
#pragma unroll
  for (int j = 0; j < Cfg::kSteps; ++j) {
    float* base = sm_o + (warp * 8) * kPad;
    const int dim = gid * (D / 8) + 2 * j;
    base[(2 * tig) * kPad + dim] = o_acc[j][0];
    base[(2 * tig + 1) * kPad + dim] = o_acc[j][1];
    base[(2 * tig) * kPad + dim + 1] = o_acc[j][2];
    base[(2 * tig + 1) * kPad + dim + 1] = o_acc[j][3];
  }
  __syncthreads();
  const int64_t part = ((int64_t)b * p.q_heads + hq0) * p.chunk_capacity + out_slot;
  // kPair: columns g and g + 4 of every warp
  merge_parts_and_store<D, kPair ? 2 * kMmaWarps : kMmaWarps, kPair ? 4 : 8>(sm_m, sm_l, sm_o, g_count, p.stats + part * 2,
                                                                             p.values + part * D, p.chunk_capacity);
  // The window kernel's partials and, when it arrives last, its merged output must be complete before this CTA
  // counts itself in (fused merge) or the kernel ends (two-pass merge).
  wait_for_prior_grids();
  if (p.fused.counters != nullptr) {
    const int64_t head0 = ((int64_t)b * p.q_heads + hq0) * p.chunk_capacity;
    __syncthreads();
    if constexpr (AHEAD)
      fused_combine_ahead<T, D, kMmaThreads, kMergeHeads<D, kPair>, MERGE>(
          p.fused, b, hq0, g_count, slots, p.chunk_capacity, p.stats + head0 * 2, p.values + head0 * D,
          reinterpret_cast<float*>(smem_raw), (int64_t)b * units + unit, arrivals);
    else
      fused_combine_tail<T, D, kMmaThreads, kMergeHeads<D, kPair>, MERGE>(
          p.fused, b, hq0, g_count, slots, p.chunk_capacity, p.stats + head0 * 2, p.values + head0 * D,
          reinterpret_cast<float*>(smem_raw), (int64_t)b * units + unit, arrivals);
  }
  // the merge buffers lie where the next segment's copies land: order those writes before the copy engine's
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncthreads();
}

template <typename T, int D, int BITS>
__device__ __forceinline__ void init_packed_barriers(uint8_t* smem_raw) {
  using Cfg = TqMmaCfg<T, D, BITS>;
  if (threadIdx.x == 0) {
    const uint32_t bars = smem_u32(smem_raw + Cfg::kWorkSmem);
    for (int i = 0; i < kMmaWarps * Cfg::kStages; ++i) mbar_init(bars + i * 8, 1);
    mbar_init_fence();
  }
  __syncthreads();
}

// Fixed chunks of the context, handed out by the block scheduler: grid (window chunks + packed chunks, units, batch).
template <typename T, int D, int BITS, bool kPair>
__global__ void __launch_bounds__(kMmaThreads, TqMmaCfg<T, D, BITS>::kMinBlocks)
    tq_decode_split_mma_kernel(const TqDecodeParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int b = blockIdx.z;
  const RowChunks row = row_chunks(p, b);
  const int chunk = (int)blockIdx.x - p.num_window_chunks;  // window chunks run in tq_window_split_mma_kernel
  if (chunk < 0 || chunk >= row.packed) {
    wait_for_prior_grids();
    return;
  }
  const int t0 = chunk * p.chunk_tokens;
  init_packed_barriers<T, D, BITS>(smem_raw);
  PackedRing ring{0, 0u, false};
  TqRawConsts<D, BITS> consts;
  consts.load(p);
  TqQueryConsts qc = load_query_consts(consts);
  // active slots stay contiguous: [window | packed]
  tq_packed_segment<T, D, BITS, kPair, MergeLoads::kAllColumns, false>(
      p, smem_raw, qc, ring, b, (int)blockIdx.y, (int)gridDim.y, t0, min(row.quantized, t0 + p.chunk_tokens), row.window + chunk,
      row.window + row.packed, row.packed);
}

// Small calls: window chunks and packed chunks in one launch, grid (window chunks + packed chunks, units, batch), all of it
// resident at once; every chunk counts on the merge counter.  The second launch of the other kernels costs the host about
// as much as the rest of such a call.  With few CTAs there are registers and shared memory to spare, but a window CTA has to
// live with what a packed one has: its ring holds one tile per warp.
template <typename T, int D, int BITS>
struct TqSmallCfg {
  static constexpr int kMinBlocks = D >= 256 ? 2 : 3;
  static constexpr int kWindowSmem = MmaCfg<D, 1>::kSmemBytes;
  static constexpr int kPackedSmem = TqMmaCfg<T, D, BITS>::kSmemBytes;
  static constexpr int kSmemBytes = kWindowSmem > kPackedSmem ? kWindowSmem : kPackedSmem;
  // the merge stages its weights in the window CTAs' shared memory, too
  static_assert(kWindowSmem >= 8 * kFusedMaxChunks * 4, "no room for the weights of the merge");
};

template <typename T, int D, int BITS, bool kPair>
__global__ void __launch_bounds__(kMmaThreads, TqSmallCfg<T, D, BITS>::kMinBlocks)
    tq_decode_small_mma_kernel(const TqDecodeParams p) {
  constexpr bool kEarly = TqSmallOrder<D, BITS, kPair>::kEarly;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int b = blockIdx.z;
  const int chunk = (int)blockIdx.x - p.num_window_chunks;
  const int t0 = chunk * p.chunk_tokens;
  int32_t first_page = kPageNotAsked;
  TqRawConsts<D, BITS> consts;
  if constexpr (kEarly) {  // the page, the constants and the lengths are read side by side
    if (chunk >= 0) first_page = first_page_of<T, D, BITS>(p, b, t0);
    consts.load(p);
  }
  const RowChunks row = row_chunks(p, b);
  if (chunk < 0) {
    tq_window_chunk<T, D, 1, kMergeHeads<D, kPair>, true>(p, smem_raw, row, b, blockIdx.y, gridDim.y, blockIdx.x, true);
    return;
  }
  if (chunk >= row.packed) return;
  init_packed_barriers<T, D, BITS>(smem_raw);
  PackedRing ring{0, 0u, false};
  TqQueryConsts qc{};
  if constexpr (!kEarly) {
    consts.load(p);
    qc = load_query_consts(consts);
  }
  const int active = row.window + row.packed;
  tq_packed_segment<T, D, BITS, kPair, MergeLoads::kAllColumns, kEarly, true>(
      p, smem_raw, qc, ring, b, (int)blockIdx.y, (int)gridDim.y, t0, min(row.quantized, t0 + p.chunk_tokens), row.window + chunk, active,
      active, first_page, &consts);
}

// What a segment costs beyond its tiles (query preparation, first copy, merge: about 6 us), in tiles.  Over 512 shapes (1 to
// 1000 rows of 129 to 16000 tokens, all widths, head_dim 128 and 256, 1 to 12 query heads per KV head) the mean time was 16 %
// longer with 0, 1.6 % with 10, 0.1 % shorter with 40.
constexpr int kTqSegmentTiles = 20;

// Persistent variant: one resident wave, every CTA takes an even share of the packed tiles (balanced_schedule.cuh).
template <typename T, int D, int BITS, bool kPair, bool kShort>
__global__ void __launch_bounds__(kMmaThreads, TqMmaCfg<T, D, BITS>::kMinBlocks)
    tq_decode_balanced_mma_kernel(const TqDecodeParams p, const int batch) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // This instance has no registers for the loads of two columns and issues them one after the other (two rows of 12000 tokens,
  // 16/2 heads: 44.7 us, one column after the other 32.4; one of 20000, 64/8 heads: 45.7 and 36.2).
  constexpr MergeLoads kMerge = D == 128 && BITS == 3 && !kPair ? MergeLoads::kOneColumn : MergeLoads::kAllColumns;
  using Order = TqShareOrder<D, BITS, kPair, kShort>;
  const int units = p.kv_heads * ((p.groups + 7) / 8);
  init_packed_barriers<T, D, BITS>(smem_raw);
  PackedRing ring{0, 0u, false};
  TqQueryConsts qc{};
  if constexpr (!Order::kEarly) {
    TqRawConsts<D, BITS> consts;
    consts.load(p);
    qc = load_query_consts(consts);
  }
  balanced_for_each_segment<kMmaThreads, false>(
      p.lengths, p.max_len, batch, units, min(p.chunk_capacity, kFusedMaxChunks) - p.num_window_chunks,
      [](int) {},  // rows without packed tokens belong to the window kernel
      [&](int b, int unit, int t0, int t1, int slot, int partials) {
        const int active_window = (p.residual_len + p.chunk_tokens - 1) / p.chunk_tokens;  // the window of this row is full
        tq_packed_segment<T, D, BITS, kPair, kMerge, Order::kEarly, Order::kAhead>(p, smem_raw, qc, ring, b, unit, units, t0, t1,
                                                                                   active_window + slot, active_window + partials,
                                                                                   partials);
      },
      p.residual_len, kMmaWarps * TqMmaCfg<T, D, BITS>::kTilesPerStep, kTqSegmentTiles, kTqSegmentTiles);
  wait_for_prior_grids();
}

// A call that is not small in the plan's chunks may be so in longer ones, up to this many tokens.  128 tokens are one step of a
// CTA's warps, of which 64 leave half idle; 256 are two, which still costs less than the scan and the second launch of even
// shares (GPU time, one row of 4000 tokens, 32/8 heads, 4 bits: 17.4 us in shares, 12.0 so; of 8000 20.8 and 13.4; 4 rows of
// 1500, 8 heads, 3 bits 16.4 and 11.7; 6 rows of 0.3-1.5 K, 8/4 heads of 256 17.5 and 13.0).
constexpr int kTqSmallChunk = 256;

static bool tq_fixed_chunks_only() {
  static const bool disabled = [] {
    const char* flag = std::getenv("ANNA_B200_DISABLE_BALANCED");
    return flag != nullptr && flag[0] != '\0' && flag[0] != '0';
  }();
  return disabled;
}

// A small call, whose chunks are resident at once, gains nothing from even shares and pays for the scan of the lengths (GPU time,
// one row of 260-2500 tokens, 8 heads, 3 bits: 13.9-16.4 us in shares, 9.9-12.7 in chunks; 4 rows of 500, 32/8 heads, 4 bits: 15.1
// and 9.9), unless it waits for the last CTA's merge, which even shares give fewer partials (eight heads of 256, two KV heads, one
// row of 6000 tokens: 92 partials of 64 tokens 31.7 us, shares 27.6; of 3712, 56 partials, 25.4 and 23.5; eight heads of 128, 120
// partials, 24.0 and 21.9).  The limits are on the safe side: 50 partials of four heads of 128 would still gain (one row of 12928
// tokens, 32/8 heads: 17.2 and 25.7), and 20 of eight heads of 256 (two of 5248, 32/4 heads: 21.8 and 31.1).
// `resident` = CTAs that fit the GPU at once.
static bool tq_small(const TqDecodeParams& p, int batch, int head_dim, int64_t ctas, int resident) {
  const int64_t chunks = p.num_chunks - p.num_window_chunks;
  const int rounds = (min(8, p.groups) * (head_dim / 4) + kMmaThreads - 1) / kMmaThreads;
  return ctas <= resident && chunks * rounds <= (rounds == 1 ? 40 : 24);
}

// Which schedule the packed prefix of a call that is not small takes; `ctas` = CTAs of the even-share kernel that are
// resident at once.
static bool tq_use_balanced(const TqDecodeParams& p, int batch, int head_dim, int ctas) {
  const int64_t units = (int64_t)p.kv_heads * ((p.groups + 7) / 8);
  const int packed_slots = min(p.chunk_capacity, kFusedMaxChunks) - p.num_window_chunks;
  if (tq_fixed_chunks_only() || p.given_chunks || p.fused.counters == nullptr) return false;
  if (!balanced_schedule_fits(batch, units, p.max_len, packed_slots, kTqSegmentTiles)) return false;
  // The plan's longest chunks mean that there are enough of them for a few waves, which the block scheduler hands out as SMs
  // get free.  With six waves or more (counted by the longest row) that is better than even shares (64 rows of 32 K tokens,
  // 32/8 heads, 6.9 waves: 590 us, shares 611; 600 rows of 0.75-6 K, 48/4 heads, 16 waves: 697 and 742), with fewer the last
  // one is too empty or too ragged (128 rows of 0.5-16 K, 16/4 heads, 3.5 waves: 227.5 and 217.4; 40 rows of 2-16 K, 32/8
  // heads: 157 and 136, of 16 K 219 and 205; 64 rows of 8-24 K, 5.2 waves: 323 and 317) -- but not of rows of no more than two
  // chunks, where even lengths leave nothing to share (128 rows of 8 K, 3.5 waves: 323 and 337; of 1-8 K 226 and 222).
  // With less work the chunks shrink, down to 64 tokens, and every CTA's fixed cost and the number of partials grow (16 rows
  // of 0.4-4 K tokens, 16/2 heads of 256: 70 us, even shares 36; 64 rows of 4-32 K: 196 and 169).
  const int64_t longest = p.num_chunks - p.num_window_chunks;
  if (p.chunk_tokens >= kTqLongestChunk && (longest <= 2 || batch * units * longest >= (int64_t)6 * ctas)) return false;
  return !tq_small(p, batch, head_dim, batch * units * (p.num_chunks - p.num_window_chunks) * 5, ctas * 4);
}

// Shares of so few tokens (counted by the longest row) are short.  4-bit pairs, GPU time in the order of short shares and of long ones,
// against neither: head_dim 128, shares of 64-256 tokens 0.989 and 1.016 (18 rows of 0.5-3 K, 2/2 heads: single calls 18.8 and 19.7
// us), 256-512 0.992 and 1.001, 512-768 0.995 and 0.993, above 2048 1.004 and 0.968; head_dim 256, of 32-128 tokens 1 and 1.08, 128-384 1
// and 1.00 (single shapes up to 1.12), 384-768 1 and 0.989, above 2048 1 and 0.980.
constexpr int64_t kTqShortShare = 512;

static bool tq_short_shares(const TqDecodeParams& p, int batch, int ctas) {
  const int64_t units = (int64_t)p.kv_heads * ((p.groups + 7) / 8);
  return batch * units * (p.max_len - p.residual_len) < kTqShortShare * ctas;
}

// The launches of a call, and the chunks it is cut into.
struct TqLaunches {
  TqSchedule schedule;
  int chunk_tokens, num_window_chunks, num_chunks;
};

// `one_launch_ctas`, `share_ctas` = CTAs of the kernels that are resident at once.
static TqLaunches tq_choose_launches(const TqDecodeParams& p, int batch, int head_dim, int one_launch_ctas, int share_ctas) {
  TqLaunches out{TqSchedule::kOneLaunch, p.chunk_tokens, p.num_window_chunks, p.num_chunks};
  if (!tq_fixed_chunks_only() && !p.given_chunks && p.fused.counters != nullptr && batch <= 65535) {
    const int64_t units = (int64_t)p.kv_heads * ((p.groups + 7) / 8);
    TqDecodeParams sp = p;
    for (int tokens = p.chunk_tokens; tokens <= max(p.chunk_tokens, kTqSmallChunk); tokens *= 2) {
      sp.chunk_tokens = tokens;
      sp.num_window_chunks = (p.residual_len + tokens - 1) / tokens;
      sp.num_chunks = sp.num_window_chunks + (int)((p.max_len - p.residual_len + tokens - 1) / tokens);
      if (!tq_small(sp, batch, head_dim, batch * units * sp.num_chunks, one_launch_ctas)) continue;
      out.chunk_tokens = tokens;
      out.num_window_chunks = sp.num_window_chunks;
      out.num_chunks = sp.num_chunks;
      return out;
    }
  }
  out.schedule = tq_use_balanced(p, batch, head_dim, share_ctas) ? TqSchedule::kEvenShares : TqSchedule::kChunks;
  return out;
}

// CTAs of a kernel that fit the whole GPU at once, worked out at its first launch on a device, which also lets it have `smem`
// bytes of shared memory.
template <typename Kernel>
static int resident_ctas(Kernel kernel, int smem, int (&known)[64], int device, int* ctas) {
  *ctas = (device >= 0 && device < 64) ? known[device] : 0;
  if (*ctas != 0) return ANNA_OK;
  ANNA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int sms = 0, per_sm = 0;
  ANNA_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  ANNA_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kMmaThreads, smem));
  *ctas = sms * (per_sm > 0 ? per_sm : 1);
  if (device >= 0 && device < 64) known[device] = *ctas;
  return ANNA_OK;
}

template <typename T, int D, int BITS, bool kPair>
static int launch_tq_mma(const TqDecodeParams& p, int batch, cudaStream_t stream) {
  using Cfg = TqMmaCfg<T, D, BITS>;
  auto kernel = tq_decode_split_mma_kernel<T, D, BITS, kPair>;
  static bool configured[64] = {};
  int device = 0;
  ANNA_CUDA_CHECK(cudaGetDevice(&device));
  if (device < 0 || device >= 64 || !configured[device]) {
    ANNA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    ANNA_CUDA_CHECK(cudaFuncSetAttribute(tq_window_split_mma_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         MmaCfg<D>::kSmemBytes));
    if (device >= 0 && device < 64) configured[device] = true;
  }
  // with 16-token pages a tile is copied as one run, so the page chunk must have exactly the stage's layout
  if (p.block_size == kTileTokens &&
      (p.layout.off_kcodes != Cfg::kOffKey || p.layout.off_knorm != Cfg::kOffNorm ||
       p.layout.off_krnorm != Cfg::kOffRnorm || p.layout.off_vdata != Cfg::kOffVal ||
       p.layout.off_vscale != Cfg::kOffScale || p.layout.off_vzero != Cfg::kOffZero ||
       p.layout.chunk_bytes < Cfg::kTileDataBytes))
    return set_error(ANNA_ERR_INVALID, "packed page layout does not match the decode kernel's tile layout");
  const int group_tiles = (p.groups + 7) / 8;
  using Small = TqSmallCfg<T, D, BITS>;
  auto small = tq_decode_small_mma_kernel<T, D, BITS, kPair>;
  auto balanced = tq_decode_balanced_mma_kernel<T, D, BITS, kPair, false>;
  static int small_resident[64] = {}, balanced_resident[64] = {};
  int small_ctas = 0, balanced_ctas = 0;
  int rc = resident_ctas(small, Small::kSmemBytes, small_resident, device, &small_ctas);
  if (rc == ANNA_OK) rc = resident_ctas(balanced, Cfg::kSmemBytes, balanced_resident, device, &balanced_ctas);
  if (rc != ANNA_OK) return rc;
  const TqLaunches launches = tq_choose_launches(p, batch, D, small_ctas, balanced_ctas);
  if (launches.schedule == TqSchedule::kOneLaunch) {
    TqDecodeParams sp = p;
    sp.chunk_tokens = launches.chunk_tokens;
    sp.num_window_chunks = launches.num_window_chunks;
    sp.num_chunks = launches.num_chunks;
    const dim3 grid((unsigned)sp.num_chunks, (unsigned)(p.kv_heads * group_tiles), (unsigned)batch);
    small<<<grid, kMmaThreads, Small::kSmemBytes, stream>>>(sp);
    return check_launch("tq_decode_small_mma_kernel");
  }
  dim3 window_grid((unsigned)p.num_window_chunks, (unsigned)(p.kv_heads * group_tiles), (unsigned)batch);
  tq_window_split_mma_kernel<T, D><<<window_grid, kMmaThreads, MmaCfg<D>::kSmemBytes, stream>>>(p);
  rc = check_launch("tq_window_split_mma_kernel");
  if (rc != ANNA_OK) return rc;
  if (p.num_chunks <= p.num_window_chunks) return rc;
  // programmatic dependent launch: the packed chunks run beside the (small) window launch instead of after it
  cudaLaunchConfig_t config = {};
  config.blockDim = dim3(kMmaThreads);
  config.dynamicSmemBytes = Cfg::kSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = 1;
  if (launches.schedule == TqSchedule::kEvenShares) {
    if constexpr (kShareOrders<D, BITS, kPair>) {
      if (tq_short_shares(p, batch, balanced_ctas)) {
        auto in_short = tq_decode_balanced_mma_kernel<T, D, BITS, kPair, true>;
        static int short_resident[64] = {};
        int short_ctas = 0;
        rc = resident_ctas(in_short, Cfg::kSmemBytes, short_resident, device, &short_ctas);
        if (rc != ANNA_OK) return rc;
        config.gridDim = dim3((unsigned)short_ctas);
        ANNA_CUDA_CHECK(cudaLaunchKernelEx(&config, in_short, p, batch));
        return check_launch("tq_decode_balanced_mma_kernel");
      }
    }
    config.gridDim = dim3((unsigned)balanced_ctas);
    ANNA_CUDA_CHECK(cudaLaunchKernelEx(&config, balanced, p, batch));
    return check_launch("tq_decode_balanced_mma_kernel");
  }
  config.gridDim = dim3((unsigned)p.num_chunks, (unsigned)(p.kv_heads * group_tiles), (unsigned)batch);
  ANNA_CUDA_CHECK(cudaLaunchKernelEx(&config, kernel, p));
  return check_launch("tq_decode_split_mma_kernel");
}

template <typename T, int D>
static int launch_window(const TqDecodeParams& p, int batch, cudaStream_t stream) {
  static bool configured[64] = {};
  int device = 0;
  ANNA_CUDA_CHECK(cudaGetDevice(&device));
  if (device < 0 || device >= 64 || !configured[device]) {
    ANNA_CUDA_CHECK(cudaFuncSetAttribute(tq_window_split_mma_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         MmaCfg<D>::kSmemBytes));
    if (device >= 0 && device < 64) configured[device] = true;
  }
  const int group_tiles = (p.groups + 7) / 8;
  dim3 window_grid((unsigned)p.num_window_chunks, (unsigned)(p.kv_heads * group_tiles), (unsigned)batch);
  tq_window_split_mma_kernel<T, D><<<window_grid, kMmaThreads, MmaCfg<D>::kSmemBytes, stream>>>(p);
  return check_launch("tq_window_split_mma_kernel");
}

int launch_tq_window_split(const TqDecodeParams& p, int batch, int head_dim, int dtype, cudaStream_t stream) {
  if (dtype == ANNA_DTYPE_BF16)
    return head_dim == 128 ? launch_window<__nv_bfloat16, 128>(p, batch, stream)
                           : launch_window<__nv_bfloat16, 256>(p, batch, stream);
  return head_dim == 128 ? launch_window<__half, 128>(p, batch, stream) : launch_window<__half, 256>(p, batch, stream);
}

int tq_decode_mma_faults(int* count) {
  int32_t value = 0;
  ANNA_CUDA_CHECK(cudaMemcpyFromSymbol(&value, g_tq_mma_faults, sizeof(value)));
  *count = (int)value;
  return ANNA_OK;
}

// Self-test of the bounded wait: nobody ever arrives on this barrier, so the wait has to give up and say so.
__global__ void wait_expiry_selftest_kernel(int32_t* result) {
  __shared__ __align__(8) unsigned long long bar_storage;
  const uint32_t bar = smem_u32(&bar_storage);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  __syncwarp();
  const bool landed = mbar_wait(bar, 0u);
  if (threadIdx.x == 0) *result = landed ? 0 : 1;
}

bool tq_split_mma_applicable(const TqDecodeParams& p, int batch, int head_dim, int dtype) {
  static const bool disabled = [] {
    const char* flag = std::getenv("ANNA_B200_DISABLE_MMA");
    return flag != nullptr && flag[0] != '\0' && flag[0] != '0';
  }();
  if (disabled) return false;
  if (dtype != ANNA_DTYPE_F16 && dtype != ANNA_DTYPE_BF16) return false;
  if (head_dim != 128 && head_dim != 256) return false;
  if (p.value_group != 32 || p.block_size % kTileTokens != 0 || p.chunk_tokens % kTileTokens != 0) return false;
  if (p.max_len >= (int64_t)1 << 31 || p.query_frags == nullptr) return false;
  // the window chunks read query rows as aligned 32-bit pairs
  if ((reinterpret_cast<uintptr_t>(p.q) & 3u) != 0 || (batch > 1 && p.q_stride_b % 2 != 0) ||
      (p.q_heads > 1 && p.q_stride_h % 2 != 0))
    return false;
  return true;
}

int launch_tq_split_mma(const TqDecodeParams& p, int batch, int head_dim, int bits, int dtype, cudaStream_t stream) {
#define ANNA_TQ_MMA_CASE(TYPE, DIM, BITS_) \
  if (head_dim == DIM && bits == BITS_)          \
    return p.groups <= 4 ? launch_tq_mma<TYPE, DIM, BITS_, true>(p, batch, stream) \
                         : launch_tq_mma<TYPE, DIM, BITS_, false>(p, batch, stream);
  if (dtype == ANNA_DTYPE_BF16) {
    ANNA_TQ_MMA_CASE(__nv_bfloat16, 128, 2) ANNA_TQ_MMA_CASE(__nv_bfloat16, 128, 3) ANNA_TQ_MMA_CASE(__nv_bfloat16, 128, 4)
    ANNA_TQ_MMA_CASE(__nv_bfloat16, 256, 2) ANNA_TQ_MMA_CASE(__nv_bfloat16, 256, 3) ANNA_TQ_MMA_CASE(__nv_bfloat16, 256, 4)
  } else {
    ANNA_TQ_MMA_CASE(__half, 128, 2) ANNA_TQ_MMA_CASE(__half, 128, 3) ANNA_TQ_MMA_CASE(__half, 128, 4)
    ANNA_TQ_MMA_CASE(__half, 256, 2) ANNA_TQ_MMA_CASE(__half, 256, 3) ANNA_TQ_MMA_CASE(__half, 256, 4)
  }
#undef ANNA_TQ_MMA_CASE
  return set_error(ANNA_ERR_UNSUPPORTED, "no tensor-core TurboQuant decode for head_dim %d, %d bits", head_dim, bits);
}

}  // namespace anna

// Launches one warp that waits on an mbarrier nothing completes and reports whether the bounded wait gave up
// (*expired = 1) -- the path every copy wait of the library takes when its data does not arrive.  Takes about a second
// (the full wait budget), synchronises the stream, and leaves the context usable.  No counterpart in the reference.
extern "C" int anna_kv_selftest_wait_expiry(int* expired, anna_stream_t stream) {
  ANNA_REQUIRE(expired != nullptr, "anna_kv_selftest_wait_expiry: null output pointer");
  int32_t* flag = nullptr;
  ANNA_CUDA_CHECK(cudaMalloc(&flag, sizeof(int32_t)));
  cudaError_t err = cudaMemsetAsync(flag, 0xff, sizeof(int32_t), (cudaStream_t)stream);
  if (err == cudaSuccess) {
    anna::wait_expiry_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(flag);
    err = cudaGetLastError();
  }
  int32_t value = -1;
  if (err == cudaSuccess)
    err = cudaMemcpyAsync(&value, flag, sizeof(value), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (err == cudaSuccess) err = cudaStreamSynchronize((cudaStream_t)stream);
  cudaFree(flag);
  if (err != cudaSuccess)
    return anna::set_error(ANNA_ERR_CUDA, "wait-expiry self-test failed: %s", cudaGetErrorString(err));
  *expired = (int)value;
  return ANNA_OK;
}

// Number of bounded waits that expired in the kernels that stage tiles with the copy engine, on the current device,
// since the library was loaded (0 in a healthy run).  Synchronises the device.
extern "C" int anna_kv_device_faults(int* count) {
  ANNA_REQUIRE(count != nullptr, "anna_kv_device_faults: null output pointer");
  int mma = 0, umma = 0, prefill = 0;
  int rc = anna::tq_decode_mma_faults(&mma);
  if (rc == ANNA_OK) rc = anna::tq_decode_umma_faults(&umma);
  if (rc == ANNA_OK) rc = anna::prefill_umma_faults(&prefill);
  if (rc != ANNA_OK) return rc;
  *count = mma + umma + prefill;
  return ANNA_OK;
}

// Host side of a call's way through the packed decode, for tests without a GPU: what the entry point and launch_tq_mma choose.
extern "C" int anna_kv_selftest_tq_schedule(const void* q, int64_t q_stride_b, int64_t q_stride_h, int batch, int q_heads,
                                            int kv_heads, int head_dim, int64_t max_blocks, int block_size, int residual_len,
                                            int value_group, int dtype, int one_launch_ctas, int share_ctas, int* schedule,
                                            int* chunk_tokens) {
  using namespace anna;
  ANNA_REQUIRE(schedule != nullptr && chunk_tokens != nullptr && kv_heads > 0 && q_heads > 0 && q_heads % kv_heads == 0,
               "anna_kv_selftest_tq_schedule: bad argument");
  TqDecodeParams p{};
  const int rc = anna_tq_decode_plan(batch, kv_heads, max_blocks, block_size, residual_len, &p.chunk_tokens, &p.num_chunks);
  if (rc != ANNA_OK) return rc;
  int32_t counters = 0;
  p.q = q; p.q_stride_b = q_stride_b; p.q_stride_h = q_stride_h;
  p.q_heads = q_heads; p.kv_heads = kv_heads; p.groups = q_heads / kv_heads;
  p.block_size = block_size; p.residual_len = residual_len; p.value_group = value_group;
  p.max_blocks = max_blocks; p.max_len = max_blocks * (int64_t)block_size + residual_len;
  p.chunk_capacity = p.num_chunks;
  p.num_window_chunks = (residual_len + p.chunk_tokens - 1) / p.chunk_tokens;
  p.query_frags = &counters;
  if (p.num_chunks <= kFusedMaxChunks) p.fused.counters = &counters;
  *chunk_tokens = p.chunk_tokens;
  *schedule = (int)TqSchedule::kCudaCores;
  if (!tq_split_mma_applicable(p, batch, head_dim, dtype)) return ANNA_OK;
  const TqLaunches launches = tq_choose_launches(p, batch, head_dim, one_launch_ctas, share_ctas);
  *chunk_tokens = launches.chunk_tokens;
  *schedule = (int)launches.schedule;
  return ANNA_OK;
}
