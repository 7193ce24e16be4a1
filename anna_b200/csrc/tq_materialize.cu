// De-quantize packed TurboQuant pages into dense keys / values in the cache dtype (a warp per run of token-heads); with the
// window ring given, the same launch also copies the un-quantized tail of every row and zero-pads up to max_len, i.e.
// it produces the whole dense view of a batch of rows.
#include "tq_bulk.cuh"

namespace anna {

struct TqMaterializeParams {
  const uint8_t* pages;
  const int32_t* block_table;
  int64_t table_stride;
  const int64_t* quantized_lengths;
  const float* signs1;
  const float* signs2;
  const float* centroids;
  void* key_out;
  void* value_out;
  int64_t out_stride_b, out_stride_h, out_stride_t;
  int kv_heads, block_size, value_group;
  int64_t num_pages, max_blocks, max_quantized_len;
  anna_tq_layout layout;
  // optional dense tail: window ring [slots, 2, Hkv, R, D], ring slot and total length per row
  const void* window;
  const int64_t* window_slots;
  const int64_t* lengths;
  int residual_len;
};

constexpr int kMaterializeWarps = 4;
constexpr int kMaterializeTokens = 8;  // consecutive tokens of one (row, kv head) per warp
constexpr int kMaterializeBulkCtasPerSm = 5;  // 96 registers per thread

// A warp walks kMaterializeTokens consecutive tokens of one (row, kv head): the sign vectors stay in registers, the
// codes of a token are one 2- or 4-byte load per lane where the geometry allows, and two tokens are in flight at a time
// so that the shuffles of one transform hide behind the arithmetic of the other.  The arithmetic per token is unchanged
// (same order of operations as the one-token-per-warp version it replaces), so the output is bit-identical.
template <typename T, int D, int BITS>
__global__ void __launch_bounds__(kMaterializeWarps * 32) tq_materialize_kernel(const TqMaterializeParams p) {
  constexpr int E = D / 32;
  constexpr int M = BITS - 1;
  constexpr int VS = BITS == 2 ? 2 : 4;
  __shared__ float sm_cent[1 << M];
  if (threadIdx.x < (1 << M)) sm_cent[threadIdx.x] = p.centroids[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int h = blockIdx.y;
  const int b = blockIdx.z;
  const int e0 = lane * E;
  const int64_t t0 = ((int64_t)blockIdx.x * kMaterializeWarps + warp) * kMaterializeTokens;
  if (t0 >= p.max_quantized_len) return;

  const bool dense_view = p.window != nullptr;
  int64_t len = 0, lq;
  if (dense_view) {
    // whole dense view: [0, len - R) from the pages, [len - R, len) from the ring, [len, max) zeros
    // (max_quantized_len is the padded length in this mode)
    len = max((int64_t)0, min(p.lengths[b], p.max_quantized_len));
    lq = len > p.residual_len ? len - p.residual_len : 0;
  } else {
    lq = min(p.quantized_lengths[b], p.max_quantized_len);
  }
  float s1[E], s2[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    s1[j] = p.signs1[e0 + j];
    s2[j] = p.signs2[e0 + j];
  }
  const int64_t out_base = (int64_t)b * p.out_stride_b + (int64_t)h * p.out_stride_h + e0;
  const int64_t t_end = min(t0 + kMaterializeTokens, p.max_quantized_len);

#pragma unroll 2
  for (int64_t t = t0; t < t_end; ++t) {
    T* kout = reinterpret_cast<T*>(p.key_out) + out_base + t * p.out_stride_t;
    T* vout = reinterpret_cast<T*>(p.value_out) + out_base + t * p.out_stride_t;
    if (t >= lq) {
      if (!dense_view) break;
      if (t < len) {
        const int64_t slot = p.window_slots[b];
        const int64_t rs = t % p.residual_len;
        const T* ring = reinterpret_cast<const T*>(p.window);
        lane_copy<T, E>(ring + (((slot * 2 + 0) * p.kv_heads + h) * p.residual_len + rs) * D + e0, kout);
        lane_copy<T, E>(ring + (((slot * 2 + 1) * p.kv_heads + h) * p.residual_len + rs) * D + e0, vout);
      } else {
#pragma unroll
        for (int j = 0; j < E; ++j) {
          kout[j] = ElemTraits<T>::from_float(0.0f);
          vout[j] = ElemTraits<T>::from_float(0.0f);
        }
      }
      continue;
    }
    const int64_t blk = t / p.block_size;
    const int tok = (int)(t % p.block_size);
    int32_t pid = -1;
    if (blk < p.max_blocks) pid = p.block_table[(int64_t)b * p.table_stride + blk];
    if (pid < 0 || pid >= p.num_pages) {
      if (dense_view) {  // the dense view has no holes: an unmapped block reads as zeros
#pragma unroll
        for (int j = 0; j < E; ++j) {
          kout[j] = ElemTraits<T>::from_float(0.0f);
          vout[j] = ElemTraits<T>::from_float(0.0f);
        }
      }
      continue;
    }
    const uint8_t* chunk = p.pages + ((int64_t)pid * p.kv_heads + h) * p.layout.chunk_bytes;

    // ---- keys: k_hat = norm / D * s1 * fwht( centroid[idx] + kappa * rnorm * s2 * fwht(2*sign - 1) ) ----------------
    const uint8_t* krow = chunk + p.layout.off_kcodes + tok * p.layout.key_bytes;
    float cent[E], sg[E];
    if constexpr (BITS == 4 && E == 4) {
      const uint32_t fields = reinterpret_cast<const uint16_t*>(krow)[lane];  // this lane's four nibbles
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const uint32_t field = (fields >> (4 * j)) & 0xFu;
        cent[j] = sm_cent[field & 7u];
        sg[j] = (field >> 3) ? 1.0f : -1.0f;
      }
    } else {
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const int d = e0 + j;
        uint32_t code, sbit;
        if constexpr (BITS == 4) {
          const uint32_t field = (krow[d >> 1] >> ((d & 1) * 4)) & 0xFu;
          code = field & 7u;
          sbit = field >> 3;
        } else if constexpr (BITS == 2) {
          const uint32_t field = (krow[d >> 2] >> ((d & 3) * 2)) & 3u;
          code = field & 1u;
          sbit = field >> 1;
        } else {
          code = (krow[d >> 2] >> ((d & 3) * 2)) & 3u;
          sbit = (krow[D / 4 + (d >> 3)] >> (d & 7)) & 1u;
        }
        cent[j] = sm_cent[code];
        sg[j] = sbit ? 1.0f : -1.0f;
      }
    }
    const float norm = reinterpret_cast<const float*>(chunk + p.layout.off_knorm)[tok];
    const float rnorm = reinterpret_cast<const float*>(chunk + p.layout.off_krnorm)[tok];
    warp_fwht<E>(sg, lane);
    const float coef = (1.2533141373155001f * rsqrt_dim_const<D>()) * rnorm;
#pragma unroll
    for (int j = 0; j < E; ++j) cent[j] = fmaf(coef, s2[j] < 0.0f ? -sg[j] : sg[j], cent[j]);
    warp_fwht<E>(cent, lane);
    const float scale = norm * (1.0f / (float)D);
    T kvals[E];
#pragma unroll
    for (int j = 0; j < E; ++j) kvals[j] = ElemTraits<T>::from_float(scale * (s1[j] < 0.0f ? -cent[j] : cent[j]));
    lane_copy<T, E>(kvals, kout);

    // ---- values: code * scale + zero --------------------------------------------------------------------------------
    const uint8_t* vrow = chunk + p.layout.off_vdata + tok * p.layout.value_bytes;
    const T* scales = reinterpret_cast<const T*>(chunk + p.layout.off_vscale) + tok * p.layout.groups;
    const T* zeros = reinterpret_cast<const T*>(chunk + p.layout.off_vzero) + tok * p.layout.groups;
    constexpr int kPerByte = 8 / VS;
    T vvals[E];
    if (p.value_group % E == 0) {  // one group per lane: its scale and zero point once
      const int g = e0 / p.value_group;
      const float v_scale = ElemTraits<T>::to_float(scales[g]), v_zero = ElemTraits<T>::to_float(zeros[g]);
      uint32_t codes = 0;
      if constexpr (E * VS == 16) codes = reinterpret_cast<const uint16_t*>(vrow)[lane];
      else if constexpr (E * VS == 8) codes = vrow[lane];
      else if constexpr (E * VS == 32) codes = reinterpret_cast<const uint32_t*>(vrow)[lane];
      else {
#pragma unroll
        for (int j = 0; j < E; ++j)
          codes |= ((vrow[(e0 + j) / kPerByte] >> (((e0 + j) % kPerByte) * VS)) & ((1u << VS) - 1u)) << (j * VS);
      }
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const uint32_t code = (codes >> (j * VS)) & ((1u << VS) - 1u);
        vvals[j] = ElemTraits<T>::from_float(__fadd_rn(__fmul_rn((float)code, v_scale), v_zero));
      }
    } else {
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const int d = e0 + j;
        const uint32_t code = (vrow[d / kPerByte] >> ((d % kPerByte) * VS)) & ((1u << VS) - 1u);
        const int g = d / p.value_group;
        const float prod = __fmul_rn((float)code, ElemTraits<T>::to_float(scales[g]));
        vvals[j] = ElemTraits<T>::from_float(__fadd_rn(prod, ElemTraits<T>::to_float(zeros[g])));
      }
    }
    lane_copy<T, E>(vvals, vout);
  }
}

// Walsh-Hadamard transform of a token's +-1 vector, exact in fp16 (whole numbers up to D): a register holds a pair (i, i + 8).
template <int LANES>
__device__ __forceinline__ void bulk_fwht_signs(__half2 (&s)[kBulkPairs], int lane) {
#pragma unroll
  for (int h = 1; h < kBulkPairs; h <<= 1) {
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i) {
      if ((i & h) == 0) {
        const __half2 a = s[i], b = s[i + h];
        s[i] = __hadd2(a, b);
        s[i + h] = __hsub2(a, b);
      }
    }
  }
  const __half2 halves = __floats2half2_rn(1.0f, -1.0f);
#pragma unroll
  for (int i = 0; i < kBulkPairs; ++i) s[i] = __hfma2(s[i], halves, __lowhigh2highlow(s[i]));
#pragma unroll
  for (int dl = 1; dl < LANES; dl <<= 1) {
    const __half2 sgn = __float2half2_rn((lane & dl) != 0 ? -1.0f : 1.0f);
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i) s[i] = __hfma2(s[i], sgn, __shfl_xor_sync(0xffffffffu, s[i], dl));
  }
}

// The same tokens and the same results as tq_materialize_kernel, several tokens per warp (tq_bulk.cuh), for value groups of 16
// or more and 16-byte aligned rows.  The codes of a warp's next tokens are on their way while it works on the current ones.
// That kernel is bound by its instructions, too: 8 x 2176 tokens, 4 heads of 128, 3 bits 45.1 -> 24.6 us (169 instructions per
// token-head); 64 x 2176, 8 heads, 4 bits 485 -> 233; one row of 1081 tokens, 2 heads of 256 22.5 -> 10.2.
template <typename T, int D, int BITS>
__global__ void __launch_bounds__(kBulkWarps * 32, kMaterializeBulkCtasPerSm)
    tq_materialize_bulk_kernel(const TqMaterializeParams p) {
  constexpr int kLanes = D / kBulkCoords;  // lanes per token
  constexpr int kTokens = 32 / kLanes;     // tokens per warp
  constexpr int M = BITS - 1;
  constexpr int VS = BITS == 2 ? 2 : 4;
  constexpr int KS = BITS == 4 ? 4 : 2;
  using Raw = BulkRaw<T>;
  __shared__ float sm_cent[1 << M];
  if (threadIdx.x < (1 << M)) sm_cent[threadIdx.x] = p.centroids[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int token_lane = lane & (kLanes - 1);
  const int e0 = token_lane * kBulkCoords;
  const int h = blockIdx.y;
  const int b = blockIdx.z;
  constexpr int kCtaTokens = kBulkWarps * kTokens;
  const int64_t my_token = (int)(threadIdx.x >> 5) * kTokens + lane / kLanes;
  const int64_t stride = (int64_t)gridDim.x * kCtaTokens;

  const bool dense_view = p.window != nullptr;
  int64_t len = 0, lq;
  if (dense_view) {
    len = max((int64_t)0, min(p.lengths[b], p.max_quantized_len));
    lq = len > p.residual_len ? len - p.residual_len : 0;
  } else {
    lq = min(p.quantized_lengths[b], p.max_quantized_len);
  }
  uint64_t sign1[kBulkPairs], sign2[kBulkPairs];
#pragma unroll
  for (int i = 0; i < kBulkPairs; ++i) {
    sign1[i] = pair_of(p.signs1[e0 + i] < 0.0f ? -1.0f : 1.0f, p.signs1[e0 + i + kBulkPairs] < 0.0f ? -1.0f : 1.0f);
    sign2[i] = pair_of(p.signs2[e0 + i] < 0.0f ? -1.0f : 1.0f, p.signs2[e0 + i + kBulkPairs] < 0.0f ? -1.0f : 1.0f);
  }
  const int64_t out_base = (int64_t)b * p.out_stride_b + (int64_t)h * p.out_stride_h + e0;
  const int group = e0 / p.value_group;

  struct Codes {
    uint32_t field[BulkFields<KS>::kWords], sign_field[1], vfield[BulkFields<VS>::kWords];
    float norm, rnorm, v_scale, v_zero;
    bool packed;
  };
  // packed tokens of the lanes that have one; the others read nothing
  auto load_codes = [&](int64_t t, Codes& c) {
    int32_t pid = -1;
    int tok = 0;
    if (t < lq) {
      const int64_t blk = t / p.block_size;
      tok = (int)(t - blk * p.block_size);
      if (blk < p.max_blocks) pid = p.block_table[(int64_t)b * p.table_stride + blk];
    }
    c.packed = pid >= 0 && pid < p.num_pages;
    if (!c.packed) return;
    const uint8_t* chunk = p.pages + ((int64_t)pid * p.kv_heads + h) * p.layout.chunk_bytes;
    const uint8_t* krow = chunk + p.layout.off_kcodes + tok * p.layout.key_bytes;
    BulkFields<KS>::load(krow, token_lane, c.field);
    if constexpr (BITS == 3) BulkFields<1>::load(krow + D / 4, token_lane, c.sign_field);
    BulkFields<VS>::load(chunk + p.layout.off_vdata + tok * p.layout.value_bytes, token_lane, c.vfield);
    c.norm = reinterpret_cast<const float*>(chunk + p.layout.off_knorm)[tok];
    c.rnorm = reinterpret_cast<const float*>(chunk + p.layout.off_krnorm)[tok];
    c.v_scale = ElemTraits<T>::to_float((reinterpret_cast<const T*>(chunk + p.layout.off_vscale) + tok * p.layout.groups)[group]);
    c.v_zero = ElemTraits<T>::to_float((reinterpret_cast<const T*>(chunk + p.layout.off_vzero) + tok * p.layout.groups)[group]);
  };
  Codes next = {};
  load_codes((int64_t)blockIdx.x * kCtaTokens + my_token, next);

  for (int64_t base = (int64_t)blockIdx.x * kCtaTokens; base < p.max_quantized_len; base += stride) {  // the same in all lanes
    const int64_t t = base + my_token;
    T* kout = reinterpret_cast<T*>(p.key_out) + out_base + t * p.out_stride_t;
    T* vout = reinterpret_cast<T*>(p.value_out) + out_base + t * p.out_stride_t;
    const Codes now = next;
    load_codes(t + stride, next);
    if (!now.packed && dense_view && t < p.max_quantized_len) {
      Raw key, val;
      if (t >= lq && t < len) {
        const int64_t slot = p.window_slots[b];
        const int64_t rs = t % p.residual_len;
        const T* ring = reinterpret_cast<const T*>(p.window) + e0;
        key.load(ring + (((slot * 2 + 0) * p.kv_heads + h) * p.residual_len + rs) * D);
        val.load(ring + (((slot * 2 + 1) * p.kv_heads + h) * p.residual_len + rs) * D);
      } else {  // padding, and holes of the block table
#pragma unroll
        for (int k = 0; k < Raw::kWords; ++k) key.w[k] = val.w[k] = 0u;
      }
      key.store(kout);
      val.store(vout);
    }
    // the exchanges below take the whole warp: lanes without a packed token go along and store nothing
    if (!__any_sync(0xffffffffu, now.packed)) continue;

    // ---- keys: k_hat = norm / D * s1 * fwht( centroid[idx] + kappa * rnorm * s2 * fwht(2*sign - 1) ) ----------------
    __half2 sg[kBulkPairs];
    uint64_t w[kBulkPairs];
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i) {
      uint32_t c_lo, c_hi, s_lo, s_hi;
      if constexpr (BITS == 4) {
        c_lo = now.field[0] >> (4 * i), c_hi = now.field[BulkFields<KS>::kWords - 1] >> (4 * i);
        s_lo = c_lo >> 3, s_hi = c_hi >> 3;
      } else {
        c_lo = now.field[0] >> (2 * i), c_hi = now.field[0] >> (16 + 2 * i);
        if constexpr (BITS == 2) s_lo = c_lo >> 1, s_hi = c_hi >> 1;
        else s_lo = now.sign_field[0] >> i, s_hi = now.sign_field[0] >> (8 + i);
      }
      w[i] = pair_of(sm_cent[c_lo & ((1u << M) - 1u)], sm_cent[c_hi & ((1u << M) - 1u)]);
      const uint32_t bits = 0xBC00BC00u ^ ((s_lo & 1u) << 15) ^ (s_hi << 31);  // -1 where the sign bit is clear
      sg[i] = *reinterpret_cast<const __half2*>(&bits);
    }
    bulk_fwht_signs<kLanes>(sg, lane);
    const float coef = (1.2533141373155001f * rsqrt_dim_const<D>()) * now.rnorm;
    const uint64_t coef2 = pair_of(coef, coef);
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i)
      w[i] = fma_pair(coef2, mul_pair(pair_of(__low2float(sg[i]), __high2float(sg[i])), sign2[i]), w[i]);
    bulk_fwht<kLanes>(w, lane);
    const float scale = now.norm * (1.0f / (float)D);
    const uint64_t scale2 = pair_of(scale, scale);
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i) w[i] = mul_pair(scale2, mul_pair(w[i], sign1[i]));
    auto put = [&](T* out) {
      Raw r;
#pragma unroll
      for (int i = 0; i < kBulkPairs; i += 2) {
        float a, b2, c, d;
        halves_of(w[i], a, c);
        halves_of(w[i + 1], b2, d);
        r.set(i, a, b2);
        r.set(i + kBulkPairs, c, d);
      }
      r.store(out);
    };
    if (now.packed) put(kout);

    // ---- values: code * scale + zero; a code under the exponent of 2^23 reads as 2^23 + code ------------------------
    const uint64_t vscale2 = pair_of(now.v_scale, now.v_scale), vzero2 = pair_of(now.v_zero, now.v_zero), bias2 = pair_of(-8388608.0f, -8388608.0f);
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i) {
      constexpr uint32_t kCode = (1u << VS) - 1u;
      const uint32_t lo = now.vfield[0] >> (VS * i);
      const uint32_t hi = VS == 4 ? now.vfield[BulkFields<VS>::kWords - 1] >> (VS * i) : now.vfield[0] >> (16 + VS * i);
      const uint64_t code = add_pair(pair_of(__uint_as_float((lo & kCode) | 0x4B000000u), __uint_as_float((hi & kCode) | 0x4B000000u)), bias2);
      w[i] = add_pair(mul_pair_rounded(code, vscale2), vzero2);
    }
    if (now.packed) put(vout);
  }
}

}  // namespace anna

using namespace anna;

static int launch_materialize(TqMaterializeParams p, int batch, int kv_heads, int head_dim, int block_size, int bits,
                              int value_group, int dtype, cudaStream_t stream) {
  if (!tq_make_layout(head_dim, bits, block_size, dtype_bytes_of(dtype), value_group, &p.layout))
    return set_error(ANNA_ERR_INVALID, "TurboQuant materialize: unsupported geometry D=%d bits=%d S=%d group=%d", head_dim,
                     bits, block_size, value_group);
  const int64_t row_bytes = dtype_bytes_of(dtype);
  const size_t access = lane_access_bytes(head_dim, (int)row_bytes);
  auto steps_aligned = [&](int64_t stride, int64_t count) { return count <= 1 || stride * row_bytes % (int64_t)access == 0; };
  ANNA_REQUIRE(aligned_to(p.key_out, access) && aligned_to(p.value_out, access) && aligned_to(p.window, access) && aligned_to(p.pages, 4) &&
                   steps_aligned(p.out_stride_b, batch) && steps_aligned(p.out_stride_h, kv_heads) &&
                   steps_aligned(p.out_stride_t, p.max_quantized_len),
               "TurboQuant materialize: outputs, their strides and the window must be aligned to %d bytes, pages to 4", (int)access);
  const int64_t per_cta = (int64_t)kMaterializeWarps * kMaterializeTokens;
  dim3 grid((unsigned)((p.max_quantized_len + per_cta - 1) / per_cta), (unsigned)kv_heads, (unsigned)batch);
  // the bulk kernel's lanes move 16 bytes of dense rows, 8 of packed ones, and hold 16 values of one group
  const bool bulk = value_group >= kBulkCoords && aligned_to(p.key_out, 16) && aligned_to(p.value_out, 16) &&
                    aligned_to(p.window, 16) && aligned_to(p.pages, 8) && p.out_stride_b * row_bytes % 16 == 0 &&
                    p.out_stride_h * row_bytes % 16 == 0 && p.out_stride_t * row_bytes % 16 == 0;
  return ANNA_DISPATCH_DTYPE(dtype, T, [&]() -> int {
    return ANNA_DISPATCH_TQ_DIM(head_dim, D, [&]() -> int {
      return ANNA_DISPATCH_TQ_BITS(bits, BITS, [&]() -> int {
        if (bulk) {
          static int resident[64] = {};
          int device = 0, ctas = 0;
          ANNA_CUDA_CHECK(cudaGetDevice(&device));
          const int rc = bulk_resident_ctas(tq_materialize_bulk_kernel<T, D, BITS>, kBulkWarps * 32, resident, device, &ctas);
          if (rc != ANNA_OK) return rc;
          constexpr int kCtaTokens = kBulkWarps * (32 * kBulkCoords / D);
          const int chunks = bulk_chunks((int64_t)kv_heads * batch, (p.max_quantized_len + kCtaTokens - 1) / kCtaTokens, ctas);
          tq_materialize_bulk_kernel<T, D, BITS><<<dim3((unsigned)chunks, (unsigned)kv_heads, (unsigned)batch), kBulkWarps * 32, 0,
                                                   stream>>>(p);
          return check_launch("tq_materialize_bulk_kernel");
        }
        tq_materialize_kernel<T, D, BITS><<<grid, kMaterializeWarps * 32, 0, stream>>>(p);
        return check_launch("tq_materialize_kernel");
      });
    });
  });
}

extern "C" int anna_tq_gather_dense(const uint8_t* packed_pages, const int32_t* block_table, int64_t table_stride,
                                    const void* window, const int64_t* window_slots, const int64_t* lengths,
                                    const float* signs1, const float* signs2, const float* centroids, void* key_out,
                                    void* value_out, int64_t out_stride_b, int64_t out_stride_h, int64_t out_stride_t,
                                    int batch, int kv_heads, int head_dim, int block_size, int residual_len, int bits,
                                    int value_group, int64_t num_pages, int64_t max_blocks, int64_t max_len, int dtype,
                                    anna_stream_t stream) {
  ANNA_REQUIRE(window && window_slots && lengths && signs1 && signs2 && centroids && key_out && value_out,
               "anna_tq_gather_dense: null pointer argument");
  ANNA_REQUIRE(packed_pages != nullptr || num_pages == 0, "anna_tq_gather_dense: null page pool with num_pages > 0");
  ANNA_REQUIRE(block_table != nullptr || max_blocks == 0, "anna_tq_gather_dense: null block table with max_blocks > 0");
  ANNA_REQUIRE(batch > 0 && kv_heads > 0 && block_size >= 1 && residual_len >= 1 && max_len >= 0,
               "anna_tq_gather_dense: sizes must be positive");
  if (max_len == 0) return ANNA_OK;
  TqMaterializeParams p{};
  p.pages = packed_pages; p.block_table = block_table; p.table_stride = table_stride;
  p.signs1 = signs1; p.signs2 = signs2; p.centroids = centroids;
  p.key_out = key_out; p.value_out = value_out;
  p.out_stride_b = out_stride_b; p.out_stride_h = out_stride_h; p.out_stride_t = out_stride_t;
  p.kv_heads = kv_heads; p.block_size = block_size; p.value_group = value_group;
  p.num_pages = num_pages; p.max_blocks = max_blocks; p.max_quantized_len = max_len;
  p.window = window; p.window_slots = window_slots; p.lengths = lengths; p.residual_len = residual_len;
  return launch_materialize(p, batch, kv_heads, head_dim, block_size, bits, value_group, dtype, (cudaStream_t)stream);
}

extern "C" int anna_tq_materialize(const uint8_t* packed_pages, const int32_t* block_table, int64_t table_stride,
                                   const int64_t* quantized_lengths, const float* signs1, const float* signs2,
                                   const float* centroids, void* key_out, void* value_out, int64_t out_stride_b,
                                   int64_t out_stride_h, int64_t out_stride_t, int batch, int kv_heads, int head_dim,
                                   int block_size, int bits, int value_group, int64_t num_pages, int64_t max_blocks,
                                   int64_t max_quantized_len, int dtype, anna_stream_t stream) {
  ANNA_REQUIRE(packed_pages && block_table && quantized_lengths && signs1 && signs2 && centroids && key_out && value_out,
               "anna_tq_materialize: null pointer argument");
  ANNA_REQUIRE(batch > 0 && kv_heads > 0 && block_size >= 1 && max_quantized_len >= 0,
               "anna_tq_materialize: sizes must be positive");
  if (max_quantized_len == 0) return ANNA_OK;
  TqMaterializeParams p{};
  p.pages = packed_pages; p.block_table = block_table; p.table_stride = table_stride;
  p.quantized_lengths = quantized_lengths; p.signs1 = signs1; p.signs2 = signs2; p.centroids = centroids;
  p.key_out = key_out; p.value_out = value_out;
  p.out_stride_b = out_stride_b; p.out_stride_h = out_stride_h; p.out_stride_t = out_stride_t;
  p.kv_heads = kv_heads; p.block_size = block_size; p.value_group = value_group;
  p.num_pages = num_pages; p.max_blocks = max_blocks; p.max_quantized_len = max_quantized_len;
  return launch_materialize(p, batch, kv_heads, head_dim, block_size, bits, value_group, dtype, (cudaStream_t)stream);
}
