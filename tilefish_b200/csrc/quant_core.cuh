// Per-thread core of the BlockScaled quantizers: one thread owns 8 consecutive bf16 values (one 128-bit load); the
// 4 (block 32) or 2 (block 16) adjacent lanes that share a scale block combine their maxima with warp shuffles.
//
// Every arithmetic step is a single correctly rounded f32 operation or an integer operation, in a fixed order, so the
// bytes are the same as the torch restatement's:
//   MX     amax on the 15 magnitude bits; E = amax >> 7; scale = amax == 0 ? 127 : max(E - emax, 0);
//          code = cast(f32(x) * 2^(127 - scale))                      (exact product)
//   NVFP4  s8 = e4m3(amax * (1 / (6 * gs))); d = f32(s8) * gs; code = e2m1(f32(x) * (1 / d)); zero when gs == 0 or d == 0
#pragma once

#include "common.cuh"

namespace tf {

// Maximum of the 15 magnitude bits of the 8 bf16 words of v (packed 16-bit unsigned maxima, then the two halves).
__device__ __forceinline__ uint32_t amax_bits8(const uint4& v) {
  const uint32_t k = 0x7FFF7FFFu;
  uint32_t t = __vimax3_u16x2(v.x & k, v.y & k, v.z & k);
  t = __vimax3_u16x2(t, v.w & k, 0u);
  return max(t & 0xFFFFu, t >> 16);
}

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// Quantizes the 8 bf16 values of `v`. All 32 lanes of the warp must call it together (lanes without data pass zeros).
// Returns the packed codes in c0 (and c1 for 8-bit elements) and the scale byte of the lane's block.
// nvfp4: gs is the tensor's global scale and inv_t = 1 / (6 * gs), both uniform over the kernel.
template <int FMT>
__device__ __forceinline__ void quantize_vec8(const uint4& v, float gs, float inv_t, uint32_t& c0, uint32_t& c1, uint32_t& scale) {
  uint32_t m = amax_bits8(v);
  m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
  if (FMT != TF_FMT_NVFP4) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));

  if (FMT == TF_FMT_NVFP4) {
    const float amax = __uint_as_float(m << 16);
    uint32_t s8 = 0;
    if (gs != 0.0f && m != 0) s8 = cvt_e4m3x2(__fmul_rn(amax, inv_t), 0.0f) & 0xFFu;
    const float d = __fmul_rn(e4m3_to_f32(s8), gs);
    const bool zero = (d == 0.0f);
    const float inv = zero ? 0.0f : __frcp_rn(d);
    scale = s8;
    c0 = cvt_e2m1x8(__fmul_rn(bf16lo_to_f32(v.x), inv), __fmul_rn(bf16hi_to_f32(v.x), inv), __fmul_rn(bf16lo_to_f32(v.y), inv),
                    __fmul_rn(bf16hi_to_f32(v.y), inv), __fmul_rn(bf16lo_to_f32(v.z), inv), __fmul_rn(bf16hi_to_f32(v.z), inv),
                    __fmul_rn(bf16lo_to_f32(v.w), inv), __fmul_rn(bf16hi_to_f32(v.w), inv));
    if (zero) c0 = 0;
    c1 = 0;
    return;
  }

  const int emax = (FMT == TF_FMT_MXFP8) ? 8 : 2;
  const int e = (int)(m >> 7) - emax;
  scale = (m == 0) ? 127u : (uint32_t)max(e, 0);
  // 2^(127 - scale) as two packed bf16: a power of two times a bf16 is exact in bf16 (a result below the normal range loses
  // bits, but it is then far below half of the smallest code and becomes a signed zero either way)
  const uint32_t inv1 = (254u - scale) << 7;
  const uint32_t inv2 = inv1 | (inv1 << 16);
  const uint32_t q0 = mul_bf16x2(v.x, inv2), q1 = mul_bf16x2(v.y, inv2), q2 = mul_bf16x2(v.z, inv2), q3 = mul_bf16x2(v.w, inv2);
  if (FMT == TF_FMT_MXFP8) {
    c0 = cvt_e4m3x4(bf16lo_to_f32(q0), bf16hi_to_f32(q0), bf16lo_to_f32(q1), bf16hi_to_f32(q1));
    c1 = cvt_e4m3x4(bf16lo_to_f32(q2), bf16hi_to_f32(q2), bf16lo_to_f32(q3), bf16hi_to_f32(q3));
  } else {
    c0 = cvt_e2m1x8(bf16lo_to_f32(q0), bf16hi_to_f32(q0), bf16lo_to_f32(q1), bf16hi_to_f32(q1), bf16lo_to_f32(q2), bf16hi_to_f32(q2),
                    bf16lo_to_f32(q3), bf16hi_to_f32(q3));
    c1 = 0;
  }
}

// nvfp4: the reciprocal of a block scale, 1 / (f32(s8) * gs), or kZeroBlock where that product is zero (no reciprocal has these bits: a NaN result is canonical).
constexpr uint32_t kZeroBlock = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t nvfp4_inverse(uint32_t s8, float gs) {
  const float d = __fmul_rn(e4m3_to_f32(s8), gs);
  return d == 0.0f ? kZeroBlock : __float_as_uint(__frcp_rn(d));
}
// (a.lo * b, a.hi * b) of the two bf16 of `w`, as two f32.
__device__ __forceinline__ void mul_bf16_pair(uint32_t w, float b, float& lo, float& hi) {
  asm("{ .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n mul.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x; }"
      : "=f"(lo), "=f"(hi)
      : "f"(bf16lo_to_f32(w)), "f"(bf16hi_to_f32(w)), "f"(b));
}

// 16 consecutive bf16 values per thread (one 256-bit load): half the shuffles, scale arithmetic and address arithmetic per element
// of the 8-value form. A block of 32 is two adjacent lanes; an nvfp4 block of 16 is the thread's own. Same arithmetic, same bytes.
// codes: 4 words (e4m3) or 2 words (e2m1). nvfp4: gs, inv_t = 1 / (6 * gs), and where there is one the table of nvfp4_inverse for gs.
template <int FMT>
__device__ __forceinline__ void quantize_vec16(const uint32_t (&w)[8], float gs, float inv_t, uint32_t (&codes)[4], uint32_t& scale, const uint32_t* inverses = nullptr) {
  const uint32_t k = 0x7FFF7FFFu;
  uint32_t t0 = __vimax3_u16x2(w[0] & k, w[1] & k, w[2] & k);
  uint32_t t1 = __vimax3_u16x2(w[3] & k, w[4] & k, w[5] & k);
  t0 = __vimax3_u16x2(t0, w[6] & k, w[7] & k);
  t0 = __vimax3_u16x2(t0, t1, 0u);
  uint32_t m = max(t0 & 0xFFFFu, t0 >> 16);
  if (FMT != TF_FMT_NVFP4) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));

  if (FMT == TF_FMT_NVFP4) {
    const float amax = __uint_as_float(m << 16);
    uint32_t s8 = 0;
    if (gs != 0.0f && m != 0) s8 = cvt_e4m3x2(__fmul_rn(amax, inv_t), 0.0f) & 0xFFu;
    const uint32_t bits = inverses ? inverses[s8 & 127u] : nvfp4_inverse(s8, gs);
    const float inv = __uint_as_float(bits);
    scale = s8;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float f[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) mul_bf16_pair(w[4 * h + j], inv, f[2 * j], f[2 * j + 1]);
      codes[h] = bits == kZeroBlock ? 0u : cvt_e2m1x8(f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
    }
    codes[2] = codes[3] = 0;
    return;
  }
  const int emax = (FMT == TF_FMT_MXFP8) ? 8 : 2;
  const int e = (int)(m >> 7) - emax;
  scale = (m == 0) ? 127u : (uint32_t)max(e, 0);
  const uint32_t inv1 = (254u - scale) << 7;
  const uint32_t inv2 = inv1 | (inv1 << 16);
  uint32_t q[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) q[j] = mul_bf16x2(w[j], inv2);
  if (FMT == TF_FMT_MXFP8) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      codes[j] = cvt_e4m3x4(bf16lo_to_f32(q[2 * j]), bf16hi_to_f32(q[2 * j]), bf16lo_to_f32(q[2 * j + 1]), bf16hi_to_f32(q[2 * j + 1]));
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      codes[h] = cvt_e2m1x8(bf16lo_to_f32(q[4 * h]), bf16hi_to_f32(q[4 * h]), bf16lo_to_f32(q[4 * h + 1]), bf16hi_to_f32(q[4 * h + 1]),
                            bf16lo_to_f32(q[4 * h + 2]), bf16hi_to_f32(q[4 * h + 2]), bf16lo_to_f32(q[4 * h + 3]), bf16hi_to_f32(q[4 * h + 3]));
    codes[2] = codes[3] = 0;
  }
}

// Zeroes the padding of a swizzled scale tensor: the rows past `rows` of the last row tile and the columns past `cols` of the last
// column tile. Thread `first` of `stride` threads that share the work. The bytes are disjoint from the scales, so no ordering is
// needed; a kernel that writes scales does this itself instead of a memset of the whole tensor in front of it (measured in captured
// graphs: the README block at one row 26.1 -> 25.0 us, its NVFP4 form at 16 rows 28.7 -> 26.7). One item of the
// row padding is 16 contiguous bytes (the four row groups of one tile row), so a tensor of one row and 2560 columns takes two stores
// per thread of a single block. `scales` is 16-byte aligned.
constexpr unsigned kPadBlocks = 8;  // a launch that pads has at least this many blocks to share the work
// COLUMNS = false: the columns are written with the row's scales (store_quantized_words): the rmsnorm kernel passes tens of megabytes
// through L2 before it comes to the later rows, whose sectors a sweep at the start would leave half written for that long (with an mxfp4 copy,
// 16026 x 1504: 61.2 us with the sweep, 54.2 with the columns behind each row, 57.2 with the memset).
template <bool COLUMNS = true>
__device__ __forceinline__ void zero_scale_padding(uint8_t* __restrict__ scales, int64_t rows, int64_t cols, int64_t first, int64_t stride) {
  const int64_t n_ct = (cols + 3) >> 2;
  const int used = (int)(rows & 127);  // rows of the last row tile that hold scales; 0: all of them
  if (used) {
    uint8_t* tiles = scales + (rows >> 7) * n_ct * 512;
    for (int64_t i = first; i < n_ct * 32; i += stride) {
      const int rr = (int)(i & 31);
      uint32_t* p = reinterpret_cast<uint32_t*>(tiles + i * 16);
      if (rr >= used) {
        *reinterpret_cast<uint4*>(p) = make_uint4(0, 0, 0, 0);
      } else {
        for (int g = 1; g < 4; ++g)
          if (g * 32 + rr >= used) p[g] = 0u;
      }
    }
  }
  if (COLUMNS && (cols & 3)) {
    for (int64_t r = first; r < rows; r += stride)
      for (int64_t c = cols; c < n_ct * 4; ++c) scales[swizzled_scale_offset(r, c, n_ct)] = 0;
  }
}

// Scales of row `row` as the bytes of `word`: columns col .. col + 3 (col a multiple of 4), or with `pair` col and col + 1 (col even). WORDS: swizzled
// scales that can be stored as words; else byte by byte in either layout (a template: the short row kernels run from a cold instruction
// cache, and the branches over the byte stores cost the README block at 1 and 512 rows 0.3 and 0.6 us). real: the row is one of the tensor's
// (the swizzled layout has more).
template <bool WORDS>
__device__ __forceinline__ void store_scale_word(uint8_t* __restrict__ scales, int layout, int64_t row, int col, int cols, int n_ct, bool real, uint32_t word,
                                                 bool pair = false) {
  if (WORDS) {
    uint8_t* dst = scales + swizzled_scale_offset(row, col, n_ct);
    if (pair) *reinterpret_cast<uint16_t*>(dst) = (uint16_t)word;
    else *reinterpret_cast<uint32_t*>(dst) = word;
    return;
  }
  uint8_t* dst = scales + (layout == TF_SCALES_PLAIN ? row * cols + col : swizzled_scale_offset(row, col, n_ct));
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if ((b < 2 || !pair) && (layout == TF_SCALES_SWIZZLED || (real && col + b < cols))) dst[b] = (uint8_t)(word >> (8 * b));
}
inline bool scales_as_words(const void* scales, int layout) { return layout == TF_SCALES_SWIZZLED && reinterpret_cast<uintptr_t>(scales) % 4 == 0; }

// One thread's codes of 8 elements (vector `vec` of row `row`), and the scales of a row's column tile as one word of the swizzled layout, the zeros of
// its padding columns included. All 32 lanes call it together, with consecutive vectors from a multiple of 32 on; `has`: this lane has data.
template <int FMT, bool WORDS>
__device__ __forceinline__ void store_quantized_words(uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, int layout, bool has, int64_t row, int vec, int d,
                                                      uint32_t c0, uint32_t c1, uint32_t scale) {
  constexpr int kLanes = (FMT == TF_FMT_NVFP4) ? 2 : 4;  // of one block
  uint32_t word = has ? scale << (8 * ((vec / kLanes) & 3)) : 0u;
  word |= __shfl_xor_sync(0xFFFFFFFFu, word, kLanes);
  word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2 * kLanes);
  if (!has) return;
  if (FMT == TF_FMT_MXFP8) *reinterpret_cast<uint2*>(codes + row * d + (int64_t)vec * 8) = make_uint2(c0, c1);
  else *reinterpret_cast<uint32_t*>(codes + row * (d >> 1) + (int64_t)vec * 4) = c0;
  if ((vec & (4 * kLanes - 1)) == 0) {
    const int cols = (d >> 3) / kLanes, col = vec / kLanes;
    store_scale_word<WORDS>(scales, layout, row, col, cols, (cols + 3) >> 2, true, word);
  }
}

// Stores one thread's codes (8 elements starting at element column `col` of row `row`) and, from the first lane of each
// block, the scale byte. `vec` is the index of the 8-element vector inside the row.
template <int FMT>
__device__ __forceinline__ void store_quantized(uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, int swizzled,
                                                int64_t row, int vec, int64_t k, uint32_t c0, uint32_t c1, uint32_t scale) {
  if (FMT == TF_FMT_MXFP8) {
    *reinterpret_cast<uint2*>(codes + row * k + (int64_t)vec * 8) = make_uint2(c0, c1);
  } else {
    *reinterpret_cast<uint32_t*>(codes + row * (k >> 1) + (int64_t)vec * 4) = c0;
  }
  const int lanes_per_block = (FMT == TF_FMT_NVFP4) ? 2 : 4;
  if ((vec & (lanes_per_block - 1)) == 0) {
    const int blk = (FMT == TF_FMT_NVFP4) ? 16 : 32;
    const int64_t cols = k / blk;
    const int64_t c = vec / lanes_per_block;
    const int64_t off = swizzled ? swizzled_scale_offset(row, c, (cols + 3) >> 2) : row * cols + c;
    scales[off] = (uint8_t)scale;
  }
}

}  // namespace tf
