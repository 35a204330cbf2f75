// The reference's other expert formats: IQ3_XXS, IQ2_S and IQ4_XS as gate/up formats (256-weight super-blocks, paired with
// Q8_K activations) and Q2_0 as a down format (64-weight blocks, paired with Q8_0), src/kernels/moe/iq_device.cuh:171-288
// and third_party/ggml-iq/ggml-iq.h:26-78 of the reference: codebooks, which the streaming kernel
// (moe_decode_experts.cuh) uses too, and the dequantization probe's decoders. Included by moe_decode.cu and probes.cu.
// (No namespace of its own: included inside namespace fb's unnamed namespace, once per translation unit.)
#pragma once

static __constant__ uint16_t c_iq3xxs_grid_packed[256] = {FB_IQ3XXS_GRID_PACKED};
static __constant__ uint16_t c_iq2s_grid_packed[1024] = {FB_IQ2S_GRID_PACKED};

constexpr int kGenericGridWords = 2048;  // shared-memory words the largest expanded codebook takes (IQ2_S: 1024 x 8 bytes)

__device__ __forceinline__ uint32_t iq3xxs_expand(uint32_t p) {
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t c = (p >> (3 * j)) & 7u;
    w |= (4u + 8u * c + (c == 7u ? 2u : 0u)) << (8 * j);  // 4, 12, ..., 52, 62
  }
  return w;
}

__device__ __forceinline__ uint2 iq2s_expand(uint32_t p) {
  uint32_t w[2] = {0, 0};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t c = (p >> (2 * j)) & 3u;
    w[j >> 2] |= (c == 0u ? 8u : c == 1u ? 25u : 43u) << (8 * (j & 3));
  }
  return make_uint2(w[0], w[1]);
}

// Expands the format's codebook into shared memory (called by every thread; caller synchronizes).
// IQ3_XXS: 256 words of four magnitudes; IQ2_S: 1024 pairs of words of four magnitudes each.
template <int FMT>
__device__ __forceinline__ void generic_grid_fill(uint32_t* grid) {
  if constexpr (FMT == FB_FMT_IQ3_XXS) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) grid[i] = iq3xxs_expand(c_iq3xxs_grid_packed[i]);
  } else if constexpr (FMT == FB_FMT_IQ2_S) {
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) reinterpret_cast<uint2*>(grid)[i] = iq2s_expand(c_iq2s_grid_packed[i]);
  }
}

__device__ __forceinline__ uint32_t ld_u16(const uint8_t* p) { return uint32_t(p[0]) | (uint32_t(p[1]) << 8); }
__device__ __forceinline__ uint32_t ld_u32_unaligned(const uint8_t* p) {  // two-byte aligned
  return ld_u16(p) | (ld_u16(p + 2) << 16);
}
__device__ __forceinline__ float fp16_bits(uint32_t h) { return __half2float(__ushort_as_half(static_cast<unsigned short>(h))); }
// bit j of an 8-bit sign pattern -> byte j = 0xFF: bits 0-3 into the first word, 4-7 into the second
__device__ __forceinline__ int sign_bytes(uint32_t s4) {
  return int(__vcmpne4((s4 * 0x00204081u) & 0x01010101u, 0u));  // bit j of the nibble at position 8j
}
__device__ __forceinline__ int apply_sign(uint32_t mag, int mask) { return int(__vsub4(mag ^ uint32_t(mask), uint32_t(mask))); }

// One 32-weight sub-block, decoded: q[0..3] = weights 0..15, q[4..7] = weights 16..31 (int8 x 4 per word),
// integer multipliers of the two halves and the float factor.
struct Sub32 {
  int q[8];
  int m0, m1;
  float d;
};

// `row` = the weight row, `sub` = index of the 32-weight sub-block inside it.
template <int FMT>
__device__ __forceinline__ void decode_sub32(const uint8_t* row, int sub, const uint32_t* grid, Sub32& s) {
  if constexpr (FMT == FB_FMT_IQ3_XXS) {
    const uint8_t* b = row + (sub >> 3) * 98;
    const int ib = sub & 7;
    const uint8_t* qs = b + 2 + 8 * ib;
    const uint32_t aux = ld_u32_unaligned(b + 2 + 64 + 4 * ib);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t idx7 = (aux >> (7 * l)) & 127u;
      const uint32_t sg = idx7 | ((__popc(idx7) & 1u) << 7);  // the sign pattern: index + parity bit
      s.q[2 * l] = apply_sign(grid[qs[2 * l]], sign_bytes(sg & 15u));
      s.q[2 * l + 1] = apply_sign(grid[qs[2 * l + 1]], sign_bytes(sg >> 4));
    }
    s.m0 = s.m1 = 2 * int(aux >> 28) + 1;
    s.d = fp16_bits(ld_u16(b)) * 0.25f;
  } else if constexpr (FMT == FB_FMT_IQ2_S) {
    const uint8_t* b = row + (sub >> 3) * 82;
    const int ib = sub & 7;
    const uint8_t* qs = b + 2 + 4 * ib;
    const uint8_t* sg = b + 2 + 32 + 4 * ib;
    const uint32_t qh = b[2 + 64 + ib];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t idx = uint32_t(qs[l]) | ((qh << (8 - 2 * l)) & 0x300u);
      s.q[2 * l] = apply_sign(grid[2 * idx], sign_bytes(uint32_t(sg[l]) & 15u));
      s.q[2 * l + 1] = apply_sign(grid[2 * idx + 1], sign_bytes(uint32_t(sg[l]) >> 4));
    }
    const uint32_t sc = b[2 + 64 + 8 + ib];
    s.m0 = 2 * int(sc & 15u) + 1;
    s.m1 = 2 * int(sc >> 4) + 1;
    s.d = fp16_bits(ld_u16(b)) * 0.125f;
  } else if constexpr (FMT == FB_FMT_IQ4_XS) {
    const uint8_t* b = row + (sub >> 3) * 136;
    const int ib = sub & 7;
    const uint8_t* qs = b + 8 + 16 * ib;  // 8-byte header: d, scales_h, scales_l[4]
    constexpr int lv[16] = {FB_IQ4NL_LEVELS};
    auto level = [&](uint32_t n) -> uint32_t {  // 16-way select on a nibble (registers only)
      int v = lv[0];
#pragma unroll
      for (int i = 1; i < 16; ++i) v = n == uint32_t(i) ? lv[i] : v;
      return uint32_t(v) & 0xFFu;
    };
#pragma unroll
    for (int wv = 0; wv < 4; ++wv) {
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t byte = qs[4 * wv + j];
        lo |= level(byte & 15u) << (8 * j);
        hi |= level(byte >> 4) << (8 * j);
      }
      s.q[wv] = int(lo);      // weights 4wv .. 4wv+3
      s.q[4 + wv] = int(hi);  // weights 16 + 4wv ..
    }
    const uint32_t sl = b[4 + (ib >> 1)], sh = ld_u16(b + 2);
    const int ls = int(((sl >> (4 * (ib & 1))) & 15u) | (((sh >> (2 * ib)) & 3u) << 4));
    s.m0 = s.m1 = ls - 32;
    s.d = fp16_bits(ld_u16(b));
  } else {  // Q2_0: the sub-block is half of a 64-weight block; weights in natural order
    const uint8_t* b = row + (sub >> 1) * 18;
    const uint8_t* qs = b + 2 + 8 * (sub & 1);
#pragma unroll
    for (int wv = 0; wv < 8; ++wv) {
      const uint32_t c = qs[wv];  // four 2-bit codes, lowest first
      const uint32_t x = (c & 3u) | ((c & 0xCu) << 6) | ((c & 0x30u) << 12) | ((c & 0xC0u) << 18);
      s.q[wv] = int(__vsub4(x, 0x01010101u));
    }
    s.m0 = s.m1 = 1;
    s.d = fp16_bits(ld_u16(b));
  }
}

// Exact fp32 values of the sub-block's 32 weights in ggml's own operation order
// (third_party/ggml-iq/ggml-iq.c:135-152, 171-229, 290-311), for the bit-exact dequantization probe.
template <int FMT>
__device__ __forceinline__ void dequant_sub32(const uint8_t* row, int sub, const uint32_t* grid, float* y) {
  Sub32 s;
  decode_sub32<FMT>(row, sub, grid, s);
  float d0, d1;
  if constexpr (FMT == FB_FMT_IQ3_XXS) {
    const float d = fp16_bits(ld_u16(row + (sub >> 3) * 98));
    d0 = d1 = d * (0.5f + float((s.m0 - 1) / 2)) * 0.5f;
  } else if constexpr (FMT == FB_FMT_IQ2_S) {
    const float d = fp16_bits(ld_u16(row + (sub >> 3) * 82));
    d0 = d * (0.5f + float((s.m0 - 1) / 2)) * 0.25f;
    d1 = d * (0.5f + float((s.m1 - 1) / 2)) * 0.25f;
  } else if constexpr (FMT == FB_FMT_IQ4_XS) {
    d0 = d1 = s.d * float(s.m0);
  } else {
    d0 = d1 = s.d;
  }
#pragma unroll
  for (int wv = 0; wv < 8; ++wv)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int v = int(int8_t(uint32_t(s.q[wv]) >> (8 * j)));
      const float dl = wv < 4 ? d0 : d1;
      float r;
      if constexpr (FMT == FB_FMT_Q2_0) r = float(v) * dl;           // (q - 1) * d
      else if constexpr (FMT == FB_FMT_IQ4_XS) r = dl * float(v);     // dl * level
      else r = dl * float(v < 0 ? -v : v) * (v < 0 ? -1.0f : 1.0f);   // dl * magnitude * sign
      y[4 * wv + j] = r;
    }
}

template <int FMT>
__global__ void __launch_bounds__(256) dequant_generic_kernel(const uint8_t* __restrict__ rows, int64_t row_bytes,
                                                              int nrows, int k, float* __restrict__ out) {
  __shared__ __align__(8) uint32_t s_grid[kGenericGridWords];
  generic_grid_fill<FMT>(s_grid);
  __syncthreads();
  const int subs = k / 32;
  for (int64_t u = int64_t(blockIdx.x) * 256 + threadIdx.x; u < int64_t(nrows) * subs; u += int64_t(gridDim.x) * 256) {
    const int r = int(u / subs), sub = int(u - int64_t(r) * subs);
    float y[32];
    dequant_sub32<FMT>(rows + int64_t(r) * row_bytes, sub, s_grid, y);
    float4* o = reinterpret_cast<float4*>(out + int64_t(r) * k + 32 * sub);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
  }
}
