// Device routines for the GGUF expert formats: codebook tables in shared memory, exact integer
// decode of IQ3_S / IQ4_NL sub-blocks into dp4a operands, and the Q8_K / Q8_0 activation
// quantizers. What the GEMV kernels and the parity probes share is said at the probes.
//
// Format definitions follow third_party/ggml-iq/ggml-iq.h:81-96 and the reference dequantizers
// third_party/ggml-iq/ggml-iq.c:231-288 of the reference project.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"
#include "iq_codebooks.h"

namespace fb {

// ------------------------------------------------------------------------------ tables
// IQ3_S codebook in shared memory, replicated once per lane: entry i of lane l lives at word
// i*32 + l, so a warp's 32 independent look-ups always hit 32 different banks.
constexpr int kGridRepWords = 512 * 32;
constexpr int kGridRepBytes = kGridRepWords * 4;  // 65536
// Sign masks: nibble n -> four bytes, 0xFF where bit j of n is set. 16 words, 16 banks.
constexpr int kSignTabWords = 16;

// One copy per translation unit (internal linkage), initialised at load time.
static __constant__ uint16_t c_iq3s_grid_packed[512] = {FB_IQ3S_GRID_PACKED};

__device__ __forceinline__ uint32_t iq3s_expand(uint32_t p) {
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) w |= (2u * ((p >> (3 * j)) & 7u) + 1u) << (8 * j);
  return w;
}
__device__ __forceinline__ uint32_t iq3s_grid_entry(int i) { return iq3s_expand(c_iq3s_grid_packed[i]); }

// Called by every thread of the block; caller synchronizes afterwards.
__device__ __forceinline__ void iq3s_tables_fill(uint32_t* gridrep, uint32_t* signtab) {
  // consecutive threads write consecutive 16-byte pieces (eight per entry): no bank conflicts
  for (int i = threadIdx.x; i < 512 * 8; i += blockDim.x) {
    const uint32_t w = iq3s_grid_entry(i >> 3);
    reinterpret_cast<uint4*>(gridrep)[i] = make_uint4(w, w, w, w);
  }
  if (threadIdx.x < 16) {
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (threadIdx.x & (1 << j)) m |= 0xFFu << (8 * j);
    signtab[threadIdx.x] = m;
  }
}

// ------------------------------------------------------------------------------ IQ3_S
// One 32-weight sub-block. Inputs: qs_lo/qs_hi = its 8 index bytes, qh = a word whose bits
// [sh, sh+8) are the 8 ninth index bits, sg = its 4 sign bytes (nibble l = signs of look-up l).
// Outputs per look-up l: g[l] = four magnitudes (bytes, element order), m[l] = 0xFF in the bytes
// whose weight is negative. grid_lane = gridrep + lane.
//
// Instruction budget matters here (the integer pipe, not HBM, bounds this kernel): the ninth
// index bits are spread to bytes with one multiply per nibble, then each 9-bit index is one
// byte-permute (low byte from qs, high byte from the spread bits) and each sign-table offset is
// one byte-permute of the pre-scaled nibbles.
// prmt.b32 in its default mode: selector nibble n picks byte (n & 7) of {a, b}; with bit 3 set the
// selected byte's sign bit is replicated over the output byte instead (0x00 for bytes < 0x80).
// (__byte_perm documents only three selector bits per byte, so the PTX form is spelled out.)
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

__device__ __forceinline__ void iq3s_decode_sub(uint32_t qs_lo, uint32_t qs_hi, uint32_t qh, int sh, uint32_t sg,
                                                const uint32_t* grid_lane, const uint32_t* signtab,
                                                uint32_t (&g)[8], uint32_t (&m)[8]) {
  // bit j of a nibble -> byte j (0 or 1): n * (1 + 2^7 + 2^14 + 2^21) has bit j at position 8j
  const uint32_t h_lo = (((qh >> sh) & 0xFu) * 0x00204081u) & 0x01010101u;
  const uint32_t h_hi = (((qh >> (sh + 4)) & 0xFu) * 0x00204081u) & 0x01010101u;
  // nibbles pre-scaled by 4 (byte offsets into the 16-word sign table)
  const uint32_t s_even = (sg << 2) & 0x3C3C3C3Cu;  // look-ups 0,2,4,6
  const uint32_t s_odd = (sg >> 2) & 0x3C3C3C3Cu;   // look-ups 1,3,5,7
  const char* signb = reinterpret_cast<const char*>(signtab);
#pragma unroll
  for (int l = 0; l < 8; ++l) {
    const int b = l & 3;
    // byte0 = qs byte b, byte1 = spread bit b, bytes 2-3 = 0 (sign-replicate of a 0/1 byte)
    const uint32_t sel = uint32_t(b) | (uint32_t(4 + b) << 4) | (uint32_t(0xC + b) << 8) | (uint32_t(0xC + b) << 12);
    const uint32_t idx = prmt(l < 4 ? qs_lo : qs_hi, l < 4 ? h_lo : h_hi, sel);
    g[l] = grid_lane[idx * 32];
    const uint32_t off = __byte_perm((l & 1) ? s_odd : s_even, 0u, 0x4440u | uint32_t(l >> 1));
    m[l] = *reinterpret_cast<const uint32_t*>(signb + off);
  }
}

// Signed int8x4 weights from (g, m): byte-wise negation where m = 0xFF; (g ^ 0xFF) + 1 never carries
// because every magnitude is odd.
__device__ __forceinline__ int iq3s_signed(uint32_t g, uint32_t m) { return int((g ^ m) + (m & 0x01010101u)); }

// dp4a of 8 signed weight words with 32 int8 activations at `a` (16-byte aligned shared memory).
__device__ __forceinline__ int dot32(const int (&w)[8], const int8_t* a) {
  const int4 a0 = *reinterpret_cast<const int4*>(a);
  const int4 a1 = *reinterpret_cast<const int4*>(a + 16);
  int s = __dp4a(w[0], a0.x, 0);
  s = __dp4a(w[1], a0.y, s);
  s = __dp4a(w[2], a0.z, s);
  s = __dp4a(w[3], a0.w, s);
  s = __dp4a(w[4], a1.x, s);
  s = __dp4a(w[5], a1.y, s);
  s = __dp4a(w[6], a1.z, s);
  s = __dp4a(w[7], a1.w, s);
  return s;
}

// The same of weights that are sums of two words' bytes.
__device__ __forceinline__ int dot32(const int (&w)[8], const int (&v)[8], const int8_t* a) {
  const int4 a0 = *reinterpret_cast<const int4*>(a);
  const int4 a1 = *reinterpret_cast<const int4*>(a + 16);
  const int av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
  int s = 0, t = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s = __dp4a(w[i], av[i], s);
    t = __dp4a(v[i], av[i], t);
  }
  return s + t;
}

// An IQ3_S block is a 2-byte scale followed by 27 words: 16 of index bytes, 2 of ninth bits, 8 of
// signs, 1 of sub-block scales. In a 220-byte unit (two blocks, word aligned) the first block's
// 27 words sit 2 bytes off word alignment, the second block's are aligned: S<MIS>(w, k) reads
// word k of the stream either way (w = the word holding the fp16 scale).
template <bool MIS>
__device__ __forceinline__ uint32_t iq3s_stream(const uint32_t* w, int k) {
  if constexpr (MIS) return __byte_perm(w[k], w[k + 1], 0x5432);
  else return w[k + 1];
}

// ------------------------------------------------------------------------------ IQ4_NL
// The 16 levels held in four registers for byte-permute look-ups.
struct Iq4nlLevels {
  uint32_t t0, t1, t2, t3;
  uint32_t u2, u3;  // the upper eight plus one
};
__host__ __device__ constexpr uint32_t iq4nl_pack4(int q, int plus = 0) {
  constexpr int lv[16] = {FB_IQ4NL_LEVELS};
  return uint32_t(uint8_t(lv[4 * q] + plus)) | (uint32_t(uint8_t(lv[4 * q + 1] + plus)) << 8) |
         (uint32_t(uint8_t(lv[4 * q + 2] + plus)) << 16) | (uint32_t(uint8_t(lv[4 * q + 3] + plus)) << 24);
}
__device__ __forceinline__ Iq4nlLevels iq4nl_levels() {
  constexpr uint32_t a = iq4nl_pack4(0), b = iq4nl_pack4(1), c = iq4nl_pack4(2), d = iq4nl_pack4(3);
  Iq4nlLevels L;
  L.t0 = a;
  L.t1 = b;
  L.t2 = c;
  L.t3 = d;
  constexpr uint32_t u2 = iq4nl_pack4(2, 1), u3 = iq4nl_pack4(3, 1);
  L.u2 = u2;
  L.u3 = u3;
  return L;
}
__host__ __device__ constexpr int iq4nl_level(int i) {
  constexpr int lv[16] = {FB_IQ4NL_LEVELS};
  return lv[i];
}
__device__ __forceinline__ uint32_t upper_half(uint32_t w) { return __dp2a_lo(w, 0x0100u, 0u); }
// One 32-weight block from its 16 code bytes, as two addends of every weight, for dot products. Word 2 m + h of either (m = word
// of the codes, h = half) holds the elements {4m+2h, 4m+2h+16, 4m+2h+1, 4m+2h+17}: activations are stored in that interleaved
// order (q8_0_interleave_index). With the upper bit of a code as a permute's sign-replicating bit, a permute of the lower eight
// levels (all negative) gives the level, or -1 for an upper code; one of the upper eight levels plus one (all positive), by the
// code with that bit turned round, gives level + 1, or 0 for a lower code. So sum of level * a = dp4a(lo, a) + dp4a(hi, a), and
// nothing has to be picked. Codes = eight half words from half word `half0` of `w` on (a permute looks at the low 16 bits of its
// selector, so halves need no alignment): 45 instructions per 32 weights and token, 21 of them on the integer pipe, which was the
// busy one, where picking the level out of two permutes by a third, and one dp4a per four weights, made 54 and 38 (eight IQ4_NL
// layers of one token 143 -> 133 us, of eight 364 -> 356, of sixteen 599 -> 585).
constexpr bool iq4nl_signs_split() {
  for (int i = 0; i < 16; ++i)
    if (i < 8 ? iq4nl_level(i) >= 0 : iq4nl_level(i) <= 0 || iq4nl_level(i) > 126) return false;
  return true;
}
static_assert(iq4nl_signs_split(), "lower levels negative, upper ones positive");
template <int WORDS>
__device__ __forceinline__ void iq4nl_addends32(const Iq4nlLevels& L, const uint32_t (&w)[WORDS], int half0, int (&lo)[8], int (&hi)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t c = w[(half0 + i) >> 1], f = c ^ 0x88888888u;
    const bool up = (half0 + i) & 1;
    lo[i] = int(prmt(L.t0, L.t1, up ? upper_half(c) : c));
    hi[i] = int(prmt(L.u2, L.u3, up ? upper_half(f) : f));
  }
}
// Position of element e (0..31) of a Q8_0 block in the interleaved activation order.
__host__ __device__ __forceinline__ int q8_0_interleave_index(int e) {
  return 2 * (e & 15) + (e >> 4);  // nibble byte e%16, low nibble first
}

// ------------------------------------------------------------------------------ quantizers
// Q8_K of one 256-value block by one warp; lane l holds elements 8l..8l+7 in v.
// quantize_row_q8_K_ref, third_party/ggml-iq/ggml-iq.c:313-350: max is the FIRST element of
// largest magnitude (signed), iscale = -127/max, q = min(127, rne(iscale*x)), d = 1/iscale; an
// all-zero block gives d = 0, q = 0, bsums = 0 (src/cpu/q8_cpu.h:7-8).
// Returns d; q[8] are this lane's codes; pair_sum is the sum of the 16 codes of this lane's group
// of 16 (valid in both lanes of the pair).
__device__ __forceinline__ float q8k_block_warp(const float (&v)[8], int (&q)[8], int& pair_sum) {
  const int lane = threadIdx.x & 31;
  float amax = 0.0f;
  int idx = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float a = fabsf(v[i]);
    if (a > amax) {
      amax = a;
      idx = 8 * lane + i;
    }
  }
  // (magnitudes, never NaN here, order like their bits; the first of the largest is the one with the smallest index)
  const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
  idx = int(__reduce_min_sync(0xffffffffu, amax == most ? uint32_t(idx) : 0x7fffffffu));
  if (most == 0.0f) {
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = 0;
    pair_sum = 0;
    return 0.0f;
  }
  float cand = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((idx & 7) == i) cand = v[i];
  const float mx = __shfl_sync(0xffffffffu, cand, idx >> 3);
  const float iscale = __fdiv_rn(-127.0f, mx);
  int s = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = __float2int_rn(__fmul_rn(iscale, v[i]));
    q[i] = r < 127 ? r : 127;
    s += q[i];
  }
  pair_sum = s + __shfl_xor_sync(0xffffffffu, s, 1);
  return __fdiv_rn(1.0f, iscale);
}

// Q8_0 of one 32-value block by one warp; lane l holds element l.
// quantize_row_q8_0_ref, third_party/ggml-iq/ggml-iq.c:75-98: d = amax/127 stored as fp16,
// id = 1/d computed in fp32 from the unrounded d, q = roundf(x*id).
__device__ __forceinline__ int q8_0_block_warp(float v, unsigned short& d_half) {
  float amax = fabsf(v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float d = __fdiv_rn(amax, 127.0f);
  const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
  d_half = __half_as_ushort(__float2half_rn(d));
  return int(roundf(__fmul_rn(v, id)));
}

// Eight Q8_0 blocks (256 values) by one warp: lane l holds elements 8l..8l+7 in v, four lanes a block. Same arithmetic as
// q8_0_block_warp. Codes go to out[0..255] in the interleaved order (16-byte stores by two lanes of four), the fp16-rounded
// scales widened to scales[0..7]. `live` = this lane's block exists (its four lanes agree).
__device__ __forceinline__ void q8_0_eight_blocks_warp(const float (&v)[8], bool live, uint8_t* out, float* scales) {
  const int lane = threadIdx.x & 31;
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  const float d = __fdiv_rn(amax, 127.0f);
  const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
  uint32_t w[2] = {0u, 0u}, o[2];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i >> 2] |= uint32_t(uint8_t(int8_t(int(roundf(__fmul_rn(v[i], id)))))) << (8 * (i & 3));
#pragma unroll
  for (int i = 0; i < 2; ++i) o[i] = __shfl_xor_sync(0xffffffffu, w[i], 2);
  if (live && (lane & 2) == 0)  // elements e and, from the lane two up, e + 16
    *reinterpret_cast<uint4*>(out + 32 * (lane >> 2) + 16 * (lane & 1)) =
        make_uint4(prmt(w[0], o[0], 0x5140u), prmt(w[0], o[0], 0x7362u), prmt(w[1], o[1], 0x5140u), prmt(w[1], o[1], 0x7362u));
  if (live && (lane & 3) == 0) scales[lane >> 2] = __half2float(__float2half_rn(d));
}

// ------------------------------------------------------------------------------ routing
// Top-10 of 512 logits by one warp (lane l holds logits l + 32 i): value descending, ties to the
// lower id, NaN never wins, -0 == +0; weights = softmax over the winners in fp32, summed in rank
// order (src/kernels/moe/moe_common.cuh:33-85 of the reference states the same contract).
// Order-preserving map of a float to uint32 (larger float -> larger key); NaN maps below every
// number and -0 equals +0.
__device__ __forceinline__ uint32_t logit_key(float x) {
  if (x != x) x = -INFINITY;
  if (x == 0.0f) x = 0.0f;
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// weights = softmax over the ten winners (fp32, expf(v - top), summed in rank order).
__device__ __forceinline__ void topk_softmax(float (&vals)[FB_TOPK], float* weights) {
  float sum = 0.0f;
  const float top = vals[0];
#pragma unroll
  for (int k = 0; k < FB_TOPK; ++k) {
    vals[k] = expf(vals[k] - top);
    sum += vals[k];
  }
  const float inv = __fdiv_rn(1.0f, sum);
#pragma unroll
  for (int k = 0; k < FB_TOPK; ++k) weights[k] = vals[k] * inv;
}
__device__ __forceinline__ float key_logit(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

template <class LoadF>
__device__ __forceinline__ void warp_topk10(LoadF load_logit, int* ids, float* weights) {
  const int lane = threadIdx.x & 31;
  uint32_t key[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) key[i] = logit_key(load_logit(lane + 32 * i));
  float vals[FB_TOPK];
#pragma unroll
  for (int k = 0; k < FB_TOPK; ++k) {
    // lane-local best as a 4-level tree: a higher slot wins only when strictly greater, so equal
    // keys resolve to the lower id; the warp step is two redux operations (max key, then min id).
    uint32_t tk[16];
    int ti[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      tk[i] = key[i];
      ti[i] = i;
    }
#pragma unroll
    for (int w = 1; w < 16; w <<= 1) {
#pragma unroll
      for (int i = 0; i < 16; i += 2 * w) {
        const bool up = tk[i + w] > tk[i];
        tk[i] = up ? tk[i + w] : tk[i];
        ti[i] = up ? ti[i + w] : ti[i];
      }
    }
    const uint32_t best = __reduce_max_sync(0xffffffffu, tk[0]);
    const uint32_t cand = tk[0] == best ? uint32_t(lane + 32 * ti[0]) : 0xffffffffu;
    const int win = int(__reduce_min_sync(0xffffffffu, cand));
    ids[k] = win;
    const uint32_t u = (best & 0x80000000u) ? (best & 0x7fffffffu) : ~best;
    vals[k] = __uint_as_float(u);
    // retire the winner: key 0 is below every real key (the smallest real key is ~0xFF800000 = 0x007FFFFF)
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (win == lane + 32 * i) key[i] = 0u;
  }
  topk_softmax(vals, weights);
}

// The same selection as a short dependent chain (a decode step runs it in every CTA): winners and their logits; the
// weights are top10_weights below. The tenth largest of the maxima of the sixteen lane pairs is a lower bound of the tenth
// largest logit (ten different logits reach it), so only logits at or above it can win (fourteen on average); they are
// compacted into `scratch` (32 entries of this warp, shared memory, 16-byte aligned), one per lane, every lane ranks its
// candidate against the others (larger logit, then lower id: a strict order), and ranks 0..9 are the winners. More than 32
// survivors (many equal logits), or a bound of -infinity (which NaN counts as), take the general path. Same winners, same
// order as warp_topk10; out_ids / out_vals (ten entries each, shared memory) are complete after the caller's next barrier.
// Bound: instructions on one warp's chain. The whole selection takes 2.1 us at one token and 3.3 at sixteen, 2.8 and 4.1 with
// 32 lane maxima, ranks by shuffles and the softmax in the chain.
// TIES: where the survivors are too many because logits equal the bound (all logits of a padded row are equal), those above it
// are ranked and the lowest of the equal ones follow, without the general path. (The prefill kernel, all rows of equal logits,
// us: the general path alone 2.2 for one token and 9.4 for 4096, behind the search 3.9 and 12.8, so 1.9 and 3.9. The decode kernels
// keep the shorter code.)
template <bool TIES, class LoadF>
__device__ __forceinline__ void warp_top10_pruned(LoadF load_logit, uint2* scratch, int* out_ids, float* out_vals) {
  const int lane = threadIdx.x & 31;
  float x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = load_logit(lane + 32 * i);
  float pm = -INFINITY;  // (fmaxf passes a NaN over; the comparisons below are false for it)
#pragma unroll
  for (int i = 0; i < 16; ++i) pm = fmaxf(pm, x[i]);
  pm = fmaxf(pm, __shfl_xor_sync(0xffffffffu, pm, 1));
  int above = 0;  // lane pairs whose maximum is larger than this pair's
#pragma unroll
  for (int j = 0; j < 16; ++j) above += __shfl_sync(0xffffffffu, pm, 2 * j) > pm ? 1 : 0;
  float thr;
  {
    const float v = above < FB_TOPK ? pm : INFINITY;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(thr) : "f"(v));
  }
  int mine = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) mine += x[i] >= thr ? 1 : 0;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  if constexpr (TIES) {
    if (total > 32 && thr != -INFINITY) {
      int above_thr = 0;  // of this lane
#pragma unroll
      for (int i = 0; i < 16; ++i) above_thr += x[i] > thr ? 1 : 0;
      int k = int(__reduce_add_sync(0xffffffffu, unsigned(above_thr)));
      if (k < FB_TOPK) {
        // (k of them: every one is ranked by the lane that holds it, against all of them)
        int n = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (n >= k) break;  // (the same for all lanes)
          const float v = x[i];
          const unsigned has = __ballot_sync(0xffffffffu, v > thr);
          if (v > thr) scratch[n + __popc(has & ((1u << lane) - 1u))] = make_uint2(__float_as_uint(v), uint32_t(lane + 32 * i));
          n += __popc(has);
        }
        __syncwarp();
        if (lane < k) {
          const uint2 c = scratch[lane];
          const float cv = __uint_as_float(c.x);
          int rank = 0;
          for (int j = 0; j < k; ++j) {
            const uint2 o = scratch[j];
            const float a = __uint_as_float(o.x);
            rank += a > cv || (a == cv && o.y < c.y) ? 1 : 0;
          }
          out_ids[rank] = int(c.y);
          out_vals[rank] = cv;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (k >= FB_TOPK) break;  // (the same for all lanes)
          const float v = x[i];
          const unsigned has = __ballot_sync(0xffffffffu, v == thr);
          const int at = k + __popc(has & ((1u << lane) - 1u));
          if (v == thr && at < FB_TOPK) {
            out_ids[at] = lane + 32 * i;
            out_vals[at] = thr;
          }
          k += __popc(has);
        }
        return;
      }
    }
  }
  if (total > 32 || thr == -INFINITY) {
    int ids[FB_TOPK];
    float w[FB_TOPK];
    warp_topk10(load_logit, ids, w);
#pragma unroll
    for (int k = 0; k < FB_TOPK; ++k)
      if (lane == k) {
        out_ids[k] = ids[k];
        out_vals[k] = key_logit(logit_key(load_logit(ids[k])));
      }
    return;
  }
  uint2* at = scratch + (incl - mine);  // (the candidates' order does not matter)
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (x[i] >= thr) *at++ = make_uint2(__float_as_uint(x[i]), uint32_t(lane + 32 * i));
  if (lane == 31 && (total & 1)) *at = make_uint2(0xff800000u, 0x7fffffffu);  // (read in pairs; -infinity beats nobody)
  __syncwarp();
  const uint2 c = scratch[lane < total ? lane : 0];
  const float cv = __uint_as_float(c.x);
  int rank = 0;
#pragma unroll 4
  for (int j = 0; j < total; j += 2) {
    const uint4 o = *reinterpret_cast<const uint4*>(scratch + j);
    const float a = __uint_as_float(o.x), b = __uint_as_float(o.z);
    rank += a > cv || (a == cv && o.y < c.y) ? 1 : 0;
    rank += b > cv || (b == cv && o.w < c.y) ? 1 : 0;
  }
  if (lane < total && rank < FB_TOPK) {
    out_ids[rank] = int(c.y);
    out_vals[rank] = cv;
  }
}

// Softmax over the winners exactly as topk_softmax: exp(v - top), summed in rank order, by one warp. Lane k computes the
// k-th term; the ten terms then reach every lane through shuffles and are added in the same order.
__device__ __forceinline__ void top10_weights(const float* vals, float* out_w) {
  const int lane = threadIdx.x & 31;
  const float e = expf(vals[lane < FB_TOPK ? lane : 0] - vals[0]);
  float sum = 0.0f;
#pragma unroll
  for (int k = 0; k < FB_TOPK; ++k) sum += __shfl_sync(0xffffffffu, e, k);
  if (lane < FB_TOPK) out_w[lane] = e * __fdiv_rn(1.0f, sum);
}

}  // namespace fb
