// The grouped GEMM kernel of the prefill path, included by moe_prefill.cu inside namespace fb's anonymous namespace.
// One persistent kernel, one CTA per SM, for both projections:
//   gate/up  unit = 64 intermediate rows of one expert x up to 256 of its tokens; the 128 tensor-memory lanes hold
//            gate and up rows in turn (lane 2i = gate row i, lane 2i + 1 = up row i), so that SwiGLU pairs a lane with
//            its neighbour;
//   down     unit = 128 output rows x up to 128 tokens (two accumulators: the epilogue, which is half of the work here,
//            overlaps the next unit; with 256 tokens per unit the projection took 667 instead of 411 us at 8192 tokens).
//
// What bounds it is the decoding of the weights: every weight passes the integer pipe once per (expert, 256-token
// unit) however few tokens the unit has. So the decoded bf16 values go from registers straight into TENSOR MEMORY,
// where tcgen05.mma takes its A operand from: no shared-memory store of the tile, no read of it by the tensor core,
// no proxy fence, and 256 columns of ring space (K = 512) that cost no shared memory. (The version before this one
// stored swizzled tiles into a three-stage shared-memory ring: 8 weights per clock and SM.)
//
// The B operand comes by TMA from rows in pair order: h for the down projection; for gate/up the token rows are first
// copied into that order (scatter_rows_kernel). (Gathered by cp.async inside this kernel, a unit of 256 tokens cost
// 2048 load/store cycles per 256 K beside the decoding's thousand; by TMA gather, 52 cycles per four rows.)
//
// Roles: warp 0 issues the MMAs, warp 1 the TMA copies, two warps copy raw weight bytes with cp.async; 16 decoding
// warps, lane = weight row (tensor-memory lane quarter = warp % 4); eight epilogue warps.
// Tensor memory: columns 0..255 accumulators (two of 128 tokens or one of 256), 256..511 two A stages of 256 K.
// All hand-offs are mbarriers with bounded waits.
//
// Times in this file are of calls (or of layers of four calls) on two states in turn, twelve passes between two device events,
// the best of four runs. With more states in turn, as a model has layers, a layer takes 9 to 15 % longer (96 IQ4_NL tokens 297 and
// 324 to 335 us, 8192 IQ3_S tokens 1120 and 1250 to 1300): compare differences, not times, with figures taken that way.
#pragma once

constexpr int kGgAStages = 2, kGgMaxRawSlots = 5, kGgMaxBStages = 4;
constexpr int kGgRawWarps = 2, kGgDecodeWarps = 16, kGgEpiWarps = 8;
constexpr int kGgFirstDecode = 2 + kGgRawWarps, kGgFirstEpi = kGgFirstDecode + kGgDecodeWarps;
constexpr int kGgThreads = (kGgFirstEpi + kGgEpiWarps) * 32;
constexpr int kGgABase = 256;  // first tensor-memory column of the A slots
// TMA boxes of token (h) rows x K steps: a stage of one or two K steps is filled with the fewest boxes of 128, 64 and 32
// rows, a stage of four or eight steps by one box.
enum { kBox32, kBox64, kBox128, kBox32x8, kBox64x4, kBoxes };
struct GgMaps {
  CUtensorMap m[kBoxes];
};

struct GgBars {
  uint64_t b_full[kGgMaxBStages], b_empty[kGgMaxBStages];
  uint64_t a_full[kGgAStages], a_empty[kGgAStages];
  uint64_t raw_full[kGgMaxRawSlots], raw_empty[kGgMaxRawSlots];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort;
};

static __constant__ int8_t c_iq4nl_levels[16] = {FB_IQ4NL_LEVELS};

// Raw weight bytes in shared memory.
// gate/up: a slot = one round (256 weights) of the unit's 128 rows, copied row piece by row piece. IQ3_S: the up to eight
//   16-byte words that cover a row's 110-byte block (single 4-byte words took four times the copies: with them the two copying
//   warps alone needed 200 us for gate/up of 96 tokens, which went from 241 to 213 us). Rows lie 1100 bytes apart, so a block starts at word 0..3 of its first 16 bytes,
//   by turns; the rows of 32 lanes are laid out so that the same word of their blocks meets 32 banks (gg_iq3s_slot_row).
//   IQ4_NL: 144 bytes, back to back (16-byte reads of eight neighbouring rows cover all banks).
//   kBStages: token stages of 32 KB. A unit of 256 tokens drains one in 512 cycles, and the L2 answers later than three of them
//   last: with the fourth in the place of a raw slot a layer of 8192 IQ3_S tokens went from 1216 to 1192 us. (With three raw
//   slots gate/up of 96 tokens lost 7 to 15 %: IQ4_NL, whose raw slots are larger, keeps three token stages.)
// down: a slot = the whole unit, 128 complete rows, which lie back to back in the matrix: one bulk copy. (Cut into pieces like
//   gate/up, rows of 360 bytes came in 8-byte copies, and the copying warps were the pace: 382 us instead of 233 at 1003
//   tokens.)
template <int FMT, bool DOWN>
struct GgRaw;
template <>
struct GgRaw<FB_FMT_IQ3_S, false> {
  static constexpr int kPiece = 110, kPitch = 132, kSlots = 4, kSlot = kTileM * kPitch, kBStages = 4;  // (128 + 16 bytes per four rows)
};
template <>
struct GgRaw<FB_FMT_IQ4_NL, false> {
  static constexpr int kPiece = 144, kPitch = 144, kSlots = 5, kSlot = kTileM * kPitch, kBStages = 3;
};
template <>
struct GgRaw<FB_FMT_IQ3_S, true> {
  static constexpr int kPiece = 110, kPitch = 220, kSlots = 3, kSlot = kTileM * kPitch, kBStages = 3;  // (intermediate 512 only)
};
template <>
struct GgRaw<FB_FMT_IQ4_NL, true> {
  static constexpr int kPiece = 144, kPitch = 360, kSlots = 2, kSlot = kTileM * kPitch, kBStages = 3;  // (288-byte rows: pitch 288)
};
// IQ3_S selectors (of an entry's weights 3, 2, 1, 0), 16 bits per index and lane: entry i of lane l at byte 64 i + 2 l. Two
// lanes share a bank, so a warp's look-up takes two passes at most where one shared copy takes three to four.
// IQ4_NL level pairs, entry b of lane l at byte 128 b + 4 l.
template <int FMT>
constexpr int kGgTableBytes = FMT == FB_FMT_IQ3_S ? 512 * 64 : 256 * 128;
template <int FMT, bool DOWN>
constexpr int gg_smem() {
  return GgRaw<FMT, DOWN>::kBStages * kTileB + GgRaw<FMT, DOWN>::kSlots * GgRaw<FMT, DOWN>::kSlot + kGgTableBytes<FMT> +
         int(sizeof(GgBars)) + 64;
}
static_assert(gg_smem<FB_FMT_IQ3_S, false>() <= 232448 && gg_smem<FB_FMT_IQ4_NL, false>() <= 232448 &&
                  gg_smem<FB_FMT_IQ3_S, true>() <= 232448 && gg_smem<FB_FMT_IQ4_NL, true>() <= 232448,
              "shared memory per block");

// Byte of an IQ3_S gate/up slot where the piece of lane l (row l / 2 of gate or up) of a lane quarter begins. Places are taken
// in the order of g = l / 8 + 4 (l % 2), four rows each, 128 bytes per row and another 16 after every four: the 16-byte words
// of a g start in bank 4 g, and its four rows' blocks in the four banks from there.
__device__ __forceinline__ uint32_t gg_iq3s_slot_row(int l) {
  const int g = (l >> 3) + 4 * (l & 1), p = 4 * g + ((l >> 1) & 3);
  return uint32_t(128 * p + 16 * g);
}

__device__ __forceinline__ uint32_t lds_u8(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}

// ------------------------------------------------------------------------------ tensor memory
// D[tmem] (+)= A[tmem] * B[smem], bf16 operands, 16 K.
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kDescHiK128)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------------------------ decoding
// Byte B of `word` times `weight` plus `acc`: one integer dot product, which runs on the multiply pipe. The decoders are
// bound by the half-rate integer pipe and by issue (74 and 72 % busy in IQ3_S gate/up with shifts and masks here), so table
// addresses and sign masks are formed this way: gate/up of 96 tokens 306 -> 278 us.
template <int B>
__device__ __forceinline__ uint32_t byte_mad(uint32_t word, uint32_t weight, uint32_t acc) {
  return __dp4a(word, weight << (8 * B), acc);
}
// IQ3_S, one sub-block (32 weights). A weight is db * g * sign with g one of the 8 odd magnitudes 1..15, so the 8
// possible bf16 values of the sub-block are computed once (db * (2k+1) is exact in fp32, then rounded like the
// reference rounds) and kept as two byte planes in four registers; the codebook table holds, per 9-bit index, the
// four 3-bit magnitude numbers as PRMT selector nibbles, so one PRMT per plane picks four weights, one XOR flips
// their signs (bit 7 of the high bytes; rounding is sign-symmetric) and two PRMTs interleave the planes into bf16
// pairs. A byte times 0x08040201 has bit 7 - j of the byte at bit 7 of byte j, whatever else the byte holds (every bit of the
// product is one bit of the byte), times sixteen bit 3 - j: a sign byte gives the masks of its eight weights by two
// multiplications, if the four weights of a look-up are taken in reverse order. The table holds them so, and the
// interleaving turns them round. The eight ninth index bits are spread the same way, look-up 7 - j (3 - j) in byte j.
// (119 -> 111 instructions per 32 weights; gate/up of 96 tokens 213 -> 207 us.)
constexpr uint32_t kSpreadHi = 0x08040201u, kSpreadLo = 0x80402010u;  // bits 7..4, 3..0 of a byte -> bit 7 of bytes 0..3
template <int B>
__device__ __forceinline__ void gg_iq3s_lookup(uint32_t qs, uint32_t bits, uint32_t signs, uint32_t lane_table,
                                               const uint32_t (&plane)[4], uint32_t& out0, uint32_t& out1) {
  const uint32_t sel = lds_u16<0>(byte_mad<B>(qs, 64u, byte_mad<3 - B>(bits, 128u, lane_table)));
  const uint32_t lo4 = prmt(plane[0], plane[1], sel);
  const uint32_t hi4 = prmt(plane[2], plane[3], sel) ^ (signs & 0x80808080u);
  out0 = prmt(lo4, hi4, 0x6273u);
  out1 = prmt(lo4, hi4, 0x4051u);
}
__device__ __forceinline__ void gg_decode_iq3s(float db, uint32_t qs_lo, uint32_t qs_hi, uint32_t B, uint32_t sg,
                                               uint32_t lane_table, uint32_t (&out)[16]) {
  float pv[8];
  pv[0] = db;
#pragma unroll
  for (int k = 1; k < 8; ++k) pv[k] = fmaf(float(2 * k), db, db);  // exact: (2k+1) * db has at most 20 significant bits
  const uint32_t t01 = pack_bf16(pv[0], pv[1]), t23 = pack_bf16(pv[2], pv[3]);
  const uint32_t t45 = pack_bf16(pv[4], pv[5]), t67 = pack_bf16(pv[6], pv[7]);
  const uint32_t plane[4] = {prmt(t01, t23, 0x6420u), prmt(t45, t67, 0x6420u), prmt(t01, t23, 0x7531u), prmt(t45, t67, 0x7531u)};
  const uint32_t b_lo = (B * kSpreadLo) & 0x80808080u, b_hi = (B * kSpreadHi) & 0x80808080u;
  const uint32_t s0 = byte_mad<0>(sg, 1u, 0u), s1 = byte_mad<1>(sg, 1u, 0u), s2 = byte_mad<2>(sg, 1u, 0u), s3 = sg >> 24;
  gg_iq3s_lookup<0>(qs_lo, b_lo, s0 * kSpreadLo, lane_table, plane, out[0], out[1]);
  gg_iq3s_lookup<1>(qs_lo, b_lo, s0 * kSpreadHi, lane_table, plane, out[2], out[3]);
  gg_iq3s_lookup<2>(qs_lo, b_lo, s1 * kSpreadLo, lane_table, plane, out[4], out[5]);
  gg_iq3s_lookup<3>(qs_lo, b_lo, s1 * kSpreadHi, lane_table, plane, out[6], out[7]);
  gg_iq3s_lookup<0>(qs_hi, b_hi, s2 * kSpreadLo, lane_table, plane, out[8], out[9]);
  gg_iq3s_lookup<1>(qs_hi, b_hi, s2 * kSpreadHi, lane_table, plane, out[10], out[11]);
  gg_iq3s_lookup<2>(qs_hi, b_hi, s3 * kSpreadLo, lane_table, plane, out[12], out[13]);
  gg_iq3s_lookup<3>(qs_hi, b_hi, s3 * kSpreadHi, lane_table, plane, out[14], out[15]);
}

// IQ4_NL, one block (32 weights) from its scale (half of `dw`, HI = the upper one) and 16 code bytes. A byte holds the codes
// of elements i and i + 16; a table in shared memory (one copy per lane: a look-up takes one pass) gives both levels as an
// fp16 pair (exact: |level| <= 127). The multiply-add of two fp16 numbers into fp32 takes the halves as they lie: d * level is
// exact in fp32 (19 significant bits; + -0 keeps it) and rounded once to bf16. Five instructions per two weights; widening
// both halves by a shift and a mask first made it seven (gate/up and down of 96 tokens 217 and 122 us, 185 and 106 so).
__device__ __forceinline__ float mul_f16(uint16_t a, uint16_t b) {
  float r;
  asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(r) : "h"(a), "h"(b), "f"(-0.0f));
  return r;
}
template <bool HI>
__device__ __forceinline__ void gg_decode_iq4nl(uint32_t dw, const uint32_t (&q)[4], uint32_t lane_table, uint32_t (&out)[16]) {
  const uint16_t d = HI ? uint16_t(dw >> 16) : uint16_t(dw);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const uint32_t v[4] = {lds_u32<0>(byte_mad<0>(q[m], 128u, lane_table)), lds_u32<0>(byte_mad<1>(q[m], 128u, lane_table)),
                           lds_u32<0>(byte_mad<2>(q[m], 128u, lane_table)), lds_u32<0>(byte_mad<3>(q[m], 128u, lane_table))};
    float lo[4], hi[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      lo[b] = mul_f16(uint16_t(v[b]), d);
      hi[b] = mul_f16(uint16_t(v[b] >> 16), d);
    }
    out[2 * m] = pack_bf16(lo[0], lo[1]);
    out[2 * m + 1] = pack_bf16(lo[2], lo[3]);
    out[8 + 2 * m] = pack_bf16(hi[0], hi[1]);
    out[8 + 2 * m + 1] = pack_bf16(hi[2], hi[3]);
  }
}

// The raw words of one warp step (64 weights of the lane's row), in registers, and their decoding half by half.
struct GgStepIq3s {
  uint32_t qs[4], sg[2], qh, sc;
  float d;
  // `row` = the row's words of the round, `shift` = 2 if the block starts in the middle of the first word, pos = K step.
  // The 27 words behind the scale then lie on word boundaries (shift 2) or two bytes off (shift 0).
  __device__ __forceinline__ void load(uint32_t row, int shift, int pos) {
    const uint32_t blk = row + shift, p = row + 2 * shift, sh = shift ? 0u : 16u;
    const uint32_t pq = p + 16 * pos, ps = p + 8 * pos;
    d = __half2float(__ushort_as_half(static_cast<unsigned short>(lds_u16<0>(blk))));
    qh = lds_u16<66>(blk + 2 * pos);
    sc = lds_u8(blk + 106 + pos);
    const uint32_t w0 = lds_u32<0>(pq), w1 = lds_u32<4>(pq), w2 = lds_u32<8>(pq), w3 = lds_u32<12>(pq), w4 = lds_u32<16>(pq);
    const uint32_t g0 = lds_u32<72>(ps), g1 = lds_u32<76>(ps), g2 = lds_u32<80>(ps);
    qs[0] = __funnelshift_r(w0, w1, sh);
    qs[1] = __funnelshift_r(w1, w2, sh);
    qs[2] = __funnelshift_r(w2, w3, sh);
    qs[3] = __funnelshift_r(w3, w4, sh);
    sg[0] = __funnelshift_r(g0, g1, sh);
    sg[1] = __funnelshift_r(g1, g2, sh);
  }
  template <int HALF>
  __device__ __forceinline__ void decode(uint32_t lane_table, uint32_t (&out)[16]) const {
    // multiplier 2 s + 1 as a float through the mantissa of 2^23
    const float m = __uint_as_float(0x4B000001u | ((HALF ? sc >> 4 : sc & 15u) << 1)) - 8388608.0f;
    gg_decode_iq3s(__fmul_rn(d, m), qs[2 * HALF], qs[2 * HALF + 1], HALF ? qh >> 8 : qh & 0xFFu, sg[HALF], lane_table,
                   out);
  }
};
// IQ4_NL: W words of the lane's row. gate/up fetches one K step (two 18-byte blocks, nine words) at a time; down both steps of
// its half round (72 bytes) in wide loads: 16 bytes where rows keep that alignment, 8 for rows of 360 bytes. (Rows are 288
// bytes apart there, single words of 32 rows meet in four banks. For gate/up, rows 144 bytes apart, the wide forms cost
// registers and gained nothing.)
template <int W>
struct GgWords {
  uint32_t w[W];
  __device__ __forceinline__ void load_step(uint32_t b) {
    w[0] = lds_u32<0>(b); w[1] = lds_u32<4>(b); w[2] = lds_u32<8>(b); w[3] = lds_u32<12>(b); w[4] = lds_u32<16>(b);
    w[5] = lds_u32<20>(b); w[6] = lds_u32<24>(b); w[7] = lds_u32<28>(b); w[8] = lds_u32<32>(b);
  }
  __device__ __forceinline__ void load_half(uint32_t row, int m, bool by16) {  // half m of the 144 bytes at `row`
    if (by16) {
      uint32_t v[20];
#pragma unroll
      for (int i = 0; i < 5; ++i)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v[4 * i]), "=r"(v[4 * i + 1]), "=r"(v[4 * i + 2]), "=r"(v[4 * i + 3])
                     : "r"(row + 64 * m + 16 * i)
                     : "memory");
#pragma unroll
      for (int i = 0; i < 18; ++i) w[i] = m ? v[i + 2] : v[i];
    } else {
#pragma unroll
      for (int i = 0; i < 9; ++i)
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[2 * i]), "=r"(w[2 * i + 1]) : "r"(row + 72 * m + 8 * i) : "memory");
    }
  }
  template <int B>  // block B of those fetched
  __device__ __forceinline__ void decode(uint32_t lane_table, uint32_t (&out)[16]) const {
    constexpr int k = 9 * B / 2;
    if constexpr (B % 2 == 0) {
      const uint32_t q[4] = {__funnelshift_r(w[k], w[k + 1], 16), __funnelshift_r(w[k + 1], w[k + 2], 16),
                             __funnelshift_r(w[k + 2], w[k + 3], 16), __funnelshift_r(w[k + 3], w[k + 4], 16)};
      gg_decode_iq4nl<false>(w[k], q, lane_table, out);
    } else {
      const uint32_t q[4] = {w[k + 1], w[k + 2], w[k + 3], w[k + 4]};
      gg_decode_iq4nl<true>(w[k], q, lane_table, out);
    }
  }
};

// ------------------------------------------------------------------------------ raw bytes into shared memory
// gate/up, IQ4_NL: one loader warp copies the pieces of 32 rows (`bytes` of each) into its part of a raw slot. row_at(r) =
// address of the piece of row r. Copy size: the largest the alignment allows; pieces two bytes off word alignment (an expert
// table may hold any even address) go through registers. Returns true if the copies are asynchronous.
template <int B, class RowF>
__device__ __forceinline__ void gg_copy_pieces(uint32_t dst, int pitch, int bytes, int lane, RowF row_at) {
  const int per_row = bytes / B;
  for (int id = lane; id < 32 * per_row; id += 32) {
    const int r = id / per_row, c = id - r * per_row;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst + r * pitch + c * B), "l"(row_at(r) + c * B), "n"(B)
                 : "memory");
  }
}
template <class RowF>
__device__ __forceinline__ bool gg_load_iq4nl(uint32_t dst, int bytes, uint32_t align, int lane, const uint8_t* base,
                                              const int (&piece)[9], bool near, RowF row_at) {
  constexpr int P = GgRaw<FB_FMT_IQ4_NL, false>::kPitch;
  if ((align & 15u) == 0 && bytes == P && near) {
    // 16-byte pieces, nine per row: piece id -> shared-memory byte 16 id. `piece[i]` = where this lane's i-th piece
    // lies from the first row's, the same for every round: recomputing it made the two loader warps, which get an
    // issue slot every eight cycles or so, the pace of the kernel (2400 cycles per round).
#pragma unroll
    for (int i = 0; i < 9; ++i)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * lane + 512 * i), "l"(base + piece[i]) : "memory");
  } else if ((align & 7u) == 0) {
    gg_copy_pieces<8>(dst, P, bytes, lane, row_at);
  } else if ((align & 3u) == 0) {
    gg_copy_pieces<4>(dst, P, bytes, lane, row_at);
  } else {
    const int per_row = bytes / 4;
    for (int id = lane; id < 32 * per_row; id += 32) {
      const int r = id / per_row, c = id - r * per_row;
      const unsigned short* p = reinterpret_cast<const unsigned short*>(row_at(r) + 4 * c);
      sts_u32<0>(dst + r * P + 4 * c, uint32_t(p[0]) | (uint32_t(p[1]) << 16));
    }
    return false;
  }
  return true;
}

// A stage of the token ring holds this many 64-wide K steps: 256 / n rounded down to 1, 2, 4 or 8. A unit of few tokens
// then takes one hand-off per 512 K instead of eight: a wait costs the MMA thread a few hundred cycles, as much as a
// whole K step of such a unit.
// (What a copy costs is the issuing thread's instructions: its warp gets an issue slot every eight cycles or so beside the
// decoding ones, and eight boxes of one K step each took it 2000 cycles, more than the 512 K they feed.)
__device__ __forceinline__ int gg_b_steps(int n) { return n <= 32 ? 8 : n <= 64 ? 4 : n <= 128 ? 2 : 1; }

struct GgArgs {
  fb_moe_expert_layout L;
  const uint8_t* const* expert_blob;  // [512] blob addresses, or nullptr: slots + e * blob_stride
  const int4* tiles;                  // token tiles {expert, 0, first pair, tokens}
  const int32_t* n_units;             // 128-row units: tiles x (rows / 128)
  const int32_t* pair_token;
  __nv_bfloat16* h;                   // gate/up: output rows, one per pair
  const float* pair_weight;           // down
  float* yp;                          // down: output rows, one per pair
  unsigned long long* y_fixed;        // down: fixed-point sums instead, one row per token
  uint32_t* status;
};

// SwiGLU of the accumulators of one lane quarter, chunks of 16 tokens from `chunk0` on, into rows of h. Even lanes hold gate
// rows, odd lanes the matching up rows: an even lane finishes tokens 0..7 of a chunk, its neighbour tokens 8..15. A unit of 256
// tokens waits for this with its accumulators (the next one needs both), so the path is short: constant row distances, no
// bounds checks in whole chunks, silu(g) = g / (1 + 2^(-g log2 e)) with the hardware's power of two and reciprocal. The exponent is
// rounded to fp32, so the power's relative error grows with |g|, about |g| / 2 ulp: 2^-18 at |g| = 85, beyond which it is
// infinite or without effect; the bf16 step of h is 2^-8.
template <int I>
__device__ __forceinline__ void gg_store_h(__nv_bfloat16* h, const int4& un, int q, int lane, int chunk0, uint32_t dcol) {
  const bool odd = (lane & 1) != 0;
  const int first = odd ? 8 : 0;
  for (int c0 = chunk0; c0 < un.w; c0 += 4 * kGgEpiWarps) {
    uint32_t r[16];
    tmem_ld16(dcol + uint32_t(c0), r);
    tmem_ld_wait();
    __nv_bfloat16* out = h + size_t(un.z + c0 + first) * I + un.y + 16 * q + (lane >> 1);
    __nv_bfloat16 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? r[i] : r[8 + i], 1);
      const float gv = __uint_as_float(odd ? got : r[i]), uv = __uint_as_float(odd ? r[8 + i] : got);
      float e, d;
      asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(gv * -1.4426950408889634f));
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(1.0f + e));
      v[i] = __float2bfloat16_rn(gv * d * uv);
    }
    if (c0 + 16 <= un.w) {
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i * I] = v[i];
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + first + i < un.w) out[i * I] = v[i];
    }
  }
}

template <int FMT, bool DOWN>
__global__ void __launch_bounds__(kGgThreads, 1)
grouped_kernel(const GgArgs A, const __grid_constant__ GgMaps maps) {
  using R = GgRaw<FMT, DOWN>;
  constexpr bool kIq3s = FMT == FB_FMT_IQ3_S;
  constexpr int kBStages = R::kBStages;
  extern __shared__ __align__(1024) uint8_t gg_smem_base[];  // (operand tiles start on swizzle atoms)
  uint8_t* ringb = gg_smem_base;
  uint8_t* rawb = ringb + kBStages * kTileB;
  uint8_t* table = rawb + R::kSlots * R::kSlot;
  GgBars* bars = reinterpret_cast<GgBars*>(table + kGgTableBytes<FMT>);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int I = A.L.inter;
  const int k_steps = (DOWN ? I : H) / kBK, rounds = (k_steps + 3) / 4;
  // (IQ3_S down comes at intermediate 512 only: its row length is a constant of the copies' addresses)
  const int row_bytes = kIq3s ? (DOWN ? 512 : H) / 256 * 110 : (DOWN ? I : H) / 32 * 18;
  const Abort ab{&bars->abort, A.status};

  // (not from down: combine blocks that sit early on the multiprocessors that are done first made 8192 tokens 1.5 % slower)
  if constexpr (!DOWN) pdl_launch_dependents();
  if constexpr (kIq3s) {
    for (int i = tid; i < 512 * 4; i += kGgThreads) {  // 16 bytes = eight lanes' copies of an entry
      const uint32_t p = c_iq3s_grid_packed[i >> 2];
      const uint32_t e = ((p & 7u) << 12) | (((p >> 3) & 7u) << 8) | (((p >> 6) & 7u) << 4) | ((p >> 9) & 7u);
      const uint32_t w = e * 0x00010001u;
      reinterpret_cast<uint4*>(table)[i] = make_uint4(w, w, w, w);
    }
  } else {
    for (int i = tid; i < 256 * 8; i += kGgThreads) {  // 16 bytes = four lanes' copies of an entry
      const uint32_t lo = __half_as_ushort(__float2half_rn(float(c_iq4nl_levels[(i >> 3) & 15])));
      const uint32_t w = lo | (uint32_t(__half_as_ushort(__float2half_rn(float(c_iq4nl_levels[i >> 7])))) << 16);
      reinterpret_cast<uint4*>(table)[i] = make_uint4(w, w, w, w);
    }
  }
  if (tid == 0) {
    for (int i = 0; i < kBStages; ++i) {
      mbar_init(&bars->b_full[i], 1);
      mbar_init(&bars->b_empty[i], 1);
    }
    for (int i = 0; i < kGgAStages; ++i) {
      mbar_init(&bars->a_full[i], 8);  // two warps per lane quarter
      mbar_init(&bars->a_empty[i], 1);
    }
    for (int i = 0; i < R::kSlots; ++i) {
      mbar_init(&bars->raw_full[i], DOWN ? 1 : 32 * kGgRawWarps);
      mbar_init(&bars->raw_empty[i], DOWN ? kGgDecodeWarps : 8);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], kGgEpiWarps);
    }
    bars->abort = 0;
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(&bars->tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
  pdl_wait_prior();
  // gate/up: 128 intermediate rows are two units here, of 64 gate and 64 up rows each
  const int n_units = DOWN ? *A.n_units : 2 * *A.n_units;
  auto unit_at = [&](int u) -> int4 {  // {expert, first weight row, first pair, tokens}
    const int per_tile = DOWN ? H / kTileM : I / 64, tile = DOWN ? u / (H / kTileM) : I == 512 ? u / 8 : u / 10;
    int4 un = A.tiles[tile];
    un.y = (u - tile * per_tile) * (DOWN ? kTileM : 64);
    return un;
  };
  // every role reads its unit one ahead of its use
  auto unit_or_none = [&](int u) -> int4 { return u < n_units ? unit_at(u) : make_int4(0, 0, 0, 0); };
  auto blob_of = [&](int e) -> const uint8_t* {
    return A.expert_blob ? A.expert_blob[e] : A.L.slots + int64_t(e) * A.L.blob_stride;
  };

  if (warp == 0) {
    // ---------------- MMA issuer. A unit of at most 128 tokens takes one of two 128-column accumulators, so its
    // epilogue overlaps the next unit's K loop; a wider unit takes both.
    // (Its instructions are on the path from hand-off to hand-off, an issue slot every eight cycles or so: the loop exists once
    // for every number of K steps a token stage holds, with all addresses a constant away from two. With the token rows in
    // few boxes, a layer of 1003 tokens went from 507 to 484 us, of 8192 from 1259 to 1240.)
    if (elect_one()) {
      const uint32_t ring_lo = umma_desc_lo_k128(smem_u32(ringb));
      uint32_t sa = 0, pa = 0, sb = 0, pb = 0;  // A and token stage, their phases
      uint32_t use0 = 0, use1 = 0, nb = 0;
      bool ok = true;
      auto unit = [&](auto steps_per_stage, uint32_t dcol, uint32_t idesc) {
        constexpr int S = decltype(steps_per_stage)::value, kGroup = S < 4 ? S : 4;  // K steps from one wait to the next
        constexpr uint32_t kStep = (kTileB >> 4) / S;                               // descriptor distance of K steps
        for (int rd = 0; rd < rounds; ++rd) {
          const int steps = min(4, k_steps - 4 * rd);
          const uint32_t la = tmem_base + kGgABase + sa * 128;
#pragma unroll
          for (int k = 0; k < 4; k += kGroup) {
            if (k >= steps) break;
            if (S < 8 || (rd & 1) == 0) {
              if (!(ok = ab.wait(&bars->b_full[sb], pb))) return;
            }
            if (k == 0 && !(ok = ab.wait(&bars->a_full[sa], pa))) return;  // (the later of the two)
            tc_fence_after();
            const uint32_t lb = ring_lo + sb * (kTileB >> 4) + (S == 8 ? (rd & 1) * (4 * kStep) : 0u);
            {
#pragma unroll
              for (int i = 0; i < kGroup; ++i) {
                if (kGroup > 2 && i >= steps) break;
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4)
                  umma_bf16_ts(dcol, la + 32 * (k + i) + 8 * k4, lb + i * kStep + 2 * k4, idesc, k + i + k4 ? 1u : uint32_t(rd));
              }
              if (S < 8 || (rd & 1) || rd == rounds - 1) umma_commit(&bars->b_empty[sb]);
            }
            if (S < 8 || (rd & 1) || rd == rounds - 1) {
              if (++sb == kBStages) {
                sb = 0;
                pb ^= 1u;
              }
            }
          }
          umma_commit(&bars->a_empty[sa]);
          pa ^= sa;
          sa ^= 1u;
        }
      };
      int tokens = unit_or_none(blockIdx.x).w;
      for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
        const int n = (tokens + 15) & ~15;
        tokens = unit_or_none(u + gridDim.x).w;
        const bool wide = n > 128;
        const uint32_t idesc = idesc_bf16(n);
        if (wide || nb == 0) ok = ab.wait(&bars->acc_empty[0], (use0 & 1) ^ 1);
        if (ok && (wide || nb == 1)) ok = ab.wait(&bars->acc_empty[1], (use1 & 1) ^ 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t dcol = tmem_base + (wide ? 0u : nb * 128u);
        const int S = gg_b_steps(n);
        if (S == 8) unit(std::integral_constant<int, 8>{}, dcol, idesc);
        else if (S == 4) unit(std::integral_constant<int, 4>{}, dcol, idesc);
        else if (S == 2) unit(std::integral_constant<int, 2>{}, dcol, idesc);
        else unit(std::integral_constant<int, 1>{}, dcol, idesc);
        if (!ok) break;
        if (wide || nb == 0) { umma_commit(&bars->acc_full[0]); ++use0; }
        if (wide || nb == 1) { umma_commit(&bars->acc_full[1]); ++use1; }
        if (!wide) nb ^= 1u;
      }
    }
  } else if (warp == 1) {
    // ---------------- token (h) rows of the unit's pairs by TMA (one thread)
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      int4 un = unit_or_none(blockIdx.x), un_next;
      for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x, un = un_next) {
        un_next = unit_or_none(u + gridDim.x);
        const int S = gg_b_steps((un.w + 15) & ~15);
        const int rows = (un.w + 31) & ~31;
        for (int k0 = 0; k0 < k_steps; k0 += S, ++it) {
          const uint32_t s = it % kBStages;
          if (!(ok = ab.wait(&bars->b_empty[s], ((it / kBStages) & 1) ^ 1))) break;
          uint64_t* full = &bars->b_full[s];
          uint8_t* dst = ringb + s * kTileB;
          if (S >= 4) {  // (steps behind the last one are filled with zeros and not used)
            mbar_expect_tx(full, kTileB);
            tma_load_3d(dst, &maps.m[S == 8 ? kBox32x8 : kBox64x4], 0, un.z, k0, full);
          } else {
            const int k1 = min(k0 + S, k_steps);
            mbar_expect_tx(full, uint32_t((k1 - k0) * rows) * 128);
            for (int k = k0; k < k1; ++k, dst += kTileB / 2) {
              int r = 0;
              for (; rows - r >= 128; r += 128) tma_load_3d(dst + r * 128, &maps.m[kBox128], 0, un.z + r, k, full);
              if (rows - r >= 64) {
                tma_load_3d(dst + r * 128, &maps.m[kBox64], 0, un.z + r, k, full);
                r += 64;
              }
              if (rows > r) tma_load_3d(dst + r * 128, &maps.m[kBox32], 0, un.z + r, k, full);
            }
          }
        }
      }
    }
  } else if (warp < kGgFirstDecode) {
    if constexpr (DOWN) {
      // ---------------- raw weight bytes of whole units, a unit or two ahead of the decoding (one warp)
      if (warp == 2) {
        uint32_t n = 0;
        const uint32_t bytes = uint32_t(kTileM * row_bytes);
        for (int u = blockIdx.x; u < n_units; u += gridDim.x, ++n) {
          const int4 un = unit_at(u);
          const uint8_t* src = blob_of(un.x) + A.L.down_offset + size_t(un.y) * row_bytes;
          const uint32_t s = n % R::kSlots;
          uint8_t* dst = rawb + s * R::kSlot;
          if (!ab.wait_warp(&bars->raw_empty[s], ((n / R::kSlots) & 1) ^ 1)) break;
          if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
            if (lane == 0) {
              mbar_expect_tx(&bars->raw_full[s], bytes);
              bulk_g2s(dst, src, bytes, &bars->raw_full[s]);
            }
          } else {  // an expert table may hold any even address
            for (uint32_t i = lane; i < bytes / 2; i += 32)
              reinterpret_cast<unsigned short*>(dst)[i] = reinterpret_cast<const unsigned short*>(src)[i];
            fence_proxy_async();  // (a later unit's bulk copy will write here)
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->raw_full[s]);
          }
        }
      }
    } else {
      // ---------------- raw weight bytes, a few rounds ahead of the decoding; a warp copies 64 of the 128 rows
      constexpr int kRows = kTileM / kGgRawWarps;
      const int row0 = kRows * (warp - 2);
      int piece[9] = {};  // IQ4_NL, see gg_load_iq4nl
      // (32-bit distances: matrices further apart, as separate tensors may be, take the copies by row address)
      const int64_t apart = A.L.up_offset - A.L.gate_offset;
      const bool near = apart > -(int64_t(1) << 30) && apart < (int64_t(1) << 30);
      if constexpr (!kIq3s) {
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const int id = lane + 32 * i, r = id / 9, c = id - 9 * r;
          piece[i] = 16 * c + (r >> 1) * row_bytes + ((r & 1) && near ? int(apart) : 0);
        }
      }
      uint32_t rcount = 0;
      int4 un = unit_or_none(blockIdx.x), un_next;
      bool ok = true;
      for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x, un = un_next) {
        un_next = unit_or_none(u + gridDim.x);
        const uint8_t* blob = blob_of(un.x);
        const uint8_t* rg = blob + A.L.gate_offset + size_t(un.y + row0 / 2) * row_bytes;   // first gate row
        const uint8_t* rup = blob + A.L.up_offset + size_t(un.y + row0 / 2) * row_bytes;  // first up row
        for (int rd = 0; rd < rounds; ++rd, ++rcount) {
          const uint32_t s = rcount % R::kSlots;
          if (!(ok = ab.wait_warp(&bars->raw_empty[s], ((rcount / R::kSlots) & 1) ^ 1))) break;
          const int off = rd * R::kPiece;
          const uint32_t slot = smem_u32(rawb) + s * R::kSlot + row0 * R::kPitch;
          bool async = true;
          if constexpr (kIq3s) {
            // lane = 16-byte word c of a block in row i of four; rows 4 k + i lie 4400 bytes apart, so they are cut alike
            const int i = lane >> 3, c = lane & 7;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              const uint8_t* p = (m ? rup : rg) + off + i * row_bytes;
              const int in = int(reinterpret_cast<uintptr_t>(p) & 15);
              p += 16 * c - in;
              if (16 * c < in + R::kPiece) {  // (no copy of 16 bytes without one of the block's)
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                  for (int hf = 0; hf < kRows / 32; ++hf)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                 ::"r"(slot + 32 * hf * R::kPitch + (4 * (4 * m + k) + i) * 128 + 16 * (4 * m + k) + 16 * c),
                                 "l"(p + (16 * hf + 4 * k) * row_bytes)
                                 : "memory");
              }
            }
          } else {
            const int bytes = min(R::kPitch, row_bytes - off);
            const uint8_t *pg = rg + off, *pu = rup + off;
            const uint32_t align = uint32_t(reinterpret_cast<uintptr_t>(pg) | reinterpret_cast<uintptr_t>(pu)) | uint32_t(row_bytes);
            for (int hf = 0; hf < kRows / 32; ++hf) {
              const uint8_t *p = pg + 16 * hf * row_bytes, *p2 = pu + 16 * hf * row_bytes;
              async = gg_load_iq4nl(slot + 32 * hf * R::kPitch, bytes, align, lane, p, piece, near,
                                    [&](int r) { return ((r & 1) ? p2 : p) + (r >> 1) * row_bytes; });
            }
          }
          if (async) cp_async_arrive_noinc(&bars->raw_full[s]);
          else mbar_arrive(&bars->raw_full[s]);
        }
      }
      cp_async_wait_all();
    }
  } else if (warp < kGgFirstEpi) {
    // ---------------- decoding warps: lane = row 32 q + lane. Two groups of eight warps take alternate rounds of 256 K
    // and own one A stage each: while one group waits (raw bytes, its stage, its tensor-memory stores) the other one
    // decodes. In a group, a quarter's two warps take 128 K each. (Sixteen warps on every round ran in phase and waited
    // in phase; four groups on 128 K each double the hand-offs of the MMA thread, which then paces the kernel.)
    const int q = warp & 3, j = (warp - kGgFirstDecode) >> 2, grp = j >> 1;
    const uint32_t raw_row = smem_u32(rawb) + (!DOWN && kIq3s ? 32 * q * R::kPitch + gg_iq3s_slot_row(lane)
                                                              : (32 * q + lane) * (DOWN ? row_bytes : R::kPitch));
    const uint32_t ta = tmem_base + (uint32_t(32 * q) << 16) + kGgABase + grp * 128;
    const uint32_t lane_table = smem_u32(table) + uint32_t(lane) * (kIq3s ? 2 : 4);
    // IQ3_S gate/up: where the lane's row begins in its first 16 bytes (units and lane quarters are multiples of four rows
    // apart, which are multiples of 16 bytes)
    auto row_start = [&](const int4& w) -> int {
      if constexpr (!kIq3s || DOWN) return 0;
      const int64_t at = ((lane & 1) ? A.L.up_offset : A.L.gate_offset) + ((lane >> 1) & 3) * row_bytes;
      return int(reinterpret_cast<uintptr_t>(blob_of(w.x) + at)) & 15;
    };
    uint32_t r0 = 0, n = 0;  // rounds, units before this unit
    int4 un_next = unit_or_none(blockIdx.x);
    for (int u = blockIdx.x; u < n_units; u += gridDim.x, r0 += rounds, ++n) {
      const int start0 = row_start(un_next);
      un_next = unit_or_none(u + gridDim.x);
      bool ok = true;
      if constexpr (DOWN) {
        if (!ab.wait_warp(&bars->raw_full[n % R::kSlots], (n / R::kSlots) & 1)) break;
      }
      for (int rd = (grp ^ int(r0)) & 1; rd < rounds; rd += 2) {
        const uint32_t rc = r0 + rd, rs = (DOWN ? n : rc) % R::kSlots, pa = ((rc / kGgAStages) & 1) ^ 1;
        const int m = (j ^ int(rc >> 1)) & 1;  // this warp's half of the round (a short round's only half changes hands)
        const int at = DOWN ? rd * R::kPiece : kIq3s ? (start0 + rd * R::kPiece) & 15 : 0;
        const uint32_t row = raw_row + rs * R::kSlot + (at & ~3), tcol = ta + m * 64;
        const int shift = at & 3;
        if constexpr (!DOWN) {
          if (!(ok = ab.wait_warp(&bars->raw_full[rs], (rc / R::kSlots) & 1))) break;
        }
        const bool mine = 4 * rd + 2 * m < k_steps;
        std::conditional_t<kIq3s, GgStepIq3s, GgWords<DOWN ? 18 : 9>> raw;
        uint32_t out[16];
        if (mine) {
          if constexpr (kIq3s) raw.load(row, shift, 2 * m);
          else if constexpr (DOWN) raw.load_half(row, m, (row_bytes & 15) == 0);
          else raw.load_step(row + 72 * m);
          raw.template decode<0>(lane_table, out);
        }
        if (!(ok = ab.wait_warp(&bars->a_empty[grp], pa))) break;
        tc_fence_after();
        if (mine) {
          tmem_st16(tcol, out);
          raw.template decode<1>(lane_table, out);
          tmem_st16(tcol + 16, out);
          if constexpr (kIq3s) raw.load(row, shift, 2 * m + 1);
          else if constexpr (!DOWN) raw.load_step(row + 72 * m + 36);
          raw.template decode<!kIq3s && DOWN ? 2 : 0>(lane_table, out);
          tmem_st16(tcol + 32, out);
          raw.template decode<!kIq3s && DOWN ? 3 : 1>(lane_table, out);
          tmem_st16(tcol + 48, out);
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bars->a_full[grp]);
          if (!DOWN) mbar_arrive(&bars->raw_empty[rs]);
        }
      }
      if (!ok) break;
      if (DOWN) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->raw_empty[n % R::kSlots]);
      }
    }
  } else {
    // ---------------- epilogue: lane quarter = warp % 4, two warps per quarter take alternate chunks of 16 tokens
    const int q = warp & 3, chunk0 = 16 * ((warp - kGgFirstEpi) >> 2);
    uint32_t use0 = 0, use1 = 0, nb = 0;
    int4 un = unit_or_none(blockIdx.x), un_next;
    for (int u = blockIdx.x; u < n_units; u += gridDim.x, un = un_next) {
      un_next = unit_or_none(u + gridDim.x);
      const bool wide = ((un.w + 15) & ~15) > 128;
      // (the routing weights of the warp's chunks, asked for ahead of the wait: a load per chunk behind it cost as much as the
      // rest of the chunk)
      float pw[kTileNDown / 32];
      if constexpr (DOWN) {
#pragma unroll
        for (int i = 0; i < kTileNDown / 32; ++i) {
          const int t = chunk0 + 32 * i + (lane & 15);
          pw[i] = t < un.w && !A.y_fixed ? A.pair_weight[un.z + t] : 0.0f;
        }
      }
      bool ok = true;
      if (wide || nb == 0) ok = ab.wait_warp(&bars->acc_full[0], use0 & 1);
      if (ok && (wide || nb == 1)) ok = ab.wait_warp(&bars->acc_full[1], use1 & 1);
      if (!ok) break;
      tc_fence_after();
      const uint32_t dcol = tmem_base + (uint32_t(32 * q) << 16) + (wide ? 0u : nb * 128u);
      if constexpr (!DOWN) {
        if (I == 512) gg_store_h<512>(A.h, un, q, lane, chunk0, dcol);
        else gg_store_h<640>(A.h, un, q, lane, chunk0, dcol);
      } else {
#pragma unroll
        for (int c = 0; c < kTileNDown / 32; ++c) {
          const int c0 = chunk0 + 32 * c;
          if (c0 >= un.w) break;
          uint32_t r[16];
          tmem_ld16(dcol + uint32_t(c0), r);
          tmem_ld_wait();
          const int n = un.y + 32 * q + lane;
          if (A.y_fixed) {  // the reference's accumulation (src/kernels/moe/moe.h:186-192): y_fixed[token] += fixed(w * v)
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c0 + i < un.w) {
                const float v = A.pair_weight[un.z + c0 + i] * __uint_as_float(r[i]);
                atomicAdd(A.y_fixed + size_t(A.pair_token[un.z + c0 + i]) * H + n,
                          static_cast<unsigned long long>(__float2ll_rn(v * 4294967296.0f)));
              }
          } else {
            // (an epilogue warp gets an issue slot every eight cycles or so: the weights reach the lanes by shuffles, and whole
            // chunks skip the bounds checks)
            float* out = A.yp + size_t(un.z + c0) * H + n;
            if (c0 + 16 <= un.w) {
#pragma unroll
              for (int i = 0; i < 16; ++i) out[i * H] = __shfl_sync(0xffffffffu, pw[c], i) * __uint_as_float(r[i]);
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const float w = __shfl_sync(0xffffffffu, pw[c], i);
                if (c0 + i < un.w) out[i * H] = w * __uint_as_float(r[i]);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (wide || nb == 0) { if (lane == 0) mbar_arrive(&bars->acc_empty[0]); ++use0; }
      if (wide || nb == 1) { if (lane == 0) mbar_arrive(&bars->acc_empty[1]); ++use1; }
      if (!wide) nb ^= 1u;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Token rows in pair order: xg[p] = x[token of p]. A warp reads its token's row (1 / PARTS of it) once and writes it to the
// token's pairs: the writes (420 MB at 8192 tokens) are the cost. (A warp per pair took 100 us there.)
template <int PARTS>
__global__ void __launch_bounds__(128) scatter_rows_kernel(const __nv_bfloat16* x, const int32_t* token_pair, int tokens,
                                                           __nv_bfloat16* xg) {
  pdl_launch_dependents();
  pdl_wait_prior();
  constexpr int kPieces = H / 256 / PARTS;
  const int w = blockIdx.x * 4 + (threadIdx.x >> 5), t = w / PARTS, lane = threadIdx.x & 31;
  if (t >= tokens) return;
  const int at = 32 * kPieces * (w - t * PARTS) + lane;
  const uint4* src = reinterpret_cast<const uint4*>(x + size_t(t) * H) + at;
  const int mine = lane < kTopK ? token_pair[t * kTopK + lane] : -1;
  uint4 v[kPieces];
#pragma unroll
  for (int i = 0; i < kPieces; ++i) v[i] = src[32 * i];
#pragma unroll
  for (int k = 0; k < kTopK; ++k) {
    const int p = __shfl_sync(0xffffffffu, mine, k);
    if (p < 0) continue;  // a pair of another rank
    uint4* dst = reinterpret_cast<uint4*>(xg + size_t(p) * H) + at;
#pragma unroll
    for (int i = 0; i < kPieces; ++i) dst[32 * i] = v[i];
  }
}
