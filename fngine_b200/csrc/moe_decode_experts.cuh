// The streaming expert kernel of the decode path, included by moe_decode.cu inside namespace fb's anonymous namespace:
// gate/up in IQ3_S, IQ4_NL, IQ2_S, IQ3_XXS or IQ4_XS, down in IQ3_S, IQ4_NL or Q2_0. Written for IQ3_S, described for IQ3_S; the
// other formats ride the same skeleton with their own tile sizes and block arithmetic (ExpertsCfg, gate_up_sub,
// iq4nl_task_terms, q2_0_task_terms). (Behind plain kernels - a warp per row, lanes = sub-blocks from global memory - an
// IQ2_S + IQ4_NL layer of five tokens took 129 us in six launches.)
//
// One persistent kernel streams the gate, up and down matrices of every routed expert of a layer:
// first all gate/up tiles (heaviest experts first), then all down tiles, through one ring of three
// 40 KB slots (four where no table takes the space), so the codebook set-up, the work-list copy and the pipeline fill are paid once per
// layer and HBM keeps streaming across the gate/up -> down boundary. A down tile needs its expert's h
// re-quantized, which the warp that finishes the expert's last gate/up tile does and then flags; the
// producer asks for a down tile's weights first and polls that flag (a bounded number of times) only
// before it asks for the activation rows. (With few tokens values carry their own arrival flags instead: DIRECT, below.) The
// same kernel runs one phase alone behind the separate gate/up and down entry points.
//
// Shape of the work. A lane owns a weight row; a warp task is one 110-byte block (256 weights) of 32
// rows (gate/up: 16 gate rows + the 16 matching up rows, ten blocks; down: five groups of 32 rows, two
// blocks), so every tile is ten tasks, five on even blocks and five on odd ones, that the consumer
// warps draw from two shared-memory tickets.
//
// Arithmetic per 4 weights (one codebook look-up). The codebook in shared memory holds G = (g - 1) / 2
// for every magnitude g in {1, 3, ..., 15}; with m = 0xFF in the bytes of negative weights, the bytes of
// x = G ^ m are G or -G-1, so that 2 x + 1 = +-g: the signed weight. Hence
//   sum_i s_i g_i a_i = 2 * sum_lookups dp4a(x, a) + sum_i a_i,
// ONE dp4a per look-up and token; the second term is the sum of the sub-block's 32 activation codes,
// which the activation quantizer stores beside the codes (it is Q8_K's bsums, pairwise added). Exact
// integer arithmetic throughout: the block sums are the same integers the reference's CPU tier forms.
#pragma once

// ------------------------------------------------------------------------------ planar activation rows
// Q8_K rows in the workspace and in the staged tiles: codes [k] | block scales float [k/256], padded to
// 64 bytes | sub-block code sums int16 [k/32].
__host__ __device__ constexpr int q8k_planar_asum_off(int k) { return q8k_asum_off(k); }
__host__ __device__ constexpr int q8k_planar_bytes(int k) { return q8k_asum_off(k) + ((k / 32 * 2 + 15) & ~15); }
static_assert(q8k_planar_bytes(2560) <= FB_XQ_STRIDE && q8k_planar_bytes(512) <= FB_HQ_STRIDE, "row strides");
static_assert(q8k_planar_bytes(2560) % 16 == 0 && q8k_planar_bytes(512) % 16 == 0, "bulk copies");

// ------------------------------------------------------------------------------ codebook for the 2x+1 form
// Entry i of lane l at word i*32 + l (as iq3s_tables_fill), bytes (g - 1) / 2.
__device__ __forceinline__ void sign_table_fill(uint32_t* signtab) {
  if (threadIdx.x < 16) {
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (threadIdx.x & (1 << j)) m |= 0xFFu << (8 * j);
    signtab[threadIdx.x] = m;
  }
}
__device__ __forceinline__ uint32_t lds_word(uint32_t a) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}

// One 32-weight sub-block: P = sum over its 8 look-ups of dp4a(G ^ m, a) for each of TT tokens.
// qs_lo/qs_hi = its 8 index bytes, qh = a word whose bits [sh, sh+8) are the ninth index bits, sg = its
// 32 sign bits (nibble l = look-up l). sign_base = shared-window address of the 16-word mask table
// (256-byte aligned, below 2^24): it rides in the upper bytes of the byte-permute that builds the
// table offset, so the mask load needs no address arithmetic.
template <int TT>
__device__ __forceinline__ void iq3s_sub_dot(uint32_t qs_lo, uint32_t qs_hi, uint32_t qh, int sh, uint32_t sg,
                                             const uint32_t* grid_lane, uint32_t sign_base,
                                             const int8_t* const (&act)[TT], int (&P)[TT]) {
  // bit j of a nibble -> byte j (0 or 1): n * (1 + 2^7 + 2^14 + 2^21) has bit j at position 8j
  const uint32_t h_lo = (((qh >> sh) & 0xFu) * 0x00204081u) & 0x01010101u;
  const uint32_t h_hi = (((qh >> (sh + 4)) & 0xFu) * 0x00204081u) & 0x01010101u;
  // sign nibbles pre-scaled by 4 (byte offsets into the mask table)
  const uint32_t s_even = (sg << 2) & 0x3C3C3C3Cu;  // look-ups 0,2,4,6
  const uint32_t s_odd = (sg >> 2) & 0x3C3C3C3Cu;   // look-ups 1,3,5,7
  // An index byte and its ninth bit side by side, times 128 (the bytes of an entry), plus the lane's entry 0: one two-way dot
  // product, which runs on the multiply pipe beside the busier integer one (a byte-permute and a shifted add each: eight
  // layers of one token 147.0 -> 145.5 us, of sixteen 630.6 -> 626.3).
  const uint32_t grid_at = smem_u32(grid_lane);
  const uint32_t idx[4] = {prmt(qs_lo, h_lo, 0x5140u), prmt(qs_lo, h_lo, 0x7362u), prmt(qs_hi, h_hi, 0x5140u),
                           prmt(qs_hi, h_hi, 0x7362u)};
  uint32_t x[8];
#pragma unroll
  for (int l = 0; l < 8; ++l) {
    const uint32_t g = lds_word(__dp2a_lo(idx[l >> 1], (l & 1) ? 0x8000u : 0x0080u, grid_at));
    // byte0 = the pre-scaled nibble of look-up l, bytes 1-3 = the table's address bytes
    // (Computing the masks instead frees a third of the shared-memory wavefronts, and loses: isolating the nibble, one wide multiply
    // that sends bit j to the top of byte j and one sign-replicating byte-permute took 96 us a layer launch of sixteen tokens where
    // loads took 80, the multiplies queuing up in the dispatch stage; a later form without the isolation, see gate_up_sub, eight
    // layers in 640 us where loads take 626.)
    const uint32_t maddr = prmt((l & 1) ? s_odd : s_even, sign_base, 0x7650u | uint32_t(l >> 1));
    x[l] = g ^ lds_word(maddr);
  }
#pragma unroll
  for (int t = 0; t < TT; ++t) {
    const int4 a0 = *reinterpret_cast<const int4*>(act[t]);
    const int4 a1 = *reinterpret_cast<const int4*>(act[t] + 16);
    int p = __dp4a(int(x[0]), a0.x, 0);
    p = __dp4a(int(x[1]), a0.y, p);
    p = __dp4a(int(x[2]), a0.z, p);
    p = __dp4a(int(x[3]), a0.w, p);
    p = __dp4a(int(x[4]), a1.x, p);
    p = __dp4a(int(x[5]), a1.y, p);
    p = __dp4a(int(x[6]), a1.z, p);
    p = __dp4a(int(x[7]), a1.w, p);
    P[t] = p;
  }
}

// Integer dot of one IQ3_S block with TT activation blocks:
//   bsum[t] = sum over its 8 sub-blocks of (2 s + 1) * (2 P + A), exact in int32 (|bsum| < 2^24).
// w = the word that holds the block's fp16 scale (MIS: in its low half, the 27 stream words then sit
// 2 bytes off word alignment; else in its high half and the stream is aligned); act[t] = the 256
// codes of the matching Q8_K block, asum[t] = its 8 sub-block code sums (16-byte aligned).
// |P| <= 32 * 8 * 127 fits 16 bits, so two sub-blocks' P (and their two code sums A) are multiplied by
// their odd multipliers with one two-way dot product each.
template <bool MIS, int TT>
__device__ __forceinline__ void iq3s_block_idot2(const uint32_t* w, const uint32_t* grid_lane, uint32_t sign_base,
                                                 const int8_t* const (&act)[TT], const int16_t* const (&asum)[TT],
                                                 int (&bsum)[TT]) {
  const uint32_t sc = iq3s_stream<MIS>(w, 26);
  // multipliers 2 s + 1 as bytes: even sub-blocks (low nibbles) and odd sub-blocks (high nibbles)
  const uint32_t m_even = ((sc << 1) & 0x1E1E1E1Eu) | 0x01010101u;
  const uint32_t m_odd = ((sc >> 3) & 0x1E1E1E1Eu) | 0x01010101u;
  int4 as[TT];
  int accP[TT], accA[TT];
#pragma unroll
  for (int t = 0; t < TT; ++t) {
    accP[t] = 0;
    as[t] = *reinterpret_cast<const int4*>(asum[t]);
  }
  {  // code-sum part: sum_sb (2 s + 1) * A_sb, four two-way dot products
    const uint32_t mi01 = __byte_perm(m_even, m_odd, 0x5140), mi23 = __byte_perm(m_even, m_odd, 0x7362);
#pragma unroll
    for (int t = 0; t < TT; ++t) {
      int a = __dp2a_lo(as[t].x, int(mi01), 0);
      a = __dp2a_hi(as[t].y, int(mi01), a);
      a = __dp2a_lo(as[t].z, int(mi23), a);
      accA[t] = __dp2a_hi(as[t].w, int(mi23), a);
    }
  }
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const uint32_t qh = iq3s_stream<MIS>(w, 16 + half);
    // bytes {m(4h), m(4h+1), m(4h+2), m(4h+3)} of this half's four sub-blocks
    const uint32_t mi = __byte_perm(m_even, m_odd, half == 0 ? 0x5140u : 0x7362u);
    int P[4][TT];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ib = 4 * half + i;
      const int8_t* a[TT];
#pragma unroll
      for (int t = 0; t < TT; ++t) a[t] = act[t] + 32 * ib;
      iq3s_sub_dot<TT>(iq3s_stream<MIS>(w, 2 * ib), iq3s_stream<MIS>(w, 2 * ib + 1), qh, 8 * i,
                       iq3s_stream<MIS>(w, 18 + ib), grid_lane, sign_base, a, P[i]);
    }
#pragma unroll
    for (int t = 0; t < TT; ++t) {
      const int p01 = int(__byte_perm(uint32_t(P[0][t]), uint32_t(P[1][t]), 0x5410));
      const int p23 = int(__byte_perm(uint32_t(P[2][t]), uint32_t(P[3][t]), 0x5410));
      accP[t] = __dp2a_lo(p01, int(mi), accP[t]);
      accP[t] = __dp2a_hi(p23, int(mi), accP[t]);
    }
  }
#pragma unroll
  for (int t = 0; t < TT; ++t) bsum[t] = 2 * accP[t] + accA[t];
}

// scale of the block, fp16 -> fp32
template <bool MIS>
__device__ __forceinline__ float iq3s_block_d(const uint32_t* w) {
  const uint32_t v = MIS ? (w[0] & 0xFFFFu) : (w[0] >> 16);
  return __half2float(__ushort_as_half(static_cast<unsigned short>(v)));
}

// The 64-byte mask table sits on a 256-byte boundary (its address bytes 1-3 ride in a byte-permute)
// inside an area of kSignArea bytes.
constexpr int kSignArea = 320;
constexpr int kIq2sTableBytes = 1024 * 64;  // eight copies of 1024 x 8 bytes
__device__ __forceinline__ uint32_t* sign_table_at(uint8_t* area) {
  return reinterpret_cast<uint32_t*>(area + ((256u - (smem_u32(area) & 255u)) & 255u));
}

// ------------------------------------------------------------------------------ multi-stage ring
template <int S>
struct RingN {
  uint64_t* full;   // [S] count 1 (DIRECT: and one for every quantizing warp) + tx bytes
  uint64_t* empty;  // [S]
  uint64_t* staged;  // [S] DIRECT: the entry's description stands (count 1, the producer)
  volatile StageMeta* meta;  // [S]
  // number of entries the producer staged in all; kRingOpen while it is still staging; 0 from a time-out on
  volatile int* end_seq;
  volatile int* staged_seq;  // -1, then the entries staged when the producer stopped, whatever made it stop
};
constexpr int kRingOpen = 0x7fffffff;
constexpr uint32_t kStopPolls = 1u << 26;  // polls of shared memory with naps of 40 ns or more: some five seconds

// Bounded: 2^21 tries of at most about a microsecond each.
__device__ __forceinline__ bool mbar_wait_hint(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < (1u << 21); ++i)
    if (mbar_try_wait_hint(bar, parity)) return true;
  return false;
}

// A wait has run out: warps that look at the end mark leave. It stays 0: the producer's count only ever takes the place of
// kRingOpen.
template <int S>
__device__ __forceinline__ void ring_abort(const RingN<S>& r, uint32_t* status) {
  *r.end_seq = 0;
  atomicMax(status, uint32_t(FB_STATUS_PIPELINE_TIMEOUT));
}
template <int S>
__device__ __forceinline__ void ring_close(const RingN<S>& r, int entries) {
  *r.staged_seq = entries;
  __threadfence_block();
  atomicCAS(const_cast<int*>(r.end_seq), kRingOpen, entries);
}
// By one lane of the warp whose wait ran out: warps that leave early leave entries behind, and no block may end with copies
// on their way into its shared memory. Waits (bounded) until the producer has stopped, then for the last entries' barriers.
// The producer may be in its wait for a slot, some two seconds at most, which does not look at the end mark (eight layers of
// one token take 148.5 us where it does, 146.5 as it is; a look at the end of every warp costs them 1 us as well).
template <int S>
__device__ __noinline__ void ring_drain(const RingN<S>& r) {
  for (uint32_t i = 0; *r.staged_seq < 0 && i < kStopPolls; ++i) __nanosleep(100);
  const int n = *r.staged_seq;
  for (int e = max(0, n - S); e < n; ++e) mbar_wait_hint(&r.full[e % S], (e / S) & 1);
}

template <int S>
__device__ __forceinline__ void ringn_init(const RingN<S>& r, int arrivals) {
  for (int s = 0; s < S; ++s) {
    mbar_init(&r.full[s], arrivals);
    mbar_init(&r.empty[s], 1);  // one arrival frees a slot: the warp that finishes the entry's last task
    mbar_init(&r.staged[s], 1);
    r.meta[s].tile = -1;
    r.meta[s].seq = -1;
  }
  *r.end_seq = kRingOpen;
  *r.staged_seq = -1;
  mbar_fence_init();
}

// Consumer side: draws the next (entry, task) ticket and waits for that entry's data; returns false
// at the end. A warp may hold a ticket for an entry that is S or more entries ahead of the one its slot
// is being filled with, and the barrier's one-bit phase cannot tell those apart. So the warp first waits
// (polling one shared-memory word, asleep in between) until the producer has written this entry's number
// into the slot, which it does before it arms the barrier; only then is the barrier's current phase the
// entry's own, and the warp can sleep inside try_wait.
template <int S, int TASKS>
__device__ __forceinline__ bool draw_task_n(const RingN<S>& r, int* ticket_ctr, uint32_t* status, int lane, int& s,
                                            int& task) {
  int ticket = 0;
  if (lane == 0) ticket = atomicAdd(ticket_ctr, 1);
  ticket = __shfl_sync(0xffffffffu, ticket, 0);
  const int seq = ticket / TASKS;
  task = ticket - seq * TASKS;
  s = seq % S;
  uint32_t tries = 0;
  while (r.meta[s].seq != seq) {
    if (*r.end_seq <= seq) return false;
    if (++tries > (1u << 20)) {  // bounded: a quarter of a second
      ring_abort(r, status);
      if (lane == 0) ring_drain(r);
      return false;
    }
    // (the producer is behind only at the start of a phase; the nap is short because at one to three tokens this
    // wait sits on the layer's critical path)
    __nanosleep(200);
  }
  const uint32_t parity = (seq / S) & 1;
  for (uint32_t i = 0; i < (1u << 21); ++i) {  // bounded: each try takes at most about a microsecond
    if (mbar_try_wait_hint(&r.full[s], parity)) return true;
    if (*r.end_seq <= seq) return false;
  }
  ring_abort(r, status);
  if (lane == 0) ring_drain(r);
  return false;
}

// ------------------------------------------------------------------------------ the expert kernel
// Gate/up tile = 16 intermediate rows: 16 gate rows and the 16 matching up rows; task b (0..9) = block b (256 weights)
// of all 32 rows, lanes 0-15 the gate rows, lanes 16-31 the up rows; the warp that finishes the tile's last task adds
// each row's ten block terms in block order, pairs gate with up through a shuffle and applies SwiGLU.
// Down tile = 160 output rows at intermediate 512, 128 at 640; task 2k + b = half b (256 or 320 weights) of rows
// 32k .. 32k+31 (at 640 the tasks 8 and 9 are empty); the finishing warp adds each row's two half terms and applies the
// routing weight. Both kinds carry the activation rows of the pass behind the weights.
// Bytes of 256 gate/up weights of one row, and the shared-memory table that decodes them (sign masks included).
template <int FMT>
struct GuFmt;
template <>
struct GuFmt<FB_FMT_IQ3_S> { static constexpr int kBlock = 110, kTable = kGridRepBytes + kSignArea; };
template <>
struct GuFmt<FB_FMT_IQ4_NL> { static constexpr int kBlock = 144, kTable = 0; };  // eight 18-byte blocks; levels in registers
template <>
struct GuFmt<FB_FMT_IQ2_S> { static constexpr int kBlock = 82, kTable = kIq2sTableBytes + kSignArea; };
template <>
struct GuFmt<FB_FMT_IQ3_XXS> { static constexpr int kBlock = 98, kTable = 256 * 32 * 4 + kSignArea; };
template <>
struct GuFmt<FB_FMT_IQ4_XS> { static constexpr int kBlock = 136, kTable = 0; };

constexpr int kStaticSmem = 7168;  // the kernel's own shared variables, at most
template <int GU, int DN, int INTER>
struct ExpertsCfg {
  static constexpr int kWarps = 24, kTasks = 10, kInter = INTER;
  // consumers, the producer, and where h rows carry their own arrival flags the warps that quantize them
  static constexpr int threads(bool direct) { return (kWarps + 1 + (direct ? direct_warps(INTER) : 0)) * 32; }
  static constexpr int kTaskBytes = GuFmt<GU>::kBlock;
  static constexpr int kGuRows = 16, kGuRowBytes = kTasks * kTaskBytes, kGuPart = kGuRows * kGuRowBytes;
  static constexpr int kDnTaskBytes = DN == FB_FMT_IQ3_S ? 110 : INTER / (DN == FB_FMT_Q2_0 ? 128 : 64) * 18;  // half a row
  static constexpr int kDnRows = INTER == 512 ? 160 : 128, kDnRowBytes = 2 * kDnTaskBytes, kDnTile = kDnRows * kDnRowBytes;
  static constexpr int kAct = act_of(GU);
  static constexpr int kGuAct = kAct == FB_ACT_Q8_K ? q8k_planar_bytes(H) : H + H / 8;
  static constexpr int kDnAct = DN == FB_FMT_IQ3_S ? q8k_planar_bytes(INTER) : INTER + INTER / 8;
  static constexpr int kGuBytes = 2 * kGuPart + kTT * kGuAct, kDnBytes = kDnTile + kTT * kDnAct;
  static constexpr int kSlot = kGuBytes > kDnBytes ? kGuBytes : kDnBytes;
  static constexpr int kDnTilesPerItem = H / kDnRows;
  static constexpr int kTableBytes = GuFmt<GU>::kTable;
  // block terms of the tasks in flight; before the first task the selection's scratch memory
  static constexpr size_t partials_of(int stages) {
    const size_t terms = size_t(stages) * kTasks * kTT * 32 * 4, scratch = (sizeof(SelectScratch) + 15) & ~size_t(15);
    return terms > scratch ? terms : scratch;
  }
  static constexpr size_t smem_of(int stages) {
    return size_t(kTableBytes) + size_t(stages) * kSlot + partials_of(stages) + 128;
  }
  // 24 warps work on 2.4 tiles at a time, so of three slots little more than a half is in flight from memory: four where
  // they fit (the formats without a table)
  static constexpr int kStages = smem_of(4) + kStaticSmem <= 232448 ? 4 : 3;
  static constexpr int kPartialFloats = int(partials_of(kStages) / 4);
  static constexpr size_t kSmem = smem_of(kStages);
  static_assert(DN == FB_FMT_IQ4_NL || DN == FB_FMT_Q2_0 || (DN == FB_FMT_IQ3_S && GU == FB_FMT_IQ3_S && INTER == 512),
                "IQ3_S down shares the gate/up codebook and needs whole blocks per half row");
  static_assert(kTableBytes % 16 == 0 && kSlot % 16 == 0 && kGuPart % 16 == 0 && kDnTile % 16 == 0 && kGuAct % 16 == 0 &&
                    kDnAct % 16 == 0 && H % kDnRows == 0 && kDnRows % 32 == 0 && 2 * (kDnRows / 32) <= kTasks,
                "tile shapes, bulk-copy sizes");
  static_assert(kSmem + kStaticSmem <= 232448, "dynamic plus static shared memory of a block");
};
// kPhaseSelect: the CTA builds the work list itself from the router logits (SelectArgs) instead of
// reading the device work list a selection kernel left.
enum { kPhaseGateUp = 1, kPhaseDown = 2, kPhaseSelect = 4 };

// ------------------------------------------------------------------------------ tables of the gate/up formats
// The packed codebooks once more in global memory: a warp reads 32 different entries, which constant memory would deliver
// one by one.
static __device__ uint16_t g_iq3s_grid_packed[512] = {FB_IQ3S_GRID_PACKED};
static __device__ uint16_t g_iq3xxs_grid_packed[256] = {FB_IQ3XXS_GRID_PACKED};
static __device__ uint16_t g_iq2s_grid_packed[1024] = {FB_IQ2S_GRID_PACKED};
// IQ3_S: the half codebook, replicated per lane. IQ2_S: 1024 entries of eight magnitudes, eight copies (entry i of
// copy c at byte 64 i + 8 c, a lane reads copy lane % 8: two lanes of a half warp share two bank groups, 3 passes per
// look-up of eight weights against 6 with one copy). IQ3_XXS: 256 entries of four magnitudes, one copy per lane.
// A warp expands 32 entries, one per lane, and its lanes then write consecutive 16-byte pieces of the copies (no bank
// conflicts), the values coming through shuffles: 0.8 us for IQ3_S, up to 1.3 for IQ2_S, between the route kernel's end and
// the selection on the multiprocessors that the route kernel leaves last (1.0 and 3.0 with a constant-memory read and an
// expansion per 16 bytes written).
template <int FMT>
__device__ __forceinline__ void experts_table_fill(uint32_t* grid, uint32_t* signtab) {
  if constexpr (FMT == FB_FMT_IQ3_S || FMT == FB_FMT_IQ2_S || FMT == FB_FMT_IQ3_XXS) {
    constexpr int kEntries = FMT == FB_FMT_IQ3_S ? 512 : FMT == FB_FMT_IQ2_S ? 1024 : 256;
    constexpr int kPieces = FMT == FB_FMT_IQ2_S ? 4 : 8;  // 16-byte pieces of an entry's copies
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int e0 = 32 * (threadIdx.x >> 5); e0 < kEntries; e0 += int(blockDim.x)) {
      uint2 w = make_uint2(0u, 0u);
      if constexpr (FMT == FB_FMT_IQ3_S) w.x = (iq3s_expand(g_iq3s_grid_packed[e0 + lane]) >> 1) & 0x07070707u;
      else if constexpr (FMT == FB_FMT_IQ2_S) w = iq2s_expand(g_iq2s_grid_packed[e0 + lane]);
      else w.x = iq3xxs_expand(g_iq3xxs_grid_packed[e0 + lane]);
      uint4* out = reinterpret_cast<uint4*>(grid) + size_t(e0) * kPieces + lane;
#pragma unroll
      for (int k = 0; k < kPieces; ++k) {
        const int src = (32 * k + lane) / kPieces;
        const uint32_t x = __shfl_sync(0xffffffffu, w.x, src);
        const uint32_t y = FMT == FB_FMT_IQ2_S ? __shfl_sync(0xffffffffu, w.y, src) : x;
        out[32 * k] = make_uint4(x, y, x, y);
      }
    }
    sign_table_fill(signtab);
  }
}

// ------------------------------------------------------------------------------ one block against the pass's tokens
// One 32-weight sub-block of the other formats as eight words of int8 weights in natural order. w = the word that holds
// the block's scale (even blocks: in its low half), as iq3s_stream reads it; IQ4_XS: the block's words. With a codebook, q =
// magnitudes ^ mask (0xFF in the bytes of negative weights): a negative weight's byte is one less than the weight, and the
// caller takes dp4a(mask, a) off. (Two more integer operations per four weights made the weights themselves: four layers
// of eight IQ3_XXS tokens 280 -> 276 us.)
template <int FMT, bool EVEN>
__device__ __forceinline__ void gate_up_sub(const uint32_t* w, int ib, const uint32_t* grid, uint32_t sign_base,
                                            const Iq4nlLevels& lv, int (&q)[8], int (&mask)[8], int& m0, int& m1) {
  if constexpr (FMT == FB_FMT_IQ4_XS) {
    const uint32_t head = w[0], sl = w[1];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint2 v = reinterpret_cast<const uint2*>(w)[1 + 2 * ib + h];
      const uint32_t qq[2] = {v.x, v.y};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t sel = qq[i] & 0x77777777u, pick = ((qq[i] >> 1) & 0x44444444u) | 0x32103210u;
        const uint32_t r0 = prmt(prmt(lv.t0, lv.t1, sel), prmt(lv.t2, lv.t3, sel), pick);
        const uint32_t sel1 = upper_half(sel);
        const uint32_t r1 = prmt(prmt(lv.t0, lv.t1, sel1), prmt(lv.t2, lv.t3, sel1), upper_half(pick));
        q[2 * h + i] = int(prmt(r0, r1, 0x6420u));      // low nibbles: weights 4j .. 4j + 3
        q[4 + 2 * h + i] = int(prmt(r0, r1, 0x7531u));  // high nibbles: weights 16 + 4j ..
      }
    }
    m0 = m1 = int(((sl >> (8 * (ib >> 1) + 4 * (ib & 1))) & 15u) | (((head >> (16 + 2 * ib)) & 3u) << 4)) - 32;
  } else {
    uint32_t g[8], sg;
    if constexpr (FMT == FB_FMT_IQ2_S) {
      const uint32_t qs = iq3s_stream<EVEN>(w, ib), qh = (iq3s_stream<EVEN>(w, 16 + (ib >> 2)) >> (8 * (ib & 3))) & 0xFFu;
      sg = iq3s_stream<EVEN>(w, 8 + ib);
      const uint32_t sc = iq3s_stream<EVEN>(w, 18 + (ib >> 2)) >> (8 * (ib & 3));
      m0 = int((sc << 1) & 30u) + 1;
      m1 = int((sc >> 3) & 30u) + 1;
      // byte offsets 64 * index + 8 * (lane % 8) of two look-ups per word: the index byte in bits 6..13 (22..29), its two
      // upper bits, taken from qh by a multiply that lands them on bits 14 and 15 (30 and 31)
      const uint32_t lane_pat = (threadIdx.x & 7) * 0x00080008u, grid_at = smem_u32(grid);
      const uint32_t a02 = ((qs << 6) & 0x3FC03FC0u) | lane_pat | ((qh * 0x04004000u) & 0xC000C000u);
      const uint32_t a13 = ((qs >> 2) & 0x3FC03FC0u) | lane_pat | ((qh * 0x01001000u) & 0xC000C000u);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const uint32_t at = __dp2a_lo((l & 1) ? a13 : a02, (l & 2) ? 0x0100u : 0x0001u, grid_at);
        asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(g[2 * l]), "=r"(g[2 * l + 1]) : "r"(at));
      }
    } else {
      const uint32_t aux = iq3s_stream<EVEN>(w, 16 + ib);
      m0 = m1 = 2 * int(aux >> 28) + 1;
      // four 7-bit sign indices into bytes, the eighth sign is their parity
      sg = (aux & 0x7Fu) | ((aux << 1) & 0x7F00u) | ((aux << 2) & 0x7F0000u) | ((aux << 3) & 0x7F000000u);
      uint32_t p = sg ^ (sg >> 4);
      p ^= p >> 2;
      p ^= p >> 1;
      sg |= (p & 0x01010101u) << 7;
      const uint32_t grid_at = smem_u32(grid) + 4 * (threadIdx.x & 31);
#pragma unroll
      for (int l = 0; l < 8; ++l)  // (byte times 128 plus base in one dot product: 276 -> 259 us)
        g[l] = lds_word(__dp4a(iq3s_stream<EVEN>(w, 2 * ib + (l >> 2)), 128u << (8 * (l & 3)), grid_at));
    }
    const uint32_t s_even = (sg << 2) & 0x3C3C3C3Cu, s_odd = (sg >> 2) & 0x3C3C3C3Cu;  // nibbles as byte offsets, see iq3s_sub_dot
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      uint32_t m;
      if constexpr (FMT == FB_FMT_IQ2_S) {
        // Shared memory is the busy unit here (look-ups of eight bytes in three passes), so the mask is made: a sign byte times
        // 0x80402010 has bit 3 - j at bit 7 of byte j, times 0x08040201 bit 7 - j, and a byte-permute spreads them over the
        // bytes and turns them round. (Eight layers of five tokens 383 -> 371 us. The others, whose look-ups take one
        // pass, lose by it: IQ3_XXS 259 -> 262, IQ3_S at sixteen tokens 626 -> 640.)
        m = prmt(__dp4a(sg, 1u << (8 * (l >> 1)), 0u) * ((l & 1) ? 0x08040201u : 0x80402010u), 0u, 0x89ABu);
      } else {
        m = lds_word(prmt((l & 1) ? s_odd : s_even, sign_base, 0x7650u | uint32_t(l >> 1)));
      }
      q[l] = int(g[l] ^ m);
      mask[l] = int(m);
    }
  }
}

template <int FMT, bool EVEN, int TT>
__device__ __forceinline__ void gate_up_block_idot(const uint32_t* w, const uint32_t* grid, uint32_t sign_base,
                                                   const Iq4nlLevels& lv, const int8_t* const (&act)[TT], int (&bsum)[TT]) {
#pragma unroll
  for (int t = 0; t < TT; ++t) bsum[t] = 0;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ib = 4 * half + i;
      int q[8], mask[8], m0, m1;
      gate_up_sub<FMT, EVEN>(w, ib, grid, sign_base, lv, q, mask, m0, m1);
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        const int4 a0 = *reinterpret_cast<const int4*>(act[t] + 32 * ib);
        const int4 a1 = *reinterpret_cast<const int4*>(act[t] + 32 * ib + 16);
        int s0 = __dp4a(q[0], a0.x, 0);
        s0 = __dp4a(q[1], a0.y, s0);
        s0 = __dp4a(q[2], a0.z, s0);
        s0 = __dp4a(q[3], a0.w, s0);
        int s1 = __dp4a(q[4], a1.x, FMT == FB_FMT_IQ2_S ? 0 : s0);
        s1 = __dp4a(q[5], a1.y, s1);
        s1 = __dp4a(q[6], a1.z, s1);
        s1 = __dp4a(q[7], a1.w, s1);
        if constexpr (FMT != FB_FMT_IQ4_XS) {
          int c0 = __dp4a(mask[0], a0.x, 0);
          c0 = __dp4a(mask[1], a0.y, c0);
          c0 = __dp4a(mask[2], a0.z, c0);
          c0 = __dp4a(mask[3], a0.w, c0);
          int c1 = __dp4a(mask[4], a1.x, FMT == FB_FMT_IQ2_S ? 0 : c0);
          c1 = __dp4a(mask[5], a1.y, c1);
          c1 = __dp4a(mask[6], a1.z, c1);
          c1 = __dp4a(mask[7], a1.w, c1);
          s0 -= c0;
          s1 -= c1;
        }
        bsum[t] += FMT == FB_FMT_IQ2_S ? m0 * s0 + m1 * s1 : m0 * s1;
      }
    }
  }
}

// One block (256 weights) of the lane's row against the pass's tokens: term[t] = bsum * d * d_act. EVEN: the block starts
// on a word; ablk = index of the Q8_K block it meets in the activation row of k values.
template <int FMT, bool EVEN>
__device__ __forceinline__ void gate_up_block_terms(const uint8_t* blk, const uint32_t* grid, uint32_t sign_base,
                                                    const Iq4nlLevels& lv, const uint8_t* act0, int act_bytes, int ablk,
                                                    int ntp, float (&term)[kTT], int k = H) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(EVEN || FMT == FB_FMT_IQ4_XS ? blk : blk - 2);
  constexpr bool kLow = EVEN || FMT == FB_FMT_IQ4_XS;  // the scale sits in the low half of its word
  constexpr float kFactor = FMT == FB_FMT_IQ2_S ? 0.125f : FMT == FB_FMT_IQ3_XXS ? 0.25f : 1.0f;
  const float d = iq3s_block_d<kLow>(w) * kFactor;
  auto dots = [&](auto& a, auto& as, auto& bs) {
    constexpr int TT = sizeof(bs) / sizeof(int);
    if constexpr (FMT == FB_FMT_IQ3_S) iq3s_block_idot2<EVEN, TT>(w, grid + (threadIdx.x & 31), sign_base, a, as, bs);
    else gate_up_block_idot<FMT, EVEN, TT>(w, grid, sign_base, lv, a, bs);
  };
  if (ntp == 1) {
    const int8_t* a[1] = {reinterpret_cast<const int8_t*>(act0) + 256 * ablk};
    const int16_t* as[1] = {reinterpret_cast<const int16_t*>(act0 + q8k_planar_asum_off(k)) + 8 * ablk};
    int bs[1];
    dots(a, as, bs);
    term[0] = float(bs[0]) * (d * reinterpret_cast<const float*>(act0 + k)[ablk]);
  } else {
    const uint8_t* act1 = act0 + act_bytes;
    const int8_t* a[2] = {reinterpret_cast<const int8_t*>(act0) + 256 * ablk,
                          reinterpret_cast<const int8_t*>(act1) + 256 * ablk};
    const int16_t* as[2] = {reinterpret_cast<const int16_t*>(act0 + q8k_planar_asum_off(k)) + 8 * ablk,
                            reinterpret_cast<const int16_t*>(act1 + q8k_planar_asum_off(k)) + 8 * ablk};
    int bs[2];
    dots(a, as, bs);
    term[0] = float(bs[0]) * (d * reinterpret_cast<const float*>(act0 + k)[ablk]);
    term[1] = float(bs[1]) * (d * reinterpret_cast<const float*>(act1 + k)[ablk]);
  }
}

// IQ4_NL: one task = eight consecutive 18-byte blocks of the lane's row at `wp`, against the pass's tokens; blk0 = index of the
// first of them in the row. Even blocks start on a word (scale in the low half, codes two bytes off), odd blocks on a half word
// (scale in the high half, codes aligned). Rows of 1440 and 288 bytes keep eight blocks on 16-byte boundaries: the widest
// loads. term[t] = sum over the blocks, in block order, of isum * (d * d_act). (Four blocks at a time, with their words moved
// into place: half the code, eight layers of eight tokens 354.6 -> 351.8 us, but of one 132.8 -> 136.0.)
__device__ __forceinline__ void iq4nl_task_terms(const uint8_t* wp, const Iq4nlLevels& lv, const uint8_t* act0,
                                                 int act_bytes, int k, int blk0, int ntp, float (&term)[kTT]) {
  uint32_t w[36];
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    const uint4 v = reinterpret_cast<const uint4*>(wp)[c];
    w[4 * c] = v.x;
    w[4 * c + 1] = v.y;
    w[4 * c + 2] = v.z;
    w[4 * c + 3] = v.w;
  }
  term[0] = term[1] = 0.0f;
  const uint8_t* act1 = act0 + (ntp == 2 ? act_bytes : 0);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int base = b % 2 == 0 ? 9 * b / 2 : (18 * b - 2) / 4;  // the word with the scale
    const float d = __half2float(__ushort_as_half(static_cast<unsigned short>(b % 2 == 0 ? w[base] & 0xFFFFu : w[base] >> 16)));
    int lo[8], hi[8];
    iq4nl_addends32(lv, w, 2 * base + (b % 2 == 0 ? 1 : 2), lo, hi);
    const int blk = blk0 + b;
    const int s0 = dot32(lo, hi, reinterpret_cast<const int8_t*>(act0) + 32 * blk);
    term[0] = fmaf(float(s0), d * reinterpret_cast<const float*>(act0 + k)[blk], term[0]);
    if (ntp == 2) {
      const int s1 = dot32(lo, hi, reinterpret_cast<const int8_t*>(act1) + 32 * blk);
      term[1] = fmaf(float(s1), d * reinterpret_cast<const float*>(act1 + k)[blk], term[1]);
    }
  }
}
// The same for half a row of 640: ten blocks, two at a time from single words (rows of 360 bytes: two lanes share a bank), so
// that the code stands in the kernel once and is short. (The warps waited for instructions most: with all ten blocks unrolled, once
// for either half, eight layers of five IQ2_S + IQ4_NL tokens took 363 us, 327 so; the decode branch of four tokens 420, 378.)
__device__ __forceinline__ void iq4nl_half_row_terms(const uint8_t* half, const Iq4nlLevels& lv, const uint8_t* act0, int act_bytes,
                                                     int k, int blk0, int ntp, float (&term)[kTT]) {
  term[0] = term[1] = 0.0f;
  const uint8_t* act1 = act0 + (ntp == 2 ? act_bytes : 0);
#pragma unroll 1
  for (int p = 0; p < 5; ++p) {
    uint32_t w[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) w[i] = reinterpret_cast<const uint32_t*>(half)[9 * p + i];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const float d = __half2float(__ushort_as_half(static_cast<unsigned short>(b == 0 ? w[0] & 0xFFFFu : w[4] >> 16)));
      int lo[8], hi[8];
      iq4nl_addends32(lv, w, b == 0 ? 1 : 10, lo, hi);
      const int blk = blk0 + 2 * p + b;
      const int s0 = dot32(lo, hi, reinterpret_cast<const int8_t*>(act0) + 32 * blk);
      term[0] = fmaf(float(s0), d * reinterpret_cast<const float*>(act0 + k)[blk], term[0]);
      if (ntp == 2) {
        const int s1 = dot32(lo, hi, reinterpret_cast<const int8_t*>(act1) + 32 * blk);
        term[1] = fmaf(float(s1), d * reinterpret_cast<const float*>(act1 + k)[blk], term[1]);
      }
    }
  }
}
// Q2_0: one task = NB consecutive 18-byte blocks (64 weights, codes 0..3 for -1..2) of the lane's row, OFF (0 or 2) bytes
// behind the word `wp`. A code is a byte-permute's selector into the four levels once every other code of a byte is masked
// off; eight more permutes put sixteen weights into the activations' interleaved order. Rows of 180 bytes (45 words) are
// read without bank conflicts word by word, rows of 144 bytes in pairs of words.
template <int NB, int OFF>
__device__ __forceinline__ void q2_0_task_terms(const uint8_t* wp, const uint8_t* act0, int act_bytes, int k, int sub0,
                                                int ntp, float (&term)[kTT]) {
  constexpr int kWords = (OFF + 18 * NB + 3) / 4;
  constexpr uint32_t kLevels = 0x020100FFu, kPairs = 0x33333333u;
  uint32_t w[kWords];
  if constexpr (NB == 4) {
#pragma unroll
    for (int c = 0; c < kWords / 2; ++c) {
      const uint2 v = reinterpret_cast<const uint2*>(wp)[c];
      w[2 * c] = v.x;
      w[2 * c + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int c = 0; c < kWords; ++c) w[c] = reinterpret_cast<const uint32_t*>(wp)[c];
  }
  term[0] = term[1] = 0.0f;
  const uint8_t* act1 = act0 + (ntp == 2 ? act_bytes : 0);
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int at = OFF + 18 * b;  // even: the block's scale is the low or the high half of its word
    const uint32_t head = w[at / 4];
    const float d = __half2float(__ushort_as_half(static_cast<unsigned short>(at % 4 ? head >> 16 : head & 0xFFFFu)));
#pragma unroll
    for (int sub = 0; sub < 2; ++sub) {
      uint32_t c[2];  // codes 0..15 and 16..31 of the sub-block
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int n = at / 4 + 2 * sub + i;
        c[i] = at % 4 ? w[n + 1] : __funnelshift_r(w[n], w[n + 1], 16);
      }
      // selectors of the even and of the odd weights
      const uint32_t e0 = c[0] & kPairs, o0 = (c[0] >> 2) & kPairs, e1 = c[1] & kPairs, o1 = (c[1] >> 2) & kPairs;
      int wq[8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t A = prmt(kLevels, 0u, h ? upper_half(e0) : e0), B = prmt(kLevels, 0u, h ? upper_half(o0) : o0);
        const uint32_t C = prmt(kLevels, 0u, h ? upper_half(e1) : e1), D = prmt(kLevels, 0u, h ? upper_half(o1) : o1);
        const uint32_t ac0 = prmt(A, C, 0x5140u), ac1 = prmt(A, C, 0x7362u), bd0 = prmt(B, D, 0x5140u), bd1 = prmt(B, D, 0x7362u);
        wq[4 * h] = int(prmt(ac0, bd0, 0x5410u));  // weights 2j, 2j + 16, 2j + 1, 2j + 17
        wq[4 * h + 1] = int(prmt(ac0, bd0, 0x7632u));
        wq[4 * h + 2] = int(prmt(ac1, bd1, 0x5410u));
        wq[4 * h + 3] = int(prmt(ac1, bd1, 0x7632u));
      }
      const int blk = sub0 + 2 * b + sub;
      const int s0 = dot32(wq, reinterpret_cast<const int8_t*>(act0) + 32 * blk);
      term[0] = fmaf(float(s0), d * reinterpret_cast<const float*>(act0 + k)[blk], term[0]);
      if (ntp == 2) {
        const int s1 = dot32(wq, reinterpret_cast<const int8_t*>(act1) + 32 * blk);
        term[1] = fmaf(float(s1), d * reinterpret_cast<const float*>(act1 + k)[blk], term[1]);
      }
    }
  }
}
// The combine of the fused layer call, by the warps that finish down tiles: a tile's rows of a token are counted, and the
// warp that brings the last of the token's pairs adds the columns' partial rows in slot order (the order, hence the
// bits, of combine_kernel). A launch of its own behind this kernel cost a layer of one token 4 us.
template <int ROWS>
__device__ __forceinline__ void combine_tile(const fb_moe_decode_workspace& ws, const SelectArgs& sel, const WorkCache& wc,
                                             int pair0, int ntp, int r0, int lane) {
  int mine = 0;
  if (lane < ntp) {  // release and acquire ride on the atomic; the warp's stores are ordered before it by the __syncwarp
    int* counter = ws.sched + kSchedParts + wc.pair_token[pair0 + lane] * kMaxDnTiles + r0 / ROWS;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(mine) : "l"(counter) : "memory");
  }
  for (int i = 0; i < ntp; ++i) {
    const int before = __shfl_sync(0xffffffffu, mine, i);
    if (before != kTopK - 1) continue;
    __syncwarp();  // (the shuffle orders no memory: the other lanes read the partial rows behind their lane's acquire by this)
    const int t = wc.pair_token[pair0 + i];
    int row[kTopK];
#pragma unroll
    for (int k = 0; k < kTopK; ++k) row[k] = wc.token_row[t][k];
    for (int c = 4 * lane; c < ROWS; c += 128) {
      float4 v[kTopK];
#pragma unroll
      for (int k = 0; k < kTopK; ++k)
        v[k] = __ldcg(reinterpret_cast<const float4*>(ws.partial + size_t(row[k]) * H + r0 + c));
      float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int k = 0; k < kTopK; ++k) {
        y.x += v[k].x;
        y.y += v[k].y;
        y.z += v[k].z;
        y.w += v[k].w;
      }
      float* out = sel.y_out + size_t(t) * H + r0 + c;  // (any 4-byte alignment)
      if ((reinterpret_cast<uintptr_t>(sel.y_out) & 15) == 0) {
        *reinterpret_cast<float4*>(out) = y;
      } else {
        out[0] = y.x;
        out[1] = y.y;
        out[2] = y.z;
        out[3] = y.w;
      }
    }
  }
}

// The same where rows are their own arrival flags: the warp that finished the tile of the token's pair that is visited last
// polls the other pairs' rows (false: a wait has run out). What it waits for comes before its own tile in the order in which
// tiles are drawn and tasks taken, so the earliest unfinished tile never waits for a polling warp.
template <int ROWS, int S>
__device__ __forceinline__ bool combine_tile_direct(const fb_moe_decode_workspace& ws, const SelectArgs& sel,
                                                    const WorkCache& wc, int pair0, int ntp, int r0, int lane,
                                                    const RingN<S>& ring) {
  for (int i = 0; i < ntp; ++i) {
    const int t = wc.pair_token[pair0 + i];
    if (wc.last_pair[t] != pair0 + i) continue;
    int row[kTopK];
#pragma unroll
    for (int k = 0; k < kTopK; ++k) row[k] = wc.token_row[t][k];
#pragma unroll 1
    for (int c0 = 0; c0 < ROWS; c0 += 128) {
      const int c = c0 + 4 * lane;
      float4 y;
      uint32_t tries = 0;
      while (true) {
        bool all = true;
        y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (c < ROWS) {
          float4 v[kTopK];
#pragma unroll
          for (int k = 0; k < kTopK; ++k) v[k] = direct_load4(ws.partial + size_t(row[k]) * H + r0 + c, all);
#pragma unroll
          for (int k = 0; k < kTopK; ++k) {
            y.x += v[k].x;
            y.y += v[k].y;
            y.z += v[k].z;
            y.w += v[k].w;
          }
        }
        if (__all_sync(0xffffffffu, all)) break;
        if (__shfl_sync(0xffffffffu, *ring.end_seq, 0) == 0) return false;
        if (++tries > value_polls(ws)) {
          if (lane == 0) {
            ring_abort(ring, ws.status);
            ring_drain(ring);
          }
          return false;
        }
        __nanosleep(20);
      }
      if (c >= ROWS) continue;
      float* out = sel.y_out + size_t(t) * H + r0 + c;  // (any 4-byte alignment)
      if ((reinterpret_cast<uintptr_t>(sel.y_out) & 15) == 0) {
        *reinterpret_cast<float4*>(out) = y;
      } else {
        out[0] = y.x;
        out[1] = y.y;
        out[2] = y.z;
        out[3] = y.w;
      }
    }
  }
  return true;
}

// DIRECT (all phases, up to direct_tokens): h and the partial rows are their own arrival flags (direct_store), and two or
// three more warps, each its 256 values, quantize the h rows of this CTA's down entries as they arrive. One token of IQ3_S:
// by counters 161 us for eight layers, with one quantizing warp 154, with two 147. (As a run-time switch it cost sixteen
// tokens 2 to 3 %.)
template <int GU, int DN, int INTER, bool DIRECT>
__global__ void __launch_bounds__(ExpertsCfg<GU, DN, INTER>::threads(DIRECT), 1)
experts_kernel(fb_moe_expert_layout L, fb_moe_decode_workspace ws, int phases, SelectArgs sel) {
  using C = ExpertsCfg<GU, DN, INTER>;
  constexpr int S = C::kStages;
  constexpr bool kSigns = GU == FB_FMT_IQ3_S || GU == FB_FMT_IQ2_S || GU == FB_FMT_IQ3_XXS;
  extern __shared__ __align__(128) uint8_t smem[];
  uint32_t* grid = reinterpret_cast<uint32_t*>(smem);  // the gate/up format's codebook, its sign masks behind it
  uint32_t* signtab = kSigns ? sign_table_at(smem + (C::kTableBytes - kSignArea)) : nullptr;
  uint8_t* stage0 = smem + C::kTableBytes;
  float* partials = reinterpret_cast<float*>(stage0 + S * C::kSlot);
  uint64_t* bars = reinterpret_cast<uint64_t*>(partials + C::kPartialFloats);
  __shared__ StageMeta s_meta[S];
  __shared__ int s_misc[3 + S];  // [1..2] task tickets (even / odd blocks), [3..] finished tasks per slot
  __shared__ int s_end, s_staged;
  __shared__ WorkCache s_work;
  static_assert(3 * S * sizeof(uint64_t) <= 128, "barriers behind the block terms");
  RingN<S> ring{bars, bars + S, bars + 2 * S, s_meta, &s_end, &s_staged};

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // (a down-only launch of another format than IQ3_S looks nothing up)
  if (DN == FB_FMT_IQ3_S || (phases & kPhaseGateUp)) experts_table_fill<GU>(grid, signtab);
  if (tid == 0) {
    ringn_init(ring, DIRECT ? 1 + direct_warps(INTER) : 1);
    for (int i = 1; i < 3 + S; ++i) s_misc[i] = 0;
  }
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait_prior();

  int n_items;
  if (phases & kPhaseSelect) {
    select_block<DIRECT>([&](int t, int e) { return __ldcg(sel.logits + size_t(t) * sel.stride + e); }, sel.slot_of, sel.tokens, ws,
                 nullptr, sel.remote_ok != 0, blockIdx.x == 0, false, s_work, *reinterpret_cast<SelectScratch*>(partials));
    n_items = s_work.n_items;
  } else {
    n_items = min(max(ws.work->n_items, 0), kMaxPairs);
  }
  const uint8_t* xq_rows = ws.xq + xq_offset(C::kAct);
  constexpr int gu_tpi = INTER / C::kGuRows;
  const int n_gu = (phases & kPhaseGateUp) ? n_items * gu_tpi : 0;
  const int n_dn = (phases & kPhaseDown) ? n_items * C::kDnTilesPerItem : 0;
  const int down_act = act_of(L.down_format);

  if (warp == C::kWarps) {
    // ---------------- producer: one lane draws tiles (two steps ahead of their use) and issues their
    // bulk copies into the ring; every pass of kTT tokens of a tile is one ring entry.
    if (!(phases & kPhaseSelect)) {
      work_cache_fill(ws, s_work, n_items);
      __syncwarp();
    }
    if (lane != 0) return;
    int* counter = ws.sched + ((phases & kPhaseGateUp) ? kSchedGateUp : kSchedDown);
    const int n_tiles = n_gu + n_dn;
    int i = 0;
    bool failed = false;
    struct EndMark {  // whichever way the loop is left, waiting warps learn how many entries exist
      const RingN<S>& r;
      const int& i;
      const bool& failed;
      __device__ ~EndMark() {
        ring_close(r, i);
        if (failed) ring_drain(r);
      }
    } end_mark{ring, i, failed};
    auto give_up = [&]() {
      failed = true;
      ring_abort(ring, ws.status);
    };
    auto slot_free = [&](int s) -> bool {
      if (*ring.end_seq == 0) {  // another warp gave up
        failed = true;
        return false;
      }
      if (i >= S && !mbar_wait_hint(&ring.empty[s], ((i / S) - 1) & 1)) {
        give_up();
        return false;
      }
      return true;
    };
    // With three slots, whatever lies between a slot's release and its next copy is lost streaming time (an exchange of a
    // few values with the idle lanes of this warp here cost a sixteen-token layer 11 us of 84): an entry is made up before
    // the wait, and behind it come the copies first, then the entry's description, then the arrival that publishes both.
    int s = 0;
    // a block's first two tiles need no ticket; the counter hands out the tiles behind those (a ticket's value is not touched
    // before its tile's turn)
    const int first_ticket = 2 * int(gridDim.x);
    int next = int(blockIdx.x) - first_ticket, next2 = int(blockIdx.x + gridDim.x) - first_ticket;
    while (true) {
      const int tile = first_ticket + next;
      if (tile >= n_tiles) break;
      next = next2;
      next2 = atomicAdd(counter, 1);
      const bool down = tile >= n_gu;
      const int tl = down ? tile - n_gu : tile;
      const int pos = down ? tl / C::kDnTilesPerItem : tl / gu_tpi;
      const int sub = down ? tl - pos * C::kDnTilesPerItem : tl - pos * gu_tpi;
      const int item = s_work.order[pos];
      const int pb = s_work.pair_begin[item];
      const int ntok = s_work.pair_begin[item + 1] - pb;
      const uint8_t* blob = L.slots + int64_t(s_work.slot[item]) * L.blob_stride;
      const uint8_t* w0 = blob + (down ? L.down_offset + size_t(sub) * C::kDnTile : L.gate_offset + size_t(sub) * C::kGuPart);
      const uint8_t* w1 = blob + L.up_offset + size_t(sub) * C::kGuPart;  // (gate/up)
      const int row0 = sub * (down ? C::kDnRows : C::kGuRows);
      bool ready = !down || !(phases & kPhaseGateUp);  // a down-only launch runs behind a finished gate/up launch
      for (int tok0 = 0; tok0 < ntok; tok0 += kTT, ++i) {
        const int ntp = min(kTT, ntok - tok0), pair0 = pb + tok0;
        float wgt[kTT];
        const uint8_t* act[kTT];
#pragma unroll
        for (int t = 0; t < kTT; ++t) {
          const int p = pair0 + (t < ntp ? t : 0);
          wgt[t] = s_work.pair_weight[p];
          act[t] = down ? ws.hq + size_t(p) * FB_HQ_STRIDE : xq_rows + size_t(s_work.pair_token[p]) * FB_XQ_STRIDE;
        }
        uint8_t* st = stage0 + s * C::kSlot;
        uint64_t* full = &ring.full[s];
        StageMeta* m = const_cast<StageMeta*>(&ring.meta[s]);
        if (!slot_free(s)) return;
        if (!down) {
          mbar_expect_tx_only(full, uint32_t(2 * C::kGuPart + ntp * C::kGuAct));
          bulk_g2s(st, w0, C::kGuPart, full);
          bulk_g2s(st + C::kGuPart, w1, C::kGuPart, full);
#pragma unroll
          for (int t = 0; t < kTT; ++t)
            if (t < ntp) bulk_g2s(st + 2 * C::kGuPart + t * C::kGuAct, act[t], C::kGuAct, full);
        } else if constexpr (DIRECT) {
          mbar_expect_tx_only(full, uint32_t(C::kDnTile));
          bulk_g2s(st, w0, C::kDnTile, full);
        } else {
          mbar_expect_tx_only(full, uint32_t(C::kDnTile + ntp * C::kDnAct));
          bulk_g2s(st, w0, C::kDnTile, full);
          if (!ready) {  // the item's h must have been re-quantized (bounded poll of its flag)
            const int* flag = ws.item_done + kMaxPairs + item;
            uint32_t tries = 0;
            while (true) {
              int v;
              asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
              if (v) break;
              if (++tries > value_polls(ws) || *ring.end_seq == 0) {
                give_up();
                break;
              }
              __nanosleep(50);
            }
            ready = true;
            // the rows were written by another SM's ordinary stores and are read by bulk copies
            asm volatile("fence.proxy.async.global;" ::: "memory");
          }
#pragma unroll
          for (int t = 0; t < kTT; ++t)
            if (t < ntp) bulk_g2s(st + C::kDnTile + t * C::kDnAct, act[t], C::kDnAct, full);
        }
        m->store(i, !down ? 0 : DIRECT && sub == 0 ? 2 : 1, pair0, ntp, row0, item, pb, ntok, wgt);
        if constexpr (DIRECT) mbar_arrive(&ring.staged[s]);
        mbar_arrive(full);
        if (failed) {  // (the entry is complete all the same: its copies are under way)
          ++i;
          return;
        }
        if (++s == S) s = 0;
      }
    }
    if (phases & kPhaseSelect) return;
    // Behind a selection of its own, the last producer of the launch clears the tile counters and the items' flags (all of
    // which have been seen by then), so that the next launch on the same work list (another layer's weights, say) starts
    // like the first; the items' counters wrap to zero. (The fused call's route kernel clears them all.)
    int before;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(before) : "l"(ws.sched + kSchedLeft) : "memory");
    if (before != int(gridDim.x) - 1) return;
#pragma unroll 1
    for (int k = 0; k < kSchedOrderBase; ++k) ws.sched[k] = 0;
    if (phases & kPhaseDown) {
#pragma unroll 1
      for (int k = 0; k < kMaxPairs; ++k) ws.item_done[kMaxPairs + k] = 0;
    }
    return;
  }

  if (DIRECT && warp > C::kWarps) {
    // ---------------- a piece of the h rows of every down entry, quantized into its slot as they arrive
    // These warps arrive on every entry's full barrier, gate/up entries included, so the producer cannot lap them and an
    // entry's phase of `staged` is its own. That barrier is what orders their reads of the description behind the producer's
    // stores, and their writes into the slot behind the consumers' reads of the entry before (those arrive on `empty`, which
    // the producer has waited for). (Probes with short naps: a try with a time limit wakes so late that eight layers of one
    // token take 152.4 us instead of 146.4.)
    const int piece = warp - (C::kWarps + 1), at = 256 * piece + 8 * lane;
    // Behind an expired wait they go on to the last entry that has been staged, with whatever h holds: the block's last wait
    // for its copies (ring_drain) needs their arrivals.
    bool expired = false;
    for (int seq = 0;; ++seq) {
      const int s = seq % S;
      uint32_t tries = 0;
      bool end = false;
      while (!__all_sync(0xffffffffu, mbar_test_wait(&ring.staged[s], (seq / S) & 1))) {
        end = uint32_t(__shfl_sync(0xffffffffu, *ring.staged_seq, 0)) <= uint32_t(seq);  // (-1: not known yet)
        if (end) break;
        if (++tries > kStopPolls) {
          if (expired) return;  // (the producer does not answer)
          expired = true;
          tries = 0;
          if (lane == 0) ring_abort(ring, ws.status);
        }
        __nanosleep(40);
      }
      if (end) break;
      const int kind = ring.meta[s].tile, pair0 = ring.meta[s].pair0, ntp = ring.meta[s].ntp;
      if (kind == 0) {  // gate/up: nothing to add
        if (lane == 0) mbar_arrive(&ring.full[s]);
        continue;
      }
      uint8_t* out = stage0 + s * C::kSlot + C::kDnTile;
      for (int t = 0; t < ntp; ++t, out += C::kDnAct) {
        const float* h = ws.h + size_t(pair0 + t) * INTER;
        float v[8];
        tries = 0;
        while (!__all_sync(0xffffffffu, direct_load8(h, at, INTER, v))) {
          if (__shfl_sync(0xffffffffu, *ring.end_seq, 0) == 0) break;
          if (++tries > value_polls(ws)) {
            expired = true;
            if (lane == 0) ring_abort(ring, ws.status);
            break;
          }
          __nanosleep(20);
        }
        quantize_h_piece<INTER>(v, piece, down_act, out);
      }
      fence_proxy_async();  // (a later entry's bulk copies will write here)
      __syncwarp();
      if (lane == 0) mbar_arrive(&ring.full[s]);
      if (kind == 2)  // an item's first tile: its rows in the workspace too, where the other form of this kernel leaves them
        for (int p = pair0; p < pair0 + ntp; ++p) {
          float v[8];
          direct_load8(ws.h + size_t(p) * INTER, at, INTER, v);
          quantize_h_piece<INTER>(v, piece, down_act, ws.hq + size_t(p) * FB_HQ_STRIDE);
        }
    }
    if (expired && lane == 0) ring_drain(ring);
    return;
  }

  // ---------------- consumers
  const uint32_t sign_base = kSigns ? smem_u32(signtab) : 0u;
  const Iq4nlLevels lv = iq4nl_levels();
  const int gu_row_off = (lane >> 4) * C::kGuPart + (lane & 15) * C::kGuRowBytes;
  // Even blocks of the formats with 2-byte alignment start on a word boundary (their words behind the scale are 2 bytes
  // off), odd blocks the other way round: two code paths. A warp keeps to one parity, and since warp w issues on
  // scheduler w % 4, each scheduler's instruction cache sees one path only.
  const int parity = warp & 1;
  while (true) {
    int s, k;
    if (!draw_task_n<S, C::kTasks / 2>(ring, &s_misc[1 + parity], ws.status, lane, s, k)) break;
    const int task = 2 * k + parity;
    const int ntp = ring.meta[s].ntp;
    const bool down = ring.meta[s].tile != 0;
    uint8_t* st = stage0 + s * C::kSlot;
    float term[kTT] = {0.0f, 0.0f};
    if constexpr (DN == FB_FMT_IQ3_S) {
      // one copy of the decode for both projections: the two parities' loops fill the instruction cache as it is
      const uint8_t* blk = down ? st + (32 * k + lane) * C::kDnRowBytes + parity * C::kDnTaskBytes
                                : st + gu_row_off + task * C::kTaskBytes;
      const uint8_t* act0 = st + (down ? C::kDnTile : 2 * C::kGuPart);
      const int act_bytes = down ? C::kDnAct : C::kGuAct, act_k = down ? INTER : H, ablk = down ? parity : task;
      if (parity == 0) gate_up_block_terms<GU, true>(blk, grid, sign_base, lv, act0, act_bytes, ablk, ntp, term, act_k);
      else gate_up_block_terms<GU, false>(blk, grid, sign_base, lv, act0, act_bytes, ablk, ntp, term, act_k);
    } else if constexpr (GU == FB_FMT_IQ4_NL && DN == FB_FMT_IQ4_NL && INTER == 512) {
      // one copy here too: instructions are what the warps wait for most (the two copies before: eight layers of
      // eight tokens 357.3 us, 354.8 so)
      if (!down || k < C::kDnRows / 32)
        iq4nl_task_terms(down ? st + (32 * k + lane) * C::kDnRowBytes + parity * C::kDnTaskBytes : st + gu_row_off + task * C::kTaskBytes,
                               lv, st + (down ? C::kDnTile : 2 * C::kGuPart), down ? C::kDnAct : C::kGuAct, down ? INTER : H,
                               8 * (down ? parity : task), ntp, term);
    } else if (!down) {
      const uint8_t* blk = st + gu_row_off + task * C::kTaskBytes;
      const uint8_t* act0 = st + 2 * C::kGuPart;
      if constexpr (GU == FB_FMT_IQ4_NL) {
        iq4nl_task_terms(blk, lv, act0, C::kGuAct, H, 8 * task, ntp, term);
      } else if (parity == 0) {
        gate_up_block_terms<GU, true>(blk, grid, sign_base, lv, act0, C::kGuAct, task, ntp, term);
      } else {
        gate_up_block_terms<GU, false>(blk, grid, sign_base, lv, act0, C::kGuAct, task, ntp, term);
      }
    } else if (k < C::kDnRows / 32) {
      const uint8_t* half = st + (32 * k + lane) * C::kDnRowBytes + parity * C::kDnTaskBytes;
      const uint8_t* act0 = st + C::kDnTile;
      if constexpr (DN == FB_FMT_Q2_0) {
        if constexpr (INTER == 512) q2_0_task_terms<4, 0>(half, act0, C::kDnAct, INTER, 8 * parity, ntp, term);
        else if (parity == 0) q2_0_task_terms<5, 0>(half, act0, C::kDnAct, INTER, 0, ntp, term);
        else q2_0_task_terms<5, 2>(half - 2, act0, C::kDnAct, INTER, 10, ntp, term);
      } else if constexpr (INTER == 512) {
        iq4nl_task_terms(half, lv, act0, C::kDnAct, INTER, 8 * parity, ntp, term);
      } else {
        iq4nl_half_row_terms(half, lv, act0, C::kDnAct, INTER, 10 * parity, ntp, term);
      }
    }
    float* part = partials + (s * C::kTasks + task) * (kTT * 32);
    part[lane] = term[0];
    part[32 + lane] = term[1];
    // The warp that finishes the entry's last task adds the block terms of every row in a fixed
    // order, finishes the rows and hands the slot back to the producer.
    __threadfence_block();
    __syncwarp();
    int done = 0;
    if (lane == 0) done = atomicAdd(&s_misc[3 + s], 1);
    done = __shfl_sync(0xffffffffu, done, 0);
    if (done != C::kTasks - 1) continue;
    __threadfence_block();
    const int pair0 = ring.meta[s].pair0, r0 = ring.meta[s].row0;
    const float* pt = partials + s * C::kTasks * (kTT * 32);
    if (!down) {
      const int item = ring.meta[s].item, ipb = ring.meta[s].item_pair0, itok = ring.meta[s].item_tok;
      for (int t = 0; t < ntp; ++t) {
        float v = 0.0f;
#pragma unroll
        for (int b = 0; b < C::kTasks; ++b) v += pt[(b * kTT + t) * 32 + lane];
        const float u = __shfl_down_sync(0xffffffffu, v, 16);
        float* out = ws.h + size_t(pair0 + t) * INTER + r0 + lane;
        if (lane < 16) {
          if constexpr (DIRECT) direct_store(out, silu_mul(v, u));
          else *out = silu_mul(v, u);
        }
      }
      __syncwarp();
      if (lane == 0) {
        s_misc[3 + s] = 0;
        mbar_arrive(&ring.empty[s]);
      }
      if constexpr (!DIRECT)
        item_contribution_done<INTER>(ws, item, ipb, itok, gu_tpi * ((itok + kTT - 1) / kTT), down_act,
                                      phases & kPhaseDown ? 1 : 0, lane);
    } else {
      const float w0 = ring.meta[s].wgt[0], w1 = ring.meta[s].wgt[1];
#pragma unroll
      for (int g = 0; g < C::kDnRows / 32; ++g) {
        const float v0 = pt[((2 * g) * kTT + 0) * 32 + lane] + pt[((2 * g + 1) * kTT + 0) * 32 + lane];
        float* out = ws.partial + size_t(pair0) * H + r0 + 32 * g + lane;
        if constexpr (DIRECT) direct_store(out, w0 * v0);
        else *out = w0 * v0;
        if (ntp == 2) {
          const float v1 = pt[((2 * g) * kTT + 1) * 32 + lane] + pt[((2 * g + 1) * kTT + 1) * 32 + lane];
          if constexpr (DIRECT) direct_store(out + H, w1 * v1);
          else out[H] = w1 * v1;
        }
      }
      __syncwarp();
      if (lane == 0) {
        s_misc[3 + s] = 0;
        mbar_arrive(&ring.empty[s]);
      }
      if (sel.y_out) {
        if constexpr (!DIRECT) combine_tile<C::kDnRows>(ws, sel, s_work, pair0, ntp, r0, lane);
        else if (!combine_tile_direct<C::kDnRows>(ws, sel, s_work, pair0, ntp, r0, lane, ring)) break;
      }
    }
  }
}
