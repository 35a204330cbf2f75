// Decode-width (T <= 16) routed-expert kernels on native GGUF expert bytes.
//
//   route    router projection, once-per-token activation quantization
//   select   top-10 and the sorted work list (stand-alone from given logits, or inside the expert kernel)
//   gate_up  h[pair][j] = silu(gate_j . x) * (up_j . x)
//   down     partial[pair][n] = w_pair * (down_n . q8(h[pair]))
//   combine  y[t] = sum of token t's partials in slot order (+ shared, + residual write)
//
// Kernels of this path start while their predecessor runs out (programmatic dependent launch) and wait for it before they
// touch global memory. None of them reads through const __restrict__ pointers or __ldg: such loads count as invariant
// and may be moved ahead of the wait.
//
// gate_up and down are one persistent kernel, one CTA per SM (moe_decode_experts.cuh): a producer thread streams
// tiles of the expert blob into a shared-memory ring of three or four slots with 1-D bulk async copies (TMA, no multicast)
// signalled through mbarriers; consumer warps decode the blocks from shared memory and accumulate exact int8 dot
// products (dp4a). Numerics are those of the
// reference's CPU expert tier (src/cpu/iq_cpu.h:12-40 of the reference project): Q8_K activations
// for IQ3_S weights, Q8_0 for IQ4_NL, integer sums per block, one fp32 scale step per block.
#include "iq_decode.cuh"
#include "host_range.h"

#include <cstring>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>

namespace fb {
namespace {

constexpr int H = FB_HIDDEN;
constexpr int kTopK = FB_TOPK;
constexpr int kExperts = FB_EXPERTS;
constexpr int kMaxTok = FB_DECODE_MAX_TOKENS;
constexpr int kMaxPairs = FB_DECODE_MAX_PAIRS;
constexpr int kTT = 2;  // tokens of one work item handled per pass over a staged tile
// ws.sched: [0] gate/up tile counter, [1] down tile counter, [2] producers that have staged their last tile,
// [8..168) item order
constexpr int kSchedLeft = 2, kSchedOrderBase = 8;
constexpr int kEpMaxRanks = FB_EP_MAX_RANKS;
constexpr uint32_t kPeerSpinLimit = 1u << 20;  // default polls of a peer-written flag before giving up (about a second)

// Flag-in-data exchange lines (the low-latency protocol of collective libraries): 16 bytes =
// {value 0, step, value 1, step}, written by ONE 16-byte store, so a reader that sees the step
// number of the current step in both flag words holds both values - no fence, no separate flag.
__device__ __forceinline__ void ll_store(uint4* line, float v0, float v1, uint32_t step) {
  asm volatile("st.relaxed.sys.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(line), "r"(__float_as_uint(v0)), "r"(step),
               "r"(__float_as_uint(v1)), "r"(step)
               : "memory");
}
// Polls the line (at most `limit` times) until both halves carry `step`.
__device__ __forceinline__ float2 ll_read(const uint4* line, uint32_t step, uint32_t* status, uint32_t limit) {
  uint4 v;
  for (uint32_t i = 0; i < limit; ++i) {
    asm volatile("ld.relaxed.sys.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(line)
                 : "memory");
    if (v.y == step && v.w == step) return make_float2(__uint_as_float(v.x), __uint_as_float(v.z));
    // once any reader of this launch has given up, the others stop waiting too (checked rarely)
    if ((i & 1023u) == 1023u && *reinterpret_cast<volatile uint32_t*>(status) >= uint32_t(FB_STATUS_PIPELINE_TIMEOUT))
      return make_float2(0.0f, 0.0f);
    __nanosleep(100);
  }
  atomicMax(status, uint32_t(FB_STATUS_PIPELINE_TIMEOUT));
  return make_float2(0.0f, 0.0f);
}
// ws.sched behind the order: [token][down tile] finished partial tiles (the expert kernel's own combine)
constexpr int kSchedParts = 192, kMaxDnTiles = H / 128;
constexpr int kSchedInts = kSchedParts + kMaxTok * kMaxDnTiles;

__host__ __device__ constexpr int act_of(int fmt) {
  return fmt == FB_FMT_IQ4_NL || fmt == FB_FMT_Q2_0 ? FB_ACT_Q8_0 : FB_ACT_Q8_K;
}
// ws.xq holds [2][16][FB_XQ_STRIDE]: the Q8_K rows of the step's tokens, then their Q8_0 rows. A workspace
// made for a layout gets the one its gate/up format needs; one made without a layout gets both from
// the stand-alone selection (which does not see the layout).
__host__ __device__ constexpr size_t xq_offset(int act) { return act == FB_ACT_Q8_0 ? size_t(kMaxTok) * FB_XQ_STRIDE : 0; }

__device__ __forceinline__ float silu_mul(float g, float u) { return __fdividef(g, 1.0f + expf(-g)) * u; }

// Planar Q8_K rows: codes [k] | block scales float [k/256] (64 bytes reserved) | code sums of every 32
// codes, int16 [k/32] (Q8_K's bsums added in pairs; the IQ3_S kernels use them, see moe_decode_experts.cuh).
__host__ __device__ constexpr int q8k_asum_off(int k) { return k + 64; }

// Stores block b of a planar Q8_K row from the calling warp's quantizer output (lane l holds codes
// 8l..8l+7 of the block in q, pair_sum the sum of its 16-code group).
__device__ __forceinline__ void store_q8k_block_planar(uint8_t* out, int k, int b, const int (&q)[8], int pair_sum,
                                                       float d) {
  const int lane = threadIdx.x & 31;
  uint2 pk;
  pk.x = uint32_t(uint8_t(q[0])) | (uint32_t(uint8_t(q[1])) << 8) | (uint32_t(uint8_t(q[2])) << 16) |
         (uint32_t(uint8_t(q[3])) << 24);
  pk.y = uint32_t(uint8_t(q[4])) | (uint32_t(uint8_t(q[5])) << 8) | (uint32_t(uint8_t(q[6])) << 16) |
         (uint32_t(uint8_t(q[7])) << 24);
  *reinterpret_cast<uint2*>(out + 256 * b + 8 * lane) = pk;
  const int sum32 = pair_sum + __shfl_xor_sync(0xffffffffu, pair_sum, 2);  // lanes 4j..4j+3 hold sub-block j
  if ((lane & 3) == 0) reinterpret_cast<int16_t*>(out + q8k_asum_off(k))[8 * b + (lane >> 2)] = int16_t(sum32);
  if (lane == 0) reinterpret_cast<float*>(out + k)[b] = d;
}

// ------------------------------------------------------------------------------ activation rows
// One row of k values -> planar codes + scales, by the calling block (any number of warps).
// Q8_K: codes [k], scales float[k/256]. Q8_0: codes [k] (interleaved per block), scales float[k/32].
template <class LoadF>
__device__ __forceinline__ void quantize_row_planar(int act, int k, LoadF load, uint8_t* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (act == FB_ACT_Q8_K) {
    for (int b = warp; b < k / 256; b += warps) {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = load(256 * b + 8 * lane + i);
      int q[8], ps;
      const float d = q8k_block_warp(v, q, ps);
      store_q8k_block_planar(out, k, b, q, ps, d);
    }
  } else {
    float* scales = reinterpret_cast<float*>(out + k);
    for (int b = warp; b < k / 32; b += warps) {
      unsigned short dh;
      const int q = q8_0_block_warp(load(32 * b + lane), dh);
      out[32 * b + q8_0_interleave_index(lane)] = uint8_t(int8_t(q));
      if (lane == 0) scales[b] = __half2float(__ushort_as_half(dh));
    }
  }
}

// ------------------------------------------------------------------------------ router
// logits[t][r] = sum_k W[r][k] * x[t][k]; one warp per row (four rows per block), the row's
// weights held in registers, tokens taken four at a time so that their loads overlap; the 32 lane
// sums are added by a butterfly. Fixed order: repeated calls are bitwise identical.
template <bool XBF16>
__global__ void __launch_bounds__(128) router_kernel(const __nv_bfloat16* w, int rows, const void* xv, int tokens,
                                                     float* logits, int stride) {
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_wait_prior();
  if (row >= rows) return;
  float wr[80];
  {
    const uint4* wp = reinterpret_cast<const uint4*>(w + size_t(row) * H);
#pragma unroll
    for (int c = 0; c < 10; ++c) {
      const uint4 v = wp[c * 32 + lane];
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        wr[8 * c + 2 * i] = __uint_as_float(u[i] << 16);
        wr[8 * c + 2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u);
      }
    }
  }
  for (int t0 = 0; t0 < tokens; t0 += 4) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < 10; ++c) {
#pragma unroll
      for (int tt = 0; tt < 4; ++tt) {
        const int t = min(t0 + tt, tokens - 1);  // clamped rows are computed and dropped
        float xs[8];
        if constexpr (XBF16) {
          const uint4 v =
              reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(xv) + size_t(t) * H)[c * 32 + lane];
          const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            xs[2 * i] = __uint_as_float(u[i] << 16);
            xs[2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u);
          }
        } else {
          const float4* xp =
              reinterpret_cast<const float4*>(static_cast<const float*>(xv) + size_t(t) * H) + (c * 32 + lane) * 2;
          const float4 a = xp[0], b = xp[1];
          xs[0] = a.x; xs[1] = a.y; xs[2] = a.z; xs[3] = a.w;
          xs[4] = b.x; xs[5] = b.y; xs[6] = b.z; xs[7] = b.w;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[tt] = fmaf(wr[8 * c + i], xs[i], acc[tt]);
      }
    }
#pragma unroll
    for (int tt = 0; tt < 4; ++tt) {
      float v = acc[tt];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0 && t0 + tt < tokens) logits[size_t(t0 + tt) * stride + row] = v;
    }
  }
}

// The same logits, bit for bit, at prefill width (tokens > kMaxTok). Bound: the fp32 pipe (tokens x rows x 2560
// multiply-adds). router_kernel above re-reads x for every row and keeps four tokens in flight: 0.96 us per token,
// 963 us at 1003 tokens; this kernel takes 87 us there (3.7 waves of blocks).
// A block owns 32 rows (ROWS) x 32 tokens; its sixteen warps split K the way router_kernel's lanes do: the partial sum of
// lane l (elements 256 c + 8 l + i, added over c, then i) belongs to warp l mod 16, which adds those of lanes l and
// l + 16; the sixteen results meet in shared memory in the butterfly's order. A thread accumulates 8 rows x 4 tokens. bf16
// activations: multiply-adds of two bf16 numbers into fp32, which take the halves of the packed words as they lie (one
// rounding, as fmaf). What bounds it is their three register operands: an instruction takes some 1.5 cycles of a scheduler.
// Packed fp32 multiply-adds of widened values (fma.rn.f32x2, half the instructions, and as many again to widen) took 103 us,
// values widened on their way into shared memory 103, half-warps on a lane class each with 8 x 8 values per thread 100.
// fp32 activations: packed pairs of rows. 256-wide K chunks lie row-major in three cp.async buffers, rows 16 bytes apart
// modulo the banks: one 16-byte load brings a row's eight elements of a lane class. (A K-major copy in fp32, widened while
// staging, took 142 us: its global loads touched 32 rows per instruction.)
// ROWS (32, 16 or 8): few tokens do not fill the GPU with tiles of 32 rows, and a block's time follows its rows; see
// fb_router_logits.
constexpr int kRtTok = 32, kRtChunk = 256, kRtBufs = 3;
template <bool XBF16>
constexpr int router_tile_pitch() { return kRtChunk * (XBF16 ? 2 : 4) + 16; }  // bytes between token rows
constexpr int kRtWPitch = kRtChunk * 2 + 16;                                  // and between weight rows
template <bool XBF16, int ROWS>
constexpr int router_tile_buf() { return ROWS * kRtWPitch + kRtTok * router_tile_pitch<XBF16>(); }
template <bool XBF16, int ROWS>
constexpr int router_tile_smem() {
  const int ring = kRtBufs * router_tile_buf<XBF16, ROWS>(), part = 16 * ROWS * kRtTok * 4;
  return ring > part ? ring : part;  // the warps' partial tiles reuse the buffers
}

__device__ __forceinline__ void fma_f32x2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// acc += lo(w) lo(x), then hi(w) hi(x), of bf16 pairs
__device__ __forceinline__ void fma_bf16_pair(float& acc, uint32_t w, uint32_t x) {
  asm("{\n\t.reg .b16 wl, wh, xl, xh;\n\tmov.b32 {wl, wh}, %1;\n\tmov.b32 {xl, xh}, %2;\n\t"
      "fma.rn.f32.bf16 %0, wl, xl, %0;\n\tfma.rn.f32.bf16 %0, wh, xh, %0;\n\t}"
      : "+f"(acc)
      : "r"(w), "r"(x));
}
__device__ __forceinline__ uint64_t pack_f32x2(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
// 16 bytes, or 16 zeros (nothing is read then).
__device__ __forceinline__ void cp_async_16(void* dst_smem, const void* src, bool read) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst_smem)), "l"(src), "r"(read ? 16 : 0) : "memory");
}

template <bool XBF16, int ROWS>
__global__ void __launch_bounds__(512, 1) router_tile_kernel(const __nv_bfloat16* w, int rows, const void* xv,
                                                             int tokens, float* logits, int stride) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int kXPitch = router_tile_pitch<XBF16>(), kBuf = router_tile_buf<XBF16, ROWS>(), kChunks = H / kRtChunk;
  pdl_launch_dependents();
  pdl_wait_prior();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row_base = blockIdx.x * ROWS, tok_base = blockIdx.y * kRtTok;
  // a warp copies two weight rows and two token rows of a chunk; rows and tokens beyond the end are zeros (they are computed
  // and not stored). Repeats of the last one in their place were read by all warps at once, and the copies waited for that
  // one line (513 rows, bf16, us: 17 tokens 13.2 -> 8.9, 33 21.5 -> 10.0, 100 17.3 -> 13.7, 1003 89.9 -> 87.2).
  auto fetch = [&](int c) {
    uint8_t* buf = smem + (c % kRtBufs) * kBuf;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int r = warp + 16 * p;
      if (r < ROWS) {
        const bool in = row_base + r < rows;
        cp_async_16(buf + r * kRtWPitch + 16 * lane, w + size_t(in ? row_base + r : 0) * H + kRtChunk * c + 8 * lane, in);
      }
      uint8_t* xd = buf + ROWS * kRtWPitch + r * kXPitch + 16 * lane;
      const bool in = tok_base + r < tokens;
      const size_t at = size_t(in ? tok_base + r : 0) * H + kRtChunk * c;
      if constexpr (XBF16) {
        cp_async_16(xd, static_cast<const __nv_bfloat16*>(xv) + at + 8 * lane, in);
      } else {
        cp_async_16(xd, static_cast<const float*>(xv) + at + 4 * lane, in);
        cp_async_16(xd + 512, static_cast<const float*>(xv) + at + 128 + 4 * lane, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // thread = rows rg + 4 j (j = 0..ROWS / 4 - 1; fp32: pairs of neighbouring j) x tokens tg + 8 t (t = 0..3)
  const int rg = lane >> 3, tg = lane & 7;
  constexpr int kAcc = XBF16 ? ROWS / 4 : ROWS / 8;
  std::conditional_t<XBF16, float, uint64_t> acc[2][kAcc][4];  // [lane class warp, warp + 16][row or row pair][token]
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < kAcc; ++r)
#pragma unroll
      for (int t = 0; t < 4; ++t) acc[c][r][t] = 0;
  fetch(0);
  fetch(1);
  for (int c = 0; c < kChunks; ++c) {
    if (c + 1 < kChunks) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // chunk c is in place, and nobody reads the buffer that the next fetch fills
    if (c + 2 < kChunks) fetch(c + 2);
    const uint8_t* buf = smem + (c % kRtBufs) * kBuf;
    if constexpr (XBF16) {
#pragma unroll
      for (int cls = 0; cls < 2; ++cls) {
        const int piece = warp + 16 * cls;  // elements 8 piece .. + 7 of the chunk
        uint4 x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t)
          x[t] = *reinterpret_cast<const uint4*>(buf + ROWS * kRtWPitch + (tg + 8 * t) * kXPitch + 16 * piece);
#pragma unroll
        for (int r = 0; r < ROWS / 4; ++r) {
          const uint4 wv = *reinterpret_cast<const uint4*>(buf + (rg + 4 * r) * kRtWPitch + 16 * piece);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            fma_bf16_pair(acc[cls][r][t], wv.x, x[t].x);
            fma_bf16_pair(acc[cls][r][t], wv.y, x[t].y);
            fma_bf16_pair(acc[cls][r][t], wv.z, x[t].z);
            fma_bf16_pair(acc[cls][r][t], wv.w, x[t].w);
          }
        }
      }
    } else {
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        const int cls = ch >> 1, e = 4 * (ch & 1);
        const int piece = warp + 16 * cls;  // elements 8 piece + e .. + 3 of the chunk
        uint64_t xx[4][4];                  // token values, both halves alike: made once, used by four row pairs
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint8_t* xp = buf + ROWS * kRtWPitch + (tg + 8 * t) * kXPitch + (8 * piece + e) * 4;
          const uint4 v = *reinterpret_cast<const uint4*>(xp);
          xx[t][0] = pack_f32x2(v.x, v.x);
          xx[t][1] = pack_f32x2(v.y, v.y);
          xx[t][2] = pack_f32x2(v.z, v.z);
          xx[t][3] = pack_f32x2(v.w, v.w);
        }
#pragma unroll
        for (int r = 0; r < ROWS / 8; ++r) {
          const uint2 a = *reinterpret_cast<const uint2*>(buf + (rg + 8 * r) * kRtWPitch + 16 * piece + 2 * e);
          const uint2 b = *reinterpret_cast<const uint2*>(buf + (rg + 8 * r + 4) * kRtWPitch + 16 * piece + 2 * e);
          const uint64_t wp[4] = {pack_f32x2(a.x << 16, b.x << 16), pack_f32x2(a.x & 0xFFFF0000u, b.x & 0xFFFF0000u),
                                  pack_f32x2(a.y << 16, b.y << 16), pack_f32x2(a.y & 0xFFFF0000u, b.y & 0xFFFF0000u)};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int t = 0; t < 4; ++t) fma_f32x2(acc[cls][r][t], wp[i], xx[t][i]);
        }
      }
    }
  }
  __syncthreads();
  float* part = reinterpret_cast<float*>(smem);  // [warp][token][row]
#pragma unroll
  for (int r = 0; r < kAcc; ++r)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float* q = part + (warp * kRtTok + tg + 8 * t) * ROWS + rg;
      if constexpr (XBF16) {
        q[4 * r] = acc[0][r][t] + acc[1][r][t];
      } else {
        const float2 a = *reinterpret_cast<const float2*>(&acc[0][r][t]), b = *reinterpret_cast<const float2*>(&acc[1][r][t]);
        q[8 * r] = a.x + b.x;
        q[8 * r + 4] = a.y + b.y;
      }
    }
  __syncthreads();
  for (int o = tid; o < ROWS * kRtTok; o += 512) {
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = part[i * ROWS * kRtTok + o];
#pragma unroll
    for (int n = 8; n >= 1; n >>= 1)
#pragma unroll
      for (int i = 0; i < n; ++i) v[i] += v[i + n];
    const int t = tok_base + o / ROWS, r = row_base + (o & (ROWS - 1));
    if (t < tokens && r < rows) logits[size_t(t) * stride + r] = v[0];
  }
}

// The part of the work list a producer needs, in shared memory: the producer is a single thread, and a
// chain of dependent global loads per tile (visiting order -> item -> its pairs -> their tokens and
// weights, about two microseconds) would pace the whole kernel. Either copied from the device work list
// (work_cache_fill) or built in place by the CTA's own selection (select_block).
struct WorkCache {
  int order[kMaxPairs];
  int pair_begin[kMaxPairs + 1];
  int slot[kMaxPairs];
  int pair_token[kMaxPairs];
  float pair_weight[kMaxPairs];
  int token_row[kMaxTok][kTopK];  // a token's pairs in slot order (only by the CTA's own selection)
  int last_pair[kMaxTok];         // the one of them whose item is visited last (the same)
  int n_items;
};
// Called by the 32 lanes of the producer warp (the only reader) after the wait on the preceding kernel;
// the caller follows with __syncwarp().
__device__ __forceinline__ void work_cache_fill(const fb_moe_decode_workspace& ws, WorkCache& c, int n_items) {
  const fb_moe_decode_work* work = ws.work;
  for (int i = threadIdx.x & 31; i < kMaxPairs; i += 32) {
    const bool live = i < n_items;
    c.order[i] = live ? ws.sched[kSchedOrderBase + i] : 0;
    c.slot[i] = live ? work->item_slot[i] : 0;
    c.pair_begin[i] = i <= n_items ? work->item_pair_begin[i] : 0;
    c.pair_token[i] = work->pair_token[i];
    c.pair_weight[i] = work->pair_weight[i];
  }
  if ((threadIdx.x & 31) == 0) {
    c.pair_begin[kMaxPairs] = n_items == kMaxPairs ? work->item_pair_begin[kMaxPairs] : 0;
    c.n_items = n_items;
  }
}

// ------------------------------------------------------------------------------ select
struct SelectScratch {
  union {
    uint2 cand[kMaxTok][32];  // a token's candidates: logit, id
    struct {  // behind those
      int begin[kExperts];         // physical slot -> first pair of its item
      int slot[kMaxTok][kTopK];    // physical slots of the winners, -1: not held here
      int16_t rank[kExperts];      // physical slot -> its item's place in the visiting order
    };
  };
  float val[kMaxTok][kTopK];             // the winners' logits
  uint32_t tok[kExperts];                // physical slot -> mask of the tokens that chose it
  int hist[kExperts / 32][kMaxTok + 1];  // [warp of slots][token count - 1] -> items (padded: no bank conflicts)
  int scan[kExperts / 32];               // [warp of slots] -> its pairs | its items << 16
};
// LAST: wc.last_pair is wanted. load(t, e): logit e of token t. `scratch`: shared memory (16-byte aligned) that is free until
// the call returns.
// Called by every thread of a block of 512 or more threads. The work list goes to `wc` in shared memory
// (complete when the call returns) and, with `publish`, to the device work list as well; `reset` clears
// the tile and item counters of the streaming kernels (only where no such kernel can be running). The
// list is a function of the logits alone: every block that runs this on the same logits builds the same
// list. Every CTA of a decode step waits for this, so it is kept a short chain of six barriers: token
// masks per physical slot (shared-memory atomics), one scan over the 512 slots (thread = slot), the items ranked by a
// counting sort on their token counts (warp matches), and the pairs placed from the scan. Few
// warps do this work and a warp on its own retires an instruction every few cycles: what counts here is the
// number of instructions on the longest chain, not the arithmetic. So the routing weights are computed by warps that
// the list does not need, and the device work list is written behind the last barrier. (Up to three tokens: one warp,
// shuffles.)
//   items  = distinct selected experts held on this rank, in physical-slot order
//   pairs  = (item, token), tokens ascending inside an item
//   order  = items by token count, most first, ties by item index (the streaming kernels' visiting order)
template <bool LAST, class LoadF>
__device__ __forceinline__ void select_block(LoadF load, const int32_t* slot_of, int T,
                                             const fb_moe_decode_workspace& ws, uint32_t* counts, bool remote_ok,
                                             bool publish, bool reset, WorkCache& wc, SelectScratch& scratch) {
  static_assert(kExperts == 512 && kMaxTok == 16, "sixteen warps of slots, lanes 0..15 hold the token-count classes");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  // (these three outlive the scratch memory)
  __shared__ int s_pair[kMaxTok][kTopK];
  __shared__ int s_id[kMaxTok][kTopK];
  __shared__ float s_w[kMaxTok][kTopK];
  auto& s_val = scratch.val;
  auto& s_tok = scratch.tok;
  auto& s_begin = scratch.begin;
  auto& s_hist = scratch.hist;
  auto& s_scan = scratch.scan;
  if (tid < kExperts) s_tok[tid] = 0;
  if (tid < kExperts / 32 * (kMaxTok + 1)) (&s_hist[0][0])[tid] = 0;
  if (reset) {
    if (tid < 2 * kMaxPairs) ws.item_done[tid] = 0;
    if (tid < kSchedOrderBase) ws.sched[tid] = 0;
  }
  // (One warp per token. All sixteen warps on each token's slices - maxima, threshold, candidates and ranking behind a
  // barrier each - was slower at every batch: 3.3 against 2.5 us at one token, 6 against 3 at sixteen.)
  if (warp < T) warp_top10_pruned<false>([&](int e) { return load(warp, e); }, scratch.cand[warp], s_id[warp], s_val[warp]);
  __syncthreads();
  const int np = T * kTopK;
  const bool small = np <= 32;
  {
    const int first = small ? 1 : warps > kMaxTok ? kMaxTok : 0;
    if (warp >= first)
      for (int t = warp - first; t < T; t += warps - first) top10_weights(s_val[t], s_w[t]);
  }
  const bool valid = tid < np;
  const int pt = tid / kTopK, pk = tid - pt * kTopK;
  if (small) {
    // Up to three tokens: the pairs fit one warp, which builds the whole list through shuffles (lane = pair).
    // Same list as the general path below.
    if (warp == 0) {
      const int e = valid ? s_id[pt][pk] : 0;
      int slot = !valid ? -1 : slot_of ? slot_of[e] : e;
      if (slot >= kExperts) slot = -1;
      const int key = slot >= 0 ? slot * kMaxTok + pt : 0x7fffffff;  // pairs not held here sort last
      // (a lone warp runs at a few cycles per instruction: the loops below take np turns, not 32, and a single
      // token, whose ten pairs are ten different experts, needs only the first)
      int idx = 0, trank = 0, cnt = 0;
#pragma unroll 5
      for (int j = 0; j < np; ++j) {
        const int kj = __shfl_sync(0xffffffffu, key, j);
        const bool same = kj != 0x7fffffff && (kj / kMaxTok) == slot;
        idx += kj < key ? 1 : 0;
        cnt += same ? 1 : 0;
        trank += same && kj < key ? 1 : 0;
      }
      const bool hot = slot >= 0, first = hot && trank == 0;
      const uint32_t hot_m = __ballot_sync(0xffffffffu, hot), first_m = __ballot_sync(0xffffffffu, first);
      const int n_pairs = __popc(hot_m), n_items = __popc(first_m);
      int item = idx, rank = idx;  // one token: every held pair is an item of one token, in key order
      if (T > 1) {
        item = 0;  // distinct slots below this pair's slot = first pairs with a smaller key
#pragma unroll 2
        for (int j = 0; j < np; ++j) {
          const int kj = __shfl_sync(0xffffffffu, key, j);
          item += ((first_m >> j) & 1u) && (kj / kMaxTok) < slot ? 1 : 0;
        }
        rank = 0;  // visiting order among the items: more tokens first, then lower item index
#pragma unroll 2
        for (int j = 0; j < np; ++j) {
          const int cj = __shfl_sync(0xffffffffu, cnt, j), ij = __shfl_sync(0xffffffffu, item, j);
          rank += ((first_m >> j) & 1u) && (cj > cnt || (cj == cnt && ij < item)) ? 1 : 0;
        }
      }
      if constexpr (LAST) {  // (the lanes of an item agree on its rank)
        const int mine = hot ? rank : -1;
        int most = -1;
#pragma unroll
        for (int k = 0; k < kTopK; ++k) most = max(most, __shfl_sync(0xffffffffu, mine, min(31, kTopK * (valid ? pt : 0) + k)));
        if (valid && hot && mine == most) wc.last_pair[pt] = idx;
      }
      if (hot) wc.pair_token[idx] = pt;
      if (first) {
        wc.slot[item] = slot;
        wc.pair_begin[item] = idx;
        wc.order[rank] = item;
      }
      if (lane == 0) {
        wc.pair_begin[n_items] = n_pairs;
        wc.n_items = n_items;
      }
      if (valid) {
        s_pair[pt][pk] = hot ? idx : -1;
        if (counts) atomicAdd(&counts[e], 1u);
      }
    }
    __syncthreads();
    if (valid) {
      const int idx = s_pair[pt][pk];
      if (idx >= 0) wc.pair_weight[idx] = s_w[pt][pk];
    }
    if (warp == 1 && lane < np) {  // a token's pairs in slot order = pair order
      const int t = lane / kTopK, idx = s_pair[t][lane - t * kTopK];
      int rank = 0;
#pragma unroll
      for (int k = 0; k < kTopK; ++k) rank += uint32_t(s_pair[t][k]) < uint32_t(idx) ? 1 : 0;  // (-1 is the largest)
      if (idx >= 0) wc.token_row[t][rank] = idx;
    }
  } else {
    int my_slot = -1;
    if (valid) {
      const int e = s_id[pt][pk];
      my_slot = slot_of ? slot_of[e] : e;
      if (my_slot >= kExperts) my_slot = -1;
      scratch.slot[pt][pk] = my_slot;
      if (my_slot >= 0) atomicOr(&s_tok[my_slot], 1u << pt);
      if (counts) atomicAdd(&counts[e], 1u);
    }
    __syncthreads();
    // Thread = slot, sixteen warps. Inside the warps: inclusive scan of (pairs, items) in one word, and each item's place
    // among the warp's items of as many tokens.
    const int c = tid < kExperts ? __popc(s_tok[tid]) : 0;
    int incl = c | (c > 0 ? 1 << 16 : 0), peer_rank = 0;
    if (warp < kExperts / 32) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      if (lane == 31) s_scan[warp] = incl;
      const uint32_t peers = __match_any_sync(0xffffffffu, c);
      peer_rank = __popc(peers & ((1u << lane) - 1u));
      if (c > 0 && peer_rank == 0) s_hist[warp][c - 1] = __popc(peers);
    }
    __syncthreads();
    if (warp < kExperts / 32) {
      const int v = lane < kExperts / 32 ? s_scan[lane] : 0;
      const int base = __reduce_add_sync(0xffffffffu, lane < warp ? v : 0), total = __reduce_add_sync(0xffffffffu, v);
      const int n_pairs = total & 0xFFFF, n_items = total >> 16;
      // Visiting order: items with more tokens first, ties by item index. Lane = token count - 1: items of that count in
      // all warps and in the warps before this one, then the items of larger counts.
      int all = 0, before = 0;
#pragma unroll
      for (int w = 0; w < kExperts / 32; ++w) {
        const int h = s_hist[w][lane & 15];
        all += h;
        before += w < warp ? h : 0;
      }
      int larger = lane < kMaxTok ? all : 0;
#pragma unroll
      for (int o = 1; o < kMaxTok; o <<= 1) {
        const int x = __shfl_down_sync(0xffffffffu, larger, o);
        larger += lane + o < kMaxTok ? x : 0;
      }
      const int order_base = __shfl_sync(0xffffffffu, larger - all + before, (c - 1) & 15);
      if (c > 0) {  // a chosen slot = an item
        const int first = base + incl;
        const int item = (first >> 16) - 1, pair_begin = (first & 0xFFFF) - c;
        s_begin[tid] = pair_begin;
        wc.slot[item] = tid;
        wc.pair_begin[item] = pair_begin;
        wc.order[order_base + peer_rank] = item;
        if constexpr (LAST) scratch.rank[tid] = int16_t(order_base + peer_rank);
      }
      if (tid == 0) {
        wc.pair_begin[n_items] = n_pairs;
        wc.n_items = n_items;
      }
    }
    // thread = pair, of the first warps, and for the pairs' places in their tokens of the last ones (of all there are)
    const int p2 = tid - (blockDim.x >= 512 + kMaxPairs ? 512 : 0), t2 = p2 / kTopK;
    int slot2 = -1, rank2 = 0;
    if (p2 >= 0 && p2 < np) {
      slot2 = scratch.slot[t2][p2 - t2 * kTopK];
#pragma unroll
      for (int k = 0; k < kTopK; ++k) rank2 += uint32_t(scratch.slot[t2][k]) < uint32_t(slot2) ? 1 : 0;
    }
    __syncthreads();
    auto pair_of = [&](int slot, int t) {  // tokens ascending inside an item
      return s_begin[slot] + __popc(s_tok[slot] & ((1u << t) - 1u));
    };
    if (valid) {
      int idx = -1;
      if (my_slot >= 0) {
        idx = pair_of(my_slot, pt);
        wc.pair_token[idx] = pt;
        wc.pair_weight[idx] = s_w[pt][pk];
      }
      s_pair[pt][pk] = idx;
    }
    if (slot2 >= 0) {
      const int pair = pair_of(slot2, t2);
      wc.token_row[t2][rank2] = pair;
      if constexpr (LAST) {
        const int mine = scratch.rank[slot2];
        bool last = true;
#pragma unroll
        for (int k = 0; k < kTopK; ++k) {
          const int other = scratch.slot[t2][k];
          last = last && (other < 0 || scratch.rank[other] <= mine);
        }
        if (last) wc.last_pair[t2] = pair;
      }
    }
  }
  __syncthreads();
  if (!publish || tid >= kExperts) return;  // (the device list is behind everything the streaming waits for)
  fb_moe_decode_work* work = ws.work;
  const int n_items = wc.n_items, n_pairs = wc.pair_begin[n_items];
  if (tid < n_items) {
    work->item_slot[tid] = wc.slot[tid];
    ws.sched[kSchedOrderBase + tid] = wc.order[tid];
  }
  if (tid <= n_items) work->item_pair_begin[tid] = wc.pair_begin[tid];
  if (tid < n_pairs) {
    work->pair_token[tid] = wc.pair_token[tid];
    work->pair_weight[tid] = wc.pair_weight[tid];
  }
  if (valid) {
    work->topk_expert[pt][pk] = s_id[pt][pk];
    work->topk_weight[pt][pk] = s_w[pt][pk];
    int held = 0;
#pragma unroll
    for (int k = 0; k < kTopK; ++k) held += s_pair[pt][k] >= 0 ? 1 : 0;
    if (pk < held) work->token_pairs[pt][pk] = wc.token_row[pt][pk];
    if (pk == 0) {
      work->token_pair_count[pt] = held;
      work->token_cold_count[pt] = kTopK - held;
    }
  }
  if (tid == 0) {
    work->n_items = n_items;
    work->n_pairs = n_pairs;
    work->n_cold = np - n_pairs;
    work->tokens = T;
    if (np - n_pairs && !remote_ok) atomicMax(ws.status, uint32_t(FB_STATUS_BAD_WORK));
  }
}

// What a streaming kernel needs to run the selection itself (the fused layer call): every CTA builds the
// work list in its own shared memory from the logits the route kernel stored, and block 0 also writes the
// device work list for the combine kernel and the host.
struct SelectArgs {
  const float* logits;  // [tokens][stride]
  int stride;
  const int32_t* slot_of;
  int tokens;
  int remote_ok;
  float* y_out;  // not null: the kernel adds up the token's partial rows itself (every expert held here)
};

// Stand-alone selection (the reference's moe_select_publish): block 0 routes, blocks 1..T quantize
// one token's activations each.
template <bool XBF16>
__global__ void __launch_bounds__(512) select_kernel(const float* logits, int logits_stride, const void* xv,
                                                     const int32_t* slot_of, int T, fb_moe_decode_workspace ws,
                                                     uint32_t* counts) {
  pdl_launch_dependents();
  pdl_wait_prior();
  if (blockIdx.x > 0) {
    const int t = blockIdx.x - 1;
    auto load = [&](int i) -> float {
      if constexpr (XBF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(xv)[size_t(t) * H + i]);
      else return static_cast<const float*>(xv)[size_t(t) * H + i];
    };
    for (int act = FB_ACT_Q8_K; act <= FB_ACT_Q8_0; ++act)
      if (ws.gate_up_format == 0 || act_of(ws.gate_up_format) == act)
        quantize_row_planar(act, H, load, ws.xq + xq_offset(act) + size_t(t) * FB_XQ_STRIDE);
    return;
  }
  __shared__ WorkCache s_work;  // the streaming kernels of this path read the device work list instead
  __shared__ __align__(16) SelectScratch s_scratch;
  select_block<false>([&](int t, int e) { return logits[size_t(t) * logits_stride + e]; },
               slot_of, T, ws, counts, false, true, true, s_work, s_scratch);
}

// Up to here values carry their own arrival flags (direct_store). At one token that is 7 to 13 % of a layer in every pair of
// formats, because the hand-off of h stands in the layer's chain; with more tokens the down tiles of the first experts cover
// the hand-off of the last ones, and each down tile quantizes its item's rows again. Eight layers, us, by counters and so:
//   512, IQ3_S + IQ3_S     one 161 144   three 245 230   four 253 253   six 312 326   sixteen 627 658
//        IQ4_NL + IQ4_NL   one 166 145   three 246 219   four 255 236   six 311 300   eight 377 363   sixteen 616 596
//        IQ4_NL + Q2_0     one 158 140   three 233 215   four 239 229   six 287 292   eight 343 349   sixteen 563 572
//        the other eight at one 158 to 174 and 137 to 155, at three 239 to 266 and 219 to 247; the lines are not drawn
//        further for them: six tokens +2 to -2 %
//   640, IQ3_S + IQ4_NL    one 178 154   two 237 227   three 292 287
//        the other nine at one 163 to 185 and 146 to 164, at two 212 to 249 and 201 to 247
__host__ __device__ constexpr int direct_tokens(int gate_up, int down, int inter) {
  return inter != 512 ? 1 : gate_up != FB_FMT_IQ4_NL ? 3 : down == FB_FMT_IQ4_NL ? kMaxTok : 4;
}
constexpr uint32_t kNotYet = 0xFFFFFFFFu;

// What route_kernel needs for an expert-parallel step with peer-memory exchange (n_ranks == 0: none).
struct EpRouteArgs {
  fb_ep_peers peers;
  const float* x_local;  // this rank's rows, fp32 [tpr][2560]
  int tpr;               // tokens per rank
  int parity;
  uint32_t step;
  uint32_t spin_limit;  // polls per awaited line
  int act;              // activation format the layer's gate/up weights pair with (set for every launch)
  int clear_h, clear_partial;  // floats at ws.h and ws.partial to set to kNotYet (multiples of four)
};

// Router projection and activation quantization in one launch (the head of the fused layer call; the
// selection runs inside the streaming kernel that follows, see SelectArgs). Bound: latency, from the predecessor's end to the
// logits. 128 blocks in clusters of four: cluster g owns router rows 16g..16g+15, its CTA q K elements [640q, 640q+640),
// two of the eight slices whose sums make a logit. The weights are asked into L2 ahead of the dependency wait, into
// registers behind it together with the x share, which goes to shared memory; every CTA sends the slice sums of rows
// 4i..4i+3 to CTA i of its cluster through distributed shared memory, and behind one cluster barrier CTA i adds them in
// slice order 0..7 (fixed: repeated calls are bitwise identical) and stores the logits. Two more warps of every block
// quantize the activation rows meanwhile, and block 0 clears the counters of the streaming kernels (none can be running:
// this kernel waited for its predecessor). From the wait to the last block's end: one token 2.3 us, sixteen 4.2, four with
// the shared rows 5.6; 4.5, 8.8 and 9.8 with clusters of eight (only fifteen of those find a multiprocessor per CTA, 33 of
// four do), x loaded in turns ahead of the weights, quantization behind the projection, and slice sums read out of the other
// CTAs, which then wait for their readers.
//
// With SHARED (the whole decode branch of a layer) the kernel also projects the shared expert's gate/up rows and router
// row 512, its gate: cluster g takes inter_s / 32 (gate, up) row pairs the same way, FP8 codes widened exactly, and
// stores h = bf16(silu(gate) * up). Five megabytes spread over 128 blocks that run anyway: as projections of their own
// on a second stream they cost four launches, two events and, the expert kernel filling every multiprocessor, no overlap.
struct SharedRouteArgs {
  const uint8_t* codes;    // [2 inter_s][2560] E4M3
  const void* scales;      // [2 inter_s], fp32 or bf16
  int scale_bf16;
  int inter_s;             // a multiple of 128, at most kSharedMaxInter
  __nv_bfloat16* h;        // [tokens][inter_s]
};
constexpr int kSharedMaxInter = 1024;
__device__ __forceinline__ float fp8_row_scale(const void* scales, int is_bf16, int row) {
  return is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(scales)[row]) : static_cast<const float*>(scales)[row];
}
__device__ __forceinline__ float2 e4m3x2_float2(uint32_t pair) {
  const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(pair), __NV_E4M3);
  return __half22float2(*reinterpret_cast<const __half2*>(&hr));
}
constexpr int kRouteSplits = 8, kRouteSlice = H / kRouteSplits;  // 320
constexpr int kRouteCluster = 4, kRouteSpan = H / kRouteCluster;  // a CTA's share of K: two slices
constexpr int kRouteRows = 4 * kRouteCluster;                     // router rows of a cluster
constexpr int kRouteBlocks = kExperts / kRouteRows * kRouteCluster;
constexpr int kRouteWarps = 16, kRouteThreads = (kRouteWarps + 2) * 32;  // projection; two warps quantize beside it
static_assert(kRouteSlice == 320, "lane layout below: two 128-element chunks and a 64-element tail");
static_assert(2 * kRouteBlocks >= kMaxTok * (H / 256), "a quantizing warp takes one 256-value piece");

template <bool XBF16, bool EP, bool SHARED = false>
__global__ void __launch_bounds__(kRouteThreads, 1) route_kernel(const __nv_bfloat16* w, const void* xv, int T, float* logits,
                                                                 int stride, fb_moe_decode_workspace ws, EpRouteArgs ep,
                                                                 SharedRouteArgs sh) {
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = blockIdx.x / kRouteCluster, q = int(cluster_cta_rank());  // (clusters are four consecutive blocks)
  const int n_sh = SHARED ? sh.inter_s / (kRouteBlocks / kRouteCluster) : 0;  // (gate, up) pairs of this cluster
  cluster_arrive();  // (its other half stands before the first store into another CTA's shared memory)
  {
    // The weights on their way into L2 while the kernel before this one runs out (nothing is read ahead of the wait).
    const void* src = nullptr;
    uint32_t bytes = 0;
    if (tid < kRouteRows) {
      src = w + size_t(g * kRouteRows + tid) * H + q * kRouteSpan;
      bytes = kRouteSpan * 2;
    } else if (SHARED && tid - kRouteRows < 2 * n_sh) {
      const int i = tid - kRouteRows, row = g * n_sh + (i < n_sh ? i : sh.inter_s + i - n_sh);
      src = sh.codes + size_t(row) * H + q * kRouteSpan;
      bytes = kRouteSpan;
    }
    if (src && (reinterpret_cast<uintptr_t>(src) & 15) == 0)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
  }
  pdl_wait_prior();
  constexpr bool ep_mode = EP;  // the single-GPU instantiation carries none of the exchange code
  const uint4* x_lines = nullptr;  // this rank's copy of all tokens' rows, as exchange lines
  if constexpr (EP) {
    // Expert-parallel step: this rank's own rows go to every rank as flag-in-data lines (block b
    // serves rank b % R with slice b / R of the rows); readers below poll the lines they need.
    const int R = ep.peers.n_ranks, d = int(blockIdx.x) % R, slice = int(blockIdx.x) / R, n_slices = int(gridDim.x) / R;
    // (the host refuses rank counts that do not divide the grid; the clamp keeps a stray block inside the rows)
    const int total = ep.tpr * (H / 4), lo = min(total, int(int64_t(total) * slice / n_slices)),
              hi = min(total, int(int64_t(total) * (slice + 1) / n_slices));
    uint4* dst = static_cast<uint4*>(ep.peers.x_all[d]) +
                 (size_t(ep.parity) * kMaxTok + size_t(ep.peers.rank) * ep.tpr) * (H / 2);
    const float4* src = reinterpret_cast<const float4*>(ep.x_local);
    for (int i = lo + tid; i < hi; i += kRouteThreads) {
      const float4 v = src[i];
      ll_store(dst + 2 * i, v.x, v.y, ep.step);
      ll_store(dst + 2 * i + 1, v.z, v.w, ep.step);
    }
    x_lines = static_cast<const uint4*>(ep.peers.x_all[ep.peers.rank]) + size_t(ep.parity) * kMaxTok * (H / 2);
  }
  // Four or eight values (the size of v) of token t from element e on, as fp32; e a multiple of four.
  auto load_x = [&](int t, int e, auto& v) {
    constexpr int n = sizeof(v) / sizeof(float);
    if constexpr (ep_mode) {
      const uint4* ln = x_lines + (size_t(t) * H + e) / 2;
#pragma unroll
      for (int i = 0; i < n / 2; ++i) {
        const float2 f = ll_read(ln + i, ep.step, ws.status, ep.spin_limit);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
      }
    } else if constexpr (XBF16) {
      const uint2* src = reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(xv) + size_t(t) * H + e);
#pragma unroll
      for (int i = 0; i < n / 4; ++i) {
        const uint2 u = src[i];
        v[4 * i] = __uint_as_float(u.x << 16);
        v[4 * i + 1] = __uint_as_float(u.x & 0xFFFF0000u);
        v[4 * i + 2] = __uint_as_float(u.y << 16);
        v[4 * i + 3] = __uint_as_float(u.y & 0xFFFF0000u);
      }
    } else {
      const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(xv) + size_t(t) * H + e);
#pragma unroll
      for (int i = 0; i < n / 4; ++i) {
        const float4 u = src[i];
        v[4 * i] = u.x;
        v[4 * i + 1] = u.y;
        v[4 * i + 2] = u.z;
        v[4 * i + 3] = u.w;
      }
    }
  };
  extern __shared__ __align__(16) float s_x[];  // this CTA's part of x [token][640]
  // what the cluster's CTAs send this one: [K slice][row][token] of the rows it finishes
  __shared__ float s_in[kRouteSplits][4][kMaxTok];
  constexpr int kShPer = SHARED ? kSharedMaxInter / kRouteBlocks : 1;  // (gate, up) pairs a CTA finishes, at most
  __shared__ float s_sh[kRouteSplits][2 * kShPer][kMaxTok];
  __shared__ float s_gate[SHARED ? kRouteSplits : 1][kMaxTok];
  const int per = n_sh / kRouteCluster;  // pairs a CTA finishes

  // Row groups of this cluster: four of four router rows; SHARED: n_sh / 2 of two (gate, up) pairs, then (cluster 0) router
  // row 512 with three rows of nothing. An item is a group and one of the CTA's two K slices; a warp takes an item for
  // every value of x it reads from shared memory to feed four rows. (Two rows and all tokens per warp: 3 us instead of
  // 1.5 at sixteen tokens, the shared-memory reads.) Without shared groups there are items for half of the warps: above two
  // tokens warps i and i + 8 share item i and take alternate pairs of tokens (neighbours would leave two schedulers idle up
  // to two tokens). Lane holds elements 128c + 4 lane .. +3 (c = 0, 1) and 256 + 2 lane, +1 of the slice.
  const int item0 = SHARED ? warp : warp & 7, tok0 = SHARED ? 0 : 2 * (warp >> 3), tok_step = SHARED ? 2 : 4;
  const int half = item0 & 1, slice = 2 * q + half, k0 = slice * kRouteSlice;  // (a warp's items are all on one slice)
  uint32_t raw[20];  // a group's rows as loaded
  float wr[4][10];
  auto fetch = [&](int row, int n) {  // n router rows
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r >= n) break;
      const __nv_bfloat16* wrow = w + size_t(row + r) * H + k0;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint2 u = reinterpret_cast<const uint2*>(wrow)[c * 32 + lane];
        raw[5 * r + 2 * c] = u.x;
        raw[5 * r + 2 * c + 1] = u.y;
      }
      raw[5 * r + 4] = reinterpret_cast<const uint32_t*>(wrow + 256)[lane];
    }
  };
  auto widen = [&](int n) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        wr[r][2 * i] = r < n ? __uint_as_float(raw[5 * r + i] << 16) : 0.0f;
        wr[r][2 * i + 1] = r < n ? __uint_as_float(raw[5 * r + i] & 0xFFFF0000u) : 0.0f;
      }
  };
  auto fetch_shared = [&](int u) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint8_t* wrow = sh.codes + size_t((r & 1 ? sh.inter_s : 0) + g * n_sh + 2 * u + (r >> 1)) * H + k0;
      raw[3 * r] = reinterpret_cast<const uint32_t*>(wrow)[lane];
      raw[3 * r + 1] = reinterpret_cast<const uint32_t*>(wrow)[32 + lane];
      raw[3 * r + 2] = reinterpret_cast<const uint16_t*>(wrow + 256)[lane];
    }
  };
  auto widen_shared = [&]() {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 a = e4m3x2_float2(raw[3 * r + c] & 0xFFFFu), b = e4m3x2_float2(raw[3 * r + c] >> 16);
        wr[r][4 * c + 0] = a.x;
        wr[r][4 * c + 1] = a.y;
        wr[r][4 * c + 2] = b.x;
        wr[r][4 * c + 3] = b.y;
      }
      const float2 a = e4m3x2_float2(raw[3 * r + 2]);
      wr[r][8] = a.x;
      wr[r][9] = a.y;
    }
  };
  // the slice's sums of the rows in wr over this warp's tokens, into the shared memory of the CTA that finishes the row
  auto project = [&](int group) {
    // lanes 4i end with row i >> 1 (of four), token i & 1 of a pair of tokens
    const int r = lane >> 3;
    const float* dst = &s_in[slice][r][0];
    uint32_t owner = uint32_t(group);
    bool live = (lane & 3) == 0;
    if (SHARED && group == 4 + n_sh / 2) {
      dst = s_gate[SHARED ? slice : 0];
      owner = kRouteCluster - 1;
      live = live && r == 0;
    } else if (SHARED && group >= 4) {
      const int p = 2 * (group - 4) + (r >> 1);
      owner = uint32_t(p / per);
      dst = &s_sh[slice][2 * (p - int(owner) * per) + (r & 1)][0];
    }
#pragma unroll 1
    for (int tg = tok0; tg < T; tg += tok_step) {  // (two at a time: registers)
      float acc[8];  // [row][token of the pair]
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (tg + t < T) {
          const float* xr = s_x + (tg + t) * kRouteSpan + half * kRouteSlice;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const float4 x4 = reinterpret_cast<const float4*>(xr)[c * 32 + lane];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              a[i] = fmaf(wr[i][4 * c + 0], x4.x, a[i]);
              a[i] = fmaf(wr[i][4 * c + 1], x4.y, a[i]);
              a[i] = fmaf(wr[i][4 * c + 2], x4.z, a[i]);
              a[i] = fmaf(wr[i][4 * c + 3], x4.w, a[i]);
            }
          }
          const float2 x2 = reinterpret_cast<const float2*>(xr + 256)[lane];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a[i] = fmaf(wr[i][8], x2.x, a[i]);
            a[i] = fmaf(wr[i][9], x2.y, a[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[2 * i + t] = a[i];
      }
      // Sum over the 32 lanes by the butterfly xor 16, 8, 4, 2, 1, halving the values a lane carries at its first three
      // steps: nine shuffles for the eight (row, token) sums.
#pragma unroll
      for (int n = 4, o = 16; n >= 1; n >>= 1, o >>= 1) {
        const bool hi = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const float send = hi ? acc[i] : acc[i + n], keep = hi ? acc[i + n] : acc[i];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
      if (live) st_cluster_u32(dst + tg + ((lane >> 2) & 1), owner, __float_as_uint(acc[0]));
    }
  };

  // Everything is asked for before anything is waited for: this warp's first rows, then its share of the x slice.
  if (warp < kRouteWarps) {
    if (!SHARED || item0 < 8) fetch(g * kRouteRows + 4 * (item0 >> 1), 4);
    else if (item0 < 8 + n_sh) fetch_shared((item0 - 8) >> 1);
    constexpr int kMaxX = kMaxTok * (kRouteSpan / 4) / (kRouteWarps * 32);
    float xs[kMaxX][4];
#pragma unroll
    for (int j = 0; j < kMaxX; ++j) {
      const int i = tid + j * kRouteWarps * 32, t = i / (kRouteSpan / 4), c = i - t * (kRouteSpan / 4);
      if (t < T) load_x(t, q * kRouteSpan + 4 * c, xs[j]);
    }
#pragma unroll
    for (int j = 0; j < kMaxX; ++j) {
      const int i = tid + j * kRouteWarps * 32;
      if (i < T * (kRouteSpan / 4)) reinterpret_cast<float4*>(s_x)[i] = make_float4(xs[j][0], xs[j][1], xs[j][2], xs[j][3]);
    }
    named_bar_sync(1, kRouteWarps * 32);
    cluster_wait();  // every CTA of the cluster runs: its shared memory may be written
    if (!SHARED || item0 < 8) {
      widen(4);
      project(item0 >> 1);
    }
    if constexpr (SHARED) {
#pragma unroll 1
      for (int i = item0 < 8 ? item0 + kRouteWarps : item0; i < 8 + n_sh; i += kRouteWarps) {
        if (i != item0) fetch_shared((i - 8) >> 1);
        widen_shared();
        project(i >> 1);
      }
      if (g == 0 && (item0 >> 1) == (4 + n_sh / 2) % (kRouteWarps / 2)) {
        fetch(kExperts, 1);
        widen(1);
        project(4 + n_sh / 2);
      }
    }
  } else {
    // activation quantization: one warp per 256 values (spread over the blocks first: a single token's ten pieces go to
    // ten different SMs); block 0 clears the counters of the streaming kernel
    const int task = (warp - kRouteWarps) * kRouteBlocks + int(blockIdx.x), t = task / (H / 256), b = task - t * (H / 256);
    if (t < T) {
      float v[8];
      load_x(t, 256 * b + 8 * lane, v);
      uint8_t* out = ws.xq + xq_offset(ep.act) + size_t(t) * FB_XQ_STRIDE;
      if (ep.act == FB_ACT_Q8_K) {
        int qv[8], ps;
        const float d = q8k_block_warp(v, qv, ps);
        store_q8k_block_planar(out, H, b, qv, ps, d);
      } else {
        q8_0_eight_blocks_warp(v, true, out + 256 * b, reinterpret_cast<float*>(out + H) + 8 * b);
      }
    }
    if (blockIdx.x == 0) {
      static_assert(kSchedOrderBase <= 2 * kMaxPairs && kMaxTok * kMaxDnTiles <= 2 * kMaxPairs, "one loop clears all");
      for (int i = tid - kRouteWarps * 32; i < 2 * kMaxPairs; i += 64) {
        ws.item_done[i] = 0;
        if (i < kSchedOrderBase) ws.sched[i] = 0;
        if (i < kMaxTok * kMaxDnTiles) ws.sched[kSchedParts + i] = 0;
      }
    }
    for (int i = int(blockIdx.x) * 64 + tid - kRouteWarps * 32; i < (ep.clear_h + ep.clear_partial) / 4; i += kRouteBlocks * 64) {
      float* dst = i < ep.clear_h / 4 ? ws.h + 4 * size_t(i) : ws.partial + 4 * size_t(i - ep.clear_h / 4);
      *reinterpret_cast<uint4*>(dst) = make_uint4(kNotYet, kNotYet, kNotYet, kNotYet);
    }
    __syncwarp();
    cluster_wait();
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();  // the sums of all slices are here; nobody reads another CTA's memory from now on
  if (tid < 4 * kMaxTok) {
    const int r = tid >> 4, t = tid & 15;
    if (t < T) {
      float v = 0.0f;
#pragma unroll
      for (int qq = 0; qq < kRouteSplits; ++qq) v += s_in[qq][r][t];
      logits[size_t(t) * stride + g * kRouteRows + 4 * q + r] = v;
    }
  }
  if constexpr (SHARED) {
    for (int i = tid; i < per * kMaxTok; i += kRouteThreads) {
      const int p = i >> 4, j = g * n_sh + q * per + p, t = i & 15;
      if (t >= T) continue;
      float gv = 0.0f, uv = 0.0f;
#pragma unroll
      for (int qq = 0; qq < kRouteSplits; ++qq) {
        gv += s_sh[qq][2 * p][t];
        uv += s_sh[qq][2 * p + 1][t];
      }
      gv *= fp8_row_scale(sh.scales, sh.scale_bf16, j);
      uv *= fp8_row_scale(sh.scales, sh.scale_bf16, sh.inter_s + j);
      sh.h[size_t(t) * sh.inter_s + j] = __float2bfloat16_rn(gv / (1.0f + expf(-gv)) * uv);
    }
    if (g == 0 && q == kRouteCluster - 1 && tid < T) {
      float v = 0.0f;
#pragma unroll
      for (int qq = 0; qq < kRouteSplits; ++qq) v += s_gate[SHARED ? qq : 0][tid];
      logits[size_t(tid) * stride + kExperts] = v;
    }
  }
}

// ------------------------------------------------------------------------------ streaming skeleton
// Tiles are handed out dynamically: the producer lane of each CTA takes the next tile index from a
// device counter (reset by the select kernel), so a CTA that drew an expert with many tokens simply
// takes fewer tiles. Work items are visited heaviest first (ws.sched[8..]). An expert with more
// than kTT tokens is staged once per group of kTT tokens (its weights come back from L2). Every
// output element is still written by exactly one thread after a fixed-order reduction: results do
// not depend on which CTA or warp ran which piece.
constexpr int kSchedGateUp = 0, kSchedDown = 1;

// What the producer tells the consumers about the entry staged in a ring slot (shared memory). A reader acquires it through
// the barrier on which the producer arrives behind store() (`full`, or `staged`); the entry number alone is also polled, to
// learn that the slot's barrier has reached the entry's phase (draw_task_n), and is therefore stored last.
struct alignas(16) StageMeta {
  int seq;         // entry number of this CTA
  int tile;        // entry kind: 0 gate/up, 1 down, 2 down and its item's first tile
  int pair0;       // first pair (row of h / partial) of this pass
  int ntp;         // tokens in this pass (1..kTT)
  int row0;        // first intermediate row (gate/up) or output row (down) of the tile
  int item;        // work item
  int item_pair0;  // first pair of the item
  int item_tok;    // tokens of the item
  float wgt[kTT];  // routing weights of the pass's pairs (down)
  __device__ __forceinline__ void store(int seq_, int tile_, int pair0_, int ntp_, int row0_, int item_, int item_pair0_,
                                        int item_tok_, const float (&wgt_)[kTT]) {
    const uint32_t a = smem_u32(this);
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a + 32), "f"(wgt_[0]), "f"(wgt_[1]) : "memory");
    asm volatile("st.shared.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(a + 16), "r"(row0_), "r"(item_), "r"(item_pair0_),
                 "r"(item_tok_)
                 : "memory");
    asm volatile("st.shared.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(seq_), "r"(tile_), "r"(pair0_), "r"(ntp_) : "memory");
  }
};
static_assert(kTT == 2 && sizeof(StageMeta) == 48, "three vector stores");

// Piece p of a row of h -> its place in a planar activation row of the down projection, by the calling warp: lane l holds
// elements 256 p + 8 l .. + 7 (none behind the row's end). `out`: the row, in global or shared memory, 16-byte aligned.
template <int I>
__device__ __forceinline__ void quantize_h_piece(const float (&v)[8], int p, int down_act, uint8_t* out) {
  if (I % 256 == 0 && down_act == FB_ACT_Q8_K) {
    int q[8], ps;
    const float d = q8k_block_warp(v, q, ps);
    store_q8k_block_planar(out, I, p, q, ps, d);
  } else {
    q8_0_eight_blocks_warp(v, 256 * p + 8 * int(threadIdx.x & 31) < I, out + 256 * p, reinterpret_cast<float*>(out + I) + 8 * p);
  }
}
// A whole row; all of its loads are in flight before the first block is quantized (the finishing warp waits on this chain:
// Q8_0 rows taken block by block, twenty round trips at 640, cost a layer of one token 8 us).
template <int I>
__device__ __forceinline__ void quantize_h_row(const float* h, int down_act, uint8_t* out) {
  constexpr int kPasses = (I + 255) / 256;
  const int lane = threadIdx.x & 31;
  float v[kPasses][8];
#pragma unroll
  for (int p = 0; p < kPasses; ++p) {
    const int e = 256 * p + 8 * lane;
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), c = a;
    if (e < I) {
      a = __ldcg(reinterpret_cast<const float4*>(h + e));
      c = __ldcg(reinterpret_cast<const float4*>(h + e) + 1);
    }
    v[p][0] = a.x; v[p][1] = a.y; v[p][2] = a.z; v[p][3] = a.w;
    v[p][4] = c.x; v[p][5] = c.y; v[p][6] = c.z; v[p][7] = c.w;
  }
#pragma unroll
  for (int p = 0; p < kPasses; ++p) quantize_h_piece<I>(v[p], p, down_act, out);
}

// Up to direct_tokens, values are their own arrival flags. The route kernel fills the rows with kNotYet, a NaN
// that no arithmetic produces; a value is stored once, by one relaxed store, and a reader polls the values it needs (a
// bounded number of times). Nothing else is read on the strength of a value, so no fence and no counter stand between a
// store and its reader: release, counter, a last contributor that re-quantizes a row, its flag, the row's copy into shared
// memory were four dependent round trips.
__device__ __forceinline__ void direct_store(float* p, float v) {
  const uint32_t b = __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(b == kNotYet ? 0x7FFFFFFFu : b) : "memory");
}
// Four values; `all` goes false where one is not there yet.
__device__ __forceinline__ float4 direct_load4(const float* p, bool& all) {
  uint4 u;
  asm volatile("ld.relaxed.gpu.global.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
               : "l"(p)
               : "memory");
  all = all && u.x != kNotYet && u.y != kNotYet && u.z != kNotYet && u.w != kNotYet;
  return make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
}
// Eight values of a row from element `at` on (zeros behind the row's end): false where one is not there yet.
__device__ __forceinline__ bool direct_load8(const float* row, int at, int n, float (&v)[8]) {
  bool all = true;
  float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), c = a;
  if (at < n) {
    a = direct_load4(row + at, all);
    c = direct_load4(row + at + 4, all);
  }
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
  return all;
}
// Polls of a value (or of an item's flag) that other multiprocessors write, unless the workspace names a number: each takes a
// round trip to L2 and a nap of 20 ns or more, two to three seconds in all. A layer may share the GPU with another stream's
// kernel, and the blocks that it waits for start behind that.
constexpr uint32_t kValuePolls = 1u << 22;
__device__ __forceinline__ uint32_t value_polls(const fb_moe_decode_workspace& ws) {
  return ws.wait_polls > 0 ? uint32_t(ws.wait_polls) : kValuePolls;
}
// Warps that quantize the h rows of a CTA's down entries, each its piece of 256 values.
constexpr int direct_warps(int inter) { return (inter + 255) / 256; }

// Counts one finished contribution to an item's h; the last one re-quantizes that item's h for the
// down projection and then sets the item's flag, ws.item_done[kMaxPairs + item], to `ready` (1 in a fused gate/up + down
// launch, which polls it before staging the item's rows). `expected` = contributions per item; the counter wraps to zero
// behind the last one.
template <int I>
__device__ __forceinline__ void item_contribution_done(const fb_moe_decode_workspace& ws, int item, int pair_begin,
                                                       int n_tok, int expected, int down_act, int ready, int lane) {
  // (release and acquire ride on the two atomics: at one token this chain is a tenth of the layer)
  __syncwarp();
  int ticket = 0;
  if (lane == 0)
    asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;" : "=r"(ticket) : "l"(&ws.item_done[item]), "r"(expected - 1) : "memory");
  ticket = __shfl_sync(0xffffffffu, ticket, 0);
  if (ticket == expected - 1) {
    __syncwarp();  // (the shuffle orders no memory: the other lanes read h behind lane 0's acquire by this)
    for (int p = pair_begin; p < pair_begin + n_tok; ++p)
      quantize_h_row<I>(ws.h + size_t(p) * I, down_act, ws.hq + size_t(p) * FB_HQ_STRIDE);
    __syncwarp();
    if (lane == 0) asm volatile("red.release.gpu.global.or.b32 [%0], %1;" ::"l"(&ws.item_done[kMaxPairs + item]), "r"(ready) : "memory");
  }
}

#include "moe_decode_generic.cuh"
#include "moe_decode_experts.cuh"

// ------------------------------------------------------------------------------ combine
// y[t][n] = partials of token t in slot order (+ y_shared); optional rank-1 ablation of the routed
// part; X[t][s][n] += inj[t][s] * y (4 residual streams) when X is given; y_out optional.
// One block per (token, 256-column slice): the projection r . y_routed needs the whole row, so
// with ablation a block first reduces the row (only then).
// Column n of token t's partial rows, added in slot order; all loads in flight at once.
__device__ __forceinline__ float sum_partials(const fb_moe_decode_workspace& ws, int t, int np, int n) {
  int row[kTopK];
  float v[kTopK];
#pragma unroll
  for (int k = 0; k < kTopK; ++k) row[k] = k < np ? ws.work->token_pairs[t][k] : 0;
#pragma unroll
  for (int k = 0; k < kTopK; ++k) v[k] = k < np ? ws.partial[size_t(row[k]) * H + n] : 0.0f;
  float y = 0.0f;
#pragma unroll
  for (int k = 0; k < kTopK; ++k)
    if (k < np) y += v[k];
  return y;
}

__global__ void __launch_bounds__(256) combine_kernel(fb_moe_decode_workspace ws, const float* y_shared,
                                                      const float* inj, float* X, float* y_out, const float* ablate,
                                                      float ablate_scale) {
  pdl_launch_dependents();
  pdl_wait_prior();
  const int t = blockIdx.y;
  const fb_moe_decode_work* work = ws.work;
  const int np = min(max(work->token_pair_count[t], 0), kTopK);
  __shared__ float s_red[8];
  __shared__ float s_proj;
  float proj = 0.0f;
  if (ablate) {
    float loc = 0.0f;
    for (int n = threadIdx.x; n < H; n += 256) {
      float y = 0.0f;
      for (int k = 0; k < np; ++k) y += ws.partial[size_t(work->token_pairs[t][k]) * H + n];
      loc = fmaf(ablate[n], y, loc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loc += __shfl_xor_sync(0xffffffffu, loc, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = loc;
    __syncthreads();
    if (threadIdx.x == 0) {
      float s = 0.0f;
      for (int i = 0; i < 8; ++i) s += s_red[i];
      s_proj = s;
    }
    __syncthreads();
    proj = s_proj;
  }
  const int n = blockIdx.x * 256 + threadIdx.x;
  float y = sum_partials(ws, t, np, n);
  if (ablate) y -= ablate_scale * ablate[n] * proj;
  if (y_shared) y += y_shared[size_t(t) * H + n];
  float x[4], g[4];  // (all loads ahead of the stores: they may meet for all the compiler knows)
  if (X) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      x[s] = X[(size_t(t) * 4 + s) * H + n];
      g[s] = inj[t * 4 + s];
    }
  }
  if (y_out) y_out[size_t(t) * H + n] = y;
  if (X) {
#pragma unroll
    for (int s = 0; s < 4; ++s) X[(size_t(t) * 4 + s) * H + n] = x[s] + g[s] * y;
  }
}

// The combine of the whole decode branch: the shared expert's down projection (y_shared[t][n] = sigmoid(gate logit) *
// scale[n] * sum_k h[t][k] W[n][k], exact products, fp32 sums) for 16 columns and all tokens first, then their sums and
// residual writes. The 1.6 MB of codes are read once, by 160 blocks; as a projection of its own in front of the combine
// it took 6 us. Warp = two columns, lanes split K; h of all tokens in shared memory.
struct SharedDownArgs {
  const uint8_t* codes;  // [2560][k] E4M3
  const void* scales;
  int scale_bf16;
  int k;                 // a multiple of 128
  const __nv_bfloat16* h;
  const float* logits;   // [tokens][stride], the gate in column 512
  int stride;
  float* y_shared;
};
constexpr int kCsCols = 16, kCsMaxK = kSharedMaxInter;
__global__ void __launch_bounds__(256) combine_shared_kernel(fb_moe_decode_workspace ws, SharedDownArgs sh, int T,
                                                             const float* inj, float* X, float* y_out) {
  extern __shared__ __align__(16) float s_h[];  // [token][k]
  __shared__ float s_y[kMaxTok][kCsCols];
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n0 = blockIdx.x * kCsCols;
  {  // on their way into L2 while the expert kernel finishes
    const int bytes = kCsCols * sh.k;
    for (int i = tid * 128; i < bytes; i += 256 * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(sh.codes + size_t(n0) * sh.k + i));
  }
  pdl_wait_prior();
  // Everything the block reads is asked for before it waits for any of it: its codes, its partial rows and residual
  // streams (thread = token, column), then h.
  constexpr int kChunks = kCsMaxK / 128;
  const int chunks = sh.k / 128, t_out = tid >> 4, n = n0 + (tid & 15);
  uint32_t codes[kChunks][2];
#pragma unroll
  for (int c = 0; c < kChunks; ++c)
    if (c < chunks) {
#pragma unroll
      for (int r = 0; r < 2; ++r)
        codes[c][r] = reinterpret_cast<const uint32_t*>(sh.codes + size_t(n0 + 2 * warp + r) * sh.k)[c * 32 + lane];
    }
  float routed = 0.0f, xs[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (t_out < T) {
    routed = sum_partials(ws, t_out, min(max(ws.work->token_pair_count[t_out], 0), kTopK), n);
    if (X) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        xs[i] = X[(size_t(t_out) * 4 + i) * H + n];
        gs[i] = inj[t_out * 4 + i];
      }
    }
  }
  for (int i = tid; i < T * sh.k / 8; i += 256) {
    const uint4 u = reinterpret_cast<const uint4*>(sh.h)[i];
    float4* d = reinterpret_cast<float4*>(s_h) + 2 * i;
    d[0] = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xFFFF0000u));
    d[1] = make_float4(__uint_as_float(u.z << 16), __uint_as_float(u.z & 0xFFFF0000u), __uint_as_float(u.w << 16),
                       __uint_as_float(u.w & 0xFFFF0000u));
  }
  __syncthreads();
  float acc[32];  // [column of the warp][token]
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    if (c >= chunks) break;
    float w[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float2 a = e4m3x2_float2(codes[c][r] & 0xFFFFu), b = e4m3x2_float2(codes[c][r] >> 16);
      w[r][0] = a.x; w[r][1] = a.y; w[r][2] = b.x; w[r][3] = b.y;
    }
#pragma unroll
    for (int t = 0; t < kMaxTok; ++t) {
      if (t < T) {
        const float4 hv = reinterpret_cast<const float4*>(s_h + t * sh.k)[c * 32 + lane];
#pragma unroll
        for (int r = 0; r < 2; ++r)
          acc[16 * r + t] = fmaf(w[r][3], hv.w, fmaf(w[r][2], hv.z, fmaf(w[r][1], hv.y, fmaf(w[r][0], hv.x, acc[16 * r + t]))));
      }
    }
  }
  // the butterfly of the route kernel: lane l ends with column l >> 4, token l & 15
#pragma unroll
  for (int m = 16, o = 16; m >= 1; m >>= 1, o >>= 1) {
    const bool hi = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < m; ++i) {
      const float send = hi ? acc[i] : acc[i + m], keep = hi ? acc[i + m] : acc[i];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  {
    const int t = lane & 15, col = 2 * warp + (lane >> 4);
    if (t < T)
      s_y[t][col] = acc[0] * fp8_row_scale(sh.scales, sh.scale_bf16, n0 + col) /
                    (1.0f + expf(-sh.logits[size_t(t) * sh.stride + kExperts]));
  }
  __syncthreads();
  if (t_out < T) {
    const float ysh = s_y[t_out][tid & 15], y = routed + ysh;
    sh.y_shared[size_t(t_out) * H + n] = ysh;
    if (y_out) y_out[size_t(t_out) * H + n] = y;
    if (X) {
#pragma unroll
      for (int i = 0; i < 4; ++i) X[(size_t(t_out) * 4 + i) * H + n] = xs[i] + gs[i] * y;
    }
  }
}

// ------------------------------------------------------------------------------ expert-parallel combine
// y[r][n] = parts[0][r][n] + parts[1][r][n] + ... in rank order (deterministic).
__global__ void __launch_bounds__(256) sum_ranks_kernel(const float* __restrict__ parts, int n_ranks, int64_t elems,
                                                        float* __restrict__ y) {
  const int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x;
  if (i >= elems) return;
  float v = 0.0f;
  for (int r = 0; r < n_ranks; ++r) v += parts[int64_t(r) * elems + i];
  y[i] = v;
}

// ------------------------------------------------------------------------------ peer-memory exchange
// Expert-parallel decode without a collective library call in the step: ranks write flag-in-data
// lines (ll_store) straight into each other's buffers over NVLink and readers poll the lines they
// need in their OWN memory, a bounded number of times. No fence, no ticket, no separate flag sits
// between the data and its arrival. Buffers are double-buffered by step parity: a rank can be at
// most one step ahead of a peer (it needs that peer's partial rows to finish a step), so the lines
// of step k+2 never overwrite lines of step k that someone still reads, and a stale line (step
// k-2) never passes for a current one.
//   x_all   [2][16][1280] lines         all tokens of the step, rows written by their owners
//   y_parts [2][8][16][1280] lines      [parity][source rank][local token]: partial rows for this rank's tokens

// The combine of an expert-parallel step. Thread = (token t, two adjacent columns): token t's partial
// row over the local pairs (slot order) goes straight into its owner's y_parts; threads of tokens
// this rank owns then read the partial rows of all ranks and add them in rank order.
__global__ void __launch_bounds__(256) ep_combine_exchange_kernel(fb_moe_decode_workspace ws, fb_ep_peers peers, int tpr,
                                                                  int parity, uint32_t step, uint32_t spin_limit,
                                                                  float* y_local) {
  pdl_launch_dependents();
  pdl_wait_prior();
  const int t = blockIdx.y;
  const fb_moe_decode_work* work = ws.work;
  const int np = min(max(work->token_pair_count[t], 0), kTopK);
  const int c = blockIdx.x * 256 + threadIdx.x;  // line = columns 2c, 2c+1
  float y0 = 0.0f, y1 = 0.0f;
  for (int k = 0; k < np; ++k) {
    const float2 v = *reinterpret_cast<const float2*>(ws.partial + size_t(work->token_pairs[t][k]) * H + 2 * c);
    y0 += v.x;
    y1 += v.y;
  }
  const int d = t / tpr, i = t - d * tpr;
  ll_store(static_cast<uint4*>(peers.y_parts[d]) + ((size_t(parity) * kEpMaxRanks + peers.rank) * kMaxTok + i) * (H / 2) + c,
           y0, y1, step);
  if (d != peers.rank) return;
  const uint4* mine = static_cast<const uint4*>(peers.y_parts[peers.rank]);
  float a0 = 0.0f, a1 = 0.0f;
  for (int s = 0; s < peers.n_ranks; ++s) {
    const float2 v =
        ll_read(mine + ((size_t(parity) * kEpMaxRanks + s) * kMaxTok + i) * (H / 2) + c, step, ws.status, spin_limit);
    a0 += v.x;
    a1 += v.y;
  }
  *reinterpret_cast<float2*>(y_local + size_t(i) * H + 2 * c) = make_float2(a0, a1);
}

// x of fb_moe_layer_decode_host from page-locked host memory. Bound: one round trip over PCIe. As a copy operation it ends
// the launch chain (the route kernel is then launched behind it, not beside it).
__global__ void __launch_bounds__(256) copy_in_kernel(const uint4* src, uint4* dst, int n) {
  pdl_launch_dependents();
  pdl_wait_prior();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) dst[i] = src[i];
}

// ------------------------------------------------------------------------------ host side
// Device address of a buffer that lies in page-locked host memory from end to end, or nullptr for any other. (The driver is
// asked, not the runtime: it also tells how far an allocation or registration reaches, in as long a call, 0.7 us.)
void* pinned_on_device(const void* host, size_t bytes) {
  using QueryFn = CUresult (*)(unsigned int, CUpointer_attribute*, void**, CUdeviceptr);
  static const QueryFn attributes = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<QueryFn>(p);
  }();
  if (!attributes) return nullptr;
  return reinterpret_cast<void*>(pinned_range(reinterpret_cast<uintptr_t>(host), bytes, [&](uintptr_t at, PinnedByte& b) {
    unsigned int type = 0, managed = 0;  // (they stay 0 for memory that CUDA does not know)
    CUdeviceptr device = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute what[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                   CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                   CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* into[5] = {&type, &managed, &device, &start, &size};
    if (attributes(5, what, into, CUdeviceptr(at)) != CUDA_SUCCESS || type != CU_MEMORYTYPE_HOST || managed) return false;
    cudaPointerAttributes pa{};
    if (!device && cudaPointerGetAttributes(&pa, reinterpret_cast<const void*>(at)) == cudaSuccess)
      device = CUdeviceptr(reinterpret_cast<uintptr_t>(pa.devicePointer));  // (a thread that has no context yet)
    b = PinnedByte{uintptr_t(device), uintptr_t(start), size};
    return true;
  }));
}

bool layout_ok(const fb_moe_expert_layout* L) {
  if (!L || !L->slots) return false;
  if ((reinterpret_cast<uintptr_t>(L->slots) | uintptr_t(L->blob_stride) | uintptr_t(L->gate_offset) |
       uintptr_t(L->up_offset) | uintptr_t(L->down_offset)) & 15)
    return false;
  if (L->inter != 512 && L->inter != 640) return false;
  if (L->gate_up_format != FB_FMT_IQ3_S && L->gate_up_format != FB_FMT_IQ4_NL &&
      L->gate_up_format != FB_FMT_IQ3_XXS && L->gate_up_format != FB_FMT_IQ2_S && L->gate_up_format != FB_FMT_IQ4_XS)
    return false;
  if (L->down_format == FB_FMT_IQ3_S) return L->inter % 256 == 0;
  return L->down_format == FB_FMT_IQ4_NL || L->down_format == FB_FMT_Q2_0;
}

// Polls a reader gives a peer-written exchange line before it records FB_STATUS_PIPELINE_TIMEOUT.
uint32_t g_peer_wait_polls = kPeerSpinLimit;

// A workspace made for a layout must be used with that layout; one made without (formats 0) fits all.
bool ws_fits(const fb_moe_decode_workspace* ws, const fb_moe_expert_layout* L, bool gate_up, bool down) {
  if (ws->inter && ws->inter != L->inter) return false;
  if (gate_up && ws->gate_up_format && ws->gate_up_format != L->gate_up_format) return false;
  if (down && ws->down_format && ws->down_format != L->down_format) return false;
  return true;
}

bool ws_ok(const fb_moe_decode_workspace* ws) {
  return ws && ws->work && ws->xq && ws->h && ws->hq && ws->partial && ws->item_done && ws->sched && ws->status;
}

// The streaming expert kernel over the given phases; with `sel` it runs the selection itself.
template <int GU, int DN, int INTER>
int32_t launch_experts_as(const fb_moe_expert_layout* layout, const fb_moe_decode_workspace* ws, int phases,
                          void* stream, const char* what, const SelectArgs* sel) {
  using C = ExpertsCfg<GU, DN, INTER>;
  auto launch = [&](auto kernel, PerDeviceOnce& once, int threads) -> int32_t {
    const cudaError_t attr = per_device_once(once, [&] { return opt_in_smem(kernel, C::kSmem); });
    if (attr != cudaSuccess) {
      set_error("%s: shared-memory opt-in: %s", what, cudaGetErrorString(attr));
      return int32_t(attr);
    }
    const cudaError_t e = launch_pdl(kernel, dim3(sm_count()), dim3(threads), C::kSmem, as_stream(stream), *layout, *ws,
                                     sel ? (phases | kPhaseSelect) : phases, sel ? *sel : SelectArgs{});
    return e != cudaSuccess ? check_launch(what) : 0;
  };
  static PerDeviceOnce once[2];
  // the fused call's few tokens (the route kernel has filled h and the partial rows: layer_decode_impl)
  if (sel && sel->tokens <= direct_tokens(GU, DN, INTER) && phases == (kPhaseGateUp | kPhaseDown))
    return launch(experts_kernel<GU, DN, INTER, true>, once[1], C::threads(true));
  return launch(experts_kernel<GU, DN, INTER, false>, once[0], C::threads(false));
}
// Every gate/up format has its kernel with an IQ4_NL or Q2_0 down projection at both intermediate sizes; IQ3_S also with
// its own.
template <int GU>
int32_t launch_experts_gu(const fb_moe_expert_layout* layout, const fb_moe_decode_workspace* ws, int phases, void* stream,
                          const char* what, const SelectArgs* sel) {
  if (layout->down_format == FB_FMT_Q2_0)
    return layout->inter == 512 ? launch_experts_as<GU, FB_FMT_Q2_0, 512>(layout, ws, phases, stream, what, sel)
                                : launch_experts_as<GU, FB_FMT_Q2_0, 640>(layout, ws, phases, stream, what, sel);
  return layout->inter == 512 ? launch_experts_as<GU, FB_FMT_IQ4_NL, 512>(layout, ws, phases, stream, what, sel)
                              : launch_experts_as<GU, FB_FMT_IQ4_NL, 640>(layout, ws, phases, stream, what, sel);
}
int32_t launch_phases(const fb_moe_expert_layout* layout, const fb_moe_decode_workspace* ws, int phases, void* stream,
                      const char* what, const SelectArgs* sel) {
  const bool dn_iq3s = layout->down_format == FB_FMT_IQ3_S;
  // a down-only launch does not care for the gate/up format: IQ4_NL's kernel has no table to fill
  const int gu = phases & kPhaseGateUp ? layout->gate_up_format : dn_iq3s ? FB_FMT_IQ3_S : FB_FMT_IQ4_NL;
  switch (gu) {
    case FB_FMT_IQ3_S:
      if (dn_iq3s) return launch_experts_as<FB_FMT_IQ3_S, FB_FMT_IQ3_S, 512>(layout, ws, phases, stream, what, sel);
      return launch_experts_gu<FB_FMT_IQ3_S>(layout, ws, phases, stream, what, sel);
    case FB_FMT_IQ4_NL: return launch_experts_gu<FB_FMT_IQ4_NL>(layout, ws, phases, stream, what, sel);
    case FB_FMT_IQ2_S: return launch_experts_gu<FB_FMT_IQ2_S>(layout, ws, phases, stream, what, sel);
    case FB_FMT_IQ3_XXS: return launch_experts_gu<FB_FMT_IQ3_XXS>(layout, ws, phases, stream, what, sel);
    default: return launch_experts_gu<FB_FMT_IQ4_XS>(layout, ws, phases, stream, what, sel);
  }
}

}  // namespace
}  // namespace fb

using namespace fb;

extern "C" {

size_t fb_moe_decode_workspace_bytes(int32_t inter) {
  (void)inter;
  auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
  return up(sizeof(fb_moe_decode_work)) + up(size_t(2 * kMaxTok) * FB_XQ_STRIDE) + up(size_t(kMaxPairs) * 640 * 4) +
         up(size_t(kMaxPairs) * FB_HQ_STRIDE) + up(size_t(kMaxPairs) * H * 4) + up(2 * kMaxPairs * 4) +
         up(kSchedInts * 4) + 256;
}

int32_t fb_moe_decode_workspace_make(void* base, const fb_moe_expert_layout* layout, fb_moe_decode_workspace* out) {
  if (!base || !out || (reinterpret_cast<uintptr_t>(base) & 255)) return invalid("decode workspace: base must be 256-byte aligned");
  if (layout && !layout_ok(layout)) return invalid("decode workspace: unsupported expert layout");
  auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
  uint8_t* p = static_cast<uint8_t*>(base);
  out->work = reinterpret_cast<fb_moe_decode_work*>(p);
  p += up(sizeof(fb_moe_decode_work));
  out->xq = p;
  p += up(size_t(2 * kMaxTok) * FB_XQ_STRIDE);
  out->h = reinterpret_cast<float*>(p);
  p += up(size_t(kMaxPairs) * 640 * 4);
  out->hq = p;
  p += up(size_t(kMaxPairs) * FB_HQ_STRIDE);
  out->partial = reinterpret_cast<float*>(p);
  p += up(size_t(kMaxPairs) * H * 4);
  out->item_done = reinterpret_cast<int32_t*>(p);
  p += up(2 * kMaxPairs * 4);
  out->sched = reinterpret_cast<int32_t*>(p);
  p += up(kSchedInts * 4);
  out->status = reinterpret_cast<uint32_t*>(p);
  out->gate_up_format = layout ? layout->gate_up_format : 0;  // 0: any (the selection quantizes x both ways)
  out->down_format = layout ? layout->down_format : 0;
  out->inter = layout ? layout->inter : 0;
  out->wait_polls = 0;
  return 0;
}

int32_t fb_router_logits(const void* w_bf16, int32_t rows, const void* x, int32_t x_dtype, int32_t tokens,
                         float* logits, int32_t logits_stride, void* stream) {
  if (!w_bf16 || !x || !logits || rows <= 0 || tokens <= 0 || logits_stride < rows)
    return invalid("router_logits: bad arguments");
  if (tokens > kMaxTok) {
    // Tiles of fewer rows while they run as one wave (513 rows, us, while rows beyond the end were still read: 17 tokens 26.7 ->
    // 14.6, 40 27.1 -> 19.2, 100 28.0 -> 20.2); beyond that each wave of smaller blocks costs as much as it saves.
    const int tok_tiles = (tokens + kRtTok - 1) / kRtTok;
    auto tiles = [&](int r) { return ((rows + r - 1) / r) * tok_tiles; };
    auto launch = [&](auto kernel, PerDeviceOnce& once, int r, int smem) {
      cudaError_t a = per_device_once(once, [&] { return opt_in_smem(kernel, smem); });
      if (a == cudaSuccess)
        a = launch_pdl(kernel, dim3((rows + r - 1) / r, tok_tiles), dim3(512), size_t(smem), as_stream(stream),
                       static_cast<const __nv_bfloat16*>(w_bf16), rows, x, tokens, logits, logits_stride);
      return a;
    };
    static PerDeviceOnce once[6];
    const bool bf = x_dtype == FB_DT_BF16;
    const cudaError_t e =
        tiles(8) <= sm_count()    ? bf ? launch(router_tile_kernel<true, 8>, once[0], 8, router_tile_smem<true, 8>())
                                       : launch(router_tile_kernel<false, 8>, once[1], 8, router_tile_smem<false, 8>())
        : tiles(16) <= sm_count() ? bf ? launch(router_tile_kernel<true, 16>, once[2], 16, router_tile_smem<true, 16>())
                                       : launch(router_tile_kernel<false, 16>, once[3], 16, router_tile_smem<false, 16>())
        : bf                      ? launch(router_tile_kernel<true, 32>, once[4], 32, router_tile_smem<true, 32>())
                                  : launch(router_tile_kernel<false, 32>, once[5], 32, router_tile_smem<false, 32>());
    if (e == cudaSuccess) return 0;
    set_error("router_logits: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return int32_t(e);
  }
  const dim3 grid((rows + 3) / 4), block(128);
  cudaError_t e = x_dtype == FB_DT_BF16
                      ? launch_pdl(router_kernel<true>, grid, block, 0, as_stream(stream),
                                   static_cast<const __nv_bfloat16*>(w_bf16), rows, x, tokens, logits, logits_stride)
                      : launch_pdl(router_kernel<false>, grid, block, 0, as_stream(stream),
                                   static_cast<const __nv_bfloat16*>(w_bf16), rows, x, tokens, logits, logits_stride);
  if (e != cudaSuccess) return check_launch("router_logits");
  return 0;
}

int32_t fb_moe_select_publish(const float* router_logits, int32_t logits_stride, const void* x, int32_t x_dtype,
                              const int32_t* slot_of, int32_t layer, const uint32_t* seq, void* exchange,
                              int32_t tokens, const fb_moe_decode_workspace* ws, void* stream,
                              uint32_t* routing_counts) {
  (void)layer;
  (void)seq;
  if (exchange) return invalid("select_publish: no CPU expert tier exists behind these kernels; exchange must be NULL");
  if (!router_logits || !x || !ws_ok(ws) || tokens < 1 || tokens > kMaxTok || logits_stride < kExperts)
    return invalid("select_publish: bad arguments (tokens must be 1..16)");
  cudaError_t e = x_dtype == FB_DT_BF16
                      ? launch_pdl(select_kernel<true>, dim3(1 + tokens), dim3(512), 0, as_stream(stream),
                                   router_logits, logits_stride, x, slot_of, tokens, *ws, routing_counts)
                      : launch_pdl(select_kernel<false>, dim3(1 + tokens), dim3(512), 0, as_stream(stream),
                                   router_logits, logits_stride, x, slot_of, tokens, *ws, routing_counts);
  if (e != cudaSuccess) return check_launch("select_publish");
  return 0;
}

// `sel`: the kernel runs the selection itself (the fused layer call), else it reads the device work list.
static int32_t launch_gate_up(const fb_moe_expert_layout* layout, const fb_moe_decode_workspace* ws, void* stream,
                              const SelectArgs* sel) {
  return launch_phases(layout, ws, kPhaseGateUp, stream, "hot_gate_up", sel);
}

int32_t fb_moe_hot_gate_up(const fb_moe_expert_layout* layout, int32_t tokens, const fb_moe_decode_workspace* ws,
                           void* stream) {
  if (!layout_ok(layout) || !ws_ok(ws) || tokens < 1 || tokens > kMaxTok) return invalid("hot_gate_up: bad arguments");
  if (!ws_fits(ws, layout, true, true))
    return invalid("hot_gate_up: workspace was made for a different layout");
  return launch_gate_up(layout, ws, stream, nullptr);
}

static int32_t launch_down(const fb_moe_expert_layout* layout, const fb_moe_decode_workspace* ws, void* stream);

static bool one_launch(const fb_moe_expert_layout* layout) {
  return layout->down_format != FB_FMT_IQ3_S || layout->gate_up_format == FB_FMT_IQ3_S;
}
// Both projections of every routed expert: one launch, but for IQ3_S down behind another gate/up format.
static int32_t launch_experts(const fb_moe_expert_layout* layout, const fb_moe_decode_workspace* ws, void* stream,
                              const SelectArgs* sel) {
  if (one_launch(layout))
    return launch_phases(layout, ws, kPhaseGateUp | kPhaseDown, stream, "hot_experts", sel);
  const int32_t st = launch_gate_up(layout, ws, stream, sel);
  return st ? st : launch_down(layout, ws, stream);
}

int32_t fb_moe_hot_experts(const fb_moe_expert_layout* layout, int32_t tokens, const fb_moe_decode_workspace* ws,
                           void* stream) {
  if (!layout_ok(layout) || !ws_ok(ws) || tokens < 1 || tokens > kMaxTok) return invalid("hot_experts: bad arguments");
  if (!ws_fits(ws, layout, true, true))
    return invalid("hot_experts: workspace was made for a different layout");
  return launch_experts(layout, ws, stream, nullptr);
}

static int32_t launch_down(const fb_moe_expert_layout* layout, const fb_moe_decode_workspace* ws, void* stream) {
  return launch_phases(layout, ws, kPhaseDown, stream, "hot_down", nullptr);
}

int32_t fb_moe_hot_down(const fb_moe_expert_layout* layout, int32_t tokens, const fb_moe_decode_workspace* ws,
                        void* stream) {
  if (!layout_ok(layout) || !ws_ok(ws) || tokens < 1 || tokens > kMaxTok) return invalid("hot_down: bad arguments");
  if (!ws_fits(ws, layout, false, true))
    return invalid("hot_down: workspace was made for a different layout");
  return launch_down(layout, ws, stream);
}

int32_t fb_moe_combine(const fb_moe_decode_workspace* ws, const float* y_shared, void* exchange, int32_t layer,
                       const uint32_t* seq, const float* inj, float* X, float* y_out, int32_t tokens,
                       long long timeout_cycles, const float* ablate_direction, float ablate_scale, void* stream) {
  (void)layer;
  (void)seq;
  (void)timeout_cycles;
  if (exchange) return invalid("combine: no CPU expert tier exists behind these kernels; exchange must be NULL");
  if (!ws_ok(ws) || tokens < 1 || tokens > kMaxTok || (X && !inj) || (!X && !y_out))
    return invalid("combine: bad arguments");
  cudaError_t e = launch_pdl(combine_kernel, dim3(H / 256, tokens), dim3(256), 0, as_stream(stream), *ws, y_shared, inj,
                             X, y_out, ablate_direction, ablate_scale);
  if (e != cudaSuccess) return check_launch("combine");
  return 0;
}

static int32_t layer_decode_impl(const void* router_w_bf16, const fb_moe_expert_layout* layout,
                                 const int32_t* slot_of, bool remote_ok, const void* x, int32_t x_dtype,
                                 int32_t tokens, const fb_moe_decode_workspace* ws, float* logits_scratch, float* y_out,
                                 void* stream, const EpRouteArgs* ep = nullptr, const SharedRouteArgs* shared = nullptr) {
  const bool with_combine = ep == nullptr && shared == nullptr;
  EpRouteArgs era{};
  if (ep) era = *ep;
  era.act = layout_ok(layout) ? act_of(layout->gate_up_format) : FB_ACT_Q8_K;
  const bool own_combine = with_combine && !slot_of && layout_ok(layout) && one_launch(layout);
  if (layout_ok(layout) && one_launch(layout) &&
      tokens <= direct_tokens(layout->gate_up_format, layout->down_format, layout->inter)) {
    era.clear_h = tokens * kTopK * layout->inter;
    era.clear_partial = own_combine ? tokens * kTopK * H : 0;
  }
  // Two launches: route (router projection + activation quantization) and the expert kernel (every CTA runs the
  // selection on the stored logits, then gate/up and down tiles in one persistent launch, whose warps also combine a
  // token's rows when its last one is there). IQ3_S down behind another gate/up format takes a gate/up and a down launch,
  // and a caller with a table of resident slots a combine launch. The expert arithmetic is that of the separate entry
  // points. The route kernel sums a logit as eight K slices of
  // 320 added in slice order, where fb_router_logits sums 80 values per lane and then the lanes: the two
  // projections agree to fp32 rounding (a few ulp), not bit for bit, so a near-tie between the tenth and
  // eleventh expert may resolve differently. Only rows 0..511 of logits_scratch are written: row 512
  // (the shared-expert gate) is not produced here.
  if (!router_w_bf16 || !x || (!y_out && with_combine) || !logits_scratch || !layout_ok(layout) || !ws_ok(ws) ||
      tokens < 1 || tokens > kMaxTok)
    return invalid("layer_decode: bad arguments (tokens must be 1..16, logits scratch [tokens][513] required)");
  if (!ws_fits(ws, layout, true, true))
    return invalid("layer_decode: workspace was made for a different layout");
  const dim3 grid(kRouteBlocks), block(kRouteThreads);
  // (one opt-in per kernel and device: the x share of sixteen tokens and the shared expert's sums pass 48 KB together)
  static PerDeviceOnce once;
  const cudaError_t attr = per_device_once(once, [] {
    constexpr size_t most = size_t(kMaxTok) * kRouteSpan * 4;
    cudaError_t a = opt_in_smem(route_kernel<false, false>, most);
    if (a == cudaSuccess) a = opt_in_smem(route_kernel<true, false>, most);
    if (a == cudaSuccess) a = opt_in_smem(route_kernel<false, true>, most);
    if (a == cudaSuccess) a = opt_in_smem(route_kernel<true, false, true>, most);
    return a;
  });
  if (attr != cudaSuccess) {
    set_error("layer_decode: shared-memory opt-in: %s", cudaGetErrorString(attr));
    return int32_t(attr);
  }
  auto launch = [&](auto kernel) {
    return launch_pdl_cluster(kernel, grid, block, size_t(tokens) * kRouteSpan * 4, as_stream(stream), unsigned(kRouteCluster),
                              static_cast<const __nv_bfloat16*>(router_w_bf16), x, tokens, logits_scratch,
                              int(FB_ROUTER_ROWS), *ws, era, shared ? *shared : SharedRouteArgs{});
  };
  cudaError_t e = ep                       ? launch(route_kernel<false, true>)
                  : shared                 ? launch(route_kernel<true, false, true>)
                  : x_dtype == FB_DT_BF16 ? launch(route_kernel<true, false>)
                                          : launch(route_kernel<false, false>);
  if (e != cudaSuccess) return check_launch("layer_decode: route");
  const SelectArgs sel{logits_scratch, int(FB_ROUTER_ROWS), slot_of, tokens, remote_ok ? 1 : 0, own_combine ? y_out : nullptr};
  const int32_t st = launch_experts(layout, ws, stream, &sel);  // selection + both projections of every routed expert
  if (st || !with_combine || own_combine) return st;
  return fb_moe_combine(ws, nullptr, nullptr, 0, nullptr, nullptr, nullptr, y_out, tokens, 0, nullptr, 0.0f, stream);
}

int32_t fb_moe_layer_decode(const void* router_w_bf16, const fb_moe_expert_layout* layout, const void* x,
                            int32_t x_dtype, int32_t tokens, const fb_moe_decode_workspace* ws, float* logits_scratch,
                            float* y_out, void* stream) {
  return layer_decode_impl(router_w_bf16, layout, nullptr, false, x, x_dtype, tokens, ws, logits_scratch, y_out,
                           stream);
}

int32_t fb_moe_forward_decode(const void* router_w_bf16, const fb_moe_expert_layout* layout, const fb_shared_expert* shared,
                              const void* x_bf16, int32_t tokens, const fb_moe_decode_workspace* ws, float* logits,
                              const float* inj, float* X, float* y_out, void* stream) {
  if (!shared || !shared->gate_up_codes || !shared->gate_up_scales || !shared->down_codes || !shared->down_scales ||
      !shared->h_bf16 || !shared->y || tokens < 1 || tokens > kMaxTok || (X && !inj) || (!X && !y_out))
    return invalid("forward_decode: bad arguments (tokens must be 1..16)");
  if (shared->inter < 128 || shared->inter > kSharedMaxInter || shared->inter % 128)
    return invalid("forward_decode: the shared expert's intermediate size must be a multiple of 128, at most %d", kSharedMaxInter);
  if ((reinterpret_cast<uintptr_t>(shared->gate_up_codes) | reinterpret_cast<uintptr_t>(shared->down_codes) |
       reinterpret_cast<uintptr_t>(shared->h_bf16) | reinterpret_cast<uintptr_t>(x_bf16)) & 15)
    return invalid("forward_decode: x, weight codes and h must be 16-byte aligned");
  const SharedRouteArgs ra{shared->gate_up_codes, shared->gate_up_scales, shared->gate_up_scales_dtype == FB_DT_BF16,
                           shared->inter, static_cast<__nv_bfloat16*>(shared->h_bf16)};
  const int32_t st = layer_decode_impl(router_w_bf16, layout, nullptr, false, x_bf16, FB_DT_BF16, tokens, ws, logits,
                                       nullptr, stream, nullptr, &ra);
  if (st) return st;
  const SharedDownArgs da{shared->down_codes, shared->down_scales, shared->down_scales_dtype == FB_DT_BF16, shared->inter,
                          static_cast<const __nv_bfloat16*>(shared->h_bf16), logits, int(FB_ROUTER_ROWS), shared->y};
  static PerDeviceOnce once;
  const cudaError_t attr =
      per_device_once(once, [] { return opt_in_smem(combine_shared_kernel, size_t(kMaxTok) * kCsMaxK * 4); });
  if (attr != cudaSuccess) {
    set_error("forward_decode: shared-memory opt-in: %s", cudaGetErrorString(attr));
    return int32_t(attr);
  }
  const cudaError_t e = launch_pdl(combine_shared_kernel, dim3(H / kCsCols), dim3(256), size_t(tokens) * shared->inter * 4,
                                   as_stream(stream), *ws, da, tokens, inj, X, y_out);
  if (e != cudaSuccess) return check_launch("forward_decode: combine");
  return 0;
}

int32_t fb_moe_layer_decode_ep(const void* router_w_bf16, const fb_moe_expert_layout* layout,
                               const int32_t* slot_of, const void* x, int32_t x_dtype, int32_t tokens,
                               const fb_moe_decode_workspace* ws, float* logits_scratch, float* y_partial,
                               void* stream) {
  if (!slot_of) return invalid("layer_decode_ep: slot_of (expert -> local slot, -1 = another rank) is required");
  return layer_decode_impl(router_w_bf16, layout, slot_of, true, x, x_dtype, tokens, ws, logits_scratch, y_partial,
                           stream);
}

int32_t fb_moe_layer_decode_ep_p2p(const void* router_w_bf16, const fb_moe_expert_layout* layout,
                                   const int32_t* slot_of, const float* x_local, int32_t tokens,
                                   const fb_ep_peers* peers, uint32_t step, const fb_moe_decode_workspace* ws,
                                   float* logits_scratch, float* y_local, void* stream) {
  if (!slot_of || !x_local || !y_local || !peers || peers->n_ranks < 1 || peers->n_ranks > kEpMaxRanks ||
      peers->rank < 0 || peers->rank >= peers->n_ranks || tokens < peers->n_ranks || tokens > kMaxTok ||
      tokens % peers->n_ranks || step == 0)
    return invalid("layer_decode_ep_p2p: bad arguments (tokens a multiple of the rank count, at most 16; step >= 1)");
  // the route kernel hands its blocks out to the ranks in equal shares
  if (kRouteBlocks % peers->n_ranks)
    return invalid("layer_decode_ep_p2p: the rank count must be 1, 2, 4 or 8");
  for (int d = 0; d < peers->n_ranks; ++d)
    if (!peers->x_all[d] || !peers->y_parts[d])
      return invalid("layer_decode_ep_p2p: a peer buffer address is missing");
  const int R = peers->n_ranks, tpr = tokens / R, parity = int(step & 1u);
  cudaStream_t s = as_stream(stream);
  // Three launches, chained like the single-GPU layer: route (publishes this rank's rows, waits for everyone's), experts
  // (selection, gate/up, down; IQ3_S down behind another gate/up format: two), combine (sends partial rows, waits, sums).
  EpRouteArgs era{};
  era.peers = *peers;
  era.x_local = x_local;
  era.tpr = tpr;
  era.parity = parity;
  era.step = step;
  era.spin_limit = g_peer_wait_polls;
  // (the route kernel reads every x row through the exchange lines; x_local only satisfies the argument check)
  int32_t st = layer_decode_impl(router_w_bf16, layout, slot_of, true, x_local, FB_DT_F32, tokens, ws, logits_scratch,
                                 nullptr, stream, &era);
  if (st) return st;
  const cudaError_t e = launch_pdl(ep_combine_exchange_kernel, dim3(H / 512, tokens), dim3(256), 0, s, *ws, *peers, tpr,
                                   parity, step, g_peer_wait_polls, y_local);
  if (e != cudaSuccess) return check_launch("layer_decode_ep_p2p: combine");
  return check_launch("layer_decode_ep_p2p");
}

// Exchange buffers of fb_moe_layer_decode_ep_p2p. They are allocated here (cudaMalloc, so a CUDA IPC
// handle names exactly the buffer) and opened by the peers in the context of THEIR OWN device with
// lazy peer access, the way collective libraries map each other's memory.
constexpr size_t kEpBytes[2] = {size_t(2) * kMaxTok * (H / 2) * 16, size_t(2) * kEpMaxRanks * kMaxTok * (H / 2) * 16};

int32_t fb_ep_exchange_create(void** x_all, void** y_parts, uint8_t* handles) {
  if (!x_all || !y_parts || !handles) return invalid("ep_exchange_create: NULL argument");
  static_assert(sizeof(cudaIpcMemHandle_t) == FB_EP_HANDLE_BYTES, "handle size");
  void** out[2] = {x_all, y_parts};
  for (int k = 0; k < 2; ++k) {
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, kEpBytes[k]);
    if (e == cudaSuccess) e = cudaMemset(p, 0, kEpBytes[k]);
    cudaIpcMemHandle_t h;
    if (e == cudaSuccess) e = cudaIpcGetMemHandle(&h, p);
    if (e != cudaSuccess) {
      cudaGetLastError();
      set_error("ep_exchange_create: %s", cudaGetErrorString(e));
      return int32_t(e);
    }
    memcpy(handles + k * FB_EP_HANDLE_BYTES, &h, FB_EP_HANDLE_BYTES);
    *out[k] = p;
  }
  return int32_t(cudaDeviceSynchronize());
}

int32_t fb_ep_exchange_open(const uint8_t* handles, void** x_all, void** y_parts) {
  if (!x_all || !y_parts || !handles) return invalid("ep_exchange_open: NULL argument");
  void** out[2] = {x_all, y_parts};
  for (int k = 0; k < 2; ++k) {
    cudaIpcMemHandle_t h;
    memcpy(&h, handles + k * FB_EP_HANDLE_BYTES, FB_EP_HANDLE_BYTES);
    void* p = nullptr;
    const cudaError_t e = cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess);
    if (e != cudaSuccess) {
      cudaGetLastError();
      set_error("ep_exchange_open: %s", cudaGetErrorString(e));
      return int32_t(e);
    }
    *out[k] = p;
  }
  return 0;
}

int32_t fb_ep_exchange_close(void* x_all, void* y_parts, int32_t own) {
  void* p[2] = {x_all, y_parts};
  int32_t st = 0;
  for (int k = 0; k < 2; ++k) {
    if (!p[k]) continue;
    const cudaError_t e = own ? cudaFree(p[k]) : cudaIpcCloseMemHandle(p[k]);
    if (e != cudaSuccess) {
      cudaGetLastError();
      st = int32_t(e);
    }
  }
  return st;
}

void fb_ep_set_wait_limit(uint32_t polls) { g_peer_wait_polls = polls ? polls : kPeerSpinLimit; }

size_t fb_ep_exchange_bytes(int32_t which) { return which == 0 ? kEpBytes[0] : which == 1 ? kEpBytes[1] : 0; }

int32_t fb_ep_sum_ranks(const float* parts, int32_t n_ranks, int32_t rows, float* y, void* stream) {
  if (!parts || !y || n_ranks < 1 || rows < 1) return invalid("ep_sum_ranks: bad arguments");
  const int64_t elems = int64_t(rows) * H;
  sum_ranks_kernel<<<unsigned((elems + 255) / 256), 256, 0, as_stream(stream)>>>(parts, n_ranks, elems, y);
  return check_launch("ep_sum_ranks");
}

int32_t fb_moe_layer_decode_host(const void* router_w_bf16, const fb_moe_expert_layout* layout, const void* x_host,
                                 int32_t x_dtype, int32_t tokens, const fb_moe_decode_workspace* ws,
                                 float* logits_scratch, void* x_dev, float* y_dev, float* y_host, void* stream) {
  if (!x_host || !x_dev || !y_dev || !y_host || tokens < 1 || tokens > kMaxTok)
    return invalid("layer_decode_host: bad arguments");
  const size_t xb = size_t(tokens) * H * (x_dtype == FB_DT_BF16 ? 2 : 4);
  // Pinned buffers are read and written by kernels (page-locked host memory has a device address under unified
  // addressing): two copy operations and their launches less per call (eight calls of four tokens with x as a copy operation
  // 423, so 415 us). Pageable memory, buffers that are page-locked in part only, and x off 16 bytes take the copies.
  const void* x_pinned = pinned_on_device(x_host, xb);
  cudaError_t e;
  if (x_pinned && ((reinterpret_cast<uintptr_t>(x_pinned) | reinterpret_cast<uintptr_t>(x_dev)) & 15) == 0) {
    const int n = int(xb / 16);
    e = launch_pdl(copy_in_kernel, dim3((n + 255) / 256), dim3(256), 0, as_stream(stream),
                   static_cast<const uint4*>(x_pinned), static_cast<uint4*>(x_dev), n);
  } else {
    e = cudaMemcpyAsync(x_dev, x_host, xb, cudaMemcpyHostToDevice, as_stream(stream));
  }
  if (e != cudaSuccess) return check_launch("layer_decode_host: copy in");
  float* y_pinned = static_cast<float*>(pinned_on_device(y_host, size_t(tokens) * H * 4));
  const bool direct = y_pinned != nullptr;
  float* y_target = direct ? y_pinned : y_dev;
  int32_t st = fb_moe_layer_decode(router_w_bf16, layout, x_dev, x_dtype, tokens, ws, logits_scratch, y_target, stream);
  if (st) return st;
  if (!direct) {
    e = cudaMemcpyAsync(y_host, y_dev, size_t(tokens) * H * 4, cudaMemcpyDeviceToHost, as_stream(stream));
    if (e != cudaSuccess) return check_launch("layer_decode_host: copy out");
  }
  e = cudaStreamSynchronize(as_stream(stream));
  if (e != cudaSuccess) {
    set_error("layer_decode_host: %s", cudaGetErrorString(e));
    return int32_t(e);
  }
  return 0;
}


// ---------------------------------------------------------------------------------------------
// fb_moe_layer_decode_static: the whole decode layer without any caller-provided scratch.
//
// Some hosts of this library may not allocate device memory at the point where they run a layer:
// an engine whose memory plan is frozen after start-up (every byte of HBM already handed to
// weights and KV cache), a plug-in that is only given tensor pointers, or code running where a
// cudaMalloc would serialize the device. For them the layer's scratch - work list, quantized
// activations, h, partial sums, router logits - lives in one array inside the library image.
// Every GPU that loads the library carries these kStaticScratchBytes until the process exits.
//
// The array's name is only a host-side handle; its device address comes from
// cudaGetSymbolAddress, taken once per device on that device's first call (so make that first
// call outside any stream capture). All calls on a device share the array and it keeps the last
// call's contents: the entry point clears the one word that must start at zero, and two calls
// that overlap on the same GPU (different streams) race on it - serialize them.
// fb_moe_layer_decode_static_status reads the status word of the last call back to the host (a
// stream-ordered copy out of the array and a wait on that stream; it allocates nothing either).
namespace {
constexpr size_t kStaticWorkspaceBytes = 2304 * 1024;  // >= fb_moe_decode_workspace_bytes(640), checked at set-up
constexpr size_t kStaticLogitsBytes = size_t(FB_DECODE_MAX_TOKENS) * FB_ROUTER_ROWS * 4;
constexpr size_t kStaticScratchBytes = kStaticWorkspaceBytes + ((kStaticLogitsBytes + 255) & ~size_t(255));
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

struct StaticScratch {
  bool ready = false;
  unsigned char* base = nullptr;
  uint32_t* status = nullptr;  // the workspace's status word inside the array (set by the first layer call)
};
StaticScratch g_static[64];
}  // namespace

int32_t fb_moe_layer_decode_static(const void* router_w_bf16, const fb_moe_expert_layout* layout, const void* x,
                                   int32_t x_dtype, int32_t tokens, float* y_out, void* stream) {
  if (tokens < 1 || tokens > kMaxTok)
    return invalid("layer_decode_static: tokens must be 1..%d (the static scratch is sized for that)", kMaxTok);
  if (!layout_ok(layout)) return invalid("layer_decode_static: unsupported expert layout");
  if (fb_moe_decode_workspace_bytes(layout->inter) > kStaticWorkspaceBytes)
    return invalid("layer_decode_static: layout needs more scratch than the %zu static bytes", kStaticWorkspaceBytes);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    set_error("layer_decode_static: cudaGetDevice: %s", cudaGetErrorString(e));
    return e != cudaSuccess ? int32_t(e) : int32_t(cudaErrorInvalidDevice);
  }
  StaticScratch& sc = g_static[dev];
  if (!sc.ready) {  // first call on this device: resolve the array's device address
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || !p) {
      set_error("layer_decode_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      return e != cudaSuccess ? int32_t(e) : int32_t(cudaErrorInvalidSymbol);
    }
    sc.base = static_cast<unsigned char*>(p);
    sc.ready = true;
  }
  fb_moe_decode_workspace ws;
  int32_t st = fb_moe_decode_workspace_make(sc.base, layout, &ws);
  if (st) return st;
  sc.status = ws.status;
  float* logits = reinterpret_cast<float*>(sc.base + kStaticWorkspaceBytes);
  // the sticky status word and the scheduler words (tile counters) are the only state a call inherits
  e = cudaMemsetAsync(ws.status, 0, sizeof(uint32_t), as_stream(stream));
  if (e == cudaSuccess) e = cudaMemsetAsync(ws.sched, 0, kSchedInts * sizeof(int32_t), as_stream(stream));
  if (e != cudaSuccess) {
    set_error("layer_decode_static: clearing scratch state: %s", cudaGetErrorString(e));
    return int32_t(e);
  }
  return fb_moe_layer_decode(router_w_bf16, layout, x, x_dtype, tokens, &ws, logits, y_out, stream);
}

int32_t fb_moe_layer_decode_static_status(uint32_t* status_host, void* stream) {
  if (!status_host) return invalid("layer_decode_static_status: status_host is NULL");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64 || !g_static[dev].status)
    return invalid("layer_decode_static_status: fb_moe_layer_decode_static has not run on this device");
  e = cudaMemcpyAsync(status_host, g_static[dev].status, sizeof(uint32_t), cudaMemcpyDeviceToHost, as_stream(stream));
  if (e == cudaSuccess) e = cudaStreamSynchronize(as_stream(stream));
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_error("layer_decode_static_status: %s", cudaGetErrorString(e));
    return int32_t(e);
  }
  return 0;
}

}  // extern "C"
