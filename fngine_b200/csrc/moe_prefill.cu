// Prefill-width routed experts: route -> grouped gate/up -> grouped down -> combine.
//
// Numerics are the reference's prefill family (src/kernels/moe/moe.h:32-35 and the CPU pool's
// prefill mode, src/cpu/iq_cpu.h:93-99): weights dequantized exactly and rounded to bf16, bf16
// activations, fp32 accumulation, h stored as bf16.
//
// Both grouped GEMMs run on tcgen05 (kind::f16, bf16 x bf16 -> fp32 in tensor memory) with the
// WEIGHT rows on the 128 TMEM lanes and the expert's TOKENS on the N axis (a multiple of 16, up to
// 256), so ragged per-expert token counts waste at most 15 columns:
//   D[128 weight rows][tokens] += W_bf16[128][64] * X[tokens][64]^T        per 64-wide K step.
// The A operand exists in tensor memory only: decoding warps write it there from registers
// (moe_prefill_grouped.cuh).
#include "iq_decode.cuh"

#include <cuda.h>
#include <cuda_bf16.h>

#include <type_traits>

namespace fb {
namespace {

constexpr int H = FB_HIDDEN;
constexpr int kExperts = FB_EXPERTS;
constexpr int kTopK = FB_TOPK;
constexpr int kBK = 64;          // K elements per pipeline stage = one 128-byte swizzled row
constexpr int kTileM = 128;      // weight rows per unit (TMEM lanes)
constexpr int kTileN = 256;      // tokens per gate/up unit
constexpr int kTileNDown = 128;  // tokens per down unit
constexpr int kTileB = kTileN * 128;  // 32 KB

// ------------------------------------------------------------------------------ PTX (tcgen05 / TMA / cp.async)
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Shared-memory operand descriptors are given by their low words (the high word is the same for every tile, see
// umma_desc_lo_k128): the issuing lane steps through a stage's K slices with 32-bit adds.
constexpr uint32_t kDescHiK128 = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// One arrival on `bar` (already counted in its expected arrivals) once every cp.async this thread has issued so far
// is complete.
__device__ __forceinline__ void cp_async_arrive_noinc(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Shared-memory operand descriptor of a K-major bf16 tile, rows of 128 bytes, 128-byte swizzle, 8-row groups 1024
// bytes apart: low word = address / 16 | leading offset 1 << 16, high word (kDescHiK128) = stride 1024 / 16 |
// descriptor version 1 << 14 | swizzle mode 2 << 29.
__device__ __forceinline__ uint32_t umma_desc_lo_k128(uint32_t smem_addr) {
  return ((smem_addr & 0x3FFFFu) >> 4) | (1u << 16);
}
static_assert((uint64_t(kDescHiK128) << 32) == ((uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61)),
              "descriptor high word");
// D fp32, A and B bf16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(kTileM >> 4) << 24);
}
struct Abort {
  volatile int* flag;
  uint32_t* status;
  __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) const {
    // The first probe of a barrier does not wait (a try with a time limit takes longer even when the phase is complete).
    // Each later one may sleep in the instruction for about a microsecond: two dozen waiting warps share the issue slots
    // with the decoding ones.
    if (mbar_test_wait(bar, parity)) return true;
    for (uint32_t i = 0; i < (1u << 21); ++i) {
      if (mbar_try_wait_hint(bar, parity)) return true;
      if ((i & 31u) == 31u && *flag) return false;  // another role gave up: fall through every later wait
    }
    *flag = 1;
    atomicMax(status, uint32_t(FB_STATUS_PIPELINE_TIMEOUT));
    return false;
  }
  // The same for a whole warp. All lanes try: a lane that polls for the others (a branch, then a shuffle) made a wait on a
  // barrier that is ready cost some 400 cycles (gate/up of 96 IQ3_S tokens 278 us, 253 so); all decisions are the warp's.
  __device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity) const {
    if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
    for (uint32_t i = 0; i < (1u << 21); ++i) {
      if (__all_sync(0xffffffffu, mbar_try_wait_hint(bar, parity))) return true;
      if ((i & 31u) == 31u && __any_sync(0xffffffffu, *flag != 0)) return false;
    }
    *flag = 1;
    if ((threadIdx.x & 31) == 0) atomicMax(status, uint32_t(FB_STATUS_PIPELINE_TIMEOUT));
    return false;
  }
};

// ------------------------------------------------------------------------------ shared-memory access, packing
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Shared-memory accesses by 32-bit window address with a compile-time offset: one instruction
// each, no 64-bit pointer arithmetic.
template <int OFF>
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFF) : "memory");
  return v;
}
template <int OFF>
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
  uint32_t v;
  asm volatile("{\n\t.reg .b16 t;\n\tld.shared.u16 t, [%1+%2];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(a), "n"(OFF) : "memory");
  return v;
}
template <int OFF>
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0+%1], %2;" ::"r"(a), "n"(OFF), "r"(v) : "memory");
}

// ------------------------------------------------------------------------------ route
// The path's launches are chained by programmatic dependent launch: a kernel's blocks start, and the grouped kernels build
// their tables and barriers, while the one before runs out. Every kernel waits for its predecessor before it touches
// global memory (so all earlier ones are complete too), and data of a predecessor is never read through const __restrict__
// pointers, which would allow the load ahead of the wait. Layers of 96 IQ4_NL
// tokens 373 -> 355 us, of 50 tokens at 640 268 -> 248.
// From kBlockNumbers tokens on, pairs are counted and numbered in one pass by blocks: a block counts its pairs in shared memory
// (the count a pair finds is its number within the block), adds the sums to the expert's count once, and the value it meets
// there plus the block's number is the pair's number within its expert, left in token_pair for the scatter kernel. (One atomic
// per pair, in two kernels, met a popular expert's counter 4000 times at 8192 tokens: the route call 41 us, 20.5 so.) With fewer
// tokens the blocks' clearing and adding costs more than it saves: the route call takes every pair's number from the expert's
// count itself (us, by blocks / so: 1 token 10.3 / 9.2, 64 11.3 / 10.4, 400 11.4 / 10.5, 1000 level, zipf-distributed experts at 1500 12.4 /
// 13.2), the one for dispatched rows counts first and numbers in the scatter kernel (100 rows 10.3 / 8.3, 300 10.3 / 8.4,
// 1000 level, 2048 10.4 / 12.4).
constexpr int kBlockNumbers = 1000;
struct PairNumbers {
  int count[kExperts];  // pairs of the block, then the pairs of blocks before it
  __device__ __forceinline__ void clear(int threads) {
    for (int e = threadIdx.x; e < kExperts; e += threads) count[e] = 0;
  }
  __device__ __forceinline__ int add(int e) { return atomicAdd(&count[e], 1); }
  __device__ __forceinline__ void publish(int32_t* total, int threads) {
    for (int e = threadIdx.x; e < kExperts; e += threads) {
      const int c = count[e];
      if (c) count[e] = atomicAdd(&total[e], c);
    }
  }
};

// Top-10 per token (one warp each, PER_WARP in turn), per-expert pair counts and the pairs' numbers (token_pair, may be absent;
// BLOCKS: by blocks).
// PER_WARP 4 from 4096 tokens on: fewer meetings on a popular expert's counter; below that single tokens fill the GPU.
// The routing launches of 8192 tokens together: 45 us, 25 so (selection by the pruned search and numbering).
template <int PER_WARP, bool BLOCKS>
__global__ void __launch_bounds__(256) pf_topk_kernel(const float* logits, int stride, int T, int32_t* topk_e, float* topk_w,
                                                      int32_t* count, int32_t* token_pair) {
  __shared__ PairNumbers s_num;  // (BLOCKS only)
  __shared__ __align__(16) uint2 s_scratch[8][32];
  __shared__ int s_ids[8][kTopK];
  __shared__ float s_vals[8][kTopK];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t0 = (blockIdx.x * 8 + warp) * PER_WARP;
  if (BLOCKS) {
    s_num.clear(256);
    __syncthreads();
  }
  pdl_wait_prior();
  int id[PER_WARP], number[PER_WARP];
#pragma unroll
  for (int i = 0; i < PER_WARP; ++i) {
    const int t = t0 + i;
    if (t >= T) break;
    warp_top10_pruned<true>([&](int e) { return logits[size_t(t) * stride + e]; }, s_scratch[warp], s_ids[warp], s_vals[warp]);
    __syncwarp();
    float vals[kTopK], w[kTopK];
#pragma unroll
    for (int k = 0; k < kTopK; ++k) vals[k] = s_vals[warp][k];
    topk_softmax(vals, w);
    if (lane < kTopK) {
      id[i] = s_ids[warp][lane];
      float wt = 0.0f;
#pragma unroll
      for (int k = 0; k < kTopK; ++k)
        if (lane == k) wt = w[k];
      topk_e[t * kTopK + lane] = id[i];
      topk_w[t * kTopK + lane] = wt;
      if constexpr (BLOCKS) number[i] = s_num.add(id[i]);
      else if (token_pair) token_pair[t * kTopK + lane] = atomicAdd(&count[id[i]], 1);
    }
    __syncwarp();
  }
  if constexpr (!BLOCKS) return;
  __syncthreads();
  s_num.publish(count, 256);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PER_WARP; ++i)
    if (t0 + i < T && lane < kTopK) token_pair[(t0 + i) * kTopK + lane] = s_num.count[id[i]] + number[i];
}

// Expert-parallel routing: the (expert, weight) lists arrive with the dispatched rows; entries of
// experts other ranks own ([lo, hi) is this rank's range) become -1 and take no part. With a share
// table (placement with copies) the rule is per expert instead: share[e] < 0 = not held here, else
// (n << 8) | i = this rank holds copy i of n and takes the rows r with r % n == i.
template <bool BLOCKS>
__global__ void __launch_bounds__(256) pf_import_kernel(const int32_t* in_e, const float* in_w, int lo, int hi,
                                                        const int32_t* share, int n, int32_t* topk_e, float* topk_w,
                                                        int32_t* count, int32_t* token_pair) {
  __shared__ PairNumbers s_num;  // (BLOCKS only)
  pdl_launch_dependents();
  if constexpr (BLOCKS) {
    s_num.clear(256);
    __syncthreads();
  }
  pdl_wait_prior();
  const int i = blockIdx.x * 256 + threadIdx.x;
  int e = -1, number = 0;
  if (i < n) {
    e = in_e[i];
    bool local = e >= lo && e < hi;
    if (share) {
      const int sh = e >= 0 && e < kExperts ? share[e] : -1;
      local = sh >= 0 && (i / kTopK) % max(sh >> 8, 1) == (sh & 255);
    }
    if (!local) e = -1;
    topk_e[i] = e;
    topk_w[i] = in_w[i];
    if constexpr (BLOCKS) {
      if (local) number = s_num.add(e);
    } else {
      if (local) atomicAdd(&count[e], 1);
    }
  }
  if constexpr (!BLOCKS) return;
  __syncthreads();
  s_num.publish(count, 256);
  __syncthreads();
  if (e >= 0) token_pair[i] = s_num.count[e] + number;
}

// Exclusive scan of the counts and the token-tile lists of both grouped GEMMs (one block of 512): tile = {expert, 0,
// first pair, tokens}; a tile stands for inter / 128 (down: 2560 / 128) units of 128 weight rows, which the GEMM kernel
// counts out itself. (Lists of units cost this single block 17 us at 8192 tokens.)
// Tiles are listed by token count, most first (in steps of sixteen; a bucket's order is whatever the atomics give, results
// do not depend on it): the GEMM's blocks take units in turn, and with tiles in expert order, a block's share of some forty
// units of unequal cost was up to a sixth above the mean.
constexpr int kTileBuckets = kTileN / 16;
template <int TILE>
__device__ __forceinline__ void list_tiles(int expert, int first_pair, int count, int* s_cursor, int4* tiles,
                                           int max_tiles) {
  const int full = count / TILE, rest = count - full * TILE;
  if (full) {
    const int at = atomicAdd(&s_cursor[0], full);
    for (int t = 0; t < full; ++t)
      if (at + t < max_tiles) tiles[at + t] = make_int4(expert, 0, first_pair + t * TILE, TILE);
  }
  if (rest) {
    const int at = atomicAdd(&s_cursor[(TILE - rest) / 16], 1);
    if (at < max_tiles) tiles[at] = make_int4(expert, 0, first_pair + full * TILE, rest);
  }
}
__global__ void __launch_bounds__(512) pf_scan_kernel(const int32_t* count, int32_t* offset, int32_t* cursor, int4* tiles_gu,
                                                      int4* tiles_dn, int32_t* meta, int inter, int max_units_gu,
                                                      int max_units_dn) {
  pdl_launch_dependents();
  pdl_wait_prior();
  __shared__ int s_scan[16];
  __shared__ int s_bucket[2][kTileBuckets], s_cursor[2][kTileBuckets];  // bucket b: TILE - 16 b - 15 .. TILE - 16 b tokens
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 2 * kTileBuckets) (&s_bucket[0][0])[tid] = 0;
  const int c = count[tid];
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += a;
  }
  if (lane == 31) s_scan[warp] = incl;
  __syncthreads();
  auto tally = [&](int tile, int* bucket) {
    const int full = c / tile, rest = c - full * tile;
    if (full) atomicAdd(&bucket[0], full);
    if (rest) atomicAdd(&bucket[(tile - rest) / 16], 1);
  };
  tally(kTileN, s_bucket[0]);
  tally(kTileNDown, s_bucket[1]);
  int first = incl - c, total = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    first += i < warp ? s_scan[i] : 0;
    total += s_scan[i];
  }
  offset[tid] = first;
  cursor[tid] = 0;
  __syncthreads();
  const int mg = inter / kTileM, md = H / kTileM;
  if (warp < 2) {  // warp k: list k
    const int n = lane < kTileBuckets ? s_bucket[warp][lane] : 0;
    int upto = n;
#pragma unroll
    for (int o = 1; o < kTileBuckets; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += a;
    }
    if (lane < kTileBuckets) s_cursor[warp][lane] = upto - n;
    if (lane == kTileBuckets - 1) meta[warp] = min(upto * (warp ? md : mg), warp ? max_units_dn : max_units_gu);
  }
  if (tid == 0) {
    offset[kExperts] = total;
    meta[2] = total;
  }
  __syncthreads();
  list_tiles<kTileN>(tid, first, c, s_cursor[0], tiles_gu, max_units_gu / mg);
  list_tiles<kTileNDown>(tid, first, c, s_cursor[1], tiles_dn, max_units_dn / md);
}

// Pairs grouped by expert, a pair's place being its number within the expert (from token_pair; CURSOR: taken here). The numbers depend on the atomics, the results do
// not: every pair's h and y rows depend only on (token, expert) and the combine adds a token's ten rows in ascending-expert
// order.
template <bool CURSOR>
__global__ void __launch_bounds__(256) pf_scatter_kernel(const int32_t* topk_e, const float* topk_w, const int32_t* offset,
                                                         int32_t* cursor, int32_t* pair_token, float* pair_weight, int32_t* token_pair, int T) {
  pdl_launch_dependents();
  pdl_wait_prior();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= T * kTopK) return;
  const int e = topk_e[i];
  if (e < 0) {  // an expert of another rank
    token_pair[i] = -1;
    return;
  }
  const int pos = offset[e] + (CURSOR ? atomicAdd(&cursor[e], 1) : token_pair[i]);
  pair_token[pos] = i / kTopK;
  pair_weight[pos] = topk_w[i];
  token_pair[i] = pos;
}

// Owner-side sum of an expert-parallel step: y[t] = sum over source ranks d, in rank order, of the
// partial row that rank d returned for token t (row_of[t][d] = its row in `recv`, -1 if rank d held
// none of the token's experts).
__global__ void __launch_bounds__(256) ep_scatter_sum_kernel(const float* __restrict__ recv,
                                                             const int32_t* __restrict__ row_of, int n_ranks,
                                                             float* __restrict__ y) {
  const int t = blockIdx.y, n = blockIdx.x * 256 + threadIdx.x;
  float acc = 0.0f;
  for (int d = 0; d < n_ranks; ++d) {
    const int r = row_of[t * n_ranks + d];
    if (r >= 0) acc += recv[size_t(r) * H + n];
  }
  y[size_t(t) * H + n] = acc;
}

#include "moe_prefill_grouped.cuh"

// ------------------------------------------------------------------------------ combine
// y[t][n] = sum over token t's ten pairs, in ascending expert id, of yp[pair][n] (+ shared);
// X[t][s][n] += inj[t][s] * y when X is given. Bound: the ten rows per token from memory. Four blocks per token, thread = four
// columns, all ten 16-byte loads in flight. (8192 tokens: 147 us, 0.97 of the copy rate. One block of 640 threads per token
// took 210: with its registers two of them share a multiprocessor, and while one orders its pairs only the other one loads.
// Two blocks of 320: 150; blocks of 640 that stay and fetch the next token's pairs ahead: 151.)
constexpr int kPcParts = 4, kPcThreads = H / 4 / kPcParts;  // 160
template <bool ALIGNED>  // y_shared, X and y_out on 16-byte boundaries (single words otherwise)
__device__ __forceinline__ float4 load4(const float* p) {
  if constexpr (ALIGNED) return *reinterpret_cast<const float4*>(p);
  else return make_float4(p[0], p[1], p[2], p[3]);
}
template <bool ALIGNED>
__device__ __forceinline__ void store4(float* p, const float4& v) {
  if constexpr (ALIGNED) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
    p[3] = v.w;
  }
}
template <bool ALIGNED>
__global__ void __launch_bounds__(kPcThreads) pf_combine_kernel(const int32_t* topk_e, const int32_t* token_pair, const float* yp,
                                                                const float* y_shared, const float* inj, float* X,
                                                                float* y_out, const long long* y_fixed) {
  pdl_launch_dependents();
  pdl_wait_prior();
  const int t = blockIdx.x / kPcParts, n4 = (blockIdx.x % kPcParts) * kPcThreads + threadIdx.x, lane = threadIdx.x & 31;
  float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (y_fixed) {  // fixed-point sums: one rounding, the scale is exact (moe_y_fixed_to_float of the reference)
    const longlong2* f = reinterpret_cast<const longlong2*>(y_fixed + size_t(t) * H) + 2 * n4;
    const longlong2 a = f[0], b = f[1];
    constexpr float kScale = 1.0f / 4294967296.0f;
    y = make_float4(float(a.x) * kScale, float(a.y) * kScale, float(b.x) * kScale, float(b.y) * kScale);
  } else {
    // Every warp orders the token's pairs by expert id (lane = list entry; the ids are distinct); entries without a local
    // pair (expert-parallel shards) sort last.
    int e = 0x7fffffff, pair = -1;
    if (lane < kTopK) {
      e = topk_e[t * kTopK + lane];
      pair = token_pair[t * kTopK + lane];
      if (e < 0) e = kExperts + lane;
    }
    int rank = 0;
#pragma unroll
    for (int k = 0; k < kTopK; ++k) rank += __shfl_sync(0xffffffffu, e, k) < e ? 1 : 0;
    int row[kTopK];
    float4 v[kTopK];
#pragma unroll
    for (int k = 0; k < kTopK; ++k) {
      const uint32_t who = __ballot_sync(0xffffffffu, lane < kTopK && rank == k);
      row[k] = __shfl_sync(0xffffffffu, pair, __ffs(who) - 1);
    }
#pragma unroll
    for (int k = 0; k < kTopK; ++k)
      if (row[k] >= 0) v[k] = __ldcs(reinterpret_cast<const float4*>(yp + size_t(row[k]) * H) + n4);
#pragma unroll
    for (int k = 0; k < kTopK; ++k)
      if (row[k] >= 0) {
        y.x += v[k].x;
        y.y += v[k].y;
        y.z += v[k].z;
        y.w += v[k].w;
      }
  }
  if (y_shared) {
    const float4 s = load4<ALIGNED>(y_shared + size_t(t) * H + 4 * n4);
    y.x += s.x;
    y.y += s.y;
    y.z += s.z;
    y.w += s.w;
  }
  if (y_out) store4<ALIGNED>(y_out + size_t(t) * H + 4 * n4, y);
  if (X) {
    float4 x[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) x[s] = load4<ALIGNED>(X + (size_t(t) * 4 + s) * H + 4 * n4);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float g = inj[t * 4 + s];
      x[s].x += g * y.x;
      x[s].y += g * y.y;
      x[s].z += g * y.z;
      x[s].w += g * y.w;
      store4<ALIGNED>(X + (size_t(t) * 4 + s) * H + 4 * n4, x[s]);
    }
  }
}

// ------------------------------------------------------------------------------ host
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// Rows of pairs as a bf16 tensor [K steps][pairs][64], 128-byte swizzle; a box that reaches behind the last pair or the last
// K step reads the zero fill.
int32_t rows_maps(GgMaps* maps, void* rows, int width, int capacity, const char* what) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) {
    set_error("%s: cuTensorMapEncodeTiled is not available", what);
    return int32_t(cudaErrorNotSupported);
  }
  static const cuuint32_t boxes[kBoxes][2] = {{32, 1}, {64, 1}, {128, 1}, {32, 8}, {64, 4}};
  const cuuint64_t dims[3] = {cuuint64_t(kBK), cuuint64_t(size_t(capacity) * kTopK), cuuint64_t(width / kBK)};
  const cuuint64_t strides[2] = {cuuint64_t(width) * 2, cuuint64_t(kBK) * 2};
  const cuuint32_t elem[3] = {1, 1, 1};
  for (int i = 0; i < kBoxes; ++i) {
    const cuuint32_t box[3] = {cuuint32_t(kBK), boxes[i][0], boxes[i][1]};
    if (fn(&maps->m[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, rows, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
      set_error("%s: cuTensorMapEncodeTiled failed", what);
      return int32_t(cudaErrorInvalidValue);
    }
  }
  return 0;
}

template <int FMT, bool DOWN>
cudaError_t launch_grouped(const GgArgs& a, const GgMaps& maps, cudaStream_t stream) {
  static PerDeviceOnce once;
  const cudaError_t e = per_device_once(once, [] { return opt_in_smem(grouped_kernel<FMT, DOWN>, gg_smem<FMT, DOWN>()); });
  if (e != cudaSuccess) return e;
  return launch_pdl(grouped_kernel<FMT, DOWN>, dim3(sm_count()), dim3(kGgThreads), size_t(gg_smem<FMT, DOWN>()), stream, a, maps);
}

// Offsets, token tiles and pair lists from the counts and the top-10 entries of `rows` tokens.
cudaError_t launch_pair_lists(const fb_moe_prefill_workspace* ws, int rows, bool numbered, cudaStream_t s) {
  const cudaError_t e = launch_pdl(pf_scan_kernel, dim3(1), dim3(512), 0, s, ws->expert_count, ws->expert_offset, ws->expert_cursor,
                                   static_cast<int4*>(ws->units_gate_up), static_cast<int4*>(ws->units_down),
                                   ws->meta, ws->inter, ws->max_units_gate_up, ws->max_units_down);
  if (e != cudaSuccess) return e;
  return launch_pdl(numbered ? pf_scatter_kernel<false> : pf_scatter_kernel<true>, dim3((rows * kTopK + 255) / 256), dim3(256), 0, s,
                    ws->topk_expert, ws->topk_weight, ws->expert_offset, ws->expert_cursor, ws->pair_token, ws->pair_weight, ws->token_pair, rows);
}

size_t up256(size_t v) { return (v + 255) & ~size_t(255); }
// Token tiles that `capacity` tokens can make: every expert's last tile may be short.
int max_tiles(int capacity, int tile_tokens) {
  return int(int64_t(capacity) * kTopK / tile_tokens) + kExperts;
}

struct PfLayout {
  size_t meta, count, offset, cursor, topk_e, topk_w, pair_token, pair_weight, token_pair, units_gu, units_dn, h, yp,
      status, total;
};
PfLayout pf_layout(int capacity, int inter) {
  PfLayout l;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = up256(o + bytes);
    return at;
  };
  const size_t pairs = size_t(capacity) * kTopK;
  l.meta = take(64);
  l.count = take(kExperts * 4);
  l.offset = take((kExperts + 1) * 4);
  l.cursor = take(kExperts * 4);
  l.topk_e = take(pairs * 4);
  l.topk_w = take(pairs * 4);
  l.pair_token = take(pairs * 4);
  l.pair_weight = take(pairs * 4);
  l.token_pair = take(pairs * 4);
  l.units_gu = take(size_t(max_tiles(capacity, kTileN)) * 16);
  l.units_dn = take(size_t(max_tiles(capacity, kTileNDown)) * 16);
  l.h = take((pairs + kTileN) * size_t(inter) * 2);  // + one tile so a TMA box never leaves the buffer
  l.yp = take(pairs * size_t(H) * 4);
  l.status = take(64);
  l.total = o;
  return l;
}

bool pf_layout_ok(const fb_moe_expert_layout* L, const void* table) {
  if (!L || (!L->slots && !table)) return false;
  if ((uintptr_t(L->blob_stride) | uintptr_t(L->gate_offset) | uintptr_t(L->up_offset) | uintptr_t(L->down_offset)) & 1)
    return false;
  if (L->inter != 512 && L->inter != 640) return false;
  if (L->gate_up_format != FB_FMT_IQ3_S && L->gate_up_format != FB_FMT_IQ4_NL) return false;
  if (L->down_format == FB_FMT_IQ3_S) return L->inter % 256 == 0;
  return L->down_format == FB_FMT_IQ4_NL;
}

bool pf_ws_ok(const fb_moe_prefill_workspace* ws, int tokens) {
  return ws && ws->meta && ws->h && ws->yp && ws->units_gate_up && ws->units_down && tokens >= 1 &&
         tokens <= ws->capacity;
}

}  // namespace
}  // namespace fb

using namespace fb;

extern "C" {

size_t fb_moe_prefill_workspace_bytes(int32_t capacity, int32_t inter) {
  if (capacity < 1 || (inter != 512 && inter != 640)) return 0;
  return pf_layout(capacity, inter).total;
}

int32_t fb_moe_prefill_workspace_make(void* base, int32_t capacity, int32_t inter, fb_moe_prefill_workspace* out) {
  if (!base || !out || (reinterpret_cast<uintptr_t>(base) & 255) || capacity < 1 || (inter != 512 && inter != 640))
    return invalid("prefill_workspace_make: bad arguments (base 256-byte aligned, inter 512 or 640)");
  const PfLayout l = pf_layout(capacity, inter);
  uint8_t* b = static_cast<uint8_t*>(base);
  out->capacity = capacity;
  out->inter = inter;
  out->max_units_gate_up = max_tiles(capacity, kTileN) * (inter / kTileM);
  out->max_units_down = max_tiles(capacity, kTileNDown) * (H / kTileM);
  out->meta = reinterpret_cast<int32_t*>(b + l.meta);
  out->expert_count = reinterpret_cast<int32_t*>(b + l.count);
  out->expert_offset = reinterpret_cast<int32_t*>(b + l.offset);
  out->expert_cursor = reinterpret_cast<int32_t*>(b + l.cursor);
  out->topk_expert = reinterpret_cast<int32_t*>(b + l.topk_e);
  out->topk_weight = reinterpret_cast<float*>(b + l.topk_w);
  out->pair_token = reinterpret_cast<int32_t*>(b + l.pair_token);
  out->pair_weight = reinterpret_cast<float*>(b + l.pair_weight);
  out->token_pair = reinterpret_cast<int32_t*>(b + l.token_pair);
  out->units_gate_up = b + l.units_gu;
  out->units_down = b + l.units_dn;
  out->h = b + l.h;
  out->yp = reinterpret_cast<float*>(b + l.yp);
  out->status = reinterpret_cast<uint32_t*>(b + l.status);
  return 0;
}

// 1: the down projection adds into fixed-point per-token sums (the reference's scheme: exact, order-free,
// no per-pair buffer to write and re-read); 0: it stores fp32 per-pair rows that the combine adds in ascending
// expert order. Both are deterministic. The sums live in the head of the yp buffer.
static int g_prefill_fixed = 0;
int32_t fb_moe_prefill_set_accumulation(int32_t fixed_point) {
  g_prefill_fixed = fixed_point ? 1 : 0;
  return 0;
}
static cudaError_t clear_fixed(const fb_moe_prefill_workspace* ws, int32_t tokens, cudaStream_t s) {
  return g_prefill_fixed ? cudaMemsetAsync(ws->yp, 0, size_t(tokens) * H * 8, s) : cudaSuccess;
}

int32_t fb_moe_route(const float* router_logits, int32_t logits_stride, const void* x, const uint8_t* const* expert_blob,
                     int32_t layer, const uint32_t* seq, void* control, int32_t tokens,
                     const fb_moe_prefill_workspace* ws, void* stream) {
  (void)x;
  (void)expert_blob;
  (void)layer;
  (void)seq;
  if (control) return invalid("route: no CPU expert tier exists behind these kernels; control must be NULL");
  if (!router_logits || logits_stride < kExperts || !pf_ws_ok(ws, tokens)) return invalid("route: bad arguments");
  cudaStream_t s = as_stream(stream);
  cudaError_t e = cudaMemsetAsync(ws->expert_count, 0, kExperts * 4, s);
  if (e == cudaSuccess) e = clear_fixed(ws, tokens, s);
  if (e != cudaSuccess) return check_launch("route: memset");
  const int per_warp = tokens >= 4096 ? 4 : 1;
  auto* kernel = per_warp == 4 ? pf_topk_kernel<4, true> : tokens >= kBlockNumbers ? pf_topk_kernel<1, true> : pf_topk_kernel<1, false>;
  e = launch_pdl(kernel, dim3((tokens + 8 * per_warp - 1) / (8 * per_warp)), dim3(256),
                 0, s, router_logits, logits_stride, tokens, ws->topk_expert, ws->topk_weight, ws->expert_count, ws->token_pair);
  if (e == cudaSuccess) e = launch_pair_lists(ws, tokens, true, s);
  const int32_t st = check_launch("route");
  return st ? st : int32_t(e);
}

int32_t fb_moe_topk(const float* router_logits, int32_t logits_stride, int32_t tokens, int32_t* topk_expert,
                    float* topk_weight, void* stream) {
  if (!router_logits || logits_stride < kExperts || tokens < 1 || !topk_expert || !topk_weight)
    return invalid("topk: bad arguments");
  const cudaError_t e = launch_pdl(pf_topk_kernel<1, false>, dim3((tokens + 7) / 8), dim3(256), 0, as_stream(stream), router_logits,
                                   logits_stride, tokens, topk_expert, topk_weight, static_cast<int32_t*>(nullptr),
                                   static_cast<int32_t*>(nullptr));
  const int32_t st = check_launch("topk");
  return st ? st : int32_t(e);
}

static int32_t route_ep_impl(const int32_t* topk_expert, const float* topk_weight, int32_t expert_lo, int32_t expert_hi,
                             const int32_t* share, int32_t rows, const fb_moe_prefill_workspace* ws, void* stream);

int32_t fb_moe_route_ep(const int32_t* topk_expert, const float* topk_weight, int32_t expert_lo, int32_t expert_hi,
                        int32_t rows, const fb_moe_prefill_workspace* ws, void* stream) {
  if (!topk_expert || !topk_weight || expert_lo < 0 || expert_hi > kExperts || expert_lo >= expert_hi ||
      !pf_ws_ok(ws, rows))
    return invalid("route_ep: bad arguments");
  return route_ep_impl(topk_expert, topk_weight, expert_lo, expert_hi, nullptr, rows, ws, stream);
}

int32_t fb_moe_route_placed(const int32_t* topk_expert, const float* topk_weight, const int32_t* share, int32_t rows,
                            const fb_moe_prefill_workspace* ws, void* stream) {
  if (!topk_expert || !topk_weight || !share || !pf_ws_ok(ws, rows)) return invalid("route_placed: bad arguments");
  return route_ep_impl(topk_expert, topk_weight, 0, 0, share, rows, ws, stream);
}

static int32_t route_ep_impl(const int32_t* topk_expert, const float* topk_weight, int32_t expert_lo, int32_t expert_hi,
                             const int32_t* share, int32_t rows, const fb_moe_prefill_workspace* ws, void* stream) {
  cudaStream_t s = as_stream(stream);
  cudaError_t e = cudaMemsetAsync(ws->expert_count, 0, kExperts * 4, s);
  if (e == cudaSuccess) e = clear_fixed(ws, rows, s);
  if (e != cudaSuccess) return check_launch("route_ep: memset");
  const int n = rows * kTopK;
  e = launch_pdl(rows >= kBlockNumbers ? pf_import_kernel<true> : pf_import_kernel<false>, dim3((n + 255) / 256), dim3(256), 0, s, topk_expert, topk_weight, expert_lo, expert_hi, share,
                 n, ws->topk_expert, ws->topk_weight, ws->expert_count, ws->token_pair);
  if (e == cudaSuccess) e = launch_pair_lists(ws, rows, rows >= kBlockNumbers, s);
  const int32_t st = check_launch("route_ep");
  return st ? st : int32_t(e);
}

int32_t fb_ep_scatter_sum(const float* recv, const int32_t* row_of, int32_t n_ranks, int32_t tokens, float* y,
                          void* stream) {
  if (!recv || !row_of || n_ranks < 1 || tokens < 1 || !y) return invalid("ep_scatter_sum: bad arguments");
  ep_scatter_sum_kernel<<<dim3(H / 256, tokens), 256, 0, as_stream(stream)>>>(recv, row_of, n_ranks, y);
  return check_launch("ep_scatter_sum");
}

int32_t fb_moe_grouped_gate_up(const fb_moe_expert_layout* layout, const uint8_t* const* expert_blob, const void* x_bf16,
                               int32_t tokens, const fb_moe_prefill_workspace* ws, void* stream) {
  if (!pf_layout_ok(layout, expert_blob) || !x_bf16 || !pf_ws_ok(ws, tokens) || layout->inter != ws->inter ||
      (reinterpret_cast<uintptr_t>(x_bf16) & 15))
    return invalid("grouped_gate_up: bad arguments");
  // The token rows in pair order use the upper half of yp, which nothing needs before the down projection writes it
  // (the fixed-point sums, cleared by the route call, sit in its first fifth).
  auto* xg = reinterpret_cast<__nv_bfloat16*>(ws->yp + size_t(ws->capacity) * kTopK * (H / 2));
  GgMaps maps;
  if (const int32_t st = rows_maps(&maps, xg, H, ws->capacity, "grouped_gate_up")) return st;
  // a few tokens: a fifth of a row per warp, so that there are enough of them (9.3 us at 96 tokens with whole rows)
  const int parts = tokens <= 1024 ? 5 : 1;
  cudaError_t e = launch_pdl(parts == 5 ? scatter_rows_kernel<5> : scatter_rows_kernel<1>, dim3((tokens * parts + 3) / 4),
                             dim3(128), 0, as_stream(stream), static_cast<const __nv_bfloat16*>(x_bf16), ws->token_pair, tokens, xg);
  if (e != cudaSuccess) {
    set_error("grouped_gate_up: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return int32_t(e);
  }
  GgArgs a{};
  a.L = *layout;
  a.expert_blob = expert_blob;
  a.tiles = static_cast<const int4*>(ws->units_gate_up);
  a.n_units = ws->meta;
  a.h = static_cast<__nv_bfloat16*>(ws->h);
  a.status = ws->status;
  e = layout->gate_up_format == FB_FMT_IQ3_S ? launch_grouped<FB_FMT_IQ3_S, false>(a, maps, as_stream(stream))
                                             : launch_grouped<FB_FMT_IQ4_NL, false>(a, maps, as_stream(stream));
  if (e != cudaSuccess) {
    set_error("grouped_gate_up: %s", cudaGetErrorString(e));
    return int32_t(e);
  }
  return check_launch("grouped_gate_up");
}

int32_t fb_moe_grouped_down(const fb_moe_expert_layout* layout, const uint8_t* const* expert_blob, int32_t tokens,
                            const fb_moe_prefill_workspace* ws, void* stream) {
  if (!pf_layout_ok(layout, expert_blob) || !pf_ws_ok(ws, tokens) || layout->inter != ws->inter)
    return invalid("grouped_down: bad arguments");
  GgMaps maps;
  if (const int32_t st = rows_maps(&maps, ws->h, ws->inter, ws->capacity, "grouped_down")) return st;
  GgArgs a{};
  a.L = *layout;
  a.expert_blob = expert_blob;
  a.tiles = static_cast<const int4*>(ws->units_down);
  a.n_units = ws->meta + 1;
  a.pair_token = ws->pair_token;
  a.pair_weight = ws->pair_weight;
  a.yp = ws->yp;
  a.y_fixed = g_prefill_fixed ? reinterpret_cast<unsigned long long*>(ws->yp) : nullptr;
  a.status = ws->status;
  const cudaError_t e = layout->down_format == FB_FMT_IQ3_S
                            ? launch_grouped<FB_FMT_IQ3_S, true>(a, maps, as_stream(stream))
                            : launch_grouped<FB_FMT_IQ4_NL, true>(a, maps, as_stream(stream));
  if (e != cudaSuccess) {
    set_error("grouped_down: %s", cudaGetErrorString(e));
    return int32_t(e);
  }
  return check_launch("grouped_down");
}

int32_t fb_moe_prefill_combine(const fb_moe_prefill_workspace* ws, const float* y_shared, void* control, int32_t layer,
                               const uint32_t* seq, const float* inj, float* X, float* y_out, int32_t tokens,
                               long long timeout_cycles, const float* ablate_direction, float ablate_scale,
                               void* stream) {
  (void)layer;
  (void)seq;
  (void)timeout_cycles;
  (void)ablate_scale;
  if (control) return invalid("prefill_combine: no CPU expert tier exists behind these kernels; control must be NULL");
  if (ablate_direction) return invalid("prefill_combine: the rank-1 ablation is not built for the prefill path");
  if (!pf_ws_ok(ws, tokens) || (X && !inj) || (!X && !y_out)) return invalid("prefill_combine: bad arguments");
  const bool aligned = ((reinterpret_cast<uintptr_t>(y_shared) | reinterpret_cast<uintptr_t>(X) |
                         reinterpret_cast<uintptr_t>(y_out)) & 15) == 0;
  auto* kernel = aligned ? pf_combine_kernel<true> : pf_combine_kernel<false>;
  const cudaError_t e = launch_pdl(kernel, dim3(unsigned(tokens) * kPcParts), dim3(kPcThreads), 0, as_stream(stream), ws->topk_expert, ws->token_pair,
                                   ws->yp, y_shared, inj, X, y_out,
                                   g_prefill_fixed ? reinterpret_cast<const long long*>(ws->yp) : nullptr);
  const int32_t st = check_launch("prefill_combine");
  return st ? st : int32_t(e);
}

}  // extern "C"
