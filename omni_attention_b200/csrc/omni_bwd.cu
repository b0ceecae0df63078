// sm_100a backward pass of block-mask ("omni") attention: dQ, dK, dV from dO with the block lists of
// the forward pass and its saved log-sum-exp. The reference is forward-only
// (omni-attn-mma/mma/omni_attn_shared_kv.cu has no gradient kernel); what is differentiated here is
// its forward definition, softmax((Q K^T) * scale + mask) V (omni-attn-mma/omni_attn_torch.py:348-387),
// with the same mask semantics as the forward kernels (omni_common.cuh).
//
//   P  = exp(S * scale - LSE)            S = Q K^T, masked entries give P = 0
//   dV = P^T dO
//   dP = dO V^T,  delta = rowsum(dO * O),  dS = P * (dP - delta)
//   dQ = scale * dS K,   dK = scale * dS^T Q
//
// Two launches on the caller's stream, all working memory in a caller-provided workspace:
//   1. omni_bwd_prep_kernel   resolves every (Q block, KV block) of the lists into a dense table of
//                             entry codes [BH, nq, nq] (so that the lists can be walked by column as
//                             well as by row) and computes delta.
//   2. omni_bwd_kernel        two kinds of CTA:
//      dK/dV                  one per (KV block, batch*head); K, V stay in shared memory, the Q
//                             blocks that visit this KV block stream through a ring; S^T and
//                             dP^T are computed transposed (TMEM lane = key) so that P^T and dS^T can be
//                             fed to the tensor cores from TMEM for dV += P^T dO and dK += dS^T Q.
//      dQ                     one per (Q block, batch*head), the mirror image: Q, dO stay, the
//                             visited K, V stream; dQ += dS K with dS from TMEM.
// S and dP are recomputed in both kinds (7 tile contractions per visited tile instead of 5), which
// buys a deterministic result with no atomics and no fp32 dQ buffer.
// Both are warp-specialised: 8 compute warps (a tile row = TMEM lane is shared by two
// threads, one per warpgroup, each taking 64 of its 128 columns), one warp of which an elected lane issues
// every tcgen05.mma and one of which an elected lane issues the TMA loads; everything is handed over through
// mbarriers (tcgen05.commit for "MMAs done", thread arrivals for "P / dS stored"). The per-element
// work of a visit is split in two (probabilities from S; dS from dP and the probabilities) and the
// MMAs of consecutive visits are interleaved so that the tensor pipe runs under both halves.
#include <type_traits>

#include "omni_common.cuh"
#include "omni_launch.h"

namespace omni {

template <int D>
struct BwdCfg {
  static constexpr int kTileBytes = kBlock * D * 2;
  static constexpr int kChunks = D / 64;
  static constexpr int kChunkBytes = kBlock * 128;
  static constexpr int kTmemCols = 512;
  // dK/dV kernel: whether S^T has two regions of TMEM (free next to dV and dK at D = 64) and is issued a visit
  // ahead, and the stages of Q, LSE and delta that this takes
  static constexpr bool kAhead = (D == 64);
  static constexpr int kQStages = kAhead ? 3 : 2;
  static constexpr int kVecBytes = 2 * kQStages * kBlock * 4;   // LSE and delta of a Q block
  static constexpr int kBitsBytes = 2 * kBlock * 16;      // bit-packed partial tiles of two visits
  static constexpr int kListBytes = kMaxKvBlocks * 4 + kMaxKvBlocks * 2 + 16;   // codes, visit list, its length
  static constexpr int kSmemBytes = (4 + kQStages) * kTileBytes + kVecBytes + kBitsBytes + kListBytes + 256;
};

// Of every eight element pairs, this many take their exponentials from the FMA pipe (exp2_fma2): the two halves of
// the per-element work alternate, so while E1 runs the MUFU unit is what it waits for (1 024 cycles a visit). dK/dV
// kernel 956 -> 942 / 934 / 938 us with 1 / 2 / 3 of eight (32 heads x 8K tokens, D = 128) and 234 -> 227 / 225 / 224
// (32 x 4K, D = 64); dQ kernel 710 -> 704 / 698 / 700 and 172 -> 170 / 167 / 166.
// Not with a soft-cap, whose own polynomial already fills that pipe (dQ kernel of 16 heads x 1.5K tokens 34 -> 36 us).
constexpr int kBwdPolyOf8 = 2;

constexpr int kBwdComputeThreads = 256;
constexpr int kBwdThreads = kBwdComputeThreads + 64;
constexpr int kBwdIssuerWarp = kBwdComputeThreads / 32;         // one elected lane issues the MMAs
constexpr int kBwdProducerWarp = kBwdComputeThreads / 32 + 1;   // one elected lane issues the TMA loads


template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (BF16) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
  } else {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
}

// ---------------------------------------------------------------------------------------------
// 1. Workspace: entry-code table and delta. Grid (nq, BH), 160 threads: warps 0-3 compute delta of 32 rows
// each, warp 4 resolves the Q block's list. Bound by the two 16-bit tensors read once, and for short batches by
// load latency alone, so each warp has kBatch loads of 16 bytes per lane and tensor in flight, several rows at a
// time (one row at a time, 4 bytes per lane: 24.7 against 4.7 us for 16 heads x 1.5K tokens, 34 against 27 for
// 32 x 8K at D = 128, which is 5 TB/s).
// ---------------------------------------------------------------------------------------------
constexpr int kPrepThreads = 160;
template <int D, bool BF16>
__global__ void __launch_bounds__(kPrepThreads) omni_bwd_prep_kernel(const BwdParams p) {
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int qb = blockIdx.x;
  const int bh = blockIdx.y;
  const int nq = p.f.nq;

  uint32_t* codes = p.codes + (static_cast<long long>(bh) * nq + qb) * nq;
  if (warp == 4) {
    for (int i = lane; i < nq; i += 32) codes[i] = 0u;
    __syncwarp();
    const long long list_base = (static_cast<long long>(bh) * nq + qb) * p.f.max_blocks;
    int n_list = __ldg(p.f.kv_num_blocks + static_cast<long long>(bh) * nq + qb);
    n_list = max(0, min(n_list, p.f.max_blocks));
    for (int i0 = 0; i0 < n_list; i0 += 32) {   // in list order; a block listed twice resolves as in the forward
      const int i = i0 + lane;
      int kvb = -1;
      uint32_t code = 0u;
      if (i < n_list) code = resolve_entry(p.f, list_base, i, qb, kvb);
      table_put(codes, code != 0u ? kvb : -1, code);
    }
    return;
  }

  constexpr int kLanes = D / 8;               // lanes per row, 16 bytes each
  constexpr int kRowsAtOnce = 32 / kLanes;
  constexpr int kBatch = 4;
  const int sub = lane / kLanes, col = (lane % kLanes) * 8;
  const bool in_row = col < p.f.d_real;       // head_dim 32 on the 64-wide instantiation: half the lanes idle
  const long long pitch = static_cast<long long>(p.f.d_real) * 2;
  const long long head = static_cast<long long>(bh) * p.f.N;
#pragma unroll 1
  for (int r0 = 0; r0 < 32; r0 += kRowsAtOnce * kBatch) {
    uint4 a[kBatch], b[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int q_abs = qb * kBlock + 32 * warp + r0 + kRowsAtOnce * i + sub;
      a[i] = b[i] = make_uint4(0u, 0u, 0u, 0u);
      if (in_row && q_abs < p.f.N) {   // the last tile of an unpadded tensor ends inside
        a[i] = __ldg(reinterpret_cast<const uint4*>(static_cast<const char*>(p.o) + (head + q_abs) * pitch + 2 * col));
        b[i] = __ldg(reinterpret_cast<const uint4*>(static_cast<const char*>(p.d_o) + (head + q_abs) * pitch + 2 * col));
      }
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int q_abs = qb * kBlock + 32 * warp + r0 + kRowsAtOnce * i + sub;
      const uint32_t wa[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, wb[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
      float acc = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float2 x = unpack2<BF16>(wa[w]), y = unpack2<BF16>(wb[w]);
        acc = fmaf(x.x, y.x, acc);
        acc = fmaf(x.y, y.y, acc);
      }
#pragma unroll
      for (int o = kLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
      if (lane % kLanes == 0 && q_abs < p.f.N) p.delta[head + q_abs] = acc;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Pieces shared by the two tile kernels.
// ---------------------------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void bwd_load_tile(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int y, int bh) {
#pragma unroll
  for (int c = 0; c < BwdCfg<D>::kChunks; ++c) tma_load_3d(dst + c * BwdCfg<D>::kChunkBytes, tm, bar, c * 64, y, bh);
}

// The issuing thread runs ahead of the tensor pipe by about eight MMAs as long as it spends less time on
// an MMA than the pipe does (64 cycles at 128x128x16): the thread is chosen with elect.sync (an MMA issued
// under a branch on the lane number costs the thread 52 cycles, under an elected branch 17), the
// descriptors are advanced as 32-bit low words (the high word is one constant) and the accumulate flags
// are compile-time constants wherever they can be.
constexpr uint32_t kBwdDescHi = umma_desc_hi_sw128(1024);

// acc[128 x 128] = A[128 x D] * B[128 x D]^T, both tiles row-major with D contiguous (K-major).
template <int D>
__device__ __forceinline__ void bwd_mma_ss(uint32_t d_tmem, uint32_t sA, uint32_t sB, uint32_t idesc) {
  const uint32_t a_lo = umma_desc_lo(sA, 16), b_lo = umma_desc_lo(sB, 16);
  umma_ss_lo<false>(d_tmem, a_lo, b_lo, kBwdDescHi, idesc);
#pragma unroll
  for (int k = 1; k < D / 16; ++k) {
    const uint32_t off = ((k / 4) * BwdCfg<D>::kChunkBytes + (k % 4) * 32) >> 4;
    umma_ss_lo<true>(d_tmem, a_lo + off, b_lo + off, kBwdDescHi, idesc);
  }
}

// acc[128 x D] (+)= A[128 x 128] * B[128 x D], A 16-bit in TMEM (lane = row of A), B a row-major tile whose rows
// are the contraction index (MN-major operand). A is stored as two runs of 32 TMEM columns, 64 columns apart
// (contraction indices [0,64) at a_region + a_off, [64,128) at a_region + 64 + a_off): the layout the
// tile kernels use so that each thread writes P / dS only over score columns it has read itself.
template <int D>
__device__ __forceinline__ void bwd_mma_ts_split(uint32_t d_tmem, uint32_t a_region, uint32_t a_off, uint32_t sB,
                                                 uint32_t idesc, bool accumulate) {
  const uint32_t b_lo = umma_desc_lo(sB, BwdCfg<D>::kChunkBytes);
  umma_ts_lo(d_tmem, a_region + a_off, b_lo, kBwdDescHi, idesc, accumulate ? 1u : 0u);
#pragma unroll
  for (int k = 1; k < kBlock / 16; ++k) {
    umma_ts_lo_acc(d_tmem, a_region + 64 * (k / 4) + a_off + 8 * (k % 4), b_lo + k * 128, kBwdDescHi, idesc);
  }
}

// One accumulator row (32-column chunks [kFirstChunk, kEndChunk) of it) out of TMEM, times `mul`, as
// 16-bit values to global memory (zeros when `have_acc` is false; nothing when the row is not in memory).
template <int D, bool BF16, int kFirstChunk = 0, int kEndChunk = D / 32>
__device__ __forceinline__ void bwd_store_row(uint32_t taddr_row, bool have_acc, float mul, void* base,
                                              long long row_index, int d_real, bool in_memory) {
  // rows of the output are d_real elements long; accumulator columns beyond that (head_dim 32 on the
  // 64-wide instantiation) are zero and are not stored
  uint4* dst = reinterpret_cast<uint4*>(static_cast<char*>(base) + row_index * (static_cast<long long>(d_real) * 2));
#pragma unroll
  for (int c = kFirstChunk; c < kEndChunk; ++c) {
    if (32 * c >= d_real) break;
    uint32_t r[32];
    if (have_acc) {
      tmem_ld32(taddr_row + 32 * c, r);
      tc_wait_ld();
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = 0u;
    }
    uint32_t w[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      w[j] = pack2<BF16>(__uint_as_float(r[2 * j]) * mul, __uint_as_float(r[2 * j + 1]) * mul);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (in_memory) dst[4 * c + j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
    }
  }
}

// One row or column of the entry-code table -> shared memory, plus the ascending list of the blocks
// it visits (walking the table in global memory instead costs one dependent load per skipped
// block). Every thread of the CTA must call it.
__device__ __forceinline__ int bwd_build_visit_list(const uint32_t* src, long long stride, int n, uint32_t* code_s,
                                                    uint16_t* vis_s, int* n_vis_s) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) code_s[i] = __ldg(src + i * stride);
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int count = 0;
    for (int base = 0; base < n; base += 32) {
      const bool on = base + lane < n && code_s[base + lane] != 0u;
      const uint32_t any = __ballot_sync(0xFFFFFFFFu, on);
      if (on) vis_s[count + __popc(any & ((1u << lane) - 1u))] = static_cast<uint16_t>(base + lane);
      count += __popc(any);
    }
    if (lane == 0) *n_vis_s = count;
  }
  __syncthreads();
  return *n_vis_s;
}

// Tanh soft-cap in the backward pass (the forward's soft_cap_scores): the raw score s stands for the
// capped scaled score softcap * tanh(s * scale / softcap), whose derivative with respect to the
// scaled raw score is 1 - tanh^2. Replaces the pair of raw scores by their capped raw-equivalents
// (cap_out * tanh) and returns the two derivative factors.
__device__ __forceinline__ float2 bwd_soft_cap(float2& s, float cap_in, float cap_out) {
  const float2 y = __fmul2_rn(s, make_float2(cap_in, cap_in));
  float2 t;
  if (fmaxf(fabsf(y.x), fabsf(y.y)) <= kTanhPolyLimit) {
    t = tanh_small2(y);   // the forward's polynomial for small arguments: no MUFU work
  } else {
    t = make_float2(tanh_exact(y.x), tanh_exact(y.y));
  }
  s = __fmul2_rn(t, make_float2(cap_out, cap_out));
  return __ffma2_rn(make_float2(-t.x, -t.y), t, make_float2(1.f, 1.f));
}

// CTA index -> (block, batch*head) for the two tile kernels. Heads are taken in groups of
// `group_heads` (sized on the host so that a group's Q, K, V and dO stay in L2 together); inside a
// group the blocks run from the longest lists to the shortest for causal-like masks (`descending`:
// from the last block to the first) with the group's heads adjacent, so that the long CTAs of every
// head start early and the grid drains with short ones.
__device__ __forceinline__ void bwd_decode_cta(const FwdParams& f, int cta, bool descending, int& block, int& bh) {
  const int G = f.group_heads;
  const int grp = cta / (f.nq * G);
  const int rem = cta - grp * f.nq * G;
  const int heads_here = min(G, f.BH - grp * G);
  const int b = rem / heads_here;
  block = descending ? f.nq - 1 - b : b;
  bh = grp * G + rem % heads_here;
}

// log-sum-exp (natural log) -> subtrahend in the log2 domain; a row that attended nothing
// (-inf) gives +inf, which turns every probability of the row into exp2(-inf) = 0.
__device__ __forceinline__ float lse_to_log2(float lse) {
  return lse == -INFINITY ? INFINITY : lse * 1.4426950408889634f;
}

// ---------------------------------------------------------------------------------------------
// 2. dK, dV. One CTA per (KV block, batch*head), see bwd_decode_cta. 320 threads:
//   warps 0-7  per-element work; threads t and t + 128 own key row t of the block (query columns
//              [0,64) and [64,128) of the visited Q block)
//   warp  8    an elected lane issues every tcgen05.mma
//   warp  9    an elected lane issues the TMA loads (at D = 64 all lanes stage LSE and delta)
// TMEM, D = 128: S^T [0,128), dP^T [128,256), dV [256,384), dK [384,512); P^T (16-bit) goes over S^T and
// dS^T over dP^T. D = 64: two regions of S^T [0,256), dP^T [256,384), dV [384,448), dK [448,512); P^T and dS^T
// both go over S^T. Each thread writes only columns it has read itself.
//
// The per-element work is split in two so that the tensor pipe always has something to do:
//   E1(i): P^T  = exp2(S^T * c - LSE)        needs S^T(i)          -> feeds dV(i)
//   E2(i): dS^T = P^T * (dP^T - delta)       needs dP^T(i), E1(i)  -> feeds dK(i)
// and the MMAs of consecutive visits are interleaved, at D = 128 in the order
//   dV(i), S^T(i+1) | dK(i), dP^T(i+1)
// The first pair is issued when P^T(i) is there and runs under E2(i), the second when dS^T(i) is there and
// runs under E1(i+1): each region is overwritten by the MMA right behind the one that read it, so neither
// half of the per-element work waits for more than the pair in front of it. (With the regions alternating,
// S^T(i+1) over dP^T(i) and so only after E2(i), the chain S^T - E1 - E2 of a visit could not overlap the next
// one's: kernel 1055 against 949 us for 32 heads x 8K tokens at D = 128, bits equal.) The 32 MMAs of a visit are
// 2 048 of its about 3 000 cycles; both kinds of CTA together keep the tensor pipe busy for 66 % of the active cycles.
// D = 64 needs half the MMAs and is bound by the per-element work; its second region of S^T lets the scores run a
// visit ahead, so that E1(i+1) starts as soon as E2(i) ends:
//   dV(i) | dP^T(i+1), dK(i), S^T(i+2)
// (32 heads x 4K tokens: 230 -> 211 us together with the vectors staged by the producer warp and kBwdPolyOf8.)
// ---------------------------------------------------------------------------------------------
template <int D, bool BF16, bool SOFTCAP>
__device__ __forceinline__ void bwd_dkdv_cta(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                                             const CUtensorMap& tmdO, const BwdParams& p, int cta, uint8_t* smem) {
  using Cfg = BwdCfg<D>;

  const uint32_t sK = smem_u32(smem);
  const uint32_t sV = sK + Cfg::kTileBytes;
  const uint32_t sQ = sV + Cfg::kTileBytes;                  // kQStages
  const uint32_t sdO = sQ + Cfg::kQStages * Cfg::kTileBytes;  // two stages
  // -LSE * log2(e) (-inf for a dead row) and -delta of the visited Q block, kQStages
  float* lse_s = reinterpret_cast<float*>(smem + (4 + Cfg::kQStages) * Cfg::kTileBytes);   // [kQStages][128]
  float* delta_s = lse_s + Cfg::kQStages * kBlock;                                         // [kQStages][128]
  uint32_t* bits_s = reinterpret_cast<uint32_t*>(delta_s + Cfg::kQStages * kBlock);        // [2][128][4]
  uint32_t* code_s = bits_s + 2 * kBlock * 4;                                // [kMaxKvBlocks]
  uint16_t* vis_s = reinterpret_cast<uint16_t*>(code_s + kMaxKvBlocks);      // [kMaxKvBlocks]
  int* n_vis_s = reinterpret_cast<int*>(vis_s + kMaxKvBlocks);
  uint64_t* bars = reinterpret_cast<uint64_t*>(n_vis_s + 4);
  const uint32_t bar_kv = smem_u32(bars + 0);       // K, V landed
  const uint32_t bar_q = smem_u32(bars + 1);        // [3] Q stage landed
  const uint32_t bar_do = smem_u32(bars + 4);       // [2] dO stage landed
  const uint32_t bar_s = smem_u32(bars + 6);        // [2] S^T of a visit complete (by visit parity)
  const uint32_t bar_dp = smem_u32(bars + 8);       // dP^T of the visit complete
  // [2] P^T of a visit stored (256 arrivals), by visit parity: with the scores issued a visit ahead, a warp can be
  // through E1(i+1) while another is still in E1(i) and the issuer has not looked yet. Two are enough: E1(i+2)
  // comes after E2(i+1), which needs dP^T(i+1), issued only after every thread has stored P^T(i) and dS^T(i).
  const uint32_t bar_p = smem_u32(bars + 9);
  const uint32_t bar_ds = smem_u32(bars + 11);      // dS^T stored (256 arrivals)
  const uint32_t bar_dvdone = smem_u32(bars + 12);  // [2] dV MMAs of the visit in this stage complete: dO stage free
  const uint32_t bar_dkdone = smem_u32(bars + 14);  // [3] dK MMAs complete: Q, LSE and delta stage free
  const uint32_t bar_vec = smem_u32(bars + 17);     // [3] LSE / delta of the visit in this stage written (32 arrivals)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const bool compute = tid < kBwdComputeThreads;
  const int half = (tid >> 7) & 1;  // which 64 query columns of the tile this thread works on
  const int t = tid & 127;          // key row of the tile = TMEM lane
  const int nq = p.f.nq;
  int kvb, bh;
  bwd_decode_cta(p.f, cta, false, kvb, bh);

  if (tid == 0) {
    mbar_init(bar_kv, 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(bar_q + 8 * s, 1);
      mbar_init(bar_dkdone + 8 * s, 1);
      mbar_init(bar_vec + 8 * s, 32);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_do + 8 * s, 1);
      mbar_init(bar_dvdone + 8 * s, 1);
      mbar_init(bar_s + 8 * s, 1);
      mbar_init(bar_p + 8 * s, kBwdComputeThreads);
    }
    mbar_init(bar_dp, 1);
    mbar_init(bar_ds, kBwdComputeThreads);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const uint32_t tmem_base = *tmem_slot;
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  auto region_s = [&](int i) { return tmem_base + (Cfg::kAhead ? 128u * static_cast<uint32_t>(i & 1) : 0u); };
  const uint32_t tdP = tmem_base + (Cfg::kAhead ? 256 : 128);
  const uint32_t tdV = tmem_base + 512 - 2 * D;
  const uint32_t tdK = tmem_base + 512 - D;
  // where dS^T goes, from a thread's 64 columns on: behind P^T over S^T, or over dP^T
  auto region_ds = [&](int i) { return Cfg::kAhead ? region_s(i) : tdP; };
  constexpr uint32_t kDsOff = Cfg::kAhead ? 32 : 0;
  constexpr int fmt = BF16 ? 1 : 0;
  constexpr uint32_t idesc_ss = umma_idesc_f16(128, 128, fmt, 0);
  constexpr uint32_t idesc_ts = umma_idesc_f16(128, D, fmt, 1);

  const long long row0 = static_cast<long long>(bh) * p.f.N;
  // column kvb of this head's code table: which Q blocks visit this KV block, and how
  const int n_vis = bwd_build_visit_list(p.codes + static_cast<long long>(bh) * nq * nq + kvb, nq, nq, code_s, vis_s,
                                         n_vis_s);
  // What the compute warps need of query row q_abs: -LSE * log2(e), -inf for a row beyond the sequence or one
  // that attended nothing, and -delta.
  auto load_vectors = [&](int q_abs, float& neg_lse2, float& neg_delta) {
    const bool live = q_abs < p.f.seqlen_orig;
    neg_lse2 = live ? -lse_to_log2(__ldg(p.lse + row0 + q_abs)) : -INFINITY;
    neg_delta = live ? -__ldg(p.delta + row0 + q_abs) : 0.f;
  };
  if constexpr (!Cfg::kAhead) {
    if (tid < kBlock) {
      for (int i = 0; i < 2 && i < n_vis; ++i) {
        load_vectors(static_cast<int>(vis_s[i]) * kBlock + tid, lse_s[i * kBlock + tid], delta_s[i * kBlock + tid]);
      }
    }
    __syncthreads();   // the vectors are read by every compute thread
  }

  if (warp == kBwdProducerWarp && (Cfg::kAhead || elect_one())) {
    // =========================== TMA producer ====================================================
    // With S^T issued ahead, the whole warp runs this loop: one elected lane issues the copies and all stage the
    // LSE / delta vectors (rows of unpadded tensors have no alignment that a bulk copy could use) in the form the
    // compute warps need them in. A stage of Q and of the vectors is free when dK of its last visit, which was
    // issued after every compute thread had stored dS^T, is complete. Without (D = 128) one lane issues the
    // copies and the compute warps stage the vectors: there the loop waits on the tensor pipe anyway, and the
    // vectors in this warp made the kernel slower (984 against 945 us; at D = 64 223 against 233).
    const bool leader = Cfg::kAhead ? elect_one() : true;
    auto wait = [&](uint32_t bar, uint32_t parity, int where) {
      if constexpr (Cfg::kAhead) {
        mbar_wait_warp(bar, parity, abort_flag, p.f.status, where);
      } else {
        mbar_wait(bar, parity, abort_flag, p.f.status, where);
      }
    };
    if (n_vis > 0 && leader) {
      mbar_expect_tx(bar_kv, 2 * Cfg::kTileBytes);
      const int y = kvb * kBlock;
      bwd_load_tile<D>(sK, &tmK, bar_kv, y, bh);
      bwd_load_tile<D>(sV, &tmV, bar_kv, y, bh);
    }
    auto load_q = [&](int i) {
      const int stage = i % Cfg::kQStages;
      const int y = static_cast<int>(vis_s[i]) * kBlock;
      float vl[4], vd[4];   // in flight while the stage is waited for
      if constexpr (Cfg::kAhead) {
#pragma unroll
        for (int j = 0; j < 4; ++j) load_vectors(y + 32 * j + lane, vl[j], vd[j]);
      }
      if (i >= Cfg::kQStages) {
        wait(bar_dkdone + 8 * stage, static_cast<uint32_t>((i / Cfg::kQStages - 1) & 1), 55);
      }
      if (leader) {
        mbar_expect_tx(bar_q + 8 * stage, Cfg::kTileBytes);
        bwd_load_tile<D>(sQ + stage * Cfg::kTileBytes, &tmQ, bar_q + 8 * stage, y, bh);
      }
      if constexpr (Cfg::kAhead) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          lse_s[stage * kBlock + 32 * j + lane] = vl[j];
          delta_s[stage * kBlock + 32 * j + lane] = vd[j];
        }
        mbar_arrive(bar_vec + 8 * stage);
      }
    };
    auto load_do = [&](int i) {
      const int stage = i & 1;
      if (i >= 2) wait(bar_dvdone + 8 * stage, static_cast<uint32_t>(((i >> 1) - 1) & 1), 56);
      if (leader) {
        mbar_expect_tx(bar_do + 8 * stage, Cfg::kTileBytes);
        bwd_load_tile<D>(sdO + stage * Cfg::kTileBytes, &tmdO, bar_do + 8 * stage, static_cast<int>(vis_s[i]) * kBlock, bh);
      }
    };
    if (Cfg::kAhead && n_vis > 0) load_q(0);
    for (int i = 0; i < n_vis; ++i) {   // in the order in which the stages come free
      if constexpr (Cfg::kAhead) {
        load_do(i);
        if (i + 1 < n_vis) load_q(i + 1);
      } else if (i < 2) {   // both stages are empty: what the visit needs first
        load_q(i);
        load_do(i);
      } else {
        load_do(i);
        load_q(i);
      }
    }
  } else if (warp == kBwdIssuerWarp && elect_one()) {
    // =========================== MMA issuer ======================================================
    auto issue_s = [&](int i) {    // S^T(i) = K Q(i)^T
      const int stage = i % Cfg::kQStages;
      mbar_wait(bar_q + 8 * stage, static_cast<uint32_t>((i / Cfg::kQStages) & 1), abort_flag, p.f.status, 51);
      tc_fence_after();
      bwd_mma_ss<D>(region_s(i), sK, sQ + stage * Cfg::kTileBytes, idesc_ss);
      tc_commit(bar_s + 8 * (i & 1));
    };
    auto issue_dp = [&](int i) {   // dP^T(i) = V dO(i)^T
      const int stage = i & 1;
      mbar_wait(bar_do + 8 * stage, static_cast<uint32_t>((i >> 1) & 1), abort_flag, p.f.status, 52);
      tc_fence_after();
      bwd_mma_ss<D>(tdP, sV, sdO + stage * Cfg::kTileBytes, idesc_ss);
      tc_commit(bar_dp);
    };
    auto issue_dk = [&](int i) {   // dK += dS^T(i) Q(i)
      const int stage = i % Cfg::kQStages;
      bwd_mma_ts_split<D>(tdK, region_ds(i), kDsOff, sQ + stage * Cfg::kTileBytes, idesc_ts, i > 0);
      tc_commit(bar_dkdone + 8 * stage);
    };
    if (n_vis > 0) {
      mbar_wait(bar_kv, 0, abort_flag, p.f.status, 50);
      issue_s(0);
      issue_dp(0);
      if (Cfg::kAhead && n_vis > 1) issue_s(1);
    }
    for (int i = 0; i < n_vis; ++i) {
      const int stage = i & 1;
      const uint32_t ph = static_cast<uint32_t>(i & 1);
      // E1(i) has read S^T(i) and stored P^T(i) over it
      mbar_wait(bar_p + 8 * stage, static_cast<uint32_t>((i >> 1) & 1), abort_flag, p.f.status, 58);
      tc_fence_after();
      bwd_mma_ts_split<D>(tdV, region_s(i), 0, sdO + stage * Cfg::kTileBytes, idesc_ts, i > 0);    // dV += P^T(i) dO(i)
      tc_commit(bar_dvdone + 8 * stage);
      if (!Cfg::kAhead && i + 1 < n_vis) issue_s(i + 1);   // over P^T(i), which the MMAs just issued read first
      // E2(i) has read dP^T(i) and stored dS^T(i)
      mbar_wait(bar_ds, ph, abort_flag, p.f.status, 57);
      tc_fence_after();
      if constexpr (Cfg::kAhead) {
        if (i + 1 < n_vis) issue_dp(i + 1);   // first: E2(i + 1) waits for it
        issue_dk(i);
        if (i + 2 < n_vis) issue_s(i + 2);    // over P^T(i) and dS^T(i)
      } else {
        issue_dk(i);
        if (i + 1 < n_vis) issue_dp(i + 1);   // over dS^T(i)
      }
    }
    if (n_vis > 0) {
      const int last = n_vis - 1;
      // keep this thread alive until every MMA has retired
      mbar_wait(bar_dkdone + 8 * (last % Cfg::kQStages), static_cast<uint32_t>((last / Cfg::kQStages) & 1), abort_flag,
                p.f.status, 59);
    }
  } else if (compute) {
    // =========================== per-element work ================================================
    const int k_abs = kvb * kBlock + t;
    const bool key_live = k_abs < p.f.seqlen_orig;
    const float2 c2 = make_float2(p.f.scale_log2, p.f.scale_log2);
    int next_qb = n_vis > 0 ? vis_s[0] : 0;   // looked up one visit ahead
    uint32_t next_code = code_s[next_qb];
    int turn = 0;   // i % 3, counted: divided, it is a register too many in the soft-capped kernel (112 bytes of spills, 32 now)
    for (int i = 0; i < n_vis; ++i, turn = turn == 2 ? 0 : turn + 1) {
      const int stage = Cfg::kAhead ? turn : i & 1;
      const uint32_t ph = static_cast<uint32_t>(i & 1);
      const int qb = next_qb;
      const uint32_t code = next_code;
      const uint32_t my_s = region_s(i) + lane_base + 64 * half;
      const uint32_t my_dp = tdP + lane_base + 64 * half;
      const uint32_t my_ds = region_ds(i) + kDsOff + lane_base + 64 * half;
      // D = 128: the vectors of the visit after next, loaded here and stored at the end of this visit, so that
      // their latency is off everybody's path
      float next_lse = -INFINITY, next_delta = 0.f;
      if (!Cfg::kAhead && tid < kBlock && i + 2 < n_vis) {
        load_vectors(static_cast<int>(vis_s[i + 2]) * kBlock + tid, next_lse, next_delta);
      }

      // Allow-bits of this thread's key over its 64 query rows of the block (bit r of word w = query
      // row 64 * half + 32 * w + r).
      const uint32_t type = code & kCodeTypeMask;
      uint32_t allow[2] = {0xFFFFFFFFu, 0xFFFFFFFFu};
      if (type == kTypePartial) {   // uniform over the compute threads
        // (the buffer's last use was two visits ago: dP^T of the last visit came after every dS^T of that one)
        uint32_t* bits = bits_s + (i & 1) * kBlock * 4;
        if (tid < kBlock) {
          uint32_t rowbits[4];
          load_partial_row(p.f, code >> 3, tid, rowbits);   // row tid of the tile = query row tid
          *reinterpret_cast<uint4*>(bits + 4 * tid) = make_uint4(rowbits[0], rowbits[1], rowbits[2], rowbits[3]);
        }
        named_barrier_sync(1, kBwdComputeThreads);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          uint32_t acc = 0u;
#pragma unroll
          for (int r = 0; r < 32; ++r) {
            acc |= ((bits[4 * (64 * half + 32 * w + r) + (t >> 5)] >> (t & 31)) & 1u) << r;
          }
          allow[w] = acc;
        }
      } else if (type == kTypeCausal) {
        // diagonal block: key t is seen by query rows r >= t
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const int d = t - 64 * half - 32 * w;   // lowest allowed bit in this word
          allow[w] = d <= 0 ? 0xFFFFFFFFu : (d > 31 ? 0u : ~((1u << d) - 1u));
        }
      }
      if (!key_live) allow[0] = allow[1] = 0u;
      const bool masked = type != kTypeFull || (code & kCodeClip) || (qb + 1) * kBlock > p.f.seqlen_orig;
      const int q_live = p.f.seqlen_orig - qb * kBlock - 64 * half;   // query rows [0, q_live) of this half exist
      if (q_live < 64) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const int d = q_live - 1 - 32 * w;
          allow[w] &= d >= 31 ? 0xFFFFFFFFu : (d < 0 ? 0u : ((2u << d) - 1u));
        }
      }

      // ---- E1: P^T -------------------------------------------------------------------------------
      const float* lse_c = lse_s + stage * kBlock + 64 * half;
      const float* del_c = delta_s + stage * kBlock + 64 * half;
      float pf[64];      // the unrounded probabilities (times the soft-cap slope, if any), kept for E2
      if constexpr (Cfg::kAhead) {
        mbar_wait_warp(bar_vec + 8 * stage, static_cast<uint32_t>((i / Cfg::kQStages) & 1), abort_flag, p.f.status, 49);
      }
      mbar_wait_warp(bar_s + 8 * (i & 1), static_cast<uint32_t>((i >> 1) & 1), abort_flag, p.f.status, 52);
      tc_fence_after();
      auto e1 = [&](auto masked_c) {
        constexpr bool kMasked = decltype(masked_c)::value;
        uint32_t rs2[2][32];
        tmem_ld32(my_s, rs2[0]);
        tmem_ld32(my_s + 32, rs2[1]);
        tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t (&rs)[32] = rs2[c];
          uint32_t pp[16];
          const uint32_t aw = allow[c];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float2 nl = *reinterpret_cast<const float2*>(lse_c + 32 * c + 2 * j);
            float2 sc = make_float2(__uint_as_float(rs[2 * j]), __uint_as_float(rs[2 * j + 1]));
            float2 slope = make_float2(1.f, 1.f);
            if constexpr (SOFTCAP) slope = bwd_soft_cap(sc, p.f.cap_in, p.f.cap_out);
            const float2 x = __ffma2_rn(sc, c2, nl);
            float2 pr = j % 8 < (SOFTCAP ? 0 : kBwdPolyOf8) ? exp2_fma2(x) : make_float2(ex2_approx(x.x), ex2_approx(x.y));
            if constexpr (kMasked) {
              pr.x = ((aw >> (2 * j)) & 1u) ? pr.x : 0.f;
              pr.y = ((aw >> (2 * j + 1)) & 1u) ? pr.y : 0.f;
            }
            pp[j] = pack2<BF16>(pr.x, pr.y);
            if constexpr (SOFTCAP) pr = __fmul2_rn(pr, slope);
            pf[32 * c + 2 * j] = pr.x;
            pf[32 * c + 2 * j + 1] = pr.y;
          }
          // P^T over this thread's S^T columns [0,32) of its half: chunk 0 has been read completely
          tmem_st16(my_s + 16 * c, pp);
        }
      };
      if (masked) {   // uniform over the compute threads
        e1(std::true_type{});
      } else {
        e1(std::false_type{});
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(bar_p + 8 * (i & 1));

      if (i + 1 < n_vis) {
        next_qb = vis_s[i + 1];
        next_code = code_s[next_qb];
      }

      // ---- E2: dS^T ------------------------------------------------------------------------------
      mbar_wait_warp(bar_dp, ph, abort_flag, p.f.status, 53);
      tc_fence_after();
      uint32_t rd2[2][32];
      tmem_ld32(my_dp, rd2[0]);
      tmem_ld32(my_dp + 32, rd2[1]);
      tc_wait_ld();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint32_t (&rd)[32] = rd2[c];
        uint32_t dd[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 nd = *reinterpret_cast<const float2*>(del_c + 32 * c + 2 * j);
          const float2 ds = __fmul2_rn(make_float2(pf[32 * c + 2 * j], pf[32 * c + 2 * j + 1]),
                                       __fadd2_rn(make_float2(__uint_as_float(rd[2 * j]), __uint_as_float(rd[2 * j + 1])),
                                                  nd));
          dd[j] = pack2<BF16>(ds.x, ds.y);
        }
        // over columns of its half that this thread has read
        tmem_st16(my_ds + 16 * c, dd);
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(bar_ds);
      if constexpr (!Cfg::kAhead) {   // this visit's vectors are free once every compute thread is through E2
        named_barrier_sync(2, kBwdComputeThreads);
        if (tid < kBlock && i + 2 < n_vis) {
          lse_s[stage * kBlock + tid] = next_lse;
          delta_s[stage * kBlock + tid] = next_delta;
        }
      }
    }
    if (n_vis > 0) {
      const int last = n_vis - 1;
      if (half == 0) {   // dV is complete before dK
        mbar_wait_warp(bar_dvdone + 8 * (last & 1), static_cast<uint32_t>((last >> 1) & 1), abort_flag, p.f.status, 54);
      } else {
        mbar_wait_warp(bar_dkdone + 8 * (last % Cfg::kQStages), static_cast<uint32_t>((last / Cfg::kQStages) & 1), abort_flag,
                       p.f.status, 54);
      }
      tc_fence_after();
    }
    const long long out_row = row0 + k_abs;
    if (half == 0) {
      bwd_store_row<D, BF16>(tdV + lane_base, n_vis > 0, 1.f, p.dv, out_row, p.f.d_real, k_abs < p.f.N);
    } else {
      bwd_store_row<D, BF16>(tdK + lane_base, n_vis > 0, p.f.scale, p.dk, out_row, p.f.d_real, k_abs < p.f.N);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

// ---------------------------------------------------------------------------------------------
// 3. dQ. One CTA per (Q block, batch*head), see bwd_decode_cta. Same roles as the dK/dV kernel
// (threads t and t + 128 own query row t, key columns [0,64) and [64,128) of the visited KV block).
// TMEM: three score regions R0, R1, R2 = [0,128), [128,256), [256,384), dQ [384,384+D). Visit i puts
// S in R(i&1) and dP in R2; dS (16-bit) goes over S. The third region is what lets the scores run
// ahead: R2 is dead once E2(i) is done and takes dP(i+1) at once, R(i&1) is free once dQ(i) has read
// dS(i) and takes S(i+2), so the tensor pipe works in the order
//   dP(i+1), dQ(i), S(i+2)
// while the compute warps do E1(i+1) (probabilities, kept in registers) under dP(i+1) and E2(i+1)
// (dS) under dQ(i) / S(i+2). K is needed by S two visits ahead and by dQ, hence a ring of three K
// tiles (two for V); with Q and dO resident that is all of an SM's shared memory at D=128, so the
// buffer is declared 1024-byte aligned instead of being aligned by hand.
// ---------------------------------------------------------------------------------------------
template <int D>
struct DqCfg {
  static constexpr int kTileBytes = kBlock * D * 2;
  static constexpr int kListBytes = kMaxKvBlocks * 2 + 16;   // visit list, its length
  static constexpr int kSmemBytes = 7 * kTileBytes + kListBytes + 256;
};

template <int D, bool BF16, bool SOFTCAP>
__device__ __forceinline__ void bwd_dq_cta(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                                           const CUtensorMap& tmdO, const BwdParams& p, int cta, uint8_t* smem) {
  using Cfg = DqCfg<D>;

  const uint32_t sQ = smem_u32(smem);
  const uint32_t sdO = sQ + Cfg::kTileBytes;
  const uint32_t sK = sdO + Cfg::kTileBytes;           // three stages
  const uint32_t sV = sK + 3 * Cfg::kTileBytes;        // two stages
  uint16_t* vis_s = reinterpret_cast<uint16_t*>(smem + 7 * Cfg::kTileBytes);   // [kMaxKvBlocks]
  int* n_vis_s = reinterpret_cast<int*>(vis_s + kMaxKvBlocks);
  uint64_t* bars = reinterpret_cast<uint64_t*>(n_vis_s + 4);
  const uint32_t bar_qdo = smem_u32(bars + 0);     // Q, dO landed
  const uint32_t bar_k = smem_u32(bars + 1);       // [3] K stage landed
  const uint32_t bar_v = smem_u32(bars + 4);       // [2] V stage landed
  const uint32_t bar_s = smem_u32(bars + 6);       // [2] S of a visit complete (by visit parity)
  const uint32_t bar_dp = smem_u32(bars + 8);      // dP of the visit complete
  const uint32_t bar_ds = smem_u32(bars + 9);      // dS stored (256 arrivals)
  const uint32_t bar_kfree = smem_u32(bars + 10);  // [3] dQ MMAs that read this K stage complete
  const uint32_t bar_vfree = smem_u32(bars + 13);  // [2] dP MMAs that read this V stage complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const bool compute = tid < kBwdComputeThreads;
  const int half = (tid >> 7) & 1;  // which 64 key columns of the tile this thread works on
  const int t = tid & 127;          // query row of the tile = TMEM lane
  const int nq = p.f.nq;
  int qb, bh;
  bwd_decode_cta(p.f, cta, true, qb, bh);

  if (tid == 0) {
    mbar_init(bar_qdo, 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(bar_k + 8 * s, 1);
      mbar_init(bar_kfree + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_v + 8 * s, 1);
      mbar_init(bar_vfree + 8 * s, 1);
      mbar_init(bar_s + 8 * s, 1);
    }
    mbar_init(bar_dp, 1);
    mbar_init(bar_ds, kBwdComputeThreads);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const uint32_t tmem_base = *tmem_slot;
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const uint32_t tdQ = tmem_base + 384;
  auto region_s = [&](int i) { return tmem_base + 128u * static_cast<uint32_t>(i & 1); };
  auto region_dp = [&](int) { return tmem_base + 256u; };
  constexpr int fmt = BF16 ? 1 : 0;
  constexpr uint32_t idesc_ss = umma_idesc_f16(128, 128, fmt, 0);
  constexpr uint32_t idesc_ts = umma_idesc_f16(128, D, fmt, 1);

  const long long row0 = static_cast<long long>(bh) * p.f.N;
  // row qb of this head's code table: the KV blocks this Q block visits, and how
  const uint32_t* codes_row = p.codes + (static_cast<long long>(bh) * nq + qb) * nq;
  if (warp == 0) {
    const int lane = tid;
    int count = 0;
    for (int base = 0; base < nq; base += 32) {
      const bool on = base + lane < nq && __ldg(codes_row + base + lane) != 0u;
      const uint32_t any = __ballot_sync(0xFFFFFFFFu, on);
      if (on) vis_s[count + __popc(any & ((1u << lane) - 1u))] = static_cast<uint16_t>(base + lane);
      count += __popc(any);
    }
    if (lane == 0) *n_vis_s = count;
  }
  __syncthreads();
  const int n_vis = *n_vis_s;

  if (warp == kBwdProducerWarp && elect_one()) {
    // =========================== TMA producer ====================================================
    if (n_vis > 0) {
      mbar_expect_tx(bar_qdo, 2 * Cfg::kTileBytes);
      const int y = qb * kBlock;
      bwd_load_tile<D>(sQ, &tmQ, bar_qdo, y, bh);
      bwd_load_tile<D>(sdO, &tmdO, bar_qdo, y, bh);
    }
    for (int j = 0; j < n_vis; ++j) {
      const int y = static_cast<int>(vis_s[j]) * kBlock;
      const int ks = j % 3, vs = j & 1;
      if (j >= 3) mbar_wait(bar_kfree + 8 * ks, static_cast<uint32_t>((j / 3 - 1) & 1), abort_flag, p.f.status, 65);
      mbar_expect_tx(bar_k + 8 * ks, Cfg::kTileBytes);
      bwd_load_tile<D>(sK + ks * Cfg::kTileBytes, &tmK, bar_k + 8 * ks, y, bh);
      if (j >= 2) mbar_wait(bar_vfree + 8 * vs, static_cast<uint32_t>(((j >> 1) - 1) & 1), abort_flag, p.f.status, 66);
      mbar_expect_tx(bar_v + 8 * vs, Cfg::kTileBytes);
      bwd_load_tile<D>(sV + vs * Cfg::kTileBytes, &tmV, bar_v + 8 * vs, y, bh);
    }
  } else if (warp == kBwdIssuerWarp && elect_one()) {
    // =========================== MMA issuer ======================================================
    auto issue_s = [&](int j) {    // S(j) = Q K(j)^T
      mbar_wait(bar_k + 8 * (j % 3), static_cast<uint32_t>((j / 3) & 1), abort_flag, p.f.status, 61);
      tc_fence_after();
      bwd_mma_ss<D>(region_s(j), sQ, sK + (j % 3) * Cfg::kTileBytes, idesc_ss);
      tc_commit(bar_s + 8 * (j & 1));
    };
    auto issue_dp = [&](int j) {   // dP(j) = dO V(j)^T
      mbar_wait(bar_v + 8 * (j & 1), static_cast<uint32_t>((j >> 1) & 1), abort_flag, p.f.status, 62);
      tc_fence_after();
      bwd_mma_ss<D>(region_dp(j), sdO, sV + (j & 1) * Cfg::kTileBytes, idesc_ss);
      tc_commit(bar_dp);
      tc_commit(bar_vfree + 8 * (j & 1));
    };
    if (n_vis > 0) {
      mbar_wait(bar_qdo, 0, abort_flag, p.f.status, 60);
      issue_s(0);
      issue_dp(0);
      if (n_vis > 1) issue_s(1);
    }
    for (int i = 0; i < n_vis; ++i) {
      mbar_wait(bar_ds, static_cast<uint32_t>(i & 1), abort_flag, p.f.status, 63);
      tc_fence_after();
      if (i + 1 < n_vis) issue_dp(i + 1);   // first: E2(i+1) is waiting for it
      bwd_mma_ts_split<D>(tdQ, region_s(i), 0, sK + (i % 3) * Cfg::kTileBytes, idesc_ts, i > 0);   // dQ += dS(i) K(i)
      tc_commit(bar_kfree + 8 * (i % 3));
      if (i + 2 < n_vis) issue_s(i + 2);
    }
    if (n_vis > 0) {
      const int last = n_vis - 1;
      mbar_wait(bar_kfree + 8 * (last % 3), static_cast<uint32_t>((last / 3) & 1), abort_flag, p.f.status, 64);
    }
  } else if (compute) {
    // =========================== per-element work ================================================
    const int q_abs = qb * kBlock + t;
    const long long my_row = row0 + q_abs;
    const bool q_live = q_abs < p.f.seqlen_orig;
    // a row beyond the sequence (or one that attended nothing) gets -LSE = -inf: every probability 0
    const float neg_lse2 = q_live ? -lse_to_log2(__ldg(p.lse + my_row)) : -INFINITY;
    const float neg_delta = q_live ? -__ldg(p.delta + my_row) : 0.f;
    const float2 c2 = make_float2(p.f.scale_log2, p.f.scale_log2);
    const float2 nl2 = make_float2(neg_lse2, neg_lse2);
    const float2 nd2 = make_float2(neg_delta, neg_delta);

    for (int i = 0; i < n_vis; ++i) {
      const int kvb = vis_s[i];
      const uint32_t code = __ldg(codes_row + kvb);
      const uint32_t my_s = region_s(i) + lane_base + 64 * half;
      const uint32_t my_dp = region_dp(i) + lane_base + 64 * half;
      const bool masked = (code & kCodeTypeMask) != kTypeFull || (code & kCodeClip);
      uint32_t allow[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
      if (masked) build_allow(p.f, code, kvb, t, allow);

      // ---- E1: probabilities (times the soft-cap slope, if any), kept in registers ---------------
      float pf[64];
      mbar_wait_warp(bar_s + 8 * (i & 1), static_cast<uint32_t>((i >> 1) & 1), abort_flag, p.f.status, 67);
      tc_fence_after();
      auto e1 = [&](auto masked_c) {
        constexpr bool kMasked = decltype(masked_c)::value;
        uint32_t rs2[2][32];
        tmem_ld32(my_s, rs2[0]);
        tmem_ld32(my_s + 32, rs2[1]);
        tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t (&rs)[32] = rs2[c];
          const uint32_t aw = allow[2 * half + c];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float2 sc = make_float2(__uint_as_float(rs[2 * j]), __uint_as_float(rs[2 * j + 1]));
            float2 slope = make_float2(1.f, 1.f);
            if constexpr (SOFTCAP) slope = bwd_soft_cap(sc, p.f.cap_in, p.f.cap_out);
            const float2 x = __ffma2_rn(sc, c2, nl2);
            float2 pr = j % 8 < (SOFTCAP ? 0 : kBwdPolyOf8) ? exp2_fma2(x) : make_float2(ex2_approx(x.x), ex2_approx(x.y));
            if constexpr (SOFTCAP) pr = __fmul2_rn(pr, slope);
            if constexpr (kMasked) {
              pr.x = ((aw >> (2 * j)) & 1u) ? pr.x : 0.f;
              pr.y = ((aw >> (2 * j + 1)) & 1u) ? pr.y : 0.f;
            }
            pf[32 * c + 2 * j] = pr.x;
            pf[32 * c + 2 * j + 1] = pr.y;
          }
        }
      };
      if (masked) {   // uniform over the compute threads
        e1(std::true_type{});
      } else {
        e1(std::false_type{});
      }

      // ---- E2: dS over this thread's S columns [0,32) of its half ---------------------------------
      mbar_wait_warp(bar_dp, static_cast<uint32_t>(i & 1), abort_flag, p.f.status, 68);
      tc_fence_after();
      uint32_t rd2[2][32];
      tmem_ld32(my_dp, rd2[0]);
      tmem_ld32(my_dp + 32, rd2[1]);
      tc_wait_ld();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint32_t (&rd)[32] = rd2[c];
        uint32_t dd[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 ds = __fmul2_rn(make_float2(pf[32 * c + 2 * j], pf[32 * c + 2 * j + 1]),
                                       __fadd2_rn(make_float2(__uint_as_float(rd[2 * j]), __uint_as_float(rd[2 * j + 1])), nd2));
          dd[j] = pack2<BF16>(ds.x, ds.y);
        }
        tmem_st16(my_s + 16 * c, dd);
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(bar_ds);
    }
    if (n_vis > 0) {
      const int last = n_vis - 1;
      mbar_wait_warp(bar_kfree + 8 * (last % 3), static_cast<uint32_t>((last / 3) & 1), abort_flag, p.f.status, 64);
      tc_fence_after();
    }
    if (half == 0) {
      bwd_store_row<D, BF16, 0, D / 64>(tdQ + lane_base, n_vis > 0, p.f.scale, p.dq, my_row, p.f.d_real, q_abs < p.f.N);
    } else {
      bwd_store_row<D, BF16, D / 64, D / 32>(tdQ + lane_base, n_vis > 0, p.f.scale, p.dq, my_row, p.f.d_real, q_abs < p.f.N);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// Both in one launch, the dK/dV CTAs first: neither needs the other's results, so the dQ CTAs fill the SMs that the
// last dK/dV ones leave idle. That is most of a wave for short batches (16 heads x 12 blocks: 1.3 waves of each, 70.6 ->
// 66.9 us with the soft-cap; 32 x 4K tokens at D = 64 369 -> 365, 32 x 8K at 128 1609 -> 1595; same bits).
template <int D, bool BF16, bool SOFTCAP>
__global__ void __launch_bounds__(kBwdThreads, 1)
omni_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_bwd[];
  if ((smem_u32(smem_bwd) & 1023u) != 0u) {   // the swizzled tile layout needs it; uniform over the CTA
    if (threadIdx.x == 0 && p.f.status != nullptr) atomicExch(p.f.status, kStatusWaitTimeout | (69 << 8));
    return;
  }
  const int ctas = p.f.nq * p.f.BH;
  const int cta = static_cast<int>(blockIdx.x);
  if (cta < ctas) {
    bwd_dkdv_cta<D, BF16, SOFTCAP>(tmQ, tmK, tmV, tmdO, p, cta, smem_bwd);
  } else {
    bwd_dq_cta<D, BF16, SOFTCAP>(tmQ, tmK, tmV, tmdO, p, cta - ctas, smem_bwd);
  }
}

template <int D, bool BF16, bool SOFTCAP>
static cudaError_t launch_bwd_t(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV,
                                const CUtensorMap& tmdO, const BwdParams& p, cudaStream_t stream) {
  constexpr int kSmem = BwdCfg<D>::kSmemBytes > DqCfg<D>::kSmemBytes ? BwdCfg<D>::kSmemBytes : DqCfg<D>::kSmemBytes;
  auto kern = omni_bwd_kernel<D, BF16, SOFTCAP>;
  static SmemAttrOnce attr[kMaxDevices];
  cudaError_t e = ensure_smem_attr(kern, kSmem, attr);
  if (e != cudaSuccess) return e;
  omni_bwd_prep_kernel<D, BF16><<<dim3(p.f.nq, p.f.BH), kPrepThreads, 0, stream>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const unsigned ctas = static_cast<unsigned>(p.f.nq) * static_cast<unsigned>(p.f.BH);
  kern<<<2 * ctas, kBwdThreads, kSmem, stream>>>(tmQ, tmK, tmV, tmdO, p);
  return cudaGetLastError();
}

cudaError_t launch_bwd(int head_dim, bool bf16, const CUtensorMap& tmQ, const CUtensorMap& tmK,
                       const CUtensorMap& tmV, const CUtensorMap& tmdO, const BwdParams& p, cudaStream_t stream) {
  const bool cap = p.f.cap_out != 0.f;
  if (head_dim == 64) {
    if (cap) {
      return bf16 ? launch_bwd_t<64, true, true>(tmQ, tmK, tmV, tmdO, p, stream)
                  : launch_bwd_t<64, false, true>(tmQ, tmK, tmV, tmdO, p, stream);
    }
    return bf16 ? launch_bwd_t<64, true, false>(tmQ, tmK, tmV, tmdO, p, stream)
                : launch_bwd_t<64, false, false>(tmQ, tmK, tmV, tmdO, p, stream);
  }
  if (cap) {
    return bf16 ? launch_bwd_t<128, true, true>(tmQ, tmK, tmV, tmdO, p, stream)
                : launch_bwd_t<128, false, true>(tmQ, tmK, tmV, tmdO, p, stream);
  }
  return bf16 ? launch_bwd_t<128, true, false>(tmQ, tmK, tmV, tmdO, p, stream)
              : launch_bwd_t<128, false, false>(tmQ, tmK, tmV, tmdO, p, stream);
}

}  // namespace omni
