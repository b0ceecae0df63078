// Block-mask construction on the GPU from modality (image span) positions.
//
// Replaces the host-side builder create_omni_block_mask_from_modality_positions
// (omni-attn-mma/omni_attn_torch.py:1518-1736), which walks every (Q block, KV block) pair in Python,
// materialises the dense [B, N, N] mask of transfusion_pytorch/transfusion.py:496-515
// (causal | any_m(q >= offset_m & k < offset_m + length_m)) and cuts the PARTIAL tiles out of it
// (build_partial_block_data, omni_attn_torch.py:148-205).
//
// Here nothing N x N is ever built. Under that rule every query row q attends one contiguous key
// range [0, limit(q)], limit(q) = max(q, max over spans with offset <= q of offset + length - 1),
// clipped to the unpadded length. A (Q block, KV block) tile is therefore fully described by the
// smallest and largest limit of the block's 128 rows:
//     all keys allowed for all rows  -> FULL          no key allowed for any row -> not listed
//     diagonal tile of a block whose rows are all plain causal rows (no row inside a span) -> CAUSAL
//     anything else -> PARTIAL, element (r, c) allowed iff c <= limit(r) - 128 * kv_block
// which is the block-type derivation of omni-attn-mma/generate_attn_data.py:200-236 applied to the
// dense rule. PARTIAL tiles are written bit-packed ([P,128,4] words) and, optionally, in the
// reference's byte-per-element form; the pool is shared by all heads of a batch element.
//
// limit(q) never decreases inside the sequence, so the limits of a block are those of its first and last
// row, the listed KV blocks are 0 .. limit_max / 128, the first (limit_min + 1) / 128 of them FULL, and
// everything there is to know about a Q block takes one pass over the spans. For few blocks one kernel therefore
// does it all: a CTA works out its own Q block and, for the position of its PARTIAL tiles in the pool, the
// PARTIAL counts of all Q blocks before it (the counts of a thread's share of them, summed over the CTA),
// writes its pool tiles and the lists of a slice of the heads. That counting grows with the square of the number of
// Q blocks in the batch; where it would take longer than two small launches (see count_first) the blocks are
// counted once and the counts summed up in the caller's scratch first. HBM-write bound for long sequences (the index
// tensors: 101 MB for a 4 x 32-head batch of 32K tokens), launch latency for short ones.
#include <cstdint>

#include "../../include/omni_attn_sm100.h"
#include "omni_common.cuh"

namespace omni {
namespace {

constexpr int kMaskThreads = 128;

struct MaskParams {
  const int32_t* modality_positions;  // [B, M, 3] (type, offset, length)
  int32_t* kv_num_blocks;             // [B, H, nq]
  int32_t* kv_indices;                // [B, H, nq, nq]
  int32_t* block_mask_types;          // [B, H, nq, nq]
  int32_t* partial_idx;               // [B, H, nq, nq]
  uint32_t* partial_bits;             // [capacity, 128, 4]
  uint8_t* partial_bool;              // [capacity, 128, 128] or null
  int32_t* num_partial_out;           // device int
  int32_t* counts;                    // [B, nq] PARTIAL tiles of each Q block, and
  int32_t* bases;                     // [B, nq] of all before it; null when every CTA counts for itself
  int B, M, H, seqlen, nq, capacity;
  int heads_per_cta;                  // heads whose lists one CTA writes (grid z = slices of the heads)
  bool vec4;                          // list rows are 16-byte aligned
};

// limit of row q (-1 = the row attends nothing)
__device__ __forceinline__ int row_limit(const MaskParams& p, int b, int q) {
  if (q >= p.seqlen) return -1;
  int lim = q;
  const int32_t* m = p.modality_positions + static_cast<long long>(b) * p.M * 3;
  for (int i = 0; i < p.M; ++i) {
    const int off = __ldg(m + 3 * i + 1);
    const int len = __ldg(m + 3 * i + 2);
    if (len > 0 && q >= off) lim = max(lim, off + len - 1);
  }
  return min(lim, p.seqlen - 1);
}

// One Q block: KV blocks [0, n_full) are FULL, [n_full, n_listed) PARTIAL, except that the diagonal one is
// CAUSAL when every row of the block is a plain causal row (no row inside a span).
struct BlockShape {
  int n_full, n_listed;
  bool causal_diag;
  __device__ __forceinline__ bool diag_in_range(int qb) const { return causal_diag && qb >= n_full && qb < n_listed; }
  __device__ __forceinline__ int partials(int qb) const { return max(0, n_listed - n_full) - (diag_in_range(qb) ? 1 : 0); }
};

__device__ __forceinline__ BlockShape block_shape(const MaskParams& p, int b, int qb) {
  const int q0 = qb * kBlock, q1 = q0 + kBlock - 1;
  const int last = min(q1, p.seqlen - 1);   // last row of the block that exists
  int lim0 = q0, lim1 = last;
  bool causal = q1 < p.seqlen;
  const int32_t* m = p.modality_positions + static_cast<long long>(b) * p.M * 3;
  for (int i = 0; i < p.M; ++i) {
    const int off = __ldg(m + 3 * i + 1);
    const int len = __ldg(m + 3 * i + 2);
    if (len <= 0) continue;
    if (q0 >= off) lim0 = max(lim0, off + len - 1);
    if (last >= off) lim1 = max(lim1, off + len - 1);
    if (max(off, q0) <= min(off + len - 1, q1)) causal = false;
  }
  const int lim_min = q1 < p.seqlen ? min(lim0, p.seqlen - 1) : -1;         // rows past the end attend nothing
  const int lim_max = q0 < p.seqlen ? min(lim1, p.seqlen - 1) : -1;
  BlockShape s;
  s.n_full = (lim_min + 1) / kBlock;
  s.n_listed = lim_max < 0 ? 0 : lim_max / kBlock + 1;
  s.causal_diag = causal;
  return s;
}

__global__ void __launch_bounds__(kMaskThreads) mask_count_kernel(const MaskParams p) {
  const int i = blockIdx.x * kMaskThreads + threadIdx.x;
  if (i < p.B * p.nq) p.counts[i] = block_shape(p, i / p.nq, i % p.nq).partials(i % p.nq);
}

// Exclusive prefix sums of the counts, one CTA: each thread sums a run of neighbours, then writes their bases.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) mask_scan_kernel(const MaskParams p) {
  __shared__ int warp_sum[kScanThreads / 32];
  const int t = threadIdx.x, n = p.B * p.nq;
  const int run = (n + kScanThreads - 1) / kScanThreads;
  const int first = min(n, t * run), last = min(n, first + run);
  int sum = 0;
  for (int i = first; i < last; ++i) sum += p.counts[i];
  int upto = sum;   // of the threads up to this one
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xFFFFFFFFu, upto, o);
    if ((t & 31) >= o) upto += x;
  }
  if ((t & 31) == 31) warp_sum[t >> 5] = upto;
  __syncthreads();
  int base = upto - sum;
  for (int w = 0; w < (t >> 5); ++w) base += warp_sum[w];
  for (int i = first; i < last; ++i) {
    p.bases[i] = base;
    base += p.counts[i];
  }
}

__global__ void __launch_bounds__(kMaskThreads) mask_build_kernel(const MaskParams p) {
  __shared__ int part[kMaskThreads / 32];
  const int qb = blockIdx.x, b = blockIdx.y, t = threadIdx.x;
  const BlockShape own = block_shape(p, b, qb);

  // pool position of this block's first PARTIAL tile
  const int me = b * p.nq + qb;
  int base;
  if (p.bases != nullptr) {
    base = p.bases[me];
  } else {
    int before = 0;
    for (int i = t; i < me; i += kMaskThreads) before += block_shape(p, i / p.nq, i % p.nq).partials(i % p.nq);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
    if ((t & 31) == 0) part[t >> 5] = before;
    __syncthreads();
    base = part[0] + part[1] + part[2] + part[3];
  }
  const bool diag = own.diag_in_range(qb);

  if (blockIdx.z == 0) {   // the pool, shared by the heads: thread t writes row t of every PARTIAL tile
    const int lim = row_limit(p, b, qb * kBlock + t);
    int pool = base;
    for (int kb = own.n_full; kb < own.n_listed; ++kb) {
      if (diag && kb == qb) continue;
      const int slot = pool++;
      if (slot >= p.capacity) break;   // reported through num_partial_out > capacity
      const int cnt = min(max(lim + 1 - kb * kBlock, 0), kBlock);   // allowed columns of this row
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int d = cnt - 32 * j;
        w[j] = d >= 32 ? 0xFFFFFFFFu : (d <= 0 ? 0u : ((1u << d) - 1u));
      }
      reinterpret_cast<uint4*>(p.partial_bits)[static_cast<size_t>(slot) * kBlock + t] = make_uint4(w[0], w[1], w[2], w[3]);
      if (p.partial_bool != nullptr) {
        uint4* dst = reinterpret_cast<uint4*>(p.partial_bool + (static_cast<size_t>(slot) * kBlock + t) * kBlock);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int c0 = 16 * j + 4 * k;
            x[k] = (c0 < cnt ? 1u : 0u) | (c0 + 1 < cnt ? 0x100u : 0u) | (c0 + 2 < cnt ? 0x10000u : 0u) |
                   (c0 + 3 < cnt ? 0x1000000u : 0u);
          }
          dst[j] = make_uint4(x[0], x[1], x[2], x[3]);
        }
      }
    }
    if (t == 0 && me == p.B * p.nq - 1) *p.num_partial_out = base + own.partials(qb);
  }

  // the lists, for this CTA's heads
  const int h0 = blockIdx.z * p.heads_per_cta, h1 = min(p.H, h0 + p.heads_per_cta);
  auto entry = [&](int i, int& idx, int& typ, int& pi) {
    const bool listed = i < own.n_listed;
    const bool part_tile = listed && i >= own.n_full && !(diag && i == qb);
    idx = listed ? i : 0;
    typ = !listed ? kTypeMasked : (i < own.n_full ? kTypeFull : (part_tile ? kTypePartial : kTypeCausal));
    pi = part_tile ? base + (i - own.n_full) - (diag && i > qb ? 1 : 0) : -1;
  };
  const long long head_stride = static_cast<long long>(p.nq) * p.nq;
  const long long row0 = (static_cast<long long>(b) * p.H * p.nq + qb) * p.nq;
  if (p.vec4) {
    for (int i = 4 * t; i < p.nq; i += 4 * kMaskThreads) {
      int4 idx, typ, pi;
      entry(i, idx.x, typ.x, pi.x);
      entry(i + 1, idx.y, typ.y, pi.y);
      entry(i + 2, idx.z, typ.z, pi.z);
      entry(i + 3, idx.w, typ.w, pi.w);
      for (int h = h0; h < h1; ++h) {
        const long long at = row0 + h * head_stride + i;
        *reinterpret_cast<int4*>(p.kv_indices + at) = idx;
        *reinterpret_cast<int4*>(p.block_mask_types + at) = typ;
        *reinterpret_cast<int4*>(p.partial_idx + at) = pi;
      }
    }
  } else {
    for (int i = t; i < p.nq; i += kMaskThreads) {
      int idx, typ, pi;
      entry(i, idx, typ, pi);
      for (int h = h0; h < h1; ++h) {
        const long long at = row0 + h * head_stride + i;
        p.kv_indices[at] = idx;
        p.block_mask_types[at] = typ;
        p.partial_idx[at] = pi;
      }
    }
  }
  for (int h = h0 + t; h < h1; h += kMaskThreads) p.kv_num_blocks[(static_cast<long long>(b) * p.H + h) * p.nq + qb] = own.n_listed;
}

// Whether the Q blocks are counted once, by kernels of their own, instead of by every CTA that comes after them. What the
// CTAs do together is half the square of the blocks, times the spans (and about four spans' worth for the rest), times the
// slices of the heads, at 1.2 span visits a nanosecond; the two kernels cost 5 to 8 us. Without : with them, us, at 8
// heads: 8 x 8K tokens and 16 spans (2.6e6 visits) 10 : 15, 16 x 8K, 6 (5e6) 12 : 15, 16 x 8K, 16 (10e6) 19 : 17, 4 x 32K,
// 16, at 32 heads (10e6, counted under the writes) 22 : 30, 32 x 8K, 16 (42e6) 45 : 19, 16 x 32K, 60 (537e6) 425 : 57.
constexpr double kCountVisits = 16e6;
bool count_first(long long blocks, int M, int slices) {
  return 0.5 * static_cast<double>(blocks) * static_cast<double>(blocks) * (M + 4.0) * slices > kCountVisits;
}

}  // namespace
}  // namespace omni

extern "C" int omni_attn_build_mask_sm100(const int32_t* modality_positions, int B, int M, int H, int seqlen,
                                          int seqlen_padded, int32_t* kv_num_blocks, int32_t* kv_indices,
                                          int32_t* block_mask_types, int32_t* partial_idx, uint32_t* partial_bits,
                                          uint8_t* partial_bool_or_null, int partial_capacity,
                                          int32_t* num_partial_out, void* scratch, long long scratch_bytes,
                                          void* cuda_stream) {
  using namespace omni;
  if (kv_num_blocks == nullptr || kv_indices == nullptr || block_mask_types == nullptr || partial_idx == nullptr ||
      num_partial_out == nullptr || scratch == nullptr || (M > 0 && modality_positions == nullptr) ||
      (partial_capacity > 0 && partial_bits == nullptr)) {
    return OMNI_ERR_NULL_POINTER;
  }
  if (B <= 0 || H <= 0 || M < 0 || B > 65535) return OMNI_ERR_SHAPE;
  if (seqlen_padded <= 0 || seqlen_padded % kBlock != 0 || seqlen <= 0 || seqlen > seqlen_padded) return OMNI_ERR_SEQLEN;
  const int nq = seqlen_padded / kBlock;
  if (nq > 1024) return OMNI_ERR_TOO_LONG;
  if (partial_capacity < 0) return OMNI_ERR_PARTIAL;
  if (scratch_bytes < 2LL * B * nq * static_cast<long long>(sizeof(int32_t))) return OMNI_ERR_SCRATCH;
  if ((reinterpret_cast<uintptr_t>(partial_bits) & 15u) || (reinterpret_cast<uintptr_t>(partial_bool_or_null) & 15u)) {
    return OMNI_ERR_ALIGNMENT;
  }
  MaskParams p;
  p.modality_positions = modality_positions;
  p.kv_num_blocks = kv_num_blocks;
  p.kv_indices = kv_indices;
  p.block_mask_types = block_mask_types;
  p.partial_idx = partial_idx;
  p.partial_bits = partial_bits;
  p.partial_bool = partial_bool_or_null;
  p.num_partial_out = num_partial_out;
  p.B = B; p.M = M; p.H = H; p.seqlen = seqlen; p.nq = nq; p.capacity = partial_capacity;
  const uintptr_t lists = reinterpret_cast<uintptr_t>(kv_indices) | reinterpret_cast<uintptr_t>(block_mask_types) |
                          reinterpret_cast<uintptr_t>(partial_idx);
  p.vec4 = nq % 4 == 0 && (lists & 15u) == 0;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  // Slices of the heads: enough CTAs to keep the memory system busy with a few (batch, Q block) pairs, but no
  // more than that, since every slice repeats the counting of the blocks before its own.
  const long long blocks = static_cast<long long>(nq) * B;
  int slices = static_cast<int>(blocks >= 592 ? 1 : 592 / blocks);
  if (slices > H) slices = H;
  p.heads_per_cta = (H + slices - 1) / slices;
  const dim3 grid(nq, B, (H + p.heads_per_cta - 1) / p.heads_per_cta);
  p.counts = p.bases = nullptr;
  if (count_first(blocks, M, static_cast<int>(grid.z))) {
    p.counts = static_cast<int32_t*>(scratch);
    p.bases = p.counts + blocks;
    mask_count_kernel<<<static_cast<unsigned>((blocks + kMaskThreads - 1) / kMaskThreads), kMaskThreads, 0, st>>>(p);
    mask_scan_kernel<<<1, kScanThreads, 0, st>>>(p);
  }
  mask_build_kernel<<<grid, kMaskThreads, 0, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? OMNI_OK : OMNI_ERR_CUDA;
}
