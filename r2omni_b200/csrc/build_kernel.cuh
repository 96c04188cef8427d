// A whole packed cache from one layer's keys and values in one launch (r2k_build_cache).
//
// One CTA takes 128 arena rows of one head: four warps quantise the key blocks, 32 rows each, the other four the same
// rows' values, each in the format of its pool.  Every key and value row is read once.  Further CTAs write the token
// bookkeeping and set what lies behind the last used row.  Source rows come from the page table (a page's rows are
// consecutive), so nothing per token is uploaded.  A build of 32768 tokens x 2 heads takes 56 us in all, host work included,
// where four launches over token-index arrays, a fill per arena and an upload per index array took 1.35 ms.
#pragma once

#include "pack_kernels.cuh"
#include "r2k_b200.h"

namespace r2k {

constexpr int kBuildRows = 128, kBuildThreads = 256;
constexpr int kMaxFills = 13;
constexpr int64_t kFillBytes = 16384;   // per CTA

struct BuildFill {            // `bytes` bytes at `at`, once per head
  uint8_t* at;
  int64_t stride, bytes;
  int heads, value;
};
struct BuildArgs {
  R2KBuild b;
  int active, chunks, chunk_ctas, meta_ctas, n_fills;
  BuildFill fill[kMaxFills];
};

// Page that holds row r of the pool order: the last one whose first row is at most r (pages without rows share theirs with
// the next page).  Pages are as a rule page_size long, so the search starts where r would then be and doubles its step:
// two or three loads there, and no more than twice the logarithm of the table for pages of any length (262144 pages of one token: 2.5 ms for the whole
// call, 97.9 with a walk in steps of one page).
__device__ __forceinline__ int page_of(const R2KBuild& b, int r) {
  int lo = min(r / b.page_size, b.n_pages - 1), hi = lo + 1, step = 1;   // looking for pages[lo].dst <= r < pages[hi].dst
  const int lo_dst = b.pages[lo].dst, hi_dst = b.pages[hi].dst;
  if (lo_dst > r) {
    do { hi = lo; lo = max(lo - step, 0); step *= 2; } while (b.pages[lo].dst > r);
  } else if (hi_dst <= r) {
    do { lo = hi; hi = min(hi + step, b.n_pages); step *= 2; } while (b.pages[hi].dst <= r);
  }
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (b.pages[mid].dst > r) hi = mid; else lo = mid;
  }
  return lo;
}

template <bool BF16>
__device__ __forceinline__ void build_keys(const R2KBuild& b, int chunk, int head, const int* src_row, float (*range)[128][2]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;   // warps 0-3: rows 32 warp ..
  const uint16_t* src = reinterpret_cast<const uint16_t*>(b.key) + (int64_t)head * b.rows * 128 + 4 * lane;
  uint2 w[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int s = src_row[32 * warp + i];
    // a row behind the last token counts as zeros, which the range contains anyway
    w[i] = s >= 0 ? __ldcs(reinterpret_cast<const uint2*>(src + (int64_t)s * 128)) : make_uint2(0u, 0u);
  }
  float lo[4], hi[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) lo[e] = hi[e] = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    float x[4];
    unpack4<BF16>(w[i], x);
#pragma unroll
    for (int e = 0; e < 4; ++e) { lo[e] = fminf(lo[e], x[e]); hi[e] = fmaxf(hi[e], x[e]); }
  }
  if (b.k_block > 32) {   // a block spans two or four warps
#pragma unroll
    for (int e = 0; e < 4; ++e) { range[warp][4 * lane + e][0] = lo[e]; range[warp][4 * lane + e][1] = hi[e]; }
    named_bar_sync(1, 128);
    const int n = b.k_block / 32, first = warp / n * n;
    for (int k = first; k < first + n; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) { lo[e] = fminf(lo[e], range[k][4 * lane + e][0]); hi[e] = fmaxf(hi[e], range[k][4 * lane + e][1]); }
  }
  float st[4], zp[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    st[e] = fmaxf(__fdiv_rn(__fsub_rn(hi[e], lo[e]), 15.f), 1.0e-6f);
    zp[e] = fminf(fmaxf(rintf(__fdiv_rn(-lo[e], st[e])), 0.f), 15.f);
  }
  uint8_t* prow = b.k_packed + ((int64_t)head * b.k_capacity + (int64_t)chunk * kBuildRows + 32 * warp) * 64 + 2 * lane;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (src_row[32 * warp + i] < 0) continue;
    float x[4];
    unpack4<BF16>(w[i], x);
    uint32_t out = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) out |= (uint32_t)fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(x[e], st[e]), zp[e])), 0.f), 15.f) << (4 * e);
    *reinterpret_cast<uint16_t*>(prow + i * 64) = (uint16_t)out;
  }
  const int row = chunk * kBuildRows + 32 * warp;
  if (row % b.k_block == 0 && src_row[32 * warp] >= 0) {
    const int64_t blk = (int64_t)head * (b.k_capacity / b.k_block) + row / b.k_block;
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(b.k_scale) + blk * 128 + 4 * lane) = make_uint2(pack_f16x2(st[0], st[1]), pack_f16x2(st[2], st[3]));
    *reinterpret_cast<uint32_t*>(b.k_zero + blk * 128 + 4 * lane) =
        (uint32_t)zp[0] | (uint32_t)zp[1] << 8 | (uint32_t)zp[2] << 16 | (uint32_t)zp[3] << 24;
  }
}

// BF16: the values' type; CACHE_BF16: the cache's.
template <bool BF16, bool CACHE_BF16>
__device__ __forceinline__ void build_values(const R2KBuild& b, int chunk, int head, const int* src_row) {
  const int warp = (threadIdx.x >> 5) - 4, lane = threadIdx.x & 31;
  const uint16_t* src = reinterpret_cast<const uint16_t*>(b.value) + (int64_t)head * b.rows * 128 + 4 * lane;
  const int lanes = b.v2_group / 4;
#pragma unroll 1
  for (int i0 = 0; i0 < 32; i0 += 8) {
    uint2 w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int s = src_row[32 * warp + i0 + k];
      w[k] = s >= 0 ? __ldcs(reinterpret_cast<const uint2*>(src + (int64_t)s * 128)) : make_uint2(0u, 0u);
    }
#pragma unroll 1
    for (int k = 0; k < 8; ++k) {
      if (src_row[32 * warp + i0 + k] < 0) return;
      uint2 v = w[0];
#pragma unroll
      for (int j = 0; j < 7; ++j) w[j] = w[j + 1];   // the next row moves to the front: one copy of the code for eight rows
      int row = chunk * kBuildRows + 32 * warp + i0 + k;
      if (row < b.n_fp) {
        if (BF16 != CACHE_BF16) {
          float x[4];
          unpack4<BF16>(v, x);
          v = CACHE_BF16 ? make_uint2(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3])) : make_uint2(pack_f16x2(x[0], x[1]), pack_f16x2(x[2], x[3]));
        }
        *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(b.fp_v) + ((int64_t)head * b.n_fp + row) * 128 + 4 * lane) = v;
        continue;
      }
      row -= b.n_fp;
      float sc, zp;
      if (row < b.n_i4) {
        const uint16_t out = encode_v_int4<BF16>(v, sc);
        const int64_t at = (int64_t)head * b.n_i4 + row;
        *reinterpret_cast<uint16_t*>(b.i4_packed + at * 64 + 2 * lane) = out;
        if (lane == 0) b.i4_scale[at] = sc;
        continue;
      }
      row -= b.n_i4;
      const uint8_t out = encode_v_int2<BF16>(v, lanes, sc, zp);
      const int64_t at = (int64_t)head * b.i2_capacity + row;
      b.i2_packed[at * 32 + lane] = out;
      if ((lane & (lanes - 1)) == 0) {
        const int64_t m = at * (128 / b.v2_group) + lane / lanes;
        reinterpret_cast<__half*>(b.i2_scale)[m] = __float2half_rn(sc);
        b.i2_zero[m] = (uint8_t)zp;
      }
    }
  }
}

template <bool BF16, bool VALUES_BF16>
__global__ void __launch_bounds__(kBuildThreads, 2) build_cache_kernel(const __grid_constant__ BuildArgs a) {
  __shared__ int src_row[kBuildRows];
  __shared__ float range[4][128][2];
  const R2KBuild& b = a.b;
  int cta = blockIdx.x;
  if (cta == 0 && threadIdx.x == 0) *b.recent_len = 0;
  if (cta < a.chunk_ctas) {
    const int chunk = cta % a.chunks, head = cta / a.chunks;
    if (threadIdx.x < kBuildRows) {
      const int r = chunk * kBuildRows + threadIdx.x;
      int s = -1;
      if (r < a.active) {
        const R2KPage page = b.pages[page_of(b, r)];
        s = page.src + (r - page.dst);
      }
      src_row[threadIdx.x] = s;
    }
    __syncthreads();
    if (threadIdx.x < 128) build_keys<BF16>(b, chunk, head, src_row, range);
    else build_values<VALUES_BF16, BF16>(b, chunk, head, src_row);
    return;
  }
  cta -= a.chunk_ctas;
  if (cta < a.meta_ctas) {
    int r = cta * kBuildThreads + threadIdx.x;
    if (r >= b.rows) return;
    const int i = page_of(b, r);
    const R2KPage page = b.pages[i];
    const int k = r - page.dst, s = page.src + k;
    const int64_t g = b.global_rows ? b.global_rows[s] : b.global_base[i] + k;
    const int64_t l = b.logical_rows ? b.logical_rows[s] : b.logical_base[i] + k;
    if (r < b.n_fp) { b.fp_global[r] = g; b.fp_logical[r] = l; return; }
    r -= b.n_fp;
    if (r < b.n_i4) { b.i4_global[r] = g; b.i4_logical[r] = l; return; }
    r -= b.n_i4;
    if (r < b.n_i2) { b.i2_global[r] = g; b.i2_logical[r] = l; return; }
    b.evicted_global[r - b.n_i2] = g;
    return;
  }
  cta -= a.meta_ctas;
  for (int k = 0; k < a.n_fills; ++k) {
    const BuildFill& f = a.fill[k];
    const int per_head = (int)((f.bytes + kFillBytes - 1) / kFillBytes), n = per_head * f.heads;
    if (cta >= n) { cta -= n; continue; }
    uint8_t* p = f.at + (cta / per_head) * f.stride + (int64_t)(cta % per_head) * kFillBytes;
    const int64_t left = f.bytes - (int64_t)(cta % per_head) * kFillBytes;
    const int bytes = (int)(left < kFillBytes ? left : kFillBytes);
    const int head_bytes = min(bytes, (int)((16u - (reinterpret_cast<uintptr_t>(p) & 15u)) & 15u)), words = (bytes - head_bytes) / 16;
    if ((int)threadIdx.x < head_bytes) p[threadIdx.x] = (uint8_t)f.value;
    const uint32_t v4 = (uint32_t)f.value * 0x01010101u;
    for (int i = threadIdx.x; i < words; i += kBuildThreads) reinterpret_cast<uint4*>(p + head_bytes)[i] = make_uint4(v4, v4, v4, v4);
    const int tail = head_bytes + words * 16;
    if (tail + (int)threadIdx.x < bytes) p[tail + threadIdx.x] = (uint8_t)f.value;
    return;
  }
}

}  // namespace r2k
