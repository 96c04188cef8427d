// A whole packed cache from one layer's keys and values in one launch (r2k_build_cache).
//
// One CTA takes 128 arena rows of one head, eight rows a warp: their keys first (the warps of a key block exchange their channels'
// ranges), then their values, each in the format of its pool.  Every key and value row is read once.  Further CTAs write the
// token bookkeeping and set what lies behind the last used row.  Source rows come from the page table (a page's rows are
// consecutive), so nothing per token is uploaded.
//
// Bound by the chain through a CTA (page search, rows, range, divide, 14 us from end to end) times its waves: 32768 tokens x 2 heads are
// 512 CTAs, two on an SM, 1.7 waves, 33.5 us.  The IEEE divisions (one per key and per quantised value) are about 10 us of issue of it,
// the rows' bytes 7 us at the copy rate.  With 32 rows a warp, keys and values on different warps and one value row at a time, a CTA
// took 27 us and the launch 48.  64 registers spill 52 to 56 bytes a thread; with all it wants (108, one CTA an SM) the launch takes 37.5.
#pragma once

#include "pack_kernels.cuh"
#include "r2k_b200.h"

namespace r2k {

constexpr int kBuildRows = 128, kBuildThreads = 512;
constexpr int kWarpRows = kBuildRows / (kBuildThreads / 32);   // 8
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

// A warp's rows of one tensor, four channels a lane; a row behind the last token reads as zeros.
__device__ __forceinline__ void load_rows(const void* base, int64_t rows, int head, const int* src_row, uint2 (&w)[kWarpRows]) {
  const uint16_t* src = reinterpret_cast<const uint16_t*>(base) + (int64_t)head * rows * 128 + 4 * (threadIdx.x & 31);
#pragma unroll
  for (int i = 0; i < kWarpRows; ++i) {
    const int s = src_row[i];
    w[i] = s >= 0 ? __ldcs(reinterpret_cast<const uint2*>(src + (int64_t)s * 128)) : make_uint2(0u, 0u);
  }
}

template <bool BF16>
__device__ __forceinline__ void build_keys(const R2KBuild& b, int chunk, int head, const int* src_row, const uint2 (&w)[kWarpRows],
                                           float4 (*range)[2][32]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float lo[4], hi[4];   // a range contains zero, so the zeros behind the last token change nothing
#pragma unroll
  for (int e = 0; e < 4; ++e) lo[e] = hi[e] = 0.f;
#pragma unroll
  for (int i = 0; i < kWarpRows; ++i) {
    float x[4];
    unpack4<BF16>(w[i], x);
#pragma unroll
    for (int e = 0; e < 4; ++e) { lo[e] = fminf(lo[e], x[e]); hi[e] = fmaxf(hi[e], x[e]); }
  }
  range[warp][0][lane] = make_float4(lo[0], lo[1], lo[2], lo[3]);
  range[warp][1][lane] = make_float4(hi[0], hi[1], hi[2], hi[3]);
  __syncthreads();
  const int n = b.k_block / kWarpRows, first = warp / n * n;   // the warps of this block: 4, 8 or 16
#pragma unroll 4
  for (int k = first; k < first + n; ++k) {
    const float4 l = range[k][0][lane], h = range[k][1][lane];
    lo[0] = fminf(lo[0], l.x); lo[1] = fminf(lo[1], l.y); lo[2] = fminf(lo[2], l.z); lo[3] = fminf(lo[3], l.w);
    hi[0] = fmaxf(hi[0], h.x); hi[1] = fmaxf(hi[1], h.y); hi[2] = fmaxf(hi[2], h.z); hi[3] = fmaxf(hi[3], h.w);
  }
  float st[4], zp[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    st[e] = fmaxf(__fdiv_rn(__fsub_rn(hi[e], lo[e]), 15.f), 1.0e-6f);
    zp[e] = fminf(fmaxf(rintf(__fdiv_rn(-lo[e], st[e])), 0.f), 15.f);
  }
  const int row = chunk * kBuildRows + kWarpRows * warp;
  uint8_t* prow = b.k_packed + ((int64_t)head * b.k_capacity + row) * 64 + 2 * lane;
#pragma unroll
  for (int i = 0; i < kWarpRows; ++i) {
    if (src_row[i] < 0) continue;
    float x[4];
    unpack4<BF16>(w[i], x);
    uint32_t out = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) out |= (uint32_t)fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(x[e], st[e]), zp[e])), 0.f), 15.f) << (4 * e);
    *reinterpret_cast<uint16_t*>(prow + i * 64) = (uint16_t)out;
  }
  if (warp == first && src_row[0] >= 0) {
    const int64_t blk = (int64_t)head * (b.k_capacity / b.k_block) + row / b.k_block;
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(b.k_scale) + blk * 128 + 4 * lane) = make_uint2(pack_f16x2(st[0], st[1]), pack_f16x2(st[2], st[3]));
    *reinterpret_cast<uint32_t*>(b.k_zero + blk * 128 + 4 * lane) =
        (uint32_t)zp[0] | (uint32_t)zp[1] << 8 | (uint32_t)zp[2] << 16 | (uint32_t)zp[3] << 24;
  }
}

// One value row: `row` counts in its pool.  BF16: the values' type; CACHE_BF16: the cache's.
template <bool BF16, bool CACHE_BF16>
__device__ __forceinline__ void build_value_fp(const R2KBuild& b, int head, int row, uint2 v) {
  const int lane = threadIdx.x & 31;
  if (BF16 != CACHE_BF16) {
    float x[4];
    unpack4<BF16>(v, x);
    v = CACHE_BF16 ? make_uint2(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3])) : make_uint2(pack_f16x2(x[0], x[1]), pack_f16x2(x[2], x[3]));
  }
  *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(b.fp_v) + ((int64_t)head * b.n_fp + row) * 128 + 4 * lane) = v;
}
template <bool BF16>
__device__ __forceinline__ void build_value_int4(const R2KBuild& b, int head, int row, const uint2& v) {
  const int lane = threadIdx.x & 31;
  float sc;
  const uint16_t out = encode_v_int4<BF16>(v, sc);
  const int64_t at = (int64_t)head * b.n_i4 + row;
  *reinterpret_cast<uint16_t*>(b.i4_packed + at * 64 + 2 * lane) = out;
  if (lane == 0) b.i4_scale[at] = sc;
}
template <bool BF16>
__device__ __forceinline__ void build_value_int2(const R2KBuild& b, int head, int row, const uint2& v) {
  const int lane = threadIdx.x & 31, lanes = b.v2_group / 4;
  float sc, zp;
  const uint8_t out = encode_v_int2<BF16>(v, lanes, sc, zp);
  const int64_t at = (int64_t)head * b.i2_capacity + row;
  b.i2_packed[at * 32 + lane] = out;
  if ((lane & (lanes - 1)) == 0) {
    const int64_t m = at * (128 / b.v2_group) + lane / lanes;
    reinterpret_cast<__half*>(b.i2_scale)[m] = __float2half_rn(sc);
    b.i2_zero[m] = (uint8_t)zp;
  }
}

// A warp whose rows are all of one pool (all but those at a pool's ends) works on them side by side: a row alone is a chain of
// shuffles and divisions.
template <bool BF16, bool CACHE_BF16>
__device__ __forceinline__ void build_values(const R2KBuild& b, int chunk, int head, const int* src_row, const uint2 (&w)[kWarpRows]) {
  const int row = chunk * kBuildRows + kWarpRows * (int)(threadIdx.x >> 5), i4 = row - b.n_fp, i2 = i4 - b.n_i4;
  const bool whole = src_row[kWarpRows - 1] >= 0;   // rows behind the last token come last
  if (whole && i4 + kWarpRows <= 0) {
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i) build_value_fp<BF16, CACHE_BF16>(b, head, row + i, w[i]);
  } else if (whole && i4 >= 0 && i2 + kWarpRows <= 0) {
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i) build_value_int4<BF16>(b, head, i4 + i, w[i]);
  } else if (whole && i2 >= 0) {
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i) build_value_int2<BF16>(b, head, i2 + i, w[i]);
  } else {
    uint2 v[kWarpRows];
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i) v[i] = w[i];
#pragma unroll 1
    for (int i = 0; i < kWarpRows && src_row[i] >= 0; ++i) {
      if (i4 + i < 0) build_value_fp<BF16, CACHE_BF16>(b, head, row + i, v[0]);
      else if (i2 + i < 0) build_value_int4<BF16>(b, head, i4 + i, v[0]);
      else build_value_int2<BF16>(b, head, i2 + i, v[0]);
#pragma unroll
      for (int j = 0; j < kWarpRows - 1; ++j) v[j] = v[j + 1];   // the next row moves to the front: one copy of the code
    }
  }
}

template <bool BF16, bool VALUES_BF16>
__global__ void __launch_bounds__(kBuildThreads, 2) build_cache_kernel(const __grid_constant__ BuildArgs a) {
  __shared__ int src_row[kBuildRows];
  __shared__ float4 range[kBuildThreads / 32][2][32];
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
    const int* mine = src_row + kWarpRows * (threadIdx.x >> 5);
    uint2 k[kWarpRows], v[kWarpRows];
    load_rows(b.key, b.rows, head, mine, k);
    load_rows(b.value, b.rows, head, mine, v);   // on their way beside the keys' arithmetic
    build_keys<BF16>(b, chunk, head, mine, k, range);
    build_values<VALUES_BF16, BF16>(b, chunk, head, mine, v);
    publish_pools();
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
    publish_pools();
    return;
  }
}

}  // namespace r2k
