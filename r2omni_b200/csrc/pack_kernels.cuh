// Quantize-and-pack kernels, bit-exact with the reference's CPU torch routines:
// IEEE divisions (__fdiv_rn), round-half-even (rintf), no fused multiply-add
// across the divide/add, steps stored as fp16 while codes use the fp32 step.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "device_utils.cuh"
#include "r2k_b200.h"

namespace r2k {

template <bool BF16>
__device__ __forceinline__ float raw_to_float(uint16_t raw) {
  if (BF16) return __uint_as_float((uint32_t)raw << 16);
  return __half2float(__ushort_as_half(raw));
}
template <bool BF16>
__device__ __forceinline__ float round_through_elem(float x) {
  if (BF16) return __bfloat162float(__float2bfloat16_rn(x));
  return __half2float(__float2half_rn(x));
}

struct PackArgs {
  const uint16_t* src;      // [B][H, src_rows, 128] 16-bit elements
  int64_t src_bstride;      // bytes
  int64_t src_rows;
  const int64_t* index;     // optional [count] source rows (shared by every request)
  int64_t count;
  int64_t capacity;         // destination rows per head
  int64_t dst_start;
  int num_heads;
  bool in_flush;            // the launch behind this one belongs to the same flush and may come in early
};

// ---- keys: per (head, block, channel) affine INT4 -------------------------
// One CTA of 64 threads per (block, head, request); thread c owns channels 2c, 2c+1.
// compact_int4_key.py:83-110 (quantiser), :210-220 (tail re-quantisation).
template <bool BF16>
__global__ void __launch_bounds__(64) pack_k_int4_kernel(PackArgs a, uint8_t* packed, __half* scale, uint8_t* zero,
                                                         int64_t packed_bstride, int64_t scale_bstride, int64_t zero_bstride,
                                                         int k_block, int64_t first_block) {
  // A flush launches the value pack behind this kernel with programmatic stream serialization: the two read
  // different halves of the residual window and write different arenas, so they may run side by side.  By itself it lets nobody
  // in: a rotation and the decode launch behind it may follow, and that one reads the pools before it waits.
  if (a.in_flush) launch_dependents();
  const int64_t blk = first_block + blockIdx.x;
  const int head = blockIdx.y, req = blockIdx.z, c = threadIdx.x;
  const int64_t blocks_per_head = a.capacity / k_block;
  const uint16_t* src = reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(a.src) + req * a.src_bstride) +
                        (int64_t)head * a.src_rows * 128;
  uint8_t* prow = packed + req * packed_bstride + ((int64_t)head * a.capacity) * 64;
  __half* srow = reinterpret_cast<__half*>(reinterpret_cast<uint8_t*>(scale) + req * scale_bstride) +
                 ((int64_t)head * blocks_per_head + blk) * 128;
  uint8_t* zrow = zero + req * zero_bstride + ((int64_t)head * blocks_per_head + blk) * 128;

  const int64_t r_begin = blk * k_block;
  const int64_t r_end = min(r_begin + (int64_t)k_block, a.dst_start + a.count);
  // rows in front of dst_start are already packed: they are re-quantised from their dequantised, element-rounded values
  const float old_s0 = __half2float(srow[2 * c]), old_s1 = __half2float(srow[2 * c + 1]);
  const float old_z0 = (float)zrow[2 * c], old_z1 = (float)zrow[2 * c + 1];

  // The block's values (raw 16-bit pairs: re-quantised rows are element-rounded, so nothing is lost) are staged in
  // shared memory by the first pass: its loads are independent and run several at a time, and the second pass
  // reads no global memory, so its stores do not wait behind loads that might alias them.
  extern __shared__ uint32_t staged_words[];   // k_block rows of 64 words (dynamic: k_block * 256 bytes)
  uint32_t (*staged)[64] = reinterpret_cast<uint32_t (*)[64]>(staged_words);
  auto fetch_raw = [&](int64_t r) -> uint32_t {
    if (r < a.dst_start) {
      const uint8_t byte = prow[r * 64 + c];
      const float x0 = __fmul_rn(__fsub_rn((float)(byte & 15), old_z0), old_s0);
      const float x1 = __fmul_rn(__fsub_rn((float)(byte >> 4), old_z1), old_s1);
      if (BF16) return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x0)) | ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x1)) << 16);
      return (uint32_t)__half_as_ushort(__float2half_rn(x0)) | ((uint32_t)__half_as_ushort(__float2half_rn(x1)) << 16);
    }
    const int64_t i = r - a.dst_start;
    const int64_t s = a.index ? a.index[i] : i;
    return *reinterpret_cast<const uint32_t*>(src + s * 128 + 2 * c);
  };

  float lo0 = INFINITY, hi0 = -INFINITY, lo1 = INFINITY, hi1 = -INFINITY;
  const int rows = (int)(r_end - r_begin);
#pragma unroll 8
  for (int i = 0; i < rows; ++i) {
    const uint32_t w = fetch_raw(r_begin + i);
    staged[i][c] = w;
    const float x0 = raw_to_float<BF16>((uint16_t)(w & 0xffffu)), x1 = raw_to_float<BF16>((uint16_t)(w >> 16));
    lo0 = fminf(lo0, x0); hi0 = fmaxf(hi0, x0);
    lo1 = fminf(lo1, x1); hi1 = fmaxf(hi1, x1);
  }
  lo0 = fminf(lo0, 0.f); hi0 = fmaxf(hi0, 0.f);
  lo1 = fminf(lo1, 0.f); hi1 = fmaxf(hi1, 0.f);
  const float st0 = fmaxf(__fdiv_rn(__fsub_rn(hi0, lo0), 15.f), 1.0e-6f);
  const float st1 = fmaxf(__fdiv_rn(__fsub_rn(hi1, lo1), 15.f), 1.0e-6f);
  const float zp0 = fminf(fmaxf(rintf(__fdiv_rn(-lo0, st0)), 0.f), 15.f);
  const float zp1 = fminf(fmaxf(rintf(__fdiv_rn(-lo1, st1)), 0.f), 15.f);
#pragma unroll 4
  for (int i = 0; i < rows; ++i) {
    const uint32_t w = staged[i][c];   // written by this very thread
    const float x0 = raw_to_float<BF16>((uint16_t)(w & 0xffffu)), x1 = raw_to_float<BF16>((uint16_t)(w >> 16));
    const float q0 = fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(x0, st0), zp0)), 0.f), 15.f);
    const float q1 = fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(x1, st1), zp1)), 0.f), 15.f);
    prow[(r_begin + i) * 64 + c] = (uint8_t)((uint32_t)q0 | ((uint32_t)q1 << 4));
  }
  srow[2 * c] = __float2half_rn(st0);
  srow[2 * c + 1] = __float2half_rn(st1);
  zrow[2 * c] = (uint8_t)zp0;
  zrow[2 * c + 1] = (uint8_t)zp1;
  if (!a.in_flush) publish_pools();   // a flush's last launch waits for this grid
}

// ---- values: one warp per (token, head, request), lane owns dims 4l..4l+3 ---
template <bool BF16>
__device__ __forceinline__ void unpack4(const uint2& w, float (&x)[4]) {
  x[0] = raw_to_float<BF16>((uint16_t)(w.x & 0xffffu)); x[1] = raw_to_float<BF16>((uint16_t)(w.x >> 16));
  x[2] = raw_to_float<BF16>((uint16_t)(w.y & 0xffffu)); x[3] = raw_to_float<BF16>((uint16_t)(w.y >> 16));
}

// Per-token symmetric INT4 (quantization.py:19-50, 77-102; fused_value_pack.py:25-70): returns the lane's two bytes.
template <bool BF16>
__device__ __forceinline__ uint16_t encode_v_int4(const uint2& w, float& sc) {
  float x[4];
  unpack4<BF16>(w, x);
  float amax = fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3])));
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
  sc = fmaxf(__fdiv_rn(amax, 7.f), 1.0e-6f);
  uint32_t out = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int q = (int)fminf(fmaxf(rintf(__fdiv_rn(x[e], sc)), -7.f), 7.f);
    out |= (uint32_t)(q & 15) << (4 * e);
  }
  return (uint16_t)out;
}

// Per-token, per-group affine INT2 (int2_reference.py:96-151; fused_value_pack.py:72-149): returns the lane's byte;
// `lanes` lanes (8, 16 or 32) share a group, its scale and its zero point.
template <bool BF16>
__device__ __forceinline__ uint8_t encode_v_int2(const uint2& w, int lanes, float& sc, float& zp) {
  float x[4];
  unpack4<BF16>(w, x);
  float lo = fminf(fminf(x[0], x[1]), fminf(x[2], x[3]));
  float hi = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
  for (int d = 1; d < lanes; d <<= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
  }
  lo = fminf(lo, 0.f);
  hi = fmaxf(hi, 0.f);
  sc = fmaxf(__fdiv_rn(__fsub_rn(hi, lo), 3.f), 1.0e-6f);
  zp = fminf(fmaxf(rintf(__fdiv_rn(-lo, sc)), 0.f), 3.f);
  uint32_t out = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t q = (uint32_t)fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(x[e], sc), zp)), 0.f), 3.f);
    out |= q << (2 * e);
  }
  return (uint8_t)out;
}

template <bool BF16>
__global__ void __launch_bounds__(128) pack_v_int4_kernel(PackArgs a, uint8_t* packed, float* scale, int64_t packed_bstride,
                                                          int64_t scale_bstride) {
  const int64_t i = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (i >= a.count) return;
  const int head = blockIdx.y, req = blockIdx.z, lane = threadIdx.x & 31;
  const int64_t s = a.index ? a.index[i] : i;
  const uint16_t* src = reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(a.src) + req * a.src_bstride) +
                        ((int64_t)head * a.src_rows + s) * 128;
  float sc;
  const uint16_t out = encode_v_int4<BF16>(*reinterpret_cast<const uint2*>(src + 4 * lane), sc);
  const int64_t row = (int64_t)head * a.capacity + a.dst_start + i;
  *reinterpret_cast<uint16_t*>(packed + req * packed_bstride + row * 64 + 2 * lane) = out;
  if (lane == 0) *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(scale) + req * scale_bstride + row * 4) = sc;
  publish_pools();
}

template <bool BF16>
__global__ void __launch_bounds__(128) pack_v_int2_kernel(PackArgs a, uint8_t* packed, __half* scale, uint8_t* zero,
                                                          int64_t packed_bstride, int64_t scale_bstride, int64_t zero_bstride,
                                                          int group) {
  if (a.in_flush) launch_dependents();   // the ring kernel follows; it waits for this grid before it touches the ring
  const int64_t i = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (i < a.count) {
    const int head = blockIdx.y, req = blockIdx.z, lane = threadIdx.x & 31;
    const int64_t s = a.index ? a.index[i] : i;
    const uint16_t* src = reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(a.src) + req * a.src_bstride) +
                          ((int64_t)head * a.src_rows + s) * 128;
    const int lanes = group / 4;  // lanes per group: 8, 16 or 32
    float sc, zp;
    const uint8_t out = encode_v_int2<BF16>(*reinterpret_cast<const uint2*>(src + 4 * lane), lanes, sc, zp);
    const int64_t row = (int64_t)head * a.capacity + a.dst_start + i;
    packed[req * packed_bstride + row * 32 + lane] = out;
    if ((lane & (lanes - 1)) == 0) {
      const int64_t m = row * (128 / group) + lane / lanes;
      reinterpret_cast<__half*>(reinterpret_cast<uint8_t*>(scale) + req * scale_bstride)[m] = __float2half_rn(sc);
      zero[req * zero_bstride + m] = (uint8_t)zp;
    }
    if (!a.in_flush) publish_pools();   // a flush's last launch waits for this grid
  }
  // In a flush this grid runs beside the key pack in front of it.  The ring kernel behind it waits for this
  // grid only, so this grid must not complete before the key pack has: every thread passes here on its way out.
  grid_dependency_wait();
}

// ---- row gather (bf16-value pool) ------------------------------------------
__global__ void __launch_bounds__(128) gather_rows_kernel(const uint16_t* src, int64_t src_rows, const int64_t* index,
                                                          int64_t count, uint16_t* dst, int64_t dst_rows, int64_t dst_start) {
  const int64_t i = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (i >= count) return;
  const int head = blockIdx.y, lane = threadIdx.x & 31;
  const int64_t s = index ? index[i] : i;
  const uint2 w = *reinterpret_cast<const uint2*>(src + ((int64_t)head * src_rows + s) * 128 + 4 * lane);
  *reinterpret_cast<uint2*>(dst + ((int64_t)head * dst_rows + dst_start + i) * 128 + 4 * lane) = w;
  publish_pools();
}

// ---- host block copy ---------------------------------------------------------
// Brings a block of page-locked, device-mapped host memory into device memory with plain loads over PCIe, 16 bytes
// per thread.  A decode launched behind it with programmatic stream serialization runs its prologue and starts
// streaming the packed pools meanwhile; it reads the block only after this grid has completed.
__global__ void __launch_bounds__(256) host_block_copy_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int n16) {
  launch_dependents();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n16) dst[i] = src[i];
}

// ---- residual ring ----------------------------------------------------------
struct RingArgs {
  uint8_t* recent_k; uint8_t* recent_v; int32_t* recent_len;
  int64_t* recent_global; int64_t* recent_logical; int64_t* recent_page_lengths;
  int64_t k_bstride, v_bstride, len_bstride, global_bstride, logical_bstride, page_bstride;
  int num_heads, capacity, page_size;
};

// One-token append (triton_fourq_splitk.py:413-447).  grid (B), block 256: K/V rows of every head, then metadata.
__global__ void append_recent_kernel(RingArgs r, const uint8_t* new_k, const uint8_t* new_v, const int64_t* idx,
                                     int64_t global_index, int64_t logical_position) {
  const int b = blockIdx.x;
  int32_t* len_ptr = reinterpret_cast<int32_t*>(reinterpret_cast<uint8_t*>(r.recent_len) + b * r.len_bstride);
  const int pos = *len_ptr;
  __syncthreads();  // everybody has read the length before thread 0 bumps it
  if (pos < r.capacity) {
    for (int i = threadIdx.x; i < r.num_heads * 16; i += blockDim.x) {  // 16-byte pieces
      const int h = i >> 4, piece = i & 15;
      const size_t s = ((size_t)b * r.num_heads + h) * 256 + 16 * piece;
      const size_t d = ((size_t)h * r.capacity + pos) * 256 + 16 * piece;
      *reinterpret_cast<uint4*>(r.recent_k + b * r.k_bstride + d) = *reinterpret_cast<const uint4*>(new_k + s);
      *reinterpret_cast<uint4*>(r.recent_v + b * r.v_bstride + d) = *reinterpret_cast<const uint4*>(new_v + s);
    }
    if (threadIdx.x == 0) {
      reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(r.recent_global) + b * r.global_bstride)[pos] = idx ? idx[2 * b] : global_index;
      reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(r.recent_logical) + b * r.logical_bstride)[pos] = idx ? idx[2 * b + 1] : logical_position;
      *len_ptr = pos + 1;
      reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(r.recent_page_lengths) + b * r.page_bstride)[pos / r.page_size] =
          pos % r.page_size + 1;
    }
  }
}

// After a flush: copy the flushed tokens' indices to the INT2 pool's metadata, slide the remaining rows
// to the front (each thread owns one 16-byte column and walks the rows in order, so overlapping
// ranges are safe), and refresh length and page lengths (dynamic_fourq_cache.py:108-117, 248-253).
__global__ void flush_ring_kernel(RingArgs r, int ring_tokens, int flush_tokens, int64_t* i2_global, int64_t* i2_logical,
                                  int64_t meta_bstride, int64_t meta_dst) {
  const int b = blockIdx.x;
  const int rest = ring_tokens - flush_tokens;
  int64_t* gl = reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(r.recent_global) + b * r.global_bstride);
  int64_t* lg = reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(r.recent_logical) + b * r.logical_bstride);
  if (i2_global != nullptr) {
    int64_t* dg = reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(i2_global) + b * meta_bstride) + meta_dst;
    int64_t* dl = reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(i2_logical) + b * meta_bstride) + meta_dst;
    for (int i = threadIdx.x; i < flush_tokens; i += blockDim.x) { dg[i] = gl[i]; dl[i] = lg[i]; }
  }
  grid_dependency_wait();   // the pack kernels read the rows that are moved and the length that is reset below
  __syncthreads();
  for (int col = threadIdx.x; col < r.num_heads * 16; col += blockDim.x) {
    const int h = col >> 4, piece = col & 15;
    uint8_t* kb = r.recent_k + b * r.k_bstride + (size_t)h * r.capacity * 256 + 16 * piece;
    uint8_t* vb = r.recent_v + b * r.v_bstride + (size_t)h * r.capacity * 256 + 16 * piece;
    for (int row = 0; row < rest; ++row) {
      *reinterpret_cast<uint4*>(kb + (size_t)row * 256) = *reinterpret_cast<const uint4*>(kb + (size_t)(row + flush_tokens) * 256);
      *reinterpret_cast<uint4*>(vb + (size_t)row * 256) = *reinterpret_cast<const uint4*>(vb + (size_t)(row + flush_tokens) * 256);
    }
  }
  if (threadIdx.x == 0) {
    for (int row = 0; row < rest; ++row) { gl[row] = gl[row + flush_tokens]; lg[row] = lg[row + flush_tokens]; }
    *reinterpret_cast<int32_t*>(reinterpret_cast<uint8_t*>(r.recent_len) + b * r.len_bstride) = rest;
    int64_t* pl = reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(r.recent_page_lengths) + b * r.page_bstride);
    for (int pg = 0; pg < r.capacity / r.page_size; ++pg) {
      const int v = rest - pg * r.page_size;
      pl[pg] = v < 0 ? 0 : (v > r.page_size ? r.page_size : v);
    }
  }
}

// ---------------------------------------------------------------------------
// Row transforms: the normalised 128-point Walsh-Hadamard transform and the multimodal rotary embedding of 16-bit
// rows of 128 channels.  fp32 arithmetic, butterflies in the reference's stage order (stride 1, 2, ..., 64), result
// rounded to the element type.
//
// Eight lanes hold a row and a warp holds four: lane s of a row owns channels 8s..8s+7 and 64+8s..64+8s+7.  Loads and
// stores are 16 bytes wide, the rotation's partner channel (d +- 64) and the butterflies of stride 1, 2, 4 and 64 are in
// the lane's own registers, and only three stages go through shuffles (12 shuffle instructions a row; one row per
// warp with four channels a lane took 24 and one table look-up per element).
// ---------------------------------------------------------------------------
struct Row16 { f32x2 x[8]; };   // channels (8s + e, 64 + 8s + e)

template <bool BF16>
__device__ __forceinline__ void unpack8(const uint4& raw, float (&x)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (BF16) {
      x[2 * i] = __uint_as_float(w[i] << 16);
      x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      x[2 * i] = f.x;
      x[2 * i + 1] = f.y;
    }
  }
}
template <bool BF16>
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  uint4 v;
  v.x = BF16 ? pack_bf16x2(x[0], x[1]) : pack_f16x2(x[0], x[1]);
  v.y = BF16 ? pack_bf16x2(x[2], x[3]) : pack_f16x2(x[2], x[3]);
  v.z = BF16 ? pack_bf16x2(x[4], x[5]) : pack_f16x2(x[4], x[5]);
  v.w = BF16 ? pack_bf16x2(x[6], x[7]) : pack_f16x2(x[6], x[7]);
  return v;
}
// 16 bytes at a pointer that is a multiple of 16 (wide) or of 8 bytes
__device__ __forceinline__ uint4 load16(const uint16_t* p, bool wide) {
  if (wide) return ld_streamed(p);   // every row is touched once
  const uint2 a = *reinterpret_cast<const uint2*>(p), b = *reinterpret_cast<const uint2*>(p + 4);
  return make_uint4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store16(uint16_t* p, const uint4& v, bool wide) {
  if (wide) { __stcs(reinterpret_cast<uint4*>(p), v); return; }
  *reinterpret_cast<uint2*>(p) = make_uint2(v.x, v.y);
  *reinterpret_cast<uint2*>(p + 4) = make_uint2(v.z, v.w);
}

// The last stage (stride 64) is left to the caller's split_scaled: its operands are the two halves of a pair.
__device__ __forceinline__ void hadamard_row(Row16& r, int s) {
  const f32x2 minus = make_f32x2(-1.f, -1.f);
#pragma unroll
  for (int span = 1; span < 8; span <<= 1) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (e & span) continue;
      const f32x2 a = r.x[e], b = r.x[e + span];
      r.x[e] = add2(a, b);
      r.x[e + span] = fma2(b, minus, a);   // a - b: the product is exact
    }
  }
#pragma unroll
  for (int sft = 1; sft < 8; sft <<= 1) {   // stride 8 * sft: own + other, or other - own
    const float sign = (s & sft) ? -1.f : 1.f;
    const f32x2 own = make_f32x2(sign, sign);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float lo, hi;
      split_f32x2(r.x[e], lo, hi);
      const f32x2 other = make_f32x2(__shfl_xor_sync(0xffffffffu, lo, sft), __shfl_xor_sync(0xffffffffu, hi, sft));
      r.x[e] = fma2(r.x[e], own, other);
    }
  }
}
__device__ __forceinline__ void split_row(const Row16& r, bool hadamard, float (&lo)[8], float (&hi)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    split_f32x2(r.x[e], lo[e], hi[e]);
    if (hadamard) {
      const f32x2 y = mul2(make_f32x2(__fadd_rn(lo[e], hi[e]), __fsub_rn(lo[e], hi[e])), make_f32x2(0.08838834764831845f, 0.08838834764831845f));
      split_f32x2(y, lo[e], hi[e]);
    }
  }
}

// In place when out == in.
template <bool BF16>
__global__ void __launch_bounds__(128) fwht128_kernel(const uint16_t* in, uint16_t* out, int64_t rows, bool wide) {
  // launched with programmatic stream serialization: only the way here overlaps the kernel in front (16384 tokens' rotation and values
  // 45.2 us as an ordinary launch, 44.0 so)
  grid_dependency_wait();
  const int64_t row = ((int64_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * 4 + ((threadIdx.x & 31) >> 3);
  const int s = threadIdx.x & 7;
  const bool valid = row < rows;   // every lane takes part in the shuffles
  uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
  if (valid) { a = load16(in + row * 128 + 8 * s, wide); b = load16(in + row * 128 + 64 + 8 * s, wide); }
  float lo[8], hi[8];
  unpack8<BF16>(a, lo);
  unpack8<BF16>(b, hi);
  Row16 r;
#pragma unroll
  for (int e = 0; e < 8; ++e) r.x[e] = make_f32x2(lo[e], hi[e]);
  hadamard_row(r, s);
  split_row(r, true, lo, hi);
  if (!valid) return;
  store16(out + row * 128 + 8 * s, pack8<BF16>(lo), wide);
  store16(out + row * 128 + 64 + 8 * s, pack8<BF16>(hi), wide);
}

// Qwen multimodal rotary embedding of the query and key rows of a step, optionally followed by the Hadamard
// transform, in one launch: row (request, head, token) of q or k, out[d] = x[d] * cos[axis(d)] + rot(x)[d] *
// sin[axis(d)] with rot(x)[d] = -x[d + 64] (d < 64), x[d - 64] (d >= 64) and axis(d) chosen by the section of d mod 64.
struct MropeArgs {
  const uint16_t* q; const uint16_t* k; uint16_t* q_out; uint16_t* k_out;
  const void* cos; const void* sin;
  int64_t cos_stride[4], sin_stride[4];   // elements: axis, request, token, channel
  int batch, hq, hkv, tokens, section0, section1, rot_dtype, hadamard;   // rot_dtype: R2K_DTYPE_* or 2 for float32
  // The whole prologue of a decode step (v != nullptr): the value rows pass through the same launch (copied, or
  // Hadamard-transformed when v_hadamard), and the three inputs may be slices of one fused projection: elements
  // between two requests' rows (a request's heads and tokens stay contiguous); the outputs are contiguous.
  const uint16_t* v; uint16_t* v_out;
  int64_t q_bstride, k_bstride, v_bstride;
  int v_hadamard;
  int heads_per_warp;     // heads a warp walks with its tokens' table rows in registers
  int wide;               // rows can be moved 16 bytes at a time
  int table_vec;          // eight channels of a table row are one or two aligned 16-byte loads of one axis
};

__device__ __forceinline__ float load_rot(const void* base, int64_t index, int dtype) {
  if (dtype == 2) return reinterpret_cast<const float*>(base)[index];
  const uint16_t raw = reinterpret_cast<const uint16_t*>(base)[index];
  return dtype == R2K_DTYPE_BF16 ? __uint_as_float((uint32_t)raw << 16) : __half2float(__ushort_as_half(raw));
}

// Channels d0..d0+7 of one (request, token)'s table row; d0 is a multiple of 8.
__device__ __forceinline__ void load_table8(const MropeArgs& a, const void* base, const int64_t (&stride)[4], int request,
                                            int token, int d0, float (&x)[8]) {
  const int64_t at = request * stride[1] + token * stride[2];
  const int sd = d0 & 63;
  if (a.table_vec) {
    const int axis = sd < a.section0 ? 0 : (sd < a.section0 + a.section1 ? 1 : 2);
    const int64_t i = at + axis * stride[0] + d0;
    if (a.rot_dtype == 2) {
      const float4* row = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + i);
      const float4 u = row[0], w = row[1];
      x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = w.x; x[5] = w.y; x[6] = w.z; x[7] = w.w;
    } else {
      const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + i);
      if (a.rot_dtype == R2K_DTYPE_BF16) unpack8<true>(u, x); else unpack8<false>(u, x);
    }
    return;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int axis = sd + e < a.section0 ? 0 : (sd + e < a.section0 + a.section1 ? 1 : 2);
    x[e] = load_rot(base, at + axis * stride[0] + (d0 + e) * stride[3], a.rot_dtype);
  }
}

// Bound by memory on a prefill: every row is read and written once, a (request, token)'s table rows are read once per
// heads_per_warp rows.  A warp takes four consecutive (request, token)s and walks heads_per_warp heads with the next
// head's rows in flight; blockIdx.y is the group of heads.  Twenty warps an SM at 94 registers: 16384 tokens of 16 + 2
// heads with the Hadamard in 39 us (151 MB of rows, 3.9 TB/s; 36 us without it), from 139 us with a row per warp.
template <bool BF16>
__global__ void __launch_bounds__(128, 5) mrope_rows_kernel(MropeArgs a) {
  // The decode launch that follows on the stream may start its CTAs and prefetch pool tiles early (it is
  // launched with programmatic stream serialization); it reads the rows written here only after its own
  // dependency wait, i.e. after this grid has completed.  It comes in behind this grid's wait: the kernel in front may have written
  // the pools, and is complete only then.  This kernel itself comes in behind a
  // projection in the same way (a batch-32 attention block 82.5 us as an ordinary launch and 79.8 so, the prefill above with its
  // value rows 45.6 and 43.7).
  grid_dependency_wait();
  launch_dependents();
  const int s = threadIdx.x & 7;
  const int64_t n = (int64_t)a.batch * a.tokens;
  const int64_t first = ((int64_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * 4;
  if (first >= n) return;
  const int64_t i = first + ((threadIdx.x & 31) >> 3);
  const bool valid = i < n;   // every lane takes part in the shuffles
  const int request = (int)((valid ? i : first) / a.tokens), token = (int)((valid ? i : first) - (int64_t)request * a.tokens);
  const int heads = a.hq + a.hkv + (a.v != nullptr ? a.hkv : 0);
  const int h_begin = blockIdx.y * a.heads_per_warp, h_end = min(h_begin + a.heads_per_warp, heads);
  // The next head's rows are in flight while one head's are worked on.
  auto locate = [&](int head, const uint16_t*& src, uint16_t*& dst) {
    const int which = head < a.hq ? 0 : (head < a.hq + a.hkv ? 1 : 2);   // query, key or value row
    const int h = which == 0 ? head : (which == 1 ? head - a.hq : head - a.hq - a.hkv);
    const int64_t in_row = ((int64_t)h * a.tokens + token) * 128 + 8 * s;
    const int64_t out_row = (((int64_t)request * (which == 0 ? a.hq : a.hkv) + h) * a.tokens + token) * 128 + 8 * s;
    src = (which == 0 ? a.q + request * a.q_bstride : which == 1 ? a.k + request * a.k_bstride : a.v + request * a.v_bstride) + in_row;
    dst = (which == 0 ? a.q_out : which == 1 ? a.k_out : a.v_out) + out_row;
  };
  const uint16_t* src;
  uint16_t* dst;
  locate(h_begin, src, dst);
  uint4 next_lo = load16(src, a.wide), next_hi = load16(src + 64, a.wide);
  f32x2 cs[8];                   // cos of (d, d + 64)
  float sin_lo[8], sin_hi[8];    // -sin of d (its partner enters negated), sin of d + 64
  if (h_begin < a.hq + a.hkv) {
    float lo[8], hi[8];
    load_table8(a, a.cos, a.cos_stride, request, token, 8 * s, lo);
    load_table8(a, a.cos, a.cos_stride, request, token, 64 + 8 * s, hi);
    load_table8(a, a.sin, a.sin_stride, request, token, 8 * s, sin_lo);
    load_table8(a, a.sin, a.sin_stride, request, token, 64 + 8 * s, sin_hi);
#pragma unroll
    for (int e = 0; e < 8; ++e) { cs[e] = make_f32x2(lo[e], hi[e]); sin_lo[e] = -sin_lo[e]; }
  }
  for (int head = h_begin; head < h_end; ++head) {
    const uint4 raw_lo = next_lo, raw_hi = next_hi;
    uint16_t* const out = dst;
    if (head + 1 < h_end) {
      locate(head + 1, src, dst);
      next_lo = load16(src, a.wide);
      next_hi = load16(src + 64, a.wide);
    }
    const bool is_value = head >= a.hq + a.hkv;
    if (is_value && !a.v_hadamard) {   // a value row that is only brought into place
      if (valid) { store16(out, raw_lo, a.wide); store16(out + 64, raw_hi, a.wide); }
      continue;
    }
    float lo[8], hi[8];
    unpack8<BF16>(raw_lo, lo);
    unpack8<BF16>(raw_hi, hi);
    Row16 x;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      x.x[e] = make_f32x2(lo[e], hi[e]);
      // the reference's compiled form of x*cos + rot*sin: one product rounded, one fused
      if (!is_value) x.x[e] = fma2(x.x[e], cs[e], make_f32x2(__fmul_rn(hi[e], sin_lo[e]), __fmul_rn(lo[e], sin_hi[e])));
    }
    const bool transform = is_value || a.hadamard;
    if (transform) hadamard_row(x, s);
    split_row(x, transform, lo, hi);
    if (valid) { store16(out, pack8<BF16>(lo), a.wide); store16(out + 64, pack8<BF16>(hi), a.wide); }
  }
}

}  // namespace r2k
