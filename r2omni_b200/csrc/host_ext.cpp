// Native host side of the operator API: what a Python caller pays for on every decode step and on every cache build.
//
// The work itself is behind the C ABI (r2k_b200.h); this module checks torch tensors, makes the tensors of a cache and
// fills the argument blocks.  A decode step through Python and ctypes cost 5.4 us of host time (7.0 with an append) around a
// launch that takes 2.2, a cache build 1.3 ms around 50 us of kernels.
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cstring>
#include <optional>
#include <string>
#include <vector>

#include "r2k_b200.h"

namespace {

void check(int status, const char* what) {
  if (status == R2K_OK) return;
  const std::string message = std::string(what) + ": " + r2k_status_string(status);
  if (status == R2K_ERR_GEOMETRY || status == R2K_ERR_ALIGNMENT || status == R2K_ERR_NULL || status == R2K_ERR_EMPTY)
    throw py::value_error(message);
  throw std::runtime_error(message);
}

int dtype_code(at::ScalarType t) {
  if (t == at::kBFloat16) return R2K_DTYPE_BF16;
  if (t == at::kHalf) return R2K_DTYPE_FP16;
  throw py::value_error("the packed-KV path stores bfloat16 or float16 keys/values");
}

// ---------------------------------------------------------------------------
// decode step
// ---------------------------------------------------------------------------
// Everything about an executor's launch that does not change from step to step: copies of its geometry and of the cache's
// addresses (the Python side makes a new Step when these are taken again), and the workspace, kept alive.  The output tensor
// and the flags are the caller's to change and come with every call.
struct Step {
  R2KGeom geom;
  R2KCacheView view;
  void* workspace;
  size_t workspace_bytes;
  at::Tensor buffer;
  at::ScalarType dtype;
  c10::Device device;
  int64_t batch, heads, kv_numel;

  Step(uintptr_t geom_, uintptr_t view_, const at::Tensor& buffer_, const at::Tensor& like)
      : geom(*reinterpret_cast<const R2KGeom*>(geom_)), view(*reinterpret_cast<const R2KCacheView*>(view_)), workspace(buffer_.data_ptr()),
        workspace_bytes((size_t)buffer_.numel()), buffer(buffer_), dtype(like.scalar_type()), device(like.device()),
        batch(geom.batch), heads(geom.num_q_heads), kv_numel((int64_t)geom.batch * geom.num_kv_heads * 128) {}

  // ap filled from (k, v); the indices are the caller's business
  void rows(R2KAppend& ap, const at::Tensor& k, const at::Tensor& v) const {
    if (k.numel() != kv_numel || v.numel() != kv_numel || k.device() != device || v.device() != device || !k.is_contiguous() ||
        !v.is_contiguous() || k.scalar_type() != dtype || v.scalar_type() != dtype)
      throw py::value_error("append K/V must be contiguous [B,Hkv,1,D] or [B,Hkv,D]");
    ap.k = k.data_ptr();
    ap.v = v.data_ptr();
  }

  void launch(const at::Tensor& query, const R2KAppend* ap, const at::Tensor& output, uint32_t flags, int32_t n_i2) const {
    const bool four = query.dim() == 4 && query.size(2) == 1;   // [B,Hq,1,128]
    if (query.dim() == 4 && query.size(2) > 1) return launch(query.select(2, 0), ap, output, flags, n_i2);   // its first token's rows
    if (!((query.dim() == 3 && query.size(2) == 128) || (four && query.size(3) == 128)) || query.size(0) != batch ||
        query.size(1) != heads || query.device() != device || query.scalar_type() != dtype || !query.is_contiguous())
      throw py::value_error("query does not match prepared split-K executor");
    if (output.numel() != batch * heads * 128 || output.scalar_type() != at::kBFloat16 || output.device() != device || !output.is_contiguous())
      throw py::value_error("workspace output does not match prepared split-K executor");
    R2KGeom now = geom;
    now.n_i2 = n_i2;   // the only extent that moves during generation (flushes)
    const int status = r2k_decode(&now, &view, query.data_ptr(), ap, workspace, workspace_bytes, output.data_ptr(), flags,
                                  at::cuda::getCurrentCUDAStream(device.index()).stream());
    if (status != R2K_OK) check(status, "r2k_decode");
  }
  void plain(const at::Tensor& query, const at::Tensor& output, uint32_t flags, int32_t n_i2) const {
    launch(query, nullptr, output, flags, n_i2);
  }
  void append(const at::Tensor& query, const at::Tensor& k, const at::Tensor& v, int64_t global_index, int64_t logical_position,
              const at::Tensor& output, uint32_t flags, int32_t n_i2) const {
    R2KAppend ap{};
    rows(ap, k, v);
    ap.global_index = global_index;
    ap.logical_position = logical_position;
    launch(query, &ap, output, flags, n_i2);
  }
};

// ---------------------------------------------------------------------------
// cache build
// ---------------------------------------------------------------------------
// The tensors of one cache share one allocation: offsets are handed out first, then the tensors are made over the storage.
struct Slab {
  struct Piece { at::ScalarType type; std::vector<int64_t> shape; int64_t offset; };
  std::vector<Piece> pieces;
  int64_t bytes = 0;
  size_t add(at::ScalarType type, std::vector<int64_t> shape) {
    int64_t n = (int64_t)c10::elementSize(type);
    for (int64_t s : shape) n *= s;
    pieces.push_back({type, std::move(shape), bytes});
    bytes += (n + 255) / 256 * 256;
    return pieces.size() - 1;
  }
  std::vector<at::Tensor> make(c10::Device device) {
    at::Tensor base = at::empty({bytes > 0 ? bytes : 1}, at::TensorOptions().dtype(at::kByte).device(device));
    std::vector<at::Tensor> out;
    out.reserve(pieces.size());
    for (const Piece& p : pieces) {
      at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(base.storage()), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                              c10::scalarTypeToTypeMeta(p.type));
      t.unsafeGetTensorImpl()->set_storage_offset(p.offset / (int64_t)c10::elementSize(p.type));
      t.unsafeGetTensorImpl()->set_sizes_contiguous(p.shape);
      out.push_back(std::move(t));
    }
    return out;
  }
};

at::Tensor host_i64(const at::Tensor& t) {
  return t.device().is_cpu() && t.scalar_type() == at::kLong && t.is_contiguous() ? t : t.to(at::kCPU, at::kLong).contiguous();
}

inline int64_t ceil_to(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// Tier of a page class: 0 bf16, 1 INT4, 2 INT2 values, 3 evicted (precision_pool.py:611-669; classes of PageClass).
inline int tier_of(int64_t cls) { return cls == 1 || cls == 3 || cls == 4 ? 0 : cls == 2 ? 1 : cls == 5 ? 2 : 3; }

// Bits in which p[0..n) differs from p[0], p[0] + 1, ...: zero for consecutive values.  Every token's two indices pass here on each
// build: at one 64-bit word a step, two fifths of the host time of a 32768-token build.  Its 65536 indices take 5 us with the clones
// that an x86 host has, 20 with the vectors that every host has.
#if defined(__x86_64__) && defined(__GNUC__) && !defined(__clang__)
__attribute__((target_clones("avx512f", "avx2", "default")))
#endif
uint64_t off_ramp(const int64_t* p, int64_t n) {
  const uint64_t first = (uint64_t)p[0];
  uint64_t odd = 0;
  for (int64_t k = 0; k < n; ++k) odd |= ((uint64_t)p[k] - first) ^ (uint64_t)k;
  return odd;
}

// build_three_precision_cache behind its argument checks.  Returns (tensors in the order of `names` on the Python side,
// n_fp, n_i4, n_i2).
std::tuple<std::vector<at::Tensor>, int64_t, int64_t, int64_t> build_cache(
    const at::Tensor& key, const at::Tensor& value, const at::Tensor& page_classes, const at::Tensor& page_offsets,
    const at::Tensor& page_lengths, const at::Tensor& global_index, const at::Tensor& logical_position,
    int64_t page_size, int64_t k_block, int64_t v2_group, int64_t recent_capacity, int64_t append_capacity) {
  const c10::cuda::CUDAGuard guard(key.device());
  const int64_t h = key.size(0), rows = key.size(1), d = 128;
  if (value.device() != key.device()) throw py::value_error("key/value must share a device");
  const int key_type = dtype_code(key.scalar_type()), value_type = dtype_code(value.scalar_type());
  const int dtype = key_type == value_type ? key_type : key_type | R2K_BUILD_OTHER_VALUES;
  const at::Tensor cls_t = host_i64(page_classes), off_t = host_i64(page_offsets), len_t = host_i64(page_lengths);
  const int64_t n = cls_t.numel();
  if (off_t.numel() != n || len_t.numel() != n) throw py::value_error("page table columns differ in length");
  const int64_t *cls = cls_t.data_ptr<int64_t>(), *off = off_t.data_ptr<int64_t>(), *len = len_t.data_ptr<int64_t>();
  int64_t tokens[4] = {0, 0, 0, 0}, total = 0;
  for (int64_t i = 0; i < n; ++i) {
    if (len[i] == 0) continue;   // its place is of no consequence
    if (len[i] < 0 || off[i] < 0 || len[i] > rows || off[i] > rows - len[i]) throw py::value_error("page lies outside the keys and values");
    tokens[tier_of(cls[i])] += len[i];
    total += len[i];
  }
  if (total != rows) throw py::value_error("compact physical pools must cover every logical token");
  if (rows > (int64_t)1 << 30) throw py::value_error("too many tokens for one cache");

  // token bookkeeping: one value per page where a page's tokens are consecutive (the ordinary case), else whole arrays
  at::Tensor global = global_index, logical = logical_position;
  if (global.numel() < rows || logical.numel() < rows) throw py::value_error("token index arrays must cover every token");
  bool by_page = global.device().is_cpu() && logical.device().is_cpu();
  if (by_page) {
    global = host_i64(global);
    logical = host_i64(logical);
    const int64_t *g = global.data_ptr<int64_t>(), *l = logical.data_ptr<int64_t>();
    for (int64_t i = 0; i < n && by_page; ++i)
      by_page = len[i] < 2 || (off_ramp(g + off[i], len[i]) | off_ramp(l + off[i], len[i])) == 0;
  }
  // the page table in pool order: R2KPage x (n + 1), then the two bases
  const int64_t words = (n + 1) + (by_page ? 2 * n : 0);
  at::Tensor table_host = at::empty({words > 0 ? words : 1}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
  {
    int64_t* w = table_host.data_ptr<int64_t>();
    R2KPage* pages = reinterpret_cast<R2KPage*>(w);
    static_assert(sizeof(R2KPage) == 8, "one table word");
    int64_t *gb = w + n + 1, *lb = gb + n, at = 0, dst = 0;
    const int64_t *g = by_page ? global.data_ptr<int64_t>() : nullptr, *l = by_page ? logical.data_ptr<int64_t>() : nullptr;
    for (int tier = 0; tier < 4; ++tier)
      for (int64_t i = 0; i < n; ++i) {
        if (tier_of(cls[i]) != tier) continue;
        pages[at] = R2KPage{(int32_t)dst, (int32_t)off[i]};
        if (by_page) { gb[at] = len[i] > 0 ? g[off[i]] : 0; lb[at] = len[i] > 0 ? l[off[i]] : 0; }
        dst += len[i];
        ++at;
      }
    pages[n] = R2KPage{(int32_t)rows, 0};
  }
  const at::TensorOptions i64 = at::TensorOptions().dtype(at::kLong).device(key.device());
  at::Tensor table = at::empty({table_host.numel()}, i64);
  table.copy_(table_host, /*non_blocking=*/true);
  if (!by_page) {
    global = global.to(key.device(), at::kLong).contiguous();
    logical = logical.to(key.device(), at::kLong).contiguous();
  }

  const int64_t n_fp = tokens[0], n_i4 = tokens[1], n_i2 = tokens[2], active = n_fp + n_i4 + n_i2;
  const int64_t k_cap = std::max<int64_t>(128, ceil_to(active + append_capacity, 128)), i2_cap = std::max<int64_t>(128, ceil_to(n_i2 + append_capacity, 128));
  const int64_t meta_cap = n_i2 + std::max<int64_t>(0, std::min(i2_cap - n_i2, k_cap - active)) / page_size * page_size;
  const int64_t groups = d / v2_group;
  const at::ScalarType T = key.scalar_type();
  Slab slab;
  slab.add(at::kByte, {1, h, k_cap, 64});
  slab.add(at::kHalf, {1, h, k_cap / k_block, d});
  slab.add(at::kByte, {1, h, k_cap / k_block, d});
  slab.add(T, {1, h, n_fp, d});
  slab.add(at::kByte, {1, h, n_i4, 64});
  slab.add(at::kFloat, {1, h, n_i4, 1});
  slab.add(at::kByte, {1, h, i2_cap, 32});
  slab.add(at::kHalf, {1, h, i2_cap, groups, 1});
  slab.add(at::kByte, {1, h, i2_cap, groups, 1});
  slab.add(T, {1, h, recent_capacity, d});
  slab.add(T, {1, h, recent_capacity, d});
  slab.add(at::kInt, {1});
  slab.add(at::kLong, {1, recent_capacity});
  slab.add(at::kLong, {1, recent_capacity});
  slab.add(at::kLong, {1, recent_capacity / page_size});
  slab.add(at::kLong, {1, meta_cap});
  slab.add(at::kLong, {1, meta_cap});
  slab.add(at::kLong, {1, n_fp});
  slab.add(at::kLong, {1, n_fp});
  slab.add(at::kLong, {1, n_i4});
  slab.add(at::kLong, {1, n_i4});
  slab.add(at::kLong, {1, tokens[3]});
  std::vector<at::Tensor> t = slab.make(key.device());
  auto ptr = [&](size_t i) { return t[i].data_ptr(); };

  R2KBuild b{};
  b.key = key.data_ptr(); b.value = value.data_ptr();
  b.rows = rows; b.dtype = dtype; b.num_kv_heads = (int32_t)h; b.page_size = (int32_t)page_size; b.k_block = (int32_t)k_block;
  b.v2_group = (int32_t)v2_group; b.n_pages = (int32_t)n;
  b.n_fp = (int32_t)n_fp; b.n_i4 = (int32_t)n_i4; b.n_i2 = (int32_t)n_i2; b.n_evicted = (int32_t)tokens[3];
  b.k_capacity = (int32_t)k_cap; b.i2_capacity = (int32_t)i2_cap; b.recent_capacity = (int32_t)recent_capacity; b.meta_capacity = (int32_t)meta_cap;
  int64_t* words_dev = table.data_ptr<int64_t>();
  b.pages = reinterpret_cast<const R2KPage*>(words_dev);
  if (by_page) { b.global_base = words_dev + n + 1; b.logical_base = words_dev + 2 * n + 1; }
  else { b.global_rows = global.data_ptr<int64_t>(); b.logical_rows = logical.data_ptr<int64_t>(); }
  b.k_packed = (uint8_t*)ptr(0); b.k_scale = ptr(1); b.k_zero = (uint8_t*)ptr(2);
  b.fp_v = ptr(3); b.i4_packed = (uint8_t*)ptr(4); b.i4_scale = (float*)ptr(5);
  b.i2_packed = (uint8_t*)ptr(6); b.i2_scale = ptr(7); b.i2_zero = (uint8_t*)ptr(8);
  b.recent_k = ptr(9); b.recent_v = ptr(10); b.recent_len = (int32_t*)ptr(11);
  b.recent_global = (int64_t*)ptr(12); b.recent_logical = (int64_t*)ptr(13); b.recent_page_lengths = (int64_t*)ptr(14);
  b.i2_global = (int64_t*)ptr(15); b.i2_logical = (int64_t*)ptr(16);
  b.fp_global = (int64_t*)ptr(17); b.fp_logical = (int64_t*)ptr(18); b.i4_global = (int64_t*)ptr(19); b.i4_logical = (int64_t*)ptr(20);
  b.evicted_global = (int64_t*)ptr(21);
  check(r2k_build_cache(&b, at::cuda::getCurrentCUDAStream().stream()), "r2k_build_cache");   // without tokens, too: it clears the cache
  return {std::move(t), n_fp, n_i4, n_i2};
}

// ---------------------------------------------------------------------------
// rotation and Hadamard of a step's or a prefill's rows
// ---------------------------------------------------------------------------
void require(bool ok, const char* message) {
  if (!ok) throw py::value_error(message);
}
void require_cuda(bool ok, const char* message) {
  if (!ok) throw std::runtime_error(message);
}
bool row_type(at::ScalarType t) { return t == at::kBFloat16 || t == at::kHalf; }

struct Rotary {
  const void *cos, *sin;
  int32_t type;
  int64_t cos_strides[4], sin_strides[4];
};
Rotary rotary(const at::Tensor& cos, const at::Tensor& sin) {
  require(cos.scalar_type() == sin.scalar_type() && (row_type(cos.scalar_type()) || cos.scalar_type() == at::kFloat),
          "rotary tables must share one of bf16 / fp16 / fp32");
  Rotary r;
  r.cos = cos.data_ptr();
  r.sin = sin.data_ptr();
  r.type = cos.scalar_type() == at::kFloat ? 2 : dtype_code(cos.scalar_type());
  for (int i = 0; i < 4; ++i) { r.cos_strides[i] = cos.stride(i); r.sin_strides[i] = sin.stride(i); }
  return r;
}
void require_sections(const std::vector<int64_t>& s) {
  require(s.size() == 3 && s[0] + s[1] + s[2] == 64, "Qwen mRoPE sections must contain three values summing to 64");
}

// triton_fwht_128 (r2omni/sspa/kernels/triton_qwen_mrope.py:325-346)
at::Tensor fwht(const at::Tensor& tensor, const std::optional<at::Tensor>& output) {
  require(tensor.dim() > 0 && tensor.size(-1) == 128 && tensor.is_floating_point(),
          "fused FWHT requires a floating tensor with last dimension 128");
  require_cuda(tensor.is_cuda(), "fused FWHT requires a CUDA tensor");
  require(row_type(tensor.scalar_type()), "fused FWHT runs on bf16 / fp16 rows (the cache's element types)");
  const c10::cuda::CUDAGuard guard(tensor.device());
  const at::Tensor in = tensor.contiguous();
  at::Tensor out;
  if (output) {
    out = *output;
    require(out.sizes() == in.sizes() && out.device() == in.device() && out.scalar_type() == in.scalar_type(),
            "fused FWHT output must match input shape, device, and dtype");
    require(out.is_contiguous(), "fused FWHT output must be contiguous");
  } else {
    out = at::empty_like(in);
  }
  if (in.numel() > 0)
    check(r2k_fwht128(in.data_ptr(), out.data_ptr(), dtype_code(in.scalar_type()), in.numel() / 128,
                      at::cuda::getCurrentCUDAStream().stream()),
          "r2k_fwht128");
  return out;
}

// qwen_qk_mrope (r2omni/sspa/kernels/triton_qwen_mrope.py:214-322)
std::pair<at::Tensor, at::Tensor> qk_mrope(const at::Tensor& query, const at::Tensor& key, const at::Tensor& cos, const at::Tensor& sin,
                                           const std::vector<int64_t>& sections, const std::optional<std::vector<at::Tensor>>& output,
                                           bool hadamard) {
  require(query.dim() == 4 && key.dim() == 4, "Qwen fused mRoPE requires rank-4 Q/K");
  const int64_t batch = query.size(0), tokens = query.size(2);
  require(key.size(0) == batch, "Qwen fused mRoPE requires equal Q/K batch sizes");
  require(tokens > 0 && key.size(2) == tokens, "Qwen fused mRoPE requires equal positive Q/K token counts");
  require(query.size(3) == 128 && key.size(3) == 128, "Qwen fused mRoPE currently requires head_dim=128");
  require(query.device() == key.device() && query.scalar_type() == key.scalar_type(), "Q/K device and dtype must match");
  require(cos.device() == query.device() && sin.device() == query.device(), "Q/K and rotary tensors must share a device");
  require(cos.dim() == 4 && cos.sizes() == sin.sizes() && cos.size(0) == 3, "Qwen fused mRoPE requires cos/sin [3,B,S,D]");
  require(cos.size(1) == batch && cos.size(2) == tokens && cos.size(3) == 128, "Qwen fused mRoPE rotary positions must match Q/K tokens");
  require_sections(sections);
  require_cuda(query.is_cuda(), "fused Qwen mRoPE requires CUDA tensors");
  require(row_type(query.scalar_type()), "fused Qwen mRoPE runs on bf16 / fp16 rows");
  const Rotary rot = rotary(cos, sin);
  const c10::cuda::CUDAGuard guard(query.device());
  const at::Tensor q = query.contiguous(), k = key.contiguous();
  at::Tensor qo, ko;
  if (output) {
    require(output->size() == 2 && (*output)[0].sizes() == q.sizes() && (*output)[1].sizes() == k.sizes(),
            "fused Qwen mRoPE output shapes must match Q/K");
    qo = (*output)[0];
    ko = (*output)[1];
    require(qo.device() == q.device() && ko.device() == q.device() && qo.scalar_type() == q.scalar_type() && ko.scalar_type() == q.scalar_type(),
            "fused Qwen mRoPE outputs must match Q/K device and dtype");
    require(qo.is_contiguous() && ko.is_contiguous(), "fused Qwen mRoPE outputs must be contiguous");
  } else {
    qo = at::empty_like(q);
    ko = at::empty_like(k);
  }
  check(r2k_qk_mrope(q.data_ptr(), k.data_ptr(), qo.data_ptr(), ko.data_ptr(), dtype_code(q.scalar_type()), (int32_t)batch,
                     (int32_t)q.size(1), (int32_t)k.size(1), (int32_t)tokens, rot.cos, rot.sin, rot.type, rot.cos_strides, rot.sin_strides,
                     (int32_t)sections[0], (int32_t)sections[1], hadamard ? 1 : 0, at::cuda::getCurrentCUDAStream().stream()),
        "r2k_qk_mrope");
  return {qo, ko};
}

// A request's rows of `t` as one run of heads * 128 elements, requests `stride` elements apart; copies where there is no such view.
struct Rows { at::Tensor t; int64_t heads, stride; };
Rows request_rows(const at::Tensor& t, int64_t batch, const char* what) {
  require_cuda(t.is_cuda(), "fused Qwen prologue requires CUDA tensors");
  if (batch < 1 || t.size(0) != batch || t.numel() % (batch * 128) != 0)
    throw py::value_error(std::string(what) + " rows do not match the batch");
  Rows r{t, t.numel() / (batch * 128), t.numel() / batch};
  if (t.is_contiguous()) return r;
  if (t.dim() == 3 && t.size(1) == 1 && t.stride(2) == 1) {
    r.stride = t.stride(0);
  } else {
    r.t = t.reshape({batch, r.heads * 128});
    r.stride = r.t.stride(0);
  }
  if ((r.t.dim() == 2 && r.t.stride(1) != 1) || r.stride % 4 || reinterpret_cast<uintptr_t>(r.t.data_ptr()) % 8) {
    r.t = r.t.contiguous();
    r.stride = r.heads * 128;
  }
  return r;
}

// qwen_qkv_prologue: see its Python entry.
std::vector<at::Tensor> qkv_prologue(const at::Tensor& query, const at::Tensor& key, const at::Tensor& value, const at::Tensor& cos,
                                     const at::Tensor& sin, const std::vector<int64_t>& sections, bool key_hadamard, bool value_hadamard,
                                     const std::optional<std::vector<at::Tensor>>& output) {
  require(query.dim() > 0 && key.dim() > 0 && value.dim() > 0, "query rows do not match the batch");
  const int64_t batch = query.size(0);
  const Rows q = request_rows(query, batch, "query"), k = request_rows(key, batch, "key"), v = request_rows(value, batch, "value");
  require(v.heads == k.heads, "key and value rows must have the same number of heads");
  const at::ScalarType T = q.t.scalar_type();
  require(row_type(T) && k.t.scalar_type() == T && v.t.scalar_type() == T, "fused Qwen prologue runs on bf16 / fp16 rows");
  require(cos.dim() == 4 && cos.sizes() == sin.sizes() && cos.size(0) == 3 && cos.size(1) == batch && cos.size(2) == 1 && cos.size(3) == 128,
          "Qwen fused prologue requires cos/sin [3,B,1,128]");
  require(cos.device() == q.t.device() && sin.device() == q.t.device(), "Q/K and rotary tensors must share a device");
  const Rotary rot = rotary(cos, sin);
  require_sections(sections);
  const c10::cuda::CUDAGuard guard(q.t.device());
  std::vector<at::Tensor> out;
  if (output) {
    out = *output;
    require(out.size() == 3, "fused Qwen prologue outputs must be contiguous [B,H,1,128] of the input type");
    for (int i = 0; i < 3; ++i)
      require(out[i].dim() == 4 && out[i].size(0) == batch && out[i].size(1) == (i == 0 ? q.heads : k.heads) && out[i].size(2) == 1 &&
                  out[i].size(3) == 128 && out[i].scalar_type() == T && out[i].device() == q.t.device() && out[i].is_contiguous(),
              "fused Qwen prologue outputs must be contiguous [B,H,1,128] of the input type");
  } else {
    for (int i = 0; i < 3; ++i) out.push_back(at::empty({batch, i == 0 ? q.heads : k.heads, 1, 128}, q.t.options()));
  }
  check(r2k_qkv_prologue(q.t.data_ptr(), q.stride, k.t.data_ptr(), k.stride, v.t.data_ptr(), v.stride, out[0].data_ptr(), out[1].data_ptr(),
                         out[2].data_ptr(), dtype_code(T), (int32_t)batch, (int32_t)q.heads, (int32_t)k.heads, rot.cos, rot.sin, rot.type,
                         rot.cos_strides, rot.sin_strides, (int32_t)sections[0], (int32_t)sections[1], key_hadamard ? 1 : 0,
                         value_hadamard ? 1 : 0, at::cuda::getCurrentCUDAStream().stream()),
        "r2k_qkv_prologue");
  return out;
}

}  // namespace

// The interpreter is left to other threads for the length of a call (no function here touches a Python object): a launch
// waits while the device's queue is full, an allocation may wait for the driver.
using unlocked = py::call_guard<py::gil_scoped_release>;

PYBIND11_MODULE(_r2k_host, m) {
  py::class_<Step>(m, "Step")
      .def(py::init<uintptr_t, uintptr_t, const at::Tensor&, const at::Tensor&>())
      .def("plain", &Step::plain, unlocked())
      .def("append", &Step::append, unlocked());
  m.def("build_cache", &build_cache, unlocked());
  m.def("fwht", &fwht, unlocked());
  m.def("qk_mrope", &qk_mrope, unlocked());
  m.def("qkv_prologue", &qkv_prologue, unlocked());
}
