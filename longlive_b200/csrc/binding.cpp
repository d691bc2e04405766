// Python binding of the C ABI (include/llnvfp4.h): argument checks, output allocation, the current stream and the call, in
// one native function per operation of longlive_b200/ops.py.
//
// Why native: a call of a small operation is bound by the host.  Through ctypes one call cost 8 to 20 us of interpreter time
// (device context manager, stream lookup, a foreign call with 20 boxed arguments, torch.empty for every output), and a
// module call on 17 rows spent 58 us on a device that was busy for 24 us.  Here the same work takes about 2 us per
// operation.  Group (sequence-parallel) forms stay on ctypes: they are bound by the exchange.
//
// Every function runs without the interpreter lock, as a ctypes call does: a launch blocks while the launch queue is full, and a first
// use loads kernels.  Only attention_nvfp4kv takes Python objects, which it unpacks before it lets the lock go.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>
#include <initializer_list>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/llnvfp4.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

[[noreturn]] void fail(const std::string& msg) { throw std::runtime_error(msg); }
[[noreturn]] void bad_value(const std::string& msg) { throw py::value_error(msg); }

void check(int rc) {
  if (rc == LLNV_OK) return;
  fail("llnvfp4 error " + std::to_string(rc) + ": " + llnv_last_error());
}

void require_cuda(const Tensor& t, const char* name) {
  if (!t.is_cuda()) bad_value(std::string(name) + " must be a CUDA tensor (the NVFP4 path has no CPU implementation)");
}

// The device of `t` made current for the duration of a call, its current stream, and the library's one-time set-up there.
struct Call {
  c10::cuda::CUDAGuard guard;
  cudaStream_t stream;
  explicit Call(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {
    static std::atomic<bool> ready[64];
    const int i = t.device().index();
    if (i < 0 || i >= 64) fail("unsupported device index");
    if (!ready[i].load(std::memory_order_acquire)) {
      check(llnv_init_device());
      ready[i].store(true, std::memory_order_release);
    }
  }
};

void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const OptTensor& t) { return t ? t->data_ptr() : nullptr; }
float* fptr(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
float* fptr(const OptTensor& t) { return t ? static_cast<float*>(t->data_ptr()) : nullptr; }
int64_t padded(int64_t m) { return (m + 127) / 128 * 128; }

Tensor empty(const Tensor& like, at::IntArrayRef shape, at::ScalarType dtype) {
  return at::empty(shape, like.options().dtype(dtype).memory_format(std::nullopt).requires_grad(false));
}

bool is_2d_bf16(const Tensor& t) { return t.dim() == 2 && t.scalar_type() == at::kBFloat16 && t.stride(1) == 1; }

// ---- quantizer ------------------------------------------------------------------------------------
struct Quantized {
  Tensor codes, sf, amax;
};

Quantized quantize_impl(Tensor x, int rule, OptTensor amax, OptTensor codes, OptTensor sf, bool given) {
  int64_t shards = 1, m, k, ldx;
  const auto dt = x.scalar_type();
  if (x.dim() == 3 && dt == at::kBFloat16 && x.is_contiguous()) {
    shards = x.size(0), m = x.size(1), ldx = x.size(2), k = shards * ldx;
  } else if (x.dim() != 2 || (dt != at::kBFloat16 && dt != at::kHalf)) {
    fail("quantize_nvfp4 expects a 2-D bfloat16 or float16 tensor (or a contiguous bfloat16 [shards, M, K/shards] one)");
  } else {
    if (x.stride(1) != 1) x = x.contiguous();
    m = x.size(0), k = x.size(1), ldx = x.stride(0);
  }
  Call call(x);
  Quantized q;
  q.codes = codes ? *codes : empty(x, {padded(m), k / 2}, at::kByte);
  q.sf = sf ? *sf : empty(x, {padded(m) * k / 16}, at::kFloat8_e4m3fn);
  if (!amax && given) bad_value("amax_given needs an amax tensor");
  q.amax = amax ? *amax : empty(x, {1}, at::kFloat);
  if (dt == at::kHalf)
    check(llnv_quantize_nvfp4_f16(ptr(x), m, k, ldx, rule, ptr(q.codes), ptr(q.sf), fptr(q.amax), given, call.stream));
  else
    check(llnv_quantize_nvfp4_ex(ptr(x), m, k, ldx, rule, ptr(q.codes), ptr(q.sf), fptr(q.amax), given, (int)shards, call.stream));
  return q;
}

std::tuple<Tensor, Tensor, Tensor> quantize(const Tensor& x, int rule, OptTensor amax, OptTensor codes, OptTensor sf, std::optional<bool> amax_given) {
  require_cuda(x, "x");
  const bool given = amax_given ? *amax_given : amax.has_value();
  Quantized q = quantize_impl(x, rule, amax, codes, sf, given);
  return {q.codes, q.sf, q.amax};
}

void quantize_pair(const Tensor& x0, const Tensor& x1, int rule, const Tensor& c0, const Tensor& s0, const Tensor& a0, const Tensor& c1,
                   const Tensor& s1, const Tensor& a1, bool given) {
  require_cuda(x0, "x0");
  if (x0.sizes() != x1.sizes() || x0.dim() != 2 || x0.stride(0) != x1.stride(0) || x0.stride(1) != 1 || x1.stride(1) != 1 ||
      x0.scalar_type() != at::kBFloat16)
    fail("quantize_nvfp4_pair expects two bfloat16 [M, K] tensors of the same shape and row stride");
  Call call(x0);
  check(llnv_quantize_nvfp4_pair(ptr(x0), ptr(x1), x0.size(0), x0.size(1), x0.stride(0), rule, ptr(c0), ptr(s0), fptr(a0), ptr(c1), ptr(s1),
                                 fptr(a1), given, call.stream));
}

using QuantizedAndY = std::tuple<OptTensor, OptTensor, OptTensor, OptTensor>;

QuantizedAndY adaln_quantize(const Tensor& x, const Tensor& scale, const Tensor& shift, int frame_rows, int rule, double eps, bool add_one,
                         bool want_y, OptTensor codes, OptTensor sf, OptTensor amax, OptTensor row_stats, int64_t row_offset, int phase,
                         bool y_only) {
  require_cuda(x, "x");
  if (!is_2d_bf16(x)) fail("adaln_quantize_nvfp4 expects a 2-D bfloat16 tensor with unit column stride");
  if (scale.dim() != 2 || shift.dim() != 2 || scale.stride(1) != 1 || shift.stride(1) != 1 || scale.stride(0) != shift.stride(0))
    fail("scale and shift must be [frames, C] views with the same row stride");
  const int64_t m = x.size(0), c = x.size(1);
  Call call(x);
  if (y_only) {
    want_y = true;
    codes.reset();
    sf.reset();
  } else {
    if (!codes) codes = empty(x, {padded(m), c / 2}, at::kByte);
    if (!sf) sf = empty(x, {padded(m) * c / 16}, at::kFloat8_e4m3fn);
  }
  if (!amax) amax = empty(x, {1}, at::kFloat);
  if (!row_stats) row_stats = empty(x, {2 * std::max<int64_t>(m, 1)}, at::kFloat);
  OptTensor y;
  if (want_y) y = empty(x, {m, c}, at::kBFloat16);
  check(llnv_adaln_quantize_nvfp4_ex(ptr(x), m, c, x.stride(0), ptr(scale), ptr(shift), scale.stride(0), frame_rows, (float)eps, add_one, rule,
                                     ptr(codes), ptr(sf), fptr(amax), ptr(y), c, fptr(row_stats), row_offset, phase, call.stream));
  return {codes, sf, amax, y};
}

QuantizedAndY layernorm_quantize(const Tensor& x, const Tensor& weight, const Tensor& bias, int rule, double eps, bool want_y, OptTensor codes,
                             OptTensor sf, OptTensor amax, OptTensor row_stats, int phase) {
  require_cuda(x, "x");
  if (!is_2d_bf16(x)) fail("layernorm_quantize_nvfp4 expects a 2-D bfloat16 tensor with unit column stride");
  const int64_t m = x.size(0), c = x.size(1);
  Call call(x);
  if (!codes) codes = empty(x, {padded(m), c / 2}, at::kByte);
  if (!sf) sf = empty(x, {padded(m) * c / 16}, at::kFloat8_e4m3fn);
  if (!amax) amax = empty(x, {1}, at::kFloat);
  if (!row_stats) row_stats = empty(x, {2 * std::max<int64_t>(m, 1)}, at::kFloat);
  OptTensor y;
  if (want_y) y = empty(x, {m, c}, at::kBFloat16);
  check(llnv_layernorm_quantize_nvfp4_ex(ptr(x), m, c, x.stride(0), ptr(weight), ptr(bias), (float)eps, rule, ptr(codes), ptr(sf), fptr(amax),
                                         ptr(y), c, fptr(row_stats), phase, call.stream));
  return {codes, sf, amax, y};
}

// ---- RMSNorm + RoPE -------------------------------------------------------------------------------
std::tuple<OptTensor, OptTensor, OptTensor> rmsnorm_rope(const Tensor& x, OptTensor weight, OptTensor cosv, OptTensor sinv, double eps, OptTensor out, OptTensor smooth,
                       bool want_smooth, OptTensor amax, bool want_amax, int shards) {
  require_cuda(x, "x");
  if (!is_2d_bf16(x)) fail("rmsnorm_rope expects a 2-D bfloat16 tensor with unit column stride");
  const int64_t s = x.size(0), c = x.size(1);
  if (shards < 1 || c % shards != 0) fail("rmsnorm_rope: " + std::to_string(c) + " channels do not divide into " + std::to_string(shards) + " shards");
  Call call(x);
  const std::vector<int64_t> shape = shards == 1 ? std::vector<int64_t>{s, c} : std::vector<int64_t>{shards, s, c / shards};
  if (!out) out = empty(x, shape, at::kBFloat16);
  if (!smooth && want_smooth) smooth = empty(x, shape, at::kBFloat16);
  if (shards > 1)
    for (const OptTensor* t : {&out, &smooth})
      if (*t && ((*t)->sizes() != at::IntArrayRef(shape) || !(*t)->is_contiguous())) fail("sharded outputs must be contiguous [shards, S, C / shards]");
  if (!amax && want_amax) amax = empty(x, {1}, at::kFloat);
  if (cosv && (cosv->scalar_type() != at::kFloat || cosv->dim() != 2 || cosv->size(0) != s || cosv->size(1) != 64 || !cosv->is_contiguous() ||
               !sinv || !sinv->is_contiguous()))
    fail("cos/sin must be contiguous float32 [S, 64]");
  check(llnv_rmsnorm_rope_ex(ptr(x), s, c, x.stride(0), ptr(weight), (float)eps, fptr(cosv), fptr(sinv), ptr(out), out->stride(-2), ptr(smooth),
                             smooth ? smooth->stride(-2) : 0, fptr(amax), shards, call.stream));
  return {out, smooth, amax};
}

using Ptrs = std::vector<uintptr_t>;
void* const* table(const Ptrs& p) { return reinterpret_cast<void* const*>(p.data()); }

void rmsnorm_rope_qk(const Tensor& xq, const Tensor& wq, const Ptrs& q, int64_t ldq, const Tensor& xk, const Tensor& wk, const Ptrs& k,
                     int64_t ldk, const std::optional<Ptrs>& ks, int64_t lds, OptTensor k_amax, const Tensor& cosv, const Tensor& sinv, double eps) {
  require_cuda(xq, "xq");
  if (k.size() != q.size() || (ks && ks->size() != q.size())) fail("rmsnorm_rope_qk: one address per head shard for each output");
  Call call(xq);
  check(llnv_rmsnorm_rope_qk(ptr(xq), xq.stride(0), ptr(wq), table(q), ldq, ptr(xk), xk.stride(0), ptr(wk), table(k), ldk,
                             ks ? table(*ks) : nullptr, lds, fptr(k_amax), xq.size(0), xq.size(1), (float)eps, fptr(cosv), fptr(sinv),
                             (int)q.size(), call.stream));
}

// ---- GEMM -----------------------------------------------------------------------------------------
void same_device(const Tensor& like, std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->device() != like.device()) fail("operands of a GEMM must be on one device (" + like.device().str() + " and " + t->device().str() + ")");
}

// The bias as the epilogue reads it, n packed bf16 values: a module in another precision has a bias of that precision.
OptTensor packed_bias(const OptTensor& bias, int64_t n, const Tensor& like) {
  if (!bias) return std::nullopt;
  same_device(like, {&*bias});
  if (bias->numel() < n) fail("bias holds " + std::to_string(bias->numel()) + " values, " + std::to_string(n) + " are needed");
  if (bias->scalar_type() == at::kBFloat16 && bias->is_contiguous()) return bias;
  return bias->to(at::kBFloat16).contiguous();
}

OptTensor gemm(const Tensor& a_codes, const Tensor& a_sf, OptTensor a_amax, int a_rule, const Tensor& b_codes, const Tensor& b_sf,
               OptTensor b_amax, int b_rule, int64_t m, int64_t n, int64_t k, OptTensor out, OptTensor alpha, OptTensor bias, int act,
               OptTensor residual, OptTensor gate, int frame_rows, OptTensor out_amax, int row_offset, int tile, OptTensor q_codes,
               OptTensor q_sf, OptTensor q_amax, bool store_out) {
  require_cuda(a_codes, "a_codes");
  same_device(a_codes, {&a_sf, &b_codes, &b_sf});
  Call call(a_codes);
  bias = packed_bias(bias, n, a_codes);
  if (!q_codes && !store_out) bad_value("store_out=False needs requant buffers");
  if (!out && store_out) out = empty(a_codes, {m, n}, at::kBFloat16);
  llnv_epilogue_t epi = {};
  epi.alpha = fptr(alpha);
  epi.bias = ptr(bias);
  epi.act = act;
  if (residual) {
    epi.residual = ptr(residual);
    epi.ldr = residual->stride(0);
  }
  if (gate) {
    epi.gate = ptr(gate);
    epi.gate_stride = gate->stride(0);
    epi.frame_rows = frame_rows;
    epi.row_offset = row_offset;
  }
  epi.out_amax = fptr(out_amax);
  if (q_codes) {
    if (!q_amax || q_amax->scalar_type() != at::kFloat)
      bad_value("requant needs requant_amax (fp32 [1]): the tensor amax must be known before the GEMM runs");
    if (q_codes->scalar_type() != at::kByte || q_codes->numel() < padded(m) * n / 2 || !q_sf || q_sf->numel() < padded(m) * n / 16)
      fail("requant buffers must hold uint8 [Mp, N/2] codes and Mp*N/16 scale bytes");
    epi.q_codes = ptr(q_codes);
    epi.q_sf = ptr(q_sf);
    epi.q_amax = fptr(q_amax);
    epi.q_rule = LLNV_RULE_MSE;
  }
  check(llnv_gemm_nvfp4_ex(ptr(a_codes), ptr(a_sf), fptr(a_amax), a_rule, ptr(b_codes), ptr(b_sf), fptr(b_amax), b_rule, m, n, k, &epi,
                           store_out ? ptr(out) : nullptr, store_out ? out->stride(0) : n, tile, call.stream));
  return store_out ? out : OptTensor();
}

void gemm_grouped(const Tensor& a_codes, const Tensor& a_sf, const Tensor& a_amax, int a_rule, const Tensor& b_codes, const Tensor& b_sf,
                  const Tensor& b_amax, int b_rule, int64_t m, int64_t n_each, int64_t k, const std::vector<Tensor>& outs, OptTensor bias, int act,
                  const std::optional<std::vector<OptTensor>>& out_amax) {
  require_cuda(a_codes, "a_codes");
  same_device(a_codes, {&a_sf, &b_codes, &b_sf, &b_amax});
  Call call(a_codes);
  bias = packed_bias(bias, n_each * (int64_t)outs.size(), a_codes);
  llnv_epilogue_t epi = {};
  epi.bias = ptr(bias);
  epi.act = act;
  void* d[8] = {};
  int64_t ldd[8] = {};
  float* am[8] = {};
  if (outs.size() > 8 || (out_amax && out_amax->size() != outs.size())) fail("gemm_nvfp4_grouped: at most 3 outputs, one amax target (or None) each");
  for (size_t g = 0; g < outs.size(); ++g) {
    d[g] = ptr(outs[g]);
    ldd[g] = outs[g].stride(0);
    if (out_amax) am[g] = fptr((*out_amax)[g]);
  }
  check(llnv_gemm_nvfp4_grouped(ptr(a_codes), ptr(a_sf), fptr(a_amax), a_rule, ptr(b_codes), ptr(b_sf), fptr(b_amax), b_rule, m, n_each, k,
                                (int)outs.size(), &epi, d, ldd, out_amax ? am : nullptr, call.stream));
}

// NVFP4 Linear: quantize the activation (leading dimensions flattened), multiply with the quantized weight [n (padded to
// n_pad rows), k], add the bias.
Tensor linear_nvfp4(const Tensor& input, int a_rule, const Tensor& w_codes, const Tensor& w_sf, const Tensor& w_amax, int w_rule, int64_t n,
                    int64_t n_pad, int64_t k, OptTensor bias) {
  const Tensor x = input.dim() == 2 ? input : input.reshape({-1, k});
  const int64_t m = x.size(0);
  same_device(x, {&w_codes, &w_sf, &w_amax});
  Quantized q = quantize_impl(x, a_rule, std::nullopt, std::nullopt, std::nullopt, false);
  Call call(x);
  Tensor out = empty(x, {m, n_pad}, at::kBFloat16);
  if (bias && bias->numel() != n_pad) bias = at::constant_pad_nd(*bias, {0, n_pad - bias->numel()});
  bias = packed_bias(bias, n_pad, x);
  llnv_epilogue_t epi = {};
  epi.bias = ptr(bias);
  check(llnv_gemm_nvfp4(ptr(q.codes), ptr(q.sf), fptr(q.amax), a_rule, ptr(w_codes), ptr(w_sf), fptr(w_amax), w_rule, m, n_pad, k, &epi,
                        ptr(out), n_pad, call.stream));
  if (n != n_pad) out = out.narrow(1, 0, n);
  if (input.dim() == 2) return out;
  std::vector<int64_t> shape = input.sizes().vec();
  shape.back() = n;
  return out.reshape(shape);
}

// ---- attention ------------------------------------------------------------------------------------
// The workspace of a call: the caller's (which has to hold at least the partial results of a split), or a fresh one of
// `want` bytes.
OptTensor attention_workspace(int64_t lq, int heads, int key_splits, int64_t want, const OptTensor& workspace, const Tensor& q) {
  const int64_t bytes = llnv_attention_workspace_bytes(lq, heads, key_splits);
  if (!workspace) return want > 0 ? OptTensor(empty(q, {want}, at::kByte)) : std::nullopt;
  if (workspace->scalar_type() != at::kByte || !workspace->is_contiguous() || workspace->numel() < bytes || workspace->device() != q.device())
    fail("attention workspace must be a contiguous uint8 tensor of at least " + std::to_string(bytes) + " bytes on the device of q");
  return workspace;
}

bool is_heads_matrix(const Tensor& t, int64_t heads) { return is_2d_bf16(t) && t.size(1) == heads * 128; }
constexpr double kDefaultScale = 0.08838834764831845;        // 128 ** -0.5

Tensor attention_bf16(const Tensor& q, const Tensor& k, const Tensor& v, int heads, std::optional<double> scale, OptTensor out,
                      std::optional<int> key_splits, OptTensor out_amax, OptTensor workspace) {
  require_cuda(q, "q");
  const Tensor* ts[3] = {&q, &k, &v};
  const char* names[3] = {"q", "k", "v"};
  for (int i = 0; i < 3; ++i)
    if (!is_heads_matrix(*ts[i], heads)) fail(std::string(names[i]) + " must be bfloat16 [tokens, heads*128] with unit column stride");
  if (k.size(0) != v.size(0)) fail("k and v must have the same number of tokens");
  Call call(q);
  const int64_t lq = q.size(0), lk = k.size(0);
  if (!out) out = empty(q, {lq, (int64_t)heads * 128}, at::kBFloat16);
  const int splits = key_splits ? *key_splits : llnv_attention_key_splits(lq, lk, heads);
  const OptTensor ws = attention_workspace(lq, heads, splits, llnv_attention_workspace_bytes(lq, heads, splits), workspace, q);
  check(llnv_attention_bf16_ex(ptr(q), lq, q.stride(0), ptr(k), ptr(v), lk, k.stride(0), v.stride(0), heads, (float)scale.value_or(kDefaultScale),
                               ptr(out), out->stride(0), splits, ptr(ws), ws ? ws->numel() : 0, fptr(out_amax), call.stream));
  return *out;
}

// One list of cache blocks (objects with `values`, `scale_factors`, `amax`) as pointer tables.
struct Blocks {
  std::vector<const void*> codes, sf;
  std::vector<const float*> amax;
  std::vector<Tensor> held;
};
Tensor attr(py::handle h, PyObject* name) {
  PyObject* o = PyObject_GetAttr(h.ptr(), name);
  if (!o) throw py::error_already_set();
  const py::object obj = py::reinterpret_steal<py::object>(o);
  if (!THPVariable_Check(o)) fail("a cache block holds tensors in values, scale_factors and amax");
  return THPVariable_Unpack(o);
}
Blocks gather_blocks(const py::sequence& blocks, const Tensor& q, int64_t rows) {
  static PyObject* s_values = PyUnicode_InternFromString("values");
  static PyObject* s_sf = PyUnicode_InternFromString("scale_factors");
  static PyObject* s_amax = PyUnicode_InternFromString("amax");
  Blocks b;
  for (const py::handle h : blocks) {
    Tensor v = attr(h, s_values), s = attr(h, s_sf), a = attr(h, s_amax);
    if (v.scalar_type() != at::kByte || v.dim() != 2 || v.size(1) != 64 || !v.is_contiguous() || v.size(0) < rows)
      fail("a cache block must be contiguous uint8 [rows_padded, 64] covering block_tokens * heads rows");
    if (v.device() != q.device() || s.device() != q.device() || a.device() != q.device() || a.scalar_type() != at::kFloat)
      fail("cache blocks must live on the device of q, with float32 amax");
    b.codes.push_back(ptr(v));
    b.sf.push_back(ptr(s));
    b.amax.push_back(fptr(a));
    b.held.insert(b.held.end(), {v, s, a});
  }
  return b;
}

Tensor attention_nvfp4kv(const Tensor& q, const py::sequence& k_blocks, const py::sequence& v_blocks, int block_tokens, OptTensor k_cur,
                         OptTensor v_cur, int heads, std::optional<double> scale, OptTensor out, std::optional<int> key_splits,
                         OptTensor out_amax, double e2m1_max, double e4m3_max, OptTensor workspace) {
  require_cuda(q, "q");
  if (!is_heads_matrix(q, heads)) fail("q must be bfloat16 [tokens, heads*128] with unit column stride");
  const int n = (int)k_blocks.size();
  if ((int)v_blocks.size() != n) fail("k_blocks and v_blocks must have the same length");
  const Blocks kb = gather_blocks(k_blocks, q, (int64_t)block_tokens * heads), vb = gather_blocks(v_blocks, q, (int64_t)block_tokens * heads);
  const py::gil_scoped_release nogil;
  int64_t l_cur = 0;
  if (k_cur) {
    if (!is_heads_matrix(*k_cur, heads)) fail("k_cur must be bfloat16 [tokens, heads*128] with unit column stride");
    if (!v_cur || !is_heads_matrix(*v_cur, heads)) fail("v_cur must be bfloat16 [tokens, heads*128] with unit column stride");
    if (k_cur->size(0) != v_cur->size(0)) fail("k_cur and v_cur must have the same number of tokens");
    l_cur = k_cur->size(0);
  }
  Call call(q);
  const int64_t lq = q.size(0), lk = (int64_t)n * block_tokens + l_cur;
  if (!out) out = empty(q, {lq, (int64_t)heads * 128}, at::kBFloat16);
  const int splits = key_splits ? *key_splits : llnv_attention_key_splits(lq, lk, heads);
  const OptTensor ws =
      attention_workspace(lq, heads, splits, llnv_attention_nvfp4kv_workspace_bytes(lq, heads, splits, n, block_tokens), workspace, q);
  check(llnv_attention_nvfp4kv(ptr(q), lq, q.stride(0), n ? kb.codes.data() : nullptr, n ? kb.sf.data() : nullptr, n ? kb.amax.data() : nullptr,
                               n ? vb.codes.data() : nullptr, n ? vb.sf.data() : nullptr, n ? vb.amax.data() : nullptr, n, block_tokens,
                               (float)e2m1_max, (float)e4m3_max, l_cur ? ptr(k_cur) : nullptr, l_cur ? ptr(v_cur) : nullptr, l_cur,
                               l_cur ? k_cur->stride(0) : 0, l_cur ? v_cur->stride(0) : 0, heads, (float)scale.value_or(kDefaultScale), ptr(out),
                               out->stride(0), splits, ptr(ws), ws ? ws->numel() : 0, fptr(out_amax), call.stream));
  return *out;
}

// ---- dequantize -----------------------------------------------------------------------------------
int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return LLNV_DTYPE_BF16;
    case at::kHalf: return LLNV_DTYPE_FP16;
    case at::kFloat: return LLNV_DTYPE_FP32;
    default: return -1;
  }
}

Tensor dequantize(const Tensor& codes, const Tensor& sf, const Tensor& amax, int64_t rows, int64_t cols, int64_t cols_padded,
                  at::ScalarType dtype, double e2m1_max, double e4m3_max, int rounding) {
  require_cuda(codes, "codes");
  Call call(codes);
  Tensor out = empty(codes, {rows, cols}, dtype);
  check(llnv_dequantize_nvfp4(ptr(codes), ptr(sf), fptr(amax), rows, cols, cols_padded, dtype_code(dtype), (float)e2m1_max, (float)e4m3_max,
                              rounding, ptr(out), out.stride(0), call.stream));
  return out;
}

Tensor kv_dequant(const std::vector<Tensor>& values, const std::vector<Tensor>& sf, const std::vector<Tensor>& amax, int64_t num_heads,
                  int64_t block_tokens, at::ScalarType dtype, double e2m1_max, double e4m3_max, int rounding, OptTensor out) {
  const size_t n = values.size();
  if (n == 0) fail("values must contain at least one cache block");
  if (sf.size() != n || amax.size() != n) fail("values, scale_factors and amax must have the same length");
  require_cuda(values[0], "values");
  const auto dev = values[0].device();
  if (dtype_code(dtype) < 0) bad_value(std::string("Unsupported fused KV dequant dtype: ") + c10::toString(dtype));
  std::vector<const void*> cp(n), sp(n);
  std::vector<const float*> ap(n);
  for (size_t i = 0; i < n; ++i) {
    const Tensor &v = values[i], &s = sf[i], &a = amax[i];
    if (v.scalar_type() != at::kByte || v.dim() != 2 || v.size(1) != 64) fail("KV dequant expects uint8 values of shape [rows_padded, 64] (head_dim 128)");
    if (v.size(0) < num_heads * block_tokens || v.size(0) % 128 != 0) fail("values rows must be padded to a multiple of 128 and cover the block");
    if (a.scalar_type() != at::kFloat) fail("amax tensors must be float32");
    if (v.device() != dev || s.device() != dev || a.device() != dev) fail("all KV block tensors must be on the same device");
    if (!(v.is_contiguous() && s.is_contiguous() && a.is_contiguous())) fail("KV block tensors must be contiguous");
    cp[i] = ptr(v), sp[i] = ptr(s), ap[i] = fptr(a);
  }
  Call call(values[0]);
  if (!out) out = empty(values[0], {1, (int64_t)n * block_tokens, num_heads, 128}, dtype);
  check(llnv_kv_dequant(cp.data(), sp.data(), ap.data(), (int)n, (int)num_heads, (int)block_tokens, dtype_code(dtype), (float)e2m1_max,
                        (float)e4m3_max, rounding, ptr(out), call.stream));
  return *out;
}

// ---- bf16 Linear, latents, scheduler ----------------------------------------------------------------
Tensor linear_bf16(const Tensor& x, const Tensor& w, OptTensor bias, int act, OptTensor out) {
  require_cuda(x, "x");
  if (!is_2d_bf16(x)) fail("x must be a 2-D bfloat16 tensor with unit column stride");
  if (!is_2d_bf16(w)) fail("w must be a 2-D bfloat16 tensor with unit column stride");
  const int64_t m = x.size(0), k = x.size(1), n = w.size(0);
  if (k != w.size(1)) fail("x is [M, " + std::to_string(k) + "] but w is [N, " + std::to_string(w.size(1)) + "]");
  if (bias && (bias->scalar_type() != at::kBFloat16 || bias->numel() != n || !bias->is_contiguous()))
    fail("bias must be a contiguous bfloat16 tensor of N values");
  Call call(x);
  if (!out) out = empty(x, {m, n}, at::kBFloat16);
  else if (!is_2d_bf16(*out) || out->size(0) != m || out->size(1) != n) fail("out must be bfloat16 [M, N] with unit column stride");
  check(llnv_linear_bf16(ptr(x), m > 1 ? x.stride(0) : std::max(k, x.stride(0)), ptr(w), w.stride(0), ptr(bias), act, m, n, k, ptr(out),
                         m > 1 ? out->stride(0) : std::max(n, out->stride(0)), call.stream));
  return *out;
}

struct Latent {
  int C, F, h, w;
  int64_t sc, sf;
  Latent(const Tensor& t, bool channels_first) {
    if (t.dim() != 4 || t.scalar_type() != at::kBFloat16 || t.stride(3) != 1 || t.stride(2) != t.size(3))
      fail("latent must be a 4-D bfloat16 tensor whose two image axes are contiguous");
    if (t.size(2) % 2 || t.size(3) % 2) fail("latent height and width must be even (patch 1 x 2 x 2)");
    const int c_ax = channels_first ? 0 : 1, f_ax = 1 - c_ax;
    C = (int)t.size(c_ax), F = (int)t.size(f_ax), sc = t.stride(c_ax), sf = t.stride(f_ax);
    h = (int)t.size(2) / 2, w = (int)t.size(3) / 2;
  }
};

Tensor patchify(const Tensor& latent, bool channels_first, OptTensor out) {
  require_cuda(latent, "latent");
  const Latent l(latent, channels_first);
  const int64_t rows = (int64_t)l.F * l.h * l.w;
  Call call(latent);
  if (!out) out = empty(latent, {rows, 4 * (int64_t)l.C}, at::kBFloat16);
  else if (!is_2d_bf16(*out) || out->size(0) != rows || out->size(1) != 4 * (int64_t)l.C) fail("out must be bfloat16 [F*h*w, 4*C] with unit column stride");
  check(llnv_patchify(ptr(latent), l.sc, l.sf, ptr(out), out->stride(0), l.C, l.F, l.h, l.w, call.stream));
  return *out;
}

Tensor unpatchify(const Tensor& tokens, const Tensor& out, bool channels_first) {
  require_cuda(tokens, "tokens");
  const Latent l(out, channels_first);
  if (!is_2d_bf16(tokens) || tokens.size(0) != (int64_t)l.F * l.h * l.w || tokens.size(1) != 4 * (int64_t)l.C || tokens.device() != out.device())
    fail("tokens must be bfloat16 [F*h*w, 4*C] with unit column stride on the device of out");
  Call call(tokens);
  check(llnv_unpatchify(ptr(tokens), tokens.stride(0), ptr(out), l.sc, l.sf, l.C, l.F, l.h, l.w, call.stream));
  return out;
}

// One scheduler step: `coef` is the address of an llnv_unipc_coef; `older` receives the new x0, `last` the corrected sample.
Tensor unipc_step(const Tensor& model_output, const Tensor& sample, const Tensor& prev, const Tensor& older, const Tensor& last, uintptr_t coef) {
  const Tensor v = model_output.contiguous(), x = sample.contiguous();
  Call call(x);
  Tensor out = at::empty_like(x);
  check(llnv_unipc_step(ptr(v), ptr(x), ptr(prev), ptr(older), ptr(last), ptr(older), ptr(last), ptr(out), x.numel(),
                        x.scalar_type() == at::kBFloat16 ? 0 : 1, reinterpret_cast<const llnv_unipc_coef*>(coef), call.stream));
  return out;
}

uintptr_t current_stream(int device) { return reinterpret_cast<uintptr_t>(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream()); }

}  // namespace

PYBIND11_MODULE(_native, m) {
  using Unlocked = py::call_guard<py::gil_scoped_release>;
  m.attr("torch_version") = LLNV_TORCH_VERSION;
  m.def("quantize", &quantize, Unlocked());
  m.def("quantize_pair", &quantize_pair, Unlocked());
  m.def("adaln_quantize", &adaln_quantize, Unlocked());
  m.def("layernorm_quantize", &layernorm_quantize, Unlocked());
  m.def("rmsnorm_rope", &rmsnorm_rope, Unlocked());
  m.def("rmsnorm_rope_qk", &rmsnorm_rope_qk, Unlocked());
  m.def("gemm", &gemm, Unlocked());
  m.def("gemm_grouped", &gemm_grouped, Unlocked());
  m.def("linear_nvfp4", &linear_nvfp4, Unlocked());
  m.def("attention_bf16", &attention_bf16, Unlocked());
  m.def("attention_nvfp4kv", &attention_nvfp4kv);       // lets the lock go itself
  m.def("dequantize", &dequantize, Unlocked());
  m.def("kv_dequant", &kv_dequant, Unlocked());
  m.def("linear_bf16", &linear_bf16, Unlocked());
  m.def("patchify", &patchify, Unlocked());
  m.def("unpatchify", &unpatchify, Unlocked());
  m.def("unipc_step", &unipc_step, Unlocked());
  m.def("current_stream", &current_stream, Unlocked());
}
