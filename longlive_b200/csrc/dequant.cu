// NVFP4 -> bf16/fp16/fp32 dequantize: a general matrix form and the multi-block KV-cache form
// (one launch for all cache blocks of a layer, pointer table passed as launch parameters).
#include <cuda_fp4.h>

#include "common.cuh"

namespace llnv {
namespace {

constexpr int kMaxBlocks = 32;

// Cache blocks of one launch: each with its own destination (a contiguous [rows, 128] matrix).
struct BlockTable {
  const uint8_t* codes[kMaxBlocks];
  const uint8_t* sf[kMaxBlocks];
  const float* amax[kMaxBlocks];
  void* out[kMaxBlocks];
};

// Rows of a bf16 matrix copied behind the blocks by the same launch (kv_window_dequant): up to two matrices.
struct RowCopies {
  const uint16_t* src[2];
  uint16_t* dst[2];
  int64_t ld[2];
  int rows, cols;
};

template <int ROUNDING>
__device__ __forceinline__ float deq_scale(float vs, float amax, float g, float denom) {
  if (ROUNDING == LLNV_DEQ_PYTORCH) return __fdiv_rn(__fmul_rn(vs, amax), denom);
  return __fmul_rn(vs, g);   // FUSED: g = amax * fp32(1/denom);  TRITON: g = amax / denom
}

template <typename T>
__device__ __forceinline__ void store16(T* out, const float (&v)[16]);

template <>
__device__ __forceinline__ void store16<__nv_bfloat16>(__nv_bfloat16* out, const float (&v)[16]) {
  uint4 a, b;
  a.x = pack_bf16x2(v[0], v[1]);   a.y = pack_bf16x2(v[2], v[3]);
  a.z = pack_bf16x2(v[4], v[5]);   a.w = pack_bf16x2(v[6], v[7]);
  b.x = pack_bf16x2(v[8], v[9]);   b.y = pack_bf16x2(v[10], v[11]);
  b.z = pack_bf16x2(v[12], v[13]); b.w = pack_bf16x2(v[14], v[15]);
  reinterpret_cast<uint4*>(out)[0] = a;
  reinterpret_cast<uint4*>(out)[1] = b;
}
template <>
__device__ __forceinline__ void store16<__half>(__half* out, const float (&v)[16]) {
  __half2 h[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
  reinterpret_cast<uint4*>(out)[0] = *reinterpret_cast<uint4*>(&h[0]);
  reinterpret_cast<uint4*>(out)[1] = *reinterpret_cast<uint4*>(&h[4]);
}
template <>
__device__ __forceinline__ void store16<float>(float* out, const float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    reinterpret_cast<float4*>(out)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}

// 16 bytes of output: 8 values of 16 bits or 4 of 32
__device__ __forceinline__ void store_vec(__nv_bfloat16* out, const float (&v)[8]) {
  *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ void store_vec(__half* out, const float (&v)[8]) {
  __half2 h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(out) = *reinterpret_cast<uint4*>(&h[0]);
}
__device__ __forceinline__ void store_vec(float* out, const float (&v)[4]) { *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]); }

// decode 8 packed bytes (16 codes) and scale them
template <int ROUNDING>
__device__ __forceinline__ void decode16(uint2 packed, float s, float amax, float g, float denom, float (&v)[16]) {
  const uint32_t words[2] = {packed.x, packed.y};
#pragma unroll
  for (int wi = 0; wi < 2; ++wi) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const uint8_t byte = (uint8_t)(words[wi] >> (8 * b));
      const __half2_raw h2 = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)byte, __NV_E2M1);
      const float lo = __half2float(__ushort_as_half(h2.x));
      const float hi = __half2float(__ushort_as_half(h2.y));
      v[wi * 8 + b * 2] = deq_scale<ROUNDING>(__fmul_rn(lo, s), amax, g, denom);
      v[wi * 8 + b * 2 + 1] = deq_scale<ROUNDING>(__fmul_rn(hi, s), amax, g, denom);
    }
  }
}

__device__ __forceinline__ float global_scale(int rounding, float amax, float denom) {
  if (rounding == LLNV_DEQ_FUSED) return __fmul_rn(amax, (float)(1.0 / (double)denom));
  return __fdiv_rn(amax, denom);
}

// rows x cols logical matrix; codes row stride = cols_padded/2 bytes; scales swizzled with
// cols_padded/16 scale columns.
template <typename T, int ROUNDING>
__global__ void __launch_bounds__(256) dequant_matrix_kernel(const uint8_t* codes, const uint8_t* sf,
                                                             const float* amax_ptr, int64_t rows, int64_t cols,
                                                             int64_t cols_padded, float denom, T* __restrict__ out, int64_t ldo) {
  pdl_begin();
  const int64_t groups_per_row = cols >> 4;
  const int64_t total = rows * groups_per_row;
  const float amax = *amax_ptr;
  const float g = global_scale(ROUNDING, amax, denom);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / groups_per_row, c = i - r * groups_per_row;
    const uint2 p = ld_global(reinterpret_cast<const uint2*>(codes + r * (cols_padded >> 1) + c * 8));
    const float s = e4m3_to_float(ld_global(sf + sf_offset(r, c, cols_padded >> 4)));
    float v[16];
    decode16<ROUNDING>(p, s, amax, g, denom, v);
    store16<T>(out + r * ldo + c * 16, v);
  }
}

// KV cache: block b holds `rows` logical rows of 128 columns.
//
// Bound by HBM writes (2 bytes out for 9/16 in).  A lane decodes the values of one 16-byte store, so a warp's store covers
// 512 contiguous bytes (with 16 values a thread the two halves of a sector came from two instructions and cost
// two partial writes); a CTA of 256 threads covers 4 KB of output a step and takes STEPS steps whose loads are issued together: four, or
// one where that leaves SMs without a CTA (660 x 3 rows with a division per value 7.3 us with four steps, 3.1 with one).
// us for 4 blocks of 2640 x 24 rows in L2: bf16 13.0, fp32 24.9 (37.0 with 8 values a lane, two stores 32 bytes apart), with a division per
// value 56 and 58.
template <typename T, int ROUNDING, int STEPS>
__global__ void __launch_bounds__(256) dequant_kv_kernel(const __grid_constant__ BlockTable tab, int num_blocks, int64_t rows, float denom,
                                                         const __grid_constant__ RowCopies copies) {
  pdl_begin();
  const int b = blockIdx.y;
  if (b >= num_blocks) {                                    // rows copied behind the blocks
    const int m = b - num_blocks;
    const int vecs = copies.cols / 8;
    const int64_t total = (int64_t)copies.rows * vecs;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
      const int64_t r = i / vecs;
      const int c = (int)(i - r * vecs);
      reinterpret_cast<uint4*>(copies.dst[m])[i] = ld_global(reinterpret_cast<const uint4*>(copies.src[m] + r * copies.ld[m]) + c);
    }
    return;
  }
  constexpr int kVals = 16 / sizeof(T), kLanes = 128 / kVals, kStepRows = 256 / kLanes;
  const int c = threadIdx.x % kLanes;                        // columns kVals * c .. kVals * c + kVals - 1
  const int64_t r0 = (int64_t)blockIdx.x * (kStepRows * STEPS) + threadIdx.x / kLanes;
  const uint8_t* codes = tab.codes[b];
  const uint8_t* sf = tab.sf[b];
  uint32_t w[STEPS], sb[STEPS];
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    const int64_t r = r0 + kStepRows * k;
    w[k] = sb[k] = 0u;
    if (r < rows) {
      if (kVals == 8) w[k] = ld_global(reinterpret_cast<const uint32_t*>(codes) + r * 16 + c);
      else w[k] = ld_global(reinterpret_cast<const uint16_t*>(codes) + r * 32 + c);
      sb[k] = ld_global(sf + sf_offset(r, c * kVals / 16, 8));
    }
  }
  const float amax = ld_global(tab.amax[b]);
  const float g = global_scale(ROUNDING, amax, denom);
  T* out = (T*)tab.out[b];
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    const int64_t r = r0 + kStepRows * k;
    if (r >= rows) continue;
    const float s = e4m3_to_float(sb[k]);
    float v[kVals];
#pragma unroll
    for (int i = 0; i < kVals / 2; ++i) {
      const __half2_raw h2 = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)(uint8_t)(w[k] >> (8 * i)), __NV_E2M1);
      v[2 * i] = deq_scale<ROUNDING>(__fmul_rn(__half2float(__ushort_as_half(h2.x)), s), amax, g, denom);
      v[2 * i + 1] = deq_scale<ROUNDING>(__fmul_rn(__half2float(__ushort_as_half(h2.y)), s), amax, g, denom);
    }
    store_vec(out + r * 128 + c * kVals, v);
  }
}

template <typename T>
int launch_matrix(const uint8_t* codes, const uint8_t* sf, const float* amax, int64_t rows, int64_t cols, int64_t cols_padded,
                  float denom, int rounding, void* out, int64_t ldo, cudaStream_t stream) {
  const int64_t total = rows * (cols / 16);
  if (total == 0) return LLNV_OK;
  int64_t blocks = (total + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  T* o = (T*)out;
  switch (rounding) {
    case LLNV_DEQ_FUSED: launch_k(dequant_matrix_kernel<T, LLNV_DEQ_FUSED>, (unsigned)blocks, 256, 0, stream, codes, sf, amax, rows, cols, cols_padded, denom, o, ldo); break;
    case LLNV_DEQ_PYTORCH: launch_k(dequant_matrix_kernel<T, LLNV_DEQ_PYTORCH>, (unsigned)blocks, 256, 0, stream, codes, sf, amax, rows, cols, cols_padded, denom, o, ldo); break;
    default: launch_k(dequant_matrix_kernel<T, LLNV_DEQ_TRITON>, (unsigned)blocks, 256, 0, stream, codes, sf, amax, rows, cols, cols_padded, denom, o, ldo); break;
  }
  return launch_status("dequant_matrix_kernel");
}

template <typename T, int STEPS>
int launch_kv_steps(const BlockTable& tab, int n, int64_t rows, float denom, int rounding, const RowCopies& copies, cudaStream_t stream) {
  constexpr int kCtaRows = 2 * 16 / sizeof(T) * STEPS;
  const int64_t gx = (rows + kCtaRows - 1) / kCtaRows;
  LLNV_REQUIRE(gx < ((int64_t)1 << 31), "llnv_kv_dequant: too many rows (%lld)", (long long)rows);
  const dim3 grid((unsigned)gx, (unsigned)(n + (copies.rows > 0 ? 2 : 0)));
  switch (rounding) {
    case LLNV_DEQ_FUSED: launch_k(dequant_kv_kernel<T, LLNV_DEQ_FUSED, STEPS>, grid, 256, 0, stream, tab, n, rows, denom, copies); break;
    case LLNV_DEQ_PYTORCH: launch_k(dequant_kv_kernel<T, LLNV_DEQ_PYTORCH, STEPS>, grid, 256, 0, stream, tab, n, rows, denom, copies); break;
    default: launch_k(dequant_kv_kernel<T, LLNV_DEQ_TRITON, STEPS>, grid, 256, 0, stream, tab, n, rows, denom, copies); break;
  }
  return launch_status("dequant_kv_kernel");
}

template <typename T>
int launch_kv(const BlockTable& tab, int n, int64_t rows, float denom, int rounding, const RowCopies& copies, cudaStream_t stream) {
  if (rows * n == 0 && copies.rows == 0) return LLNV_OK;
  const int64_t ctas = (rows + 63) / 64 * n;                 // of four steps of 16 rows
  if (ctas < 2 * (int64_t)sm_count()) return launch_kv_steps<T, 1>(tab, n, rows, denom, rounding, copies, stream);
  return launch_kv_steps<T, 4>(tab, n, rows, denom, rounding, copies, stream);
}

}  // namespace

// Keys and values of the cached part of an attention window as bf16 [tokens, heads * 128] matrices (FUSED rounding), with
// n_pad rows of the current chunk copied behind them so that the attention kernel's last tile of the cached part is whole.
int kv_window_dequant(const void* const* k_codes, const void* const* k_sf, const float* const* k_amax, const void* const* v_codes,
                      const void* const* v_sf, const float* const* v_amax, int num_blocks, int heads, int block_tokens, float denom,
                      const void* k_cur, const void* v_cur, int64_t ldk, int64_t ldv, int n_pad, void* k_out, void* v_out, cudaStream_t stream) {
  const int64_t rows = (int64_t)heads * block_tokens;
  BlockTable tab;
  for (int b = 0; b < num_blocks; ++b)
    for (int m = 0; m < 2; ++m) {
      const int i = 2 * b + m;
      tab.codes[i] = (const uint8_t*)(m ? v_codes : k_codes)[b];
      tab.sf[i] = (const uint8_t*)(m ? v_sf : k_sf)[b];
      tab.amax[i] = (m ? v_amax : k_amax)[b];
      tab.out[i] = (uint16_t*)(m ? v_out : k_out) + (int64_t)b * rows * 128;
    }
  RowCopies copies = {};
  if (n_pad > 0)
    copies = RowCopies{{(const uint16_t*)k_cur, (const uint16_t*)v_cur},
                       {(uint16_t*)k_out + (int64_t)num_blocks * rows * 128, (uint16_t*)v_out + (int64_t)num_blocks * rows * 128},
                       {ldk, ldv}, n_pad, heads * 128};
  return launch_kv<__nv_bfloat16>(tab, 2 * num_blocks, rows, denom, LLNV_DEQ_FUSED, copies, stream);
}

}  // namespace llnv

using namespace llnv;

extern "C" int llnv_dequantize_nvfp4(const void* codes, const void* sf, const float* amax, int64_t rows, int64_t cols,
                                     int64_t cols_padded, int dtype_code, float e2m1_max, float e4m3_max, int rounding,
                                     void* out, int64_t ldo, llnv_stream_t stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  LLNV_REQUIRE(codes && sf && amax && out, "llnv_dequantize_nvfp4: null pointer");
  LLNV_REQUIRE(rows >= 0 && cols >= 0 && cols % 16 == 0 && cols_padded % 64 == 0 && cols_padded >= cols,
               "llnv_dequantize_nvfp4: cols must be a multiple of 16 and cols_padded a multiple of 64 (cols=%lld padded=%lld)",
               (long long)cols, (long long)cols_padded);
  LLNV_REQUIRE(rounding >= 0 && rounding <= 2, "llnv_dequantize_nvfp4: unknown rounding %d", rounding);
  LLNV_REQUIRE(e2m1_max > 0 && e4m3_max > 0, "llnv_dequantize_nvfp4: e2m1_max and e4m3_max must be positive");
  LLNV_REQUIRE(ldo >= cols && ldo % 8 == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)codes & 7) == 0,
               "llnv_dequantize_nvfp4: out must be 16-byte aligned with ldo a multiple of 8, codes 8-byte aligned");
  const float denom = e2m1_max * e4m3_max;
  const uint8_t* c = (const uint8_t*)codes;
  const uint8_t* s = (const uint8_t*)sf;
  switch (dtype_code) {
    case LLNV_DTYPE_BF16: return launch_matrix<__nv_bfloat16>(c, s, amax, rows, cols, cols_padded, denom, rounding, out, ldo, stream);
    case LLNV_DTYPE_FP16: return launch_matrix<__half>(c, s, amax, rows, cols, cols_padded, denom, rounding, out, ldo, stream);
    case LLNV_DTYPE_FP32: return launch_matrix<float>(c, s, amax, rows, cols, cols_padded, denom, rounding, out, ldo, stream);
    default: set_error("llnv_dequantize_nvfp4: unsupported dtype code %d", dtype_code); return LLNV_E_INVALID;
  }
}

extern "C" int llnv_kv_dequant(const void* const* codes, const void* const* sf, const float* const* amax, int num_blocks,
                               int num_heads, int block_token_size, int dtype_code, float e2m1_max, float e4m3_max,
                               int rounding, void* out, llnv_stream_t stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  LLNV_REQUIRE(codes && sf && amax && out, "llnv_kv_dequant: null pointer");
  LLNV_REQUIRE(num_blocks > 0, "llnv_kv_dequant: values must contain at least one cache block");
  LLNV_REQUIRE(num_heads > 0, "llnv_kv_dequant: num_heads must be positive");
  LLNV_REQUIRE(block_token_size > 0, "llnv_kv_dequant: block_token_size must be positive");
  LLNV_REQUIRE(e2m1_max > 0 && e4m3_max > 0, "llnv_kv_dequant: e2m1_max and e4m3_max must be positive");
  LLNV_REQUIRE(rounding >= 0 && rounding <= 2, "llnv_kv_dequant: unknown rounding %d", rounding);
  LLNV_REQUIRE(((uintptr_t)out & 15) == 0, "llnv_kv_dequant: out must be 16-byte aligned");
  const int64_t rows = (int64_t)num_heads * block_token_size;
  const float denom = e2m1_max * e4m3_max;
  const size_t esize = dtype_code == LLNV_DTYPE_FP32 ? 4 : 2;
  LLNV_REQUIRE(dtype_code >= 0 && dtype_code <= 2, "llnv_kv_dequant: unsupported dtype code %d", dtype_code);
  for (int base = 0; base < num_blocks; base += kMaxBlocks) {
    const int n = num_blocks - base < kMaxBlocks ? num_blocks - base : kMaxBlocks;
    BlockTable tab;
    for (int i = 0; i < n; ++i) {
      LLNV_REQUIRE(codes[base + i] && sf[base + i] && amax[base + i], "llnv_kv_dequant: null pointer in block %d", base + i);
      LLNV_REQUIRE(((uintptr_t)codes[base + i] & 7) == 0, "llnv_kv_dequant: codes of block %d must be 8-byte aligned", base + i);
      tab.codes[i] = (const uint8_t*)codes[base + i];
      tab.sf[i] = (const uint8_t*)sf[base + i];
      tab.amax[i] = amax[base + i];
      tab.out[i] = (char*)out + (size_t)(base + i) * rows * 128 * esize;
    }
    int rc;
    if (dtype_code == LLNV_DTYPE_BF16) rc = launch_kv<__nv_bfloat16>(tab, n, rows, denom, rounding, RowCopies{}, stream);
    else if (dtype_code == LLNV_DTYPE_FP16) rc = launch_kv<__half>(tab, n, rows, denom, rounding, RowCopies{}, stream);
    else rc = launch_kv<float>(tab, n, rows, denom, rounding, RowCopies{}, stream);
    if (rc != LLNV_OK) return rc;
  }
  return LLNV_OK;
}
