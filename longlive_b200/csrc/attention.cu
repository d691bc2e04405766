// Non-causal attention of a query chunk over a key/value window, bf16 in / bf16 out, fp32
// softmax, on tcgen05 tensor cores (kind::f16) with the score and output accumulators in tensor
// memory.  head_dim = 128.
//
//   O[q, h, :] = softmax_k( Q[q, h, :] . K[k, h, :] * scale ) V[k, h, :]
//
// One CTA per (256-query tile, head), three warpgroups.  The tile is processed as two independent
// 128-query halves a and b that share the K/V tiles and ONE score buffer in tensor memory:
//
//   columns   0..127  S   scores of the half whose turn it is (fp32)
//           128..255  P   probabilities as packed bf16, 64 columns per half
//           256..511  O   output accumulators, 128 columns per half
//
// A softmax thread (one per query row) takes its 128 scores into registers at once, so the buffer is
// free for the other half a few hundred cycles after it was filled: S of half b is computed while half a
// is in its exponentials and the next S of half a before half a has finished with the present one.
// The softmax therefore never waits for a score tile, the halves run half a tile apart (so that one
// uses the special-function unit while the other waits, loads and reduces), and S = Q K^T still runs as
// 128 x 128 MMAs (64-key pieces would read Q from shared memory twice).  Roles:
//   warp 0       TMA: both Q halves once, then K and V tiles of 128 keys (two 64-channel halves each,
//                128-byte swizzle), two stages.
//   warps 1, 2   MMA issue for half a / half b (warp 1 owns the TMEM allocation).  Per key tile: S(j+1) once the other half
//                has read the buffer, then O += P V in two groups of 64 keys as the softmax finishes them (P read from
//                tensor memory, V MN-major in shared memory).  Two issuing threads, because a satisfied mbarrier wait takes
//                an issuing thread 150 cycles and more while the tensor cores stream operands, and with one thread
//                those add up to a third of a tile.
//   warps 4-7    softmax of half a, warps 8-11 of half b.  The output accumulator is rescaled lazily: only when a row
//                maximum grows by more than 2^8 is O multiplied by exp2(m_old - m_new), so in steady state O is touched only
//                by the tensor pipe.  After the last tile the same warps normalise O and store it through swizzled shared
//                memory (the Q tile's buffer) with TMA.
// All mbarrier waits are bounded (sm100.cuh).
//
// What bounds it: at 2640 x 13200 x 24 a 256 x 128 tile takes about 2570 cycles against 2048 of MMA time, at the 1.53 GHz the
// power limit leaves under back-to-back launches: 349 us = 1227 TFLOP/s (423 us with both halves' softmax waiting on their
// own score buffers and one issuing thread).
//
// The window may come in two pieces (keys [0, 128 * first_tiles) and the rest): the NVFP4 window of llnv_attention_nvfp4kv is
// expanded to bf16 in a workspace by one dequantize launch (26 us of HBM time on the shape above) and read from there, while
// the current chunk is read in place.
//
// A call whose workspace has no room for the expanded window takes attention_kernel<true>, which needs none: four more warps
// (12-15) decode the cached keys and values inside the load stage.  That repeats the decode for each of a head's query tiles and is
// bound by shared-memory bandwidth (MMA operands plus the expanded tiles).  us with the expansion / without, 4 cached blocks and the
// chunk: 2640 x 24 heads 371 / 467, 2640 x 12 190 / 250, 660 x 24 48 / 54, 660 x 3 25.5 / 27.4; 2 blocks, 2640 x 6 74.5 / 100.
// Warp 0 loads Q and the K side, warp 3 the V side: the 128 x 64-byte code tile of the stage's next key tile (one box per cache block
// the tile touches, at most two) goes into the tail of the K / V stage itself, which is free at that point.  Decode thread i owns key row i: it
// takes the row's 64 code bytes from there and its 8 scale bytes from global memory (one tile ahead) and writes the bf16 row over the
// stage in the swizzled layout the MMAs read, the bytes a TMA load of the expanded window would have put there.  The value of a code,
//     bf16((e2m1 * e4m3) * (amax * fp32(1 / (e2m1_max * e4m3_max)))),
// depends within one block only on scale byte and code: when a tile first touches a block, the eight bf16 magnitudes of each of the
// 128 scale bytes go into a 2 KiB table (byte-split for prmt), and a row is decoded with byte permutes alone.  A tile that holds the last
// cached keys and the first keys of the current chunk is built by these warps too; tiles in the current chunk come from TMA.  One
// thread issues the MMAs of both halves, and the softmax reads its scores twice in a rolled loop: with the decode's code the
// unrolled one overflows the instruction cache (467 -> 498 us).  Registers: load / MMA warpgroup 56, decode 104, softmax 176.
//
// Work split.  blockIdx.z = key split: with nsplit > 1 every (query tile, head) item is cut into nsplit equal ranges of key
// tiles, each CTA writes unnormalised fp32 partials and (m, l), and attention_combine_kernel merges them (head shards with
// too few items to fill the device).  Tail balancing (tail_cut > 0) cuts only the items of the last partial wave, once, into a
// long and a short CTA, so that the short ones fill the SMs the long ones leave free (see tail_cut_for).
#include <climits>

#include <cuda.h>

#include "common.cuh"
#include "sm100.cuh"

namespace llnv {

// dequant.cu: cached blocks -> bf16 [tokens, heads * 128] matrices of keys and values, n_pad rows of the current chunk behind them
int kv_window_dequant(const void* const* k_codes, const void* const* k_sf, const float* const* k_amax, const void* const* v_codes,
                      const void* const* v_sf, const float* const* v_amax, int num_blocks, int heads, int block_tokens, float denom,
                      const void* k_cur, const void* v_cur, int64_t ldk, int64_t ldv, int n_pad, void* k_out, void* v_out, cudaStream_t stream);

namespace {

using namespace sm100;
constexpr int kD = 128;            // head dim
constexpr int kBQ = 256;           // queries per CTA (two halves of 128)
constexpr int kHQ = 128;           // queries per half
constexpr int kBK = 128;           // keys per tile
constexpr int kStages = 2;
constexpr uint32_t kHalfBytes = 128 * 128;        // 128 rows x 64 bf16
constexpr uint32_t kTileBytes = 2 * kHalfBytes;   // 32 KiB
constexpr uint32_t kQOff = 0;
constexpr uint32_t kKOff = 2 * kTileBytes;
constexpr uint32_t kVOff = kKOff + kStages * kTileBytes;
constexpr uint32_t kBarOff = kVOff + kStages * kTileBytes;
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxKvBlocks = 16;
// attention_kernel<true>: decode tables behind the barriers, kTabSlots cache blocks x (K, V) x 128 scale bytes x 16 bytes
constexpr int kTabSlots = 2;                      // a tile of 128 keys touches at most two cache blocks (blocks hold >= 128 tokens)
constexpr uint32_t kCodeBytes = 128 * 64;         // code tile of one cache block: 128 key rows x 64 bytes, 64-byte swizzle
constexpr uint32_t kCodeOff = kTileBytes - 2 * kCodeBytes;      // two code tiles in the tail of the stage they expand into
constexpr uint32_t kTabOff = kBarOff + 1024;
constexpr uint32_t kSmemBytesFused = kTabOff + kTabSlots * 2 * 128 * 16;
static_assert(kSmemBytesFused <= 232448, "more shared memory than one CTA may use");

constexpr uint32_t kSmemBytes = kBarOff + 1024;
constexpr uint32_t kSCol = 0, kPCol = 128, kOCol = 256;      // one S tile, P_h at kPCol + 64 h, O_h at kOCol + 128 h
constexpr int kThreads = 384;      // three warpgroups: load + MMA, softmax a, softmax b
constexpr int kThreadsFused = 512; // and a fourth: decode

struct AttnParams {
  int64_t Lq, Lk;
  int heads;
  float scale_log2;            // scale * log2(e)
  unsigned int* status;
  // key splits: CTA z of a (query tile, head) handles a contiguous range of the key tiles and,
  // when there is more than one split, writes its unnormalised output and (m, l) to the workspace
  // tail balancing (tail_cut > 0, nsplit == 1, grid z = 2): (query tile, head) items are numbered in launch order
  // (tile + tiles * head); items below tail_first run whole in their z = 0 CTA, the others are cut at key tile
  // tail_cut into a z = 0 CTA and a shorter z = 1 CTA, both writing partial results
  int nsplit, tail_first, tail_cut;
  float* part_o;               // [nsplit][Lq][heads][128] fp32
  float* part_ml;              // [nsplit][Lq][heads][2]   fp32: exponent offset m (raw score units), sum l
  float* out_amax;             // optional: max |out| over all written elements (zeroed by the host before the launch)
  // key tiles [0, first_tiles) come from the first K / V tensors (rows from 0), the others from the second ones,
  // whose row second_row holds the first key of tile first_tiles
  int first_tiles, second_row;
};

// Tensor-memory columns of a half's scores and probabilities.  FUSED: a score buffer for each half, which the probabilities overwrite
// (S(j + 1) is issued behind the products of tile j).  The K tiles are late there, and with the shared buffer one that half a has read
// waits for half b's turn: 2640 x 7920 x 6 heads 111 us, with a buffer each 99.
template <bool FUSED>
__device__ __forceinline__ uint32_t s_col(int h) { return kSCol + (FUSED ? 128 * h : 0); }
template <bool FUSED>
__device__ __forceinline__ uint32_t p_col(int h) { return FUSED ? kSCol + 128 * h : kPCol + 64 * h; }

// The cached blocks of an attention_kernel<true> launch (oldest first); the kernel without them takes an empty table.
template <bool FUSED>
struct KvTable {};
template <>
struct KvTable<true> {
  const uint8_t* k_sf[kMaxKvBlocks];
  const float* k_amax[kMaxKvBlocks];
  const uint8_t* v_sf[kMaxKvBlocks];
  const float* v_amax[kMaxKvBlocks];
  // codes of block b viewed as [block_tokens, heads * 64 bytes]: box = 128 tokens x the 64 bytes of one head
  CUtensorMap k_codes[kMaxKvBlocks];
  CUtensorMap v_codes[kMaxKvBlocks];
  int n_cached, block_tokens;
  float inv_denom;             // fp32(1 / (e2m1_max * e4m3_max))
  const uint16_t* k_cur;       // current chunk: rows of the tile it shares with the cache
  const uint16_t* v_cur;
  int64_t ldk, ldv;
};

// The CTA's share of the key tiles: [j0, j0 + nt).  False: this CTA has nothing to do (tail balancing, whole item).
__device__ __forceinline__ bool key_range(const AttnParams& p, int qt, int head, int& j0, int& nt, bool& partial) {
  const int nt_all = (int)((p.Lk + kBK - 1) / kBK);
  j0 = (int)((int64_t)blockIdx.z * nt_all / p.nsplit);
  nt = (int)((int64_t)(blockIdx.z + 1) * nt_all / p.nsplit) - j0;           // >= 1: the host keeps nsplit <= nt_all
  partial = p.part_o != nullptr;
  if (p.tail_cut > 0) {
    if (qt + (int)gridDim.x * head < p.tail_first) {
      if (blockIdx.z != 0) return false;
      partial = false;
    } else {
      j0 = blockIdx.z == 0 ? 0 : p.tail_cut;
      nt = blockIdx.z == 0 ? p.tail_cut : nt_all - p.tail_cut;
    }
  }
  return true;
}

template <int N>
__device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// What a decode thread keeps of its key row between the prefetch and the decode.
struct RowInfo {
  uint32_t ksf[2], vsf[2];      // kind 0: the row's 8 K and 8 V scale bytes
  int kind;                     // 0 = cache block, 1 = current chunk, 2 = beyond the window
  int where;                    // kind 0: row inside the staged code tiles (128.. = second tile) | table slot << 8;
                                // kind 1: row of the current chunk
};

// Decode table of one (cache block, scale byte): the bf16 magnitudes of the eight E2M1 magnitudes
// {0, .5, 1, 1.5, 2, 3, 4, 6} under that scale, computed as decode16<LLNV_DEQ_FUSED> of the standalone
// dequantize kernel computes them, stored byte-split: x = low bytes of magnitudes 0..3, y = low bytes of
// 4..7, z / w = the high bytes.
__device__ __forceinline__ uint4 decode_table_entry(uint32_t scale_byte, float g) {
  const float s = e4m3_to_float(scale_byte);
  const float mags[8] = {0.f, 0.5f, 1.f, 1.5f, 2.f, 3.f, 4.f, 6.f};
  uint32_t pk[4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
    pk[m] = pack_bf16x2(__fmul_rn(__fmul_rn(mags[2 * m], s), g), __fmul_rn(__fmul_rn(mags[2 * m + 1], s), g));
  uint4 t;
  t.x = __byte_perm(pk[0], pk[1], 0x6420);
  t.y = __byte_perm(pk[2], pk[3], 0x6420);
  t.z = __byte_perm(pk[0], pk[1], 0x7531);
  t.w = __byte_perm(pk[2], pk[3], 0x7531);
  return t;
}

// 8 codes (one word) -> 8 bf16 (16 bytes) with the table entry `t` of the codes' scale byte: four byte lookups
// (low / high bytes of codes 0..3 and 4..7), the sign bits, four interleaves.
__device__ __forceinline__ uint4 decode_word(uint32_t w, const uint4& t) {
  const uint32_t sel = w & 0x77777777u;             // magnitude indices of codes 0..3 (low half) and 4..7
  const uint32_t selb = sel >> 16;
  const uint32_t w4 = w << 4;                       // bit 7 of byte k: sign of code 2k (of w: sign of code 2k+1)
  const uint32_t lo_a = __byte_perm(t.x, t.y, sel), lo_b = __byte_perm(t.x, t.y, selb);
  uint32_t hi_a = __byte_perm(t.z, t.w, sel), hi_b = __byte_perm(t.z, t.w, selb);
  hi_a |= __byte_perm(w4, w, 0x5140) & 0x80808080u;
  hi_b |= __byte_perm(w4, w, 0x7362) & 0x80808080u;
  return make_uint4(__byte_perm(lo_a, hi_a, 0x5140), __byte_perm(lo_a, hi_a, 0x7362), __byte_perm(lo_b, hi_b, 0x5140),
                    __byte_perm(lo_b, hi_b, 0x7362));
}

// Decode a cached row (code words w[0..15], scale bytes sf0 | sf1) into row i of a K / V stage: two halves of 64
// channels, rows of 128 bytes, 16-byte chunks XOR-swizzled with the row index as a TMA load with the 128-byte
// swizzle writes them.  `tab` is the row's block's table (128 entries of 16 bytes) in shared memory.  The loop
// over the four 32-channel groups stays rolled (the words rotate through w[0..3]): unrolled, this code and the
// softmax's together overflow the instruction cache.
__device__ __forceinline__ void decode_row(uint32_t (&w)[16], uint32_t sf0, uint32_t sf1, const uint8_t* tab, uint8_t* stage, int i) {
  uint8_t* dst = stage + i * 128;
  const int x = i & 7;
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {                       // 32 channels: two scale bytes, four 16-byte chunks
    const uint32_t sfw = (c & 2 ? sf1 : sf0) >> (16 * (c & 1));
    // table entries of the two scale bytes (bit 7 of a UE4M3 scale is never set): byte * 16
    const uint4 t0 = *reinterpret_cast<const uint4*>(tab + ((sfw << 4) & 0x7F0u));
    const uint4 t1 = *reinterpret_cast<const uint4*>(tab + ((sfw >> 4) & 0x7F0u));
    uint8_t* half = dst + (c >> 1) * kHalfBytes;
    const int k0 = (c & 1) * 4;                       // first chunk of the group inside its half
    *reinterpret_cast<uint4*>(half + (((k0 + 0) ^ x) << 4)) = decode_word(w[0], t0);
    *reinterpret_cast<uint4*>(half + (((k0 + 1) ^ x) << 4)) = decode_word(w[1], t0);
    *reinterpret_cast<uint4*>(half + (((k0 + 2) ^ x) << 4)) = decode_word(w[2], t1);
    *reinterpret_cast<uint4*>(half + (((k0 + 3) ^ x) << 4)) = decode_word(w[3], t1);
#pragma unroll
    for (int k = 0; k < 12; ++k) w[k] = w[k + 4];
  }
}

// Row i of a stage from 128 bf16 values in global memory (src == nullptr: zeros).
__device__ __forceinline__ void copy_row(const uint16_t* src, uint8_t* stage, int i) {
#pragma unroll 4
  for (int chunk = 0; chunk < 16; ++chunk) {
    const uint4 v = src ? ld_global(reinterpret_cast<const uint4*>(src) + chunk) : make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(stage + (chunk >> 3) * kHalfBytes + i * 128 + (((chunk & 7) ^ (i & 7)) << 4)) = v;
  }
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// three-input maximum (one instruction on sm_100) and packed two-lane fp32 arithmetic: they halve
// the instruction count of the row maximum, the score scaling and the row sum.  The maxima pass a NaN on (see row_max).
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float fmax2(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b, float c) {
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\tmov.b64 rc, {%5, %5};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d0), "=f"(d1)
      : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void add2(float& d0, float& d1, float a0, float a1) {
  asm("{\n\t.reg .b64 ra, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rd, {%0, %1};\n\t"
      "add.rn.f32x2 rd, rd, ra;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "+f"(d0), "+f"(d1)
      : "f"(a0), "f"(a1));
}

// exp2 of two values on the FMA pipe, for a share of the scores: floor by a round-down add of 1.5 * 2^23, a quartic for
// 2^frac on [0, 1) (equal-ripple fit of the relative error with the constant term fixed at 1, by linear programming: 3e-6,
// a thousandth of the bf16 rounding of P; the cubic of the same kind has 8.6e-5), exponent added as an integer.  The clamp takes
// a NaN for -125: the caller's row maximum has to carry it.
__device__ __forceinline__ F2 ex2_poly2(F2 x) {
  x.x = fmaxf(x.x, -125.f);
  x.y = fmaxf(x.y, -125.f);
  F2 r;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\t"
      "add.rm.ftz.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(12582912.f));
  const F2 f = f2_sub(x, f2_add(r, f2_splat(-12582912.f)));            // fraction in [0, 1)
  F2 pl = f2_fma(f, f2_splat(0.013425155f), f2_splat(0.052245375f));
  pl = f2_fma(pl, f, f2_splat(0.24127856f));
  pl = f2_fma(pl, f, f2_splat(0.69304514f));
  pl = f2_fma(pl, f, f2_splat(1.f));
  return F2{__int_as_float(__float_as_int(pl.x) + (__float_as_int(r.x) << 23)), __int_as_float(__float_as_int(pl.y) + (__float_as_int(r.y) << 23))};
}
// Pair p of a row's scores takes the FMA-pipe exp2.  One pair in four: per 256 x 128 tile the special-function unit is then
// busy 1540 cycles of about 2570.  (2640 x 13200 x 24 heads, us: a quarter of the pairs 350.5, a third 349.0, two fifths 356, half
// 368: the quarter leaves the FMA pipe and the issue slots more room at the same time within the spread of runs.)
__host__ __device__ constexpr bool poly_pair(int p) { return p % 4 == 1; }

// Maximum of a row's scores: independent chains of three-input maxima.  NaN if a score is NaN, whatever its column: the FMA-pipe
// exponential would lose it.
template <int G>
__device__ __forceinline__ float row_max(const uint32_t (&sr)[G][32]) {
  constexpr int kChains = 8;
  float mx[kChains];
#pragma unroll
  for (int i = 0; i < kChains; ++i) mx[i] = fmax2(__uint_as_float(sr[0][2 * i]), __uint_as_float(sr[0][2 * i + 1]));
#pragma unroll
  for (int i = 2 * kChains; i < 32 * G; i += 2) {
    float& x = mx[(i >> 1) % kChains];
    x = fmax3(x, __uint_as_float(sr[i >> 5][i & 31]), __uint_as_float(sr[i >> 5][(i & 31) + 1]));
  }
#pragma unroll
  for (int w = kChains / 2; w > 0; w >>= 1)
#pragma unroll
    for (int i = 0; i < w; ++i) mx[i] = fmax2(mx[i], mx[i + w]);
  return mx[0];
}

// Columns at or beyond `valid` become -inf (only the last key tile of a window can be ragged).
template <int G>
__device__ __forceinline__ void mask_scores(uint32_t (&sr)[G][32], int valid) {
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int nv = valid - 32 * g;                // valid columns of this group of 32
    const uint32_t keep = nv >= 32 ? 0xFFFFFFFFu : (nv <= 0 ? 0u : ((1u << nv) - 1u));
#pragma unroll
    for (int i = 0; i < 32; ++i) sr[g][i] = ((keep >> i) & 1u) ? sr[g][i] : 0xFF800000u;
  }
}

// exp2(s * c + nmc) of 32 scores, the g-th quarter of a row: the row's running sums (four packed accumulators) and the packed bf16 values.
__device__ __forceinline__ void exp_group(const uint32_t (&s)[32], int g, float c, float nmc, float (&l)[8], uint32_t (&pk)[16]) {
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    F2 x, e;
    fma2(x.x, x.y, __uint_as_float(s[i]), __uint_as_float(s[i + 1]), c, nmc);
    if (poly_pair((32 * g + i) >> 1)) {
      e = ex2_poly2(x);
    } else {
      e.x = ex2(x.x);
      e.y = ex2(x.y);
    }
    const int a = ((i >> 1) & 3) * 2;
    add2(l[a], l[a + 1], e.x, e.y);
    pk[i >> 1] = pack2(e.x, e.y);
  }
}

// Multiply the output accumulator of this thread's row by alpha.
__device__ __forceinline__ void rescale_output(uint32_t o_tmem, float alpha) {
#pragma unroll 1
  for (int g = 0; g < 4; ++g) {
    uint32_t o[32];
    tmem_ld32(o_tmem + 32 * g, o);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
    tmem_st32(o_tmem + 32 * g, o);
  }
  tmem_st_wait();
}

// Epilogue of one softmax warp: O / l -> bf16 -> swizzled staging (the Q tile's shared memory) -> TMA store, or the
// unnormalised fp32 output and (m, l) for the combine kernel.  o_tmem: this warp's lanes of the half's accumulator.
__device__ __forceinline__ void write_output(const AttnParams& p, const CUtensorMap* tmO, uint8_t* smem, uint32_t o_tmem, int qt, int head,
                                             int half, int q, int lane, bool partial, float m, float lsum) {
  const int row0 = qt * kBQ + half * kHQ + q * 32;
  if (partial) {
    // one of several key splits: unnormalised fp32 output and (m, l) for the combine kernel
    const int64_t grow = (int64_t)row0 + lane;
    const int64_t slot = ((int64_t)blockIdx.z * p.Lq + grow) * p.heads + head;
    float4* dst = reinterpret_cast<float4*>(p.part_o + slot * kD);
#pragma unroll 1
    for (int g = 0; g < 4; ++g) {
      uint32_t o[32];
      tmem_ld32(o_tmem + 32 * g, o);
      tmem_ld_wait();
      if (grow < p.Lq) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          dst[g * 8 + i] = make_float4(__uint_as_float(o[4 * i]), __uint_as_float(o[4 * i + 1]), __uint_as_float(o[4 * i + 2]),
                                       __uint_as_float(o[4 * i + 3]));
      }
    }
    if (grow < p.Lq) *reinterpret_cast<float2*>(p.part_ml + slot * 2) = make_float2(m, lsum);
    return;
  }
  const float inv_l = 1.f / lsum;
  uint32_t amax2 = 0u;          // packed running max of |out| (bf16 pairs; the magnitudes compare as integers)
#pragma unroll 1
  for (int dh = 0; dh < 2; ++dh) {
    uint32_t o[2][32];
    tmem_ld32(o_tmem + 64 * dh, o[0]);
    tmem_ld32(o_tmem + 64 * dh + 32, o[1]);
    tmem_ld_wait();
    uint8_t* buf = smem + kQOff + half * kTileBytes + dh * kHalfBytes + q * 4096;      // 32 rows x 128 bytes
#pragma unroll
    for (int v8 = 0; v8 < 8; ++v8) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int cc = v8 * 8 + 2 * e;
        const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(o[cc >> 5][cc & 31]) * inv_l,
                                                        __uint_as_float(o[(cc + 1) >> 5][(cc + 1) & 31]) * inv_l);
        w[e] = *reinterpret_cast<const uint32_t*>(&b2);
        amax2 = __vmaxu2(amax2, w[e] & 0x7FFF7FFFu);
      }
      *reinterpret_cast<uint4*>(buf + lane * 128 + ((v8 ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0 && row0 < p.Lq) {
      tma_store_2d(tmO, buf, head * kD + dh * 64, row0);
      bulk_commit();
    }
  }
  if (p.out_amax) {
    // rows at or beyond Lq are not written (the TMA store clips them) and must not count
    float a = row0 + lane < p.Lq ? __uint_as_float(max(amax2 & 0xFFFFu, amax2 >> 16) << 16) : 0.f;
    a = warp_max(a);
    if (lane == 0 && a > 0.f) atomic_max_nonneg(p.out_amax, a);
  }
  if (lane == 0) bulk_wait<0>();
}

// S = Q K^T of one half and key tile
__device__ __forceinline__ void issue_scores(uint32_t s_tmem, uint32_t q_addr, uint32_t k_addr) {
  constexpr uint32_t idesc = make_idesc_bf16(kHQ, kBK, 0, 0);     // A, B K-major
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    // 16 channels per MMA: 32 bytes along the swizzled 128-byte row, second half after 4 steps
    const uint32_t off = (ks >> 2) * kHalfBytes + (ks & 3) * 32;
    mma_f16_ss(s_tmem, make_kmajor_sw128_desc(q_addr + off), make_kmajor_sw128_desc(k_addr + off), idesc, ks != 0);
  }
}
// O (+)= P V of one half, keys 16 * KS0 .. 16 * KS1 - 1 of a tile
template <int KS0, int KS1>
__device__ __forceinline__ void issue_products(uint32_t o_tmem, uint32_t p_tmem, uint32_t v_addr, bool accumulate) {
  constexpr uint32_t idesc = make_idesc_bf16(kHQ, kD, 0, 1);      // B (V) MN-major
#pragma unroll
  for (int ks = KS0; ks < KS1; ++ks) {
    // 16 keys per MMA: P columns 8*ks..8*ks+7 (two bf16 per column), V rows 16*ks.. (2048 bytes apart)
    // V is MN-major: 64 channels contiguous per key row, the second 64 channels one half-tile further
    mma_f16_ts(o_tmem, p_tmem + 8 * ks, make_smem_desc(v_addr + ks * 2048, kHalfBytes, 1024, 2), idesc, accumulate || ks != 0);
  }
}

template <bool FUSED>
__global__ void __launch_bounds__(FUSED ? kThreadsFused : kThreads, 1)
attention_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                 const __grid_constant__ CUtensorMap tmK2, const __grid_constant__ CUtensorMap tmV2, const __grid_constant__ CUtensorMap tmO,
                 const AttnParams p, const __grid_constant__ KvTable<FUSED> tab) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + kBarOff);
  uint64_t* k_full = q_full + 1;
  uint64_t* k_empty = k_full + kStages;
  uint64_t* v_full = k_empty + kStages;
  uint64_t* v_empty = v_full + kStages;
  uint64_t* s_full = v_empty + kStages;        // [2 halves]: the S buffer holds the half's scores
  uint64_t* s_free = s_full + 2;               // [2 halves]: the half has its scores in registers
  uint64_t* p_ready = s_free + 2;              // [2 halves][2 key groups of 64]
  uint64_t* pv_done = p_ready + 4;             // [2 halves][2 key groups]
  uint64_t* kc_full = pv_done + 4;             // [kStages] code tiles of a K / V stage have landed (FUSED)
  uint64_t* vc_full = kc_full + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(vc_full + kStages);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = blockIdx.x, head = blockIdx.y;
  int j0, nt;
  bool partial;
  if (!key_range(p, qt, head, j0, nt, partial)) {                // nothing is set up yet: the CTA just leaves
    pdl_wait();
    return;
  }
  const int n_half = ((int64_t)qt * kBQ + kHQ < p.Lq) ? 2 : 1;     // the second half may lie entirely beyond Lq

  if ((smem_u32(smem) & 1023u) != 0) {
    pdl_wait();
    if (threadIdx.x == 0 && p.status && atomicCAS(p.status, 0u, 2u) == 0u) p.status[1] = 901u;
    return;
  }
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], FUSED ? 1 : n_half);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], FUSED ? 1 : n_half);
      mbar_init(&kc_full[i], 1);
      mbar_init(&vc_full[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 4);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&p_ready[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    *abort_flag = 0u;
    fence_barrier_init();
    prefetch_tensormap(&tmQ);
    prefetch_tensormap(&tmK);
    prefetch_tensormap(&tmV);
    prefetch_tensormap(&tmK2);
    prefetch_tensormap(&tmV2);
    prefetch_tensormap(&tmO);
  }
  pdl_wait();
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  pdl_trigger();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // The register file is re-divided at the top of every warpgroup's branch (all four warps of a warpgroup execute the same
  // instruction; an increase waits for the other warpgroups' releases): 12 warps x 32 x 168 registers at launch = 64512 >=
  // 128 x (80 + 2 x 208); FUSED: 16 warps x 32 x 128 = 65536 = 128 x (56 + 2 x 176 + 104).
  if (warp < 4) setmaxnreg_dec<FUSED ? 56 : 80>();

  if (warp == 0 || (FUSED && warp == 3)) {
    // ------------------------------------------------------------------ TMA producer
    // FUSED: warp 0 loads Q and feeds the K stages, warp 3 feeds the V stages, so that neither side queues behind the other's stage
    const bool do_k = warp == 0, do_v = !FUSED || warp == 3;
    if (elect_one()) {
      const int col = head * kD;
      if (do_k) {
        mbar_arrive_expect_tx(q_full, n_half * kTileBytes);
        for (int h = 0; h < n_half; ++h) {
          tma_load_2d(smem + kQOff + h * kTileBytes, &tmQ, col, qt * kBQ + h * kHQ, q_full);
          tma_load_2d(smem + kQOff + h * kTileBytes + kHalfBytes, &tmQ, col + 64, qt * kBQ + h * kHQ, q_full);
        }
      }
      // (block, token) of the first key of tile j, advanced tile by tile
      int b0 = 0, tok0 = 0;
      if constexpr (FUSED) {
        b0 = (int)(((int64_t)j0 * kBK) / tab.block_tokens);
        tok0 = (int)((int64_t)j0 * kBK - (int64_t)b0 * tab.block_tokens);
      }
      for (int j = 0; j < nt; ++j) {
        const int s = j % kStages;
        const uint32_t ph = (uint32_t)((j / kStages) & 1);
        const int t = j0 + j;
        const bool first = t < p.first_tiles;
        if constexpr (FUSED) {
          if (first) {
            // a tile the decode warps build: its codes go into the tail of the (free) stage, one box of 128 token rows per cache
            // block the tile touches; rows beyond a block's end arrive as zeros and are not used
            const bool two = tok0 + kBK > tab.block_tokens && (int64_t)(b0 + 1) * tab.block_tokens < tab.n_cached;
            const uint32_t bytes = two ? 2 * kCodeBytes : kCodeBytes;
            uint8_t* stage = smem + (do_k ? kKOff : kVOff) + s * kTileBytes + kCodeOff;
            uint64_t* full = do_k ? &kc_full[s] : &vc_full[s];
            const CUtensorMap* codes = do_k ? tab.k_codes : tab.v_codes;
            mbar_wait(do_k ? &k_empty[s] : &v_empty[s], ph ^ 1u, abort_flag, p.status, do_k ? 102u : 103u);
            mbar_arrive_expect_tx(full, bytes);
            tma_load_2d(stage, &codes[b0], head * 64, tok0, full);
            if (two) tma_load_2d(stage + kCodeBytes, &codes[b0 + 1], head * 64, 0, full);
            tok0 += kBK;
            if (tok0 >= tab.block_tokens) { tok0 -= tab.block_tokens; ++b0; }
            continue;
          }
        }
        const CUtensorMap* mk = first ? &tmK : &tmK2;
        const CUtensorMap* mv = first ? &tmV : &tmV2;
        const int krow = first ? t * kBK : (t - p.first_tiles) * kBK + p.second_row;
        if (do_k) {
          mbar_wait(&k_empty[s], ph ^ 1u, abort_flag, p.status, 100u);
          mbar_arrive_expect_tx(&k_full[s], kTileBytes);
          tma_load_2d(smem + kKOff + s * kTileBytes, mk, col, krow, &k_full[s]);
          tma_load_2d(smem + kKOff + s * kTileBytes + kHalfBytes, mk, col + 64, krow, &k_full[s]);
        }
        if (do_v) {
          mbar_wait(&v_empty[s], ph ^ 1u, abort_flag, p.status, 101u);
          mbar_arrive_expect_tx(&v_full[s], kTileBytes);
          tma_load_2d(smem + kVOff + s * kTileBytes, mv, col, krow, &v_full[s]);
          tma_load_2d(smem + kVOff + s * kTileBytes + kHalfBytes, mv, col + 64, krow, &v_full[s]);
        }
      }
    }
  } else if (FUSED && warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of both halves
    // A K tile is free as soon as both halves have read it, and one that is still being decoded holds up no products.
    if (elect_one()) {
      auto issue_qk = [&](int t, int h) {
        const int s = t % kStages;
        issue_scores(tmem_base + s_col<FUSED>(h), smem_u32(smem + kQOff + h * kTileBytes), smem_u32(smem + kKOff + s * kTileBytes));
        tc_commit(&s_full[h]);
        if (h == n_half - 1) tc_commit(&k_empty[s]);
      };
      mbar_wait(q_full, 0u, abort_flag, p.status, 201u);
      mbar_wait(&k_full[0], 0u, abort_flag, p.status, 200u);
      tc_fence_after();
      for (int h = 0; h < n_half; ++h) issue_qk(0, h);
      for (int j = 0; j < nt; ++j) {
        const int s = j % kStages;
        mbar_wait(&v_full[s], (uint32_t)((j / kStages) & 1), abort_flag, p.status, 203u);
        for (int h = 0; h < n_half; ++h) {
          mbar_wait(&p_ready[2 * h + 1], (uint32_t)(j & 1), abort_flag, p.status, 202u);
          tc_fence_after();
          issue_products<0, 8>(tmem_base + kOCol + 128 * h, tmem_base + p_col<FUSED>(h), smem_u32(smem + kVOff + s * kTileBytes), j != 0);
          tc_commit(&pv_done[2 * h + 1]);
          if (h == n_half - 1) tc_commit(&v_empty[s]);
          if (j + 1 < nt) {
            if (h == 0) {
              mbar_wait(&k_full[(j + 1) % kStages], (uint32_t)(((j + 1) / kStages) & 1), abort_flag, p.status, 204u);
              tc_fence_after();
            }
            issue_qk(j + 1, h);
          }
        }
      }
    }
  } else if (!FUSED && (warp == 1 || warp == 2)) {
    // ------------------------------------------------------------------ MMA issuers, one per half
    const int h = warp - 1;
    if (h < n_half && elect_one()) {
      const uint32_t q_addr = smem_u32(smem + kQOff + h * kTileBytes);
      const uint32_t s_tmem = tmem_base + s_col<FUSED>(h), p_tmem = tmem_base + p_col<FUSED>(h), o_tmem = tmem_base + kOCol + 128 * h;
      const int before = n_half == 2 ? h ^ 1 : 0;          // whose scores occupy the S buffer before mine do

      // S of tile t: the buffer must have been read by its previous user (half b's tile t - 1 before half a's tile t, half
      // a's tile t before half b's)
      auto issue_qk = [&](int t) {
        const int s = t % kStages;
        mbar_wait(&k_full[s], (uint32_t)((t / kStages) & 1), abort_flag, p.status, 204u);
        const int use = h == 1 ? t : t - 1;
        if (use >= 0) mbar_wait(&s_free[before], (uint32_t)(use & 1), abort_flag, p.status, 205u);
        tc_fence_after();
        issue_scores(s_tmem, q_addr, smem_u32(smem + kKOff + s * kTileBytes));
        tc_commit(&s_full[h]);
        tc_commit(&k_empty[s]);
      };

      mbar_wait(q_full, 0u, abort_flag, p.status, 201u);
      issue_qk(0);
      for (int j = 0; j < nt; ++j) {
        const int s = j % kStages;
        const uint32_t v_addr = smem_u32(smem + kVOff + s * kTileBytes);
        if (j + 1 < nt) issue_qk(j + 1);
        mbar_wait(&v_full[s], (uint32_t)((j / kStages) & 1), abort_flag, p.status, 203u);
        mbar_wait(&p_ready[2 * h], (uint32_t)(j & 1), abort_flag, p.status, 202u);
        tc_fence_after();
        issue_products<0, 4>(o_tmem, p_tmem, v_addr, j != 0);
        tc_commit(&pv_done[2 * h]);
        mbar_wait(&p_ready[2 * h + 1], (uint32_t)(j & 1), abort_flag, p.status, 202u);
        tc_fence_after();
        issue_products<4, 8>(o_tmem, p_tmem, v_addr, true);
        tc_commit(&pv_done[2 * h + 1]);
        tc_commit(&v_empty[s]);
      }
    }
  } else if (FUSED && warp >= 12) {
    if constexpr (FUSED) {
      // ------------------------------------------------------------------ NVFP4 decode (warps 12..15)
      // Thread i builds key row i of every tile: first the K stage (the MMAs need it first), then the V stage.
      setmaxnreg_dec<104>();
      const int nd = min(nt, p.first_tiles - j0);          // tiles of this CTA that hold cached keys; none where <= 0
      const int i = (int)threadIdx.x - 384;               // key row of the tile this thread builds; also its table entry
      const int H = p.heads;
      const int T = tab.block_tokens;
      const int n_cached = tab.n_cached, Lk = (int)p.Lk;      // the host keeps the window below 2^31 keys
      uint8_t* tabs = smem + kTabOff;                       // slot * 4096 + (K: 0, V: 2048) + entry * 16
      // (block, token) of the first key of the tile being fetched, advanced tile by tile (no divisions in the loop)
      int fb = (int)(((int64_t)j0 * kBK) / T);
      int ft = (int)((int64_t)j0 * kBK - (int64_t)fb * T);
      int fkey = j0 * kBK;
      // where key row i of the next tile lives, and its scale bytes (global loads, consumed one tile later)
      auto fetch = [&](RowInfo& r) {
        const int key = fkey + i;
        if (key >= n_cached) {
          r.where = key - n_cached;
          r.kind = key < Lk ? 1 : 2;
        } else {
          const bool second = ft + i >= T;                  // the row lies in the next cache block: second staged code tile
          const int b = second ? fb + 1 : fb;
          const int tok = second ? ft + i - T : ft + i;
          r.kind = 0;
          r.where = (second ? 128 + tok : i) | ((b % kTabSlots) << 8);
          const int row = tok * H + head;                   // row of the block: token-major, head-minor
          const int sf_off = (row >> 7) * 1024 + (row & 31) * 16 + ((row & 127) >> 5) * 4;   // scale columns 0..3; 4..7 are 512 bytes on
          r.ksf[0] = ld_global(reinterpret_cast<const uint32_t*>(tab.k_sf[b] + sf_off));
          r.ksf[1] = ld_global(reinterpret_cast<const uint32_t*>(tab.k_sf[b] + sf_off + 512));
          r.vsf[0] = ld_global(reinterpret_cast<const uint32_t*>(tab.v_sf[b] + sf_off));
          r.vsf[1] = ld_global(reinterpret_cast<const uint32_t*>(tab.v_sf[b] + sf_off + 512));
        }
        fkey += kBK;
        ft += kBK;
        if (ft >= T) { ft -= T; ++fb; }
      };
      // one of K / V of a tile: expand the staged codes (or copy the current chunk's rows) into stage `st`
      auto build = [&](const RowInfo& row, int kv, uint32_t sf0, uint32_t sf1, uint8_t* st, uint64_t* codes_full, uint64_t* full,
                       uint32_t ph) {
        // the stage is free and its code tiles have landed (the producer waited for the stage before it loaded them)
        mbar_wait(codes_full, ph, abort_flag, p.status, 400u + kv);
        uint32_t w[16];
        if (row.kind == 0) {
          // 64-byte rows, 16-byte chunks XOR-swizzled with bits 1-2 of the row index (TMA's 64-byte swizzle)
          const int cr = row.where & 0xFF;
          const uint8_t* src = st + kCodeOff + cr * 64;
          const int sw = (cr >> 1) & 3;
  #pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 v4 = *reinterpret_cast<const uint4*>(src + ((c ^ sw) << 4));
            w[4 * c] = v4.x; w[4 * c + 1] = v4.y; w[4 * c + 2] = v4.z; w[4 * c + 3] = v4.w;
          }
        }
        // Both barriers are executed by all 128 threads outside any divergent branch (a tile that mixes cache rows and
        // current-chunk rows splits a warp between the branches above and below; bar.sync needs converged warps).
        __syncwarp();
        asm volatile("bar.sync 1, 128;" ::: "memory");      // every thread holds its codes: the stage's tail may be overwritten
        if (row.kind == 0) {
          decode_row(w, sf0, sf1, tabs + (row.where >> 8) * 4096 + kv * 2048, st, i);
        } else {
          const uint16_t* src = nullptr;
          if (row.kind == 1) src = (kv ? tab.v_cur + (int64_t)row.where * tab.ldv : tab.k_cur + (int64_t)row.where * tab.ldk) + (int64_t)head * kD;
          copy_row(src, st, i);
        }
        fence_proxy_async();
        __syncwarp();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (i == 0) mbar_arrive(full);
      };
      // decode tables exist for cache blocks up to `built`; (lb, lt) = (block, token) of the last key of the current tile
      int built = fb - 1;
      int lb = (int)(((int64_t)j0 * kBK + kBK - 1) / T);
      int lt = (int)((int64_t)j0 * kBK + kBK - 1 - (int64_t)lb * T);
      const int last_block = n_cached > 0 ? (n_cached - 1) / T : 0;
      RowInfo nxt;
      nxt.kind = 2;
      if (nd > 0) fetch(nxt);
      for (int j = 0; j < nd; ++j) {
        const int s = j % kStages;
        const uint32_t ph = (uint32_t)((j / kStages) & 1);
        const RowInfo row = nxt;
        if (j + 1 < nd) fetch(nxt);                         // in flight while this tile is decoded
        const int b_hi = lb < last_block ? lb : last_block;
        lt += kBK;
        if (lt >= T) { lt -= T; ++lb; }
        if (b_hi > built) {               // the same for all 128 threads; the first barrier of `build` publishes the tables
          for (int b = built + 1; b <= b_hi; ++b) {
            uint8_t* tb = tabs + (b % kTabSlots) * 4096;
            *reinterpret_cast<uint4*>(tb + i * 16) = decode_table_entry((uint32_t)i, __fmul_rn(ld_global(tab.k_amax[b]), tab.inv_denom));
            *reinterpret_cast<uint4*>(tb + 2048 + i * 16) = decode_table_entry((uint32_t)i, __fmul_rn(ld_global(tab.v_amax[b]), tab.inv_denom));
          }
          built = b_hi;
        }
  #pragma unroll 1
        for (int kv = 0; kv < 2; ++kv)                      // K, then V: one copy of the build code
          build(row, kv, kv ? row.vsf[0] : row.ksf[0], kv ? row.vsf[1] : row.ksf[1], smem + (kv ? kVOff : kKOff) + s * kTileBytes,
                kv ? &vc_full[s] : &kc_full[s], kv ? &v_full[s] : &k_full[s], ph);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax + epilogue
    setmaxnreg_inc<FUSED ? 176 : 208>();
    const int q = warp & 3;
    const int half = warp >= 8 ? 1 : 0;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const float c = p.scale_log2;
    if (half < n_half) {
    float m = -INFINITY;          // exponent offset of the row (raw score units): the row maximum, updated lazily
    float l[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};        // running sum of exp: four packed accumulators
    const uint32_t s_tmem = tmem_base + lane_base + s_col<FUSED>(half);
    const uint32_t p_tmem = tmem_base + lane_base + p_col<FUSED>(half);
    const uint32_t o_tmem = tmem_base + lane_base + kOCol + 128 * half;
#pragma unroll 1
    for (int j = 0; j < nt; ++j) {
      const int valid = (int)min((int64_t)kBK, p.Lk - (int64_t)(j0 + j) * kBK);
      mbar_wait(&s_full[half], (uint32_t)(j & 1), abort_flag, p.status, 300u);
      tc_fence_after();
      // FUSED: 64 scores at a time in rolled loops, read for the maximum and again for the exponentials
      constexpr int kGroups = FUSED ? 2 : 4, kParts = 4 / kGroups;
      uint32_t sr[kGroups][32];
      auto load_scores = [&](int part) {
#pragma unroll
        for (int g = 0; g < kGroups; ++g) tmem_ld32(s_tmem + 32 * (kGroups * part + g), sr[g]);
        tmem_ld_wait();
        if (valid < kBK) mask_scores(sr, valid - 32 * kGroups * part);
      };
      float mt;
      if constexpr (FUSED) {
        mt = -INFINITY;
#pragma unroll 1
        for (int part = 0; part < kParts; ++part) {
          load_scores(part);
          mt = fmax2(mt, row_max(sr));
        }
      } else {
#pragma unroll
        for (int g = 0; g < 4; ++g) tmem_ld32(s_tmem + 32 * g, sr[g]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free[half]);       // the other half's scores may take the buffer
        if (valid < kBK) mask_scores(sr, valid);
        mt = row_max(sr);
      }
      // lazy rescale: keep the old offset unless this tile's maximum exceeds it by more than 2^8
      const bool grow = !((mt - m) * c <= 8.f);       // also true for the first tile (m = -inf) and for a NaN
      if (__any_sync(0xFFFFFFFFu, grow)) {
        if (j > 0) {
          // everything accumulated so far must have landed in O before it is rescaled
          mbar_wait(&pv_done[2 * half + 1], (uint32_t)((j - 1) & 1), abort_flag, p.status, 301u);
          tc_fence_after();
          const float m_new = grow ? mt : m;
          const float alpha = ex2((m - m_new) * c);
#pragma unroll
          for (int i = 0; i < 8; ++i) l[i] *= alpha;
          m = m_new;
          rescale_output(o_tmem, alpha);
        } else if (grow) {
          m = mt;                                      // nothing accumulated yet
        }
      }
      // A NaN or +inf score makes the row NaN, as inf - inf does in a softmax: NaN here reaches every exponential of the
      // special-function unit, and with them the row sum.
      const float nmc = __fmaf_rn(-m, c, m - m);
#pragma unroll 1
      for (int part = 0; part < kParts; ++part) {
        if constexpr (FUSED) load_scores(part);
#pragma unroll
        for (int gg = 0; gg < kGroups; ++gg) {
          const int g = kGroups * part + gg;
          uint32_t pk[16];
          exp_group(sr[gg], gg, c, nmc, l, pk);
          // the previous tile's products with this P group must have finished (FUSED: they have, S of this tile was issued behind them)
          if (!FUSED && (g & 1) == 0 && j > 0) {
            mbar_wait(&pv_done[2 * half + (g >> 1)], (uint32_t)((j - 1) & 1), abort_flag, p.status, 303u);
            tc_fence_after();
          }
          tmem_st16(p_tmem + 16 * g, pk);
          if (FUSED ? g == 3 : (g & 1)) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[2 * half + (g >> 1)]);
          }
        }
      }
    }
    const float lsum = ((l[0] + l[1]) + (l[2] + l[3])) + ((l[4] + l[5]) + (l[6] + l[7]));
    mbar_wait(&pv_done[2 * half + 1], (uint32_t)((nt - 1) & 1), abort_flag, p.status, 302u);
    tc_fence_after();
    write_output(p, &tmO, smem, o_tmem, qt, head, half, q, lane, partial, m, lsum);
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Merges the key splits: out = sum_z 2^((m_z - M) c) O_z / sum_z 2^((m_z - M) c) l_z with M = max_z m_z, z in order.
// One warp per query row of a (query tile, head) item, a lane owns four of the 128 channels.  Only items that were cut are visited
// (first_item: the first one; 0 with uniform splits).  Bound by latency: lane z holds (m_z, l_z), so that the weights cost one round of
// loads whatever the number of splits, and the outputs of four splits are loaded at a time.  us, cold caches, 1980 rows in 6 parts / 16896 in
// 2 / 29696 in 2: 4.6 / 7.4 / 10.9; four rows a warp with the loads of one split at a time 17.4 / 9.9 / 14, two rows 5.2 / 7.5 / 10.5.
__global__ void __launch_bounds__(256) attention_combine_kernel(const float* part_o, const float* part_ml, int nsplit, int64_t Lq, int heads,
                                                                float scale_log2, uint16_t* __restrict__ out, int64_t ldo,
                                                                float* __restrict__ out_amax, int first_item, int q_tiles) {
  pdl_begin();
  constexpr int kBatch = 4;
  const int lane = threadIdx.x & 31;
  const int item = first_item + (int)blockIdx.x / (kBQ / 8);
  const int head = item / q_tiles;
  const int64_t row = (int64_t)(item % q_tiles) * kBQ + ((int)blockIdx.x % (kBQ / 8)) * 8 + (threadIdx.x >> 5);
  if (row >= Lq) return;                                        // the whole warp
  const int64_t unit = row * heads + head, stride = Lq * heads;
  float2 ml[2];                                                 // of splits lane and lane + 32 (at most 64)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    ml[h] = make_float2(-INFINITY, 0.f);
    if (lane + 32 * h < nsplit) ml[h] = ld_global(reinterpret_cast<const float2*>(part_ml + ((lane + 32 * h) * stride + unit) * 2));
  }
  float4 o[kBatch];
  auto load = [&](int z0) {
#pragma unroll
    for (int i = 0; i < kBatch; ++i)
      if (z0 + i < nsplit) o[i] = ld_global(reinterpret_cast<const float4*>(part_o + ((z0 + i) * stride + unit) * kD) + lane);
  };
  load(0);
  const float mmax = warp_max(fmaxf(ml[0].x, ml[1].x));
#pragma unroll
  for (int h = 0; h < 2; ++h) ml[h].x = exp2f((ml[h].x - mmax) * scale_log2);       // the split's weight
  float lsum = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int z0 = 0; z0 < nsplit; z0 += kBatch) {
    if (z0 > 0) load(z0);
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int z = z0 + i;
      if (z >= nsplit) break;
      const float w = __shfl_sync(0xFFFFFFFFu, z < 32 ? ml[0].x : ml[1].x, z & 31);
      const float l = __shfl_sync(0xFFFFFFFFu, z < 32 ? ml[0].y : ml[1].y, z & 31);
      acc.x = __fmaf_rn(w, o[i].x, acc.x);
      acc.y = __fmaf_rn(w, o[i].y, acc.y);
      acc.z = __fmaf_rn(w, o[i].z, acc.z);
      acc.w = __fmaf_rn(w, o[i].w, acc.w);
      lsum = __fmaf_rn(w, l, lsum);
    }
  }
  const float inv = 1.f / lsum;
  uint2 packed;
  packed.x = pack2(acc.x * inv, acc.y * inv);
  packed.y = pack2(acc.z * inv, acc.w * inv);
  *reinterpret_cast<uint2*>(out + row * ldo + (int64_t)head * kD + lane * 4) = packed;
  if (out_amax) {
    const uint32_t m2 = __vmaxu2(packed.x & 0x7FFF7FFFu, packed.y & 0x7FFF7FFFu);
    const float a = warp_max(__uint_as_float(max(m2 & 0xFFFFu, m2 >> 16) << 16));
    if (lane == 0 && a > 0.f) atomic_max_nonneg(out_amax, a);
  }
}

}  // namespace
}  // namespace llnv

using namespace llnv;

// Tail balancing.  `items` (query tile, head) CTAs of `nt` key tiles each on `sms` SMs run floor(items / sms) full
// waves and then r = items % sms CTAs on an otherwise idle device.  Cutting each of those r items at key tile
// c = r * nt / sms gives r long CTAs (c tiles) and r short ones (nt - c tiles) that the hardware scheduler, which
// hands the next CTA to whichever SM frees up, packs onto the sms - r remaining SMs: the last wave then lasts about c
// tile times instead of nt.  Returns c, or 0 when there is no last partial wave or the saving is below 5 %.
static int tail_cut_for(int64_t items, int64_t nt, int sms) {
  const int64_t r = items % sms;
  if (items <= sms || r == 0 || nt < 16) return 0;
  int64_t c = (r * nt + sms - 1) / sms + 1;            // one extra tile pays for the second set-up of the short CTAs
  if (c < 4) c = 4;
  if (c > nt - 4) return 0;
  const int64_t before = (items / sms + 1) * nt, after = (items / sms) * nt + c;
  return (before - after) * 20 >= before ? (int)c : 0;
}

extern "C" int llnv_attention_key_splits(int64_t Lq, int64_t Lk, int heads) {
  if (Lq <= 0 || Lk <= 0 || heads <= 0) return 1;
  const int64_t ctas = ((Lq + kBQ - 1) / kBQ) * heads;
  const int64_t nt = (Lk + kBK - 1) / kBK;
  const int sms = sm_count();
  if (sms > 0 && ctas > sms && tail_cut_for(ctas, nt, sms) > 0) return LLNV_ATTN_SPLIT_TAIL;
  if (sms <= 0 || 2 * ctas > sms) return 1;                 // the grid already fills most of the device
  int64_t splits = sms / ctas;
  // every split should still run a few key tiles, so that the set-up and the combine pass stay small
  splits = splits < nt / 4 ? splits : nt / 4;
  splits = splits < 16 ? splits : 16;
  return (int)(splits < 1 ? 1 : splits);
}

extern "C" int64_t llnv_attention_workspace_bytes(int64_t Lq, int heads, int key_splits) {
  if (key_splits == LLNV_ATTN_SPLIT_TAIL) key_splits = 2;
  if (key_splits <= 1 || Lq <= 0 || heads <= 0) return 0;
  return (int64_t)key_splits * Lq * heads * (kD + 2) * (int64_t)sizeof(float);
}

namespace {

// The NVFP4 window of a call: cache blocks behind pointer tables.
struct CachedWindow {
  const void* const* k_codes;
  const void* const* k_sf;
  const float* const* k_amax;
  const void* const* v_codes;
  const void* const* v_sf;
  const float* const* v_amax;
  int num_blocks, block_tokens;
  float denom;                      // e2m1_max * e4m3_max
  int64_t tokens() const { return (int64_t)num_blocks * block_tokens; }
};

int64_t align256(int64_t n) { return (n + 255) / 256 * 256; }
// bf16 keys and values of the cached tokens, filled up to whole key tiles with rows of the current chunk
int64_t window_bytes(int64_t cached, int heads) { return 2 * align256((cached + kBK - 1) / kBK * kBK * heads * kD * 2); }

template <bool FUSED>
int launch_tiles(dim3 grid, cudaStream_t stream, const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmK2,
                 const CUtensorMap& tmV2, const CUtensorMap& tmO, const AttnParams& p, const KvTable<FUSED>& tab) {
  constexpr uint32_t smem = FUSED ? kSmemBytesFused : kSmemBytes;
  static bool attr_set[64] = {};
  int dev = 0;
  LLNV_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    LLNV_CUDA(cudaFuncSetAttribute(attention_kernel<FUSED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set[dev] = true;
  }
  launch_k(attention_kernel<FUSED>, grid, FUSED ? kThreadsFused : kThreads, smem, stream, tmQ, tmK, tmV, tmK2, tmV2, tmO, p, tab);
  return launch_status("attention_kernel");
}

// The launch that decodes win's cache blocks in its load stage.
int launch_fused(dim3 grid, cudaStream_t stream, const CUtensorMap& tmQ, const CUtensorMap& tmK2, const CUtensorMap& tmV2, const CUtensorMap& tmO,
                 AttnParams p, const CachedWindow& win, const void* k_cur, const void* v_cur, int64_t ldk, int64_t ldv) {
  LLNV_REQUIRE(p.Lk < INT_MAX - kBK, "llnv_attention_nvfp4kv: a window of %lld keys is too long", (long long)p.Lk);
  KvTable<true> tab;
  for (int b = 0; b < win.num_blocks; ++b) {
    tab.k_sf[b] = (const uint8_t*)win.k_sf[b];
    tab.k_amax[b] = win.k_amax[b];
    tab.v_sf[b] = (const uint8_t*)win.v_sf[b];
    tab.v_amax[b] = win.v_amax[b];
    // byte matrix [tokens, heads * 64], box 128 tokens x 64 bytes, 64-byte swizzle
    const uint64_t cols = (uint64_t)p.heads * 64;
    int rc = cached_tensor_map(&tab.k_codes[b], 0, win.k_codes[b], (uint64_t)win.block_tokens, cols, cols, 128, 64, 2);
    if (rc == LLNV_OK) rc = cached_tensor_map(&tab.v_codes[b], 0, win.v_codes[b], (uint64_t)win.block_tokens, cols, cols, 128, 64, 2);
    if (rc != LLNV_OK) return rc;
  }
  tab.n_cached = (int)win.tokens();
  tab.block_tokens = win.block_tokens;
  tab.inv_denom = (float)(1.0 / (double)win.denom);
  tab.k_cur = (const uint16_t*)k_cur;
  tab.v_cur = (const uint16_t*)v_cur;
  tab.ldk = ldk;
  tab.ldv = ldv;
  // what the last tile of the cached part holds of the current chunk is not loaded again
  p.first_tiles = (tab.n_cached + kBK - 1) / kBK;
  p.second_row = p.first_tiles * kBK - tab.n_cached;
  return launch_tiles<true>(grid, stream, tmQ, tmK2, tmV2, tmK2, tmV2, tmO, p, tab);
}

// Shared host side of the two entry points.  win == nullptr: k / v are the whole window (bf16).  Otherwise the window is win's
// cache blocks followed by the bf16 tensors k / v of Lk - win->tokens() keys.
int attention_launch(const void* q, int64_t Lq, int64_t ldq, const void* k, const void* v, int64_t Lk, int64_t ldk, int64_t ldv,
                     int heads, float scale, void* out, int64_t ldo, int key_splits, void* workspace, int64_t workspace_bytes,
                     float* out_amax, const CachedWindow* win, cudaStream_t stream, const char* who) {
  int tail_cut = 0;
  const int64_t split_bytes = llnv_attention_workspace_bytes(Lq, heads, key_splits);
  if (key_splits == LLNV_ATTN_SPLIT_TAIL) {
    const int sms = sm_count();
    if (sms > 0 && Lq > 0 && Lk > 0) tail_cut = tail_cut_for(((Lq + kBQ - 1) / kBQ) * heads, (Lk + kBK - 1) / kBK, sms);
    if (tail_cut > 0)
      LLNV_REQUIRE(workspace != nullptr && ((uintptr_t)workspace & 15) == 0 && workspace_bytes >= split_bytes,
                   "%s: tail balancing needs a 16-byte aligned workspace of llnv_attention_workspace_bytes() bytes", who);
    key_splits = 1;
  }
  LLNV_REQUIRE(key_splits >= 1 && key_splits <= 64, "%s: key_splits must be in 1..64 or LLNV_ATTN_SPLIT_TAIL (got %d)", who, key_splits);
  LLNV_REQUIRE(Lk <= 0 || key_splits <= (Lk + kBK - 1) / kBK, "%s: more key splits (%d) than key tiles of 128", who, key_splits);
  if (key_splits > 1) {
    LLNV_REQUIRE(workspace != nullptr && ((uintptr_t)workspace & 15) == 0 && workspace_bytes >= split_bytes,
                 "%s: key splits need a 16-byte aligned workspace of llnv_attention_workspace_bytes() bytes", who);
  }
  const int64_t n_cached = win ? win->tokens() : 0;
  const int64_t L_cur = Lk - n_cached;               // keys held in bf16
  LLNV_REQUIRE(q && out && (L_cur == 0 || (k && v)), "%s: null pointer", who);
  LLNV_REQUIRE(Lq >= 0 && Lk > 0 && L_cur >= 0 && heads > 0, "%s: need Lq >= 0, Lk > 0, heads > 0 (Lq=%lld Lk=%lld heads=%d)", who,
               (long long)Lq, (long long)Lk, heads);
  const int64_t C = (int64_t)heads * kD;
  LLNV_REQUIRE(ldq >= C && ldo >= C && ldq % 8 == 0 && ldo % 8 == 0 && (L_cur == 0 || (ldk >= C && ldv >= C && ldk % 8 == 0 && ldv % 8 == 0)),
               "%s: row strides must be >= heads*128 and multiples of 8", who);
  LLNV_REQUIRE(((uintptr_t)q & 15) == 0 && ((uintptr_t)k & 15) == 0 && ((uintptr_t)v & 15) == 0 && ((uintptr_t)out & 15) == 0,
               "%s: pointers must be 16-byte aligned", who);
  LLNV_REQUIRE(heads <= 65535, "%s: too many heads", who);
  if (out_amax && !amax_accumulate(1)) LLNV_CUDA(cudaMemsetAsync(out_amax, 0, sizeof(float), stream));
  if (Lq == 0) return LLNV_OK;

  AttnParams p = {};
  p.Lq = Lq;
  p.Lk = Lk;
  p.heads = heads;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = device_status_word();
  const int q_tiles = (int)((Lq + kBQ - 1) / kBQ);
  const int zdim = tail_cut > 0 ? 2 : key_splits;     // partial-result slices in the workspace
  p.nsplit = key_splits;
  p.tail_cut = tail_cut;
  p.tail_first = tail_cut > 0 ? (int)(((int64_t)q_tiles * heads / sm_count()) * sm_count()) : 0;
  p.part_o = zdim > 1 ? (float*)workspace : nullptr;
  p.part_ml = zdim > 1 ? (float*)workspace + (int64_t)zdim * Lq * heads * kD : nullptr;
  p.out_amax = key_splits > 1 ? nullptr : out_amax;   // with tail balancing the whole items report their own maximum
  p.first_tiles = INT_MAX;
  const dim3 grid((unsigned)q_tiles, (unsigned)heads, (unsigned)zdim);

  CUtensorMap tmQ, tmK, tmV, tmK2, tmV2, tmO;
  int rc = cached_tensor_map(&tmQ, 1, q, (uint64_t)Lq, (uint64_t)C, (uint64_t)ldq, 128, 64, 3);
  if (rc == LLNV_OK) rc = cached_tensor_map(&tmO, 1, out, (uint64_t)Lq, (uint64_t)C, (uint64_t)ldo, 32, 64, 3);
  if (rc == LLNV_OK && L_cur > 0) {
    rc = cached_tensor_map(&tmK2, 1, k, (uint64_t)L_cur, (uint64_t)C, (uint64_t)ldk, 128, 64, 3);
    if (rc == LLNV_OK) rc = cached_tensor_map(&tmV2, 1, v, (uint64_t)L_cur, (uint64_t)C, (uint64_t)ldv, 128, 64, 3);
  } else {
    tmK2 = tmV2 = tmQ;          // no key lives there: never used
  }
  if (rc != LLNV_OK) return rc;
  tmK = tmK2;
  tmV = tmV2;

  // the cached part as bf16: behind the partial results in the workspace
  const int64_t at = align256(zdim > 1 ? split_bytes : 0), bytes = window_bytes(n_cached, heads);
  if (n_cached > 0 && (!workspace || ((uintptr_t)workspace & 15) != 0 || workspace_bytes < at + bytes)) {
    rc = launch_fused(grid, stream, tmQ, tmK2, tmV2, tmO, p, *win, k, v, ldk, ldv);
  } else {
    if (n_cached > 0) {
      uint8_t* kw = (uint8_t*)workspace + at;
      uint8_t* vw = kw + bytes / 2;
      const int64_t first_tiles = (n_cached + kBK - 1) / kBK, rows = first_tiles * kBK;
      const int64_t pad = rows - n_cached < L_cur ? rows - n_cached : L_cur;
      rc = kv_window_dequant(win->k_codes, win->k_sf, win->k_amax, win->v_codes, win->v_sf, win->v_amax, win->num_blocks, heads,
                             win->block_tokens, win->denom, k, v, ldk, ldv, (int)pad, kw, vw, stream);
      if (rc == LLNV_OK) rc = cached_tensor_map(&tmK, 1, kw, (uint64_t)(n_cached + pad), (uint64_t)C, (uint64_t)C, 128, 64, 3);
      if (rc == LLNV_OK) rc = cached_tensor_map(&tmV, 1, vw, (uint64_t)(n_cached + pad), (uint64_t)C, (uint64_t)C, 128, 64, 3);
      p.first_tiles = (int)first_tiles;
      p.second_row = (int)pad;
    }
    if (rc == LLNV_OK) rc = launch_tiles<false>(grid, stream, tmQ, tmK, tmV, tmK2, tmV2, tmO, p, {});
  }
  if (rc == LLNV_OK && zdim > 1) {
    const int first_item = tail_cut > 0 ? p.tail_first : 0;
    const int64_t blocks = ((int64_t)q_tiles * heads - first_item) * (kBQ / 8);
    launch_k(attention_combine_kernel, (unsigned)blocks, 256, 0, stream, p.part_o, p.part_ml, zdim, Lq, heads, p.scale_log2, (uint16_t*)out, ldo,
             out_amax, first_item, q_tiles);
    rc = launch_status("attention_combine_kernel");
  }
  return rc;
}

}  // namespace

extern "C" int llnv_attention_bf16_ex(const void* q, int64_t Lq, int64_t ldq, const void* k, const void* v, int64_t Lk,
                                      int64_t ldk, int64_t ldv, int heads, float scale, void* out, int64_t ldo,
                                      int key_splits, void* workspace, int64_t workspace_bytes, float* out_amax,
                                      llnv_stream_t stream) {
  LLNV_REQUIRE(k && v, "llnv_attention_bf16: null pointer");
  return attention_launch(q, Lq, ldq, k, v, Lk, ldk, ldv, heads, scale, out, ldo, key_splits, workspace, workspace_bytes, out_amax,
                          nullptr, (cudaStream_t)stream, "llnv_attention_bf16");
}

extern "C" int64_t llnv_attention_nvfp4kv_workspace_bytes(int64_t Lq, int heads, int key_splits, int num_blocks, int block_token_size) {
  const int64_t split = llnv_attention_workspace_bytes(Lq, heads, key_splits);
  if (num_blocks <= 0 || block_token_size <= 0 || heads <= 0) return split;
  return align256(split) + window_bytes((int64_t)num_blocks * block_token_size, heads);
}

extern "C" int llnv_attention_nvfp4kv(const void* q, int64_t Lq, int64_t ldq, const void* const* k_codes, const void* const* k_sf,
                                      const float* const* k_amax, const void* const* v_codes, const void* const* v_sf,
                                      const float* const* v_amax, int num_blocks, int block_token_size, float e2m1_max,
                                      float e4m3_max, const void* k_cur, const void* v_cur, int64_t L_cur, int64_t ldk, int64_t ldv,
                                      int heads, float scale, void* out, int64_t ldo, int key_splits, void* workspace,
                                      int64_t workspace_bytes, float* out_amax, llnv_stream_t stream) {
  const char* who = "llnv_attention_nvfp4kv";
  LLNV_REQUIRE(num_blocks >= 0 && num_blocks <= kMaxKvBlocks, "%s: 0 to %d cache blocks (got %d)", who, kMaxKvBlocks, num_blocks);
  LLNV_REQUIRE(L_cur >= 0 && (num_blocks > 0 || L_cur > 0), "%s: the window is empty", who);
  if (num_blocks == 0)
    return attention_launch(q, Lq, ldq, k_cur, v_cur, L_cur, ldk, ldv, heads, scale, out, ldo, key_splits, workspace, workspace_bytes,
                            out_amax, nullptr, (cudaStream_t)stream, who);
  LLNV_REQUIRE(k_codes && k_sf && k_amax && v_codes && v_sf && v_amax, "%s: null pointer table", who);
  LLNV_REQUIRE(block_token_size >= 128 && heads > 0, "%s: block_token_size must be at least 128 (got %d) and heads positive", who,
               block_token_size);
  LLNV_REQUIRE(e2m1_max > 0 && e4m3_max > 0, "%s: e2m1_max and e4m3_max must be positive", who);
  for (int b = 0; b < num_blocks; ++b) {
    LLNV_REQUIRE(k_codes[b] && k_sf[b] && k_amax[b] && v_codes[b] && v_sf[b] && v_amax[b], "%s: null pointer in block %d", who, b);
    LLNV_REQUIRE(((uintptr_t)k_codes[b] & 15) == 0 && ((uintptr_t)v_codes[b] & 15) == 0 && ((uintptr_t)k_sf[b] & 3) == 0 &&
                     ((uintptr_t)v_sf[b] & 3) == 0,
                 "%s: codes of block %d must be 16-byte, scales 4-byte aligned", who, b);
  }
  const CachedWindow win = {k_codes, k_sf, k_amax, v_codes, v_sf, v_amax, num_blocks, block_token_size, e2m1_max * e4m3_max};
  return attention_launch(q, Lq, ldq, k_cur, v_cur, win.tokens() + L_cur, ldk, ldv, heads, scale, out, ldo, key_splits, workspace,
                          workspace_bytes, out_amax, &win, (cudaStream_t)stream, who);
}

extern "C" int llnv_attention_bf16(const void* q, int64_t Lq, int64_t ldq, const void* k, const void* v, int64_t Lk,
                                   int64_t ldk, int64_t ldv, int heads, float scale, void* out, int64_t ldo,
                                   llnv_stream_t stream) {
  return llnv_attention_bf16_ex(q, Lq, ldq, k, v, Lk, ldk, ldv, heads, scale, out, ldo, 1, nullptr, 0, nullptr, stream);
}
