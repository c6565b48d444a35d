// Fused PDQ hash kernel: 512x512 image -> tent compress -> DCT -> quality -> exact median
// quantize -> the 8 dihedral hashes, for a batch of images, one image per CTA at a time.
//
// Reference semantics (yume-pdq):
//   compress  DefaultKernel::jarosz_compress   src/kernel/mod.rs:644-666
//   DCT       DefaultKernel::dct2d_impl        src/kernel/mod.rs:543-574
//   quality   sum_of_gradients / adjust_quality src/kernel/mod.rs:611-642
//   median    torben_median                    src/kernel/mod.rs:212-253 (the 128th smallest)
//   packing   quantize / threshold_2d_f32      src/kernel/mod.rs:595-608, threshold.rs:37-119
//   dihedrals visit_dihedrals                  src/lib.rs:358-420
//
// The FP32 path reproduces the reference's f32 results bit for bit for finite inputs.
// Every product and sum is a separately rounded __fmul_rn / __fadd_rn (the reference is
// Rust, which never contracts a*b+c). Sums run in the reference's order: taps row by row;
// the DCT in four interleaved partial sums combined as ((s0+s1)+s2)+s3. The tent table is
// 7x7, but only 27 taps are nonzero: the 5x5 centre (k/81) and two subnormal residues in
// row 0 that the reference's 128-bit constant generation leaves behind. A zero tap adds +0
// to a finite partial sum, which changes nothing, so the kernel skips those taps.
//
// CTA layout (192 threads):
//   warps 0-3  compute: thread j owns output column j (j < 127) of the compressed image,
//              accumulates DCT stage 1 (16 x 127 x 127) as each compressed row appears,
//              then computes the 16 x 16 stage 2 together.
//   warp 4     producer: one lane streams the image into a shared-memory ring with 1-D
//              bulk async copies (8 or 16 input rows = one stage), a few stages deep.
//   warp 5     epilogue: quality, exact medians, bits and dihedrals of image k while the
//              compute warps already work on image k+1 (double-buffered PDQF).
//
// f32 input is bound by HBM (1,024 images 164 us, 6.6 TB/s). The others are bound by issue
// slots and latency (two compute warps per scheduler at 152 registers), so what counts is
// instructions per compressed value, ~115, and how long its serial sum of 27 terms takes:
//   * a 4-row group finishes one value and starts the next from one carried sum, so nothing
//     is read or converted twice and a stage of 2-4 groups costs one wait and one release;
//   * byte input: two groups' sums go side by side in packed pairs (an f32x2 instruction takes
//     two cycles of the FMA pipe but one issue slot): two values per 27 dependent adds (one
//     value each: 346 us below, RGB8 148). f32 rows come as 16-byte loads whose pairs would
//     have to be moved together, so f32 keeps the scalar sums;
//   * byte conversion and product are one fma, and the DCT's accumulators are pairs as well;
//   * RGB pixels become luma where they are read, without a staging of their own;
//   * the epilogue, which shares the issue slots, selects three key bits per round and stops
//     at a bin of one key, two slots side by side (one bit per round over all 32 for four
//     slots: 375 us before the pairs; one slot after another: 1.3 us more for a single wave).
// 4,096 u8 images: 552 -> 324 us (12.6 M images/s); 801 RGB8 images 262 -> 136 us; u8 with
// the separable compress and the BF16x3 DCT, 1,024 images: 133 -> 72 us. No gain, measured: a
// third CTA per SM (127 registers, copies and epilogue in one warp: 320 us against 324, but
// single waves 4 us longer and 801 RGB8 images 148 against 136), compress and DCT in warps of
// their own (388 against 375 us, none at f32), a pair's DCT steps put beside the next pair's
// sums (the same times).
#include <cuda_bf16.h>

#include <cstring>

#include <type_traits>

#include "ypdq_internal.cuh"
#include "ypdq_tables.h"

namespace ypdq {

__device__ float g_dct[16 * 127];  // D[k][i] = sqrt(2/127) cos(pi (k+1) (2i+1) / 254), f32
__device__ alignas(16) float g_dct_t[128 * 16];  // the same as D^T: [i][k]; row 127 is zero

constexpr int kGroupsPerImage = 128;  // group g holds rows 4g+1 .. 4g+4 (group 127: 509, 510)
constexpr int kComputeThreads = 128;
constexpr int kProducerWarp = 4;
constexpr int kEpilogueWarp = 5;
constexpr int kMmaWarpHash = 6;   // tensor-core DCT only: allocates TMEM, issues the MMAs
template <int kDct>
constexpr int hash_threads() { return kDct == 0 ? 192 : 224; }
// RGB8 / RGBA8 pixels, converted to f32 luma where they are read (see load_row).
struct rgb8_t {
  uint8_t c[3];
};
struct rgba8_t {
  uint8_t c[4];
};
template <typename Tin>
constexpr bool is_rgb() {
  return std::is_same<Tin, rgb8_t>::value || std::is_same<Tin, rgba8_t>::value;
}

// A stage of the input ring is one bulk copy of kGroups groups of 4 rows: the compute warps
// wait once for it and free it once, so a wider stage spreads that over more rows, as far as
// a few stages in flight still fit beside each other. In bytes per CTA: u8 4 x 8 KB, RGB8
// 6 (tensor-core DCT: 3) x 12 KB, f32 and RGBA8 5 (3) x 16 KB.
template <typename Tin>
constexpr int stage_groups() { return sizeof(Tin) == 1 ? 4 : 2; }
template <typename Tin, int kDct>
constexpr int ring_stages() {
  return sizeof(Tin) == 1 ? 4 : kDct != 0 ? 3 : sizeof(Tin) == 3 ? 6 : 5;
}
constexpr int kComputeBarrier = 1;  // named barrier id used by the 128 compute threads

// Stage 1 of the DCT on tensor cores (kDct = 1: TF32, 2: BF16x3). The compressed values
// are written, chunk by chunk of compressed rows, into a 128-byte-swizzled K-major operand
// A[j][i] (M = 128 columns j, K = rows i); B is the DCT matrix D[k][i] (N = 16).
template <int kDct>
struct DctTraits {
  static constexpr int kRowsPerChunk = 128;  // unused for kDct = 0
  static constexpr int kBufBytes = 16;
  static constexpr int kDBytes = 16;
};
template <>
struct DctTraits<1> {  // TF32: 32 rows x 4 B = 128 B per column per chunk
  static constexpr int kRowsPerChunk = 32;
  static constexpr int kBufBytes = 128 * 128;
  static constexpr int kDBytes = 4 * 2048;  // 4 K-chunks x 16 rows x 128 B
  static constexpr int kDChunkBytes = 2048;
  static constexpr int kKSteps = 4;         // MMAs of K = 8 (32 B) per chunk
};
template <>
struct DctTraits<2> {  // BF16x3: 32 rows x 2 B (64-byte swizzle), hi at +0 and lo at +8192
  static constexpr int kRowsPerChunk = 32;
  static constexpr int kBufBytes = 2 * 128 * 64;
  static constexpr int kDBytes = 2 * 4 * 1024;  // hi, lo x 4 K-chunks x 16 rows x 64 B
  static constexpr int kDChunkBytes = 1024;
  static constexpr int kKSteps = 2;             // MMAs of K = 16 (32 B) per chunk
  static constexpr int kALo = 8192, kDLo = 4096;  // byte offsets of the lo operands
};

template <int kStageBytes, int kNumStages, int kDct>
struct HashSmem {
  alignas(1024) uint8_t ops[2][DctTraits<kDct>::kBufBytes];  // A operand, double-buffered
  alignas(1024) uint8_t dops[DctTraits<kDct>::kDBytes];      // B operand (DCT matrix)
  alignas(128) unsigned char ring[kNumStages][kStageBytes];
  alignas(16) float dt[128][16];  // dt[i + 1][k] = D[k][i]; row 0 is zero
  float t[16][129];               // DCT stage 1 result T = D * B
  float p[2][16][17];             // PDQF, double-buffered between compute and epilogue
  uint64_t full[kNumStages];
  uint64_t empty[kNumStages];
  uint64_t pfull[2];
  uint64_t pempty[2];
  uint64_t a_full[2], a_empty[2], acc_full[2], acc_empty[2], tc_exit, mma_done;
  uint32_t tmem_base;
  int abort_flag;
};

template <typename Tin>
struct InputTraits;
template <>
struct InputTraits<float> {
  static constexpr int kRowBytes = 512 * 4;
};
template <>
struct InputTraits<uint8_t> {
  static constexpr int kRowBytes = 512;
};
template <>
struct InputTraits<rgb8_t> {
  static constexpr int kRowBytes = 512 * 3;
};
template <>
struct InputTraits<rgba8_t> {
  static constexpr int kRowBytes = 512 * 4;
};
// The five columns 4j + 2 .. 4j + 6 of one input row in shared memory that compressed column
// j reads: two pairs and one. f32 input and luma as they are, u8 biased (byte_biased).
struct RowX {
  float2 a, b;
  float c;
};
__device__ __forceinline__ RowX load_row(const float* row, int j) {
  const float4* r = reinterpret_cast<const float4*>(row);
  const float4 a = r[j], b = r[j + 1];
  return {make_float2(a.z, a.w), make_float2(b.x, b.y), b.z};
}
__device__ __forceinline__ RowX load_row(const uint8_t* row, int j) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(row);
  const uint32_t a = r[j], b = r[j + 1];
  return {make_float2(byte_biased<2>(a), byte_biased<3>(a)),
          make_float2(byte_biased<0>(b), byte_biased<1>(b)), byte_biased<2>(b)};
}
// RGB columns as f32 luma, converted on load (9 of 8 columns' work: each column is read by
// 1.25 threads). Converting whole stages into a luma staging first cost more: its stores,
// its loads and a barrier per row.
__device__ __forceinline__ RowX load_row(const rgb8_t* row, int j) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(row) + 3 * j;
  return {luma23(r[0], r[1], r[2]), luma01(r[3], r[4], r[5]), luma23(r[3], r[4], r[5]).x};
}
__device__ __forceinline__ RowX load_row(const rgba8_t* row, int j) {
  const uint4* r = reinterpret_cast<const uint4*>(row);
  const uint4 a = r[j], b = r[j + 1];
  return {luma_rgba(a.z, a.w), luma_rgba(b.x, b.y), luma_rgba(b.z, b.z).x};
}

#define YPDQ_W(di, dj) __uint_as_float(YPDQ_TENT_BITS_##di##_##dj)
// The weights of a tap row are (w1, w2, w3, w2, w1), and rows 1, 2 equal rows 5, 4.
static_assert(YPDQ_TENT_BITS_1_1 == YPDQ_TENT_BITS_1_5 && YPDQ_TENT_BITS_1_2 == YPDQ_TENT_BITS_1_4 &&
              YPDQ_TENT_BITS_2_1 == YPDQ_TENT_BITS_2_5 && YPDQ_TENT_BITS_2_2 == YPDQ_TENT_BITS_2_4 &&
              YPDQ_TENT_BITS_3_1 == YPDQ_TENT_BITS_3_5 && YPDQ_TENT_BITS_3_2 == YPDQ_TENT_BITS_3_4 &&
              YPDQ_TENT_BITS_1_1 == YPDQ_TENT_BITS_5_1 && YPDQ_TENT_BITS_1_2 == YPDQ_TENT_BITS_5_2 &&
              YPDQ_TENT_BITS_1_3 == YPDQ_TENT_BITS_5_3 && YPDQ_TENT_BITS_5_1 == YPDQ_TENT_BITS_5_5 &&
              YPDQ_TENT_BITS_5_2 == YPDQ_TENT_BITS_5_4 && YPDQ_TENT_BITS_2_1 == YPDQ_TENT_BITS_4_1 &&
              YPDQ_TENT_BITS_2_2 == YPDQ_TENT_BITS_4_2 && YPDQ_TENT_BITS_2_3 == YPDQ_TENT_BITS_4_3 &&
              YPDQ_TENT_BITS_4_1 == YPDQ_TENT_BITS_4_5 && YPDQ_TENT_BITS_4_2 == YPDQ_TENT_BITS_4_4,
              "the tent table is symmetric");

// RN(w x) of one value and of a whole tap row. The sums that take the products are scalar
// adds (a packed multiply is only contracted with a packed add).
template <typename T>
__device__ __forceinline__ float weighted(float w, float x) {
  if constexpr (sizeof(T) == 1) return __fmaf_rn(w, x, -kByteBias * w);
  else return __fmul_rn(w, x);
}
template <typename T>
__device__ __forceinline__ float2 weighted2(float w0, float w1, float2 x) {
  const float2 w = make_float2(w0, w1);
  if constexpr (sizeof(T) == 1) return fma2_rn(w, x, make_float2(-kByteBias * w0, -kByteBias * w1));
  else return mul2_contractible_rn(w, x);
}
template <typename T>
__device__ __forceinline__ RowX weighted_row(float w1, float w2, float w3, const RowX& x) {
  return {weighted2<T>(w1, w2, x.a), weighted2<T>(w3, w2, x.b), weighted<T>(w1, x.c)};
}
__device__ __forceinline__ float add_row(float s, const RowX& p) {
  return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, p.a.x), p.a.y), p.b.x), p.b.y), p.c);
}

// The compress walks a column group by group. Compressed value i takes rows 4i + 1 .. 4i + 6
// in the reference's tap order; row 4i + 1 holds only the two residue taps (columns 4j + 5
// and 4j + 6). Group g's rows 4g + 1 and 4g + 2 are the last two of value g - 1 and the first
// two of value g, and its rows 4g + 3 and 4g + 4 the next two of value g. So one group
// finishes value g - 1 from the sum carried over and starts value g, with nothing but that
// sum between groups; the products of row 4g + 2 serve both values (tap rows 1 and 5 have
// equal weights).
struct TapSum {
  float s = 0.0f;  // value g through tap row 3
};
template <typename Tin>
__device__ __forceinline__ float compress_group(const Tin* rows, int j, bool last, TapSum& c) {
  using T = typename std::conditional<is_rgb<Tin>(), float, Tin>::type;
  const RowX x = load_row(rows, j);
  const RowX p = weighted_row<T>(YPDQ_W(1, 1), YPDQ_W(1, 2), YPDQ_W(1, 3), load_row(rows + 512, j));
  const RowX p4 = weighted_row<T>(YPDQ_W(4, 1), YPDQ_W(4, 2), YPDQ_W(4, 3), x);
  const float done = add_row(add_row(c.s, p4), p);
  if (!last) {
    float s = __fadd_rn(__fadd_rn(0.0f, weighted<T>(YPDQ_W(0, 4), x.b.y)),
                        weighted<T>(YPDQ_W(0, 5), x.c));
    s = add_row(s, p);
    s = add_row(s, weighted_row<T>(YPDQ_W(2, 1), YPDQ_W(2, 2), YPDQ_W(2, 3),
                                   load_row(rows + 2 * 512, j)));
    c.s = add_row(s, weighted_row<T>(YPDQ_W(3, 1), YPDQ_W(3, 2), YPDQ_W(3, 3),
                                     load_row(rows + 3 * 512, j)));
  }
  return done;
}

// The same five columns of two rows, paired row by row.
struct RowX2 {
  float2 v[5];
};
__device__ __forceinline__ RowX2 load_rows(const uint8_t* p, const uint8_t* q, int j) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(p);
  const uint32_t* s = reinterpret_cast<const uint32_t*>(q);
  const uint32_t a = r[j], b = r[j + 1], c = s[j], d = s[j + 1];
  return {make_float2(byte_biased<2>(a), byte_biased<2>(c)),
          make_float2(byte_biased<3>(a), byte_biased<3>(c)),
          make_float2(byte_biased<0>(b), byte_biased<0>(d)),
          make_float2(byte_biased<1>(b), byte_biased<1>(d)),
          make_float2(byte_biased<2>(b), byte_biased<2>(d))};
}
template <int kR, int kG, int kB>  // bytes of the two words' channels
__device__ __forceinline__ float2 luma_rows(uint32_t r, uint32_t g, uint32_t b, uint32_t r1,
                                            uint32_t g1, uint32_t b1) {
  return luma2_bt601(make_float2(byte_biased<kR>(r), byte_biased<kR>(r1)),
                     make_float2(byte_biased<kG>(g), byte_biased<kG>(g1)),
                     make_float2(byte_biased<kB>(b), byte_biased<kB>(b1)));
}
__device__ __forceinline__ RowX2 load_rows(const rgb8_t* p, const rgb8_t* q, int j) {
  // pixels 0-3 in three words: r g b r | g b r g | b r g b
  const uint32_t* r = reinterpret_cast<const uint32_t*>(p) + 3 * j;
  const uint32_t* s = reinterpret_cast<const uint32_t*>(q) + 3 * j;
  return {luma_rows<2, 3, 0>(r[1], r[1], r[2], s[1], s[1], s[2]),
          luma_rows<1, 2, 3>(r[2], r[2], r[2], s[2], s[2], s[2]),
          luma_rows<0, 1, 2>(r[3], r[3], r[3], s[3], s[3], s[3]),
          luma_rows<3, 0, 1>(r[3], r[4], r[4], s[3], s[4], s[4]),
          luma_rows<2, 3, 0>(r[4], r[4], r[5], s[4], s[4], s[5])};
}
__device__ __forceinline__ RowX2 load_rows(const rgba8_t* p, const rgba8_t* q, int j) {
  const uint4* r = reinterpret_cast<const uint4*>(p);
  const uint4* s = reinterpret_cast<const uint4*>(q);
  const uint4 a = r[j], b = r[j + 1], c = s[j], d = s[j + 1];
  return {luma_rgba(a.z, c.z), luma_rgba(a.w, c.w), luma_rgba(b.x, d.x), luma_rgba(b.y, d.y),
          luma_rgba(b.z, d.z)};
}
// RN(w x) of both rows. Packed adds take these products, so the multiply must be one that is
// not contracted.
template <typename T>
__device__ __forceinline__ float2 weighted_both(float w, float2 x, float nz) {
  if constexpr (sizeof(T) == 1)
    return fma2_rn(make_float2(w, w), x, make_float2(-kByteBias * w, -kByteBias * w));
  else
    return mul2_rn(make_float2(w, w), x, nz);
}
template <typename T>
__device__ __forceinline__ RowX2 weighted_rows(float w1, float w2, float w3, const RowX2& x,
                                               float nz) {
  return {weighted_both<T>(w1, x.v[0], nz), weighted_both<T>(w2, x.v[1], nz),
          weighted_both<T>(w3, x.v[2], nz), weighted_both<T>(w2, x.v[3], nz),
          weighted_both<T>(w1, x.v[4], nz)};
}
__device__ __forceinline__ float2 add_rows(float2 s, const RowX2& p) {
#pragma unroll
  for (int k = 0; k < 5; ++k) s = add2_rn(s, p.v[k]);
  return s;
}

// Groups g and g + 1 (8 rows): finishes values g - 1 and g and starts value g + 1. The two
// groups' sums go side by side in packed pairs (half the issue slots of the serial sums, and
// twice the work between two steps of one); the finishing pair continues the sum carried in
// and the one just started by group g. The last pair starts a value that does not exist from
// whatever its two missing rows' place holds; nothing reads it.
template <typename Tin>
__device__ __forceinline__ float2 compress_pair(const Tin* rows, int j, bool last, float nz,
                                                TapSum& c) {
  if constexpr (std::is_same<Tin, float>::value) {
    const float a = compress_group(rows, j, false, c);
    return make_float2(a, compress_group(rows + 4 * 512, j, last, c));
  } else {
    using T = typename std::conditional<is_rgb<Tin>(), float, Tin>::type;
    const Tin* second = rows + 4 * 512;
    const RowX2 x = load_rows(rows, second, j);
    const RowX2 p = weighted_rows<T>(YPDQ_W(1, 1), YPDQ_W(1, 2), YPDQ_W(1, 3),
                                     load_rows(rows + 512, second + 512, j), nz);
    float2 s = add2_rn(add2_rn(make_float2(0.0f, 0.0f), weighted_both<T>(YPDQ_W(0, 4), x.v[3], nz)),
                       weighted_both<T>(YPDQ_W(0, 5), x.v[4], nz));
    s = add_rows(s, p);
    s = add_rows(s, weighted_rows<T>(YPDQ_W(2, 1), YPDQ_W(2, 2), YPDQ_W(2, 3),
                                     load_rows(rows + 2 * 512, second + 2 * 512, j), nz));
    s = add_rows(s, weighted_rows<T>(YPDQ_W(3, 1), YPDQ_W(3, 2), YPDQ_W(3, 3),
                                     load_rows(rows + 3 * 512, second + 3 * 512, j), nz));
    const RowX2 p4 = weighted_rows<T>(YPDQ_W(4, 1), YPDQ_W(4, 2), YPDQ_W(4, 3), x, nz);
    const float2 done = add_rows(add_rows(make_float2(c.s, s.x), p4), p);
    c.s = s.y;
    return done;
  }
}

// Separable compress (YPDQ_COMPRESS_SEPARABLE; not the reference's operation order). The
// tent weights are W[di][dj] = c[di] c[dj] / 81 with c = (0, 1, 2, 3, 2, 1, 0) (the 128-bit
// table also holds two subnormal residue taps, ~1e-40, which this form drops). So
//   out[i][j] = S / 81,  S = sum_{r = 2..6} c[r] h(4i + r),  h(row) = sum_{k = 2..6} c[k] x[row][4j + k]
// Each h row serves two output rows. For u8 input h and S are exact integers (two dp4a per
// h), so the only rounding is the final scale.
template <typename Tin>
__device__ __forceinline__ float hsum(const Tin* row, int j) {
  if constexpr (std::is_same<Tin, uint8_t>::value) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(row);
    // bytes of r[j]: columns 4j .. 4j+3 (weights 0, 0, 1, 2); r[j+1]: 4j+4 .. 4j+7 (3, 2, 1, 0)
    return static_cast<float>(__dp4a(r[j], 0x02010000u, __dp4a(r[j + 1], 0x00010203u, 0u)));
  } else {
    const RowX x = load_row(row, j);
    return (x.a.x + x.c) + 2.0f * (x.a.y + x.b.y) + 3.0f * x.b.x;
  }
}
// h of rows 4g + 2 .. 4g + 4, carried to the group that finishes value g.
struct HCarry {
  float h1 = 0.0f, h2 = 0.0f, h3 = 0.0f;
};
template <typename Tin>
__device__ __forceinline__ float compress_group(const Tin* rows, int j, bool last, HCarry& c) {
  const float n0 = hsum(rows, j), n1 = hsum(rows + 512, j);
  const float S = (c.h1 + n1) + 2.0f * (c.h2 + n0) + 3.0f * c.h3;
  if (!last) {
    c.h1 = n1;
    c.h2 = hsum(rows + 2 * 512, j);
    c.h3 = hsum(rows + 3 * 512, j);
  }
  return S * (1.0f / 81.0f);
}
template <typename Tin>
__device__ __forceinline__ float2 compress_pair(const Tin* rows, int j, bool last, float,
                                                HCarry& c) {
  const float a = compress_group(rows, j, false, c);
  return make_float2(a, compress_group(rows + 4 * 512, j, last, c));
}

// ---------------------------------------------------------------- epilogue

__device__ __forceinline__ uint32_t f32_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_f32(uint32_t k) {
  uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

// The rank-127 values of kSets sets of 256 held 8 per lane: MSB-first radix selection on
// order-preserving keys, three bits at a time: each lane counts its keys per digit in eight
// 4-bit counters (at most 8 each), which are widened to 16 bits and summed over the warp by
// four independent reductions. Once the digit's bin holds one key, that key is the answer
// (after 4 or 5 of the 11 rounds on images); the loop ends when every set has its answer.
template <int kSets>
__device__ __forceinline__ void select_rank127(const float (&v)[kSets][8], float (&out)[kSets]) {
  uint32_t key[kSets][8], prefix[kSets];
  int rank[kSets], width[kSets];  // the rank within the digit's bin, the keys in it
#pragma unroll
  for (int s = 0; s < kSets; ++s) {
#pragma unroll
    for (int e = 0; e < 8; ++e) key[s][e] = f32_key(v[s][e]);
    prefix[s] = 0u;
    rank[s] = 127;
  }
  int shift = 29;
#pragma unroll 1
  for (;;) {
    uint32_t two[kSets][4];  // digits i and i + 4 in 16-bit halves
#pragma unroll
    for (int s = 0; s < kSets; ++s) {
      uint32_t counts = 0u;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t k = (key[s][e] ^ prefix[s]) >> shift;  // above 7: another prefix
        counts += k < 8u ? 1u << (4 * k) : 0u;
      }
      // (in the last round, shift 0 with two bits left, digits 4-7 are keys of another prefix;
      // the rank lies below them)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        two[s][i] = __reduce_add_sync(0xffffffffu, (counts >> (4 * i)) & 0x000F000Fu);
    }
    bool single = true;
#pragma unroll
    for (int s = 0; s < kSets; ++s) {
      int below = 0, upto = 256, digit = 0, cum = 0;  // keys below and up to the rank's digit
#pragma unroll
      for (int d = 0; d < 8; ++d) {
        cum += static_cast<int>((d & 4) ? two[s][d & 3] >> 16 : two[s][d & 3] & 0xFFFFu);
        if (cum <= rank[s]) {
          below = cum;
          digit = d + 1;
        } else {
          upto = min(upto, cum);
        }
      }
      prefix[s] |= static_cast<uint32_t>(digit) << shift;
      width[s] = upto - below;
      rank[s] -= below;
      single = single && width[s] == 1;
    }
    if (shift == 0) break;
    if (single) {
#pragma unroll
      for (int s = 0; s < kSets; ++s) {
        uint32_t found = 0u;
#pragma unroll
        for (int e = 0; e < 8; ++e)
          found |= ((key[s][e] ^ prefix[s]) >> shift) == 0u ? key[s][e] : 0u;
        prefix[s] = __reduce_or_sync(0xffffffffu, found);
      }
      break;
    }
    shift = shift > 3 ? shift - 3 : 0;
  }
#pragma unroll
  for (int s = 0; s < kSets; ++s) out[s] = key_f32(prefix[s]);
}

// Slot s of the 8 outputs: value at (r, c) is sign * (s < 4 ? P[r][c] : P[c][r]).
// Row signs (row_mask) apply in slots 2, 3, 5, 6; column signs (col_mask) in 1, 2, 6, 7.
__device__ __forceinline__ bool slot_rows(int s) { return s == 2 || s == 3 || s == 5 || s == 6; }
__device__ __forceinline__ bool slot_cols(int s) { return s == 1 || s == 2 || s == 6 || s == 7; }

// Slot s as signs and strides over P (pitch 17): value (r, c) is P[r row + c col] with its sign bit
// flipped where bit r of `rows` and bit c of `cols` differ (see slot_rows).
struct SlotView {
  const float* P;
  int row, col;
  uint32_t rows, cols;
  __device__ __forceinline__ SlotView(const float* P_, int s, uint32_t rm, uint32_t cm)
      : P(P_), row(s < 4 ? 17 : 1), col(s < 4 ? 1 : 17), rows(slot_rows(s) ? rm : 0u),
        cols(slot_cols(s) ? cm : 0u) {}
  __device__ __forceinline__ float at(int r, int c) const {
    return __uint_as_float(__float_as_uint(P[r * row + c * col]) ^
                           (((rows >> r) ^ (cols >> c)) << 31));
  }
};

// Sum of gradients of slot s, summed sequentially in the reference order.
__device__ float slot_gradient(const SlotView& m) {
  float g = 0.0f;
  float prev[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) prev[c] = m.at(0, c);
#pragma unroll 1
  for (int r = 0; r < 15; ++r) {
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const float next = m.at(r + 1, c);
      g = __fadd_rn(g, fabsf(__fsub_rn(prev[c], next)));
      prev[c] = next;
    }
  }
#pragma unroll 1
  for (int r = 0; r < 16; ++r) {
#pragma unroll
    for (int c = 0; c < 16; ++c) prev[c] = m.at(r, c);
#pragma unroll
    for (int c = 0; c < 15; ++c) g = __fadd_rn(g, fabsf(__fsub_rn(prev[c], prev[c + 1])));
  }
  return g;
}

struct EpilogueOut {
  uint8_t* hashes;   // [8][32]
  float* quality;    // [8]
  float* thresholds; // [8]
  float* pdqf;       // [pdqf_slots][256]
  int pdqf_slots;
};

// Medians, bits and outputs of slots s .. s + kSets - 1 and the four after each (s < 4; slot
// s + 4 is slot s's transpose with the other axis' signs, at slot s's threshold) by one warp.
// With thr_given the threshold of slot s is the caller's.
template <int kSets>
__device__ __forceinline__ void slot_pairs(const float* P, int s, uint32_t rm, uint32_t cm,
                                           int lane, const EpilogueOut& o, bool thr_given,
                                           float thr_in) {
  const int i = lane >> 1, j0 = (lane & 1) << 3;
  float v[kSets][8], thr[kSets];
#pragma unroll
  for (int x = 0; x < kSets; ++x) {
    const SlotView m(P, s + x, rm, cm);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[x][e] = m.at(i, j0 + e);
  }
  select_rank127(v, thr);
  if (thr_given) thr[0] = thr_in;
#pragma unroll
  for (int h = 0; h < 2 * kSets; ++h) {
    const int x = h % kSets, slot = s + x + 4 * (h / kSets);
    if (h >= kSets) {
      const SlotView m(P, slot, rm, cm);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[x][e] = m.at(i, j0 + e);
    }
    uint32_t byte = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) byte |= (v[x][e] > thr[x] ? 1u : 0u) << e;
    if (o.hashes) o.hashes[slot * 32 + 31 - lane] = static_cast<uint8_t>(byte);
    if (o.pdqf && (slot == 0 || o.pdqf_slots == 8)) {
      float4* dst = reinterpret_cast<float4*>(o.pdqf + slot * 256 + lane * 8);
      dst[0] = make_float4(v[x][0], v[x][1], v[x][2], v[x][3]);
      dst[1] = make_float4(v[x][4], v[x][5], v[x][6], v[x][7]);
    }
    if (o.thresholds && lane == 0) o.thresholds[slot] = thr[x];
  }
}

// One warp turns a PDQF held in shared memory (16 rows at a pitch of 17) into the 8 slot hashes,
// thresholds and qualities. With thr0_given the slot-0 threshold is taken from the caller.
__device__ __forceinline__ void epilogue_warp(const float* P, bool thr0_given, float thr0_in,
                                              uint32_t rm, uint32_t cm, int lane,
                                              const EpilogueOut& o) {
#pragma unroll 1
  for (int s = 0; s < 4; s += 2)
    slot_pairs<2>(P, s, rm, cm, lane, o, s == 0 && thr0_given, thr0_in);
  if (o.quality && lane < 8)
    o.quality[lane] = fminf(__fdiv_rn(slot_gradient(SlotView(P, lane, rm, cm)), 180.0f), 1.0f);
}

// ------------------------------------------------------------------- kernel

// tcgen05 MMAs for the tensor-core DCT (M = 128, N = 16, f32 accumulate in TMEM).
__device__ __forceinline__ void mma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// D f32, A/B tf32 (format 2) or bf16 (format 1), K-major, M = 128, N = 16.
constexpr uint32_t kIdescTf32 = (1u << 4) | (2u << 7) | (2u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kIdescBf16 = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void split_bf16(float x, uint16_t& hi, uint16_t& lo) {
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
  hi = __bfloat16_as_ushort(h);
  lo = __bfloat16_as_ushort(l);
}
// split_bf16 of two values at once (packed conversions); a in the low halves.
__device__ __forceinline__ void split_bf16x2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const float2 hf = __bfloat1622float2(h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(a - hf.x, b - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// Byte offset of element e (of `esize` bytes) in row r of a 128B-swizzled K-major chunk.
__device__ __forceinline__ uint32_t sw128_offset(uint32_t r, uint32_t e, uint32_t esize) {
  const uint32_t byte = e * esize;
  return r * 128 + ((((byte >> 4) ^ (r & 7))) << 4) + (byte & 15);
}
// Byte offset of element e (of esize bytes) of row r in a 64-byte-swizzled K-major tile:
// rows of 64 B, 8-row atoms of 512 B, 16-byte chunk c stored at c ^ ((r >> 1) & 3).
__device__ __forceinline__ uint32_t sw64_offset(uint32_t r, uint32_t e, uint32_t esize) {
  const uint32_t byte = e * esize;
  return r * 64 + ((((byte >> 4) ^ ((r >> 1) & 3))) << 4) + (byte & 15);
}
// Operand descriptor of the tensor-core DCT's layout (TF32: 128 B swizzle, BF16: 64 B).
template <int kDct>
__device__ __forceinline__ uint64_t dct_desc(uint32_t saddr) {
  if constexpr (kDct == 1) return sw128_desc(saddr);
  else return sw64_desc(saddr);
}
// 16 consecutive TMEM columns of this warp's 32 lanes (valid after tmem_ld_wait).
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_take16(uint32_t (&r)[16]) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
}

template <typename Tin, int kDct, bool kSep>
__global__ void __launch_bounds__(hash_threads<kDct>(), 2)
    hash_kernel(const HashLaunch prm) {
  constexpr int kRowBytes = InputTraits<Tin>::kRowBytes;
  constexpr int kGroups = stage_groups<Tin>();
  constexpr int kStageBytes = 4 * kGroups * kRowBytes;
  constexpr int kNumStages = ring_stages<Tin, kDct>();
  constexpr int kStagesPerImage = kGroupsPerImage / kGroups;
  constexpr int kThreads = hash_threads<kDct>();
  using Smem = HashSmem<kStageBytes, kNumStages, kDct>;
  extern __shared__ unsigned char smem_raw[];
  // Align by offsetting the shared array itself so the compiler keeps the shared address
  // space (an integer round trip would turn every access into a generic one).
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;

  for (int idx = tid; idx < 16 * 127; idx += kThreads) {
    const int k = idx / 127, i = idx - k * 127;
    sm.dt[i + 1][k] = g_dct[idx];
  }
  if (tid < 16) sm.dt[0][tid] = 0.0f;
  if constexpr (kDct != 0) {
    // the DCT matrix as the MMA's B operand: N = 16 rows k, K = 128 (column 127 is zero)
    for (int idx = tid; idx < 16 * 128; idx += kThreads) {
      const int k = idx >> 7, i = idx & 127;
      const float d = i < 127 ? g_dct[k * 127 + i] : 0.0f;
      if constexpr (kDct == 1) {
        *reinterpret_cast<uint32_t*>(sm.dops + (i >> 5) * 2048 + sw128_offset(k, i & 31, 4)) = to_tf32(d);
      } else {
        uint16_t hi, lo;
        split_bf16(d, hi, lo);
        const uint32_t off = (i >> 5) * 1024 + sw64_offset(k, i & 31, 2);
        *reinterpret_cast<uint16_t*>(sm.dops + off) = hi;
        *reinterpret_cast<uint16_t*>(sm.dops + 4096 + off) = lo;
      }
    }
    fence_proxy_async_smem();
  }
  if (tid == 0) {
    for (int s = 0; s < kNumStages; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], kComputeThreads / 32);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.pfull[b], kComputeThreads / 32);
      mbar_init(&sm.pempty[b], 1);
      mbar_init(&sm.a_full[b], kComputeThreads / 32);
      mbar_init(&sm.a_empty[b], 1);
      mbar_init(&sm.acc_full[b], 1);
      mbar_init(&sm.acc_empty[b], kComputeThreads / 32);
    }
    mbar_init(&sm.tc_exit, kComputeThreads / 32);
    mbar_init(&sm.mma_done, 1);
    sm.abort_flag = 0;
    fence_mbar_init();
  }
  if constexpr (kDct != 0) {
    if (warp == kMmaWarpHash) {
      tmem_alloc(&sm.tmem_base, 32);  // two 16-column accumulators
      tmem_relinquish();
    }
    tc_fence_before();
  }
  __syncthreads();
  if constexpr (kDct != 0) tc_fence_after();

  volatile int* abort_flag = &sm.abort_flag;
  const int64_t n_images = prm.n_dev ? min(*prm.n_dev, prm.n) : prm.n;
  const unsigned char* images = static_cast<const unsigned char*>(prm.images);
  constexpr int64_t kImageBytes = 512ll * kRowBytes;

  if (warp == kProducerWarp) {
    if (lane != 0) return;
    const uint64_t policy = policy_evict_first();
    uint32_t g = 0;
    bool ok = true;
    for (int64_t n = blockIdx.x; n < n_images && ok; n += gridDim.x) {
      const unsigned char* img = images + n * kImageBytes;
      for (int s = 0; s < kStagesPerImage; ++s, ++g) {
        const uint32_t slot = g % kNumStages;
        if (!mbar_wait(&sm.empty[slot], ((g / kNumStages) & 1u) ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        // rows past 510 are read by no output
        const uint32_t bytes = kStageBytes - (s < kStagesPerImage - 1 ? 0 : 2 * kRowBytes);
        mbar_arrive_expect_tx(&sm.full[slot], bytes);
        bulk_g2s(sm.ring[slot], img + kRowBytes + static_cast<int64_t>(s) * kStageBytes, bytes,
                 &sm.full[slot], policy);
      }
    }
    if (!ok) {
      *abort_flag = 1;
      atomicOr(prm.dev_err, kDevErrTimeout);
      // Let the copies already issued land before the CTA exits (bounded wait each).
      for (uint32_t k = 1; k <= kNumStages && k <= g; ++k) {
        const uint32_t gi = g - k;
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&sm.full[gi % kNumStages], (gi / kNumStages) & 1u)) {
          if (globaltimer_ns() - t0 > kWaitLimitNs / 4) break;
        }
      }
    }
    return;
  }

  if (warp == kEpilogueWarp) {
    uint32_t it = 0;
    for (int64_t n = blockIdx.x; n < n_images; n += gridDim.x, ++it) {
      const int pb = it & 1;
      if (!mbar_wait(&sm.pfull[pb], (it >> 1) & 1u, abort_flag)) {
        *abort_flag = 1;
        if (lane == 0) atomicOr(prm.dev_err, kDevErrTimeout);
        return;
      }
      EpilogueOut o;
      o.hashes = prm.hashes ? prm.hashes + n * 256 : nullptr;
      o.quality = prm.quality ? prm.quality + n * 8 : nullptr;
      o.thresholds = prm.thresholds ? prm.thresholds + n * 8 : nullptr;
      o.pdqf_slots = prm.pdqf_slots;
      o.pdqf = prm.pdqf ? prm.pdqf + n * (prm.pdqf_slots == 8 ? 8 : 1) * 256 : nullptr;
      epilogue_warp(sm.p[pb][0], false, 0.0f, prm.row_mask, prm.col_mask, lane, o);
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.pempty[pb]);
    }
    return;
  }

  if constexpr (kDct != 0) {
    if (warp == kMmaWarpHash) {
      constexpr int kChunks = 128 / DctTraits<kDct>::kRowsPerChunk;
      const uint32_t tmem = sm.tmem_base;
      if (lane == 0) {
        bool ok = true;
        uint32_t gc = 0, it = 0;
        for (int64_t n = blockIdx.x; n < n_images && ok; n += gridDim.x, ++it) {
          const uint32_t acc = it & 1;
          if (!mbar_wait(&sm.acc_empty[acc], ((it >> 1) & 1u) ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          for (int c = 0; c < kChunks; ++c, ++gc) {
            const uint32_t buf = gc & 1;
            if (!mbar_wait(&sm.a_full[buf], (gc >> 1) & 1u, abort_flag)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t a = smem_u32(sm.ops[buf]);
            using TR = DctTraits<kDct>;
            const uint32_t d = smem_u32(sm.dops) + c * TR::kDChunkBytes;
#pragma unroll
            for (int ks = 0; ks < TR::kKSteps; ++ks) {
              const uint32_t accumulate = (c > 0 || ks > 0) ? 1u : 0u;
              if constexpr (kDct == 1) {
                mma_tf32(tmem + acc * 16, dct_desc<kDct>(a + ks * 32), dct_desc<kDct>(d + ks * 32),
                         kIdescTf32, accumulate);
              } else {
                // x * y ~ xh*yh + xh*yl + xl*yh   (x = A, y = D)
                mma_bf16(tmem + acc * 16, dct_desc<kDct>(a + ks * 32),
                         dct_desc<kDct>(d + ks * 32), kIdescBf16, accumulate);
                mma_bf16(tmem + acc * 16, dct_desc<kDct>(a + ks * 32),
                         dct_desc<kDct>(d + TR::kDLo + ks * 32), kIdescBf16, 1u);
                mma_bf16(tmem + acc * 16, dct_desc<kDct>(a + TR::kALo + ks * 32),
                         dct_desc<kDct>(d + ks * 32), kIdescBf16, 1u);
              }
            }
            mma_commit(&sm.a_empty[buf]);
          }
          if (ok) mma_commit(&sm.acc_full[acc]);
        }
        if (!ok) {
          *abort_flag = 1;
          atomicOr(prm.dev_err, kDevErrTimeout);
        }
        mma_commit(&sm.mma_done);
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&sm.mma_done, 0))
          if (globaltimer_ns() - t0 > kWaitLimitNs) {
            // the MMAs did not drain: the results are not trustworthy, so flag the launch
            *abort_flag = 1;
            atomicOr(prm.dev_err, kDevErrTimeout);
            break;
          }
      }
      __syncwarp();
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(&sm.tc_exit, 0))
        if (globaltimer_ns() - t0 > kWaitLimitNs) {
          // the compute warps did not report that they stopped reading tensor memory
          if (lane == 0) {
            *abort_flag = 1;
            atomicOr(prm.dev_err, kDevErrTimeout);
          }
          break;
        }
      tc_fence_after();
      tmem_dealloc(tmem, 32);
      return;
    }
  }

  // ---- compute warps: thread j <-> compressed column j (thread 127 repeats column 126 and
  // drops it)
  const int j = tid, jc = min(tid, 126);
  const bool active = j < 127;
  const float nz = prm.neg_zero;
  uint32_t it = 0, slot = 0, phase = 0;  // the stage being read
  for (int64_t n = blockIdx.x; n < n_images; n += gridDim.x, ++it) {
    typename std::conditional<kSep, HCarry, TapSum>::type carry;
    float* const buf1 = prm.buf1 && active ? prm.buf1 + n * 127 * 128 + j : nullptr;
    // FP32: the 16 x 4 accumulators [pair of frequencies][partial sum]
    float2 acc[kDct == 0 ? 8 : 1][4];
#pragma unroll
    for (int k = 0; k < (kDct == 0 ? 8 : 1); ++k)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[k][r] = make_float2(0.0f, 0.0f);
    // tensor cores: values 4 q - 4 .. 4 q - 1, written to the operand as one unit
    float unit[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    auto write_unit = [&](int u) -> bool {  // rows 4 u .. 4 u + 3 of the operand
      constexpr int kR = DctTraits<kDct>::kRowsPerChunk;
      const uint32_t within = static_cast<uint32_t>(4 * u % kR);
      const uint32_t chunk = it * (128 / kR) + static_cast<uint32_t>(4 * u / kR);
      const uint32_t buf = chunk & 1;
      if (within == 0 && !mbar_wait(&sm.a_empty[buf], ((chunk >> 1) & 1u) ^ 1u, abort_flag))
        return false;
      if constexpr (kDct == 1) {
        const uint4 w = make_uint4(to_tf32(unit[0]), to_tf32(unit[1]), to_tf32(unit[2]), to_tf32(unit[3]));
        *reinterpret_cast<uint4*>(sm.ops[buf] + sw128_offset(j, within, 4)) = w;
      } else if constexpr (kDct == 2) {
        uint32_t h01, l01, h23, l23;
        split_bf16x2(unit[0], unit[1], h01, l01);
        split_bf16x2(unit[2], unit[3], h23, l23);
        const uint32_t off = sw64_offset(j, within, 2);
        *reinterpret_cast<uint2*>(sm.ops[buf] + off) = make_uint2(h01, h23);
        *reinterpret_cast<uint2*>(sm.ops[buf] + DctTraits<kDct>::kALo + off) = make_uint2(l01, l23);
      }
      if (within + 4 == static_cast<uint32_t>(kR)) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.a_full[buf]);
      }
      return true;
    };
    // groups 4 q .. 4 q + 3 finish values 4 q - 1 .. 4 q + 2, so that each value's partial sum
    // (value % 4) is known at compile time
#pragma unroll 1
    for (int q = 0; q < kGroupsPerImage / 4; ++q) {
      float2 pair = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        if (o % 2 == 0) {
          if (o % kGroups == 0 && !mbar_wait(&sm.full[slot], phase, abort_flag)) goto fail;
          const Tin* rows =
              reinterpret_cast<const Tin*>(sm.ring[slot] + (o % kGroups) * 4 * kRowBytes);
          pair = compress_pair(rows, jc, o == 2 && q == kGroupsPerImage / 4 - 1, nz, carry);
          if (o % kGroups == kGroups - 2) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.empty[slot]);
            if (++slot == kNumStages) {
              slot = 0;
              phase ^= 1u;
            }
          }
        }
        float b = o % 2 == 0 ? pair.x : pair.y;
        const int i = 4 * q + o - 1;
        if (o == 0 && q == 0) b = 0.0f;  // there is no value -1
        if (buf1 && i >= 0) buf1[i * 128] = b;
        if constexpr (kDct == 0) {
          const float4* d4 = reinterpret_cast<const float4*>(sm.dt[i + 1]);
          const float2 bb = make_float2(b, b);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 d = d4[k];
            float2& a0 = acc[2 * k][(o + 3) & 3];
            float2& a1 = acc[2 * k + 1][(o + 3) & 3];
            a0 = add2_rn(a0, mul2_rn(make_float2(d.x, d.y), bb, nz));
            a1 = add2_rn(a1, mul2_rn(make_float2(d.z, d.w), bb, nz));
          }
        } else {
          unit[(o + 3) & 3] = active ? b : 0.0f;
          if (o == 0 && q > 0 && !write_unit(q - 1)) goto fail;
        }
      }
    }
    if constexpr (kDct == 0) {
      if (active) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float2 t = add2_rn(add2_rn(add2_rn(acc[k][0], acc[k][1]), acc[k][2]), acc[k][3]);
          sm.t[2 * k][j] = t.x;
          sm.t[2 * k + 1][j] = t.y;
        }
      }
    } else {
      unit[3] = 0.0f;  // value 127
      if (!write_unit(kGroupsPerImage / 4 - 1)) goto fail;
      const uint32_t ac = it & 1;
      if (!mbar_wait(&sm.acc_full[ac], (it >> 1) & 1u, abort_flag)) goto fail;
      tc_fence_after();
      uint32_t tr[16];
      tmem_ld16_nowait(sm.tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + ac * 16, tr);
      tmem_ld_wait();
      tmem_take16(tr);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.acc_empty[ac]);
      if (active) {
#pragma unroll
        for (int k = 0; k < 16; ++k) sm.t[k][j] = __uint_as_float(tr[k]);
      }
    }
    named_bar_sync(kComputeBarrier, kComputeThreads);
    {
      // stage 2: P[k][c] = sum_m T[k][m] * D[c][m]; thread -> (k, c0), (k, c0 + 1)
      const int k = tid >> 3, c0 = (tid & 7) * 2;
      float2 sum[4] = {};
#pragma unroll 8
      for (int m0 = 0; m0 < 128; m0 += 4) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int m = m0 + r;
          if (m < 127) {
            const float tv = sm.t[k][m];
            const float2 d = *reinterpret_cast<const float2*>(&sm.dt[m + 1][c0]);
            sum[r] = add2_rn(sum[r], mul2_rn(d, make_float2(tv, tv), nz));
          }
        }
      }
      const float2 p = add2_rn(add2_rn(add2_rn(sum[0], sum[1]), sum[2]), sum[3]);
      const int pb = it & 1;
      if (!mbar_wait(&sm.pempty[pb], ((it >> 1) & 1u) ^ 1u, abort_flag)) goto fail;
      sm.p[pb][k][c0] = p.x;
      sm.p[pb][k][c0 + 1] = p.y;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.pfull[pb]);
    }
    named_bar_sync(kComputeBarrier, kComputeThreads);
  }
  if constexpr (kDct != 0) {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.tc_exit);
  }
  return;
fail:
  *abort_flag = 1;
  if (lane == 0) atomicOr(prm.dev_err, kDevErrTimeout);
  if constexpr (kDct != 0) {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.tc_exit);
  }
}

// --------------------------------------------------------------- split kernel
//
// hash_split_kernel: the FP32 hash of a small batch, one image per cluster of 8 CTAs.
//
// hash_kernel walks an image's 128 groups of rows one after another on one CTA, 27-39 us however
// small the batch, so a batch of fewer images than CTAs leaves most of the chip idle and waits for a
// latency chain. Here the image is cut by rows: CTA c of the cluster copies the 66 input
// rows of compressed rows 16 c .. 16 c + 15 at once (five bulk copies, no ring), and the
// chains that are serial by definition are cut along their independent directions:
//   compress  CTA c, thread (column j, group g): rows 16 c + 4 g .. + 3 of column j, each
//             value sent to the CTA that owns column j (16 columns per CTA) by an
//             asynchronous store into its shared memory;
//   stage 1   CTA c: T[k][j] of its 16 columns, the reference's four partial sums over i in
//             four lanes, each 32 steps long; T goes to the cluster's first CTA;
//   stage 2   first CTA: P[k][c], the same routine with T in the place of the image;
//   epilogue  first CTA: four warps select one median each and pack its two slots; eight
//             warps sum one slot's gradients (480 dependent additions, the longest chain).
// Every sum keeps its order, so the results are hash_kernel's bit for bit.
//
// Bound by the latency of that sequence: of ~12,500 clk for one f32 image, ~2,800 until the
// rows are there, ~2,000 compress (8 conflict-free 16-byte loads per value), ~500 for each of
// the two exchanges, ~1,150 per DCT stage and ~4,200 epilogue (2,150 of them the gradient
// sum). Back to back, one image: 8.5 us (hash_kernel 31 us for f32, 27 u8); RGB8 9.6 us (39);
// 37 u8 images 13.4 us (27), or 14.2 when each call brings new ones, from HBM; 56 f32 images
// 27.3 us (31).
constexpr int kSplitCtas = 8;        // CTAs per image (the portable cluster size)
constexpr int kSplitThreads = 512;
constexpr int kSplitRows = 128 / kSplitCtas;           // compressed rows per CTA
constexpr int kSplitInRows = 4 * kSplitRows + 2;       // input rows they read
// compress_pair's last pair reads two rows more, for a start that nothing continues
template <typename Tin>
constexpr int kSplitPadRows = sizeof(Tin) == 1 ? 2 : 0;
constexpr int kSplitCopies = (kSplitInRows + 15) / 16; // bulk copies of up to 16 rows

constexpr int kSplitPitch = 132;  // floats per column of a stage's input (16-byte columns)

struct SplitSmem {
  // stage inputs column by column: the lanes of the four partial sums read values
  // 4 s .. 4 s + 3 of 8 columns, 32 different banks at this pitch.
  // [0]: compressed columns 16 c .. 16 c + 15; [1], first CTA only: T[k][j]
  alignas(16) float in[2][16][kSplitPitch];
  alignas(16) float dt[128][16];   // dt[i][k] = D[k][i]; row 127 is zero
  float p[16][17];                 // PDQF, padded: slots 4-7 read it by columns
  alignas(16) float grad[8][500];  // |differences| of a slot in summation order, padded
  uint64_t full[kSplitCopies];     // input rows
  uint64_t dt_full, in_full[2];    // DCT matrix; stage inputs, from all CTAs
  int abort_flag;
};
constexpr int kSplitRowsOffset = (sizeof(SplitSmem) + 127) & ~127;  // the input rows follow

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// Address of `p` (a place in this CTA's shared memory) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_cluster(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// Asynchronous stores to another CTA that count their bytes on its mbarrier: the receiver
// waits for the data alone (one way), where a cluster barrier after plain stores waits for
// their acknowledgement and then for the barrier (~1,300 clk measured).
__device__ __forceinline__ void st_async4(uint32_t dst, uint32_t bar, float x, float y, float z,
                                          float w) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
      ::"r"(dst), "r"(__float_as_uint(x)), "r"(__float_as_uint(y)), "r"(__float_as_uint(z)),
      "r"(__float_as_uint(w)), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void st_async1(uint32_t dst, uint32_t bar, float x) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
               "r"(__float_as_uint(x)), "r"(bar)
               : "memory");
}

// One DCT stage of 16 x 16 outputs by 128 threads: out(x, y) = sum over m < 127 of
// in[stage][x][m] * D[y][m] in the reference's four partial sums. Thread (warp w, lane):
// partial sum r = lane / 8, x = lane % 8 and x + 8, y = 4 w .. + 3 (the D values serve two
// columns: the loads, four wavefronts for four D values, are what bounds this loop); the
// sums are combined in lanes 0-7. Stage 0 (stage 1 of the DCT) sends T[y][16 rank + x] to
// the first CTA, stage 1 writes P[x][y].
// (Row 127 of the input and of D^T is zero: it adds +-0 to a sum that is never -0.)
__device__ __forceinline__ void split_dct_stage(SplitSmem& sm, int stage, int rank, int w,
                                                int lane, float neg_zero) {
  const int r = lane >> 3, x = lane & 7, y0 = 4 * w;
  const float* src = &sm.in[stage][x][r];
  const float* dsrc = &sm.dt[r][y0];
  float2 a[2][2] = {};  // [column][pair of y]
#pragma unroll 8
  for (int s = 0; s < 32; ++s) {  // m = 4 s + r
    const float b0 = src[4 * s], b1 = src[4 * s + 8 * kSplitPitch];
    const float4 d = *reinterpret_cast<const float4*>(dsrc + 64 * s);
    const float2 d0 = make_float2(d.x, d.y), d1 = make_float2(d.z, d.w);
    a[0][0] = add2_rn(a[0][0], mul2_rn(d0, make_float2(b0, b0), neg_zero));
    a[0][1] = add2_rn(a[0][1], mul2_rn(d1, make_float2(b0, b0), neg_zero));
    a[1][0] = add2_rn(a[1][0], mul2_rn(d0, make_float2(b1, b1), neg_zero));
    a[1][1] = add2_rn(a[1][1], mul2_rn(d1, make_float2(b1, b1), neg_zero));
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float v[4] = {a[h][0].x, a[h][0].y, a[h][1].x, a[h][1].y};
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const float s1 = __shfl_down_sync(0xffffffffu, v[y], 8);
      const float s2 = __shfl_down_sync(0xffffffffu, v[y], 16);
      const float s3 = __shfl_down_sync(0xffffffffu, v[y], 24);
      v[y] = __fadd_rn(__fadd_rn(__fadd_rn(v[y], s1), s2), s3);
    }
    if (lane < 8) {
      if (stage == 0) {
        const uint32_t bar = map_cluster(&sm.in_full[1], 0);
        const uint32_t dst = map_cluster(&sm.in[1][y0][16 * rank + x + 8 * h], 0);
#pragma unroll
        for (int y = 0; y < 4; ++y) st_async1(dst + 4 * kSplitPitch * y, bar, v[y]);
      } else {
#pragma unroll
        for (int y = 0; y < 4; ++y) sm.p[x + 8 * h][y0 + y] = v[y];
      }
    }
  }
}

// Quality of slot s by one warp: its 480 absolute differences in parallel into `g` in the
// reference's order (240 down the columns, row by row, then 240 along the rows), then the
// sequential sum in lane 0 (480 dependent additions, the loads 16 values ahead of them).
// Of |s x - s' y| with signs s and s' only their product matters.
__device__ __forceinline__ void split_quality(const float* P, int s, uint32_t rm, uint32_t cm,
                                              int lane, float* g, float* quality) {
  const SlotView m(P, s, rm, cm);
  const int r0 = lane >> 4, c = lane & 15;
  const float* p = P + r0 * m.row + c * m.col;
  const int right = c < 15 ? m.col : 0;
  // bit 2 t: rows r0 + 2 t and r0 + 2 t + 1 differ in sign; all bits: columns c and c + 1 do
  const uint32_t rdiff = (m.rows ^ (m.rows >> 1)) >> r0;
  const uint32_t cdiff = ((m.cols ^ (m.cols >> 1)) >> c) << 31;
#pragma unroll
  for (int t = 0; t < 8; ++t, p += 2 * m.row) {
    // (the last row's lower neighbour is past the matrix, inside the shared struct: unused)
    const float x = p[0];
    const float below = __uint_as_float(__float_as_uint(p[m.row]) ^ ((rdiff >> (2 * t)) << 31));
    const float beside = __uint_as_float(__float_as_uint(p[right]) ^ cdiff);
    if (t < 7 || r0 == 0) g[16 * (r0 + 2 * t) + c] = fabsf(__fsub_rn(x, below));
    if (c < 15) g[240 + 15 * (r0 + 2 * t) + c] = fabsf(__fsub_rn(x, beside));
  }
  __syncwarp();
  if (lane != 0) return;
  const float4* g4 = reinterpret_cast<const float4*>(g);
  float4 a[4], b[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) a[q] = g4[q];
  float sum = 0.0f;
#pragma unroll 1
  for (int t = 0; t < 120; t += 8) {
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = g4[t + 4 + q];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, a[q].x), a[q].y), a[q].z), a[q].w);
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = g4[t + 8 + q];  // the last step reads the padding
#pragma unroll
    for (int q = 0; q < 4; ++q)
      sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, b[q].x), b[q].y), b[q].z), b[q].w);
  }
  quality[s] = fminf(__fdiv_rn(sum, 180.0f), 1.0f);
}

template <typename Tin>
__global__ void __cluster_dims__(kSplitCtas, 1, 1) __launch_bounds__(kSplitThreads, 2)
    hash_split_kernel(const HashLaunch prm) {
  constexpr int kRowBytes = InputTraits<Tin>::kRowBytes;
  extern __shared__ unsigned char smem_raw[];
  SplitSmem& sm =
      *reinterpret_cast<SplitSmem*>(smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u));
  unsigned char* const rows = reinterpret_cast<unsigned char*>(&sm) + kSplitRowsOffset;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int64_t n = blockIdx.x / kSplitCtas;
  if (prm.n_dev && n >= *prm.n_dev) return;  // the whole cluster
  const int row0 = 4 * kSplitRows * rank + 1;  // first input row
  if (tid < kSplitCopies) {  // one lane per copy
    mbar_init(&sm.full[tid], 1);
    fence_mbar_init();
    const unsigned char* img =
        static_cast<const unsigned char*>(prm.images) + n * (512ll * kRowBytes);
    // rows past 510 are read by no output
    const int first = row0 + 16 * tid;
    const int count = min(min(16, kSplitInRows - 16 * tid), 511 - first);
    if (count > 0) {
      const uint32_t bytes = static_cast<uint32_t>(count) * kRowBytes;
      mbar_arrive_expect_tx(&sm.full[tid], bytes);
      bulk_g2s(rows + 16 * tid * kRowBytes, img + static_cast<int64_t>(first) * kRowBytes, bytes,
               &sm.full[tid], policy_evict_first());
    }
  } else if (tid == 32) {
    mbar_init(&sm.dt_full, 1);
    mbar_init(&sm.in_full[0], 1);
    mbar_init(&sm.in_full[1], 1);
    sm.abort_flag = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(&sm.in_full[0], 16 * 128 * 4);
    if (rank == 0) mbar_arrive_expect_tx(&sm.in_full[1], 16 * 128 * 4);
    mbar_arrive_expect_tx(&sm.dt_full, sizeof(sm.dt));
    bulk_g2s(sm.dt, g_dct_t, sizeof(sm.dt), &sm.dt_full, policy_evict_last());
  }
  __syncthreads();
  cluster_arrive();  // this CTA runs and its barriers are set: the others may write to it

  // ---- compress: thread (j, g), rows 4 g .. 4 g + 3 of the CTA's 16
  const int j = tid & 127, g = tid >> 7;
  volatile int* abort_flag = &sm.abort_flag;
  bool ok = mbar_wait(&sm.full[g], 0, abort_flag);
  // the last output's last two input rows are in the next copy (none past the image's end)
  if (row0 + 16 * (g + 1) <= 510) ok &= mbar_wait(&sm.full[g + 1], 0, abort_flag);
  float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  const int i0 = kSplitRows * rank + 4 * g;
  if (j < 127) {
    // the group before the first value starts it; group r + 1 finishes value r (there is no
    // value 127: what stands in its rows' place is summed and dropped)
    const Tin* st = reinterpret_cast<const Tin*>(rows + 16 * g * kRowBytes);
    TapSum carry;
    compress_group(st, j, false, carry);
#pragma unroll
    for (int r = 0; r < 4; r += 2) {
      const Tin* next = st + 4 * (r + 1) * 512;
      float2 pair;
      if constexpr (sizeof(Tin) == 1) {  // 37 images from L2 14.6 -> 13.4 us (RGB: 0.5 % slower)
        pair = compress_pair(next, j, r == 2, prm.neg_zero, carry);
      } else {
        pair.x = compress_group(next, j, false, carry);
        pair.y = compress_group(next + 4 * 512, j, r == 2, carry);
      }
      b[r] = pair.x;
      b[r + 1] = i0 + r + 1 < 127 ? pair.y : 0.0f;
      if (prm.buf1) {
        prm.buf1[(n * 127 + i0 + r) * 128 + j] = pair.x;
        if (i0 + r + 1 < 127) prm.buf1[(n * 127 + i0 + r + 1) * 128 + j] = pair.y;
      }
    }
  }
  cluster_wait();
  {
    const uint32_t owner = static_cast<uint32_t>(j >> 4);
    st_async4(map_cluster(&sm.in[0][j & 15][i0], owner), map_cluster(&sm.in_full[0], owner), b[0],
              b[1], b[2], b[3]);
  }

  // ---- stage 1: T[k][16 rank + x], to the first CTA; stage 2 there, by the same code:
  // P[x][y] = sum over m of T[x][m] D[y][m]
  if (warp < 4) {
    ok &= mbar_wait(&sm.dt_full, 0, abort_flag);
#pragma unroll 1
    for (int stage = 0; stage < (rank == 0 ? 2 : 1); ++stage) {
      ok &= mbar_wait(&sm.in_full[stage], 0, abort_flag);
      split_dct_stage(sm, stage, rank, warp, lane, prm.neg_zero);
      __syncwarp();
    }
  }
  cluster_arrive_relaxed();  // waited for at the end: no CTA leaves while another may write to it
  if (!ok && lane == 0) {
    // data did not land in time (or another warp's did not): the outputs are not trustworthy.
    // Everything still on its way into this CTA, copies and the other CTAs' stores alike, gets a
    // last bounded wait before the CTA may exit.
    *abort_flag = 1;
    atomicOr(prm.dev_err, kDevErrTimeout);
    const uint64_t t0 = globaltimer_ns();
    const auto landed = [t0](uint64_t* bar) {
      while (!mbar_try_wait(bar, 0) && globaltimer_ns() - t0 < kWaitLimitNs / 4) {
      }
    };
#pragma unroll 1
    for (int c = 0; c < kSplitCopies; ++c)
      if (row0 + 16 * c <= 510) landed(&sm.full[c]);
    landed(&sm.dt_full);
    landed(&sm.in_full[0]);
    if (rank == 0) landed(&sm.in_full[1]);
  }
  if (rank == 0) {
    __syncthreads();
    if (warp < 8) {
      if (prm.quality)
        split_quality(sm.p[0], warp, prm.row_mask, prm.col_mask, lane, sm.grad[warp],
                      prm.quality + n * 8);
    } else if (warp < 12) {
      EpilogueOut o;
      o.hashes = prm.hashes ? prm.hashes + n * 256 : nullptr;
      o.quality = nullptr;
      o.thresholds = prm.thresholds ? prm.thresholds + n * 8 : nullptr;
      o.pdqf_slots = prm.pdqf_slots;
      o.pdqf = prm.pdqf ? prm.pdqf + n * (prm.pdqf_slots == 8 ? 8 : 1) * 256 : nullptr;
      slot_pairs<1>(sm.p[0], warp - 8, prm.row_mask, prm.col_mask, lane, o, false, 0.0f);
    }
  }
  cluster_wait();
}

// Dihedrals of given PDQF matrices: one warp per matrix.
__global__ void __launch_bounds__(128) dihedral_kernel(const DihedralLaunch prm) {
  __shared__ float P[4][16 * 17];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t n = static_cast<int64_t>(blockIdx.x) * 4 + w;
  if (n >= prm.n) return;
  const float4* src = reinterpret_cast<const float4*>(prm.pdqf + n * 256);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 x = src[lane + 32 * h];
    float* dst = &P[w][17 * ((lane + 32 * h) >> 2) + 4 * (lane & 3)];
    dst[0] = x.x;
    dst[1] = x.y;
    dst[2] = x.z;
    dst[3] = x.w;
  }
  __syncwarp();
  EpilogueOut o;
  o.hashes = prm.hashes ? prm.hashes + n * 256 : nullptr;
  o.quality = prm.quality ? prm.quality + n * 8 : nullptr;
  o.thresholds = prm.thresholds ? prm.thresholds + n * 8 : nullptr;
  o.pdqf = prm.pdqf_out ? prm.pdqf_out + n * 8 * 256 : nullptr;
  o.pdqf_slots = 8;
  const bool given = prm.thr_in != nullptr;
  epilogue_warp(P[w], given, given ? prm.thr_in[n] : 0.0f, prm.row_mask, prm.col_mask, lane, o);
}

// ------------------------------------------------------------------ host side

template <typename Tin, int kDct>
static size_t hash_smem_bytes() {
  return sizeof(HashSmem<4 * stage_groups<Tin>() * InputTraits<Tin>::kRowBytes,
                         ring_stages<Tin, kDct>(), kDct>) +
         1024;  // + base alignment
}

// Dynamic shared memory size, and the largest shared-memory carveout so that the
// occupancy query (and the grid) count the two CTAs per SM that fit.
template <typename Tin, int kDct, bool kSep>
static cudaError_t set_smem_attr_one() {
  cudaError_t e = cudaFuncSetAttribute(hash_kernel<Tin, kDct, kSep>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(hash_smem_bytes<Tin, kDct>()));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(hash_kernel<Tin, kDct, kSep>,
                              cudaFuncAttributePreferredSharedMemoryCarveout,
                              static_cast<int>(cudaSharedmemCarveoutMaxShared));
}



// Resident CTAs per SM. The runtime's occupancy query answers 1 for the tcgen05 variants
// although their registers and shared memory admit 2 (ncu's occupancy section agrees on 2),
// so the count is also derived from the per-SM limits and the larger answer is used.
template <typename Tin, int kDct, bool kSep>
static cudaError_t occupancy_of(int* ctas) {
  int api = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &api, hash_kernel<Tin, kDct, kSep>, hash_threads<kDct>(), hash_smem_bytes<Tin, kDct>());
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa{};
  int dev = 0, smem_sm = 0, reserved = 0, regs_sm = 0, threads_sm = 0;
  e = cudaFuncGetAttributes(&fa, hash_kernel<Tin, kDct, kSep>);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&threads_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
  if (e != cudaSuccess) return e;
  const int threads = hash_threads<kDct>();
  const size_t smem_block = hash_smem_bytes<Tin, kDct>() + fa.sharedSizeBytes + reserved;
  const int regs_warp = ((fa.numRegs * 32 + 255) / 256) * 256;  // allocation unit: 256
  const int by_smem = static_cast<int>(smem_sm / smem_block);
  const int by_regs = regs_sm / (regs_warp * (threads / 32));
  const int by_threads = threads_sm / threads;
  int derived = by_smem < by_regs ? by_smem : by_regs;
  if (by_threads < derived) derived = by_threads;
  *ctas = api > derived ? api : derived;
  return cudaSuccess;
}

cudaError_t hash_occupancy(int input_kind, int* ctas_per_sm) {
  return hash_occupancy_variant(input_kind, 0, 0, ctas_per_sm);
}

// Calls F<Tin, kDct, kSep>::run(args...) for the runtime (input kind, DCT, separable).
template <template <typename, int, bool> class F, typename... A>
static cudaError_t dispatch(int kind, int dct, int sep, A&&... args) {
#define YPDQ_CASE(K, T)                                                        \
  case K:                                                                      \
    switch (dct * 2 + (sep ? 1 : 0)) {                                         \
      case 0: return F<T, 0, false>::run(args...);                             \
      case 1: return F<T, 0, true>::run(args...);                              \
      case 2: return F<T, 1, false>::run(args...);                             \
      case 3: return F<T, 1, true>::run(args...);                              \
      case 4: return F<T, 2, false>::run(args...);                             \
      case 5: return F<T, 2, true>::run(args...);                              \
      default: return cudaErrorInvalidValue;                                   \
    }
  switch (kind) {
    YPDQ_CASE(YPDQ_INPUT_F32, float)
    YPDQ_CASE(YPDQ_INPUT_U8, uint8_t)
    YPDQ_CASE(YPDQ_INPUT_RGB8, rgb8_t)
    YPDQ_CASE(YPDQ_INPUT_RGBA8, rgba8_t)
    default: return cudaErrorInvalidValue;
  }
#undef YPDQ_CASE
}

template <typename Tin, int kDct, bool kSep>
struct OccupancyOf {
  static cudaError_t run(int* ctas) { return occupancy_of<Tin, kDct, kSep>(ctas); }
};
template <typename Tin, int kDct, bool kSep>
struct SetSmemAttr {
  static cudaError_t run() { return set_smem_attr_one<Tin, kDct, kSep>(); }
};
template <typename Tin, int kDct, bool kSep>
struct LaunchOne {
  static cudaError_t run(const HashLaunch& p, int64_t grid, cudaStream_t s) {
    hash_kernel<Tin, kDct, kSep><<<static_cast<int>(grid), hash_threads<kDct>(),
                                   hash_smem_bytes<Tin, kDct>(), s>>>(p);
    return cudaGetLastError();
  }
};

template <typename Tin>
static size_t split_smem_bytes() {
  return kSplitRowsOffset + (kSplitInRows + kSplitPadRows<Tin>) * InputTraits<Tin>::kRowBytes +
         128;  // + base alignment
}
template <typename Tin>
static cudaError_t set_split_smem() {
  return cudaFuncSetAttribute(hash_split_kernel<Tin>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(split_smem_bytes<Tin>()));
}
template <typename Tin>
static cudaError_t launch_split(const HashLaunch& p, cudaStream_t s) {
  hash_split_kernel<Tin><<<static_cast<unsigned>(kSplitCtas * p.n), kSplitThreads,
                           split_smem_bytes<Tin>(), s>>>(p);
  return cudaGetLastError();
}

// Largest batch that hash_split_kernel takes. Its time grows with the waves of clusters (16 or
// more images at once), hash_kernel's is that of one image on a CTA up to 152 images (f32
// 31-38 us, u8 27 us, RGB 39 us). Measured on both sides, split against persistent: f32
// 27.3 / 31.1 us at 56 images and 32.0 / 31.4 at 64; u8 25.4 / 27.0 at 104 and 27.4 / 27.0 at
// 112; RGB8 35.4 / 39.3 at 72 and 41.0 / 39.3 at 80; RGBA8 37.6 / 39.3 and 43.3 / 39.3.
static int64_t split_max_images(int input_kind) {
  switch (input_kind) {
    case YPDQ_INPUT_F32: return 56;
    case YPDQ_INPUT_U8: return 104;
    default: return 72;
  }
}

cudaError_t hash_occupancy_variant(int input_kind, int dct, int separable, int* ctas_per_sm) {
  return dispatch<OccupancyOf>(input_kind, dct, separable, ctas_per_sm);
}

cudaError_t launch_hash(const HashLaunch& prm, int num_sms, int ctas_per_sm, cudaStream_t s) {
  if (prm.n <= 0) return cudaSuccess;
  HashLaunch p = prm;
  p.neg_zero = -0.0f;
  if (p.dct == 0 && !p.separable && p.n <= split_max_images(p.input_kind)) {
    switch (p.input_kind) {
      case YPDQ_INPUT_F32: return launch_split<float>(p, s);
      case YPDQ_INPUT_U8: return launch_split<uint8_t>(p, s);
      case YPDQ_INPUT_RGB8: return launch_split<rgb8_t>(p, s);
      case YPDQ_INPUT_RGBA8: return launch_split<rgba8_t>(p, s);
      default: return cudaErrorInvalidValue;
    }
  }
  int64_t grid = static_cast<int64_t>(num_sms) * (ctas_per_sm > 0 ? ctas_per_sm : 1);
  if (grid > p.n) grid = p.n;
  return dispatch<LaunchOne>(p.input_kind, p.dct, p.separable, p, grid, s);
}

cudaError_t upload_constants() {
  float d[16 * 127], dt[128 * 16] = {};
  for (int i = 0; i < 16 * 127; ++i) {
    uint32_t b = YPDQ_DCT_F32_BITS[i];
    memcpy(&d[i], &b, 4);
    dt[(i % 127) * 16 + i / 127] = d[i];
  }
  cudaError_t e = cudaMemcpyToSymbol(g_dct, d, sizeof(d));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_dct_t, dt, sizeof(dt));
  for (int kind = 0; kind < 4 && e == cudaSuccess; ++kind)
    for (int dct = 0; dct < 3 && e == cudaSuccess; ++dct)
      for (int sep = 0; sep < 2 && e == cudaSuccess; ++sep) e = dispatch<SetSmemAttr>(kind, dct, sep);
  if (e == cudaSuccess) e = set_split_smem<float>();
  if (e == cudaSuccess) e = set_split_smem<uint8_t>();
  if (e == cudaSuccess) e = set_split_smem<rgb8_t>();
  if (e == cudaSuccess) e = set_split_smem<rgba8_t>();
  return e;
}

cudaError_t launch_dihedrals(const DihedralLaunch& p, cudaStream_t s) {
  if (p.n <= 0) return cudaSuccess;
  const int64_t grid = (p.n + 3) / 4;
  dihedral_kernel<<<static_cast<unsigned>(grid), 128, 0, s>>>(p);
  return cudaGetLastError();
}

}  // namespace ypdq
