// ReferenceKernel<f32> on the GPU (YPDQ_COMPRESS_JAROSZ): yume-pdq's pdqhash-faithful kernel.
//
// jarosz_compress (src/kernel/mod.rs:790-820) filters the whole 512x512 image with
// jarosz_filter_float (src/kernel/ref.rs): two repetitions of a box filter along rows, then
// along columns, with window ceil(512 / 254) = 3. Each line is filtered by a running sum in
// four phases (fill, grow, slide, shrink) with correctly rounded f32 divisions, so every
// output depends on the rounding of the whole prefix of its line; the kernels below replay
// that sum in the same order. The filtered image is sampled at ((2 o + 1) 512) / 254 and
// transformed by the reference kernel's DCT (one sequential accumulator per output,
// src/kernel/mod.rs:711-735).
// Median, packing, quality and dihedrals are the batched dihedral kernel's.
//
// Two ways through the filter, bit for bit the same:
//   * jarosz_image_kernel, one CTA per image with every line's running sum kept on the chip
//     (below): reads the image once and writes the PDQF. 1,500 u8 images 1,434 -> 378 us,
//     456 f32 images 150 us.
//   * for fewer than 32 f32 or RGB images, where one CTA's walk over an image takes longer
//     than short passes with a thread per line (one image 97 against 85 us f32, 106 against 88
//     RGB8; at 32 images 101 against 110, 108 against 111): four launches through two f32
//     planes (X, Y) per image. Each thread keeps the loads of its next 16 or 32 values in
//     registers while it filters the current ones.
//   rows1      : Y = box along rows of the input (BT.601 luma on load for RGB8/RGBA8). A warp
//                owns 32 rows; 32x32 tiles transposed in shared memory keep the global
//                accesses coalesced.
//   cols1      : X = box along columns of Y (a thread owns a column; coalesced by construction)
//   rows2      : Yc = box along rows of X, keeping only the 127 sampled columns
//                (512 x 128 per image)
//   cols2+dct  : box along the columns of Yc, and at each of the 127 sampled rows the first
//                DCT stage takes the sample into its accumulators, in the reference's order;
//                the second DCT stage follows in shared memory.
#include "ypdq_internal.cuh"
#include "ypdq_tables.h"

namespace ypdq {

__device__ float g_dct[16 * 127];  // the f32 DCT matrix D[i][k]
__device__ alignas(16) float g_dct_t[127 * 16];  // and its transpose [k][i]

namespace {

constexpr int kN = 512;
constexpr size_t kPlane = static_cast<size_t>(kN) * kN;

// x / 3 correctly rounded (IEEE round to nearest even) without a division: Markstein's
// correction of the product by the reciprocal (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990).
// q0 = RN(x c) with c = RN(1/3); the remainder r = x - 3 q0 is exact in one FMA, and
// q = RN(q0 + r c). This equals x / 3 for every finite x: tests/test_div3.py compares all
// 2^31 non-negative patterns with IEEE division, and each step is odd in x. For x = +-inf
// the remainder is NaN and q0 (= x) is the quotient; NaN stays NaN.
__device__ __forceinline__ float div3_rn(float x) {
  const float c = 0x1.555556p-2f;  // RN(1/3)
  const float q0 = __fmul_rn(x, c);
  const float r = __fmaf_rn(-q0, 3.0f, x);
  return r == r ? __fmaf_rn(r, c, q0) : q0;
}

// The reference's running-sum box filter of window 3 over one line, one input at a time:
// fill takes in[0]; the value that grow2 / grow3 / slide take as in[ri] yields the output
// for position ri - 1; finish yields position 511. The reference divides by its running
// window count, which is 2 at positions 0 and 511 and 3 everywhere else: x / 2 is exactly
// RN(x * 0.5), and x / 3 is div3_rn. History holds in[ri-1], in[ri-2], in[ri-3].
struct Box3 {
  float sum = 0.0f;
  float h1 = 0.0f, h2 = 0.0f, h3 = 0.0f;
  __device__ __forceinline__ void shift(float v) {
    h3 = h2;
    h2 = h1;
    h1 = v;
  }
  __device__ __forceinline__ void fill(float v) {  // ri = 0 (half window - 1 = 1 value)
    sum = __fadd_rn(sum, v);
    shift(v);
  }
  __device__ __forceinline__ float grow2(float v) {  // ri = 1: position 0, window 2
    sum = __fadd_rn(sum, v);
    shift(v);
    return __fmul_rn(sum, 0.5f);
  }
  __device__ __forceinline__ float grow3(float v) {  // ri = 2: position 1, window 3
    sum = __fadd_rn(sum, v);
    shift(v);
    return div3_rn(sum);
  }
  __device__ __forceinline__ float slide(float v) {  // ri >= 3: position ri - 1, drop in[ri-3]
    sum = __fadd_rn(sum, v);
    sum = __fsub_rn(sum, h3);
    shift(v);
    return div3_rn(sum);
  }
  __device__ __forceinline__ float finish() {  // shrink: position 511 drops in[509] = h3
    sum = __fsub_rn(sum, h3);
    return __fmul_rn(sum, 0.5f);
  }
  // in[ri] for any ri; returns whether an output (for position ri - 1) was produced
  __device__ __forceinline__ bool push(int ri, float v, float& out) {
    if (ri == 0) {
      fill(v);
      return false;
    }
    out = ri == 1 ? grow2(v) : ri == 2 ? grow3(v) : slide(v);
    return true;
  }
};

__device__ __forceinline__ float byte_as_float(uint32_t b) { return static_cast<float>(b); }
__device__ __forceinline__ float luma601(uint32_t r, uint32_t g, uint32_t b) {
  return __fadd_rn(__fadd_rn(__fmul_rn(0.299f, byte_as_float(r)), __fmul_rn(0.587f, byte_as_float(g))),
                   __fmul_rn(0.114f, byte_as_float(b)));
}

constexpr size_t kCompactPlane = static_cast<size_t>(kN) * 128;  // rows2 output per image

__device__ __forceinline__ int sample_at(int o) { return ((2 * o + 1) * kN) / (127 * 2); }

// Four consecutive pixels (from pixel idx, a multiple of 4) of one image as raw words, and
// as f32: the reference's input buffer (u8 cast, or BT.601 luma for RGB8/RGBA8). The f32
// planes between the passes are read with kKind = YPDQ_INPUT_F32.
template <int kKind>
struct Px4;
template <>
struct Px4<YPDQ_INPUT_F32> {
  using Raw = float4;
  static __device__ __forceinline__ Raw load(const uint8_t* img, size_t idx) {
    return *reinterpret_cast<const float4*>(img + 4 * idx);
  }
  static __device__ __forceinline__ float4 cvt(Raw r) { return r; }
};
template <>
struct Px4<YPDQ_INPUT_RGB8> {  // 12 bytes, 4-byte aligned: r0 g0 b0 r1 | g1 b1 r2 g2 | b2 r3 g3 b3
  using Raw = uint3;
  static __device__ __forceinline__ Raw load(const uint8_t* img, size_t idx) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(img + 3 * idx);
    return make_uint3(w[0], w[1], w[2]);
  }
  static __device__ __forceinline__ float4 cvt(Raw r) {
    return make_float4(luma601(r.x & 0xffu, (r.x >> 8) & 0xffu, (r.x >> 16) & 0xffu),
                       luma601(r.x >> 24, r.y & 0xffu, (r.y >> 8) & 0xffu),
                       luma601((r.y >> 16) & 0xffu, r.y >> 24, r.z & 0xffu),
                       luma601((r.z >> 8) & 0xffu, (r.z >> 16) & 0xffu, r.z >> 24));
  }
};
template <>
struct Px4<YPDQ_INPUT_RGBA8> {
  using Raw = uint4;
  static __device__ __forceinline__ Raw load(const uint8_t* img, size_t idx) {
    return *reinterpret_cast<const uint4*>(img + 4 * idx);
  }
  static __device__ __forceinline__ float rgba(uint32_t w) {
    return luma601(w & 0xffu, (w >> 8) & 0xffu, (w >> 16) & 0xffu);
  }
  static __device__ __forceinline__ float4 cvt(Raw r) {
    return make_float4(rgba(r.x), rgba(r.y), rgba(r.z), rgba(r.w));
  }
};

template <int kKind>
__host__ __device__ constexpr size_t bytes_per_px() {
  return kKind == YPDQ_INPUT_U8 ? 1 : kKind == YPDQ_INPUT_RGB8 ? 3 : 4;
}

constexpr int kTileStride = 36;  // floats per tile row: 16-byte rows, conflict-free float4

__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}

// Box along rows: block = 4 warps; warp w of block b owns rows 32 (4 b + w) .. +31 of image
// blockIdx.y, in 16 tiles of 32 columns.
//   * Tile t is loaded with 16-byte accesses (lane l: rows l/8 + 4 i, columns 4 (l%8) .. +3;
//     each warp access covers four whole 128-byte rows) into one of two shared buffers,
//     while the loads of tile t+1 go out into registers.
//   * Lane l filters row l of the tile, four values per vector read. The output for position
//     p is produced by input p + 1, so outputs trail inputs by one: each float4 of outputs
//     (positions 4 g .. 4 g + 3) is written in place once input 4 g + 4 has been read, and
//     the last group of tile t - 1 is completed by the first input of tile t.
//   * Tile t - 1 (complete now) goes out with 16-byte stores; kCompact keeps the sampled
//     columns only: output column sample_at(j) goes to Yc[row][j].
// Images at or past *n_dev (graph replay with fewer images than the capture's bound; image
// blockIdx.y of the chunk is image i0 + blockIdx.y of the call) are skipped.
__device__ __forceinline__ bool past_count(const int64_t* n_dev, int64_t i0, unsigned img) {
  return n_dev && i0 + static_cast<int64_t>(img) >= *n_dev;
}

template <int kKind, bool kCompact>
__global__ void __launch_bounds__(128) rows_kernel(const uint8_t* __restrict__ in,
                                                   float* __restrict__ out,
                                                   const int64_t* n_dev, int64_t i0) {
  using P = Px4<kKind>;
  if (past_count(n_dev, i0, blockIdx.y)) return;
  __shared__ __align__(16) float tiles[4][2][32][kTileStride];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lr = lane >> 3, lc = 4 * (lane & 7);
  const int r0 = 32 * (4 * blockIdx.x + w);
  const uint8_t* img = in + blockIdx.y * kPlane * bytes_per_px<kKind>();
  const size_t base = static_cast<size_t>(r0) * kN;
  float* dst = kCompact ? out + blockIdx.y * kCompactPlane + static_cast<size_t>(r0) * 128
                        : out + blockIdx.y * kPlane + base;
  typename P::Raw pre[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) pre[i] = P::load(img, base + (lr + 4 * i) * kN + lc);
  Box3 box;
  float h0 = 0.0f, h1 = 0.0f, h2 = 0.0f;  // outputs waiting for their group's last one
  int jlo = 0;                              // kCompact: first sampled column not yet stored

  // tile buffer b holds global columns c0 .. c0 + 31 of the warp's rows, all filtered
  auto store_tile = [&](float (*b)[kTileStride], int c0) {
    if constexpr (kCompact) {
      // n <= 8 sample columns fall in a tile (they are 4 or 5 apart); lane l stores sample
      // l % 8 of rows l / 8 + 4 i, so each store covers four rows' 32-byte runs of Yc
      const int jt = jlo + lane;
      const int n = __popc(__ballot_sync(0xffffffffu, jt < 127 && sample_at(jt) < c0 + 32));
      const int j = jlo + (lane & 7);
      const bool mine = (lane & 7) < n;
      const int pos = mine ? sample_at(j) - c0 : 0;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (mine) dst[(lr + 4 * i) * 128 + j] = b[lr + 4 * i][pos];
      jlo += n;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(dst + (lr + 4 * i) * kN + c0 + lc) =
            *reinterpret_cast<const float4*>(&b[lr + 4 * i][lc]);
    }
  };

  for (int t = 0; t < kN / 32; ++t) {
    float (*cur)[kTileStride] = tiles[w][t & 1];
    float (*prv)[kTileStride] = tiles[w][(t & 1) ^ 1];
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(&cur[lr + 4 * i][lc]) = P::cvt(pre[i]);
    __syncwarp();
    if (t + 1 < kN / 32) {
#pragma unroll
      for (int i = 0; i < 8; ++i) pre[i] = P::load(img, base + (lr + 4 * i) * kN + 32 * (t + 1) + lc);
    }
    float* row = cur[lane];
    float4 x = *reinterpret_cast<const float4*>(row);
    if (t == 0) {
      box.fill(x.x);
    } else {
      const float o = box.slide(x.x);
      st4(prv[lane] + 28, h0, h1, h2, o);
    }
    h0 = t == 0 ? box.grow2(x.y) : box.slide(x.y);
    h1 = t == 0 ? box.grow3(x.z) : box.slide(x.z);
    h2 = box.slide(x.w);
#pragma unroll
    for (int g = 1; g < 8; ++g) {
      x = *reinterpret_cast<const float4*>(row + 4 * g);
      const float o = box.slide(x.x);
      st4(row + 4 * (g - 1), h0, h1, h2, o);
      h0 = box.slide(x.y);
      h1 = box.slide(x.z);
      h2 = box.slide(x.w);
    }
    __syncwarp();
    if (t > 0) store_tile(prv, 32 * (t - 1));
    __syncwarp();
  }
  float (*last)[kTileStride] = tiles[w][(kN / 32 - 1) & 1];
  st4(last[lane] + 28, h0, h1, h2, box.finish());
  __syncwarp();
  store_tile(last, kN - 32);
}

// Box along columns of full planes: thread c of block b owns column 128 b + c of image
// blockIdx.y, with the next 16 rows' loads in flight while it filters the current 16.
__global__ void __launch_bounds__(128) cols_kernel(const float* __restrict__ Y,
                                                   float* __restrict__ X,
                                                   const int64_t* n_dev, int64_t i0) {
  if (past_count(n_dev, i0, blockIdx.y)) return;
  const int col = 128 * blockIdx.x + threadIdx.x;
  const float* src = Y + blockIdx.y * kPlane + col;
  float* dst = X + blockIdx.y * kPlane + col;
  Box3 box;
  float cur[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) cur[q] = src[q * kN];
  for (int rb = 0; rb < kN / 16; ++rb) {
    float nxt[16];
    if (rb + 1 < kN / 16) {
#pragma unroll
      for (int q = 0; q < 16; ++q) nxt[q] = src[static_cast<size_t>(16 * (rb + 1) + q) * kN];
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int r = 16 * rb + q;
      float o;
      if (box.push(r, cur[q], o)) dst[static_cast<size_t>(r - 1) * kN] = o;
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) cur[q] = nxt[q];
  }
  dst[static_cast<size_t>(kN - 1) * kN] = box.finish();
}

// Box along the sampled columns of Yc and the reference kernel's DCT (one sequential
// accumulator per output, src/kernel/mod.rs:711-735), one CTA of 128 threads per image.
// Thread j filters sampled column j; at sampled row sample_at(k) its output is B[k][j], which
// enters T[i][j] = sum_k D[i][k] B[k][j] at step k (D column k read as four broadcast
// float4). Then P = T D^T from shared memory, k in order; rows padded to 129 floats keep the
// 16 different D rows of a warp in 16 banks. Thread 127 filters a copy of column 126 so
// that every thread reaches the barrier.
__global__ void __launch_bounds__(128) cols_dct_kernel(const float* __restrict__ Yc,
                                                       float* __restrict__ pdqf,
                                                       float* __restrict__ buf1,
                                                       const int64_t* n_dev, int64_t i0) {
  if (past_count(n_dev, i0, blockIdx.x)) return;  // the whole block: no barrier is split
  __shared__ float4 dk[127][4];  // dk[k][q] = D[4 q .. 4 q + 3][k]
  __shared__ float dj[16][129];  // D[i][k]
  __shared__ float t[16][129];   // T[i][j]
  const int j = threadIdx.x;
  for (int e = j; e < 16 * 127; e += 128) {
    const int i = e / 127, k = e % 127;
    const float d = g_dct[e];
    dj[i][k] = d;
    reinterpret_cast<float*>(&dk[k][i >> 2])[i & 3] = d;
  }
  const bool live = j < 127;
  const float* src = Yc + blockIdx.x * kCompactPlane + (live ? j : 126);
  float acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.0f;
  int k = 0, next_row = sample_at(0);
  Box3 box;
  float cur[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) cur[q] = src[q * 128];
  __syncthreads();  // dk, dj
  for (int rb = 0; rb < kN / 16; ++rb) {
    float nxt[16];
    if (rb + 1 < kN / 16) {
#pragma unroll
      for (int q = 0; q < 16; ++q) nxt[q] = src[(16 * (rb + 1) + q) * 128];
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int r = 16 * rb + q;
      float b;
      if (box.push(r, cur[q], b) && r - 1 == next_row) {  // the same rows for every thread
        if (buf1 && live) buf1[(static_cast<size_t>(blockIdx.x) * 127 + k) * 128 + j] = b;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const float4 d = dk[k][q4];
          acc[4 * q4 + 0] = __fadd_rn(acc[4 * q4 + 0], __fmul_rn(d.x, b));
          acc[4 * q4 + 1] = __fadd_rn(acc[4 * q4 + 1], __fmul_rn(d.y, b));
          acc[4 * q4 + 2] = __fadd_rn(acc[4 * q4 + 2], __fmul_rn(d.z, b));
          acc[4 * q4 + 3] = __fadd_rn(acc[4 * q4 + 3], __fmul_rn(d.w, b));
        }
        ++k;
        next_row = k < 127 ? sample_at(k) : -1;
      }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) cur[q] = nxt[q];
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) t[i][j] = acc[i];
  __syncthreads();
  for (int o = j; o < 256; o += 128) {
    const int i = o >> 4, jj = o & 15;
    float s = 0.0f;
    for (int kk = 0; kk < 127; ++kk) s = __fadd_rn(s, __fmul_rn(t[i][kk], dj[jj][kk]));
    pdqf[static_cast<size_t>(blockIdx.x) * 256 + o] = s;
  }
}

// ---------------------------------------------------------------------- one kernel per image
//
// jarosz_image_kernel: both repetitions, the sampling and the DCT of one image in one CTA,
// without planes in memory. The image is walked in tiles of 32 rows x 64 columns, along the
// rows first. Every line's running sum is kept between the tiles it crosses, so each sum is
// replayed in the reference's order over its whole line. Four warps, each with a part of its
// own, work on consecutive tiles at the same time (one block barrier per step):
//   A  rows1 of tile u: lane = row. u8: the window's sum directly (the running sum of
//      integers is exact, so it is the same number), four columns at a time; other input: the
//      running sum. The raw tile comes by cp.async, one tile ahead;
//   B  cols1 of tile u - 1, in place: lane = two columns, in f32 pairs;
//   C  rows2 of tile u - 2: lane = row; only the sampled columns' outputs are divided and kept;
//   D  cols2 of the 32 (31) samples of tiles u - 4 and u - 3: lane = sample, half of the rows
//      per step; each sampled value enters the lane's 16 DCT accumulators.
// Outputs trail inputs by one position. A value is stored at the slot of the input that
// completed it, so slot g holds the output of position g - 1; slot 0 holds 0, which leaves
// the next running sum unchanged, and the outputs of position 511, which no sampled value
// needs (the last one is 509), are never formed. The sample at position p completes at slot
// p + 2 of the next pass.
//
// A step takes as long as its longest part: ~1,040 clk alone (u8: A 920, C 775, D 660, B 600),
// ~1,300 with three CTAs per SM (shared memory), which keep the issue slots ~64 % busy. A
// running sum is two dependent additions per value, 8 clk, so 64 columns cannot take less
// than ~510. The loads of each part come before its stores: the compiler may not move a
// shared load over a shared store, and a load per quad of values made C take 1,900 clk. All
// four parts by all warps in turn, between block barriers, took 209 us for 608 u8 images
// (187 now) and 160 us for one (79). Four CTAs per SM, with D's sums in registers, made 608
// images 160 us but 1,500 429 us (412) and RGB slower; wider tiles leave two CTAs.
constexpr int kTileR = 32, kTileC = 64;
constexpr int kStrips = kN / kTileC;
constexpr int kTiles = (kN / kTileR) * kStrips;
constexpr int kPitch = kTileC + 4;  // floats per tile row: 16-byte rows, conflict-free float4
template <int kKind>
constexpr int raw_row_bytes() { return kTileC * static_cast<int>(bytes_per_px<kKind>()); }
template <int kKind>
constexpr int raw_pitch() { return raw_row_bytes<kKind>() + 16; }  // an odd number of 16-byte units

// Where D reads the DCT matrix: shared memory if three CTAs per SM fit with it, else global.
template <int kKind>
constexpr bool shared_dct() { return bytes_per_px<kKind>() < 4; }

template <int kKind>
struct ImageSmem {
  alignas(16) float s[3][kTileR][kPitch];
  alignas(16) uint8_t raw[2][kTileR][raw_pitch<kKind>()];
  float q[2][kTileR][33];                      // samples of two tiles
  alignas(16) float4 col[kStrips][2][32];      // B: column sums of a row block's tiles
  alignas(16) float4 sample[4][5][32];         // D: accumulators and sums of each quarter
  alignas(16) float dt[shared_dct<kKind>() ? 127 : 1][16];  // dt[k][i] = D[i][k]
};

__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

// x / 3 in two operations for sums of byte images: RN(x c + RN(x c')) with c = RN(1/3) and
// c' = RN(1/3 - c). x c + x c' is x / 3 to 2^-49, and x / 3 of a 24-bit x is at least 1/6 ulp
// from a rounding boundary, so the result is correctly rounded as long as x c' keeps its
// precision: for |x| >= 2^-120 (tests/test_div3_split.py checks every such float). A byte
// image's sums are 0 or far above that: luma values are multiples of 2^-27, so the first
// pass' sums are too, and each pass' division adds at most 25 bits below that, 2^-102 for the
// fourth. f32 input may hold anything and takes div3_rn.
template <int kKind>
__device__ __forceinline__ float div3(float x) {
  if constexpr (kKind == YPDQ_INPUT_F32) return div3_rn(x);
  else return __fmaf_rn(x, 0x1.555556p-2f, __fmul_rn(x, -0x1.555556p-27f));
}
template <int kKind>
__device__ __forceinline__ float2 div3(float2 x) {
  if constexpr (kKind == YPDQ_INPUT_F32) {
    const float2 q0 = mul2_contractible_rn(x, f2(0x1.555556p-2f));
    const float2 r = fma2_rn(q0, f2(-3.0f), x);
    const float2 q = fma2_rn(r, f2(0x1.555556p-2f), q0);
    return make_float2(r.x == r.x ? q.x : q0.x, r.y == r.y ? q.y : q0.y);
  } else {
    return fma2_rn(x, f2(0x1.555556p-2f), mul2_contractible_rn(x, f2(-0x1.555556p-27f)));
  }
}

// A line's running sum over window 3: one input, sum += v, sum -= the input three before it
// (0 before the line: x - 0 is x). p1, p2, p3: the last three inputs.
template <typename T>
struct Running {
  T sum, p1, p2, p3;
};
__device__ __forceinline__ float advance(float sum, float v, float out) {
  return __fsub_rn(__fadd_rn(sum, v), out);
}
__device__ __forceinline__ float2 advance(float2 sum, float2 v, float2 out) {
  return fma2_rn(out, f2(-1.0f), add2_rn(sum, v));
}
// Four inputs in a row; s[i] = the sum after input i.
template <typename T>
__device__ __forceinline__ void advance4(Running<T>& r, const T (&v)[4], T (&s)[4]) {
  s[0] = advance(r.sum, v[0], r.p1);
  s[1] = advance(s[0], v[1], r.p2);
  s[2] = advance(s[1], v[2], r.p3);
  s[3] = advance(s[2], v[3], v[0]);
  r.sum = s[3];
  r.p1 = v[1];
  r.p2 = v[2];
  r.p3 = v[3];
}

// C: the 64 slots of one row in a tile of the image's quarter JJ (128 columns). Each quad of
// slots completes one sample, at slot JJ of it; only the first quad of quarter 0 completes
// none and that of quarter 1 one at slot 0 (`first`: the tile starts with it).
template <int kKind, int JJ>
__device__ __forceinline__ void keep_samples(const float* row, float* kept, bool first,
                                             Running<float>& line) {
  float4 x[kTileC / 4];
#pragma unroll
  for (int q = 0; q < kTileC / 4; ++q) x[q] = *reinterpret_cast<const float4*>(row + 4 * q);
  float at[kTileC / 4];
#pragma unroll
  for (int q = 0; q < kTileC / 4; ++q) {
    const float v[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
    float s[4];
    advance4(line, v, s);
    at[q] = JJ == 1 && q == 0 && first ? s[0] : s[JJ];
  }
#pragma unroll
  for (int q = 0; q < kTileC / 4; ++q) {
    const float v = div3<kKind>(at[q]);
    if (JJ != 0) kept[q] = v;
    else if (q != 0 || !first) kept[q - 1] = v;
  }
}

// D: sixteen rows of kept samples, lane = sample of a quarter (31 in quarter 0, else 32). The
// quads of rows complete samples as the quads of columns do: quad n the image's row n - 1, at
// slot n / 32 of it; quad 0 none (its value counts 0) and quad 32 at slot 0.
struct Samples {
  Running<float> line;
  float2 acc[8];  // T[2 i], T[2 i + 1] of the lane's sample
};
template <int kKind>
__device__ __forceinline__ void take_samples(const float* kept, const float (*dt)[16], int n0,
                                             float* buf1, float nz, Samples& st) {
  float v[16], at[4];
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = kept[33 * q];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float x[4] = {v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]};
    float s[4];
    advance4(st.line, x, s);
    const int off = n0 + q == 32 ? 0 : n0 >> 5;
    const float lo = off & 1 ? s[1] : s[0], hi = off & 1 ? s[3] : s[2];
    at[q] = off & 2 ? hi : lo;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = max(n0 + q - 1, 0);
    const float b = n0 + q == 0 ? 0.0f : div3<kKind>(at[q]);
    if (buf1 && n0 + q != 0) buf1[k * 128] = b;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 d;
      if constexpr (shared_dct<kKind>()) d = reinterpret_cast<const float4*>(dt[k])[i];
      else d = __ldg(reinterpret_cast<const float4*>(g_dct_t + 16 * k) + i);
      st.acc[2 * i] = add2_rn(st.acc[2 * i], mul2_rn(make_float2(d.x, d.y), f2(b), nz));
      st.acc[2 * i + 1] = add2_rn(st.acc[2 * i + 1], mul2_rn(make_float2(d.z, d.w), f2(b), nz));
    }
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A for u8: sixteen pixels (four words) of one row. `before`: the word left of them (0 at the
// image's edge). Window sums of three in 16-bit halves, then biased floats and thirds.
__device__ __forceinline__ void rows1_u8(const uint4 px, uint32_t& before, float* out, bool edge) {
  const uint32_t words[4] = {px.x, px.y, px.z, px.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = words[i];
    const uint32_t m = __funnelshift_r(before, w, 16);  // columns -2 .. 1 of the word
    before = w;
    const uint32_t mid = ((m >> 8) & 0x00FF00FFu) + (w & 0x00FF00FFu);
    const uint32_t even = (m & 0x00FF00FFu) + mid;  // windows ending at columns 0, 2
    const uint32_t odd = mid + ((w >> 8) & 0x00FF00FFu);  // 1, 3
    float2 a = make_float2(__uint_as_float(__byte_perm(even, 0x4B000000u, 0x7610)),
                           __uint_as_float(__byte_perm(odd, 0x4B000000u, 0x7610)));
    float2 b = make_float2(__uint_as_float(__byte_perm(even, 0x4B000000u, 0x7632)),
                           __uint_as_float(__byte_perm(odd, 0x4B000000u, 0x7632)));
    a = add2_rn(a, f2(-8388608.0f));
    b = add2_rn(b, f2(-8388608.0f));
    const float half = __fmul_rn(a.y, 0.5f);  // position 0: a window of two
    a = div3<YPDQ_INPUT_U8>(a);
    b = div3<YPDQ_INPUT_U8>(b);
    if (i == 0 && edge) a = make_float2(0.0f, half);
    *reinterpret_cast<float4*>(out + 4 * i) = make_float4(a.x, a.y, b.x, b.y);
  }
}

// Where the four parts run, and when the CTAs of an SM start.
//
// A warp's scheduler is its hardware warp number modulo 4; a CTA's warps take consecutive ones
// from a place that differs from CTA to CTA. Part A on one scheduler in all three CTAs makes
// that scheduler the slowest, so the parts are turned by the CTA's place (hw_warp / 4), which
// puts different parts on every scheduler: 456 u8 images 115 us, 1,500 378, 4,000 917 (turned
// by the block index, which the hardware spreads over the SMs in an order of its own: 126, 410,
// 962; the worst turn: 166, 394).
//
// CTAs that share an SM evenly also end together, and the SMs that end first take three of the
// next images while others take none. So in the first of two or three waves the second and
// third CTA start kStaggerNs and twice that later: 912 u8 images 225 us (231 without, 263 by
// block index), 1,216 292 (315, 351), 912 RGB8 289 (306, 343); with more waves the ends drift
// apart by themselves (2,000 images 500 us with, 477 without). With at most one image per SM
// left over, none of this beats the turn by block index: 608 f32 images 246 us staggered, 237
// by block; u8 185 both, 208 without a stagger. (On 152 SMs. The delay is u8's best of 0, 10 and
// 20 us, and the lines go by the number of images launched: a server step that replays a larger
// bucket's graph with fewer keeps that bucket's rule.)
struct Parts {
  bool by_block;           // parts turned by block index
  uint32_t stagger_first;  // this many blocks start staggered
};
constexpr uint32_t kStaggerNs = 10000;

template <int kKind>
__global__ void __launch_bounds__(128, 3)
    jarosz_image_kernel(const uint8_t* __restrict__ in, float* __restrict__ pdqf,
                        float* __restrict__ buf1, const int64_t* n_dev, int64_t i0, float nz, Parts parts) {
  if (past_count(n_dev, i0, blockIdx.x)) return;  // the whole block: no barrier is split
  extern __shared__ __align__(16) uint8_t smem_raw[];
  ImageSmem<kKind>& sm = *reinterpret_cast<ImageSmem<kKind>*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Each scheduler runs another part in each of its CTAs (see Parts).
  __shared__ uint32_t hw_warp;
  if (tid == 0) asm volatile("mov.u32 %0, %%warpid;" : "=r"(hw_warp));
  __syncthreads();
  const uint32_t slot = hw_warp >> 2;
  const int part = (warp + (parts.by_block ? blockIdx.x : hw_warp + slot)) & 3;
  constexpr int kRowBytes = raw_row_bytes<kKind>();
  const uint8_t* img = in + blockIdx.x * kPlane * bytes_per_px<kKind>();
  auto fetch = [&](int t) {  // A: tile t's pixels into raw[t % 2], 16 bytes per lane and step
    constexpr int kUnits = kRowBytes / 16;  // per row
    const uint8_t* src = img + static_cast<size_t>(kTileR * (t / kStrips)) * kN * bytes_per_px<kKind>() +
                         static_cast<size_t>(t % kStrips) * kRowBytes;
#pragma unroll
    for (int e = 0; e < kUnits; ++e) {
      const int unit = 32 * e + lane, row = unit / kUnits, x = unit % kUnits;
      cp_async16(&sm.raw[t & 1][row][16 * x], src + static_cast<size_t>(row) * kN * bytes_per_px<kKind>() + 16 * x);
    }
    cp_async_commit();
  };
  if constexpr (shared_dct<kKind>())
    for (int e = tid; e < 127 * 4; e += 128)
      reinterpret_cast<float4*>(sm.dt[0])[e] = reinterpret_cast<const float4*>(g_dct_t)[e];
  for (int e = tid; e < 4 * 5 * 32; e += 128) (&sm.sample[0][0][0])[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int e = tid; e < kStrips * 2 * 32; e += 128) (&sm.col[0][0][0])[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (part == 1) fetch(0);
  if (tid == 0 && blockIdx.x < parts.stagger_first) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < slot % 3 * kStaggerNs) __nanosleep(500);
  }
  __syncthreads();

  Running<float> line = {};  // A: row sums of rows1; C: of rows2
  uint32_t before = 0;       // A, u8
  Samples st = {};           // D: the quarter at hand

#pragma unroll 1
  for (int u = 0; u < kTiles + 4; ++u) {
    if (part == 1) {
      if (u < kTiles) {  // ---- A
        const int J = u % kStrips;
        cp_async_wait_all();
        __syncwarp();
        if (u + 1 < kTiles) fetch(u + 1);
        const uint8_t* raw = sm.raw[u & 1][lane];
        float* row = sm.s[u % 3][lane];
        if (J == 0) {
          line = {};
          before = 0;
        }
        float first = 0.0f;
        uint4 px[kRowBytes / 16];
#pragma unroll
        for (int e = 0; e < kRowBytes / 16; ++e) px[e] = *reinterpret_cast<const uint4*>(raw + 16 * e);
        // sixteen pixels at a time
#pragma unroll
        for (int g = 0; g < kTileC / 16; ++g) {
          if constexpr (kKind == YPDQ_INPUT_U8) {
            rows1_u8(px[g], before, row + 16 * g, g == 0 && J == 0);
          } else {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(px + g * (kRowBytes / kTileC));
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float v[4], s[4];
              if constexpr (kKind == YPDQ_INPUT_F32) {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = __uint_as_float(w[4 * q + e]);
              } else {
                float2 lo, hi;
                if constexpr (kKind == YPDQ_INPUT_RGB8) {
                  lo = luma01(w[3 * q], w[3 * q + 1], w[3 * q + 2]);
                  hi = luma23(w[3 * q], w[3 * q + 1], w[3 * q + 2]);
                } else {
                  lo = luma_rgba(w[4 * q], w[4 * q + 1]);
                  hi = luma_rgba(w[4 * q + 2], w[4 * q + 3]);
                }
                v[0] = lo.x;
                v[1] = lo.y;
                v[2] = hi.x;
                v[3] = hi.y;
              }
              advance4(line, v, s);
              if (g == 0 && q == 0) first = s[1];
              *reinterpret_cast<float4*>(row + 16 * g + 4 * q) =
                  make_float4(div3<kKind>(s[0]), div3<kKind>(s[1]), div3<kKind>(s[2]), div3<kKind>(s[3]));
            }
          }
        }
        if (kKind != YPDQ_INPUT_U8 && J == 0) {
          row[0] = 0.0f;
          row[1] = __fmul_rn(first, 0.5f);  // position 0: a window of two
        }
      }
    } else if (part == 2) {
      if (u >= 1 && u - 1 < kTiles) {  // ---- B: columns 2 lane, 2 lane + 1
        const int t = u - 1, J = t % kStrips;
        float* at = &sm.s[t % 3][0][2 * lane];
        const float4 c0 = sm.col[J][0][lane], c1 = sm.col[J][1][lane];
        Running<float2> r = {make_float2(c0.x, c0.y), make_float2(c0.z, c0.w),
                             make_float2(c1.x, c1.y), make_float2(c1.z, c1.w)};
        float2 v[kTileR / 4][4], first = f2(0.0f);
#pragma unroll
        for (int q = 0; q < kTileR; ++q) v[q / 4][q % 4] = *reinterpret_cast<const float2*>(at + q * kPitch);
#pragma unroll
        for (int q = 0; q < kTileR / 4; ++q) {
          float2 s[4];
          advance4(r, v[q], s);
          if (q == 0) first = s[1];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            *reinterpret_cast<float2*>(at + (4 * q + e) * kPitch) = div3<kKind>(s[e]);
        }
        if (t < kStrips) {
          *reinterpret_cast<float2*>(at) = f2(0.0f);
          *reinterpret_cast<float2*>(at + kPitch) =
              make_float2(__fmul_rn(first.x, 0.5f), __fmul_rn(first.y, 0.5f));
        }
        sm.col[J][0][lane] = make_float4(r.sum.x, r.sum.y, r.p1.x, r.p1.y);
        sm.col[J][1][lane] = make_float4(r.p2.x, r.p2.y, r.p3.x, r.p3.y);
      }
    } else if (part == 0) {
      if (u >= 2 && u - 2 < kTiles) {  // ---- C: row `lane`
        const int t = u - 2, J = t % kStrips;
        const float* row = sm.s[t % 3][lane];
        float* kept = &sm.q[(t >> 1) & 1][lane][16 * (J & 1)];
        if (J == 0) line = {};
        switch (J >> 1) {
          case 0: keep_samples<kKind, 0>(row, kept, J == 0, line); break;
          case 1: keep_samples<kKind, 1>(row, kept, J == 2, line); break;
          case 2: keep_samples<kKind, 2>(row, kept, false, line); break;
          default: keep_samples<kKind, 3>(row, kept, false, line); break;
        }
      }
    } else if (u >= 4) {  // ---- D
      const int pair = (u - 4) >> 1, half = u & 1, I = pair >> 2;
      const int JJ = pair & 3, o = (JJ == 0 ? 0 : 32 * JJ - 1) + lane;
      if (half == 0) {
        const float4 r = sm.sample[JJ][4][lane];
        st.line = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 a = sm.sample[JJ][i][lane];
          st.acc[2 * i] = make_float2(a.x, a.y);
          st.acc[2 * i + 1] = make_float2(a.z, a.w);
        }
      }
      take_samples<kKind>(&sm.q[pair & 1][16 * half][lane], sm.dt, (kTileR / 4) * I + 4 * half,
                          buf1 && (JJ != 0 || lane < 31)
                              ? buf1 + static_cast<size_t>(blockIdx.x) * 127 * 128 + o
                              : nullptr,
                          nz, st);
      if (half == 1) {
        sm.sample[JJ][4][lane] = make_float4(st.line.sum, st.line.p1, st.line.p2, st.line.p3);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          sm.sample[JJ][i][lane] =
              make_float4(st.acc[2 * i].x, st.acc[2 * i].y, st.acc[2 * i + 1].x, st.acc[2 * i + 1].y);
      }
    }
    __syncthreads();
  }
  // second DCT stage, k in order: T[i][j] over the tile buffers
  float* T = sm.s[0][0];
  if (tid < 127) {
    const int JJ = (tid + 1) >> 5, l = tid - (JJ == 0 ? 0 : 32 * JJ - 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 a = sm.sample[JJ][i][l];
      T[(4 * i + 0) * 129 + tid] = a.x;
      T[(4 * i + 1) * 129 + tid] = a.y;
      T[(4 * i + 2) * 129 + tid] = a.z;
      T[(4 * i + 3) * 129 + tid] = a.w;
    }
  }
  __syncthreads();
  {
    const int i = tid >> 3, jj = 2 * (tid & 7);
    float2 sum = f2(0.0f);
#pragma unroll 8
    for (int kk = 0; kk < 127; ++kk)
      sum = add2_rn(sum, mul2_rn(__ldg(reinterpret_cast<const float2*>(g_dct_t + 16 * kk + jj)), f2(T[i * 129 + kk]), nz));
    *reinterpret_cast<float2*>(pdqf + static_cast<size_t>(blockIdx.x) * 256 + 16 * i + jj) = sum;
  }
}

template <int kKind>
cudaError_t image_init() {
  return cudaFuncSetAttribute(jarosz_image_kernel<kKind>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(sizeof(ImageSmem<kKind>)));
}
template <int kKind>
void launch_image(const uint8_t* in, float* pdqf, float* buf1, unsigned n, const int64_t* n_dev,
                  int64_t i0, int num_sms, cudaStream_t s) {
  const unsigned sms = static_cast<unsigned>(num_sms), wave = 3 * sms;
  const Parts parts = {n > wave && n <= wave + sms,
                       n > wave + sms && n <= 3 * wave ? wave : 0u};
  jarosz_image_kernel<kKind><<<n, 128, sizeof(ImageSmem<kKind>), s>>>(in, pdqf, buf1, n_dev, i0, -0.0f,
                                                                       parts);
}

template <int kKind>
void launch_rows1(const uint8_t* in, float* Y, dim3 grid, const int64_t* n_dev, int64_t i0,
                  cudaStream_t s) {
  rows_kernel<kKind, false><<<grid, 128, 0, s>>>(in, Y, n_dev, i0);
}

}  // namespace

cudaError_t jarosz_init() {
  float d[16 * 127], dt[127 * 16];
  for (int i = 0; i < 16 * 127; ++i) {
    const uint32_t b = YPDQ_DCT_F32_BITS[i];
    memcpy(&d[i], &b, 4);
    dt[(i % 127) * 16 + i / 127] = d[i];
  }
  cudaError_t e = cudaMemcpyToSymbol(g_dct, d, sizeof(d));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_dct_t, dt, sizeof(dt));
  if (e == cudaSuccess) e = image_init<YPDQ_INPUT_F32>();
  if (e == cudaSuccess) e = image_init<YPDQ_INPUT_U8>();
  if (e == cudaSuccess) e = image_init<YPDQ_INPUT_RGB8>();
  if (e == cudaSuccess) e = image_init<YPDQ_INPUT_RGBA8>();
  return e;
}

// Images from which jarosz_image_kernel runs (the header comment has both sides' times).
static int64_t image_kernel_from(int input_kind) { return input_kind == YPDQ_INPUT_U8 ? 1 : 32; }
static int64_t plane_images(int64_t chunk) { return chunk < 31 ? chunk : 31; }

// The planes of as many images as the planes version may get, and every image's PDQF.
size_t jarosz_scratch_bytes(int64_t chunk) {
  return static_cast<size_t>(plane_images(chunk)) * 2 * kPlane * sizeof(float) +
         static_cast<size_t>(chunk) * 256 * sizeof(float);
}

cudaError_t launch_hash_jarosz(const HashLaunch& p, void* scratch, int64_t chunk, int num_sms,
                               cudaStream_t s) {
  if (p.n <= 0) return cudaSuccess;
  static const size_t kBytesPerPixel[4] = {4, 1, 3, 4};
  if (p.input_kind < 0 || p.input_kind > 3) return cudaErrorInvalidValue;
  float* X = static_cast<float*>(scratch);
  float* Y = X + plane_images(chunk) * kPlane;
  float* P = Y + plane_images(chunk) * kPlane;
  for (int64_t i0 = 0; i0 < p.n; i0 += chunk) {
    const int64_t m = p.n - i0 < chunk ? p.n - i0 : chunk;
    const uint8_t* in =
        static_cast<const uint8_t*>(p.images) + static_cast<size_t>(i0) * kPlane * kBytesPerPixel[p.input_kind];
    float* buf1 = p.buf1 ? p.buf1 + static_cast<size_t>(i0) * 127 * 128 : nullptr;
    const int64_t* nd = p.n_dev;
    if (p.n >= image_kernel_from(p.input_kind)) {
      const unsigned g = static_cast<unsigned>(m);
      switch (p.input_kind) {
        case YPDQ_INPUT_F32: launch_image<YPDQ_INPUT_F32>(in, P, buf1, g, nd, i0, num_sms, s); break;
        case YPDQ_INPUT_U8: launch_image<YPDQ_INPUT_U8>(in, P, buf1, g, nd, i0, num_sms, s); break;
        case YPDQ_INPUT_RGB8: launch_image<YPDQ_INPUT_RGB8>(in, P, buf1, g, nd, i0, num_sms, s); break;
        default: launch_image<YPDQ_INPUT_RGBA8>(in, P, buf1, g, nd, i0, num_sms, s); break;
      }
    } else {
      const dim3 grid(kN / 128, static_cast<unsigned>(m));
      switch (p.input_kind) {
        case YPDQ_INPUT_F32: launch_rows1<YPDQ_INPUT_F32>(in, Y, grid, nd, i0, s); break;
        case YPDQ_INPUT_RGB8: launch_rows1<YPDQ_INPUT_RGB8>(in, Y, grid, nd, i0, s); break;
        default: launch_rows1<YPDQ_INPUT_RGBA8>(in, Y, grid, nd, i0, s); break;
      }
      cols_kernel<<<grid, 128, 0, s>>>(Y, X, nd, i0);
      rows_kernel<YPDQ_INPUT_F32, true><<<grid, 128, 0, s>>>(reinterpret_cast<const uint8_t*>(X), Y,
                                                             nd, i0);
      cols_dct_kernel<<<static_cast<unsigned>(m), 128, 0, s>>>(Y, P, buf1, nd, i0);
    }
    DihedralLaunch d{};
    d.pdqf = P;
    d.thr_in = nullptr;
    d.n = m;
    d.row_mask = p.row_mask;
    d.col_mask = p.col_mask;
    d.hashes = p.hashes ? p.hashes + static_cast<size_t>(i0) * 256 : nullptr;
    d.quality = p.quality ? p.quality + static_cast<size_t>(i0) * 8 : nullptr;
    d.thresholds = p.thresholds ? p.thresholds + static_cast<size_t>(i0) * 8 : nullptr;
    // the dihedral kernel writes all 8 slots; with one slot requested, copy slot 0 instead
    d.pdqf_out = (p.pdqf && p.pdqf_slots == 8) ? p.pdqf + static_cast<size_t>(i0) * 8 * 256 : nullptr;
    cudaError_t e = launch_dihedrals(d, s);
    if (e == cudaSuccess && p.pdqf && p.pdqf_slots != 8)
      e = cudaMemcpyAsync(p.pdqf + static_cast<size_t>(i0) * 256, P, static_cast<size_t>(m) * 1024,
                          cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

}  // namespace ypdq
