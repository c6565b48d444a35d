// Exact linear Hamming scan of 256-bit rows against a batch of 256-bit queries, with
// warp-aggregated hit compaction.
//
// Reference: CpuMatcher::find (scalar, src/matching/mod.rs:336-362) reports every
// (row, needle) with popcount(row ^ needle) <= threshold; the WGSL matcher
// (src/matching/vulkan.rs:98-147) evaluates the same predicate, one row per thread.
// Both kernels here return the full hit set with distances. They differ only in how
// they compute distances:
//   SIMT   one row per thread, eight 32-bit XOR + POPC per (row, query);
//   B1MMA  16 rows x 8 queries per warp instruction with the binary tensor-core MMA
//          (mma.sync m16n8k256 .b1 .xor.popc), whose accumulator is the distance.
#include <cstddef>

#include "ypdq_internal.cuh"

namespace ypdq {

constexpr int kScanThreads = 256;
constexpr uint32_t kMaxSmemQueries = 2048;  // queries per launch (64 KiB of shared memory)

// Hit emission from lanes that found a hit in the same converged step: one atomic per warp.
__device__ __forceinline__ void emit_hits_ballot(bool pred, uint64_t row, uint32_t query,
                                                 uint32_t dist, ypdq_hit* hits, uint64_t cap,
                                                 unsigned long long* count) {
  const uint32_t ballot = __ballot_sync(0xffffffffu, pred);
  if (ballot == 0) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(ballot) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(count, static_cast<unsigned long long>(__popc(ballot)));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (pred) {
    const uint64_t pos = base + __popc(ballot & lanemask_lt());
    if (pos < cap) {
      ypdq_hit h;
      h.index = row;
      h.query = query;
      h.distance = dist;
      hits[pos] = h;
    }
  }
}

__device__ __forceinline__ uint4 ld_stream(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// One 32-byte row. kWide: in one load, which fetches a warp's 32 sectors once; as two loads of 16
// bytes each fetches all of them, and without a place in L1 they come from L2 twice. 8 queries:
// 100 M rows 536 -> 523 us, 10 M 64.2 -> 62.4 (bound by popcounts and logic by then; 1 query,
// bound by HBM, 50.2 both).
template <bool kWide>
__device__ __forceinline__ void ld_row(const uint4* p, uint4& a, uint4& b) {
  if constexpr (kWide) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z),
                   "=r"(b.w)
                 : "l"(p));
  } else {
    a = ld_stream(p);
    b = ld_stream(p + 1);
  }
}

// ------------------------------------------------------------------- SIMT

// Popcounts of several words through carry-save adders: a full adder turns three words into
// a sum word and a carry word with x0 + x1 + x2 = s + 2 c bit by bit, so fewer popcounts
// (the scarce pipe) are needed; the adders are single three-input logic ops.
__device__ __forceinline__ void csa(uint32_t a, uint32_t b, uint32_t c, uint32_t& s, uint32_t& cy) {
  s = a ^ b ^ c;
  cy = (a & b) | (c & (a ^ b));
}
__device__ __forceinline__ uint32_t popc3(uint32_t x0, uint32_t x1, uint32_t x2) {
  uint32_t s, c;
  csa(x0, x1, x2, s, c);
  return __popc(s) + 2 * __popc(c);
}
__device__ __forceinline__ uint32_t popc5(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                          uint32_t x4) {
  uint32_t s1, c1, s2, c2;
  csa(x0, x1, x2, s1, c1);
  csa(s1, x3, x4, s2, c2);
  return __popc(s2) + 2 * (__popc(c1) + __popc(c2));
}
__device__ __forceinline__ uint32_t popc8(uint4 x, uint4 y) {
  uint32_t s1, c1, s2, c2, s3, c3, t1, f1;
  csa(x.x, x.y, x.z, s1, c1);
  csa(x.w, y.x, y.y, s2, c2);
  csa(s1, s2, y.z, s3, c3);
  const uint32_t ones = s3 ^ y.w, c4 = s3 & y.w;
  csa(c1, c2, c3, t1, f1);
  const uint32_t twos = t1 ^ c4, f2 = t1 & c4;
  const uint32_t fours = f1 ^ f2, eights = f1 & f2;
  return __popc(ones) + 2 * __popc(twos) + 4 * __popc(fours) + 8 * __popc(eights);
}

// kPrefix words (3, 5 or 8 of 8) are counted first. Their popcount is a lower bound of the
// distance, so once it exceeds t in every lane of the warp no pair of this query can be a
// hit; rows that pass are finished exactly, so hits and distances do not change. The host
// picks kPrefix by threshold: a random row is 48 +- 5 bits from a query in 96 bits and
// 80 +- 6 in 160, so for t <= 34 (or <= 62) nearly every warp stops after 2 (or 3) of the
// 8 popcounts that a plain count needs; above that the whole row is counted with 4.
// Rows per thread and resident blocks per SM of each variant (register-bound). With a
// prefix bound a thread takes two rows, so each query's shared load, vote and loop step
// serve both; the full count (4 popcounts per pair) runs out of registers first and keeps
// one row at higher occupancy. The grid-stride grid is exactly this many blocks per SM so
// that no block starts late.
__host__ __device__ constexpr int simt_rows(int prefix) { return prefix == 8 ? 1 : 2; }
__host__ __device__ constexpr int simt_blocks_per_sm(int prefix) { return prefix == 8 ? 6 : 4; }

template <int kPrefix, bool kWide>
__global__ void __launch_bounds__(kScanThreads, simt_blocks_per_sm(kPrefix))
    scan_simt_kernel(const uint4* __restrict__ rows, uint64_t n_rows,
                     const uint4* __restrict__ queries, uint32_t nq, uint32_t q_base,
                     uint32_t t, ypdq_hit* hits, uint64_t cap, unsigned long long* count,
                     const uint32_t* nq_dev) {
  constexpr int R = simt_rows(kPrefix);
  extern __shared__ uint4 sq[];
  if (nq_dev) nq = min(*nq_dev, nq);
  for (uint32_t i = threadIdx.x; i < 2 * nq; i += blockDim.x) sq[i] = queries[i];
  __syncthreads();
  // A warp owns 32 R consecutive rows per step, lane l rows l + 32 i. Every lane of a warp
  // runs the same number of steps so the ballots stay converged.
  const int lane = threadIdx.x & 31;
  const uint64_t stride = static_cast<uint64_t>(R) * gridDim.x * blockDim.x;
  const uint64_t warp_first =
      ((static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * (32 * R);
  // the next step's rows are in flight while the queries run over the current ones
  uint4 na[R], nb[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const uint64_t r = warp_first + lane + 32 * i;
    na[i] = nb[i] = make_uint4(0, 0, 0, 0);
    if (r < n_rows) ld_row<kWide>(rows + 2 * r, na[i], nb[i]);
  }
  for (uint64_t base = warp_first; base < n_rows; base += stride) {
    uint64_t r[R];
    bool v[R];
    uint4 a[R], b[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      r[i] = base + lane + 32 * i;
      v[i] = r[i] < n_rows;
      a[i] = na[i];
      b[i] = nb[i];
      if (r[i] + stride < n_rows) ld_row<kWide>(rows + 2 * (r[i] + stride), na[i], nb[i]);
    }
#pragma unroll(R == 1 ? 4 : 2)
    for (uint32_t q = 0; q < nq; ++q) {
      const uint4 qa = sq[2 * q];
      uint32_t d[R];
      if constexpr (kPrefix == 3) {
        bool near = false;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          d[i] = popc3(a[i].x ^ qa.x, a[i].y ^ qa.y, a[i].z ^ qa.z);
          near |= d[i] <= t;
        }
        if (!__any_sync(0xffffffffu, near)) continue;
        const uint4 qb = sq[2 * q + 1];
#pragma unroll
        for (int i = 0; i < R; ++i)
          d[i] += popc5(a[i].w ^ qa.w, b[i].x ^ qb.x, b[i].y ^ qb.y, b[i].z ^ qb.z, b[i].w ^ qb.w);
      } else if constexpr (kPrefix == 5) {
        const uint4 qb = sq[2 * q + 1];
        bool near = false;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          d[i] = popc5(a[i].x ^ qa.x, a[i].y ^ qa.y, a[i].z ^ qa.z, a[i].w ^ qa.w, b[i].x ^ qb.x);
          near |= d[i] <= t;
        }
        if (!__any_sync(0xffffffffu, near)) continue;
#pragma unroll
        for (int i = 0; i < R; ++i) d[i] += popc3(b[i].y ^ qb.y, b[i].z ^ qb.z, b[i].w ^ qb.w);
      } else {
        const uint4 qb = sq[2 * q + 1];
#pragma unroll
        for (int i = 0; i < R; ++i)
          d[i] = popc8(make_uint4(a[i].x ^ qa.x, a[i].y ^ qa.y, a[i].z ^ qa.z, a[i].w ^ qa.w),
                       make_uint4(b[i].x ^ qb.x, b[i].y ^ qb.y, b[i].z ^ qb.z, b[i].w ^ qb.w));
      }
      bool h[R], any_hit = false;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        h[i] = v[i] && d[i] <= t;
        any_hit |= h[i];
      }
      if (__any_sync(0xffffffffu, any_hit)) {
#pragma unroll
        for (int i = 0; i < R; ++i) emit_hits_ballot(h[i], r[i], q_base + q, d[i], hits, cap, count);
      }
    }
  }
}

// ------------------------------------------------------------------ B1 MMA

__device__ __forceinline__ void mma_b1_xor_popc(uint32_t a0, uint32_t a1, uint32_t a2,
                                                uint32_t a3, uint32_t b0, uint32_t b1,
                                                uint32_t& d0, uint32_t& d1, uint32_t& d2,
                                                uint32_t& d3) {
  asm volatile(
      "mma.sync.aligned.m16n8k256.row.col.s32.b1.b1.s32.xor.popc "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d0), "=r"(d1), "=r"(d2), "=r"(d3)
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

// Fragment layout of m16n8k256 (.b1): lane = 4*g + tq holds
//   a0: row g,   k = 32 tq .. 32 tq + 31      a2: row g,   k = 128 + 32 tq ..
//   a1: row g+8, k = 32 tq ..                 a3: row g+8, k = 128 + 32 tq ..
//   b0: col (query) g, k = 32 tq ..           b1: col g,   k = 128 + 32 tq ..
//   d0,d1: row g, queries 2tq, 2tq+1          d2,d3: row g+8, queries 2tq, 2tq+1
// The distance is a popcount over all k, so any fixed word <-> k-slot assignment works as
// long as rows and queries use the same one: k-slot tq <-> word 2tq, slot 128+32tq <->
// word 2tq+1. Each lane then loads one 8-byte pair of words per row.
__global__ void __launch_bounds__(kScanThreads)
    scan_b1_kernel(const uint2* __restrict__ rows, uint64_t n_rows,
                   const uint2* __restrict__ queries, uint32_t nq, uint32_t q_base, uint32_t t,
                   ypdq_hit* hits, uint64_t cap, unsigned long long* count) {
  extern __shared__ uint2 sfrag[];  // [chunks][32 lanes]
  const uint32_t chunks = (nq + 7) / 8;
  for (uint32_t idx = threadIdx.x; idx < chunks * 32; idx += blockDim.x) {
    const uint32_t c = idx >> 5, l = idx & 31, g = l >> 2, tq = l & 3;
    const uint32_t qi = 8 * c + g;
    sfrag[idx] = qi < nq ? queries[qi * 4 + tq] : make_uint2(0, 0);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint32_t g = lane >> 2, tq = lane & 3;
  const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const uint64_t n_warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
  const uint64_t n_tiles = (n_rows + 15) / 16;
  for (uint64_t tile = warp; tile < n_tiles; tile += n_warps) {
    const uint64_t r0 = tile * 16 + g, r1 = r0 + 8;
    uint2 A0 = make_uint2(0, 0), A1 = make_uint2(0, 0);
    if (r0 < n_rows) A0 = rows[r0 * 4 + tq];
    if (r1 < n_rows) A1 = rows[r1 * 4 + tq];
    for (uint32_t c = 0; c < chunks; ++c) {
      const uint2 B = sfrag[c * 32 + lane];
      uint32_t d0, d1, d2, d3;
      mma_b1_xor_popc(A0.x, A1.x, A0.y, A1.y, B.x, B.y, d0, d1, d2, d3);
      const uint32_t q0 = 8 * c + 2 * tq, q1 = q0 + 1;
      const bool h0 = r0 < n_rows && q0 < nq && d0 <= t;
      const bool h1 = r0 < n_rows && q1 < nq && d1 <= t;
      const bool h2 = r1 < n_rows && q0 < nq && d2 <= t;
      const bool h3 = r1 < n_rows && q1 < nq && d3 <= t;
      if (__any_sync(0xffffffffu, h0 | h1 | h2 | h3)) {
        emit_hits_ballot(h0, r0, q_base + q0, d0, hits, cap, count);
        emit_hits_ballot(h1, r0, q_base + q1, d1, hits, cap, count);
        emit_hits_ballot(h2, r1, q_base + q0, d2, hits, cap, count);
        emit_hits_ballot(h3, r1, q_base + q1, d3, hits, cap, count);
      }
    }
  }
}

cudaError_t sort_init();

cudaError_t scan_init() {
  const int smem = static_cast<int>(kMaxSmemQueries * 32);
  cudaError_t e = cudaSuccess;
  for (const void* f : {reinterpret_cast<const void*>(scan_simt_kernel<3, true>),
                        reinterpret_cast<const void*>(scan_simt_kernel<5, true>),
                        reinterpret_cast<const void*>(scan_simt_kernel<8, true>),
                        reinterpret_cast<const void*>(scan_simt_kernel<3, false>),
                        reinterpret_cast<const void*>(scan_simt_kernel<5, false>),
                        reinterpret_cast<const void*>(scan_simt_kernel<8, false>)}) {
    e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  e = cudaFuncSetAttribute(scan_b1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  e = sort_init();
  if (e != cudaSuccess) return e;
  return scan_tc_init();
}

// SIMT is HBM-bound up to a few queries; past that it is bound by its popcount and logic
// pipes, at 2, 3 or 4 popcounts per pair depending on the threshold (the prefix bound in
// scan_simt_kernel). A narrow tensor-core pass (at most 128 queries) costs about the time of
// 9 SIMT queries at t <= 34 (10M rows without hits: 0.070-0.078 ms; SIMT 0.062 ms for 8
// queries, 0.069 for 9, 0.074 for 10), 6 at t = 35..36 (the SIMT side at three popcounts: 0.068
// ms for 6, 0.077 for 7), 24 at t <= 62 and 12 above (the FP8 passes, neither side pruned as far).
// A tensor-core launch takes ~8 us on any database (query expansion, a pipeline to fill), SIMT
// ~6, and a few hits cost the tensor cores 2-5 us more, SIMT next to nothing, so small databases
// move the line. SIMT against tensor cores, t <= 34, 16 queries: 8.2 / 8.4 us at 200,000 rows,
// 10.5 / 10.3 at 500,000, 16.6 / 14.2 at 1 M, 20.8 / 16.6 at 1.5 M where nothing hits; 15.4 / 17.6
// at 1 M and 21.1 / 21.3 at 1.5 M with some tens of hits; 16.9 / 22.9 and 23.1 / 29.2 with 0.1 % of
// the rows. 32 queries 8.5 / 8.1 at 100,000 rows and 10.3 / 8.4 at 200,000 without a hit, 9.1 / 11.3
// and 11.1 / 12.6 with 0.1 %. At t = 35..36 16 queries 8.5 / 8.9 at 200,000 rows (9.2 / 12.9 with
// hits), 8 queries 21.6 / 21.6 at 2 M (22.1 / 35.5).
// Whole lookups from host queries to sorted hits, with 0.1 %: 16 queries against 100,000 rows
// 57.8 -> 47.7 us, 1.5 M 81.5 -> 71.5; at t = 36 8 queries against 2 M rows 94 -> 81. Where nothing
// hits, the line costs up to 4 us of 31-44: 16 queries 31.1 / 30.6 at 200,000 rows, 43.8 / 40.6 at
// 1.5 M, 32 queries 34.8 / 30.7 at 200,000.
int auto_scan_algo(uint32_t n_queries, uint32_t threshold, uint64_t n_rows) {
  uint32_t simt_max = threshold <= 34 ? 9 : threshold <= 36 ? 6 : threshold <= 62 ? 24 : 12;
  if (threshold <= 34 && n_rows <= 1500000) simt_max = n_rows <= 200000 ? 32 : 16;
  if (threshold > 34 && threshold <= 36 && n_rows <= 2000000) simt_max = n_rows <= 200000 ? 16 : 8;
  return n_queries <= simt_max ? YPDQ_SCAN_SIMT : YPDQ_SCAN_TC;
}

cudaError_t launch_scan(const ScanLaunch& p, int algo, int num_sms, cudaStream_t s) {
  cudaError_t e = p.append ? cudaSuccess : cudaMemsetAsync(p.count, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess || p.n_rows == 0 || p.n_queries == 0) return e;
  if (algo == YPDQ_SCAN_AUTO) algo = auto_scan_algo(p.n_queries, p.threshold, p.n_rows);
  if (algo == YPDQ_SCAN_TC) return launch_scan_tc(p, num_sms, s);
  if (algo == YPDQ_SCAN_TC_FP4) {
    ScanLaunch q = p;
    if (p.threshold <= 36) q.pair_n = kPairFp4N;  // FP4, three queries per column
    return launch_scan_tc(q, num_sms, s);
  }
  if (algo == YPDQ_SCAN_TC_FP8) {
    // FP8 at t <= 36 too: query pairs past 256 queries, else one pass of up to 256
    ScanLaunch q = p;
    if (p.threshold <= 36) {
      if (p.n_queries > 256)
        q.pair_n = 256;
      else
        q.n_tile = (p.n_queries + 63u) & ~63u;
    }
    return launch_scan_tc(q, num_sms, s);
  }
  // a device-side query count needs the whole query set in one launch
  if (p.nq_dev && (algo != YPDQ_SCAN_SIMT || p.n_queries > kMaxSmemQueries))
    return cudaErrorInvalidValue;
  for (uint32_t q0 = 0; q0 < p.n_queries; q0 += kMaxSmemQueries) {
    const uint32_t nq = (p.n_queries - q0) < kMaxSmemQueries ? (p.n_queries - q0) : kMaxSmemQueries;
    const uint8_t* qptr = p.queries + static_cast<size_t>(q0) * 32;
    if (algo == YPDQ_SCAN_B1MMA) {
      const uint64_t tiles = (p.n_rows + 15) / 16;
      uint64_t blocks = (tiles + (kScanThreads / 32) - 1) / (kScanThreads / 32);
      const uint64_t cap_blocks = static_cast<uint64_t>(num_sms) * 8;
      if (blocks > cap_blocks) blocks = cap_blocks;
      const size_t smem = static_cast<size_t>((nq + 7) / 8) * 32 * sizeof(uint2);
      scan_b1_kernel<<<static_cast<unsigned>(blocks), kScanThreads, smem, s>>>(
          reinterpret_cast<const uint2*>(p.rows), p.n_rows, reinterpret_cast<const uint2*>(qptr),
          nq, p.query_base + q0, p.threshold, p.hits, p.capacity, p.count);
    } else {
      const size_t smem = static_cast<size_t>(nq) * 32;
      const int prefix = p.threshold <= 34 ? 3 : p.threshold <= 62 ? 5 : 8;
      // 32-byte loads want rows on 32-byte boundaries
      const bool wide = reinterpret_cast<uintptr_t>(p.rows) % 32 == 0;
      auto kern = prefix == 3   ? (wide ? scan_simt_kernel<3, true> : scan_simt_kernel<3, false>)
                  : prefix == 5 ? (wide ? scan_simt_kernel<5, true> : scan_simt_kernel<5, false>)
                                : (wide ? scan_simt_kernel<8, true> : scan_simt_kernel<8, false>);
      // blocks per SM: registers allow simt_blocks_per_sm; the queries' shared memory (plus
      // the 1 KiB the runtime reserves per block, of 228 KiB per SM) may allow fewer
      const uint64_t fit = (228u << 10) / (smem + 1024);
      const uint64_t bps = static_cast<uint64_t>(simt_blocks_per_sm(prefix));
      const uint64_t rows_per_block = static_cast<uint64_t>(kScanThreads) * simt_rows(prefix);
      uint64_t blocks = (p.n_rows + rows_per_block - 1) / rows_per_block;
      const uint64_t cap_blocks = static_cast<uint64_t>(num_sms) * (fit < bps ? fit : bps);
      if (blocks > cap_blocks) blocks = cap_blocks;
      kern<<<static_cast<unsigned>(blocks), kScanThreads, smem, s>>>(
          reinterpret_cast<const uint4*>(p.rows), p.n_rows, reinterpret_cast<const uint4*>(qptr),
          nq, p.query_base + q0, p.threshold, p.hits, p.capacity, p.count, p.nq_dev);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------- hit sorting
//
// By (index, query), the scalar matcher's visit order, through a second buffer: few hits by
// counting for each the hits before it; more by sorting tiles on the chip and merging these
// runs, all at once while they are few, else in passes that merge them in pairs.

// A hit as two words: the index, and query | distance << 32.
struct Hit2 {
  uint64_t k, v;
};
static_assert(sizeof(Hit2) == sizeof(ypdq_hit) && offsetof(ypdq_hit, query) == 8 &&
                  offsetof(ypdq_hit, distance) == 12,
              "a hit is its index and query | distance << 32");
__device__ __forceinline__ bool less2(const Hit2& a, const Hit2& b) {
  return a.k < b.k || (a.k == b.k && static_cast<uint32_t>(a.v) < static_cast<uint32_t>(b.v));
}
__device__ __forceinline__ Hit2 load_hit(const ypdq_hit* h, uint64_t i) {  // 8-byte aligned
  const uint64_t* p = reinterpret_cast<const uint64_t*>(h + i);
  return {p[0], p[1]};
}
__device__ __forceinline__ void store_hit(ypdq_hit* h, uint64_t i, const Hit2& x) {
  uint64_t* p = reinterpret_cast<uint64_t*>(h + i);
  p[0] = x.k;
  p[1] = x.v;
}

// Whether the hit with keys y (index; query, then position) comes before one with k and s.
__device__ __forceinline__ uint32_t is_before(uint64_t yk, uint64_t ys, uint64_t k, uint64_t s) {
  return yk < k || (yk == k && ys < s) ? 1u : 0u;
}

// Rank of each hit among all n (of equal ones the first first), and the hit to its place.
// Block: 32 hits, one per lane; its warps share the comparisons with all n, every lane of a
// warp with the same hit at a time (a broadcast load from cache; 32 hits at a time through
// shared memory with two hits per lane was slower, 70 against 45 us for 8,192). Quadratic, but
// one launch over the whole chip.
constexpr int kRankWarps = 16;
__global__ void __launch_bounds__(32 * kRankWarps)
    rank_hits_kernel(const ypdq_hit* __restrict__ in, ypdq_hit* __restrict__ out, uint32_t n) {
  __shared__ uint32_t before[32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = 32 * blockIdx.x + lane;
  if (warp == 0) before[lane] = 0;
  __syncthreads();
  const Hit2 x = load_hit(in, min(i, n - 1));
  const uint64_t xs = (x.v << 32) | i;
  const uint32_t each = (n + kRankWarps - 1) / kRankWarps, first = warp * each;
  const uint32_t end = min(first + each, n);
  uint32_t c = 0;
#pragma unroll 8
  for (uint32_t j = first; j < end; ++j) {
    const Hit2 y = load_hit(in, j);
    c += is_before(y.k, (y.v << 32) | j, x.k, xs);
  }
  atomicAdd(&before[lane], c);
  __syncthreads();
  if (warp == 0 && i < n) store_hit(out, before[lane], x);
}

// Tile blockIdx.x of 256 hits sorted by ranks: each thread counts the hits of the tile before
// its own (of equal ones the first first). in may be out.
constexpr int kRankTile = 256;
__global__ void __launch_bounds__(kRankTile)
    rank_tiles_kernel(const ypdq_hit* in, ypdq_hit* out, uint64_t n) {
  __shared__ ulonglong2 all[kRankTile];
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kRankTile;
  const uint32_t i = threadIdx.x;
  const uint32_t m = static_cast<uint32_t>(n - base < kRankTile ? n - base : kRankTile);
  Hit2 x{};
  if (i < m) {
    x = load_hit(in, base + i);
    all[i] = make_ulonglong2(x.k, (x.v << 32) | i);
  }
  __syncthreads();
  if (i >= m) return;
  const uint64_t xs = (x.v << 32) | i;
  uint32_t c = 0;
#pragma unroll 8
  for (uint32_t j = 0; j < m; ++j) {
    const ulonglong2 y = all[j];
    c += is_before(y.x, y.y, x.k, xs);
  }
  store_hit(out, base + c, x);
}

// Up to 512 hits in place by one cluster of 8 CTAs: each keeps all hits in shared memory and
// ranks 64 of them, eight warps to the same 32 hits; nobody writes before all have read.
constexpr int kClusterSort = 512, kClusterSortCtas = 8, kClusterSortEach = 64;
__global__ void __cluster_dims__(kClusterSortCtas, 1, 1) __launch_bounds__(512)
    rank_cluster_kernel(ypdq_hit* h, uint32_t n) {
  __shared__ ulonglong2 all[kClusterSort];
  __shared__ uint32_t before[kClusterSortEach];
  const uint32_t tid = threadIdx.x, own = tid % kClusterSortEach, part = tid / kClusterSortEach;
  const uint32_t i = kClusterSortEach * blockIdx.x + own;
  if (tid < n) {
    const Hit2 y = load_hit(h, tid);
    all[tid] = make_ulonglong2(y.k, (y.v << 32) | tid);
  }
  const Hit2 x = load_hit(h, min(i, n - 1));
  if (tid < kClusterSortEach) before[tid] = 0;
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  const uint64_t xs = (x.v << 32) | i;
  constexpr uint32_t kParts = 512 / kClusterSortEach;
  const uint32_t each = (n + kParts - 1) / kParts, first = min(part * each, n), end = min(first + each, n);
  uint32_t c = 0;
#pragma unroll 8
  for (uint32_t j = first; j < end; ++j) {
    const ulonglong2 y = all[j];
    c += is_before(y.x, y.y, x.k, xs);
  }
  atomicAdd(&before[own], c);
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (tid < kClusterSortEach && i < n) store_hit(h, before[tid], x);
}

// All runs of w = 2^k sorted hits merged in one pass: a hit's place is its place in its run
// plus, for every other run, how many of that run's hits come before it (of equal hits those
// of the earlier run), k + 1 steps of a binary search. Block: 32 consecutive hits, one per
// lane, whose searches stay close to each other; its warps share the runs.
constexpr int kPlaceWarps = 16;
__global__ void __launch_bounds__(32 * kPlaceWarps)
    place_runs_kernel(const ypdq_hit* __restrict__ in, ypdq_hit* __restrict__ out, uint64_t n,
                      uint32_t w) {
  __shared__ uint32_t before[32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t i = 32ull * blockIdx.x + lane;
  if (warp == 0) before[lane] = 0;
  __syncthreads();
  const Hit2 x = load_hit(in, i < n ? i : n - 1);
  const uint32_t runs = static_cast<uint32_t>((n + w - 1) / w);
  const uint32_t own = static_cast<uint32_t>(32ull * blockIdx.x / w);
  uint32_t c = 0;
#pragma unroll 4
  for (uint32_t r = warp; r < runs; r += kPlaceWarps) {
    const ypdq_hit* run = in + static_cast<uint64_t>(r) * w;
    const uint64_t left = n - static_cast<uint64_t>(r) * w;
    const uint32_t m = left < w ? static_cast<uint32_t>(left) : w;
    uint32_t at = 0;
    if (r == own) {
      at = static_cast<uint32_t>(i - static_cast<uint64_t>(own) * w);
    } else {
      for (uint32_t h = w; h > 0; h >>= 1) {
        if (at + h > m) continue;
        const Hit2 y = load_hit(run, at + h - 1);
        if (r < own ? !less2(x, y) : less2(y, x)) at += h;
      }
    }
    c += at;
  }
  atomicAdd(&before[lane], c);
  __syncthreads();
  if (warp == 0 && i < n) store_hit(out, before[lane], x);
}

constexpr int kSortItems = 8;  // hits per thread
// Place of item i in a shared tile: one hit of padding after every eight, so that threads
// reading eight consecutive hits each (16 bytes at a time) meet different banks.
__host__ __device__ constexpr int padded(int i) { return i + i / kSortItems; }
__device__ __forceinline__ ulonglong2& slot_of(Hit2* sh, int i) {
  return *reinterpret_cast<ulonglong2*>(sh + padded(i));
}
__device__ __forceinline__ Hit2 get(Hit2* sh, int i) {
  const ulonglong2 x = slot_of(sh, i);
  return {x.x, x.y};
}
__device__ __forceinline__ void put(Hit2* sh, int i, const Hit2& h) {
  slot_of(sh, i) = make_ulonglong2(h.k, h.v);
}

// The kSortItems outputs from position d on of merging sh[a .. a + na) and sh[b .. b + nb)
// (each sorted; equal hits from the first run first) into out. Items past the end are whatever
// lies there: the caller drops them.
__device__ __forceinline__ void merge_items(Hit2* sh, int a, int na, int b, int nb, int d,
                                            Hit2 (&out)[kSortItems]) {
  int lo = d > nb ? d - nb : 0, hi = d < na ? d : na;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (!less2(get(sh, b + d - 1 - mid), get(sh, a + mid))) lo = mid + 1;
    else hi = mid;
  }
  int i = lo, j = d - lo;
  // the item a run offers next; past its end (or of an empty run) any item of the tile
  const auto of_a = [&](int at) { return get(sh, na > 0 ? a + min(at, na - 1) : b); };
  const auto of_b = [&](int at) { return get(sh, nb > 0 ? b + min(at, nb - 1) : a); };
  Hit2 x = of_a(i), y = of_b(j);
#pragma unroll
  for (int q = 0; q < kSortItems; ++q) {
    const bool first = j >= nb || (i < na && !less2(y, x));
    out[q] = first ? x : y;
    i += first ? 1 : 0;
    j += first ? 0 : 1;
    const Hit2 z = first ? of_a(i) : of_b(j);
    if (first) x = z;
    else y = z;
  }
}

// Tile blockIdx.x of kThreads * 8 hits: eight sorted in each thread's registers, then merged
// in pairs of runs through shared memory. Positions past n hold +infinity.
template <int kThreads>
__global__ void __launch_bounds__(kThreads) sort_tiles_kernel(const ypdq_hit* in, ypdq_hit* out,
                                                              uint64_t n) {
  constexpr int kTile = kThreads * kSortItems;
  extern __shared__ __align__(16) uint8_t sort_smem[];
  Hit2* sh = reinterpret_cast<Hit2*>(sort_smem);
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kTile;
  const int count = static_cast<int>(n - base < kTile ? n - base : kTile);
  const int tid = threadIdx.x;
#pragma unroll
  for (int q = 0; q < kSortItems; ++q) {
    const int i = q * kThreads + tid;
    put(sh, i, i < count ? load_hit(in, base + i) : Hit2{~0ull, ~0ull});
  }
  __syncthreads();
  Hit2 x[kSortItems];
#pragma unroll
  for (int q = 0; q < kSortItems; ++q) x[q] = get(sh, tid * kSortItems + q);
  // odd-even transposition: 8 rounds sort 8 items
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
#pragma unroll
    for (int q = r & 1; q + 1 < kSortItems; q += 2)
      if (less2(x[q + 1], x[q])) {
        const Hit2 t = x[q];
        x[q] = x[q + 1];
        x[q + 1] = t;
      }
#pragma unroll
  for (int q = 0; q < kSortItems; ++q) put(sh, tid * kSortItems + q, x[q]);
  __syncthreads();
  for (int w = kSortItems; w < count; w <<= 1) {
    const int at = tid * kSortItems, first = at / (2 * w) * (2 * w);
    merge_items(sh, first, w, first + w, w, at - first, x);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kSortItems; ++q) put(sh, at + q, x[q]);
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < kSortItems; ++q) {
    const int i = q * kThreads + tid;
    if (i < count) store_hit(out, base + i, get(sh, i));
  }
}

// How many of the first d outputs of merging runs a (na hits) and b (nb) come from a: the
// merge path's crossing of diagonal d, by one warp with 32 probes at a time.
__device__ __forceinline__ uint64_t merge_path_warp(const ypdq_hit* a, uint64_t na,
                                                    const ypdq_hit* b, uint64_t nb, uint64_t d,
                                                    int lane) {
  uint64_t lo = d > nb ? d - nb : 0, hi = d < na ? d : na;
  while (lo < hi) {
    const uint64_t span = hi - lo;
    const uint64_t mid = span <= 32 ? lo + lane : lo + span * (lane + 1) / 33;
    const bool right = mid < hi && !less2(load_hit(b, d - 1 - mid), load_hit(a, mid));
    const int c = __popc(__ballot_sync(0xffffffffu, right));  // true for a prefix of the lanes
    if (span <= 32) return lo + c;
    const uint64_t next_lo = c > 0 ? __shfl_sync(0xffffffffu, mid, c > 0 ? c - 1 : 0) + 1 : lo;
    const uint64_t next_hi = c < 32 ? __shfl_sync(0xffffffffu, mid, c < 32 ? c : 31) : hi;
    lo = next_lo;
    hi = next_hi;
  }
  return lo;
}

// One pass: runs of w hits (a multiple of the block's 2,048 outputs) merged in pairs.
constexpr int kMergeThreads = 256;
constexpr int kMergeTile = kMergeThreads * kSortItems;
__global__ void __launch_bounds__(kMergeThreads)
    merge_runs_kernel(const ypdq_hit* in, ypdq_hit* out, uint64_t n, uint64_t w) {
  __shared__ __align__(16) Hit2 sh[padded(kMergeTile)];
  __shared__ uint64_t cut[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint64_t o = static_cast<uint64_t>(blockIdx.x) * kMergeTile;
  const uint64_t first = o / (2 * w) * (2 * w);
  const uint64_t na = n - first < w ? n - first : w;
  const uint64_t nb = n - first - na < w ? n - first - na : w;
  const ypdq_hit* a = in + first;
  const ypdq_hit* b = a + na;
  const uint64_t d0 = o - first, d1 = d0 + kMergeTile < na + nb ? d0 + kMergeTile : na + nb;
  if (warp < 2) {
    const uint64_t c = merge_path_warp(a, na, b, nb, warp == 0 ? d0 : d1, lane);
    if (lane == 0) cut[warp] = c;
  }
  __syncthreads();
  const uint64_t a0 = cut[0], b0 = d0 - a0;
  const int ca = static_cast<int>(cut[1] - a0), count = static_cast<int>(d1 - d0);
#pragma unroll
  for (int q = 0; q < kSortItems; ++q) {
    const int i = q * kMergeThreads + tid;
    if (i < count) put(sh, i, i < ca ? load_hit(a, a0 + i) : load_hit(b, b0 + (i - ca)));
  }
  __syncthreads();
  Hit2 x[kSortItems];
  const int at = tid * kSortItems;
  if (at < count) merge_items(sh, 0, ca, ca, count - ca, at, x);
  __syncthreads();
  if (at < count)
#pragma unroll
    for (int q = 0; q < kSortItems; ++q) put(sh, at + q, x[q]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kSortItems; ++q) {
    const int i = q * kMergeThreads + tid;
    if (i < count) store_hit(out, o + i, get(sh, i));
  }
}

// The bitonic sort in place. Order by (index, query): the scalar matcher's visit order.
__device__ __forceinline__ bool hit_less(const ypdq_hit& a, const ypdq_hit& b) {
  return a.index < b.index || (a.index == b.index && a.query < b.query);
}

// One compare-exchange step of a bitonic sort in the "flip" form: every comparison puts
// the smaller hit at the lower index, so the virtual +infinity padding past n (up to the
// next power of two) never has to move and is never stored.
__global__ void bitonic_step_kernel(ypdq_hit* h, uint64_t n, uint64_t k, uint64_t j, int flip) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t l;
  if (flip) {
    if (i & (k >> 1)) return;
    l = i ^ (k - 1);
  } else {
    if (i & j) return;
    l = i ^ j;
  }
  if (l >= n) return;  // partner is padding: the real element is already the smaller
  const ypdq_hit a = h[i], b = h[l];
  if (hit_less(b, a)) {
    h[i] = b;
    h[l] = a;
  }
}

// The steps of the same sort whose partners lie inside one 2,048-hit block, done in shared
// memory in one launch. full != 0: every stage k = 2 .. k_last (<= 2,048), each its flip
// step and then j = k/4 .. 1. full == 0: the steps j = 1,024 .. 1 of stage k_last (> 2,048),
// whose wider steps ran as global launches. Positions past n hold a +infinity hit, which
// compares above every real one exactly as the global kernel's skipped padding does.
constexpr int kSortBlock = 2048;
__global__ void __launch_bounds__(kSortBlock / 2)
    bitonic_block_kernel(ypdq_hit* h, uint64_t n, uint64_t k_last, int full) {
  __shared__ ypdq_hit sh[kSortBlock];
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kSortBlock;
  const int t = threadIdx.x;
  ypdq_hit inf;
  inf.index = ~0ull;
  inf.query = ~0u;
  inf.distance = ~0u;
  for (int x = t; x < kSortBlock; x += kSortBlock / 2)
    sh[x] = base + x < n ? h[base + x] : inf;
  __syncthreads();
  auto step = [&](uint32_t j, bool flip, uint32_t k) {
    // thread t owns the pair whose lower position has bit j clear
    const uint32_t i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
    const uint32_t l = flip ? (i ^ (k - 1)) : (i | j);
    const ypdq_hit a = sh[i], b = sh[l];
    if (hit_less(b, a)) {
      sh[i] = b;
      sh[l] = a;
    }
    __syncthreads();
  };
  if (full) {
    for (uint32_t k = 2; k <= k_last; k <<= 1) {
      step(k >> 1, true, k);
      for (uint32_t j = k >> 2; j > 0; j >>= 1) step(j, false, k);
    }
  } else {
    for (uint32_t j = kSortBlock / 2; j > 0; j >>= 1) step(j, false, 0);
  }
  for (int x = t; x < kSortBlock; x += kSortBlock / 2)
    if (base + x < n) h[base + x] = sh[x];
}

static cudaError_t launch_sort_in_place(ypdq_hit* hits, uint64_t n, cudaStream_t s) {
  uint64_t padded = 1;
  while (padded < n) padded <<= 1;
  const unsigned threads = 256;
  const unsigned blocks = static_cast<unsigned>((n + threads - 1) / threads);
  const unsigned sblocks = static_cast<unsigned>((n + kSortBlock - 1) / kSortBlock);
  const uint64_t first = padded < static_cast<uint64_t>(kSortBlock) ? padded : kSortBlock;
  bitonic_block_kernel<<<sblocks, kSortBlock / 2, 0, s>>>(hits, n, first, 1);
  for (uint64_t k = 2 * kSortBlock; k <= padded; k <<= 1) {
    bitonic_step_kernel<<<blocks, threads, 0, s>>>(hits, n, k, k >> 1, 1);
    for (uint64_t j = k >> 2; j >= static_cast<uint64_t>(kSortBlock); j >>= 1)
      bitonic_step_kernel<<<blocks, threads, 0, s>>>(hits, n, k, j, 0);
    bitonic_block_kernel<<<sblocks, kSortBlock / 2, 0, s>>>(hits, n, k, 0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

constexpr int kTileThreads = 512;
constexpr size_t kSortSmem = sizeof(Hit2) * padded(kTileThreads * kSortItems);

cudaError_t sort_init() {
  return cudaFuncSetAttribute(sort_tiles_kernel<kTileThreads>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(kSortSmem));
}

// Up to 256 hits: one block, in place. Up to 512 one cluster, in place too: 11.2 us for 512 hits,
// event-timed with the launches, against 16.5 with rank_hits, a second buffer and a copy back; a
// whole lookup with 500 hits 58.2 -> 52.7 us. (Up to 1,024 hits, 128 a CTA, it took 16.9 for 1,000
// and lookups with 700 to 1,000 hits got 1-3 us longer.) Past that (us):
//                     1,000  2,000  4,096  8,192  10,000  16,000  20,000  30,000  50,000  100,000
//   rank_hits          18.6   20.8   30.0   44.7    67
//   tiles 256, place   23.0   23.2   22.9   24.8    26.9    33.5    45.8    59.9   122.8
//   tiles 1,024, place 30.6   33.9   33.3   33.7    33.8    35.9    39.5    43.0    64.1    145
//   tiles 4,096, place 35.9   40.1   43.3   47.8    47.4    47.1    49.3    51.0    56.0     83
//   tiles 4,096, pairs                              59.3    60.5    69.8    70.6    80.2     90
// Placing costs hits x runs x log(run), which the pairs' passes overtake between 100,000 and
// 150,000 hits (125 against 100 us). The bitonic sort that did all of this before, in place
// with every step wider than 2,048 hits a launch of its own, took 23 us for 100 hits (now 11),
// 39 for 1,000, 85 for 8,192, 107 for 10,000, 200 for 100,000 and 751 for 1.02 M (184); it
// stays for a stream under capture and where the second buffer cannot be had. For the pairs,
// tiles of 2,048 and 8,192 hits take 190 and 177 us for 1.02 M, but 8,192 longer below it.
constexpr uint64_t kRankMax = 2560, kPlaceMax256 = 16384, kPlaceMax1024 = 32768, kPlaceMax = 98304;

cudaError_t launch_sort_hits(ypdq_hit* hits, uint64_t n, cudaMemPool_t pool, cudaStream_t s) {
  if (n < 2) return cudaSuccess;
  if (n <= kRankTile) {
    rank_tiles_kernel<<<1, kRankTile, 0, s>>>(hits, hits, n);
    return cudaGetLastError();
  }
  if (n <= kClusterSort) {
    rank_cluster_kernel<<<kClusterSortCtas, 512, 0, s>>>(hits, static_cast<uint32_t>(n));
    return cudaGetLastError();
  }
  // (Under capture the buffer would become allocation nodes of the graph, which then can be
  // neither cloned nor a child graph nor instantiated twice.)
  void* second = nullptr;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (!pool || cudaStreamIsCapturing(s, &capture) != cudaSuccess ||
      capture != cudaStreamCaptureStatusNone ||
      cudaMallocFromPoolAsync(&second, n * sizeof(ypdq_hit), pool, s) != cudaSuccess) {
    cudaGetLastError();
    return launch_sort_in_place(hits, n, s);
  }
  ypdq_hit* const other = static_cast<ypdq_hit*>(second);
  cudaError_t e = cudaSuccess;
  constexpr uint64_t kTile = kTileThreads * kSortItems;
  const auto blocks = [n](uint64_t each) { return static_cast<unsigned>((n + each - 1) / each); };
  const auto place = [&](uint32_t w) {
    place_runs_kernel<<<blocks(32), 32 * kPlaceWarps, 0, s>>>(other, hits, n, w);
  };
  if (n <= kRankMax) {
    rank_hits_kernel<<<blocks(32), 32 * kRankWarps, 0, s>>>(hits, other, static_cast<uint32_t>(n));
    e = cudaMemcpyAsync(hits, other, n * sizeof(ypdq_hit), cudaMemcpyDeviceToDevice, s);
  } else if (n <= kPlaceMax256) {
    rank_tiles_kernel<<<blocks(kRankTile), kRankTile, 0, s>>>(hits, other, n);
    place(kRankTile);
  } else if (n <= kPlaceMax1024) {
    sort_tiles_kernel<128><<<blocks(1024), 128, sizeof(Hit2) * padded(1024), s>>>(hits, other, n);
    place(1024);
  } else if (n <= kPlaceMax) {
    sort_tiles_kernel<kTileThreads><<<blocks(kTile), kTileThreads, kSortSmem, s>>>(hits, other, n);
    place(kTile);
  } else {
    // the tiles go where an even number of passes from there ends in `hits`
    int passes = 0;
    for (uint64_t w = kTile; w < n; w <<= 1) ++passes;
    ypdq_hit* from = passes % 2 ? other : hits;
    ypdq_hit* to = passes % 2 ? hits : other;
    sort_tiles_kernel<kTileThreads><<<blocks(kTile), kTileThreads, kSortSmem, s>>>(hits, from, n);
    for (uint64_t w = kTile; w < n; w <<= 1) {
      merge_runs_kernel<<<blocks(kMergeTile), kMergeThreads, 0, s>>>(from, to, n, w);
      ypdq_hit* t = from;
      from = to;
      to = t;
    }
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  const cudaError_t f = cudaFreeAsync(second, s);
  return e != cudaSuccess ? e : f;
}

}  // namespace ypdq
