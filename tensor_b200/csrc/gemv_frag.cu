// Decode GEMV with the activations in registers: out[m, n] = x[m, k] . dequant(w[n, k])^T for all four formats, every
// activation type, every K a format allows (up to 32768) and every alignment of the weight rows.
//
// Replaces the reference's `gemv_packed` (benchmarks/kernels/showcase/kernels.py:116-119; fp32 weights x fp32
// activations, benchmarks/kernels/showcase/benchmark.py:468-470).
//
// Regime: HBM-bound as long as an SM spends fewer than about 100 (4-bit) to 190 (Q8_0) clocks on 16 x 256 weights.
// A warp owns one 256-weight slice of K for its whole life and walks over tiles of 16 weight rows:
//
//  * its slice of the activations is the B operand of mma.sync.m16n8k16 (batch on the columns) and stays in registers
//    as fp16 fragments, so that nothing but raw weight bytes passes through shared memory in the loop;
//  * it copies its own weight bytes with 16-byte asynchronous copies, several tiles ahead, without a producer warp or
//    a barrier; the skew of a row against the 16-byte granules is the same in every tile (16 rows are a multiple of 16
//    bytes apart), so rows of any 2-byte alignment cost one funnel shift a word;
//  * weights become EXACT fp16 integers: Q4_K's 6-bit scale times its nibble (at most 945) by one HFMA2 for two
//    weights, so the block scale d is applied once per 256 weights and the minimums are one more MMA against the group
//    sums (kept as two fp16 parts); the other formats' centred integers, with d (and Q6_K's 8-bit scale, whose product
//    with the quant would not fit 11 bits) applied to the fp32 accumulators of a scale group;
//  * bf16 activations are multiplied by one power of two per (row, slice) and then fit fp16 exactly down to 2^-29 of the
//    slice's largest value (smaller ones are off by up to 2^-40 of it; fp16 ones, for Q4_K, by one that keeps them
//    exact); fp32 ones are split into three fp16 parts on three columns, exactly down to 2^-15 of the largest value and
//    to 2^-40 of it below.
//
// The warps of a CTA cover up to 4096 of K; a longer K is spread over the CTAs of a cluster, which add their sums through
// distributed shared memory.  All sums are added in K order: no scratch, no atomics, the same bits on every launch.
//
// What bounds it is instruction issue: 600 (Q4_K, batch 8) to 830 (Q6_K, batch 4) warp instructions per 16 x 256 weights,
// half of the issue slots used by the four warps a scheduler that 128 registers allow, DRAM at a fifth of its rate.  Measured (us, this kernel | the one before; graph replay over weights larger
// than the L2): Q6_K 4096 x 12288 at batch 4 / 16 19.1 | 39.7 and 26.2 | 46.5 (tensor memory), Q8_0 12288 x 4096 18.5 | 72.3
// and 23.6 | 228, Q4_0 13.6 | 60.9 and 18.5 | 178 (SIMT), Q4_K 24576 x 4096 20.9 | 24.5 and 28.3 | 41.2 (gemv_mma.cu).
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace tb200 {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kRows = 16;       // weight rows of a tile (MMA M)
constexpr int kMaxSplits = 8;   // CTAs of a cluster along K
constexpr int kBarrierBytes = 1024;
constexpr int kColPitch = 20;   // floats between the columns of a partial tile (16 rows; conflict-free stores)

// Bytes of 256 weights, the row pitch of a stage (an odd number of 16-byte granules: eight rows hit eight bank groups),
// stages a warp, buffers of partial tiles, and how 32 lanes share the granules of a tile: kLanes lanes x kPer granules a row, 32 / kLanes rows at a time.
template <int FMT> struct Cfg;
template <> struct Cfg<kQ4_K> { static constexpr int kBytes = 144, kPitch = 144, kStages = 4, kReds = 3, kLanes = 9, kPer = 1; };
template <> struct Cfg<kQ6_K> { static constexpr int kBytes = 210, kPitch = 240, kStages = 3, kReds = 2, kLanes = 14, kPer = 1; };
template <> struct Cfg<kQ8_0> { static constexpr int kBytes = 272, kPitch = 304, kStages = 2, kReds = 3, kLanes = 6, kPer = 3; };
template <> struct Cfg<kQ4_0> { static constexpr int kBytes = 144, kPitch = 176, kStages = 4, kReds = 2, kLanes = 10, kPer = 1; };

struct FragArgs {
  const void* x;
  const uint8_t* w;
  const uint8_t* w2;   // rows [n1, n) of a grouped launch, as if its row 0 were row n1 of one matrix
  float* out;
  float* out2;         // its columns
  long long out_ld, row_bytes, w_bytes, w2_bytes;
  int m, n, n1, k;
  int row_tiles, nsb;
  int fast1, fast2;    // tiles [0, fast1) and [n1 / 16, fast2): every copy of whole granules stays inside the weight
  int warps_per_row;   // warps of a CTA along K
  int streams;         // row tiles a CTA works on at once
  int splits;          // CTAs of a cluster along K
  int iters;           // tiles of a stream
  int phase;           // splits > 1: tiles between two exchanges
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void sts32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float lds_half(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(mask), "r"(bits));
  return d;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// 4 bytes at any 2-byte aligned shared address; `shift` is 16 where it is not 4-byte aligned
__device__ __forceinline__ uint32_t lds32_half(uint32_t aligned, uint32_t shift) {
  return __funnelshift_r(lds32(aligned), lds32(aligned + 4), shift);
}
// The constants of the logic ops live in registers: with two immediates the compiler makes two instructions of one.
__device__ __forceinline__ uint32_t pinned(uint32_t v) {
  uint32_t r;
  asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

constexpr uint32_t kMagic = 0x64006400u;  // fp16 1024, twice: 0x6400 | q is 1024 + q
constexpr uint32_t half2_const(unsigned short h) { return (uint32_t)h << 16 | h; }
constexpr uint32_t kMinus1024 = half2_const(0xE400), kMinus1032 = half2_const(0xE408), kMinus1056 = half2_const(0xE420),
                   kMinus1152 = half2_const(0xE480), kMinus72 = half2_const(0xD480), kMinus64 = half2_const(0xD400),
                   kSixteenth = half2_const(0x2C00);

// Which four neighbouring elements of the slice lane tig feeds into k-step s (as (0, 2) and (1, 3)).
template <int FMT>
__device__ __forceinline__ int element(int s, int tig) {
  if constexpr (FMT == kQ4_K) return 64 * tig + 32 * (s >> 3) + 4 * (s & 7);  // low nibbles, then high ones
  else return 16 * s + 4 * tig;
}

template <int NT>
struct Frag {
  uint32_t b[16][NT][2];
  uint32_t bm[NT][2];  // Q4_K: group sums / 64 as high and low fp16 parts
  float u[NT][2];      // factors that undo the scaling of columns 2 tig and 2 tig + 1
  bool non_finite;     // Q4_K: some activation of the warp's slice is an infinity or a NaN
};

__device__ __forceinline__ float scale_for(uint32_t exponent) {  // largest magnitude -> [2^14, 2^15)
  int sh = 141 - (int)exponent;
  sh = sh > 126 ? 126 : (sh < -126 ? -126 : sh);
  return __uint_as_float((uint32_t)(sh + 127) << 23);
}

// Columns of the MMA: the batch row itself, or three columns a row (the fp16 parts of fp32 activations).  `spare`: a
// stage of this warp that holds no weights yet.
template <int FMT, int XT, int NT>
__device__ __forceinline__ void load_fragments(Frag<NT>& f, const FragArgs& a, int sb, bool live, int gid, int tig, uint32_t spare) {
  constexpr int kParts = XT == kF32 ? 3 : 1;
  const int rest = a.k - sb * 256;  // elements of the slice that exist
  f.non_finite = false;
  if constexpr (XT != kF32) {
    // Whole rows of the slice (512 bytes, a warp's 16-byte loads) go through shared memory, four at a time, and come
    // back in fragment order: loaded in that order from global memory, an instruction would touch a line per lane.
    // Q4_K lanes read 16-byte granule 8 tig + j, kept at 8 tig + (j ^ tig); with these pitches the lanes of a phase do
    // not share banks.
    constexpr uint32_t kPitch = FMT == kQ4_K ? 576 : 544;
    const int lane = 4 * gid + tig;
    uint4 raw[8 * NT];
#pragma unroll
    for (int row = 0; row < 8 * NT; ++row) {
      raw[row] = make_uint4(0, 0, 0, 0);
      if (live && row < a.m && 8 * lane < rest)
        raw[row] = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.x) + (long long)row * a.k + sb * 256 + 8 * lane);
    }
    const uint32_t to = FMT == kQ4_K ? 16u * (uint32_t)((lane & ~7) | ((lane ^ (lane >> 3)) & 7)) : 16u * (uint32_t)lane;
#pragma unroll
    for (int q = 0; q < 2 * NT; ++q) {
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 4; ++r) ptx::sts128(spare + (uint32_t)r * kPitch + to, raw[4 * q + r]);
      __syncwarp();
      if ((gid >> 2) == (q & 1)) {
        const uint32_t from = spare + (uint32_t)(gid & 3) * kPitch;
        if constexpr (FMT == kQ4_K) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint4 v = ptx::lds128(from + 16u * (uint32_t)(8 * tig + (j ^ tig)));
            const int s = 8 * (j >> 2) + 2 * (j & 3);
            f.b[s][q >> 1][0] = v.x;
            f.b[s][q >> 1][1] = v.y;
            f.b[s + 1][q >> 1][0] = v.z;
            f.b[s + 1][q >> 1][1] = v.w;
          }
        } else {
#pragma unroll
          for (int s = 0; s < 16; ++s) {
            const uint2 v = ptx::lds64(from + (uint32_t)(32 * s + 8 * tig));
            f.b[s][q >> 1][0] = v.x;
            f.b[s][q >> 1][1] = v.y;
          }
        }
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    float scale = 1.f;
    if constexpr (XT == kF32) {
      const int col = 8 * t + gid, row = col / kParts, part = col - kParts * row;
      const bool ok = live && row < a.m;
      const float* x = static_cast<const float*>(a.x) + (long long)row * a.k + sb * 256;
      uint32_t mx = 0;
#pragma unroll
      for (int s = 0; s < 16; ++s) {
        const int e = element<FMT>(s, tig);
        if (ok && e < rest) {
          const uint4 v = *reinterpret_cast<const uint4*>(x + e);
          const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t mag = q[i] & 0x7FFFFFFFu;
            if (mag < 0x7F800000u) mx = max(mx, mag);
            else f.non_finite = true;
          }
        }
      }
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      if (mx >> 23) scale = scale_for(mx >> 23);
#pragma unroll
      for (int s = 0; s < 16; ++s) {
        const int e = element<FMT>(s, tig);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (ok && e < rest) v = *reinterpret_cast<const uint4*>(x + e);
        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
        float p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // parts of a value that is not finite: itself, then zeros
          const float r = __uint_as_float(q[i]) * scale;
          const bool finite = (q[i] & 0x7F800000u) != 0x7F800000u;
          const float r1 = finite ? r - __half2float(__float2half_rn(r)) : 0.f;
          const float mid = __half2float(__float2half_rn(r1));
          p[i] = part == 0 ? r : (part == 1 ? r1 : r1 - mid);
        }
        f.b[s][t][0] = pack_f16(p[0], p[2]);
        f.b[s][t][1] = pack_f16(p[1], p[3]);
      }
    } else {
#pragma unroll
      for (int s = 0; s < 16; ++s) {
        const uint32_t lo = f.b[s][t][0], hi = f.b[s][t][1];
        f.b[s][t][0] = __byte_perm(lo, hi, 0x5410);
        f.b[s][t][1] = __byte_perm(lo, hi, 0x7632);
      }
      // fp16 values are MMA operands as they are; only Q4_K scales them, because its group sums become fp16 parts below:
      // unscaled, the low part of a sum / 64 falls under fp16's smallest step from magnitudes of about 2^-6 on (error
      // against fp64 at 4 x 2048 x 4096, weights of mean zero: 3e-5 at 2^-7, 2e-2 at 2^-16)
      if constexpr (XT == kBF16 || FMT == kQ4_K) {
        constexpr uint32_t kNonFinite = XT == kBF16 ? 0x7F80u : 0x7C00u;
        uint32_t both = 0;
#pragma unroll
        for (int s = 0; s < 16; ++s)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            asm("max.u16x2 %0, %0, %1;" : "+r"(both) : "r"(f.b[s][t][j] & 0x7FFF7FFFu));
        uint32_t mx = max(both & 0xFFFFu, both >> 16);
        if (__any_sync(0xffffffffu, mx >= kNonFinite)) {  // the scale follows the finite values
          f.non_finite = true;
          mx = 0;
#pragma unroll
          for (int s = 0; s < 16; ++s)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint32_t lo = f.b[s][t][j] & 0x7FFFu, hi = (f.b[s][t][j] >> 16) & 0x7FFFu;
              if (lo < kNonFinite) mx = max(mx, lo);
              if (hi < kNonFinite) mx = max(mx, hi);
            }
        }
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        if constexpr (XT == kBF16) {
          if (mx >> 7) scale = scale_for(mx >> 7);
#pragma unroll
          for (int s = 0; s < 16; ++s)
#pragma unroll
            for (int j = 0; j < 2; ++j)
              f.b[s][t][j] = pack_f16(__uint_as_float(f.b[s][t][j] << 16) * scale,
                                      __uint_as_float(f.b[s][t][j] & 0xFFFF0000u) * scale);
        } else {
          // upwards only and by at most 2^15, so that the product is exact; a sum / 64 of values that the cap leaves
          // small is still a multiple of 2^-15
          const int sh = min(15, max(0, 29 - (int)(mx >> 10)));
          scale = __uint_as_float((uint32_t)(127 + sh) << 23);
          const uint32_t scale2 = (uint32_t)(15 + sh) * 0x04000400u;
#pragma unroll
          for (int s = 0; s < 16; ++s)
#pragma unroll
            for (int j = 0; j < 2; ++j) f.b[s][t][j] = hmul2(f.b[s][t][j], scale2);
        }
      }
    }
    const float unscale = __uint_as_float((254u << 23) - __float_as_uint(scale));  // both are powers of two
    f.u[t][0] = __shfl_sync(0xffffffffu, unscale, 8 * tig);
    f.u[t][1] = __shfl_sync(0xffffffffu, unscale, 8 * tig + 4);
    if constexpr (FMT == kQ4_K) {
      // group sums by MMA: row i of A is one where lane i of a column feeds it, so that row i of D is the sum over lane
      // i's elements; lane (column, i) then fetches its own from the lane that holds it (an infinity or a NaN reaches
      // every group of its column: see non_finite_sum)
      const uint32_t ones = gid == tig ? 0x3C003C00u : 0u;
      float hi[2], lo[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < 8; ++s) ptx::mma16816<true>(c, ones, 0u, ones, 0u, f.b[8 * h + s][t][0], f.b[8 * h + s][t][1], c);
        const float even = __shfl_sync(0xffffffffu, c[0], 4 * tig + (gid >> 1)), odd = __shfl_sync(0xffffffffu, c[1], 4 * tig + (gid >> 1));
        const float sum = (gid & 1 ? odd : even) * 0.015625f;
        hi[h] = __half2float(__float2half_rn(sum));
        lo[h] = sum - hi[h];
      }
      f.bm[t][0] = pack_f16(hi[0], hi[1]);
      f.bm[t][1] = pack_f16(lo[0], lo[1]);
    }
  }
  if constexpr (FMT == kQ4_K) f.non_finite = __any_sync(0xffffffffu, f.non_finite);
}

// What a Q4_K block and the slice of one activation row come to where the slice holds an infinity or a NaN (`sum`: where it
// does not).  The kernel multiplies quants and minimums apart, which makes inf - inf of an infinity; the product with the
// decoded weight is an infinity of its sign.  Only terms that are not finite count.
template <int XT>
__device__ __noinline__ float non_finite_sum(float sum, const uint8_t* block, const void* x, long long at) {
  bool found = false;
#pragma unroll 1
  for (int e = 0; e < 256; ++e) {
    float v;
    if constexpr (XT == kF32) v = static_cast<const float*>(x)[at + e];
    else if constexpr (XT == kBF16) v = __bfloat162float(static_cast<const __nv_bfloat16*>(x)[at + e]);
    else v = __half2float(static_cast<const __half*>(x)[at + e]);
    if ((__float_as_uint(v) & 0x7F800000u) == 0x7F800000u) {
      sum = (found ? sum : 0.f) + decode_one<kQ4_K>(block, e) * v;
      found = true;
    }
  }
  return sum;
}

// What a lane needs to know about its two rows (gid and gid + 8) of a staged tile.
struct LaneRows {
  uint32_t row[2];    // byte offset of the slice's first byte inside a stage
  bool upper;         // Q4_K: groups 4..7
  uint32_t m_lo, m_hi, sel0, sel1, sel01;
  uint32_t nib_lo, nib_hi, magic;  // 0x000F000F, 0x00F000F0 (Q6_K: 0x0F0F0F0F, 0x30303030) and kMagic
  int valid;          // 32-weight blocks of the slice that exist
};

template <int FMT, int XT, int NT>
__device__ __forceinline__ void tile_item(const Frag<NT>& f, uint32_t stage, const LaneRows& ln, int tig, float (&acc)[NT][4]) {
  const float zero[4] = {0.f, 0.f, 0.f, 0.f};
  const uint32_t rA = stage + ln.row[0], rB = stage + ln.row[1];
  if constexpr (FMT == kQ4_K) {
    uint32_t s_lo[2], o_lo[2], s_hi[2], o_hi[2], mn[2];
    float d[2], dm[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint4 hdr = ptx::lds128(r ? rB : rA);
      const float2 dd = __half22float2(*reinterpret_cast<const __half2*>(&hdr.x));
      d[r] = dd.x;
      dm[r] = dd.y * -64.f;
      const uint32_t scv = and_or(ln.upper ? hdr.w : hdr.y, ln.m_lo, (hdr.y >> 2) & ln.m_hi);
      const uint32_t mnv = and_or(ln.upper ? hdr.w >> 4 : hdr.z, ln.m_lo, (hdr.z >> 2) & ln.m_hi);
      s_lo[r] = hadd2(__byte_perm(scv, kMagic, ln.sel0), kMinus1024);
      const uint32_t sc1 = hadd2(__byte_perm(scv, kMagic, ln.sel1), kMinus1024);
      mn[r] = hadd2(__byte_perm(mnv, kMagic, ln.sel01), kMinus1024);
      o_lo[r] = hmul2(s_lo[r], kMinus1024);
      s_hi[r] = hmul2(sc1, kSixteenth);
      o_hi[r] = hmul2(sc1, kMinus64);
    }
    // products scale * nibble, in two chains where only one column tile gives the tensor pipe something to overlap, and
    // for fp32 activations: a chain truncates at every MMA (16 x 4096 x 4096: 3.3e-7 off fp64 in one chain)
    constexpr int kChains = NT == 1 || XT == kF32 ? 2 : 1;
    float c[kChains][NT][4];
#pragma unroll
    for (int h = 0; h < kChains; ++h)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[h][t][j] = 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint4 qa = ptx::lds128(rA + 16 + 32 * tig + 16 * half), qb = ptx::lds128(rB + 16 + 32 * tig + 16 * half);
      const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int s = 4 * half + i;
        const uint32_t va = wa[i] >> 8, vb = wb[i] >> 8;
        const uint32_t a0 = hfma2(and_or(wa[i], ln.nib_lo, ln.magic), s_lo[0], o_lo[0]);
        const uint32_t a1 = hfma2(and_or(wb[i], ln.nib_lo, ln.magic), s_lo[1], o_lo[1]);
        const uint32_t a2 = hfma2(and_or(va, ln.nib_lo, ln.magic), s_lo[0], o_lo[0]);
        const uint32_t a3 = hfma2(and_or(vb, ln.nib_lo, ln.magic), s_lo[1], o_lo[1]);
#pragma unroll
        for (int t = 0; t < NT; ++t) ptx::mma16816<true>(c[0][t], a0, a1, a2, a3, f.b[s][t][0], f.b[s][t][1], c[0][t]);
        const uint32_t h0 = hfma2(and_or(wa[i], ln.nib_hi, ln.magic), s_hi[0], o_hi[0]);
        const uint32_t h1 = hfma2(and_or(wb[i], ln.nib_hi, ln.magic), s_hi[1], o_hi[1]);
        const uint32_t h2 = hfma2(and_or(va, ln.nib_hi, ln.magic), s_hi[0], o_hi[0]);
        const uint32_t h3 = hfma2(and_or(vb, ln.nib_hi, ln.magic), s_hi[1], o_hi[1]);
#pragma unroll
        for (int t = 0; t < NT; ++t)
          ptx::mma16816<true>(c[kChains - 1][t], h0, h1, h2, h3, f.b[8 + s][t][0], f.b[8 + s][t][1], c[kChains - 1][t]);
      }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      float cm[4];
      ptx::mma16816<true>(cm, mn[0], mn[1], mn[0], mn[1], f.bm[t][0], f.bm[t][1], zero);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float v = c[0][t][j];
        if constexpr (kChains == 2) v += c[1][t][j];
        acc[t][j] = fmaf(d[j >> 1], v, dm[j >> 1] * cm[j]);
      }
    }
  } else if constexpr (FMT == kQ6_K) {
    const uint32_t shA = (rA & 2u) * 8u, shB = (rB & 2u) * 8u, baseA = rA & ~3u, baseB = rB & ~3u;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[t][j] = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // the eight 8-bit scales of this half of the block, each plus 128
      uint32_t sc[2][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        sc[0][i] = lds32_half(baseA + 192 + 8 * h + 4 * i, shA) ^ 0x80808080u;
        sc[1][i] = lds32_half(baseB + 192 + 8 * h + 4 * i, shB) ^ 0x80808080u;
      }
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        uint32_t v[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t at = (r ? baseB : baseA) + 16 * jj + 4 * tig, sh = r ? shB : shA;
          const uint32_t l0 = lds32_half(at + 64 * h, sh), l1 = lds32_half(at + 64 * h + 32, sh);
          const uint32_t q = lds32_half(at + 128 + 32 * h, sh);
          v[r][0] = and_or(l0, ln.nib_lo, (q << 4) & ln.nib_hi);
          v[r][1] = and_or(l1, ln.nib_lo, (q << 2) & ln.nib_hi);
          v[r][2] = and_or(l0 >> 4, ln.nib_lo, q & ln.nib_hi);
          v[r][3] = and_or(l1 >> 4, ln.nib_lo, (q >> 2) & ln.nib_hi);
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int g = 8 * h + 2 * p + jj;  // scale group: 16 elements from 16 g on
          const uint32_t a0 = hadd2(__byte_perm(v[0][p], kMagic, 0x5250), kMinus1056), a1 = hadd2(__byte_perm(v[1][p], kMagic, 0x5250), kMinus1056);
          const uint32_t a2 = hadd2(__byte_perm(v[0][p], kMagic, 0x5351), kMinus1056), a3 = hadd2(__byte_perm(v[1][p], kMagic, 0x5351), kMinus1056);
          // byte (2 p + jj) of the half's scales as a float: 2^23 + 128 + scale
          const int byte = 2 * p + jj;
          const float fa = __uint_as_float(__byte_perm(sc[0][byte >> 2], 0x4B000000u, 0x7540u | (byte & 3))) - 8388736.f;
          const float fb = __uint_as_float(__byte_perm(sc[1][byte >> 2], 0x4B000000u, 0x7540u | (byte & 3))) - 8388736.f;
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            float c[4];
            ptx::mma16816<true>(c, a0, a1, a2, a3, f.b[g][t][0], f.b[g][t][1], zero);
            acc[t][0] = fmaf(fa, c[0], acc[t][0]);
            acc[t][1] = fmaf(fa, c[1], acc[t][1]);
            acc[t][2] = fmaf(fb, c[2], acc[t][2]);
            acc[t][3] = fmaf(fb, c[3], acc[t][3]);
          }
        }
      }
    }
    const float dA = lds_half(rA + 208), dB = lds_half(rB + 208);
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      acc[t][0] *= dA;
      acc[t][1] *= dA;
      acc[t][2] *= dB;
      acc[t][3] *= dB;
    }
  } else {
    constexpr int kBlock = FMT == kQ8_0 ? 34 : 18;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[t][j] = 0.f;
    const uint32_t baseA = rA & ~3u, baseB = rB & ~3u;
    const uint32_t halfA = rA & 2u, halfB = rB & 2u;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int at = kBlock * b + 2;  // the block's quants: the word grid's other half for every other block
      uint32_t v[2][4];               // k-step 0: (0, 2), (1, 3); k-step 1
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t half = (r ? halfB : halfA) + (uint32_t)(at & 2);  // 0, 2 or 4
        const uint32_t word = (r ? baseB : baseA) + (uint32_t)(at & ~3) + (half & 4u) + 4u * (uint32_t)tig;
        const uint32_t sh = (half & 2u) * 8u;
        if constexpr (FMT == kQ8_0) {
          const uint32_t q0 = lds32_half(word, sh) ^ 0x80808080u, q1 = lds32_half(word + 16, sh) ^ 0x80808080u;
          v[r][0] = hadd2(__byte_perm(q0, kMagic, 0x5250), kMinus1152);
          v[r][1] = hadd2(__byte_perm(q0, kMagic, 0x5351), kMinus1152);
          v[r][2] = hadd2(__byte_perm(q1, kMagic, 0x5250), kMinus1152);
          v[r][3] = hadd2(__byte_perm(q1, kMagic, 0x5351), kMinus1152);
        } else {
          const uint32_t q = lds32_half(word, sh), q8 = q >> 8;
          v[r][0] = hadd2(and_or(q, ln.nib_lo, ln.magic), kMinus1032);
          v[r][1] = hadd2(and_or(q8, ln.nib_lo, ln.magic), kMinus1032);
          v[r][2] = hfma2(and_or(q, ln.nib_hi, ln.magic), kSixteenth, kMinus72);
          v[r][3] = hfma2(and_or(q8, ln.nib_hi, ln.magic), kSixteenth, kMinus72);
        }
      }
      // (past the end of K the bytes belong to no block: their scale may be anything)
      const bool exists = b < ln.valid;
      const float dA = exists ? lds_half(rA + kBlock * b) : 0.f, dB = exists ? lds_half(rB + kBlock * b) : 0.f;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        float c[4];
        ptx::mma16816<true>(c, v[0][0], v[1][0], v[0][1], v[1][1], f.b[2 * b][t][0], f.b[2 * b][t][1], zero);
        ptx::mma16816<true>(c, v[0][2], v[1][2], v[0][3], v[1][3], f.b[2 * b + 1][t][0], f.b[2 * b + 1][t][1], c);
        acc[t][0] = fmaf(dA, c[0], acc[t][0]);
        acc[t][1] = fmaf(dA, c[1], acc[t][1]);
        acc[t][2] = fmaf(dB, c[2], acc[t][2]);
        acc[t][3] = fmaf(dB, c[3], acc[t][3]);
      }
    }
  }
}

// Shared memory: barriers, kStages tiles a warp, kReds buffers of the warps' partial tiles, then (splits > 1) two buffers of
// a phase's summed tiles for the other CTAs of the cluster.
//
// The warps of a row tile do not meet: each leaves its partial tile in a buffer and goes on, and the tile's owner (they
// take turns; two of them above eight rows) adds the sums one tile later.  Meeting at a barrier once a tile made all warps load, compute and wait at the
// same time: Q4_K 18944 x 3584 at batch 8 ran 18.2 us so.
template <int FMT, int XT, int NT>
__global__ void __launch_bounds__(kThreads, 1) gemv_frag_kernel(const FragArgs a) {
  using C = Cfg<FMT>;
  constexpr int kParts = XT == kF32 ? 3 : 1;
  constexpr int kStageBytes = kRows * C::kPitch;
  constexpr int kRed = NT * 8 * kColPitch;  // floats of a partial tile
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int warps = blockDim.x >> 5;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);  // [streams][kReds] partial tiles of all warps are in place
  uint64_t* empty = full + kWarps * C::kReds;          // [streams][kReds] ... and have been added
  static_assert(2 * kWarps * C::kReds * 8 <= kBarrierBytes, "barriers");
  float* red = reinterpret_cast<float*>(smem + kBarrierBytes + warps * C::kStages * kStageBytes);  // [kReds][warps][kRed]
  float* part = red + C::kReds * warps * kRed;                                                     // [2][phase * streams][m][kRows]
  ptx::grid_launch_dependents();

  const int rank = a.splits > 1 ? (int)cluster_rank() : 0;
  const int cluster = (int)blockIdx.x / a.splits, clusters = (int)gridDim.x / a.splits;
  const int sb0 = rank * a.nsb / a.splits, sbs = (rank + 1) * a.nsb / a.splits - sb0;
  const int stream = warp / a.warps_per_row, seg = warp - stream * a.warps_per_row;
  const int sb = sb0 + seg;
  const bool live = seg < sbs;
  const uint32_t stage0 = ptx::smem_addr(smem) + kBarrierBytes + (uint32_t)(warp * C::kStages * kStageBytes);

  // ---- weights: this lane's granules of a tile, tiles of this warp's stream one after another ----
  constexpr int kRowsAtOnce = 32 / C::kLanes;
  const int sub = lane / C::kLanes, gl = lane - sub * C::kLanes;
  const uint32_t row_bytes32 = (uint32_t)a.row_bytes, tile_bytes = kRows * row_bytes32;
  const uint32_t lane_from = (uint32_t)sub * row_bytes32 + (uint32_t)(sb * C::kBytes);
  const uint32_t lane_to = stage0 + (uint32_t)(sub * C::kPitch + 16 * gl);
  const int tile_step = clusters * a.streams, tile0 = cluster * a.streams + stream;
  const int second_tile = a.w2 ? a.n1 / kRows : a.row_tiles;
  const bool fetches = live && sub < kRowsAtOnce;
  int fetch_tile = tile0;
  uint32_t fetch_to = lane_to;
  auto fetch = [&]() {
    if (fetches && fetch_tile < a.row_tiles) {
      const bool second = fetch_tile >= second_tile;
      const uint8_t* base = (second ? a.w2 : a.w) + (unsigned long long)(uint32_t)fetch_tile * tile_bytes;
      if (fetch_tile < (second ? a.fast2 : a.fast1)) {
#pragma unroll
        for (int i = 0; i < (kRows + kRowsAtOnce - 1) / kRowsAtOnce; ++i) {
          if ((i + 1) * kRowsAtOnce <= kRows || i * kRowsAtOnce + sub < kRows) {
            const uint8_t* at = base + ((lane_from + (uint32_t)(i * kRowsAtOnce) * row_bytes32) & ~15u) + 16 * gl;
            const uint32_t to = fetch_to + (uint32_t)(i * kRowsAtOnce * C::kPitch);
#pragma unroll
            for (int g = 0; g < C::kPer; ++g)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16u * (uint32_t)(g * C::kLanes)),
                           "l"(at + 16 * g * C::kLanes)
                           : "memory");
          }
        }
      } else {
        // the end of a weight: rows that exist, and its last granule up to the last byte
        const int rows = (second ? a.n : a.n1) - fetch_tile * kRows;
        const uint8_t* end = second ? a.w2 + a.w2_bytes : a.w + a.w_bytes;
#pragma unroll 1
        for (int r = sub; r < min(kRows, rows); r += kRowsAtOnce) {
          const uint8_t* at = base + (((uint32_t)r * row_bytes32 + (uint32_t)(sb * C::kBytes)) & ~15u) + 16 * gl;
#pragma unroll
          for (int g = 0; g < C::kPer; ++g) {
            const long long left = end - (at + 16 * g * C::kLanes);
            if (left > 0)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                               fetch_to + (uint32_t)((r - sub) * C::kPitch) + 16u * (uint32_t)(g * C::kLanes)),
                           "l"(at + 16 * g * C::kLanes), "r"((int)min(16ll, left))
                           : "memory");
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    fetch_tile += tile_step;
    fetch_to += kStageBytes;
    if (fetch_to == lane_to + C::kStages * kStageBytes) fetch_to = lane_to;
  };
#pragma unroll 1
  for (int i = 0; i < C::kStages - 1; ++i) fetch();  // (weights never depend on the kernel before)

  const int row_warps = min(a.warps_per_row, sbs);
  const int slot_quads = a.m * (kRows / 4);  // a tile's sums, four rows each
  const int owners = slot_quads > 32 && row_warps > 1 ? 2 : 1;
  if (threadIdx.x < a.streams * C::kReds) {
    ptx::mbar_init(&full[threadIdx.x], row_warps);
    ptx::mbar_init(&empty[threadIdx.x], owners);
    ptx::fence_mbar_init();
  }
  __syncthreads();
  full += stream * C::kReds;
  empty += stream * C::kReds;

  LaneRows ln;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = gid + 8 * r;
    // 16 rows are a multiple of 16 bytes, so the skew of row `row` is the same in every tile
    ln.row[r] = (uint32_t)(row * C::kPitch) + (((uint32_t)row * row_bytes32 + (uint32_t)(sb * C::kBytes)) & 15u);
  }
  ln.upper = tig >= 2;
  ln.m_lo = ln.upper ? 0x0F0F0F0Fu : 0x3F3F3F3Fu;
  ln.m_hi = ln.upper ? 0x30303030u : 0u;
  const uint32_t byte = 2u * (uint32_t)(tig & 1);
  ln.sel0 = 0x5050u | byte | byte << 8;
  ln.sel1 = 0x5050u | (byte + 1) | (byte + 1) << 8;
  ln.sel01 = 0x5050u | byte | (byte + 1) << 8;
  ln.nib_lo = pinned(FMT == kQ6_K ? 0x0F0F0F0Fu : 0x000F000Fu);
  ln.nib_hi = pinned(FMT == kQ6_K ? 0x30303030u : 0x00F000F0u);
  ln.magic = pinned(kMagic);
  ln.valid = min(8, (a.k - sb * 256) >> 5);

  ptx::grid_dependency_wait();  // activations and outputs may belong to the kernel before
  Frag<NT> f;
  load_fragments<FMT, XT, NT>(f, a, sb, live, gid, tig, stage0 + (C::kStages - 1) * kStageBytes);

  // four rows of one column
  auto store = [&](int tile, int col, int r, const float4& v) {
    const int row = tile * kRows + r;
    const bool second = row >= a.n1;
    float* o = (second ? a.out2 - a.n1 : a.out) + (long long)col * a.out_ld + row;
    const int rows = (second ? a.n : a.n1) - row;
    if (rows >= 4 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
      *reinterpret_cast<float4*>(o) = v;
    } else {
      if (rows > 0) o[0] = v.x;
      if (rows > 1) o[1] = v.y;
      if (rows > 2) o[2] = v.z;
      if (rows > 3) o[3] = v.w;
    }
  };
  const uint32_t red0 = ptx::smem_addr(red), red_bytes = (uint32_t)(warps * kRed) * 4;
  const uint32_t mine = red0 + (uint32_t)(warp * kRed + 2 * tig * kColPitch + gid) * 4;
  const uint32_t first = red0 + (uint32_t)((warp - seg) * kRed) * 4;
  uint32_t stage = stage0;
  int slot = 0, part_buf = 0, tile = tile0;
  bool ok = true;  // no wait of this warp has run out
  // what the owner does: the partial tiles of tile `which` (buffer b, for the use-th time) added in K order
  auto add_up = [&](int which, int b, int use, int to_slot, int share) {
    if (ok && !ptx::mbar_wait(&full[b], use & 1)) {
      report_timeout(0xA0000u);
      ok = false;
    }
    if (!ok) return;
    for (int o = lane + 32 * share; o < slot_quads; o += 32 * owners) {
      const int col = o >> 2, r = 4 * (o & 3);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      // (the small parts of fp32 activations first: added to the sum of the large ones each would cost it a rounding)
#pragma unroll
      for (int p = kParts - 1; p >= 0; --p) {
        uint32_t at = first + (uint32_t)b * red_bytes + (uint32_t)((col * kParts + p) * kColPitch + r) * 4;
#pragma unroll 4
        for (int wi = 0; wi < row_warps; ++wi, at += kRed * 4) {
          const uint4 q = ptx::lds128(at);
          v.x += __uint_as_float(q.x), v.y += __uint_as_float(q.y), v.z += __uint_as_float(q.z), v.w += __uint_as_float(q.w);
        }
      }
      if (a.splits == 1) store(which, col, r, v);
      else reinterpret_cast<float4*>(part)[((part_buf * a.phase + to_slot) * a.streams + stream) * slot_quads + o] = v;
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&empty[b]);
  };
  int buf = 0, use = 0;               // this tile's buffer and how often it has been used before
  int last_buf = 0, last_use = 0;     // the same of the tile before
  int first_owner = 0, second_owner = row_warps / 2;  // of this tile
  int owed = -1;                      // this warp's share of the tile before, or -1
#pragma unroll 1
  for (int it = 0; it < a.iters; ++it, tile += tile_step) {
    fetch();
    cp_async_wait<C::kStages - 1>();
    __syncwarp();
    const bool has_tile = live && tile < a.row_tiles;
    if (has_tile) {
      float acc[NT][4];
      tile_item<FMT, XT, NT>(f, stage, ln, tig, acc);
      if constexpr (FMT == kQ4_K)
        if (f.non_finite) {
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int col = 8 * t + 2 * tig + (j & 1), row = tile * kRows + gid + 8 * (j >> 1);
              const bool exists = row < (tile >= second_tile ? a.n : a.n1);
              if (col % kParts == 0 && col / kParts < a.m && exists)
                acc[t][j] = non_finite_sum<XT>(acc[t][j], smem + (stage - ptx::smem_addr(smem)) + ln.row[j >> 1], a.x,
                                               (long long)(col / kParts) * a.k + sb * 256);
            }
        }
      if (use > 0 && ok && !ptx::mbar_wait(&empty[buf], (use - 1) & 1)) {
        report_timeout(0xB0000u);
        ok = false;
      }
      const uint32_t to = mine + (uint32_t)buf * red_bytes;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const uint32_t c0 = to + (uint32_t)(8 * t * kColPitch) * 4;
        sts32(c0, acc[t][0] * f.u[t][0]);
        sts32(c0 + 4 * kColPitch, acc[t][1] * f.u[t][1]);
        sts32(c0 + 32, acc[t][2] * f.u[t][0]);
        sts32(c0 + 4 * kColPitch + 32, acc[t][3] * f.u[t][1]);
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&full[buf]);
    }
    stage += kStageBytes;
    if (stage == stage0 + C::kStages * kStageBytes) stage = stage0;
    if (owed >= 0) add_up(tile - tile_step, last_buf, last_use, slot - 1, owed);
    owed = !has_tile ? -1 : seg == first_owner ? 0 : (owners == 2 && seg == second_owner) ? 1 : -1;
    last_buf = buf, last_use = use;
    if (++buf == C::kReds) buf = 0, ++use;
    if (++first_owner == row_warps) first_owner = 0;
    if (++second_owner == row_warps) second_owner = 0;
    const bool exchange = a.splits > 1 && (slot + 1 == a.phase || it + 1 == a.iters);
    if (owed >= 0 && (exchange || it + 1 == a.iters)) {
      add_up(tile, last_buf, last_use, slot, owed);
      owed = -1;
    }
    ++slot;
    if (exchange) {
      // every CTA of the cluster adds its share of the phase's tiles over all K ranges; the other buffer takes the next
      // phase's tiles meanwhile
      __syncwarp();
      cluster_sync();
      const uint32_t from = ptx::smem_addr(part) + (uint32_t)(part_buf * a.phase * a.streams * slot_quads) * 16;
      const int total = slot * a.streams * slot_quads, it0 = it + 1 - slot;
      for (int i = rank * (int)blockDim.x + (int)threadIdx.x; i < total; i += a.splits * (int)blockDim.x) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < kMaxSplits; ++p)
          if (p < a.splits) {
            const float4 q = ld_cluster_f32x4(map_rank(from, (uint32_t)p) + 16u * (uint32_t)i);
            v.x += q.x, v.y += q.y, v.z += q.z, v.w += q.w;
          }
        const int which = i / slot_quads, o = i - which * slot_quads;
        const int t = ((it0 + which / a.streams) * clusters + cluster) * a.streams + which % a.streams;
        if (t < a.row_tiles) store(t, o >> 2, 4 * (o & 3), v);
      }
      slot = 0;
      part_buf ^= 1;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  if (a.splits > 1) cluster_sync();  // nobody may still read the sums of a CTA that has left
}

struct FragPlan {
  int warps_per_row, streams, splits, clusters, iters, phase, smem;
};

template <int FMT, int XT, int NT>
int resident(int splits, const DeviceInfo& dev) {
  if (splits == 1) return dev.sm_count;
  static int known[64][kMaxSplits + 1];  // 0 = not asked yet (a race writes the same number twice)
  int& entry = known[dev.ordinal & 63][splits];
  if (entry > 0) return entry;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(dev.sm_count / splits * splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)dev.max_smem_optin;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int count = 0;
  if (cudaOccupancyMaxActiveClusters(&count, gemv_frag_kernel<FMT, XT, NT>, &cfg) != cudaSuccess || count < 1) {
    cudaGetLastError();
    count = std::max(1, dev.sm_count / splits - splits);
  }
  entry = count;
  return count;
}

// CTAs along K (a cluster) and row tiles at once.  The unit is one warp's work on 16 x 256 weights, of which an SM does one
// after another at its own rate (about 100 clocks): a plan costs the units of its busiest SM, what a tile costs beyond its
// decode (three units: buffers, barriers, adding up), and the exchange of a cluster (about a thousand clocks).
template <int FMT, int XT, int NT>
FragPlan plan_frag(int m, int row_tiles, int nsb, const DeviceInfo& dev) {
  using C = Cfg<FMT>;
  FragPlan best{};
  double best_cost = 1e300;
  for (int s = 1; s <= kMaxSplits && s <= nsb; ++s) {
    const int kw = (nsb + s - 1) / s;
    if (kw > kWarps) continue;
    const int clusters_max = resident<FMT, XT, NT>(s, dev);
    const int streams = std::min(kWarps / kw, std::max(1, (row_tiles + clusters_max - 1) / clusters_max));
    const int warps = kw * streams;
    const int clusters = std::min(clusters_max, (row_tiles + streams - 1) / streams);
    const int iters = (row_tiles + clusters * streams - 1) / (clusters * streams);
    const double cost = iters * (double)(warps + 3) + (s > 1 ? 10.0 + 0.5 * s : 0.0) + 0.25 * (kWarps - warps);
    if (cost >= best_cost) continue;
    const int smem = kBarrierBytes + warps * (C::kStages * kRows * C::kPitch + C::kReds * NT * 8 * kColPitch * 4);
    const int slot = streams * m * kRows * 4;
    const int phase = s > 1 ? std::min(iters, (dev.max_smem_optin - smem) / (2 * slot)) : 1;
    if (smem > dev.max_smem_optin || phase < 1) continue;
    best_cost = cost;
    best = FragPlan{kw, streams, s, clusters, iters, phase, smem + (s > 1 ? 2 * phase * slot : 0)};
  }
  return best;
}

template <int FMT, int XT, int NT>
cudaError_t launch_typed(FragArgs a, cudaStream_t stream) {
  cudaError_t e;
  const DeviceInfo* dev = device_info(&e);
  if (!dev) return e;
  auto kernel = gemv_frag_kernel<FMT, XT, NT>;
  e = allow_full_shared_memory(kernel);
  if (e != cudaSuccess) return e;
  const FragPlan plan = plan_frag<FMT, XT, NT>(a.m, a.row_tiles, a.nsb, *dev);
  if (!plan.splits) return cudaErrorInvalidValue;
  a.warps_per_row = plan.warps_per_row;
  a.streams = plan.streams;
  a.splits = plan.splits;
  a.iters = plan.iters;
  a.phase = plan.phase;
  // A cluster launch that may start while a plain one drains (or the other way round) costs about 4 us: Q4_K 24576 x 4096 and
  // 4096 x 12288 in turn at batch 8 take 45.1 us so and 37.3 with the cluster launches serialized, which is the sum of
  // the two alone; cluster launches one after another lose 1.6 us each by it (Q4_K and Q6_K 4096 x 12288 in turn: 34.7 us
  // for the two when they may overlap, 37.9 so).
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = plan.splits > 1 ? 0 : 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)plan.splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(plan.clusters * plan.splits));
  cfg.blockDim = dim3((unsigned)(plan.warps_per_row * plan.streams * 32));
  cfg.dynamicSmemBytes = (size_t)plan.smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = plan.splits > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <int FMT>
cudaError_t launch_format(int xt, const FragArgs& a, cudaStream_t stream) {
  const bool two = a.m * (xt == kF32 ? 3 : 1) > 8;
  if (xt == kBF16) return two ? launch_typed<FMT, kBF16, 2>(a, stream) : launch_typed<FMT, kBF16, 1>(a, stream);
  if (xt == kF16) return two ? launch_typed<FMT, kF16, 2>(a, stream) : launch_typed<FMT, kF16, 1>(a, stream);
  return two ? launch_typed<FMT, kF32, 2>(a, stream) : launch_typed<FMT, kF32, 1>(a, stream);
}

}  // namespace

TB200_DEFINE_STATUS_READER(read_gemv_frag_status)

bool gemv_frag_supported(int fmt, int xt, long long m, long long n, long long k) {
  if (!valid_format(fmt) || (xt != kBF16 && xt != kF16 && xt != kF32)) return false;
  return m >= 1 && m <= 16 && n >= 1 && n <= (1 << 28) && k >= block_weights(fmt) && k % block_weights(fmt) == 0 &&
         k <= 256 * kWarps * kMaxSplits;
}

cudaError_t launch_gemv_frag(int fmt, int xt, const void* x, const uint8_t* w, const OutSpec& out, long long m, long long n,
                             long long k, cudaStream_t stream, const uint8_t* w2, long long n1) {
  FragArgs a{};
  a.w = w;
  a.out_ld = out.ld;
  a.n = (int)n;
  a.n1 = w2 ? (int)n1 : (int)n;
  a.k = (int)k;
  a.row_bytes = row_bytes(fmt, k);
  a.w_bytes = a.row_bytes * a.n1;
  a.w2 = w2 ? w2 - a.w_bytes : nullptr;
  a.w2_bytes = a.row_bytes * n;
  a.row_tiles = (int)((n + kRows - 1) / kRows);
  a.nsb = (int)((k + 255) / 256);
  // (a copy of whole granules reads up to 288 bytes from the granule of a slice's first byte on)
  const long long tile_bytes = kRows * a.row_bytes;
  a.fast1 = (int)std::max(0ll, (a.w_bytes - 320) / tile_bytes);
  a.fast2 = (int)std::max(0ll, (a.w2_bytes - 320) / tile_bytes);
  // fp32 activations take three columns a row: five rows a launch
  const int step = xt == kF32 ? 5 : 16;
  for (int row = 0; row < m; row += step) {
    a.m = std::min(step, (int)m - row);
    a.x = static_cast<const uint8_t*>(x) + (long long)row * k * (xt == kF32 ? 4 : 2);
    a.out = out.ptr[0] + row * out.ld;
    a.out2 = w2 ? out.ptr2[0] + row * out.ld : nullptr;
    cudaError_t e = cudaErrorInvalidValue;
    switch (fmt) {
      case kQ4_0: e = launch_format<kQ4_0>(xt, a, stream); break;
      case kQ8_0: e = launch_format<kQ8_0>(xt, a, stream); break;
      case kQ4_K: e = launch_format<kQ4_K>(xt, a, stream); break;
      case kQ6_K: e = launch_format<kQ6_K>(xt, a, stream); break;
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace tb200
