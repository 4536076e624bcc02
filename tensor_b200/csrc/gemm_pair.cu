// Prefill GEMM on sm_100a, CTA pairs: out[m, n] (fp32) = x[m, k] (bf16) . dequant(w[n, k])^T for all four formats,
// weights rounded to bf16 (round-to-nearest-even of the exact fp32 decode), fp32 accumulation in tensor memory.
//
// Replaces the reference's `_packed` kernel (benchmarks/kernels/showcase/kernels.py:116-119), which decodes GGML
// blocks to 16-bit operands in shared memory and runs `mma.sync` (benchmarks/kernels/showcase/benchmark.py:471-477).
//
// Two CTAs of a cluster work on one tile of 256 weight rows x T tokens with tcgen05.mma.cta_group::2: each decodes
// 128 of the rows and loads half of the tokens, so an SM moves half the activation bytes of a one-CTA tile of the
// same size through its shared memory and from the L2.  The decoded weights never touch shared memory: a thread
// owns one row, which is one TMEM lane, and tcgen05.st puts its 64 bf16 weights where the MMA reads its A operand.
// What is left of shared memory is activation and raw weight stages: a stage is reused only after commit -> wake-up ->
// L2 -> wake-up (about 1700 clocks measured), so their number is what sets the rate (four stages of both operands
// in shared memory: 780 clocks per k-block of T = 192, where the MMAs take 384).  24 warps per CTA:
//
//   warp 0       TMA producer: activation tiles [T / 2 tokens x 64 k] bf16, 128-byte swizzle
//   warp 1       allocates TMEM; in the pair's first CTA one lane issues the MMAs of both and commits to both
//   warp 2       raw weight producer: 128 rows x 256 weights per stage, one tiled TMA copy where the row stride is a
//                multiple of 16 bytes, else (with warp 3) asynchronous copies of the 16-byte granules around a row's bytes
//   warps 4..7   epilogue: tcgen05.ld of one accumulator set while the MMAs fill the other (T <= 192: two sets)
//                (Q8_0, Q4_0: with warps 24..27, the products of every two k-blocks; see kFp32Sums)
//   warps 8..23  decode: four groups of four warps; group j decodes k-block 4 c + j (64 k) of raw chunk c, a thread
//                one row: scales once per 64 weights, 16-byte shared loads without bank conflicts
//
// Persistent over tiles where a tile's K is not split.  Few tiles (short prompts, small weights): 2 or 4 pairs of
// one cluster take a K range each and add their accumulators through distributed shared memory in K order, so that
// no scratch is needed and the result does not depend on timing.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace tb200 {
namespace {

constexpr int kPairRows = 256;   // weight rows of a pair's tile (MMA M)
constexpr int kCtaRows = 128;    // ... of which each CTA decodes half
constexpr int kBlockK = 64;      // K of a pipeline stage: one 128-byte swizzle row of bf16
constexpr int kChunkK = 256;     // K of a raw stage: four k-blocks, one per decode group
constexpr int kMaxAStages = 8;   // decoded k-blocks in tensor memory, 32 columns each (4 or 8: a power of two)
constexpr int kMaxBStages = 16;
constexpr int kMaxRawStages = 6;
constexpr int kMaxTokens = 256;
constexpr int kDecodeWarp0 = 8;
constexpr int kDecodeWarps = 16;
constexpr int kGroups = 6;       // of four warps that wait together: four that decode, up to two that drain
// The 32-weight formats: the tensor cores add up one k-block only, eight drain warps the k-blocks, in fp32 registers, and
// every kInnerSums of them in shared memory.  Accumulating in tensor memory truncates: about 1.3e-8 of the result per 16
// of K, 2.1e-6 against fp64 at K = 4096 and 1.6e-5 at 28672, where the fp32 sums of the SIMT kernel that these formats had
// before are 1.1e-7 and 2.8e-7 off; so they are 1.0e-7 and 1.6e-7 off (K = 512: 8.0e-8 | SIMT 6.6e-8).
// It costs: a drained k-block takes 710 to 750 clocks instead of 540 (waits of the issuer and the drain warps; two
// k-blocks per wait, one at a time took 1000), and 32 sums a thread next to 16 loaded products are all that 72 registers
// hold, so a tile has 64 tokens (96, with the drain warps given more registers: the longer code does not stay in the
// instruction cache, 333 x 12288 x 4096 131 us).  Q8_0 333 x 12288 x 4096 takes 109 us so, 47 accumulated in tensor
// memory, 4519 on the SIMT kernel; 64 x 4096 x 4096 20 | 17 | 283.
template <int FMT>
constexpr bool kFp32Sums = FMT == kQ8_0 || FMT == kQ4_0;
constexpr int kInnerSums = 8;
constexpr int kMaxTokensFp32 = 64;
constexpr int kSumSets = 4;  // accumulator sets: two pairs of k-blocks
template <int FMT>
constexpr int max_tokens() { return kFp32Sums<FMT> ? kMaxTokensFp32 : kMaxTokens; }
template <int FMT>
constexpr int threads_of() { return (kDecodeWarp0 + kDecodeWarps + (kFp32Sums<FMT> ? 4 : 0)) * 32; }
constexpr int kSmemLimit = 232448;
constexpr int kBarrierBytes = 1024;
constexpr int kRing = kSmemLimit - 1024 /*alignment*/ - kBarrierBytes;  // activation and raw stages (and sums)
constexpr int kSumBytes = kMaxTokensFp32 * kCtaRows * 4;

// Raw stages: bytes of 256 weights, shared-memory row pitch of the tiled copy and of the per-row copies (room for the
// up to 14 bytes in front, an odd number of 16-byte granules so that eight rows hit eight bank groups), stages.
template <int FMT> struct RawCfg;
template <> struct RawCfg<kQ4_K> { static constexpr int kBytes = 144, kPitch = 144, kRowPitch = 144, kStages = 4; };
template <> struct RawCfg<kQ6_K> { static constexpr int kBytes = 210, kPitch = 240, kRowPitch = 240, kStages = 3; };
template <> struct RawCfg<kQ8_0> { static constexpr int kBytes = 272, kPitch = 272, kRowPitch = 304, kStages = 3; };
template <> struct RawCfg<kQ4_0> { static constexpr int kBytes = 144, kPitch = 144, kRowPitch = 176, kStages = 4; };

struct PairArgs {
  const uint8_t* w;
  float* out;
  long long row_bytes;
  long long w_bytes;   // row_bytes * n
  int m, n, k;
  int tokens;          // T: a multiple of 32, at most 256
  int token_tiles, tiles;
  int splits;          // pairs of a cluster along K: 1, 2 or 4
  int chunks;          // 256-weight chunks of K (the last may be shorter for the 32-weight formats)
  int tiled;           // raw weights by tiled TMA copies
  int acc_sets;        // accumulator sets of T columns in tensor memory (2: the epilogue overlaps the next tile)
  int a_log;           // log2 of the decoded stages behind them
  int b_stages, b_bytes, raw_stages, raw_bytes, pitch;
};

// ---- cluster helpers --------------------------------------------------------------------------------------------
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
__device__ __forceinline__ void arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Bounded wait.  No suspend-time hint, so that a waiting warp sees the completing arrival at once; the clock is
// consulted only after thousands of failed probes (reading the global timer takes about as long as a wait of this kernel).
// Barriers order TMA copies and tensor-memory traffic here, also across the two CTAs of a pair: no generic access to
// another CTA's memory hangs on them, so no wait or arrival needs cluster scope (whose fences cost hundreds of clocks).
__device__ __forceinline__ bool try_wait_now(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool wait_bar(uint64_t* b, uint32_t parity) {
  const uint32_t bar = ptx::smem_addr(b);
#pragma unroll 1
  for (int i = 0; i < 4096; ++i)
    if (try_wait_now(bar, parity)) return true;
  const uint64_t start = ptx::global_timer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (try_wait_now(bar, parity)) return true;
    if (ptx::global_timer_ns() - start > ptx::kWaitLimitNs) return false;
  }
}
// Bounded wait for four barriers at once: a satisfied wait takes about 200 clocks from issue to result, four of them in
// one go take hardly more.
__device__ __forceinline__ uint32_t all_done(const uint32_t (&bar)[4], const uint32_t (&parity)[4]) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q, r, s;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 r, [%5], %6;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 s, [%7], %8;\n\t"
      "and.pred p, p, q;\n\tand.pred r, r, s;\n\tand.pred p, p, r;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar[0]), "r"(parity[0]), "r"(bar[1]), "r"(parity[1]), "r"(bar[2]), "r"(parity[2]), "r"(bar[3]), "r"(parity[3])
      : "memory");
  return ok;
}
__device__ __forceinline__ uint32_t all_done(const uint32_t (&bar)[5], const uint32_t (&parity)[5]) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q, r, s, t;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 r, [%5], %6;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 s, [%7], %8;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 t, [%9], %10;\n\t"
      "and.pred p, p, q;\n\tand.pred r, r, s;\n\tand.pred p, p, r;\n\tand.pred p, p, t;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar[0]), "r"(parity[0]), "r"(bar[1]), "r"(parity[1]), "r"(bar[2]), "r"(parity[2]), "r"(bar[3]), "r"(parity[3]),
        "r"(bar[4]), "r"(parity[4])
      : "memory");
  return ok;
}
template <int N>
__device__ __forceinline__ bool wait_all(const uint32_t (&bar)[N], const uint32_t (&parity)[N]) {
#pragma unroll 1
  for (int i = 0; i < 16384; ++i)
    if (all_done(bar, parity)) return true;
  const uint64_t start = ptx::global_timer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (all_done(bar, parity)) return true;
    if (ptx::global_timer_ns() - start > ptx::kWaitLimitNs) return false;
  }
}
// The same for a group of four warps: one polls, the others wait at a hardware barrier.  (With every decode warp
// polling, the polls queue up in front of the MMA warp's own and a satisfied wait takes 200 clocks there.)
// `late`: two words a group, in turn, that say whether a wait has run out.  Only the group's own poller writes them, before
// the barrier, and not again before every warp of the group has passed the next one: the four read the same and go on or
// leave together.  (A word shared with other groups could change between two of the reads, and part of a group would
// wait for the rest at the next barrier without end.)
struct GroupWait {
  uint32_t late;  // shared address of the word of this wait; the other one is 4 bytes on or back
  int group;
  __device__ __forceinline__ void ran_out() { asm volatile("st.shared.u32 [%0], 1;" ::"r"(late) : "memory"); }
  __device__ __forceinline__ bool verdict() {
    ptx::bar_sync(1 + group, 128);
    uint32_t word;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(word) : "r"(late) : "memory");
    late ^= 4u;
    return word == 0;
  }
  __device__ __forceinline__ bool one(uint64_t* bar, uint32_t parity) {
    if ((threadIdx.x & 96) == 0 && !wait_bar(bar, parity)) ran_out();
    return verdict();
  }
  __device__ __forceinline__ bool two(uint64_t* bar0, uint32_t parity0, uint64_t* bar1, uint32_t parity1) {
    if ((threadIdx.x & 96) == 0) {
      const uint32_t b0 = ptx::smem_addr(bar0), b1 = ptx::smem_addr(bar1);
      const uint32_t bar[4] = {b0, b1, b0, b1}, par[4] = {parity0, parity1, parity0, parity1};
      if (!wait_all(bar, par)) ran_out();
    }
    return verdict();
  }
};
// Activation half-tile into this CTA's shared memory, counted on the pair's first CTA's barrier (no multicast).
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          ptx::smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}
// A (the pair's 256 weight rows) in tensor memory, B (tokens) in shared memory, half of each in either CTA.
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate));
}
// Both CTAs of the pair see an arrival at the same offset once every MMA issued so far has completed.
__device__ __forceinline__ void commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   ptx::smem_addr(bar)),
               "h"(mask)
               : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
  return ok != 0;
}
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
      "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
      "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
  return v;
}

// tcgen05 shared-memory matrix descriptor, K-major, 128-byte swizzle (see gemm_tcgen05.cu)
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}

// ---- decode: one row's 64 weights of a k-block ---------------------------------------------------------------------
// fp32 arithmetic in pairs (one instruction for two weights); every product is exact except Q4_K's single rounding at
// the subtraction, so the pairs round as the scalar statement of the formats does (common.cuh).
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint32_t bf16x2(uint64_t v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(mask), "r"(bits));
  return d;
}
__device__ __forceinline__ float half_bits(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }

// Conversions.  Measured on B200, clocks per warp instruction and scheduler: logic, shift, permute, select and
// cvt.bf16x2 2.0, the mixed add.f32.f16 1.7 (as FFMA), the paired fp32 forms 2.1.  So an integer becomes fp16 1024 + q
// by ONE logic op or permute for two weights, and fp32 q by one mixed-precision add a weight, off the logic pipe.
__device__ __forceinline__ float add_f32_f16(uint32_t half2_, bool high, float c) {
  float r;
  if (high)
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tadd.rn.f32.f16 %0, h, %2;\n\t}" : "=f"(r) : "r"(half2_), "f"(c));
  else
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tadd.rn.f32.f16 %0, l, %2;\n\t}" : "=f"(r) : "r"(half2_), "f"(c));
  return r;
}
// two fp16 integers of different words (their low or their high halves) plus c, as a pair
__device__ __forceinline__ uint64_t pair_f32(uint32_t a, uint32_t b, bool high, float c) {
  return pack2(add_f32_f16(a, high, c), add_f32_f16(b, high, c));
}
constexpr uint32_t kMagic16 = 0x64006400u;  // fp16 1024, twice

// The four bytes of `bytes` plus c - 1024, times s, as four bf16 (two words).
__device__ __forceinline__ uint2 bytes_to_bf16(uint32_t bytes, float c, uint64_t s) {
  const uint32_t a = __byte_perm(bytes, kMagic16, 0x5150), b = __byte_perm(bytes, kMagic16, 0x5352);
  return make_uint2(bf16x2(mul2(pack2(add_f32_f16(a, false, c), add_f32_f16(a, true, c)), s)),
                    bf16x2(mul2(pack2(add_f32_f16(b, false, c), add_f32_f16(b, true, c)), s)));
}

// NW words from a shared address through aligned 16-byte loads.  WS >= 0: the address is 4 WS (+ 2) bytes past a 16-byte
// boundary for every lane of the warp, so words are picked at compile time.  WS < 0: each lane's row has its own 2-byte
// alignment; two selects a word.  HALF: the address may be 2 bytes off the word grid (one funnel shift a word).
template <int NW, int WS, bool HALF>
__device__ __forceinline__ void load_words(uint32_t addr, uint32_t (&out)[NW]) {
  constexpr int L = (NW + (WS < 0 ? 3 : WS) + (HALF ? 1 : 0) + 3) / 4;
  uint32_t w[4 * L];
  const uint32_t base = addr & ~15u;
#pragma unroll
  for (int i = 0; i < L; ++i) {
    const uint4 v = ptx::lds128(base + 16 * i);
    w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
  }
  constexpr int kAt = WS < 0 ? 0 : WS;
  if constexpr (WS < 0) {
    const bool two = addr & 8u, one = addr & 4u;
#pragma unroll
    for (int i = 0; i < NW + 2 && i + 2 < 4 * L; ++i) w[i] = two ? w[i + 2] : w[i];
#pragma unroll
    for (int i = 0; i < NW + 1 && i + 1 < 4 * L; ++i) w[i] = one ? w[i + 1] : w[i];
  }
  const uint32_t shift = (addr & 2u) * 8u;
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    if constexpr (HALF) out[i] = __funnelshift_r(w[kAt + i], kAt + i + 1 < 4 * L ? w[kAt + i + 1] : 0u, shift);
    else out[i] = w[kAt + i];
  }
}

__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}

// One word of nibbles -> fp16 integers: low nibbles of bytes (0, 2) and (1, 3) as 1024 + q, high ones as 1024 + 16 q.
struct NibbleHalves {
  uint32_t lo02, lo13, hi02, hi13;
};
__device__ __forceinline__ NibbleHalves nibble_halves(uint32_t w) {
  const uint32_t w8 = w >> 8;
  return NibbleHalves{and_or(w, 0x000F000Fu, kMagic16), and_or(w8, 0x000F000Fu, kMagic16), and_or(w, 0x00F000F0u, kMagic16),
                      and_or(w8, 0x00F000F0u, kMagic16)};
}

// Decodes k-block j of the chunk whose row bytes start at shared address `row`; v[i] holds weights 2 i, 2 i + 1.
// WS: see load_words (the word offset of the quants, the same for the whole warp, or -1).
// `valid`: 32-weight blocks of the k-block that exist (32-weight formats; the others always have both).
template <int FMT, int WS>
__device__ __forceinline__ void decode_row(uint32_t row, int j, int valid, uint32_t (&v)[32]) {
  if constexpr (FMT == kQ4_K) {
    const uint4 hdr = ptx::lds128(row);
    const uint4 q0 = ptx::lds128(row + 16 + 32 * j), q1 = ptx::lds128(row + 32 + 32 * j);
    const float d = half_bits(hdr.x & 0xFFFFu), dmin = half_bits(hdr.x >> 16);
    const bool upper = j >= 2;  // the same for the whole warp
    const int sh = 16 * (j & 1);
    const uint32_t sc4 = upper ? ((hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u)) : (hdr.y & 0x3F3F3F3Fu);
    const uint32_t mn4 = upper ? (((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u)) : (hdr.z & 0x3F3F3F3Fu);
    const uint32_t sc = sc4 >> sh, mn = mn4 >> sh;
    const float ml = -(dmin * (float)(mn & 0xFFu)), mh = -(dmin * (float)((mn >> 8) & 0xFFu));
    const float sl = d * (float)(sc & 0xFFu), sg = d * (float)((sc >> 8) & 0xFFu) * 0.0625f;
    const uint64_t s_lo = pack2(sl, sl), s_hi = pack2(sg, sg), off_lo = pack2(ml, ml), off_hi = pack2(mh, mh);
    const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const NibbleHalves w = nibble_halves(words[i]);
      v[2 * i] = bf16x2(fma2(s_lo, pair_f32(w.lo02, w.lo13, false, -1024.f), off_lo));
      v[2 * i + 1] = bf16x2(fma2(s_lo, pair_f32(w.lo02, w.lo13, true, -1024.f), off_lo));
      v[16 + 2 * i] = bf16x2(fma2(s_hi, pair_f32(w.hi02, w.hi13, false, -1024.f), off_hi));
      v[16 + 2 * i + 1] = bf16x2(fma2(s_hi, pair_f32(w.hi02, w.hi13, true, -1024.f), off_hi));
    }
  } else if constexpr (FMT == kQ6_K) {
    const int h = j >> 1;
    uint32_t ql[16], qh[8];
    load_words<16, WS, true>(row + 64 * h, ql);
    load_words<8, WS, true>(row + 128 + 32 * h, qh);
    const uint32_t s01 = lds_u16(row + 192 + 4 * j), s23 = lds_u16(row + 194 + 4 * j);
    const float d = half_bits(lds_u16(row + 208));
    float s[4];
    s[0] = d * (float)(int)(int8_t)(s01 & 0xFFu);
    s[1] = d * (float)(int)(int8_t)(s01 >> 8);
    s[2] = d * (float)(int)(int8_t)(s23 & 0xFFu);
    s[3] = d * (float)(int)(int8_t)(s23 >> 8);
    const bool odd = j & 1;  // high nibbles and the upper bit pairs (the same for the whole warp)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t ha = odd ? qh[i] : qh[i] << 4, hb = odd ? qh[i] >> 2 : qh[i] << 2;
      const uint32_t qa = and_or(odd ? ql[i] >> 4 : ql[i], 0x0F0F0F0Fu, ha & 0x30303030u);
      const uint32_t qb = and_or(odd ? ql[8 + i] >> 4 : ql[8 + i], 0x0F0F0F0Fu, hb & 0x30303030u);
      const uint2 a = bytes_to_bf16(qa, -1056.f, pack2(s[i >> 2], s[i >> 2]));  // 1024 + 32
      const uint2 b = bytes_to_bf16(qb, -1056.f, pack2(s[2 + (i >> 2)], s[2 + (i >> 2)]));
      v[2 * i] = a.x, v[2 * i + 1] = a.y;
      v[16 + 2 * i] = b.x, v[16 + 2 * i + 1] = b.y;
    }
  } else if constexpr (FMT == kQ8_0) {
    uint32_t w[17];  // fp16 d, 32 bytes, fp16 d, 32 bytes
    load_words<17, WS, (WS < 0)>(row + 68 * j, w);
    const float d0 = half_bits(w[0] & 0xFFFFu), d1 = half_bits(w[8] >> 16);
    const uint64_t s0 = pack2(d0, d0), s1 = pack2(d1, d1);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint2 a = bytes_to_bf16(__funnelshift_r(w[i], w[i + 1], 16) ^ 0x80808080u, -1152.f, s0);  // 1024 + 128
      const uint2 b = bytes_to_bf16(w[9 + i] ^ 0x80808080u, -1152.f, s1);
      v[2 * i] = a.x, v[2 * i + 1] = a.y;
      v[16 + 2 * i] = b.x, v[16 + 2 * i + 1] = b.y;
    }
  } else {
    uint32_t w[9];  // fp16 d, 16 bytes, fp16 d, 16 bytes; low nibbles are weights 0..15 of a block, high ones 16..31
    load_words<9, WS, (WS < 0)>(row + 36 * j, w);
    const float d0 = half_bits(w[0] & 0xFFFFu), d1 = half_bits(w[4] >> 16);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const float d = b ? d1 : d0, dh = d * 0.0625f;
      const uint64_t s_lo = pack2(d, d), s_hi = pack2(dh, dh);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const NibbleHalves q = nibble_halves(b ? w[5 + i] : __funnelshift_r(w[i], w[i + 1], 16));
        v[16 * b + 2 * i] = bf16x2(mul2(pair_f32(q.lo02, q.lo13, false, -1032.f), s_lo));           // 1024 + 8
        v[16 * b + 2 * i + 1] = bf16x2(mul2(pair_f32(q.lo02, q.lo13, true, -1032.f), s_lo));
        v[16 * b + 8 + 2 * i] = bf16x2(mul2(pair_f32(q.hi02, q.hi13, false, -1152.f), s_hi));       // 1024 + 16 * 8
        v[16 * b + 8 + 2 * i + 1] = bf16x2(mul2(pair_f32(q.hi02, q.hi13, true, -1152.f), s_hi));
      }
    }
  }
  if constexpr (FMT == kQ8_0 || FMT == kQ4_0) {
    if (valid < 2) {  // past the end of K: zeros (the bytes there belong to no block)
#pragma unroll
      for (int i = 0; i < 16; ++i) v[16 + i] = 0u;
      if (valid < 1)
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0u;
    }
  }
}
// `skew`: bytes of the row in front of the chunk's first (16-byte granules are copied).
template <int FMT>
__device__ __forceinline__ void decode_chunk_row(uint32_t row, uint32_t skew, bool tiled, int j, int valid, uint32_t (&v)[32]) {
  if constexpr (FMT == kQ4_K) {
    decode_row<FMT, 0>(row, j, valid, v);
  } else {
    const int ws = FMT == kQ6_K ? (int)(skew >> 2) : j;  // 68 j and 36 j are 4 j past a 16-byte boundary
    if (!tiled) decode_row<FMT, -1>(row + skew, j, valid, v);
    else if (ws == 0) decode_row<FMT, 0>(row + skew, j, valid, v);
    else if (ws == 1) decode_row<FMT, 1>(row + skew, j, valid, v);
    else if (ws == 2) decode_row<FMT, 2>(row + skew, j, valid, v);
    else decode_row<FMT, 3>(row + skew, j, valid, v);
  }
}

template <int FMT>
__global__ void __launch_bounds__(threads_of<FMT>(), 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const PairArgs a) {
  using R = RawCfg<FMT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* b_tiles = smem;  // (128-byte swizzle: 1024-byte aligned)
  uint8_t* raw_tiles = smem + a.b_stages * a.b_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kRing);
  uint64_t* full_a = bars;                        // decoded weights of a stage are in place in both CTAs (first CTA)
  uint64_t* empty_a = full_a + kMaxAStages;       // the MMAs that read it are done (both CTAs)
  uint64_t* full_b = empty_a + kMaxAStages;       // activations of both CTAs have landed (first CTA)
  uint64_t* empty_b = full_b + kMaxBStages;       // the MMAs that read them are done (both CTAs)
  uint64_t* raw_full = empty_b + kMaxBStages;     // raw chunk has landed
  uint64_t* raw_empty = raw_full + kMaxRawStages;
  uint64_t* acc_full = raw_empty + kMaxRawStages;  // [2] an accumulator set (kFp32Sums: pair of sets) is complete (both CTAs)
  uint64_t* acc_empty = acc_full + 2;              // [2] both CTAs have drained it (first CTA)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  uint32_t* late = tmem_slot + 2;  // [kGroups][2], see GroupWait
  volatile uint32_t* gave_up = tmem_slot + 1;  // some wait of this CTA has run out (read once all its warps are through)
  static_assert((2 * kMaxAStages + 2 * kMaxBStages + 2 * kMaxRawStages + 4) * 8 + 8 + 8 * kGroups <= kBarrierBytes, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();      // CTA of the cluster
  const uint32_t half = rank & 1;            // CTA of the pair
  const uint32_t leader = rank & ~1u;
  const int split = (int)(rank >> 1);
  const int cluster_ctas = 2 * a.splits;
  const int cluster = (int)blockIdx.x / cluster_ctas, clusters = (int)gridDim.x / cluster_ctas;
  const int c0 = (int)((long long)split * a.chunks / a.splits), c1 = (int)((long long)(split + 1) * a.chunks / a.splits);
  const int k_blocks = (a.k + kBlockK - 1) / kBlockK;
  const int kb0 = 4 * c0, kb1 = min(4 * c1, k_blocks), kbs = kb1 - kb0;
  const int T = a.tokens;
  const int a_mask = (1 << a.a_log) - 1;
  constexpr int kThreads = threads_of<FMT>();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxAStages; ++s) {
      ptx::mbar_init(&full_a[s], 2 * 4);  // four decode warps of each CTA
      ptx::mbar_init(&empty_a[s], 1);
    }
    for (int s = 0; s < kMaxBStages; ++s) {
      ptx::mbar_init(&full_b[s], 1);
      ptx::mbar_init(&empty_b[s], 1);
    }
    for (int s = 0; s < kMaxRawStages; ++s) {
      ptx::mbar_init(&raw_full[s], a.tiled ? 1 : 64);
      ptx::mbar_init(&raw_empty[s], 16);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&acc_full[b], 1);
      ptx::mbar_init(&acc_empty[b], 2 * (kFp32Sums<FMT> ? 8 : 4));
    }
    for (int i = 0; i < 2 * kGroups; ++i) late[i] = 0u;
    *gave_up = 0u;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_x);
    if (a.tiled) ptx::prefetch_tensormap(&map_w);
    ptx::grid_launch_dependents();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(ptx::smem_addr(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  ptx::tc_fence_before();
  __syncthreads();
  cluster_sync();  // the peers' barriers are initialised before anything arrives at them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_a = tmem_base + (uint32_t)(a.acc_sets * T);

  // Waits that can only end once the activations are there start after grid_dependency_wait(): the kernel before may
  // run for longer than their limit.
  if (warp == 0) {
    // ---------------- TMA producer: this CTA's half of the tile's tokens ----------------
    if (elect_one()) {
      ptx::grid_dependency_wait();  // activations may come from the kernel before
      const uint32_t full_leader = map_rank(ptx::smem_addr(full_b), leader);
      const int group = a.b_stages >= 12 ? 4 : (a.b_stages >= 6 ? 2 : 1);  // k-blocks per wait
      int s = 0;
      uint32_t parity = 1;  // (waits on an unused stage pass at once)
      bool ok = true;
      for (int tile = cluster; tile < a.tiles && ok; tile += clusters) {
        const int tok0 = (tile % a.token_tiles) * T + (int)half * (T / 2);
        for (int kb = kb0; kb < kb1; kb += group) {
          // stages are given back in order: the last one of the group is free when all are
          const int count = min(group, kb1 - kb);
          int last = s + count - 1;
          const uint32_t last_parity = last >= a.b_stages ? parity ^ 1 : parity;
          if (last >= a.b_stages) last -= a.b_stages;
          if (!wait_bar(&empty_b[last], last_parity)) {
            report_timeout(0x10000u | (unsigned)kb);
            *gave_up = 1u;
            ok = false;
            break;
          }
          for (int i = 0; i < count; ++i) {
            if (half == 0) ptx::mbar_arrive_expect_tx(&full_b[s], 2u * (uint32_t)a.b_bytes);
            tma_load_pair(b_tiles + s * a.b_bytes, &map_x, (kb + i) * kBlockK, tok0, full_leader + 8u * (uint32_t)s);
            if (++s == a.b_stages) s = 0, parity ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer of the pair ----------------
    if (half == 0 && elect_one()) {
      ptx::grid_dependency_wait();
      // kind::f16: fp32 accumulate, bf16 x bf16, both K-major, M = 256, N = T
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(T >> 3) << 17) | ((uint32_t)(kPairRows >> 4) << 24);
      const uint16_t mask = (uint16_t)(3u << leader);
      const uint32_t fa = ptx::smem_addr(full_a), fb = ptx::smem_addr(full_b);
      int seq = 0, s = 0, t = 0;
      uint32_t parity = 0;
      bool ok = true;
      if constexpr (kFp32Sums<FMT>) {
        const uint32_t ae = ptx::smem_addr(acc_empty);
        for (int tile = cluster; tile < a.tiles && ok; tile += clusters) {
          for (int kb = kb0; kb < kb1; kb += 2, ++t) {
            // two k-blocks at a time (an odd last one twice), each into an accumulator set of its own
            const int count = min(2, kb1 - kb), seq1 = seq + count - 1, pair = t & 1;
            const int s0 = s, s1 = count == 2 ? (s + 1 == a.b_stages ? 0 : s + 1) : s;
            const uint32_t parity1 = s1 < s0 ? parity ^ 1 : parity;
            const int a0 = seq & a_mask, a1 = seq1 & a_mask;
            const uint32_t bar[5] = {fb + 8u * (uint32_t)s0, fa + 8u * (uint32_t)a0, fb + 8u * (uint32_t)s1, fa + 8u * (uint32_t)a1,
                                     ae + 8u * (uint32_t)pair};
            const uint32_t par[5] = {parity, (uint32_t)(seq >> a.a_log) & 1u, parity1, (uint32_t)(seq1 >> a.a_log) & 1u,
                                     ((uint32_t)(t >> 1) & 1u) ^ 1u};
            if (!wait_all(bar, par)) {
              report_timeout(0x20000u | (unsigned)kb);
              *gave_up = 1u;
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const uint32_t d = tmem_base + (uint32_t)(2 * pair * T);
            uint64_t b_desc = smem_desc_sw128(ptx::smem_addr(b_tiles + s0 * a.b_bytes));
#pragma unroll
            for (int i = 0; i < kBlockK / 16; ++i)
              umma_pair(d, tmem_a + 32u * (uint32_t)a0 + 8u * i, b_desc + 2 * i, idesc, i ? 1u : 0u);
            commit_pair(&empty_a[a0], mask);
            commit_pair(&empty_b[s0], mask);
            if (count == 2) {
              b_desc = smem_desc_sw128(ptx::smem_addr(b_tiles + s1 * a.b_bytes));
#pragma unroll
              for (int i = 0; i < kBlockK / 16; ++i)
                umma_pair(d + (uint32_t)T, tmem_a + 32u * (uint32_t)a1 + 8u * i, b_desc + 2 * i, idesc, i ? 1u : 0u);
              commit_pair(&empty_a[a1], mask);
              commit_pair(&empty_b[s1], mask);
            }
            commit_pair(&acc_full[pair], mask);
            seq += count;
            s = s1 + 1 == a.b_stages ? 0 : s1 + 1;
            parity = s1 + 1 == a.b_stages ? parity1 ^ 1 : parity1;
          }
        }
      } else {
        for (int tile = cluster; tile < a.tiles && ok; tile += clusters, ++t) {
          const int b = a.acc_sets == 2 ? (t & 1) : 0, use = a.acc_sets == 2 ? (t >> 1) : t;
          if (!wait_bar(&acc_empty[b], (use & 1) ^ 1)) {
            report_timeout(0x50000u | (unsigned)t);
            *gave_up = 1u;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t d = tmem_base + (uint32_t)(b * T);
          for (int kb = kb0; kb < kb1; kb += 2) {
            // two k-blocks at a time (an odd last one twice)
            const int count = min(2, kb1 - kb), seq1 = seq + count - 1;
            const int s0 = s, s1 = count == 2 ? (s + 1 == a.b_stages ? 0 : s + 1) : s;
            const uint32_t parity1 = s1 < s0 ? parity ^ 1 : parity;
            const int a0 = seq & a_mask, a1 = seq1 & a_mask;
            const uint32_t bar[4] = {fb + 8u * (uint32_t)s0, fa + 8u * (uint32_t)a0, fb + 8u * (uint32_t)s1, fa + 8u * (uint32_t)a1};
            const uint32_t par[4] = {parity, (uint32_t)(seq >> a.a_log) & 1u, parity1, (uint32_t)(seq1 >> a.a_log) & 1u};
            if (!wait_all(bar, par)) {
              report_timeout(0x20000u | (unsigned)kb);
              *gave_up = 1u;
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            {
              const uint64_t b_desc = smem_desc_sw128(ptx::smem_addr(b_tiles + s0 * a.b_bytes));
  #pragma unroll
              for (int i = 0; i < kBlockK / 16; ++i)
                umma_pair(d, tmem_a + 32u * (uint32_t)a0 + 8u * i, b_desc + 2 * i, idesc, (kb > kb0 || i) ? 1u : 0u);
              commit_pair(&empty_a[a0], mask);
              commit_pair(&empty_b[s0], mask);
            }
            if (count == 2) {
              const uint64_t b_desc = smem_desc_sw128(ptx::smem_addr(b_tiles + s1 * a.b_bytes));
  #pragma unroll
              for (int i = 0; i < kBlockK / 16; ++i)
                umma_pair(d, tmem_a + 32u * (uint32_t)a1 + 8u * i, b_desc + 2 * i, idesc, 1u);
              commit_pair(&empty_a[a1], mask);
              commit_pair(&empty_b[s1], mask);
            }
            seq += count;
            s = s1 + 1 == a.b_stages ? 0 : s1 + 1;
            parity = s1 + 1 == a.b_stages ? parity1 ^ 1 : parity1;
          }
          commit_pair(&acc_full[b], mask);
        }
      }
    }
  } else if (warp == 2 || (warp == 3 && !a.tiled)) {
    // ---------------- raw weight producers ----------------
    int s = 0, it = 0;
    uint32_t parity = 1;
    bool ok = true;
    for (int tile = cluster; tile < a.tiles && ok; tile += clusters) {
      const int row0 = (tile / a.token_tiles) * kPairRows + (int)half * kCtaRows;
      for (int c = c0; c < c1; ++c, ++it) {
        if (it == a.raw_stages) ptx::grid_dependency_wait();
        if (!wait_bar(&raw_empty[s], parity)) {
          report_timeout(0x60000u | (unsigned)c);
          *gave_up = 1u;
          ok = false;
          break;
        }
        uint8_t* dst = raw_tiles + s * a.raw_bytes;
        uint64_t* bar = &raw_full[s];
        if (++s == a.raw_stages) s = 0, parity ^= 1;
        if (a.tiled) {
          // rows past N and bytes past a row's end arrive as zeros and count towards the transaction bytes; the copy
          // starts on the 16-byte boundary at or below the chunk (8-byte words: an even coordinate)
          if (elect_one()) {
            ptx::mbar_arrive_expect_tx(bar, kCtaRows * R::kPitch);
            ptx::tma_load_2d(dst, &map_w, ((c * R::kBytes) & ~15) >> 3, row0, bar);
          }
          continue;
        }
        // rows of any 2-byte alignment: the 16-byte granules around a row's bytes, eight lanes a row, 64 rows a warp (one
        // bulk copy per row took 70 clocks each, 9000 a chunk); the weight's last granule is read up to its end only
        const int row_len = (int)min((long long)R::kBytes, a.row_bytes - (long long)c * R::kBytes);
        const int r0 = 64 * (warp - 2) + (lane >> 3), g0 = lane & 7;
        long long first = (long long)(row0 + r0) * a.row_bytes + (long long)c * R::kBytes;
        uint32_t to = ptx::smem_addr(dst) + (uint32_t)(r0 * R::kRowPitch);
        const int rows = a.n - row0 - r0;  // of this lane's sequence, four apart
#pragma unroll 4
        for (int i = 0; i < 16; ++i, first += 4 * a.row_bytes, to += 4 * R::kRowPitch) {
          if (4 * i >= rows) break;
          const long long begin = first & ~15ll;
          const int granules = (int)(first - begin + row_len + 15) >> 4;
#pragma unroll
          for (int g = g0; g < R::kRowPitch / 16 + 7; g += 8) {
            if (g < granules) {
              const long long at = begin + 16 * g;
              const int bytes = (int)min(16ll, a.w_bytes - at);
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + 16u * (uint32_t)g), "l"(a.w + at), "r"(bytes)
                           : "memory");
            }
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(ptx::smem_addr(bar)) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= kDecodeWarp0 && warp < kDecodeWarp0 + kDecodeWarps) {
    // ---------------- decode ----------------
    const int j = (warp - kDecodeWarp0) >> 2;                     // k-block of every chunk
    const int r = (warp & 3) * 32 + lane;                         // row of this CTA's half of the tile = TMEM lane
    const uint32_t full_leader = map_rank(ptx::smem_addr(full_a), leader);
    const uint32_t tmem_row = tmem_a + ((uint32_t)((warp & 3) * 32) << 16);
    GroupWait group{ptx::smem_addr(late + 2 * j), j};
    int s = 0, base = 0;
    uint32_t parity = 0;
    bool ok = true;
    for (int tile = cluster; tile < a.tiles && ok; tile += clusters, base += kbs) {
      const long long row = (long long)(tile / a.token_tiles) * kPairRows + (int)half * kCtaRows + r;
      for (int c = c0; c < c1; ++c) {
        const int kb = 4 * c + j, seq = base + kb - kb0, sa = seq & a_mask;
        const bool live = kb < kb1;
        if (seq > a_mask && (seq >> a.a_log) == 1) ptx::grid_dependency_wait();  // (returns at once after the first time)
        const uint32_t a_parity = ((seq >> a.a_log) & 1) ^ 1;
        // with two stages of its own a group asks for the raw bytes and the stage in one go (T = 128, Q6_K: 265 -> 249 us
        // at M = 2048, N = 12288, K = 4096); with one the stage is waited for after the decode
        const bool together = live && a.a_log == 3;
        if (together ? !group.two(&raw_full[s], parity, &empty_a[sa], a_parity) : !group.one(&raw_full[s], parity)) {
          report_timeout(0x70000u | (unsigned)c);
          *gave_up = 1u;
          ok = false;
          break;
        }
        uint32_t v[32];
        if (live) {
          const uint32_t skew = a.tiled ? (uint32_t)(c * R::kBytes) & 15u
                                        : (uint32_t)(row * a.row_bytes + (long long)c * R::kBytes) & 15u;
          decode_chunk_row<FMT>(ptx::smem_addr(raw_tiles + s * a.raw_bytes) + (uint32_t)(r * a.pitch), skew, a.tiled != 0, j,
                                (a.k - kb * kBlockK + 31) >> 5, v);
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&raw_empty[s]);  // the row's bytes are in registers
        if (++s == a.raw_stages) s = 0, parity ^= 1;
        if (!live) continue;
        if (!together && !group.one(&empty_a[sa], a_parity)) {
          report_timeout(0x30000u | (unsigned)kb);
          *gave_up = 1u;
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        tmem_st_32(tmem_row + 32u * (uint32_t)sa, v);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_remote(full_leader + 8u * (uint32_t)sa);
      }
    }
  } else if (kFp32Sums<FMT> && warp >= 4) {
    // ---------------- drain: two k-blocks' products at a time, half of the token columns a group of four warps ----------
    ptx::grid_dependency_wait();  // the kernel before may still read or write the output
    const int quarter = warp & 3, id = warp < kDecodeWarp0 ? 4 : 5, col0 = id == 4 ? 0 : T / 2;
    GroupWait group{ptx::smem_addr(late + 2 * id), id};
    const uint32_t products = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col0;
    const uint32_t sums = ptx::smem_addr(smem) + (uint32_t)(kRing - kSumBytes + (col0 * kCtaRows + quarter * 32 + lane) * 4);
    const uint32_t release = map_rank(ptx::smem_addr(acc_empty), leader);
    constexpr int kParts = max_tokens<FMT>() / 32;
    int t = 0;
    bool ok = true;
    for (int tile = cluster; tile < a.tiles && ok; tile += clusters) {
      const int n = (tile / a.token_tiles) * kPairRows + (int)half * kCtaRows + quarter * 32 + lane;
      const int tok = (tile % a.token_tiles) * T + col0;
      const int cols = min(T / 2, a.m - tok);  // (none left: these warps keep the others company)
      float sum[kParts][16];
      for (int i = 0; i < kbs; i += 2, ++t) {
        const int pair = t & 1;
        if (!group.one(&acc_full[pair], (uint32_t)(t >> 1) & 1u)) {
          report_timeout(0x40000u);
          *gave_up = 1u;
          ok = false;
          break;
        }
        ptx::tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (i + h == kbs) break;
          const bool fresh = h == 0 && i % kInnerSums == 0;
#pragma unroll
          for (int c = 0; c < kParts; ++c)
            if (16 * c < cols) {
              uint32_t p[16];
              tmem_ld_16(products + (uint32_t)((2 * pair + h) * T + 16 * c), p);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) sum[c][j] = (fresh ? 0.f : sum[c][j]) + __uint_as_float(p[j]);
            }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_remote(release + 8u * (uint32_t)pair);
        if (i + 2 < kbs && (i + 2) % kInnerSums) continue;
#pragma unroll
        for (int c = 0; c < kParts; ++c)
          if (16 * c < cols) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const uint32_t at = sums + (uint32_t)((16 * c + j) * kCtaRows * 4);
              if (i >= kInnerSums) {
                float before;
                asm volatile("ld.shared.f32 %0, [%1];" : "=f"(before) : "r"(at));
                sum[c][j] += before;
              }
              if (i + 2 < kbs) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(sum[c][j]) : "memory");
            }
          }
      }
      if (!ok) break;
      if (a.splits > 1) {
        // into the stages, which no MMA reads any more
        float* part = reinterpret_cast<float*>(smem) + col0 * kCtaRows + quarter * 32 + lane;  // [tokens][128 rows]
#pragma unroll
        for (int c = 0; c < kParts; ++c)
          if (16 * c < cols)
#pragma unroll
            for (int j = 0; j < 16; ++j) part[(16 * c + j) * kCtaRows] = sum[c][j];
      } else if (n < a.n) {
        float* o = a.out + (long long)tok * a.n + n;
#pragma unroll
        for (int c = 0; c < kParts; ++c)
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (16 * c + j < cols) *o = sum[c][j];
            o += a.n;
            asm volatile("" : "+l"(o));  // (else the compiler keeps 32 addresses in registers through the loop above)
          }
      }
    }
  } else if (!kFp32Sums<FMT> && warp >= 4 && a.splits == 1) {
    // ---------------- epilogue: the accumulators of one tile while the next one's are being filled ----------------
    ptx::grid_dependency_wait();  // the kernel before may still read or write the output
    const int quarter = warp & 3;
    GroupWait group{ptx::smem_addr(late + 2 * 4), 4};
    int t = 0;
    for (int tile = cluster; tile < a.tiles; tile += clusters, ++t) {
      const int b = a.acc_sets == 2 ? (t & 1) : 0, use = a.acc_sets == 2 ? (t >> 1) : t;
      if (!group.one(&acc_full[b], use & 1)) {
        report_timeout(0x40000u);
        *gave_up = 1u;
        break;
      }
      ptx::tc_fence_after();
      const int n = (tile / a.token_tiles) * kPairRows + (int)half * kCtaRows + quarter * 32 + lane;
      const int tok0 = (tile % a.token_tiles) * T, tok_end = min(T, a.m - tok0);
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * T);
      float* o = a.out + (long long)tok0 * a.n + n;
      for (int col = 0; col < tok_end; col += 16) {
        uint32_t acc[16];
        tmem_ld_16(taddr + (uint32_t)col, acc);
        ptx::tmem_ld_wait();
        if (n < a.n) {
          if (col + 16 <= tok_end) {
#pragma unroll
            for (int i = 0; i < 16; ++i) o[(long long)(col + i) * a.n] = __uint_as_float(acc[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (col + i < tok_end) o[(long long)(col + i) * a.n] = __uint_as_float(acc[i]);
          }
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_remote(map_rank(ptx::smem_addr(&acc_empty[b]), leader));
    }
  }
  if (a.splits > 1) {
    // ---------------- K split over the pairs of this cluster (one tile per cluster) ----------------
    // Every CTA lays its accumulators out in its stages, which no MMA reads any more; then each pair adds its share of
    // the token columns over all pairs, in K order.
    const int tile = cluster;
    const int tok0 = (tile % a.token_tiles) * T, tok_end = min(T, a.m - tok0);
    float* part = reinterpret_cast<float*>(smem);  // [tokens][128 rows]
    __syncwarp();
    if (!kFp32Sums<FMT> && warp >= 4 && warp < 8) {
      ptx::grid_dependency_wait();
      const int quarter = warp & 3;
      if (!GroupWait{ptx::smem_addr(late + 2 * 4), 4}.one(&acc_full[0], 0)) {
        report_timeout(0x40000u);
        *gave_up = 1u;
      } else {
        ptx::tc_fence_after();
        for (int col = 0; col < tok_end; col += 16) {
          uint32_t acc[16];
          tmem_ld_16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col, acc);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) part[(col + i) * kCtaRows + quarter * 32 + lane] = __uint_as_float(acc[i]);
        }
        ptx::tc_fence_before();
      }
    }
    __syncwarp();
    cluster_sync();
    ptx::grid_dependency_wait();
    const int row0 = (tile / a.token_tiles) * kPairRows + (int)half * kCtaRows;
    const int first = split * tok_end / a.splits, last = (split + 1) * tok_end / a.splits;
    uint32_t src[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) src[p] = map_rank(ptx::smem_addr(part), (uint32_t)(2 * min(p, a.splits - 1)) + half);
    for (int i = first * kCtaRows + (int)threadIdx.x; i < last * kCtaRows; i += kThreads) {
      float v = ld_cluster_f32(src[0] + 4u * (uint32_t)i);
#pragma unroll
      for (int p = 1; p < 4; ++p)
        if (p < a.splits) v += ld_cluster_f32(src[p] + 4u * (uint32_t)i);
      const int n = row0 + (i & (kCtaRows - 1));
      if (n < a.n) a.out[(long long)(tok0 + i / kCtaRows) * a.n + n] = v;
    }
  }
  __syncwarp();
  ptx::tc_fence_before();
  __syncthreads();
  if (*gave_up) {
    // copies and MMAs still in flight get 50 us to end before the memory is given back, in both CTAs of the pair
    const uint64_t start = ptx::global_timer_ns();
    while (ptx::global_timer_ns() - start < 50000ull) __nanosleep(1000);
    __syncwarp();
  }
  cluster_sync();  // nobody may still arrive at, or read, a CTA that has left
  if (warp == 1) {
    ptx::tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

// ---- host side ----------------------------------------------------------------------------------------------------

// Clusters of `ctas` CTAs that the device holds at once (one CTA per SM); found once per device.
template <int FMT>
int resident_clusters(int splits, const DeviceInfo& dev) {
  static int known[64][3];  // [device][log2 splits], 0 = not asked yet (a race writes the same number twice)
  const int slot = splits == 1 ? 0 : (splits == 2 ? 1 : 2);
  int& entry = known[dev.ordinal & 63][slot];
  if (entry > 0) return entry;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(dev.sm_count / (2 * splits) * 2 * splits));
  cfg.blockDim = dim3(threads_of<FMT>());
  cfg.dynamicSmemBytes = kSmemLimit;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int count = 0;
  if (cudaOccupancyMaxActiveClusters(&count, gemm_pair_kernel<FMT>, &cfg) != cudaSuccess || count < 1) {
    cudaGetLastError();
    count = std::max(1, dev.sm_count / (2 * splits) - splits);
  }
  entry = count;
  return count;
}

// Two accumulator sets (four of 64 columns with fp32 sums) where four decoded stages fit beside them in tensor memory,
// eight stages where they do (log2).
int accumulator_sets(int fmt, int tokens) { return fmt == kQ8_0 || fmt == kQ4_0 ? kSumSets : tokens <= 192 ? 2 : 1; }
int decoded_log(int fmt, int tokens) { return accumulator_sets(fmt, tokens) * tokens <= 256 ? 3 : 2; }

constexpr long long kMaxTiles = 0x3fffffff;

struct PairPlan {
  int tokens, splits, clusters, tiles, token_tiles;
};

// Tokens per tile and pairs along K by a cost model in SM clocks.  A k-block of 64 costs its MMAs (2 T clocks) or its
// decode (128 rows x 64 weights by 16 warps, each with its waits), whichever is longer, and a little of the other
// (measured at N = 12288, K = 4096, M = 2048: clocks per k-block at T = 128 / 192 / 256 are 550 / 620 / 515 + epilogue
// for Q4_K, 680 / 770 / 600 for Q6_K; for the formats with fp32 sums what the drain costs is in it); above T = 192 one accumulator set leaves the epilogue exposed.  A tile adds its fill
// and drain, a K split the exchange of accumulators.  Tiles go out in rounds of as many clusters as the device holds,
// so a narrower T pays where it fills the last round better.
//
// A decode group takes every fourth k-block of a tile and begins the next tile where it left off, so that its k-blocks are
// up to 4 + r apart where r = k-blocks of a tile mod 4.  It waits for a decoded stage by the parity of the stage's laps,
// which says nothing of a stage a whole lap behind: with four stages (T = 160, 192) and r > 0 the group could write a
// stage that has not been read yet.  Such K take a T with eight stages there, unless a cluster has one tile only.
template <int FMT>
PairPlan plan_pair(long long m, long long n, long long k, const DeviceInfo& dev) {
  const int decode = FMT == kQ4_K ? 500 : FMT == kQ6_K ? 650 : FMT == kQ8_0 ? 730 : 710;
  const long long row_tiles = (n + kPairRows - 1) / kPairRows;
  const int chunks = (int)((k + kChunkK - 1) / kChunkK);
  const bool every_fourth = (k + kBlockK - 1) / kBlockK % 4 == 0;
  PairPlan best{};
  double best_cost = 1e300;
  for (int t = 32; t <= max_tokens<FMT>(); t += 32) {
    if (t > 32 && t - 32 >= m) break;
    const long long token_tiles = (m + t - 1) / t, tiles = token_tiles * row_tiles;
    if (tiles > kMaxTiles) continue;
    const double per_block = t > 192 ? std::max(2.0 * t, decode + 50.0) : decode + 0.6 * std::max(0, 2 * t - 200);
    for (int s = 1; s <= 4; s *= 2) {
      if (s > 1 && (s > chunks || tiles * s > dev.sm_count / 2)) break;
      const int resident = resident_clusters<FMT>(s, dev);
      if (!every_fourth && s == 1 && tiles > resident && decoded_log(FMT, t) == 2) continue;
      const long long rounds = (tiles + resident - 1) / resident;
      const double blocks = 4.0 * ((chunks + s - 1) / s);
      const double tile_cost = blocks * per_block + (s > 1 ? 1500.0 + 12.0 * t : t > 192 ? 42.0 * t : 300.0);
      const double cost = 3000.0 + rounds * tile_cost + (t > 192 && s == 1 ? 0.0 : 16.0 * t);
      if (cost < best_cost) {
        best_cost = cost;
        best.tokens = t;
        best.splits = s;
        best.token_tiles = (int)token_tiles;
        best.tiles = (int)tiles;
        best.clusters = s > 1 ? (int)tiles : (int)std::min<long long>(tiles, resident);
      }
    }
  }
  return best;
}

template <int FMT>
cudaError_t launch_pair(const void* x, const uint8_t* w, float* out, long long m, long long n, long long k,
                        cudaStream_t stream, const char** detail) {
  using R = RawCfg<FMT>;
  cudaError_t e;
  const DeviceInfo* dev = device_info(&e);
  if (!dev) return e;
  auto kernel = gemm_pair_kernel<FMT>;
  e = allow_full_shared_memory(kernel);
  if (e != cudaSuccess) return e;
  const PairPlan plan = plan_pair<FMT>(m, n, k, *dev);
  PairArgs a{};
  a.w = w;
  a.out = out;
  a.row_bytes = row_bytes(FMT, k);
  a.w_bytes = a.row_bytes * n;
  a.m = (int)m;
  a.n = (int)n;
  a.k = (int)k;
  a.tokens = plan.tokens;
  a.token_tiles = plan.token_tiles;
  a.tiles = plan.tiles;
  a.splits = plan.splits;
  a.chunks = (int)((k + kChunkK - 1) / kChunkK);
  a.tiled = a.row_bytes % 16 == 0;
  a.acc_sets = accumulator_sets(FMT, plan.tokens);
  a.a_log = decoded_log(FMT, plan.tokens);
  a.b_bytes = plan.tokens / 2 * kBlockK * 2;
  a.pitch = a.tiled ? R::kPitch : R::kRowPitch;
  a.raw_bytes = kCtaRows * a.pitch;
  a.raw_stages = R::kStages;
  a.b_stages = std::min(kMaxBStages, (kRing - (kFp32Sums<FMT> ? kSumBytes : 0) - a.raw_stages * a.raw_bytes) / a.b_bytes);
  alignas(64) CUtensorMap map_x, map_w{};
  // tokens past m and columns past k read as zero
  bool ok = make_tensor_map_2d(&map_x, TmaType::kBF16, x, (unsigned long long)k, (unsigned long long)m,
                               (unsigned long long)k * 2, kBlockK, (unsigned)(plan.tokens / 2), true);
  if (ok && a.tiled)
    ok = make_tensor_map_2d(&map_w, TmaType::kU64, w, (unsigned long long)(a.row_bytes / 8), (unsigned long long)n,
                            (unsigned long long)a.row_bytes, R::kPitch / 8, kCtaRows, false);
  if (!ok) {
    if (detail) *detail = "cuTensorMapEncodeTiled is unavailable or rejected the layout";
    return cudaErrorNotSupported;
  }
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * plan.splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(plan.clusters * 2 * plan.splits));
  cfg.blockDim = dim3(threads_of<FMT>());
  cfg.dynamicSmemBytes = kSmemLimit;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, map_x, map_w, a);
}

}  // namespace

TB200_DEFINE_STATUS_READER(read_gemm_pair_status)

bool gemm_pair_supported(int fmt, long long m, long long n, long long k, const DeviceInfo& dev) {
  if (!valid_format(fmt) || m < 1 || n < 1 || k < block_weights(fmt) || k % block_weights(fmt)) return false;
  if (m > (1 << 24) || n > (1 << 24) || k > (1 << 24)) return false;
  // (the planner has nothing to offer above so many of the largest tiles)
  const long long tokens = fmt == kQ8_0 || fmt == kQ4_0 ? kMaxTokensFp32 : kMaxTokens;
  if ((m + tokens - 1) / tokens * ((n + kPairRows - 1) / kPairRows) > kMaxTiles) return false;
  return dev.max_smem_optin >= kSmemLimit;
}

void gemm_pair_plan(int fmt, long long m, long long n, long long k, const DeviceInfo& dev, int* out8) {
  const PairPlan plan = fmt == kQ4_0   ? plan_pair<kQ4_0>(m, n, k, dev)
                        : fmt == kQ8_0 ? plan_pair<kQ8_0>(m, n, k, dev)
                        : fmt == kQ4_K ? plan_pair<kQ4_K>(m, n, k, dev)
                                       : plan_pair<kQ6_K>(m, n, k, dev);
  const int values[8] = {plan.tokens, plan.splits, plan.clusters, plan.tiles, 1 << decoded_log(fmt, plan.tokens),
                         accumulator_sets(fmt, plan.tokens), 0, 0};
  std::copy(values, values + 8, out8);
}

cudaError_t launch_gemm_pair(int fmt, const void* x, const uint8_t* w, float* out, long long m, long long n, long long k,
                             cudaStream_t stream, const char** detail) {
  switch (fmt) {
    case kQ4_0: return launch_pair<kQ4_0>(x, w, out, m, n, k, stream, detail);
    case kQ8_0: return launch_pair<kQ8_0>(x, w, out, m, n, k, stream, detail);
    case kQ4_K: return launch_pair<kQ4_K>(x, w, out, m, n, k, stream, detail);
    case kQ6_K: return launch_pair<kQ6_K>(x, w, out, m, n, k, stream, detail);
  }
  return cudaErrorInvalidValue;
}

}  // namespace tb200
