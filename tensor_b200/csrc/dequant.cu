// Standalone fp32 dequantisation: out[n, k] = dequant(w).  This kernel carries the bit-exact
// gate against the reference's decode (benchmarks/kernels/showcase/triton_kernels.py:133-181).
//
// Bound: the fp32 stores (4 B per weight out, 0.56 .. 1.06 B in).  Rows are consecutive blocks with no padding, so
// the matrix is ONE flat sequence of blocks and the output one flat array: no row arithmetic.  A warp takes
// units of 256 weights; a lane owns the 4-byte words of quants whose decoded values are whole 16-byte stores, so a
// quant byte is loaded once for both of its nibbles and every store instruction fills whole 32-byte sectors.
// kUnroll units are loaded before the first is stored: loads of one unit per lane left the kernel waiting.
// Q6_K 12288 x 4096 (41 MB in, 201 MB out; the copy rate allows 37 us): 41.6 us = 5.8 TB/s; 82 us when
// every lane decoded four neighbouring weights byte by byte with a 64-bit division for its row.
#include "common.cuh"
#include "kernels.h"

namespace tb200 {
namespace {

constexpr int kThreads = 256;
constexpr int kUnroll = 4;  // units of 256 weights per warp and step

__device__ __forceinline__ uint32_t ldg_u16(const uint8_t* p) {
  return __ldg(reinterpret_cast<const unsigned short*>(p));
}
__device__ __forceinline__ uint32_t ldg_word2(const uint8_t* p) { return ldg_u16(p) | (ldg_u16(p + 2) << 16); }
__device__ __forceinline__ float half_bits(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }
// byte j of v as an exact float (2^23 + byte, minus 2^23 + bias)
__device__ __forceinline__ float byte_f32(uint32_t v, int j, float bias) {
  return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540u | (uint32_t)j)) - (8388608.f + bias);
}

// What a lane loads of one unit, and the two groups of four weights it makes of it: values a at offset_a of the
// unit, values b at offset_b.
template <int FMT> struct Unit;

template <> struct Unit<kQ4_0> {  // lane: word lane % 4 of block lane / 4; low nibbles, then the high ones 16 further on
  uint32_t q, d;
  __device__ static int offset_a(int lane) { return 32 * (lane >> 2) + 4 * (lane & 3); }
  __device__ static int offset_b(int lane) { return offset_a(lane) + 16; }
  __device__ void load(const uint8_t* u, int lane) {
    const uint8_t* b = u + 18 * (lane >> 2);
    d = ldg_u16(b);
    q = ldg_word2(b + 2 + 4 * (lane & 3));
  }
  __device__ void decode(int, float (&a)[4], float (&b)[4]) const {
    const float s = half_bits(d);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = __fmul_rn(byte_f32(q & 0x0F0F0F0Fu, j, 8.f), s);
      b[j] = __fmul_rn(byte_f32((q >> 4) & 0x0F0F0F0Fu, j, 8.f), s);
    }
  }
};

template <> struct Unit<kQ8_0> {  // lane: words lane and lane + 32 of the unit's 64 words of quants
  uint32_t q[2], d[2];
  __device__ static int offset_a(int lane) { return 4 * lane; }
  __device__ static int offset_b(int lane) { return 128 + 4 * lane; }
  __device__ void load(const uint8_t* u, int lane) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint8_t* b = u + 34 * (4 * i + (lane >> 3));
      d[i] = ldg_u16(b);
      q[i] = ldg_word2(b + 2 + 4 * (lane & 7));
    }
  }
  __device__ void decode(int, float (&a)[4], float (&b)[4]) const {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = __fmul_rn(half_bits(d[0]), byte_f32(q[0] ^ 0x80808080u, j, 128.f));
      b[j] = __fmul_rn(half_bits(d[1]), byte_f32(q[1] ^ 0x80808080u, j, 128.f));
    }
  }
};

template <> struct Unit<kQ4_K> {  // lane: quant word lane: low nibbles are group 2 p, high ones group 2 p + 1
  uint4 hdr;
  uint32_t q;
  __device__ static int offset_a(int lane) { return 64 * (lane >> 3) + 4 * (lane & 7); }
  __device__ static int offset_b(int lane) { return offset_a(lane) + 32; }
  __device__ void load(const uint8_t* u, int lane) {
    hdr = __ldg(reinterpret_cast<const uint4*>(u));
    q = __ldg(reinterpret_cast<const uint32_t*>(u + 16) + lane);
  }
  __device__ void decode(int lane, float (&a)[4], float (&b)[4]) const {
    const int p = lane >> 3, sh = 16 * (p & 1);
    const bool upper = p >= 2;
    // both groups' 6-bit scales / mins sit in neighbouring bytes of the packed words
    const uint32_t sc4 = upper ? ((hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u)) : (hdr.y & 0x3F3F3F3Fu);
    const uint32_t mn4 = upper ? (((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u)) : (hdr.z & 0x3F3F3F3Fu);
    const uint32_t sc = sc4 >> sh, mn = mn4 >> sh;
    const float d = half_bits(hdr.x & 0xFFFFu), dmin = half_bits(hdr.x >> 16);
    const float sa = __fmul_rn(d, (float)(sc & 0xFFu)), sb = __fmul_rn(d, (float)((sc >> 8) & 0xFFu));
    const float ma = __fmul_rn(dmin, (float)(mn & 0xFFu)), mb = __fmul_rn(dmin, (float)((mn >> 8) & 0xFFu));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = __fsub_rn(__fmul_rn(sa, byte_f32(q & 0x0F0F0F0Fu, j, 0.f)), ma);
      b[j] = __fsub_rn(__fmul_rn(sb, byte_f32((q >> 4) & 0x0F0F0F0Fu, j, 0.f)), mb);
    }
  }
};

template <> struct Unit<kQ6_K> {  // lane: `ql` word lane; its low nibbles, and its high ones 64 weights further on
  uint32_t ql, qh, sc, d;
  __device__ static int offset_a(int lane) { return 128 * (lane >> 4) + 32 * ((lane >> 3) & 1) + 4 * (lane & 7); }
  __device__ static int offset_b(int lane) { return offset_a(lane) + 64; }
  __device__ void load(const uint8_t* u, int lane) {
    const int h = lane >> 4;
    ql = ldg_word2(u + 4 * lane);
    qh = ldg_word2(u + 128 + 32 * h + 4 * (lane & 7));
    const uint8_t* s = u + 192 + (offset_a(lane) >> 4);
    sc = (uint32_t)__ldg(s) | ((uint32_t)__ldg(s + 4) << 8);
    d = ldg_u16(u + 208);
  }
  __device__ void decode(int lane, float (&a)[4], float (&b)[4]) const {
    const int pair = 2 * ((lane >> 3) & 1);
    const uint32_t qa = (ql & 0x0F0F0F0Fu) | (((qh >> pair) & 0x03030303u) << 4);
    const uint32_t qb = ((ql >> 4) & 0x0F0F0F0Fu) | (((qh >> (4 + pair)) & 0x03030303u) << 4);
    const float dd = half_bits(d);
    const float sa = (float)(int)(int8_t)(sc & 0xFFu), sb = (float)(int)(int8_t)((sc >> 8) & 0xFFu);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = __fmul_rn(__fmul_rn(byte_f32(qa, j, 32.f), sa), dd);
      b[j] = __fmul_rn(__fmul_rn(byte_f32(qb, j, 32.f), sb), dd);
    }
  }
};

template <int FMT>
__global__ void __launch_bounds__(kThreads) dequant_kernel(const uint8_t* __restrict__ w, float* __restrict__ out,
                                                           long long weights, int vector) {
  using U = Unit<FMT>;
  constexpr int kUnitBytes = 256 / Fmt<FMT>::kWeights * Fmt<FMT>::kBytes;
  const int lane = threadIdx.x & 31;
  const int oa = U::offset_a(lane), ob = U::offset_b(lane);
  const long long units = (weights + 255) >> 8;
  const long long warps = (long long)gridDim.x * (kThreads / 32);
  for (long long u0 = ((long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * kUnroll; u0 < units; u0 += warps * kUnroll) {
    if (vector && (u0 + kUnroll) * 256 <= weights) {
      U unit[kUnroll];
#pragma unroll
      for (int i = 0; i < kUnroll; ++i) unit[i].load(w + (u0 + i) * kUnitBytes, lane);
#pragma unroll
      for (int i = 0; i < kUnroll; ++i) {
        float a[4], b[4];
        unit[i].decode(lane, a, b);
        float* o = out + (u0 + i) * 256;
        __stcs(reinterpret_cast<float4*>(o + oa), make_float4(a[0], a[1], a[2], a[3]));
        __stcs(reinterpret_cast<float4*>(o + ob), make_float4(b[0], b[1], b[2], b[3]));
      }
    } else {
      // the last units: whole blocks, but not always whole units (Q8_0 / Q4_0); and a Q4_K weight whose address is
      // only 2-byte aligned: one weight at a time
      const int end = (int)(weights - u0 * 256 < kUnroll * 256 ? weights - u0 * 256 : kUnroll * 256);
      for (int c = lane; c < end; c += 32) out[u0 * 256 + c] = decode_one<FMT>(w + u0 * kUnitBytes, c);
    }
  }
}

template <int FMT>
void launch(const uint8_t* w, float* out, long long weights, int sm_count, cudaStream_t stream) {
  const long long per_block = (long long)(kThreads / 32) * kUnroll * 256;
  const long long want = (weights + per_block - 1) / per_block, most = (long long)sm_count * 32;
  const int vector = FMT != kQ4_K || reinterpret_cast<uintptr_t>(w) % 16 == 0;
  dequant_kernel<FMT><<<(unsigned)(want < most ? want : most), kThreads, 0, stream>>>(w, out, weights, vector);
}

}  // namespace

cudaError_t launch_dequant(int fmt, const uint8_t* w, float* out, long long n, long long k,
                           cudaStream_t stream) {
  if (n == 0 || k == 0) return cudaSuccess;
  cudaError_t err;
  const DeviceInfo* dev = device_info(&err);
  if (!dev) return err;
  switch (fmt) {
    case kQ4_0: launch<kQ4_0>(w, out, n * k, dev->sm_count, stream); break;
    case kQ8_0: launch<kQ8_0>(w, out, n * k, dev->sm_count, stream); break;
    case kQ4_K: launch<kQ4_K>(w, out, n * k, dev->sm_count, stream); break;
    case kQ6_K: launch<kQ6_K>(w, out, n * k, dev->sm_count, stream); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace tb200
