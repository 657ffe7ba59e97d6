// digits64.cuh -- FP64 products as exact sums of digit products on the tensor
// cores, shared by the transforms (k_dft64.cu, which derives the bounds) and
// the implicit solve (k_solve64.cu): 61-bit integers of values against a power
// of two, their eight balanced 8-bit digits as FP16, m16n8k16 products of
// digits accumulated exactly per level in FP32, and the levels combined in
// 64-bit integers.
#pragma once
#include <cuda_fp16.h>

#include <cstdint>

namespace chf {

__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// two digit bytes (as 128 + d) to FP16: 1024 + byte - 1152
__device__ __forceinline__ uint32_t to_half2(uint32_t w, uint32_t sel) {
  const uint32_t h = __byte_perm(w, 0x64646464u, sel);
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&h), __half2half2(__ushort_as_half(0x6480)));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// x 2^(61 - e) rounded to an integer, |x| < 2^e, e = emax - 1022, emax >= 1
// (zeros and subnormals have the exponent of 1, without its leading bit)
__device__ __forceinline__ long long fixed_of(uint32_t lo, uint32_t hi, int emax) {
  const int ex = (int)((hi >> 20) & 0x7ffu);
  const int d = emax - max(ex, 1);  // >= 0
  if (d > 62) return 0;
  const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (ex ? 0x100000u : 0u)) << 32 | lo) << 8;
  unsigned long long t = m >> d;
  if (d > 0) t += (m >> (d - 1)) & 1ull;
  return (int)hi < 0 ? -(long long)t : (long long)t;
}

// eight planes of FP16 digit pairs (top plane first) of two integers
__device__ __forceinline__ void digit_pairs(long long x0, long long x1, uint32_t (&w)[8]) {
  const unsigned long long a = (unsigned long long)x0 + 0x8080808080808080ull;
  const unsigned long long b = (unsigned long long)x1 + 0x8080808080808080ull;
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // bytes 7..4, then 3..0
    const uint32_t u = h ? (uint32_t)a : (uint32_t)(a >> 32), v = h ? (uint32_t)b : (uint32_t)(b >> 32);
    const uint32_t top = __byte_perm(u, v, 0x7362), low = __byte_perm(u, v, 0x5140);  // bytes 2, 3 and 0, 1 of both
    w[4 * h + 0] = to_half2(top, 0x4342);
    w[4 * h + 1] = to_half2(top, 0x4140);
    w[4 * h + 2] = to_half2(low, 0x4342);
    w[4 * h + 3] = to_half2(low, 0x4140);
  }
}

// eight planes of digit bytes (biased by 128) of four integers, one word per plane
__device__ __forceinline__ void digit_bytes(const long long* x, uint32_t (&w)[8]) {
  uint32_t lo[4], hi[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const unsigned long long y = (unsigned long long)x[i] + 0x8080808080808080ull;
    lo[i] = (uint32_t)y;
    hi[i] = (uint32_t)(y >> 32);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t* v = h ? lo : hi;
    const uint32_t a = __byte_perm(v[0], v[1], 0x7362), b = __byte_perm(v[2], v[3], 0x7362);  // bytes 2, 3
    const uint32_t c = __byte_perm(v[0], v[1], 0x5140), d = __byte_perm(v[2], v[3], 0x5140);  // bytes 0, 1
    w[4 * h + 0] = __byte_perm(a, b, 0x7632);
    w[4 * h + 1] = __byte_perm(a, b, 0x5410);
    w[4 * h + 2] = __byte_perm(c, d, 0x7632);
    w[4 * h + 3] = __byte_perm(c, d, 0x5410);
  }
}

// hi 2^32 + lo += sum_p lev_p 256^(7-p), the eight level sums
__device__ __forceinline__ void add_levels(const float (&lev)[8], long long& hi, long long& lo) {
  int a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = __float2int_rn(lev[i]);
  hi += (long long)(a[0] * 256 + a[1]) * 65536ll + (long long)(a[2] * 256 + a[3]);
  lo += (long long)a[4] * 16777216ll + (long long)a[5] * 65536ll + ((long long)a[6] * 256ll + a[7]);
}

}  // namespace chf
