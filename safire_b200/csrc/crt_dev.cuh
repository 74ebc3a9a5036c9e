// Device pieces of the modular FP64 products: residues of a scaled value and values of residues.
#pragma once
#include "crt.cuh"

namespace sfq {
namespace crt {

static constexpr Tables kTabD = make_tables();
static __constant__ Tables c_crt = kTabD;
static constexpr double kTwoM64P = kTabD.P / 18446744073709551616.0;  // P 2^-64

__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double((long long)((e < -1022 ? -1022 : e > 1023 ? 1023 : e) + 1023) << 52);
}

// the scale exponent of a row with squared norm n2: |row| 2^-e < 2^kNormBits.  Rows that cannot be held
// (not finite, or so large or small that their squares leave the range) raise *flag.
__device__ __forceinline__ int row_exponent(double n2, bool any, int* flag) {
  if (!any && n2 == 0.0) return 0;
  if (!(n2 > 1e-300 && n2 < 1e300)) {
    if (flag) *flag = 1;
    return 0;
  }
  const int e2 = int((__double_as_longlong(n2) >> 52) & 0x7ff) - 1023;  // n2 < 2^(e2 + 1)
  return ((e2 + 2) >> 1) - kNormBits;
}

// four scaled values, ready to be reduced modulo each p
struct Quad {
  uint32_t lo[4], hi[4];
  __device__ __forceinline__ void set(const double* x, double sc) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const unsigned long long u = (unsigned long long)(__double2ll_rn(x[j] * sc) + (1ll << 60));
      lo[j] = uint32_t(u);
      hi[j] = uint32_t(u >> 32);
    }
  }
  // the four residues of modulus i, centred in [-(p - 1) / 2, (p - 1) / 2] (p = 256: the low bytes)
  __device__ __forceinline__ uint32_t word(int i) const {
    uint32_t r[4];
    if (i == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = lo[j];
    } else {
      const uint32_t p = kModuli_d(i), h = (p - 1) / 2;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t t = __dp4a(lo[j], c_crt.clo[i], __dp4a(hi[j], c_crt.chi[i], c_crt.init[i]));
        r[j] = t - __umulhi(t + h, c_crt.m32[i]) * p;
      }
    }
    return __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
  }
  static __device__ __forceinline__ constexpr uint32_t kModuli_d(int i) {
    constexpr uint32_t m[15] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197};
    return m[i];
  }
  __device__ __forceinline__ void store(int8_t* at, long plane) const {
#pragma unroll
    for (int i = 0; i < NMOD; ++i) *reinterpret_cast<uint32_t*>(at + i * plane) = word(i);
  }
  // the residues at `at` and those of the negated values at `neg`
  __device__ __forceinline__ void store2(int8_t* at, int8_t* neg, long plane) const {
#pragma unroll
    for (int i = 0; i < NMOD; ++i) {
      const uint32_t w = word(i);
      *reinterpret_cast<uint32_t*>(at + i * plane) = w;
      *reinterpret_cast<uint32_t*>(neg + i * plane) = __vneg4(w);  // -128 of p = 256 stays itself
    }
  }
};

// C' 2^64 / P (centred, rounded) of one element from its residues: w[q] holds moduli 4q .. 4q+3.  The
// sum of r_i G_i in 80-bit fixed point, byte by byte (each partial sum below 2^20), modulo 1
__device__ __forceinline__ long long reconstruct(const uint32_t w[4]) {
  uint32_t s[10];
#pragma unroll
  for (int j = 0; j < 10; ++j) {
    uint32_t a = j == 0 ? 0x8000u : 0u;  // half a unit of the 64 bits kept
#pragma unroll
    for (int q = 0; q < 4; ++q) a = __dp4a(w[q], c_crt.g[j][q], a);
    s[j] = a;
  }
  const uint32_t A = s[0] + (s[1] << 8), B = s[2] + (s[3] << 8) + (A >> 16), C = s[4] + (s[5] << 8),
                 D = s[6] + (s[7] << 8), E = s[8] + (s[9] << 8);
  return (long long)((unsigned long long)B + ((unsigned long long)C << 16) + ((unsigned long long)D << 32) +
                     ((unsigned long long)E << 48));
}

// the same for four consecutive elements whose residues lie at c + i * plane
__device__ __forceinline__ void reconstruct4(const uint8_t* c, long plane, long long X[4]) {
  uint32_t p[16];
#pragma unroll
  for (int i = 0; i < NMOD; ++i) p[i] = *reinterpret_cast<const uint32_t*>(c + i * plane);
  p[15] = 0;
  uint32_t e[4][4];  // [element][group of four moduli]
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t x0 = __byte_perm(p[4 * q], p[4 * q + 1], 0x5140), x1 = __byte_perm(p[4 * q + 2], p[4 * q + 3], 0x5140);
    const uint32_t y0 = __byte_perm(p[4 * q], p[4 * q + 1], 0x7362), y1 = __byte_perm(p[4 * q + 2], p[4 * q + 3], 0x7362);
    e[0][q] = __byte_perm(x0, x1, 0x5410);
    e[1][q] = __byte_perm(x0, x1, 0x7632);
    e[2][q] = __byte_perm(y0, y1, 0x5410);
    e[3][q] = __byte_perm(y0, y1, 0x7632);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) X[j] = reconstruct(e[j]);
}

}  // namespace crt
}  // namespace sfq
