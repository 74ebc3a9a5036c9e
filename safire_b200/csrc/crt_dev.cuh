// Device pieces of the modular FP64 products: residues of a scaled value and values of residues.
#pragma once
#include "crt.cuh"

namespace sfq {
namespace crt {

static constexpr Tables kTabD = make_tables();
static __constant__ Tables c_crt = kTabD;

__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double((long long)((e < -1022 ? -1022 : e > 1023 ? 1023 : e) + 1023) << 52);
}

// the scale exponent of a row with squared norm n2: |row| 2^-e < 2^kNormBits.  Rows that cannot be held
// (not finite, or a norm outside 1e+-120, beyond which two rows' scales could leave the exponent range) are asked for
// again by the thread that `asks`: their walker w, or all of them (w < 0).
__device__ __forceinline__ int row_exponent(double n2, bool any, bool asks, const Redo& redo, long w) {
  if (!any && n2 == 0.0) return 0;
  if (!(n2 > 1e-240 && n2 < 1e240)) {
    if (asks && w < 0) redo.ask_all();
    else if (asks) redo.ask(w);
    return 0;
  }
  const int e2 = int((__double_as_longlong(n2) >> 52) & 0x7ff) - 1023;  // n2 < 2^(e2 + 1)
  return ((e2 + 2) >> 1) - kNormBits;
}

// Residues of four scaled values.  A value y (an integer in FP64, up to 2^58) is first reduced modulo the
// product Q < 2^24 of a group of two or three moduli, q = rint(y / Q), x = y - q Q in one exact fma, and x,
// now exact in FP32, modulo each of them: the FP64, conversion, FP32 and byte-permute pipes share the
// work.  About 0.65 cycles an element and SM; integer dot products and high multiplies of the value's
// bytes, two pipes for everything, took 1.5.
// a row's magnitudes: their scale, and 127 for all of a row of zeros, whose products are exact
struct Mag {
  double scale;
  uint32_t fill;
};
__device__ __forceinline__ Mag mag_of(double scale, bool zero) { return {scale, zero ? 0x7f7f7f7fu : 0u}; }
struct Quad {
  double y[4];
  __device__ __forceinline__ void set(const double* x, double sc) {
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = rint(x[j] * sc);
  }
  // f(i, word): the four residues of modulus i as bytes, centred (-p / 2 .. p / 2)
  template <typename F>
  __device__ __forceinline__ void words(F&& f) const {
#pragma unroll
    for (int g = 0; g < 6; ++g) {
      constexpr int at[7] = {0, 2, 4, 7, 10, 13, 15};
      const int i0 = at[g], n = at[g + 1] - at[g];
      const double Q = double(modulus(i0)) * modulus(i0 + 1) * (n == 3 ? modulus(i0 + n - 1) : 1u);
      const double inv = 1.0 / Q;
      float x[4];
      uint32_t lo[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double q = fma(y[j], inv, 6755399441055744.0) - 6755399441055744.0;  // 1.5 2^52: rint
        const double r = fma(-q, Q, y[j]);                                          // |r| <= Q / 2, exact
        if (n == 3) {
          x[j] = __double2float_rn(r);  // exact: |r| <= 2^23
        } else {                        // |r| < 2^16: through the low words of the magic numbers
          lo[j] = uint32_t(__double_as_longlong(r + 6755399441055744.0));
          x[j] = __uint_as_float(0x4B400000u + lo[j]) - 12582912.0f;
        }
      }
#pragma unroll
      for (int i = i0; i < i0 + n; ++i) {
        uint32_t b[4];
        if (modulus(i) == 256) {  // Q is a multiple of 256
#pragma unroll
          for (int j = 0; j < 4; ++j) b[j] = lo[j];
        } else {
          const float p = float(modulus(i)), ip = 1.0f / p;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float q = __fadd_rn(fmaf(x[j], ip, 12582912.0f), -12582912.0f);
            b[j] = __float_as_uint(__fadd_rn(fmaf(-q, p, x[j]), 12582912.0f));  // low byte: the residue
          }
        }
        f(i, __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410));
      }
    }
  }
  // the four magnitudes (see crt.cuh)
  __device__ __forceinline__ uint32_t magnitudes(Mag m) const {
    uint32_t b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)  // floor: added to 1.5 2^52 rounding down
      b[j] = min(uint32_t(__double_as_longlong(__fma_rd(fabs(y[j]), m.scale, 6755399441055744.0))), 127u);
    return __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410) | m.fill;
  }
  __device__ __forceinline__ void store(int8_t* at, long plane, Mag m) const {
    words([&](int i, uint32_t w) { *reinterpret_cast<uint32_t*>(at + i * plane) = w; });
    *reinterpret_cast<uint32_t*>(at + NMOD * plane) = magnitudes(m);
  }
  // the residues at `at` and those of the negated values at `neg`
  __device__ __forceinline__ void store2(int8_t* at, int8_t* neg, long plane, Mag m) const {
    words([&](int i, uint32_t w) {
      *reinterpret_cast<uint32_t*>(at + i * plane) = w;
      *reinterpret_cast<uint32_t*>(neg + i * plane) = __vneg4(w);  // -128 of p = 256 stays itself
    });
    const uint32_t w = magnitudes(m);
    *reinterpret_cast<uint32_t*>(at + NMOD * plane) = w;
    *reinterpret_cast<uint32_t*>(neg + NMOD * plane) = w;
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
