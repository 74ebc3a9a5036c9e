// FP64 products on the int8 tensor cores by modular arithmetic (Ozaki scheme II: K. Ozaki,
// Y. Uchino, T. Imamura, "Ozaki Scheme II: A GEMM-oriented emulation of floating-point matrix
// multiplication using an integer modular technique", 2025).
//
// Every operand row is scaled by a power of two and rounded to integers a' with a 2-norm below
// 2^58; a product C' = sum_k a'_k b'_k is then an integer with |C'| < 2^116 < P/2 (Cauchy-Schwarz),
// P = prod p_i over 15 pairwise coprime moduli p_i <= 256 (log2 P = 117.78).  C' is known from its
// residues, and each residue is one exact int8 product with int32 accumulation (tcgen05
// kind::i8) of the operands' residues.  The only roundings are those of the operands, at most half a
// unit, 2^-58 of their row's norm, and of the result to FP64.
//
// An element far below its row's norm keeps fewer bits that way than FP64's 53: rows graded in opposite
// directions, |a_k| falling where |b_k| rises, would lose what FP64 keeps.  Every output is therefore checked:
// a sixteenth plane of each operand holds lower bounds of its magnitudes, |x_k| in units of the row's norm / 32
// sqrt(K), cut off at 127, and one more int8 product of these planes bounds sum_k |a_k| |b_k| from below.
// Where the modular error's bound,
//   sum_k (2^-58 |a| |b_k| + 2^-58 |b| |a_k|) <= 2^-57 sqrt(K) |a| |b|   (norms),
// is not within the FP64 chain's own, K 2^-53 sum_k |a_k| |b_k|, the walker is computed on the FP64 tensor pipe
// instead.  (Both bounds hold with sqrt(K) less for roundings that are independent, so the line is the same.)
// Operands that are not graded pass by a factor of 10 to 100; the check costs a sixteenth of the product.
//
// Rows that the scheme cannot hold (an Inf or a NaN, a norm outside 1e+-120) raise a flag in device memory, their
// walker's or, for an operand that all walkers share, the call's (Redo); the FP64 tensor-pipe product (gemm_f64),
// launched behind it, then computes what the flags ask for and leaves the other walkers' results as they are.
#pragma once
#include <cmath>

#include "common.cuh"

namespace sfq {
namespace crt {

constexpr int NMOD = 15;
constexpr int kPlanes = NMOD + 1;    // of an operand: its residues and its magnitudes
constexpr int kNormBits = 58;        // operand rows are scaled to a 2-norm below 2^kNormBits
constexpr long kMaxK = 90000;        // |sum of K residue products| <= K 2^14 < 2^30.5

// Magnitudes: floor(|a'| mag_scale(K)), 32 for an element of the row's root mean square at least.  From 8 to 64 the
// margins of typical operands differ little; 32 still sees elements of 1/32 of it beside one that holds the norm.
constexpr double kMag = 32.0;
inline double mag_scale(long K) { return std::ldexp(kMag * std::sqrt(double(K)), 1 - kNormBits); }
// the least product of magnitudes that passes: 2^-4 / sqrt(segs K) of the norms, which lie below 2 kMag sqrt(K) each,
// and an eighth more for the rounding of the result's integer
inline int mag_least(long K, int segs) { return int(std::ceil(1.125 * kMag * kMag / 4.0 * std::sqrt(double(K) / segs))); }

typedef unsigned __int128 u128;

struct Tables {
  unsigned mod[16];        // p_i; the 16th is a placeholder (never used)
  int m32[16];             // ceil(2^32 / p): floor(x / p) of |x| <= 2^24 as mulhi(x, m32), or one less
  unsigned m39[16];        // ceil(2^39 / p): floor(u / p) of u < 2^28 as umulhi(u, m39) >> 7
  unsigned big27[16];      // the smallest multiple of p >= 2^27
  unsigned big30[16];      // the smallest multiple of p >= 3 * 2^29
  unsigned r16[16];        // 2^16 mod p
  // C'/P mod 1 = sum_i r_i G_i mod 1 with G_i = ((P / p_i)^-1 mod p_i) / p_i, in 80-bit fixed point;
  // byte j of the G_i of moduli 4q .. 4q+3 in g[j][q]
  unsigned g[10][4];
  double P_hi, P_lo;       // P 2^-64 as the sum of two doubles
};

__host__ __device__ constexpr unsigned modulus(int i) {
  constexpr unsigned p[NMOD] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197};
  return p[i];
}

constexpr Tables make_tables() {
  Tables t{};
  u128 P = 1;
  for (int i = 0; i < NMOD; ++i) P *= modulus(i);
  // the top 53 bits of P and the rest, exactly
  int sh = 0;
  while ((P >> sh) >= (u128(1) << 53)) ++sh;
  double w = 1.0;
  for (int i = 0; i < sh; ++i) w *= 2.0;
  t.P_hi = double((unsigned long long)(P >> sh)) * (w / 18446744073709551616.0);
  const u128 rest = P - ((P >> sh) << sh);
  t.P_lo = (double((unsigned long long)(rest >> 32)) * 4294967296.0 + double((unsigned long long)(rest & 0xffffffffu))) /
           18446744073709551616.0;
  for (int i = 0; i < NMOD; ++i) {
    const unsigned p = modulus(i);
    t.mod[i] = p;
    t.m32[i] = int(((1ull << 32) + p - 1) / p);
    t.m39[i] = unsigned(((1ull << 39) + p - 1) / p);
    t.big27[i] = unsigned(((1ull << 27) + p - 1) / p * p);
    t.big30[i] = unsigned(((3ull << 29) + p - 1) / p * p);
    t.r16[i] = 65536u % p;
    unsigned rest = 1;  // P / p_i mod p_i
    for (int j = 0; j < NMOD; ++j)
      if (j != i) rest = rest * (modulus(j) % p) % p;
    unsigned inv = 0;
    for (unsigned x = 1; x < p; ++x)
      if (rest * x % p == 1) inv = x;
    const u128 G = ((u128(inv) << 80) + p / 2) / p;
    for (int j = 0; j < 10; ++j) t.g[j][i / 4] |= unsigned(G >> (8 * j) & 255) << (8 * (i % 4));
  }
  t.mod[15] = 1;
  return t;
}

// ---- operands ---------------------------------------------------------------------------------
// kPlanes planes of an operand: plane i at q + i * plane, rows of ld bytes (a multiple of 16),
// the row's scale exponent in e: x = a' 2^e
struct Planes {
  int8_t* q = nullptr;
  int* e = nullptr;
  long rows = 0, ld = 0, plane = 0;
};
inline long ld_of(long K) { return (K + 63) / 64 * 64; }
inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
inline size_t planes_bytes(long rows, long K) { return align256((size_t)rows * ld_of(K)) * kPlanes; }
inline size_t exps_bytes(long rows) { return align256(sizeof(int) * (size_t)rows); }
// lays the planes of rows x K out at *at and advances it (e_rows exponents behind them)
inline Planes lay_out(char*& at, long rows, long K, long e_rows) {
  Planes p;
  p.rows = rows;
  p.ld = ld_of(K);
  p.plane = (long)align256((size_t)rows * p.ld);
  p.q = reinterpret_cast<int8_t*>(at);
  at += planes_bytes(rows, K);
  p.e = reinterpret_cast<int*>(at);
  at += exps_bytes(e_rows);
  return p;
}

// the flags of a call over W walkers, at *at, which advances
inline size_t flag_bytes(long W) { return 256 + align256(sizeof(int) * (size_t)W); }
inline Redo lay_out_flags(char*& at, long W) {
  Redo r;
  r.call = reinterpret_cast<int*>(at);
  r.row = reinterpret_cast<int*>(at + 256);
  at += flag_bytes(W);
  return r;
}

// ---- the product of residues: C_i = A_i B_i^T mod p_i for every modulus ------------------------
// Output row part * M + m, column n, at C + i * c_plane + row * ldc + n (bytes).
// A rows a_off[part][seg] + m, B rows b_off[seg] + n, summed over the segments
// (a complex product: parts re, im; segments against Re B and Im B).  Rows whose magnitudes do not pass raise the
// flag of walker m % wmod.
struct Gemm {
  Planes A, B;
  int M = 0, N = 0, K = 0, parts = 1, segs = 1;
  long a_off[2][2] = {{0, 0}, {0, 0}};
  long b_off[2] = {0, 0};
  uint8_t* C = nullptr;
  long ldc = 0, c_plane = 0;
  Redo redo;                       // call[1]: set when a bounded wait expires
  int wmod = 0;
  bool check = true;               // false: the residues alone, for operands that are known not to be graded
  unsigned long long wait_ns = 0;  // limit of one wait without progress (0: 2 s)
  const int* hold = nullptr;       // self-test: loads from the hold_at-th K slice on wait for *hold
  unsigned hold_at = 0;
};
int gemm(const Gemm& g, cudaStream_t st);

// The same for products whose left rows are a walker's: [re; im] rows (w, a) of A's blocks (re, im, -im at
// block strides a_blk; row w N + a) against cols rows of B (row w b_bs + n; segs = 2: complex B, its
// imaginary rows b_off1 further).  Output row c c_part + w N + a.  The magnitudes' product runs first, and
// the others not where all walkers then have a flag (padding columns must not raise one: pass_padding).
struct WalkerGemm {
  Planes A, B;
  int N = 0, cols = 0, K = 0, batch = 1, segs = 1;
  long a_blk = 0, b_bs = 0, b_off1 = 0;
  uint8_t* C = nullptr;
  long ldc = 0, c_plane = 0, c_part = 0;
  Redo redo;
  bool check = true;               // as in Gemm
  unsigned long long wait_ns = 0;  // as in Gemm
  const int* hold = nullptr;
  unsigned hold_at = 0;
};
bool walker_gemm_fits(int N, int cols, int K, int segs);
int walker_gemm(const WalkerGemm& g, cudaStream_t st);
// calls on this device since the process began in which a bounded wait expired
int expiries(unsigned long long* n);

// the output of a product: NMOD planes of rows x ldc bytes
struct Out {
  uint8_t* q = nullptr;
  long ldc = 0, plane = 0;
};
inline long ldc_of(long N) { return (N + 31) / 32 * 32; }  // rows of whole sectors
inline size_t out_bytes(long rows, long N) { return align256((size_t)rows * ldc_of(N)) * NMOD; }
inline Out lay_out_c(char*& at, long rows, long N) {
  Out o;
  o.q = reinterpret_cast<uint8_t*>(at);
  o.ldc = ldc_of(N);
  o.plane = (long)align256((size_t)rows * o.ldc);
  at += out_bytes(rows, N);
  return o;
}

// ---- operands to residues -----------------------------------------------------------------------
// A row that cannot be held raises redo.call[0] (per_walker 0: the operand is all walkers') or the flag of
// walker r / per_walker.
// real rows (row r of `rows` at src + r * stride, K doubles) -> planes row (r / inner) * outer + r % inner
// (inner 0: row r), exponent e[r]
int rows_real(const double* src, long rows, long K, long stride, const Planes& out, Redo redo, long per_walker,
              cudaStream_t st, long inner = 0, long outer = 0);
// complex rows (K complex each) -> blocks re, im (, -im): row r's block k at plane row k * blk_stride + (r / inner) *
// outer + r % inner.  Against a complex operand the parts share one exponent, e[r]; against a real one they are rows
// of their own (e[r] and e[rows + r]), so that a small imaginary part keeps its own bits
enum class Parts { kApart, kJoint, kJointNeg };
int rows_cplx(const cplx* src, long rows, long K, long stride, Parts parts, long blk_stride, long inner, long outer,
              const Planes& out, Redo redo, long per_walker, cudaStream_t st);
// the magnitudes of a whole operand, before its rows are written, as those of rows of zeros, for rows that nothing writes
int pass_padding(const Planes& out, cudaStream_t st);
// walkers (W npol, M, N) complex -> rows (w, q, a) over the M orbitals, blocks re, im, -im: plane row
// k * W npol N + (w npol + q) N + a; and the rows themselves, S (W npol N, M)
int walkers_in(const cplx* SM, int W, int npol, int M, int N, const Planes& out, cplx* S, Redo redo, cudaStream_t st);

// alpha P 2^-64 as a sum of two doubles, so that values are rounded twice (as integers, as products) and not
// pulled by a rounded constant as well
struct Scale {
  double hi, lo;
};
Scale scale_of(double alpha);

// ---- residues to FP64 ---------------------------------------------------------------------------
// out[m][n] = alpha (C_re + i C_im) for parts = 2 products with M rows; exponents eA[m] (and eA[im + m] of the
// imaginary part), eB[n]
int out_cplx(const Out& c, long M, long N, const int* eA, long im, const int* eB, double alpha, cplx* out, long ldo,
             cudaStream_t st);
int out_real(const Out& c, long M, long N, const int* eA, const int* eB, double alpha, double* out, long ldo,
             cudaStream_t st);
// one Taylor term: T = (i / k) C, S (W, N, M) += T, and the residues of T, blocks re, im, -im -> `next` (not of the
// last one).  C rows (part, w, a), columns j; exponents eA[w N + a], eB[w M + j].
int taylor_update(const Out& c, int W, int N, int M, int k, bool last, const int* eA, const int* eB, cplx* S,
                  const Planes& next, Redo redo, cudaStream_t st);
// exx[w, n0 + n] = sum_ab T[w,a,n,b] T[w,b,n,a] and kl[w, n0 + n] = sum_a T[w,a,n,a] of T[w,b,n,a] = rows
// (part, w, b), columns n * N4 + a (exponents eA[w N + b], the imaginary part's im further, and eB[n * N + a]); nup as
// in energy_exx_reduce; not of the walkers that redo asks for
constexpr int kExxMaxN = 116;  // a walker's N x N block of one n in shared memory
int exx_reduce(const Out& c, int W, int N, int N4, int nv, int n0, int Nc, const int* eA, long im, const int* eB,
               cplx* exxn, cplx* kl, int nup, Redo redo, cudaStream_t st);

}  // namespace crt
}  // namespace sfq
