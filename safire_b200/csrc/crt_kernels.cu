// Residues of FP64 operands and FP64 values of residue products (see crt.cuh).
#include "crt.cuh"
#include "crt_dev.cuh"

#include <cmath>

namespace sfq {
namespace crt {

namespace {

// the loads of four consecutive elements from k on, zeros past K
__device__ __forceinline__ void load4(const double* row, long k, long K, bool vec, double x[4]) {
  if (vec && k + 3 < K) {
    const double2 a = *reinterpret_cast<const double2*>(row + k), b = *reinterpret_cast<const double2*>(row + k + 2);
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = k + j < K ? row[k + j] : 0.0;
  }
}

// sum over the TPR threads of a row (TPR = 32: a warp; else the whole block)
template <int TPR>
__device__ __forceinline__ double row_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (TPR == 32) return v;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < TPR / 32; ++w) s += sh[w];
  return s;
}

// Real rows.  Two passes over a row: its norm, then its residues (the second read comes from L1 or
// L2: a row is at most a few hundred KB).  One warp per row below 1024 elements, one block above.
template <int TPR>
__global__ void __launch_bounds__(256) rows_real_kernel(const double* src, long rows, long K, long stride, int8_t* q,
                                                        long ld, long plane, int* e, Redo redo, long per_walker,
                                                        int vec, long inner, long outer, double mag) {
  __shared__ double sh[8];
  const long r = TPR == 32 ? (long)blockIdx.x * 8 + (threadIdx.x >> 5) : blockIdx.x;
  const int t = TPR == 32 ? (threadIdx.x & 31) : threadIdx.x;
  if (r >= rows) return;  // TPR = 32: whole warps
  const double* row = src + r * stride;
  double n2 = 0.0, nz = 0.0;
  for (long k = 4 * t; k < K; k += 4 * TPR) {
    double x[4];
    load4(row, k, K, vec, x);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      n2 = fma(x[j], x[j], n2);
      nz = fmax(nz, fabs(x[j]));
    }
  }
  n2 = row_sum<TPR>(n2, sh);
  // a row of zeros has the norm 0; one whose squares all vanish does not
  const bool any = TPR == 32 ? __any_sync(0xffffffffu, nz != 0.0) : __syncthreads_or(nz != 0.0) != 0;
  const int ex = row_exponent(n2, any, t == 0, redo, per_walker ? r / per_walker : -1);
  if (t == 0) e[r] = ex;
  const double sc = pow2(-ex);
  const Mag m = mag_of(mag, !any);
  int8_t* qr = q + (inner ? (r / inner) * outer + r % inner : r) * ld;
  for (long k = 4 * t; k < K; k += 4 * TPR) {
    double x[4];
    load4(row, k, K, vec, x);
    Quad qd;
    qd.set(x, sc);
    qd.store(qr + k, plane, m);
  }
}

// Complex rows: the same, the parts with one exponent or each with its own
template <int TPR, Parts P>
__global__ void __launch_bounds__(256) rows_cplx_kernel(const cplx* src, long rows, long K, long stride,
                                                        long blk_stride, long inner, long outer, int8_t* q, long ld,
                                                        long plane, int* e, Redo redo, long per_walker, double mag) {
  __shared__ double sh[8];
  const long r = TPR == 32 ? (long)blockIdx.x * 8 + (threadIdx.x >> 5) : blockIdx.x;
  const int t = TPR == 32 ? (threadIdx.x & 31) : threadIdx.x;
  if (r >= rows) return;
  const cplx* row = src + r * stride;
  double x2 = 0.0, y2 = 0.0, xm = 0.0, ym = 0.0;
  for (long k = t; k < K; k += TPR) {
    const cplx z = row[k];
    x2 = fma(z.x, z.x, x2);
    y2 = fma(z.y, z.y, y2);
    xm = fmax(xm, fabs(z.x));
    ym = fmax(ym, fabs(z.y));
  }
  auto any_of = [](bool b) { return TPR == 32 ? __any_sync(0xffffffffu, b) != 0 : __syncthreads_or(b) != 0; };
  const long wk = per_walker ? r / per_walker : -1;
  int ex, ey;
  bool xs, ys;  // parts that are not zeros
  if (P == Parts::kApart) {
    x2 = row_sum<TPR>(x2, sh);
    y2 = row_sum<TPR>(y2, sh);
    xs = any_of(xm != 0.0);
    ys = any_of(ym != 0.0);
    ex = row_exponent(x2, xs, t == 0, redo, wk);
    ey = row_exponent(y2, ys, t == 0, redo, wk);
    if (t == 0) e[rows + r] = ey;
  } else {
    x2 = row_sum<TPR>(x2 + y2, sh);
    xs = ys = any_of(xm != 0.0 || ym != 0.0);
    ex = ey = row_exponent(x2, xs, t == 0, redo, wk);
  }
  if (t == 0) e[r] = ex;
  const double sx = pow2(-ex), sy = pow2(-ey);
  const Mag mx = mag_of(mag, !xs), my = mag_of(mag, !ys);
  int8_t* qr = q + ((r / inner) * outer + r % inner) * ld;
  for (long k = 4 * t; k < K; k += 4 * TPR) {
    double x[4], y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const cplx z = k + j < K ? row[k + j] : mk(0.0, 0.0);
      x[j] = z.x;
      y[j] = z.y;
    }
    Quad a;
    a.set(x, sx);
    a.store(qr + k, plane, mx);
    a.set(y, sy);
    if (P == Parts::kJointNeg) a.store2(qr + blk_stride * ld + k, qr + 2 * blk_stride * ld + k, plane, my);
    else a.store(qr + blk_stride * ld + k, plane, my);
  }
}

// Walkers' components (w, M, N), npol to a walker -> rows (w, a) over the orbitals: a block takes 16 columns of one, their
// norms first, then 64 orbitals at a time through shared memory (the transpose): their residues, and the rows as they are.
__global__ void __launch_bounds__(256) walkers_in_kernel(const cplx* SM, int W, int npol, int M, int N, int8_t* q,
                                                         long ld, long plane, int* e, cplx* rows, Redo redo,
                                                         double mag) {
  __shared__ cplx tile[64][17];
  __shared__ double sh[16][17];
  __shared__ double scs[16];
  __shared__ int nz[16];
  const int w = blockIdx.y, a0 = blockIdx.x * 16;
  const int ca = threadIdx.x & 15, ri = threadIdx.x >> 4;
  const cplx* S = SM + (long)w * M * N;
  double n2 = 0.0, mx = 0.0;
  if (threadIdx.x < 16) nz[threadIdx.x] = 0;
  __syncthreads();
  if (a0 + ca < N) {
    for (int i = ri; i < M; i += 16) {
      const cplx z = S[(long)i * N + a0 + ca];
      n2 = fma(z.x, z.x, fma(z.y, z.y, n2));
      mx = fmax(mx, fmax(fabs(z.x), fabs(z.y)));
    }
  }
  sh[ri][ca] = n2;
  if (mx != 0.0) nz[ca] = 1;
  __syncthreads();
  if (threadIdx.x < 16 && a0 + ca < N) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 16; ++j) s += sh[j][ca];
    const int ex = row_exponent(s, nz[ca] != 0, true, redo, w / npol);
    e[(long)w * N + a0 + ca] = ex;
    scs[ca] = pow2(-ex);
  }
  const long WN = (long)W * N;
  for (int i0 = 0; i0 < M; i0 += 64) {
    __syncthreads();
    for (int s = ri; s < 64; s += 16) {
      const int i = i0 + s;
      tile[s][ca] = i < M && a0 + ca < N ? S[(long)i * N + a0 + ca] : mk(0.0, 0.0);
    }
    __syncthreads();
    const int a = threadIdx.x >> 4, i4 = 4 * (threadIdx.x & 15);  // 16 rows x 16 groups of four orbitals
    if (a0 + a < N && i0 + i4 < M) {
      double x[4], y[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[j] = tile[i4 + j][a].x;
        y[j] = tile[i4 + j][a].y;
      }
      const long r = (long)w * N + a0 + a;
      int8_t* qr = q + r * ld + i0 + i4;
      const Mag m = mag_of(mag, nz[a] == 0);
      Quad d;
      d.set(x, scs[a]);
      d.store(qr, plane, m);
      d.set(y, scs[a]);
      d.store2(qr + WN * ld, qr + 2 * WN * ld, plane, m);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i0 + i4 + j < M) rows[r * M + i0 + i4 + j] = mk(x[j], y[j]);
    }
  }
}

// four columns of one output row from its residue planes
struct Vals {
  double v[4];
};
__device__ __forceinline__ Vals values4(const uint8_t* c, long plane, int ea, const int eb[4], Scale s) {
  long long X[4];
  reconstruct4(c, plane, X);
  Vals o;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double x = double(X[j]), p = pow2(ea + eb[j]);
    o.v[j] = fma(x, s.hi * p, x * (s.lo * p));
  }
  return o;
}

__device__ __forceinline__ void load_e4(const int* e, long n, long N, int eb[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) eb[j] = n + j < N ? e[n + j] : 0;
}

// complex output, 4 columns per thread, 128 per warp; the warp's values go through shared memory so that
// its stores are whole 512-byte rows
__global__ void __launch_bounds__(256) out_cplx_kernel(const uint8_t* c, long ldc, long plane, long M, long N,
                                                       const int* eA, long im0, const int* eB, Scale s, cplx* out,
                                                       long ldo) {
  __shared__ cplx sh[8][130];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long m = blockIdx.y, nw = ((long)blockIdx.x * 8 + warp) * 128;
  if (nw >= N) return;
  const long n = nw + 4 * lane;
  if (n < N) {
    int eb[4];
    load_e4(eB, n, N, eb);
    const Vals re = values4(c + m * ldc + n, plane, eA[m], eb, s);
    const Vals im = values4(c + (M + m) * ldc + n, plane, eA[im0 + m], eb, s);
#pragma unroll
    for (int j = 0; j < 4; ++j) sh[warp][4 * lane + j] = mk(re.v[j], im.v[j]);
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int t = 32 * j + lane;
    if (nw + t < N) out[m * ldo + nw + t] = sh[warp][t];
  }
}

__global__ void __launch_bounds__(256) out_real_kernel(const uint8_t* c, long ldc, long plane, long M, long N,
                                                       const int* eA, const int* eB, Scale s, double* out,
                                                       long ldo) {
  const long m = blockIdx.y, n = 4 * ((long)blockIdx.x * 256 + threadIdx.x);
  if (n >= N) return;
  int eb[4];
  load_e4(eB, n, N, eb);
  const Vals re = values4(c + m * ldc + n, plane, eA[m], eb, s);
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (n + j < N) out[m * ldo + n + j] = re.v[j];
}

// One Taylor term (see taylor_update) of R rows (w, a): items of four columns, both parts, over the R rows
// together, so that a block's threads stay busy whatever M is (100 items a row at M = 400: one row in a
// block of 128 threads left a fifth of the lanes idle).  Each complex element: 30 residues in, S in and
// out, 48 residues and magnitudes out; a row's T waits in shared memory for its norm.
template <bool LAST>
__global__ void __launch_bounds__(256, 4) taylor_kernel(const uint8_t* c, long ldc, long plane, long WN, int N, int M,
                                                     Scale sc, const int* eA, const int* eB, cplx* S, int8_t* q,
                                                     long ld, long qplane, int* e, Redo redo, int R, double mag) {
  extern __shared__ double rows[];  // [R][2][M4] T, then [R * M4 / 4] squared norms, [R] scales (negative: zeros)
  const int M4 = (M + 3) / 4 * 4, q4 = M4 / 4;
  double* part = rows + 2 * R * M4;
  double* scs = part + R * q4;
  if (redo.none_left(int(WN / N))) return;
  const long r0 = (long)blockIdx.x * R;
  const int nr = int(WN - r0 < R ? WN - r0 : R), items = nr * q4;
  for (int it = threadIdx.x; it < items; it += 256) {
    const int rr = it / q4, j0 = 4 * (it - rr * q4);
    const long r = r0 + rr;
    int eb[4];
    load_e4(eB + (r / N) * M, j0, M, eb);
    const int ea = eA[r];
    const Vals re = values4(c + r * ldc + j0, plane, ea, eb, sc);
    const Vals im = values4(c + (WN + r) * ldc + j0, plane, ea, eb, sc);
    cplx* Sr = S + r * M + j0;
    double n2 = 0.0, nz = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double x = 0.0, y = 0.0;
      if (j0 + j < M) {
        x = -im.v[j];  // T = (i / k) C
        y = re.v[j];
        Sr[j] = cadd(Sr[j], mk(x, y));
      }
      if (!LAST) {
        n2 = fma(x, x, fma(y, y, n2));
        nz = fmax(nz, fmax(fabs(x), fabs(y)));
        rows[(2 * rr) * M4 + j0 + j] = x;
        rows[(2 * rr + 1) * M4 + j0 + j] = y;
      }
    }
    if (!LAST) part[it] = n2 == 0.0 && nz != 0.0 ? 1e-320 : n2;  // squares that vanish: not a row of zeros
  }
  if (LAST) return;
  __syncthreads();
  for (int rr = threadIdx.x >> 5; rr < nr; rr += 8) {
    double n2 = 0.0;
    for (int i = threadIdx.x & 31; i < q4; i += 32) n2 += part[rr * q4 + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    if ((threadIdx.x & 31) == 0) {
      const int ex = row_exponent(n2, n2 != 0.0, true, redo, (r0 + rr) / N);
      e[r0 + rr] = ex;
      scs[rr] = n2 == 0.0 ? -1.0 : pow2(-ex);
    }
  }
  __syncthreads();
  for (int it = threadIdx.x; it < items; it += 256) {  // this thread's own entries again
    const int rr = it / q4, j0 = 4 * (it - rr * q4);
    int8_t* qr = q + (r0 + rr) * ld + j0;
    const Mag m = mag_of(mag, scs[rr] < 0.0);
    Quad d;
    d.set(rows + (2 * rr) * M4 + j0, scs[rr]);
    d.store(qr, qplane, m);
    d.set(rows + (2 * rr + 1) * M4 + j0, scs[rr]);
    d.store2(qr + WN * ld, qr + 2 * WN * ld, qplane, m);
  }
}

// One block per (n, w): the walker's T of this n, reconstructed once into shared memory, then its
// exchange trace.  Bound by the reconstruction (two residue groups per complex element) and its reads.
__global__ void __launch_bounds__(256) exx_kernel(const uint8_t* c, long ldc, long plane, long WN, int N, int N4,
                                                  const int* eA, long im0, const int* eB, int n0, int Nc, cplx* exxn,
                                                  cplx* kl, int nup, Redo redo, Scale sc) {
  extern __shared__ cplx T[];  // T[b][a], rows of P
  __shared__ cplx red[2][8];
  const int n = blockIdx.x, w = blockIdx.y, P = N | 1, q4 = N4 / 4;
  if (redo.asked(w)) return;
  for (int it = threadIdx.x; it < N * q4; it += 256) {
    const int b = it / q4, a = 4 * (it % q4);
    const long r = (long)w * N + b, col = (long)n * N4 + a;
    int eb[4];
    load_e4(eB + (long)n * N, a, N, eb);
    const Vals re = values4(c + r * ldc + col, plane, eA[r], eb, sc);
    const Vals im = values4(c + (WN + r) * ldc + col, plane, eA[im0 + r], eb, sc);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (a + j < N) T[b * P + a + j] = mk(re.v[j], im.v[j]);
  }
  __syncthreads();
  cplx acc = mk(0.0, 0.0), tr = mk(0.0, 0.0);
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x >> 5; i < N; i += 8) {
    const int j0 = i < nup ? 0 : nup, j1 = i < nup ? nup : N;  // orbitals of i's spin
    for (int j = j0 + lane; j < j1; j += 32) {
      const cplx x = T[i * P + j], y = T[j * P + i];
      acc.x = fma(x.x, y.x, fma(-x.y, y.y, acc.x));
      acc.y = fma(x.x, y.y, fma(x.y, y.x, acc.y));
    }
    if (lane == 0) tr = cadd(tr, T[i * P + i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    tr.x += __shfl_xor_sync(0xffffffffu, tr.x, o);
    tr.y += __shfl_xor_sync(0xffffffffu, tr.y, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = acc;
    red[1][threadIdx.x >> 5] = tr;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    cplx s = mk(0.0, 0.0);
    for (int i = 0; i < 8; ++i) s = cadd(s, red[threadIdx.x][i]);
    (threadIdx.x == 0 ? exxn : kl)[(long)w * Nc + n0 + n] = s;
  }
}

}  // namespace

Scale scale_of(double alpha) {
  constexpr Tables t = make_tables();
  Scale s;
  s.hi = alpha * t.P_hi;
  s.lo = std::fma(alpha, t.P_hi, -s.hi) + alpha * t.P_lo;
  return s;
}

int rows_real(const double* src, long rows, long K, long stride, const Planes& o, Redo redo, long per_walker,
              cudaStream_t st, long inner, long outer) {
  if (rows <= 0 || K <= 0) return SFQ_OK;
  const int vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && stride % 2 == 0;
  if (K < 1024)
    rows_real_kernel<32><<<ceil_div(rows, 8), 256, 0, st>>>(src, rows, K, stride, o.q, o.ld, o.plane, o.e, redo,
                                                            per_walker, vec, inner, outer, mag_scale(K));
  else
    rows_real_kernel<256><<<unsigned(rows), 256, 0, st>>>(src, rows, K, stride, o.q, o.ld, o.plane, o.e, redo,
                                                          per_walker, vec, inner, outer, mag_scale(K));
  SFQ_LAUNCHED();
  return SFQ_OK;
}

int rows_cplx(const cplx* src, long rows, long K, long stride, Parts parts, long blk, long inner, long outer,
              const Planes& o, Redo redo, long per_walker, cudaStream_t st) {
  if (rows <= 0 || K <= 0) return SFQ_OK;
  const bool wide = K >= 1024;
  const unsigned grid = wide ? unsigned(rows) : unsigned(ceil_div(rows, 8));
  auto k = parts == Parts::kApart ? (wide ? rows_cplx_kernel<256, Parts::kApart> : rows_cplx_kernel<32, Parts::kApart>)
           : parts == Parts::kJoint
               ? (wide ? rows_cplx_kernel<256, Parts::kJoint> : rows_cplx_kernel<32, Parts::kJoint>)
               : (wide ? rows_cplx_kernel<256, Parts::kJointNeg> : rows_cplx_kernel<32, Parts::kJointNeg>);
  k<<<grid, 256, 0, st>>>(src, rows, K, stride, blk, inner, outer, o.q, o.ld, o.plane, o.e, redo, per_walker,
                          mag_scale(K));
  SFQ_LAUNCHED();
  return SFQ_OK;
}

int pass_padding(const Planes& o, cudaStream_t st) {
  SFQ_CUDA_TRY(cudaMemsetAsync(o.q + NMOD * o.plane, 127, (size_t)o.rows * o.ld, st));
  return SFQ_OK;
}

int walkers_in(const cplx* SM, int W, int npol, int M, int N, const Planes& o, cplx* S, Redo redo, cudaStream_t st) {
  walkers_in_kernel<<<dim3((N + 15) / 16, W * npol), 256, 0, st>>>(SM, W * npol, npol, M, N, o.q, o.ld, o.plane, o.e, S,
                                                                   redo, mag_scale(M));
  SFQ_LAUNCHED();
  return SFQ_OK;
}

int out_cplx(const Out& c, long M, long N, const int* eA, long im, const int* eB, double alpha, cplx* out, long ldo,
             cudaStream_t st) {
  out_cplx_kernel<<<dim3(ceil_div(N, 1024), unsigned(M)), 256, 0, st>>>(c.q, c.ldc, c.plane, M, N, eA, im, eB, scale_of(alpha), out,
                                                                        ldo);
  SFQ_LAUNCHED();
  return SFQ_OK;
}

int out_real(const Out& c, long M, long N, const int* eA, const int* eB, double alpha, double* out, long ldo,
             cudaStream_t st) {
  out_real_kernel<<<dim3(ceil_div(N, 1024), unsigned(M)), 256, 0, st>>>(c.q, c.ldc, c.plane, M, N, eA, eB, scale_of(alpha), out,
                                                                        ldo);
  SFQ_LAUNCHED();
  return SFQ_OK;
}

// of one row of 4096 orbitals, the most that the propagation takes this way
constexpr size_t kTaylorSmem = sizeof(double) * (2 * 4096 + 4096 / 4 + 1);

int taylor_update(const Out& c, int W, int N, int M, int k, bool last, const int* eA, const int* eB, cplx* S,
                  const Planes& o, Redo redo, cudaStream_t st) {
  const int M4 = (M + 3) / 4 * 4, q4 = M4 / 4;
  const long WN = (long)W * N;
  // rows per block: the count up to 8 that wastes least of the last round of 256 items, in 48 KB of rows
  int R = 1;
  double best = 0.0;
  for (int n = 1; n <= 8 && (n == 1 || 16L * n * M4 <= 40 * 1024); ++n) {
    const double use = double(n) * q4 / ((n * q4 + 255) / 256 * 256);
    if (use > best + 0.02) {
      best = use;
      R = n;
    }
  }
  const size_t sm = sizeof(double) * (2L * R * M4 + (long)R * q4 + R);
  auto kern = last ? taylor_kernel<true> : taylor_kernel<false>;
  if (sm > kTaylorSmem) return record_error(SFQ_ERR_SHAPE, "crt taylor: M=%d too large", M);
  SFQ_MAX_SMEM(kern, kTaylorSmem);
  kern<<<unsigned((WN + R - 1) / R), 256, sm, st>>>(c.q, c.ldc, c.plane, WN, N, M, scale_of(1.0 / double(k)), eA, eB, S,
                                                    o.q, o.ld, o.plane, o.e, redo, R, mag_scale(M));
  SFQ_LAUNCHED();
  return SFQ_OK;
}

int exx_reduce(const Out& c, int W, int N, int N4, int nv, int n0, int Nc, const int* eA, long im, const int* eB,
               cplx* exxn, cplx* kl, int nup, Redo redo, cudaStream_t st) {
  const size_t sm = sizeof(cplx) * N * (N | 1);
  if (N > kExxMaxN) return record_error(SFQ_ERR_SHAPE, "crt exx: N=%d above %d", N, kExxMaxN);
  SFQ_MAX_SMEM(exx_kernel, sizeof(cplx) * kExxMaxN * (kExxMaxN | 1));
  exx_kernel<<<dim3(nv, W), 256, sm, st>>>(c.q, c.ldc, c.plane, (long)W * N, N, N4, eA, im, eB, n0, Nc, exxn, kl,
                                           nup < 0 ? N : nup, redo, scale_of(1.0));
  SFQ_LAUNCHED();
  return SFQ_OK;
}

}  // namespace crt
}  // namespace sfq
