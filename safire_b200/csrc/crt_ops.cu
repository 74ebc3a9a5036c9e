// The FP64 path's large products on the int8 tensor cores (see crt.cuh): force bias, vHS and the
// propagation.  Each raises flags where the modular scheme cannot hold an operand, and launches the
// FP64 tensor-pipe version behind it for the walkers that the flags name.
#include "crt.cuh"
#include "crt_ops.cuh"
#include "ops.cuh"

#include <algorithm>
#include <cmath>

namespace sfq {
namespace ops {
using namespace crt;

namespace {
// What a call holds of the shared operand at a time, with its output, and of the walkers' operand: large enough to fill
// the GPU several times over.  A call's scratch is bounded by two of these, whatever its sizes (but one walker's and 256
// rows' worth are always held).
constexpr size_t kChunkBytes = size_t(3) << 29;  // 1.5 GiB

size_t slack() { return 256 * (2 * kPlanes + 4); }  // plane roundings
// n in equal parts of at most `most`
long part_of(long n, long most) {
  const long parts = (n + most - 1) / most;
  return parts <= 1 ? n : (n + parts - 1) / parts;
}
// walkers at a time, each with `bytes` of planes
int walkers_at_a_time(int W, size_t bytes) { return int(part_of(W, std::max<long>(1, long(kChunkBytes / bytes)))); }
// rows of the shared operand at a time: all of them, or equal parts of a multiple of 16 rows
long rows_at_a_time(long rows, size_t row_bytes) {
  const long n = part_of(rows, std::max<long>(256, long(kChunkBytes / row_bytes)));
  return n == rows ? rows : (n + 15) / 16 * 16;
}
// force bias and vHS, of `rows` shared rows of K (planes of them made once: prepared): walkers and rows at a time
struct Parted {
  int w;
  long n;
};
Parted part(int W, long rows, long K, int a_blocks, int b_blocks, bool all_rows) {
  Parted p;
  p.w = walkers_at_a_time(W, (size_t)kPlanes * a_blocks * ld_of(K) + (all_rows ? (size_t)NMOD * 2 * rows : 0));
  p.n = all_rows ? rows : rows_at_a_time(rows, (size_t)kPlanes * b_blocks * ld_of(K) + (size_t)NMOD * 2 * p.w + sizeof(int));
  return p;
}
size_t parted_bytes(int W, const Parted& p, long K, int a_blocks, int b_blocks, bool prepared) {
  size_t b = flag_bytes(W) + planes_bytes((long)a_blocks * p.w, K) + exps_bytes(2L * p.w) + out_bytes(2L * p.w, p.n);
  if (!prepared) b += planes_bytes(b_blocks * p.n, K) + exps_bytes(p.n);
  return b + slack();
}
}  // namespace

// ---- force bias -----------------------------------------------------------------------------------
size_t vbias_crt_bytes(int W, int N, int M, int Nc, bool l_cplx, bool prepared) {
  const long K = (long)N * M;
  const int na = l_cplx ? 3 : 2, nb = l_cplx ? 2 : 1;
  return parted_bytes(W, part(W, Nc, K, na, nb, prepared), K, na, nb, prepared);
}

// The FP64 tensor-pipe product walks K = N M in one chain per tile, of few tiles; this path's launches cost more and its
// time hardly depends on W: with 8 walkers 64 us against 123 at K = 4096, Nc = 640, and 0.95 ms against 1.98 at
// K = 40000, Nc = 2400.  At K = 1024 the outputs decide: 37 against 35 us with 8 x 640 of them, 41 against 35 with
// 300 x 65 (K = 1030), 39 against 43 with 64 x 640, 45 against 59 with 256 x 640; a complex Lnak, twice the flops there,
// gains from K = 2323 (70 against 78 us) on at least.
bool vbias_crt_ok(int W, int N, int M, int Nc, bool l_cplx) {
  const long K = (long)N * M;
  return W >= 8 && W <= 65535 && Nc >= 64 && K >= 1024 && K * (l_cplx ? 2 : 1) <= kMaxK;
}
bool vbias_crt_gains(int W, int N, int M, int Nc, bool l_cplx) {
  return l_cplx || (long)N * M >= 1536 || (long)W * Nc >= 40000;
}

int vbias_crt(const cplx* G, const void* Lnak, bool l_cplx, const Planes* Lq, cplx* v, int W, int N, int M, int Nc,
              double a, char* ws, cudaStream_t st) {
  const long K = (long)N * M;
  const int na = l_cplx ? 3 : 2, nb = l_cplx ? 2 : 1;
  const Parted p = part(W, Nc, K, na, nb, Lq != nullptr);
  char* at = ws;
  const Redo redo = lay_out_flags(at, W);
  int rc;
  SFQ_CUDA_TRY(cudaMemsetAsync(redo.call, 0, flag_bytes(W), st));
  Planes A = lay_out(at, (long)na * p.w, K, 2L * p.w);
  Planes B = Lq ? *Lq : lay_out(at, nb * p.n, K, p.n);
  Out C = lay_out_c(at, 2L * p.w, p.n);
  for (long n0 = 0; n0 < Nc; n0 += p.n) {
    const long n = std::min<long>(p.n, Nc - n0);
    if (!Lq) {
      if (l_cplx) rc = rows_cplx((const cplx*)Lnak + n0 * K, n, K, K, Parts::kJoint, p.n, n, n, B, redo, 0, st);
      else rc = rows_real((const double*)Lnak + n0 * K, n, K, K, B, redo, 0, st);
      if (rc) return rc;
    }
    for (int w0 = 0; w0 < W; w0 += p.w) {
      const int w = std::min(p.w, W - w0);
      const Redo rw{redo.call, redo.row + w0};
      if ((n0 == 0 || p.w < W) && (rc = rows_cplx(G + w0 * K, w, K, K, l_cplx ? Parts::kJointNeg : Parts::kApart, w, w,
                                                  w, A, rw, 1, st)))
        return rc;
      crt::Gemm g;
      g.A = A; g.B = B; g.K = int(K); g.N = int(n);
      if (l_cplx) {
        g.M = w; g.parts = g.segs = 2;
        g.a_off[0][0] = 0; g.a_off[0][1] = 2L * w; g.a_off[1][0] = w; g.a_off[1][1] = 0;
        g.b_off[1] = Lq ? Nc : p.n;
      } else {
        g.M = 2 * w;
      }
      Out c = C;
      c.ldc = ldc_of(n);
      g.C = c.q; g.ldc = c.ldc; g.c_plane = c.plane; g.redo = rw; g.wmod = w;
      if ((rc = crt::gemm(g, st))) return rc;
      if ((rc = out_cplx(c, w, n, A.e, l_cplx ? 0 : w, B.e, a, v + (long)w0 * Nc + n0, Nc, st))) return rc;
    }
  }
  return vbias(G, Lnak, l_cplx, v, W, N, M, Nc, a, st, &redo);
}

// ---- vHS --------------------------------------------------------------------------------------
size_t vhs_crt_bytes(int W, long rows, int Nc, bool prepared) {
  return parted_bytes(W, part(W, rows, Nc, 2, 1, false), Nc, 2, 1, prepared);
}

// Converting L (M^2 Nc elements) costs what the FP64 product of about 64 walkers does: 160 us against 186 with 96 walkers
// at M = 128, Nc = 640, 167 against 222 with 128, 0.98 ms against 1.57 with 96 at M = 256, Nc = 1536, 4.96 against
// 13.2 with 256 at M = 400, Nc = 2400; at 64 it is even.  With L's planes prepared the product alone counts.
bool vhs_crt_ok(int W, long rows, int Nc, bool prepared) {
  const double flops = 4.0 * W * double(rows) * Nc;
  if (W > 65535 || Nc > kMaxK || Nc < 96) return false;
  return prepared ? W >= 32 && flops >= 1e9 : W >= 96 && flops >= 4e9;
}

int vhs_crt(const double* L, long rows, const Planes* Lq, const cplx* X, cplx* V, int W, int Nc, double a, char* ws,
            cudaStream_t st) {
  const Parted p = part(W, rows, Nc, 2, 1, false);
  char* at = ws;
  const Redo redo = lay_out_flags(at, W);
  int rc;
  SFQ_CUDA_TRY(cudaMemsetAsync(redo.call, 0, flag_bytes(W), st));
  Planes A = lay_out(at, 2L * p.w, Nc, 2L * p.w);
  Planes B = Lq ? *Lq : lay_out(at, p.n, Nc, p.n);
  Out C = lay_out_c(at, 2L * p.w, p.n);
  for (long r0 = 0; r0 < rows; r0 += p.n) {
    const long n = std::min<long>(p.n, rows - r0);
    if (!Lq && (rc = rows_real(L + r0 * Nc, n, Nc, Nc, B, redo, 0, st))) return rc;
    for (int w0 = 0; w0 < W; w0 += p.w) {
      const int w = std::min(p.w, W - w0);
      const Redo rw{redo.call, redo.row + w0};
      if ((r0 == 0 || p.w < W) &&
          (rc = rows_cplx(X + (long)w0 * Nc, w, Nc, Nc, Parts::kApart, w, w, w, A, rw, 1, st)))
        return rc;
      crt::Gemm g;
      g.A = A; g.B = B; g.M = 2 * w; g.N = int(n); g.K = Nc;
      g.b_off[0] = Lq ? r0 : 0;
      Out c = C;
      c.ldc = ldc_of(n);
      g.C = c.q; g.ldc = c.ldc; g.c_plane = c.plane; g.redo = rw; g.wmod = w;
      if ((rc = crt::gemm(g, st))) return rc;
      if ((rc = out_cplx(c, w, n, A.e, w, B.e + (Lq ? r0 : 0), a, V + w0 * rows + r0, rows, st))) return rc;
    }
  }
  return vhs_rows(L, rows, X, V, W, Nc, a, st, &redo);
}

// ---- propagation --------------------------------------------------------------------------------
namespace {
size_t prop_walker_bytes(int M, int Nr) {  // Nr = npol * N rows per walker
  return (size_t)kPlanes * (3 * (size_t)Nr * ld_of(M) + 2 * (size_t)M * ld_of(M)) + (size_t)NMOD * 2 * Nr * ldc_of(M) +
         32 * (size_t)Nr * M + 4 * (size_t)(Nr + M);
}
int prop_chunk(int W, int M, int Nr) { return walkers_at_a_time(W, prop_walker_bytes(M, Nr)); }
}  // namespace

size_t propagate_crt_bytes(int W, int M, int N, int npol) {
  const int Nr = N * npol, wc = prop_chunk(W, M, Nr);
  const long R = (long)wc * Nr;
  const size_t blk = align256(sizeof(cplx) * (size_t)R * M);
  const size_t b = planes_bytes(3 * R, M) + exps_bytes(R) + planes_bytes(2L * wc * M, M) + exps_bytes((long)wc * M) +
                   out_bytes(2 * R, M) + blk;
  return flag_bytes(wc) + blk + std::max(b, 2 * blk) + slack();  // the FP64 terms' buffers share the space
}

// The conversion of V and of the terms grows as M^2 and M N, the products as M^2 N a term.  Order 6, this path against
// the FP64 tensor pipe: 7.17 ms against 11.3 at M = 400 with 100 electrons and 256 walkers, 4.45 against 4.97 with 48,
// 0.71 against 0.81 with 100 and 16 walkers; 1.21 against 1.31 at M = 256 with 64 and 128; even with 64 walkers there,
// 0.76 against 0.68 at M = 240 with 48 and 80.  V is converted once for all terms: order 1, 2, 3, 4 take 0.50, 0.64,
// 0.78, 0.92 ms against 0.41, 0.59, 0.77, 0.95 at M = 256 (128 walkers), 3.40 and 4.15 against 3.45 and 5.02 for 1 and
// 2 at M = 400.
bool propagate_crt_ok(int W, int M, int N, int npol, bool p_cplx, int order) {
  const double flops = 64.0 * W * M * double(M) * N * npol;
  return !p_cplx && (long)order * M >= 800 && W <= 30000 && M >= 250 && M <= 4096 && N * npol >= 48 && flops >= 1.4e10 &&
         walker_gemm_fits(N * npol, M, M, 2);
}

// P1 is the identity and a little more: a product with it keeps the small elements of the walkers to their own bits in
// FP64, and would fail the magnitudes' check here, so both stay on the FP64 tensor pipe (4 M^2 N of 64 M^2 N flops each).
int propagate_crt(cplx* SM, const double* P1, const cplx* V, int W, int M, int N, int npol, int order, char* ws,
                  cudaStream_t st) {
  const int Nr = N * npol, wc = prop_chunk(W, M, Nr);
  const long MN = (long)M * N;
  char* at = ws;
  const Redo rw = lay_out_flags(at, wc);
  int rc;
  for (int w0 = 0; w0 < W; w0 += wc) {
    const int w = std::min(wc, W - w0);
    const long R = (long)w * Nr;
    const size_t blk = align256(sizeof(cplx) * (size_t)R * M);
    SFQ_CUDA_TRY(cudaMemsetAsync(rw.call, 0, flag_bytes(wc), st));
    cplx* S0 = SM + (long)w0 * Nr * M;
    const cplx* Vw = V + (long)w0 * M * M;
    cplx* TMN = reinterpret_cast<cplx*>(at);
    char* o = at + blk;
    Planes A = lay_out(o, 3 * R, M, R);
    Planes B = lay_out(o, 2L * w * M, M, (long)w * M);
    Out C = lay_out_c(o, 2 * R, M);
    cplx* S = reinterpret_cast<cplx*>(o);  // rows (w, q, a) over the orbitals
    if ((rc = p1_apply(P1, false, S0, TMN, w, npol, M, N, st))) return rc;
    if ((rc = walkers_in(TMN, w, npol, M, N, A, S, rw, st))) return rc;
    if ((rc = rows_cplx(Vw, (long)w * M, M, M, Parts::kJoint, M, M, 2L * M, B, rw, M, st))) return rc;
    crt::WalkerGemm t;  // C = V T: re = Vr Tr + Vi (-Ti), im = Vr Ti + Vi Tr
    t.A = A; t.B = B; t.N = Nr; t.cols = M; t.K = M; t.batch = w; t.segs = 2;
    t.a_blk = R; t.b_bs = 2L * M; t.b_off1 = M;
    t.C = C.q; t.ldc = C.ldc; t.c_plane = C.plane; t.c_part = R; t.redo = rw;
    for (int k = 1; k <= order; ++k) {
      if ((rc = crt::walker_gemm(t, st))) return rc;
      if ((rc = taylor_update(C, w, Nr, M, k, k == order, A.e, B.e, S, A, rw, st))) return rc;
    }
    for (int q = 0; q < npol; ++q) {  // SM = P1 S of the walkers that passed
      GemmDesc d;
      d.M = M; d.N = N; d.K = M; d.batch = w;
      d.A = P1; d.sAm = M; d.sAk = 1;
      d.B = S + q * MN; d.sBk = 1; d.sBn = M; d.sBb = npol * MN; d.b_cplx = true;
      d.C = S0 + q * MN; d.sCm = N; d.sCn = 1; d.sCb = npol * MN;
      d.redo = rw; d.redo_rest = true;
      if ((rc = gemm_f64(d, st))) return rc;
    }
    cplx* T1 = reinterpret_cast<cplx*>(at + blk);
    if ((rc = taylor(TMN, Vw, w, M, N, npol, order, T1, reinterpret_cast<cplx*>(at + 2 * blk), st, &rw))) return rc;
    if ((rc = p1_apply(P1, false, TMN, S0, w, npol, M, N, st, &rw))) return rc;
  }
  return SFQ_OK;
}

// ---- local energy ---------------------------------------------------------------------------
namespace {
int n4_of(int N) { return (N + 3) / 4 * 4; }
int energy_walkers(int W, int N, int M, bool l_cplx) {
  return walkers_at_a_time(W, (size_t)kPlanes * (l_cplx ? 3 : 2) * N * ld_of(M));
}
size_t energy_n_bytes(int w, int N, int M, bool l_cplx) {  // per Cholesky vector
  return (size_t)kPlanes * (l_cplx ? 2 : 1) * n4_of(N) * ld_of(M) + (size_t)NMOD * 2 * w * N * n4_of(N) +
         sizeof(int) * N;
}
int energy_nv(int w, int N, int M, int Nc, bool l_cplx) {
  return int(part_of(Nc, std::max<long>(1, long(kChunkBytes / energy_n_bytes(w, N, M, l_cplx)))));
}
}  // namespace

// A walker's [re; im] rows fill 128-row tiles: with 50 electrons 112 of them, with 32 half, where the product and the
// reconstruction together take what the FP64 product does.  Below 40 GFLOP (about a millisecond there) its launches
// count.  Storing and reconstructing T does not depend on M, the FP64 product does: 1.65 ms against 1.47 at M = 150 and
// 1.67 both at 180 (20 walkers, N = 45, Nc = 1100), 4.05 against 4.68 at 170 (64, 50, 900), 3.74 against 3.26 at 160 and
// 3.84 against 4.39 at 240 (24, 80, 700), 2.29 both at 200 (12, 100, 500), 11.6 against 13.9 at 200 (128, 50, 1200); with a
// complex Lnak, twice the flops there, 2.26 both at M = 90 (30, 45, 900), 2.29 against 2.58 at 90 (16, 70, 800), 1.89
// against 2.54 at 110 (30, 45, 900).
bool energy_crt_ok(int W, int N, int M, int Nc, bool l_cplx) {
  return W <= 65535 && N >= 40 && N <= kExxMaxN && M >= 32 && 8.0 * W * N * double(N) * M * Nc >= 4e10 &&
         energy_n_bytes(energy_walkers(W, N, M, l_cplx), N, M, l_cplx) <= kChunkBytes &&
         walker_gemm_fits(N, 16 * n4_of(N), M, l_cplx ? 2 : 1);
}

bool energy_crt_gains(int M, bool l_cplx) { return M * (l_cplx ? 2 : 1) >= 180; }

size_t energy_crt_bytes(int W, int N, int M, int Nc, bool l_cplx) {
  const int w = energy_walkers(W, N, M, l_cplx), nv = energy_nv(w, N, M, Nc, l_cplx), N4 = n4_of(N);
  const long R = (long)w * N;
  return flag_bytes(w) + planes_bytes((l_cplx ? 3 : 2) * R, M) + exps_bytes(2 * R) +
         planes_bytes((l_cplx ? 2L : 1L) * nv * N4, M) + exps_bytes((long)nv * N) + out_bytes(2 * R, (long)nv * N4) +
         slack();
}

int energy_crt(cplx* E3, const cplx* G, const cplx* haj, const void* Lnak, bool l_cplx, double E0, int W, int N, int M,
               int Nc, int addH1, int addEJ, char* scratch, size_t bytes, cplx* exxn, cplx* kl, cudaStream_t st,
               int nup) {
  int rc;
  const double scl = nup < 0 ? 2.0 : 1.0;
  const int wc = energy_walkers(W, N, M, l_cplx), nv = energy_nv(wc, N, M, Nc, l_cplx), N4 = n4_of(N);
  if ((rc = energy_e1(G, haj, E3, W, N, M, E0, scl, addH1, st))) return rc;
  for (int w0 = 0; w0 < W; w0 += wc) {
    const int w = std::min(wc, W - w0);
    const long R = (long)w * N;
    const cplx* Gw = G + (long)w0 * N * M;
    cplx *ew = exxn + (long)w0 * Nc, *kw = kl + (long)w0 * Nc;
    char* at = scratch;
    const Redo redo = lay_out_flags(at, wc);
    // the FP64 product's chunk takes the same space afterwards: 16 w N^2 bytes a vector at least, less than C's
    cplx* Tchunk = reinterpret_cast<cplx*>(at);
    const long tchunk = std::min<long>(long((bytes - flag_bytes(wc)) / sizeof(cplx)), 1L << 27);
    SFQ_CUDA_TRY(cudaMemsetAsync(redo.call, 0, flag_bytes(wc), st));
    const Planes A = lay_out(at, (l_cplx ? 3 : 2) * R, M, 2 * R);
    const Planes B = lay_out(at, (l_cplx ? 2L : 1L) * nv * N4, M, (long)nv * N);
    const Out C = lay_out_c(at, 2 * R, (long)nv * N4);
    if ((rc = rows_cplx(Gw, R, M, M, l_cplx ? Parts::kJointNeg : Parts::kApart, R, R, R, A, redo, N, st))) return rc;
    if (N4 != N && (rc = pass_padding(B, st))) return rc;
    for (int n0 = 0; n0 < Nc; n0 += nv) {
      const int n = std::min(nv, Nc - n0);
      // rows (n, a) of Lnak on rows n N4 + a: the columns of a vector then start on words
      const long off = (long)n0 * N * M;
      if (l_cplx)
        rc = rows_cplx((const cplx*)Lnak + off, (long)n * N, M, M, Parts::kJoint, (long)nv * N4, N, N4, B, redo, 0, st);
      else
        rc = rows_real((const double*)Lnak + off, (long)n * N, M, M, B, redo, 0, st, N, N4);
      if (rc) return rc;
      crt::WalkerGemm g;
      g.A = A; g.B = B; g.N = N; g.cols = n * N4; g.K = M; g.batch = w; g.segs = l_cplx ? 2 : 1;
      g.a_blk = R; g.b_off1 = (long)nv * N4;
      Out c = C;
      c.ldc = ldc_of((long)n * N4);
      g.C = c.q; g.ldc = c.ldc; g.c_plane = c.plane; g.c_part = R; g.redo = redo;
      if ((rc = crt::walker_gemm(g, st))) return rc;
      if ((rc = exx_reduce(c, w, N, N4, n, n0, Nc, A.e, l_cplx ? 0 : R, B.e, ew, kw, nup, redo, st))) return rc;
    }
    if ((rc = energy_exx_f64(Gw, Lnak, l_cplx, w, N, M, Nc, Tchunk, tchunk, ew, kw, st, nup, &redo))) return rc;
  }
  return energy_finish(exxn, kl, E3, W, Nc, scl, 1, addEJ, st);
}

}  // namespace ops
}  // namespace sfq

namespace sfq {
namespace {
// C = A B^T by either kernel, the bare product; the self-test's limit and hold, and whether a wait expired
int modular_product(const double* A, const double* B, double* C, int M, int N, int K, bool walker, cudaStream_t st,
                    unsigned long long wait_ns = 0, int hold_at = -1, int* expired = nullptr) {
  char* ws = nullptr;
  const size_t bytes = crt::flag_bytes(M) + crt::planes_bytes(M, K) + crt::exps_bytes(M) + crt::planes_bytes(N, K) +
                       crt::exps_bytes(N) + crt::out_bytes(M, N);
  SFQ_CUDA_TRY(cudaMallocAsync((void**)&ws, bytes, st));
  char* at = ws;
  const Redo redo = crt::lay_out_flags(at, M);
  const int per = walker ? M : 1;  // rows of A to a walker
  const crt::Planes a = crt::lay_out(at, M, K, M), b = crt::lay_out(at, N, K, N);
  const crt::Out c = crt::lay_out_c(at, M, N);
  const int* hold = hold_at < 0 ? nullptr : redo.call + 4;  // nothing sets it
  int rc = SFQ_OK;
  cudaError_t ce = cudaMemsetAsync(redo.call, 0, crt::flag_bytes(M), st);
  if (ce != cudaSuccess) rc = record_cuda(ce, "gemm_f64_modular", __FILE__, __LINE__);
  if (!rc) rc = crt::rows_real(A, M, K, K, a, redo, per, st);
  if (!rc) rc = crt::rows_real(B, N, K, K, b, redo, 0, st);
  if (!rc && walker) {  // the rows as the [re; im] of one walker
    crt::WalkerGemm g;
    g.A = a; g.B = b; g.N = M / 2; g.cols = N; g.K = K; g.a_blk = M / 2;
    g.C = c.q; g.ldc = c.ldc; g.c_plane = c.plane; g.c_part = M / 2; g.redo = redo; g.check = false;
    g.wait_ns = wait_ns; g.hold = hold; g.hold_at = unsigned(hold_at);
    rc = crt::walker_gemm(g, st);
  } else if (!rc) {
    crt::Gemm g;
    g.A = a; g.B = b; g.M = M; g.N = N; g.K = K; g.C = c.q; g.ldc = c.ldc; g.c_plane = c.plane; g.redo = redo; g.wmod = M; g.check = false;
    g.wait_ns = wait_ns; g.hold = hold; g.hold_at = unsigned(hold_at);
    rc = crt::gemm(g, st);
  }
  if (!rc) rc = crt::out_real(c, M, N, a.e, b.e, 1.0, C, N, st);
  if (!rc) {
    GemmDesc d;
    d.M = M; d.N = N; d.K = K;
    d.A = A; d.sAm = K; d.sAk = 1;
    d.B = B; d.sBk = 1; d.sBn = K;
    d.C = C; d.sCm = N; d.sCn = 1;
    d.redo = redo;
    d.redo_div = per;
    rc = gemm_f64(d, st);
  }
  if (!rc && expired) {
    ce = cudaMemcpyAsync(expired, redo.call + 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
    if (ce != cudaSuccess) rc = record_cuda(ce, "gemm_f64_modular", __FILE__, __LINE__);
  }
  cudaFreeAsync(ws, st);
  return rc;
}
}  // namespace
}  // namespace sfq

extern "C" int sfq_gemm_f64_modular(const double* A, const double* B, double* C, int M, int N, int K, void* stream) {
  using namespace sfq;
  if (M < 0 || N < 0 || K < 0) return record_error(SFQ_ERR_SHAPE, "negative size");
  if (!M || !N) return SFQ_OK;
  if (!A || !B || !C) return record_error(SFQ_ERR_ARG, "null pointer");
  if (K < 1 || K > crt::kMaxK || M > 65535)
    return record_error(SFQ_ERR_SHAPE, "gemm_f64_modular: 1 <= K <= %ld, M <= 65535", crt::kMaxK);
  return modular_product(A, B, C, M, N, K, false, static_cast<cudaStream_t>(stream));
}

extern "C" int sfq_selftest_modular_expiry(const double* A, const double* B, double* C, int M, int N, int K, int walker,
                                           int hold_at, unsigned long long wait_ns, void* stream) {
  using namespace sfq;
  if (wait_ns == 0 || wait_ns > 1000000000ull) return record_error(SFQ_ERR_ARG, "selftest: wait of 1 ns .. 1 s");
  if (M < 2 || M > 65534 || M % 2 || N < 1 || K < 1 || K > 4096 || hold_at < 0)
    return record_error(SFQ_ERR_SHAPE, "selftest: M even, K <= 4096");
  if (!A || !B || !C) return record_error(SFQ_ERR_ARG, "null pointer");
  int expired = 0;
  const int rc = modular_product(A, B, C, M, N, K, walker != 0, static_cast<cudaStream_t>(stream), wait_ns, hold_at,
                                 &expired);
  return rc ? rc : expired ? SFQ_ERR_TIMEOUT : SFQ_OK;
}

extern "C" int sfq_modular_expiries(unsigned long long* n) {
  using namespace sfq;
  if (!n) return record_error(SFQ_ERR_ARG, "null pointer");
  return crt::expiries(n);
}
