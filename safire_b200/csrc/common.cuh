// Shared device/host helpers for the SAFIRE-B200 AFQMC kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstddef>

#include "../../include/safire_b200.h"

namespace sfq {

// ---- complex double helpers (interleaved re,im -- the layout of std::complex<double>) -------
struct __align__(16) cplx {
  double x, y;
};

__host__ __device__ __forceinline__ cplx mk(double r, double i) { cplx c; c.x = r; c.y = i; return c; }
__host__ __device__ __forceinline__ cplx cadd(cplx a, cplx b) { return mk(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ cplx csub(cplx a, cplx b) { return mk(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ cplx cmul(cplx a, cplx b) {
  return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ cplx cscale(cplx a, double s) { return mk(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ cplx cconj(cplx a) { return mk(a.x, -a.y); }
__device__ __forceinline__ double cabs_(cplx a) { return hypot(a.x, a.y); }
// Smith's algorithm for a/b
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  if (fabs(b.x) >= fabs(b.y)) {
    double r = b.y / b.x, d = b.x + r * b.y;
    return mk((a.x + a.y * r) / d, (a.y - a.x * r) / d);
  } else {
    double r = b.x / b.y, d = b.y + r * b.x;
    return mk((a.x * r + a.y) / d, (a.y * r - a.x) / d);
  }
}
// principal complex log
__device__ __forceinline__ cplx clog_(cplx a) { return mk(log(hypot(a.x, a.y)), atan2(a.y, a.x)); }
__device__ __forceinline__ cplx cexp_(cplx a) {
  double e = exp(a.x);
  double s, c;
  sincos(a.y, &s, &c);
  return mk(e * c, e * s);
}

// ---- error reporting -------------------------------------------------------------------
#define SFQ_CUDA_TRY(expr)                                    \
  do {                                                        \
    cudaError_t _e = (expr);                                  \
    if (_e != cudaSuccess) return ::sfq::record_cuda(_e, #expr, __FILE__, __LINE__); \
  } while (0)

int record_cuda(cudaError_t e, const char* what, const char* file, int line);
void count_launch();

// after every kernel launch: count it and surface launch-configuration errors
#define SFQ_LAUNCHED()                        \
  do {                                        \
    ::sfq::count_launch();                    \
    SFQ_CUDA_TRY(cudaGetLastError());         \
  } while (0)
int record_error(int code, const char* fmt, ...);

// A kernel's dynamic shared-memory limit belongs to the function, not to the launch: it is always set to the
// kernel's largest, so that a call never lowers it between another host thread's setting and launch, nor below
// what a captured graph's node needs.
#define SFQ_MAX_SMEM(kernel, bytes) \
  SFQ_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)))

// What a modular product (crt.cuh) could not hold and asks of the FP64 kernels launched behind it, in device memory:
// call[0] (an operand that all walkers share) or call[1] (an expired wait): the whole call, row[w]: walker w, and
// call[2] the number of such walkers.  One load tells the many blocks of those kernels that nothing is asked for.
// call[3] is call[2] as the last modular product found it: kernels that may raise flags themselves, in which call[2] could
// change under way, look at that to see whether any walker is left for them.
struct Redo {
  int* call = nullptr;  // four of them, on a 16-byte boundary
  int* row = nullptr;
#ifdef __CUDACC__
  __device__ __forceinline__ int4 asked() const { return *reinterpret_cast<const int4*>(call); }
  __device__ __forceinline__ bool asked(long w) const {
    const int4 c = asked();
    return (c.x | c.y) != 0 || (c.z != 0 && row[w] != 0);
  }
  __device__ __forceinline__ bool all_asked(int nwalk) const {
    const int4 c = asked();
    return c.x != 0 || c.z == nwalk;
  }
  __device__ __forceinline__ void settle() const { call[3] = call[2]; }
  __device__ __forceinline__ bool none_left(int nwalk) const { return call[3] == nwalk; }
  __device__ __forceinline__ void ask(long w) const {
    if (!row[w] && atomicExch(row + w, 1) == 0) atomicAdd(call + 2, 1);
  }
  __device__ __forceinline__ void ask_all() const { call[0] = 1; }
#endif
};

inline int ceil_div(long a, long b) { return int((a + b - 1) / b); }

}  // namespace sfq
