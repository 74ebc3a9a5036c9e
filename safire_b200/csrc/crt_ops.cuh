// The FP64 path's products by modular arithmetic on the int8 tensor cores.  *_ok: whether it takes these sizes, *_gains
// (where there is one): whether it is then the faster path; *_bytes: device scratch of a call; Lq: the operand's planes
// prepared once (null: converted on every call).
#pragma once
#include "crt.cuh"

namespace sfq {
namespace ops {

bool vbias_crt_ok(int W, int N, int M, int Nc, bool l_cplx);
bool vbias_crt_gains(int W, int N, int M, int Nc, bool l_cplx);
size_t vbias_crt_bytes(int W, int N, int M, int Nc, bool l_cplx, bool prepared);
int vbias_crt(const cplx* G, const void* Lnak, bool l_cplx, const crt::Planes* Lq, cplx* v, int W, int N, int M,
              int Nc, double a, char* ws, cudaStream_t st);

bool vhs_crt_ok(int W, long rows, int Nc, bool prepared);
size_t vhs_crt_bytes(int W, long rows, int Nc, bool prepared);
int vhs_crt(const double* L, long rows, const crt::Planes* Lq, const cplx* X, cplx* V, int W, int Nc, double a,
            char* ws, cudaStream_t st);

bool propagate_crt_ok(int W, int M, int N, int npol, bool p_cplx, int order);
size_t propagate_crt_bytes(int W, int M, int N, int npol);
int propagate_crt(cplx* SM, const double* P1, const cplx* V, int W, int M, int N, int npol, int order, char* ws,
                  cudaStream_t st);

// the local energy (as ops::energy) with the exchange tensor's product this way, in `bytes` of scratch
bool energy_crt_ok(int W, int N, int M, int Nc, bool l_cplx);
bool energy_crt_gains(int M, bool l_cplx);
size_t energy_crt_bytes(int W, int N, int M, int Nc, bool l_cplx);
int energy_crt(cplx* E3, const cplx* G, const cplx* haj, const void* Lnak, bool l_cplx, double E0, int W, int N, int M,
               int Nc, int addH1, int addEJ, char* scratch, size_t bytes, cplx* exxn, cplx* kl, cudaStream_t st,
               int nup);

}  // namespace ops
}  // namespace sfq
