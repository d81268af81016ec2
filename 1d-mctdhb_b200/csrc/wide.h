// wide.h -- pair-space H.C and densities for more than 8 orbitals (wide.cu).
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace mctdhb {

// FP64 mma.sync m8n8k4: lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4)], D[l/4][2(l%4) + 1]
__device__ __forceinline__ void wide_dmma884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// whether the wide kernels apply to (N, M): N >= 2, 8 < M <= 30
bool wide_eligible(int N, int M);
// launch attributes (call before any stream capture)
int wide_prepare();
// the pair matrix of h and g into sp.pair_w
int wide_prep(const SpaceView& sp, const double2* hob, const double2* hint, cudaStream_t st);
// HC = H C (with the Lanczos epilogue) through the scratch sp.pair_y
int wide_hc(const SpaceView& sp, const double2* C, double2* HC, const HcEpilogue& ep,
            cudaStream_t st);
// rho1 and rho2; `partial` holds wide_gram_elems(M, D2) complex, D2 = D(N-2, M)
size_t wide_gram_elems(int M, uint32_t D2);
int wide_dens(const SpaceView& sp, uint32_t D2, const double2* C, double2* partial, double2* rho1,
              double2* rho2, cudaStream_t st);

}  // namespace mctdhb
