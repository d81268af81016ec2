// smallsys.h -- H.C and the short iterative Lanczos step of a small Fock space on
// one cluster of blocks (smallsys.cuh): H.C in one launch; a step of one system in
// two an iteration and one for the combination (its densities take the Gram
// kernels); in the batch the recurrence, the combination and rho2 in one each.
#pragma once
#include "batch.h"
#include "common.cuh"
#include "kernels.h"

namespace mctdhb {

// Spaces this path takes: 2..8 orbitals, N >= 2.  One product is two
// cluster-wide passes on eight SMs, which save launches; beyond, the whole GPU's
// tensor cores win.  Measured on one B200, here against the general path:
//   one product, up to 0.25 M complex multiply-adds of the contraction (rows of
//     the (N-2)-space times pairs^2): 0.02 M (N=10 M=4)  8.4 us against 12.0;
//     0.23 M (N=24 M=4) level; 0.45 M (N=30 M=4) 16.7 against 13
//   a step of one system, up to 2,048 rows, one a thread, and up to 4,096 where
//     a product has at most 0.21 M.  Captured steps of 5 vectors with densities:
//     1,501 rows (N=1500 M=2) 82 us against 86; 1,716 (N=6 M=8) 145 against
//     158; 2,145 (N=64 M=3) 101 against 103; 2,556 (N=70 M=3) 111 against 99;
//     2,600 (N=23 M=4, 0.20 M) 111 against 119; 4,001 (N=4000 M=2) 95 against
//     97.  Past the line: 2,380 (N=13 M=5, 0.31 M) 127 against 123; 2,925 (N=24
//     M=4, 0.23 M) 123 against 119; 4,656 (N=95 M=3) 130 against 109; 5,001
//     (N=5000 M=2) 109 against 99; 18,336 (N=190 M=3) 230 against 111.  A step
//     by the reference's C entry, where each launch costs the host time, in the
//     same order of sizes from 2,145 rows: 212 / 226 / 232 / 216 us against 238
//     / 241 / 257 / 233, past the line 248 / 241 / 258 / 236 against 259 / 257 /
//     261 / 241
//   a slot of the batch, where the general path's iteration has twice the
//     launches, up to 0.7 M: 0.69 M (N=16 M=5) 2 / 32 / 128 / 256 jobs 281 /
//     387 / 1,174 / 2,283 us against 392 / 504 / 1,130 / 2,022; 0.43 M (N=6 M=8)
//     363 / 526 / 1,552 / 3,039 against 496 / 625 / 1,403 / 2,542; the path
//     follows (N, M) alone, for a job's bits
constexpr double kSmallHcMacs = 2.5e5, kSmallSlotMacs = 7e5;
constexpr uint32_t kSmallStepRows = 2048;
constexpr double kSmallStepMacs = 2.1e5;  // from there to twice the rows
bool small_eligible(int N, int M, uint32_t D2, double macs);
// whether a step of one system with m Lanczos vectors runs here
inline bool sil_small(const SpaceView& sp, int m) {
    if (m > kBatchMaxLz || sp.pair_y == nullptr || sp.dim > 2 * kSmallStepRows) return false;
    return small_eligible(sp.N, sp.M, sp.dim2,
                          sp.dim <= kSmallStepRows ? kSmallSlotMacs : kSmallStepMacs);
}

// what one system's step works on; every pointer is device memory
struct SmallSys {
    SpaceView sp;     // with pair_w and the scratch pair_y
    double2* C;       // coefficients, in and out
    double2* V;       // m x nc Krylov vectors (V[0] may be C)
    double2* out;     // nc
    double2 *diag, *offd, *y;  // m each
    double2* misc;    // [0] max beta, [1] 1 / beta
    double2* norm2;   // |C|^2 before the renormalisation
    int* iflag;       // [0] breakdown, [1] vectors built, [2] eigensolver status
    double2* rho2;
    int m;            // Krylov vectors, at most kBatchMaxLz
    double2 pdt;      // exp(-i H pdt)
    int shift;        // exponents less their maximum (a step that renormalises)
    int renorm;
};

// parts of a step
constexpr int kSmallHc = 0;       // out = H C
constexpr int kSmallProduct = 1;  // iteration i of the Lanczos recurrence: H v_i, alpha_i
constexpr int kSmallOrth = 2;     // and the reorthogonalisation, beta_i
constexpr int kSmallLanczos = 3;  // the whole recurrence (batched slots)
constexpr int kSmallCombine = 4;  // C <- exp(-i H pdt) C from the recurrence
constexpr int kSmallDens = 5;     // rho2 of C (batched slots)
constexpr int kSmallMonitor = 6;  // eigen residual where due (batched slots)

int small_launch(const SmallSys& s, int part, int i, cudaStream_t st);
// a part of the step of the batched slots of orbital count M in the list
// (count in *nlist, at most nslots)
int small_batch_launch(int M, const BatchSlot* slots, const int* list, const int* nlist,
                       int nslots, int part, int blocks, cudaStream_t st);
int small_prepare(int M);  // launch attributes (before any stream capture)
int small_waves(int M, int (&at)[kClusterSizes]);  // clusters that run at a time

}  // namespace mctdhb
