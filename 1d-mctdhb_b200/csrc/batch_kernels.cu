// batch_kernels.cu -- the slot-level and vector kernels of the batched engine
// (batch.h).  Per slot, one step is the full step of the single-system
// solver (driver.c:159-201):
//   orb_step_launch     (orbstep.cu) one cluster of blocks per slot:
//                       Runge-Kutta step of the orbital equation with the
//                       slot's rho1^{-1} and rho2, Gram-Schmidt in imaginary
//                       time, h_kl and g_ksql of the new orbitals, the pair
//                       matrix of H.C, Lanczos set-up
//   Lanczos             the pair-space H.C (per M, batch_tmpl.cuh) and the
//                       vector kernels below, multiconfig_lanczos.c:12-90
//                       operation for operation
//   SIL                 tridiagonal eigenproblem, C = V U exp(-i D dt) U^T e1,
//                       renormalisation in imaginary time
//                       (coefficients_integration.c:59-160)
//   densities           Gram-matrix rho2 (per M, batch_tmpl.cuh)
//   bt_tail_kernel      rho1 from rho2, its regularisation and inverse (synchronize.c:42-57),
//                       energy (integrator_monitor.c:56-88), step count and
//                       the imaginary-time stop rule (driver.c:47-67)
// Vector kernels walk tiles of kBatchVecRows rows; every per-slot sum is
// formed from per-tile partials in tile order.
#include <cuda_runtime.h>

#include "batch.h"
#include "batch_kernels.h"
#include "common.cuh"
#include "gram_tmpl.cuh"
#include "moves.cuh"
#include "orbital_dev.cuh"
#include "small_linalg.cuh"

namespace mctdhb {

namespace {

__device__ __forceinline__ bool slot_running(const BatchSlot& S) {
    return S.flags[BF_STATE] == SLOT_RUNNING;
}

}  // namespace

// ---------------------------------------------------------------------------
// vector kernels over tiles of kBatchVecRows rows
// ---------------------------------------------------------------------------
#define BT_TILE_LOOP                                                              \
    const int nt = *ntiles;                                                       \
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {                            \
        const BatchTile tl = tiles[t];                                            \
        const BatchSlot& S = slots[tl.slot];                                      \
        const uint32_t nc = S.nc;                                                 \
        const uint32_t r0 = tl.idx * (uint32_t)kBatchVecRows;
#define BT_ROWS(r)                                                                \
    for (uint32_t r = r0 + threadIdx.x; r < nc && r < r0 + kBatchVecRows; r += kBatchVecThreads)

// part[tile] = <V[i], out>   (alpha_i, multiconfig_lanczos.c:40-41, :83)
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_dot_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                  const int* __restrict__ ntiles, int i) {
    BT_TILE_LOOP
    if (!slot_running(S) || S.flags[BF_BREAK]) continue;
    const double2* v = S.V + (size_t)i * nc;
    double2 acc = make_double2(0.0, 0.0);
    BT_ROWS(r) acc = cfma_conj(v[r], S.out[r], acc);
    const double2 s = block_sum(acc);
    if (threadIdx.x == 0) S.part[tl.idx] = s;
    }
}

// out -= alpha_i V[i]; part[k * vtiles + tile] = <V[k], out>, k <= i
// (multiconfig_lanczos.c:46, :57-62)
// (the iteration is a template parameter: only the i + 1 accumulators in
// use take registers, which keeps enough warps resident)
template <int I>
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_subdots_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                      const int* __restrict__ ntiles) {
    BT_TILE_LOOP
    if (!slot_running(S) || S.flags[BF_BREAK]) continue;
    const double2 alpha = S.scal[BS_DIAG + I];
    double2 acc[I + 1];
#pragma unroll
    for (int k = 0; k <= I; k++) acc[k] = make_double2(0.0, 0.0);
    BT_ROWS(r) {
        // every Krylov value is loaded before the store to out (which may
        // alias V as far as the compiler knows), V[I] once
        double2 v[I + 1];
#pragma unroll
        for (int k = 0; k <= I; k++) v[k] = S.V[(size_t)k * nc + r];
        double2 o = S.out[r];
        const double2 av = cmul(alpha, v[I]);
        o.x -= av.x;
        o.y -= av.y;
        S.out[r] = o;
#pragma unroll
        for (int k = 0; k <= I; k++) acc[k] = cfma_conj(v[k], o, acc[k]);
    }
#pragma unroll
    for (int k = 0; k <= I; k++) {
        const double2 s = block_sum(acc[k]);
        if (threadIdx.x == 0) S.part[(size_t)k * S.vtiles + tl.idx] = s;
    }
    }
}

template <int I>
static void subdots_launch(int i, int grid, cudaStream_t st, const BatchSlot* slots,
                           const BatchTile* tiles, const int* ntiles) {
    if (i == I)
        bt_subdots_kernel<I><<<grid, kBatchVecThreads, 0, st>>>(slots, tiles, ntiles);
    else if constexpr (I > 0)
        subdots_launch<I - 1>(i, grid, st, slots, tiles, ntiles);
}

// out -= sum_{k<=i} o_k V[k]; part[tile] = |out|^2 (multiconfig_lanczos.c:57-64)
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_orth_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                   const int* __restrict__ ntiles, int i) {
    BT_TILE_LOOP
    if (!slot_running(S) || S.flags[BF_BREAK]) continue;
    double acc = 0.0;
    BT_ROWS(r) {
        double2 o = S.out[r];
        for (int k = 0; k <= i; k++) {
            const double2 tv = cmul(S.V[(size_t)k * nc + r], S.scal[BS_ORTHO + k]);
            o.x -= tv.x;
            o.y -= tv.y;
        }
        S.out[r] = o;
        acc += o.x * o.x + o.y * o.y;
    }
    const double2 s = block_sum(make_double2(acc, 0.0));
    if (threadIdx.x == 0) S.part[tl.idx] = s;
    }
}

// V[i+1] = out / beta_i (multiconfig_lanczos.c:74)
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_scale_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                    const int* __restrict__ ntiles, int i) {
    BT_TILE_LOOP
    if (!slot_running(S) || S.flags[BF_BREAK]) continue;
    const double inv = S.scal[BS_MISC + 1].x;
    BT_ROWS(r) {
        const double2 o = S.out[r];
        S.V[(size_t)(i + 1) * nc + r] = make_double2(o.x * inv, o.y * inv);
    }
    }
}

// C = sum_j y_j V[j] over the vectors built (coefficients_integration.c:127-154);
// C is V[0], overwritten row by row after its own rows are read
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_combine_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                      const int* __restrict__ ntiles) {
    BT_TILE_LOOP
    if (!slot_running(S)) continue;
    const int it = S.flags[BF_ITERS];
    BT_ROWS(r) {
        double2 s = make_double2(0.0, 0.0);
        for (int j = 0; j < it; j++) s = cfma(S.V[(size_t)j * nc + r], S.scal[BS_Y + j], s);
        S.V[r] = s;
    }
    }
}

// part[tile] = |C|^2
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_norm2_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                    const int* __restrict__ ntiles) {
    BT_TILE_LOOP
    if (!slot_running(S) || !S.imag) continue;
    double acc = 0.0;
    BT_ROWS(r) acc += S.V[r].x * S.V[r].x + S.V[r].y * S.V[r].y;
    const double2 s = block_sum(make_double2(acc, 0.0));
    if (threadIdx.x == 0) S.part[tl.idx] = s;
    }
}

// C /= |C| (imaginary time, coefficients_integration.c:156-159)
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_renorm_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                     const int* __restrict__ ntiles) {
    BT_TILE_LOOP
    if (!slot_running(S) || !S.imag) continue;
    const double rn = 1.0 / sqrt(S.scal[BS_MISC + 2].x);
    BT_ROWS(r) {
        S.V[r].x *= rn;
        S.V[r].y *= rn;
    }
    }
}

#undef BT_TILE_LOOP
#undef BT_ROWS

// ---------------------------------------------------------------------------
// slot kernels: one block per slot of the list
// ---------------------------------------------------------------------------
#define BT_SLOT                                                                   \
    if ((int)blockIdx.x >= *nlist) return;                                        \
    const BatchSlot& S = slots[list[blockIdx.x]];                                 \
    if (!slot_running(S)) return;

// fixed-order sum of part[k * vtiles + t] over t, for k < nvals, into
// scal[dst + k]: threads take strided partial sums, then a tree (256 threads)
__device__ double2 bt_sum_parts(const double2* part, int ntile) {
    __shared__ double2 sh[kBatchVecThreads];
    double2 s = make_double2(0.0, 0.0);
    for (int b = threadIdx.x; b < ntile; b += blockDim.x) {
        s.x += part[b].x;
        s.y += part[b].y;
    }
    __syncthreads();
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sh[threadIdx.x].x += sh[threadIdx.x + o].x;
            sh[threadIdx.x].y += sh[threadIdx.x + o].y;
        }
        __syncthreads();
    }
    return sh[0];
}

// scal[dst + k] = sum_t part[k * vtiles + t], k < nvals.  skip_break: the
// value belongs to a Lanczos iteration a breakdown has cancelled.
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_reduce_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                     const int* __restrict__ nlist, int nvals, int dst, int skip_break) {
    BT_SLOT
    if (skip_break && S.flags[BF_BREAK]) return;
    for (int k = 0; k < nvals; k++) {
        const double2 s = bt_sum_parts(S.part + (size_t)k * S.vtiles, S.vtiles);
        if (threadIdx.x == 0) S.scal[dst + k] = s;
        __syncthreads();
    }
}

// beta_i = |out|; breakdown when beta_i / max beta < 1e-14 (or beta_i = 0);
// 1/beta_i for the scaling (multiconfig_lanczos.c:64-74)
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_norm_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                   const int* __restrict__ nlist, int i) {
    BT_SLOT
    if (S.flags[BF_BREAK]) return;
    const double2 s = bt_sum_parts(S.part, S.vtiles);
    if (threadIdx.x != 0) return;
    const double beta = sqrt(s.x);
    S.scal[BS_OFFD + i] = make_double2(beta, 0.0);
    double mx = S.scal[BS_MISC + 0].x;
    if (mx < beta) mx = beta;
    S.scal[BS_MISC + 0].x = mx;
    if (beta == 0.0 || beta / mx < 1e-14) {
        S.flags[BF_BREAK] = 1;
        S.flags[BF_ITERS] = i + 1;
        return;
    }
    S.scal[BS_MISC + 1] = make_double2(1.0 / beta, 0.0);
}

// y = U exp(-i D pdt) U^T e1 of the tridiagonal (alpha, beta) (implicit QL),
// one warp per slot as lz_small_kernel
__global__ void __launch_bounds__(32)
    bt_small_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                    const int* __restrict__ nlist) {
    BT_SLOT
    __shared__ double z[kBatchMaxLz * kBatchMaxLz];
    __shared__ double2 aux[kBatchMaxLz];
    const int lane = threadIdx.x, n = S.flags[BF_ITERS];
    double d[kBatchMaxLz], e[kBatchMaxLz];
    for (int k = 0; k < n; k++) {
        d[k] = S.scal[BS_DIAG + k].x;
        e[k] = S.scal[BS_OFFD + k].x;
    }
    const int rc = tridiag_ql_warp(n, d, e, z);
    if (lane == 0) S.flags[BF_QL] = rc;
    const double2 pdt = S.pdt;
    // imaginary time: exponents shifted by their maximum (a constant factor
    // the renormalisation at the end of the step removes), so exp cannot
    // overflow at |E| dt > 709; real time: no shift
    double shift = 0.0;
    if (pdt.y != 0.0)
        for (int k = 0; k < n; k++) shift = k == 0 ? d[k] * pdt.y : fmax(shift, d[k] * pdt.y);
    __syncwarp();
    if (lane < n) {
        const double re = d[lane] * pdt.y, im = -d[lane] * pdt.x;
        const double mag = exp(re - shift);
        double sn, cs;
        sincos(im, &sn, &cs);
        const double u = z[lane];
        aux[lane] = make_double2(u * mag * cs, u * mag * sn);
    }
    __syncwarp();
    if (lane < n) {
        double2 s = make_double2(0.0, 0.0);
        for (int j = 0; j < n; j++) {
            s.x += z[lane * n + j] * aux[j].x;
            s.y += z[lane * n + j] * aux[j].y;
        }
        S.scal[BS_Y + lane] = s;
    }
}

// rho1 from rho2, its regularisation and inverse, energy, step count, stop
// rules.
// prologue: set-up of a new slot (no step counted; the energy seeds the
// imaginary-time stop rule as driver.c:229 does).
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_tail_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                   const int* __restrict__ nlist, int prologue, int* __restrict__ mon) {
    BT_SLOT
    const int M = S.M;
    rho1_from_rho2(S.N, M, S.rho2, S.rho1, threadIdx.x, blockDim.x);
    __syncthreads();
    if (threadIdx.x < 32) {
        // the first warp, on copies in shared memory
        __shared__ double2 r1[kBatchMaxOrb * kBatchMaxOrb], ri[kBatchMaxOrb * kBatchMaxOrb];
        __shared__ double2 w[3 * kBatchMaxOrb * kBatchMaxOrb];
        const int M2 = M * M;
        for (int i = threadIdx.x; i < M2; i += 32) r1[i] = S.rho1[i];
        __syncwarp();
        const int info = sync_rho1_warp(M, r1, ri, S.reg_fac, w);
        if (threadIdx.x == 0) S.flags[BF_INFO] = info;
        for (int i = threadIdx.x; i < M2; i += 32) {
            S.rho1[i] = r1[i];
            S.rinv[i] = ri[i];
        }
    }
    __syncthreads();
    const double2 E = energy_block(M, S.rho1, S.rho2, S.hob, S.hint);
    if (threadIdx.x != 0) return;
    S.scal[BS_MISC + 3] = E;
    if (prologue) {
        S.scal[BS_MISC + 4] = make_double2(E.x / S.N, 0.0);
        S.scal[BS_MISC + 6] = make_double2(-1.0, 0.0);  // no eigen residual yet
        return;
    }
    const int steps = S.flags[BF_STEPS] + 1;
    S.flags[BF_STEPS] = steps;
    int state = SLOT_RUNNING;
    const bool check = S.check_every > 0 && steps % S.check_every == 0;
    if (S.imag && check) {
        // driver.c:47-67: |E/N - prev| < tol * prev, and with eig_tol set the
        // eigen residual below it: that half is decided by bt_monitor_kernel
        // after the monitor's H.C of this step
        const double curr = E.x / S.N, prev = S.scal[BS_MISC + 4].x;
        if (fabs(curr - prev) < S.etol * prev) {
            if (S.eig_tol > 0.0) {
                S.flags[BF_MON] = 1;
                mon[S.M] = 1;
            } else {
                state = SLOT_DONE;
                S.flags[BF_CONV] = 1;
            }
        }
        S.scal[BS_MISC + 4] = make_double2(curr, 0.0);
    }
    if (!S.imag && check) {
        // driver.c:69-96: switch the robust projector on above the
        // threshold; above the critical residual the reference exits, the
        // engine stops this job
        const double o = S.scal[BS_MISC + 5].x;
        if (o > S.ortho_tol && !S.flags[BF_ROBUST]) S.flags[BF_ROBUST] = 1;
        if (o > kOverlapAbort) state = SLOT_ABORTED;
    }
    if ((uint32_t)steps >= S.max_steps && state == SLOT_RUNNING) state = SLOT_DONE;
    S.flags[BF_STATE] = state;
}

// max_i |E C_i - (H C)_i| over a vector tile of the slots whose eigen
// residual is due (integrator_monitor.c:9-28), into part[tile].x
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_resid_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                    const int* __restrict__ ntiles) {
    __shared__ double sh[kBatchVecThreads];
    const int nt = *ntiles;
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const BatchTile tl = tiles[t];
        const BatchSlot& S = slots[tl.slot];
        if (!S.flags[BF_MON]) continue;  // block-uniform
        const uint32_t nc = S.nc;
        const uint32_t r0 = tl.idx * (uint32_t)kBatchVecRows;
        const double e = S.scal[BS_MISC + 3].x;
        double m = 0.0;
        for (uint32_t r = r0 + threadIdx.x; r < nc && r < r0 + kBatchVecRows;
             r += kBatchVecThreads) {
            const double2 c = S.V[r], h = S.out[r];
            m = fmax(m, hypot(e * c.x - h.x, e * c.y - h.y));
        }
        sh[threadIdx.x] = m;
        __syncthreads();
        for (int o = kBatchVecThreads / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + o]);
            __syncthreads();
        }
        if (threadIdx.x == 0) S.part[tl.idx] = make_double2(sh[0], 0.0);
        __syncthreads();
    }
}

// the eigen-residual half of the imaginary-time stop rule (driver.c:47-67):
// res = max over the tiles / N; the slot stops (converged) when res is
// below eig_tol
__global__ void __launch_bounds__(kBatchVecThreads)
    bt_monitor_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                      const int* __restrict__ nlist) {
    __shared__ double sh[kBatchVecThreads];
    if ((int)blockIdx.x >= *nlist) return;
    const BatchSlot& S = slots[list[blockIdx.x]];
    if (!S.flags[BF_MON]) return;
    double m = 0.0;
    for (int t = threadIdx.x; t < S.vtiles; t += blockDim.x) m = fmax(m, S.part[t].x);
    sh[threadIdx.x] = m;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    const double res = sh[0] / S.N;
    S.scal[BS_MISC + 6] = make_double2(res, 0.0);
    if (res < S.eig_tol) {
        S.flags[BF_STATE] = SLOT_DONE;
        S.flags[BF_CONV] = 1;
    }
    S.flags[BF_MON] = 0;
}

#undef BT_SLOT

__global__ void __launch_bounds__(kBatchVecThreads)
    bt_fetch_kernel(BatchFetch f, double2* __restrict__ out) {
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    if (t0 == 0) {
        out[0] = make_double2(f.scal[BS_MISC + 3].x, 0.0);
        out[1] = make_double2((double)f.flags[BF_STEPS], (double)f.flags[BF_CONV]);
    }
    double2* o = out + kFetchHead;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        for (uint32_t i = t0; i < f.n[a]; i += nt) o[i] = f.src[a][i];
        o += f.n[a];
    }
}

void bt_subdots(int i, int grid, cudaStream_t st, const BatchSlot* slots, const BatchTile* tiles,
                const int* ntiles) {
    subdots_launch<kBatchMaxLz - 2>(i, grid, st, slots, tiles, ntiles);
}

}  // namespace mctdhb
