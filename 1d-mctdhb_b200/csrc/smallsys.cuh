// smallsys.cuh -- one cluster of blocks per small system (smallsys.h; explicit
// instantiations in small_m*.cu): eight blocks for one system, 8, 4, 2 or 1 for
// a slot of the batch (batch.h, cluster_blocks).
//
// The general path spends a small space's time in launches: a Lanczos
// iteration is four of them (nine in the batch), 3 us each, for vectors of a few
// hundred to a few thousand rows.  Here a thread owns rows; vectors, Krylov
// vectors and Y are in global memory, where the thread that wrote a row reads it
// again from its L1, and a step is a fixed chain of passes over 2,048 numbered
// threads with a cluster barrier between two: the contraction
// Y = W A (a thread per row of the (N-2)-space and group of output pairs; W, the
// rank tables and the pieces of sums are in shared memory), the gather-back with the dot product, the dots of the
// reorthogonalisation, its subtraction with the norm, and the scaling.  A
// thread's sums over its rows stay in its registers.  Sums:
// rows of a thread in order, the 32 threads of a warp by a butterfly, the 64
// warps by another; the mapping of rows to threads depends on nothing but the
// row, so a value depends on the system alone.
#pragma once
#include <cooperative_groups.h>

#include <algorithm>

#include "gram_tmpl.cuh"
#include "orbital_dev.cuh"
#include "pairhc_tmpl.cuh"
#include "small_linalg.cuh"
#include "smallsys.h"

namespace mctdhb {

constexpr int kSmThreads = 256, kSmAll = kClusterMax * kSmThreads;  // numbered threads
constexpr int kSmWarps = kSmAll / 32;

template <int M>
struct SmallShared {
    static constexpr int P = M * (M + 1) / 2;
    double2 W[P * P];
    double2 piece[kBatchMaxLz * kSmWarps];
    double z[kBatchMaxLz * kBatchMaxLz];
    double2 y[kBatchMaxLz];
    double2 tab[kPairTabBytes / sizeof(double2)];
};

// blocks and threads of the cluster: constants for the single system, B = 0 any
// number for the batch (one instance alone, as orbstep.cu says)
template <int B>
struct SmallSize {
    static constexpr int blocks = B, threads = B * kSmThreads;
};
template <>
struct SmallSize<0> {
    int blocks, threads;
};

template <int M, int B>
struct SmallRun : SmallSize<B> {
    using SmallSize<B>::blocks;
    using SmallSize<B>::threads;
    static constexpr int P = M * (M + 1) / 2;
    using Sh = SmallShared<M>;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const SmallSys& s;
    Sh* sh;
    SpaceView sp;  // tables in shared memory
    int rank, lane, gtid;

    __device__ SmallRun(const SmallSys& sys, Sh* mem) : s(sys), sh(mem) {
        if constexpr (B == 0) {
            blocks = (int)cl.num_blocks();
            threads = blocks * kSmThreads;
        }
        rank = (int)cl.block_rank();
        lane = threadIdx.x & 31;
        gtid = rank * kSmThreads + threadIdx.x;
        sp = pair_stage_tab(s.sp, sh->tab, threadIdx.x, kSmThreads);
        for (int i = threadIdx.x; i < P * P; i += kSmThreads) sh->W[i] = s.sp.pair_w[i];
        cl.sync();  // own tables ready, and every block of the cluster runs
    }

    // f(n) for the numbers of the 2,048 that this thread stands for, whole warps
    // together: rows go to numbers, so that neither the sums nor who owns a row
    // depend on how many blocks the cluster has
    template <class F>
    __device__ __forceinline__ void each(F&& f) {
        const int per = kClusterMax / blocks;
#pragma unroll 1
        for (int b = rank * per; b < (rank + 1) * per; b++) f(b * kSmThreads + (int)threadIdx.x);
    }
    // the share of the warp with number n in sum k, into every block's table
    __device__ __forceinline__ void put(int k, int n, double2 v) {
        v = warp_sum(v);
        if (lane < blocks) cl.map_shared_rank(sh, lane)->piece[k * kSmWarps + (n >> 5)] = v;
    }
    // sum k, in every lane (after the barrier that follows its put)
    __device__ __forceinline__ double2 total(int k) {
        const double2* p = sh->piece + k * kSmWarps;
        return warp_sum(cadd(p[lane], p[lane + 32]));
    }

    // A_m(Q) of row m of the (N-2)-space, all pairs
    __device__ __forceinline__ void amplitudes(uint32_t row, const double2* C, double2 (&a)[P]) {
        int n[M];
        uint32_t U1[M], U2[M];
        gram_unrank<M, true>(sp.T, sp.N, sp.N - 2, sp.dim2, row, n, U1, U2);
        const uint32_t j0 = sp.dim - sp.dim2 + row;
        double s1[M], s2[M];
#pragma unroll
        for (int x = 0; x < M; x++) {
            s1[x] = sp.sq[n[x] + 1];
            s2[x] = sp.sq[n[x] + 2];
        }
        static_for<P>([&](auto pi) {
            constexpr int p = decltype(pi)::value;
            constexpr int q = kPairs<M>.q[p], l = kPairs<M>.l[p];
            a[p] = cscale(C[j0 - (U1[q] - U1[l]) - U2[l]], q == l ? s1[q] * s2[q] : s1[q] * s1[l]);
        });
    }

    // Y = W A of C: items (row, group of output pairs), the groups as many as
    // keep every thread busy
    __device__ __forceinline__ void contract(const double2* C) {
        const uint32_t D2 = sp.dim2;
        const int ng = max(1, min(P, threads / (int)D2)), per = (P + ng - 1) / ng;
        for (uint32_t e = gtid; e < D2 * ng; e += threads) {
            const uint32_t row = e % D2;
            const int p0 = (int)(e / D2) * per, p1 = min(p0 + per, P);
            if (p0 >= p1) continue;
            double2 a[P];
            amplitudes(row, C, a);
            for (int p = p0; p < p1; p++) {
                const double2* w = sh->W + p * P;
                double2 v0 = make_double2(0.0, 0.0), v1 = make_double2(0.0, 0.0);
                static_for<P>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    if constexpr (q % 2 == 0)
                        v0 = cfma(w[q], a[q], v0);
                    else
                        v1 = cfma(w[q], a[q], v1);
                });
                s.sp.pair_y[(size_t)p * D2 + row] = cadd(v0, v1);
            }
        }
        cl.sync();
    }

    // (H C)_row from Y (pair_gather_back with the tables in shared memory)
    __device__ __forceinline__ double2 back(uint32_t row) {
        const int N = sp.N;
        const uint32_t D2 = sp.dim2;
        int n[M], L[M - 1];
        uint32_t V1[M], V2[M];
        uint32_t S = sp.dim - 1u - row;
        int Lnext = N;
#pragma unroll
        for (int x = M - 2; x >= 0; x--) {
            const uint32_t* Tx = sp.T + x * (N + 1);
            const int lo = cns_level<true>(Tx, x, Lnext, S);
            S -= Tx[lo];
            n[x + 1] = Lnext - lo;
            L[x] = lo;
            Lnext = lo;
        }
        n[0] = Lnext;
        V1[M - 1] = 0u;
        V2[M - 1] = 0u;
#pragma unroll
        for (int x = M - 2; x >= 0; x--) {
            const uint32_t* Tx = sp.T + x * (N + 1);
            const uint32_t t0 = Tx[L[x]];
            V1[x] = V1[x + 1] + (t0 - Tx[L[x] >= 1 ? L[x] - 1 : 0]);
            V2[x] = V2[x + 1] + (t0 - Tx[L[x] >= 2 ? L[x] - 2 : 0]);
        }
        double r0[M], r1[M];  // sqrt(n), sqrt(n - 1)
#pragma unroll
        for (int x = 0; x < M; x++) {
            r0[x] = sp.sq[n[x]];
            r1[x] = sp.sq[n[x] >= 1 ? n[x] - 1 : 0];
        }
        const uint32_t base = D2 - sp.dim + row;
        double2 acc = make_double2(0.0, 0.0);
        static_for<P>([&](auto pi) {
            constexpr int p = decltype(pi)::value;
            constexpr int k = kPairs<M>.q[p], q = kPairs<M>.l[p];
            const bool valid = k == q ? n[k] >= 2 : (n[k] >= 1 && n[q] >= 1);
            const double f = k == q ? r0[k] * r1[k] : r0[k] * r0[q];
            const uint32_t m = valid ? base + (V1[k] - V1[q]) + V2[q] : 0u;
            const double2 v = s.sp.pair_y[(size_t)p * D2 + m];
            acc.x = fma(f, v.x, acc.x);
            acc.y = fma(f, v.y, acc.y);
        });
        return acc;
    }

    __device__ __forceinline__ void hc() {
        contract(s.C);
        for (uint32_t r = gtid; r < sp.dim; r += threads) s.out[r] = back(r);
    }

    // The Lanczos recurrence (multiconfig_lanczos.c:12-90), the operations of
    // lanczos_run, in two passes an iteration that meet in global memory: the
    // whole recurrence is one launch for a slot of the batch, each pass one for a
    // single system.
    // product(i):  v_i = out / beta_{i-1}, out = H v_i - beta_{i-1} v_{i-1},
    //              alpha_i = <v_i, out>
    __device__ __forceinline__ double2 product(int i) {
        const uint32_t nc = sp.dim;
        double2* v = s.V + (size_t)i * nc;
        double beta = 0.0;
        if (i == 0) {
            if (s.V != s.C)
                each([&](int n) {
                    for (uint32_t r = n; r < nc; r += kSmAll) v[r] = s.C[r];
                });
        } else {
            beta = s.offd[i - 1].x;
            const double inv = s.misc[1].x;
            each([&](int n) {
                for (uint32_t r = n; r < nc; r += kSmAll) v[r] = cscale(s.out[r], inv);
            });
            cl.sync();
        }
        contract(i == 0 ? s.C : v);
        each([&](int n) {
            double2 acc = make_double2(0.0, 0.0);
            for (uint32_t r = n; r < nc; r += kSmAll) {
                double2 h = back(r);
                const double2 c = i == 0 ? s.C[r] : v[r];
                if (i > 0) {
                    const double2 pv = s.V[(size_t)(i - 1) * nc + r];
                    h.x -= beta * pv.x;
                    h.y -= beta * pv.y;
                }
                s.out[r] = h;
                acc = cfma_conj(c, h, acc);
            }
            put(0, n, acc);
        });
        cl.sync();
        const double2 alpha = total(0);
        if (gtid == 0) {
            s.diag[i] = alpha;
            if (i == 0) {
                s.misc[0] = make_double2(0.0, 0.0);
                s.offd[s.m - 1] = make_double2(0.0, 0.0);
                s.iflag[0] = 0;
                s.iflag[1] = s.m;
                s.iflag[2] = 0;
            }
        }
        return alpha;
    }

    // orthogonalise(i):  out -= alpha_i v_i, out -= sum_k <v_k, out> v_k,
    // beta_i = |out|; true on a breakdown.  The pieces of alpha are added in
    // every warp before the call (one kernel: a barrier in between).
    __device__ __forceinline__ bool orthogonalise(int i, double2 alpha) {
        const uint32_t nc = sp.dim;
        const double2* v = s.V + (size_t)i * nc;
        each([&](int n) {
            for (uint32_t r = n; r < nc; r += kSmAll) {
                double2 o = s.out[r];
                const double2 av = cmul(alpha, v[r]);
                o.x -= av.x;
                o.y -= av.y;
                s.out[r] = o;
            }
            for (int k = 0; k <= i; k++) {
                double2 acc = make_double2(0.0, 0.0);
                for (uint32_t r = n; r < nc; r += kSmAll)
                    acc = cfma_conj(s.V[(size_t)k * nc + r], s.out[r], acc);
                put(k, n, acc);
            }
        });
        cl.sync();
        for (int k = 0; k <= i; k++) {
            const double2 ok = total(k);
            each([&](int n) {
                for (uint32_t r = n; r < nc; r += kSmAll) {
                    const double2 t = cmul(s.V[(size_t)k * nc + r], ok);
                    double2 o = s.out[r];
                    o.x -= t.x;
                    o.y -= t.y;
                    s.out[r] = o;
                }
            });
        }
        each([&](int n) {
            double nrm = 0.0;
            for (uint32_t r = n; r < nc; r += kSmAll) {
                const double2 o = s.out[r];
                nrm += o.x * o.x + o.y * o.y;
            }
            // the last table: no dot is there (i < m - 1 <= kBatchMaxLz - 1)
            put(kBatchMaxLz - 1, n, make_double2(nrm, 0.0));
        });
        cl.sync();
        const double beta = sqrt(total(kBatchMaxLz - 1).x), mx = fmax(s.misc[0].x, beta);
        const bool broke = beta == 0.0 || beta / mx < 1e-14;
        cl.sync();  // every thread has read the maximum before it changes
        if (gtid == 0) {
            s.offd[i] = make_double2(beta, 0.0);
            s.misc[0].x = mx;
            if (broke) {
                s.iflag[0] = 1;
                s.iflag[1] = i + 1;
            } else {
                s.misc[1] = make_double2(1.0 / beta, 0.0);
            }
        }
        return broke;
    }

    __device__ __forceinline__ void lanczos() {
        for (int i = 0; i < s.m; i++) {
            const double2 alpha = product(i);
            if (i == s.m - 1) break;
            cl.sync();
            if (orthogonalise(i, alpha)) break;
            cl.sync();
        }
    }

    // C = sum_k y_k v_k, y = U exp(-i D pdt) U^T e1 of the tridiagonal matrix
    // by the first warp of every block (lz_small_kernel), renormalised
    // (coefficients_integration.c:127-160)
    __device__ __forceinline__ void combine() {
        const uint32_t nc = sp.dim;
        const int built = s.iflag[1];
        if (threadIdx.x < 32) {
            double d[kBatchMaxLz], e[kBatchMaxLz];
            for (int k = 0; k < built; k++) {
                d[k] = s.diag[k].x;
                e[k] = s.offd[k].x;
            }
            const int rc = tridiag_ql_warp(built, d, e, sh->z);
            if (gtid == 0) s.iflag[2] = rc;
            double shift = 0.0, dk = 0.0;
            for (int k = 0; k < built; k++) {
                if (s.shift && s.pdt.y != 0.0)
                    shift = k == 0 ? d[k] * s.pdt.y : fmax(shift, d[k] * s.pdt.y);
                if (k == lane) dk = d[k];
            }
            __syncwarp();
            double2 aux = make_double2(0.0, 0.0);
            if (lane < built) {
                const double mag = exp(dk * s.pdt.y - shift), u = sh->z[lane];
                double sn, cs;
                sincos(-dk * s.pdt.x, &sn, &cs);
                aux = make_double2(u * mag * cs, u * mag * sn);
            }
            double2 yk = make_double2(0.0, 0.0);
            for (int j = 0; j < built; j++) {
                const double ax = __shfl_sync(0xffffffffu, aux.x, j);
                const double ay = __shfl_sync(0xffffffffu, aux.y, j);
                const double zk = lane < built ? sh->z[lane * built + j] : 0.0;
                yk.x += zk * ax;
                yk.y += zk * ay;
            }
            if (lane < built) {
                sh->y[lane] = yk;
                if (rank == 0) s.y[lane] = yk;
            }
        }
        __syncthreads();
        each([&](int n) {
            double nrm = 0.0;
            for (uint32_t r = n; r < nc; r += kSmAll) {
                double2 c = make_double2(0.0, 0.0);
                for (int j = 0; j < built; j++) c = cfma(s.V[(size_t)j * nc + r], sh->y[j], c);
                s.C[r] = c;
                nrm += c.x * c.x + c.y * c.y;
            }
            if (s.renorm) put(0, n, make_double2(nrm, 0.0));
        });
        if (!s.renorm) return;
        cl.sync();
        const double n2 = total(0).x, rn = 1.0 / sqrt(n2);
        if (gtid == 0) *s.norm2 = make_double2(n2, 0.0);
        each([&](int n) {
            for (uint32_t r = n; r < nc; r += kSmAll) {
                s.C[r].x *= rn;
                s.C[r].y *= rn;
            }
        });
    }

    // rho2 as the Gram matrix of the A planes (in the scratch of Y), a warp an
    // entry of the upper triangle
    __device__ __forceinline__ void densities() {
        const uint32_t D2 = sp.dim2;
        double2* A = s.sp.pair_y;
        for (uint32_t row = gtid; row < D2; row += threads) {
            double2 a[P];
            amplitudes(row, s.C, a);
            static_for<P>([&](auto pi) {
                constexpr int p = decltype(pi)::value;
                A[(size_t)p * D2 + row] = a[p];
            });
        }
        cl.sync();
        constexpr int M2 = M * M, M3 = M2 * M;
        for (int e = gtid >> 5; e < P * (P + 1) / 2; e += threads / 32) {
            int pa = 0, pb = e;
            while (pb >= P - pa) {
                pb -= P - pa;
                pa++;
            }
            pb += pa;
            const double2 *x = A + (size_t)pa * D2, *y = A + (size_t)pb * D2;
            double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
            for (uint32_t r = lane; r < D2; r += 32) acc = cfma_conj(x[r], y[r], acc);
            acc = warp_sum(acc);
            if (pa == pb) acc.y = 0.0;
            const double2 cc = make_double2(acc.x, -acc.y);
            // lanes 0..7: the orders of the two pairs and the conjugates
            int k0 = 0, s0 = pa, q0 = 0, l0 = pb;
            while (s0 >= M - k0) s0 -= M - k0++;
            while (l0 >= M - q0) l0 -= M - q0++;
            s0 += k0;
            l0 += q0;
            if (lane < 8) {
                const int k = lane & 1 ? s0 : k0, t = lane & 1 ? k0 : s0;
                const int q = lane & 2 ? l0 : q0, l = lane & 2 ? q0 : l0;
                if (lane & 4)
                    s.rho2[q + l * M + k * M2 + t * M3] = cc;
                else
                    s.rho2[k + t * M + q * M2 + l * M3] = acc;
            }
        }
        // rho1 follows from rho2 in bt_tail_kernel
    }
};

// one system: a part of its step (smallsys.h), iteration i of the Lanczos
// recurrence
template <int M>
__global__ void __launch_bounds__(kSmThreads)
    small_kernel(SmallSys s, int part, int i) {
    extern __shared__ __align__(16) unsigned char small_mem[];
    if ((part == kSmallProduct || part == kSmallOrth) && i > 0 && s.iflag[0]) return;  // breakdown
    SmallRun<M, kClusterMax> r(s, (SmallShared<M>*)small_mem);
    switch (part) {
        case kSmallHc: r.hc(); break;
        case kSmallProduct: r.product(i); break;
        case kSmallOrth: r.orthogonalise(i, s.diag[i]); break;
        case kSmallCombine: r.combine(); break;
    }
}

// a part of the step of the slots of orbital count M; kSmallMonitor: the eigen
// residual max_i |E C_i - (H C)_i| / N where it is due, and the eigen-residual
// half of the stop rule (bt_monitor_kernel)
template <int M>
__global__ void __launch_bounds__(kSmThreads)
    small_batch_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                       const int* __restrict__ nlist, int part) {
    const int at = blockIdx.x / (int)cooperative_groups::this_cluster().num_blocks();
    if (at >= *nlist) return;  // the same in every block of the cluster
    const BatchSlot& S = slots[list[at]];
    if (part == kSmallMonitor ? !S.flags[BF_MON] : S.flags[BF_STATE] != SLOT_RUNNING) return;
    extern __shared__ __align__(16) unsigned char small_mem[];
    SmallSys s;
    s.sp = S.sp;
    s.C = S.V;
    s.V = S.V;
    s.out = S.out;
    s.diag = S.scal + BS_DIAG;
    s.offd = S.scal + BS_OFFD;
    s.y = S.scal + BS_Y;
    s.misc = S.scal + BS_MISC;
    s.norm2 = S.scal + BS_MISC + 2;
    s.iflag = S.flags;
    s.rho2 = S.rho2;
    s.m = S.lz;
    s.pdt = S.pdt;
    s.shift = 1;
    s.renorm = S.imag;
    static_assert(BF_BREAK == 0 && BF_ITERS == 1 && BF_QL == 2, "iflag is the head of the flags");
    SmallRun<M, 0> r(s, (SmallShared<M>*)small_mem);
    if (part == kSmallLanczos) {
        r.lanczos();
        return;
    }
    if (part == kSmallCombine) {
        r.combine();
        return;
    }
    if (part == kSmallDens) {
        r.densities();
        return;
    }
    r.contract(s.C);
    const double e = S.scal[BS_MISC + 3].x;
    double worst = 0.0;
    for (uint32_t i = r.gtid; i < S.nc; i += r.threads) {
        const double2 c = s.C[i], h = r.back(i);
        worst = fmax(worst, hypot(e * c.x - h.x, e * c.y - h.y));
    }
    worst = warp_max_f64(worst);
    const int warps = r.threads / 32;
    if (r.lane < r.blocks)
        r.cl.map_shared_rank(r.sh, r.lane)->piece[r.gtid >> 5] = make_double2(worst, 0.0);
    r.cl.sync();
    if (r.rank != 0 || threadIdx.x >= 32) return;
    worst = 0.0;
    for (int w = r.lane; w < warps; w += 32) worst = fmax(worst, r.sh->piece[w].x);
    worst = warp_max_f64(worst);
    if (r.lane != 0) return;
    const double res = worst / S.N;
    S.scal[BS_MISC + 6] = make_double2(res, 0.0);
    if (res < S.eig_tol) {
        S.flags[BF_STATE] = SLOT_DONE;
        S.flags[BF_CONV] = 1;
    }
    S.flags[BF_MON] = 0;
}

template <int M>
int small_prepare_tmpl() {
    static std::atomic<uint64_t> done{0};
    return set_attributes_once(done, []() -> int {
        const auto kind = cudaFuncAttributeMaxDynamicSharedMemorySize;
        const int bytes = (int)sizeof(SmallShared<M>);
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(small_kernel<M>, kind, bytes));
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(small_batch_kernel<M>, kind, bytes));
        return 0;
    });
}

template <int M>
int small_waves_tmpl(int (&at)[kClusterSizes]) {
    return cluster_waves(small_batch_kernel<M>, kSmThreads, sizeof(SmallShared<M>), at);
}

template <int M>
int small_launch_tmpl(const SmallSys& s, int part, int i, cudaStream_t st) {
    ClusterLaunch c(kClusterMax, kSmThreads, sizeof(SmallShared<M>), kClusterMax, st);
    MCTDHB_CUDA_TRY(cudaLaunchKernelEx(&c.cfg, small_kernel<M>, s, part, i));
    return 0;
}

template <int M>
int small_batch_tmpl(const BatchSlot* slots, const int* list, const int* nlist, int nslots,
                     int part, int blocks, cudaStream_t st) {
    ClusterLaunch c(nslots * blocks, kSmThreads, sizeof(SmallShared<M>), blocks, st);
    MCTDHB_CUDA_TRY(cudaLaunchKernelEx(&c.cfg, small_batch_kernel<M>, slots, list, nlist, part));
    return 0;
}

}  // namespace mctdhb
