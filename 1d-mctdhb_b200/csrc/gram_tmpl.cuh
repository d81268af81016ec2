// gram_tmpl.cuh -- density matrices as a Gram matrix of annihilated states,
// for 2 <= M <= 8 orbitals (explicit instantiations in dens_m*.cu).
//
// rho2[k,s,q,l] = <a+_k a+_s a_q a_l> (density_matrices.c:9-443) is the inner
// product of states with two bosons removed.  Inserting the identity of the
// (N-2)-boson space,
//     rho2[k,s,q,l] = sum_m conj(A_m(k,s)) A_m(q,l),  A_m(q,l) = <m|a_q a_l|C>,
// with m over the D(N-2, M) configurations; rho1[k][l] =
// sum_s rho2[k,s,s,l] / (N-1) (rho1_from_rho2).  With one boson rho2 vanishes
// and rho1[k][l] = conj(C_k) C_l.  Each A value is one scaled coefficient,
// A_m(q,l) = sqrt((m_q+1)(m_l+1+[q=l])) C[m+e_q+e_l]: at N=30, M=8 that is
// 6.7 M rows x 36 pairs = 242 M gathers (against the ~3 G coupling gathers of a
// per-row pass) and a 36 x 36 Hermitian Gram matrix.
//
// Ranking.  With the cumulative occupations L_x of m and the rank-weight
// table T_x(L) = C(L+x, x+1) (common.cuh), the rank of m + e_q + e_l in the
// N-boson space is
//     j = (D_N - D_{N-2}) + rank(m) - (U1[q] - U1[l]) - U2[l],
//     U_d[x] = sum_{y=x}^{M-2} (T_y(L_y + d) - T_y(L_y)),
// two subtractions per pair once U1, U2 are formed per row.
//
// The Gram matrix on the FP64 tensor cores.  With the real columns X = [Re A,
// Im A] (2P of them) the real Gram matrix S = X^T X holds everything:
//     Re G[a][b] = S(Re a, Re b) + S(Im a, Im b),
//     Im G[a][b] = S(Re a, Im b) - S(Im a, Re b).
// S is symmetric, so only the upper triangle of its 8 x 8 tiles is formed: 45
// tiles at P = 36 (9 tiles a side, none of them padding) against 55 tile
// products of a complex Hermitian form.  In mma.sync m8n8k4 the A and the B
// fragment of a column tile are the same value per lane (column lane / 4, row
// lane % 4), so one 16-byte load gives the fragments of a real and an
// imaginary tile for both sides: 5 loads feed 45 products of 16 cycles.
// FP64 FMA register tiles, which read 8 operands for 16 complex FMAs, ran at
// 0.41 of the FP64 peak by the algorithmic count.
// What bounds it now: at N=60 M=6 the products alone take 611 us (512 us at the
// FP64 MMA peak) and the gathers alone, L2-bound, 365 us; together 770 us (903
// with the FMA tiles).  Eight producer and four consumer warps a block around a
// ring of 32-row chunks gave 786 us, with one block an SM 765 us: the gathers
// need 16 warps an SM, which leaves the products too few.
//
// Work split.  A block takes tiles of 128 or 256 rows: every thread unranks its
// row and gathers its share of the row's A values into shared memory (gram.h
// gives the layout), then the warps take the rows four at a time; from six
// orbitals two warps share them (four at eight), each with its part of the
// products, so that the accumulators of two blocks fit an SM.  At the end the warps are added in order
// and the block writes one partial; gram_finalize_kernel adds the partials in
// block order.  The grid is a function of (N, M) only, so the result is
// deterministic and the same in any launch context.
#pragma once
#include "common.cuh"
#include "kernels.h"
#include "gram.h"
#include "movelist.cuh"

namespace mctdhb {

// pair p <-> (q, l), q <= l, in row-major order of the upper triangle
template <int M>
struct PairList {
    int q[M * (M + 1) / 2], l[M * (M + 1) / 2];
    constexpr PairList() : q{}, l{} {
        int p = 0;
        for (int a = 0; a < M; a++)
            for (int b = a; b < M; b++) {
                q[p] = a;
                l[p] = b;
                p++;
            }
    }
};
template <int M>
inline constexpr PairList<M> kPairs{};

// Unrank `row` of the space of Np bosons (dimension Dp) with the rank table
// of a space of N >= Np bosons (row stride N + 1): occupations n[] and the
// suffix sums U1, U2 of the rank offsets of adding one / two bosons.
// GEN: generic table loads (the table may be staged in shared memory).
template <int M, bool GEN = false>
__device__ __forceinline__ void gram_unrank(const uint32_t* __restrict__ T, int N, int Np,
                                            uint32_t Dp, uint32_t row, int (&n)[M],
                                            uint32_t (&U1)[M], uint32_t (&U2)[M]) {
    uint32_t S = Dp - 1u - row;
    int Lnext = Np;
    int L[M > 1 ? M - 1 : 1];
#pragma unroll
    for (int x = M - 2; x >= 0; x--) {
        const uint32_t* Tx = T + x * (N + 1);
        const int lo = cns_level<GEN>(Tx, x, Lnext, S);
        S -= tab_ld<GEN>(Tx + lo);
        n[x + 1] = Lnext - lo;
        L[x] = lo;
        Lnext = lo;
    }
    n[0] = Lnext;
    U1[M - 1] = 0u;
    U2[M - 1] = 0u;
#pragma unroll
    for (int x = M - 2; x >= 0; x--) {
        const uint32_t* Tx = T + x * (N + 1);
        const uint32_t t0 = tab_ld<GEN>(Tx + L[x]);
        U1[x] = U1[x + 1] + (tab_ld<GEN>(Tx + L[x] + 1) - t0);
        U2[x] = U2[x + 1] + (tab_ld<GEN>(Tx + L[x] + 2) - t0);
    }
}

// ---------------------------------------------------------------------------
// building blocks (shared with the batched engine, batch_tmpl.cuh)
// ---------------------------------------------------------------------------
template <int M>
struct GramShape {
    static constexpr int P = gram_p(M);
    static constexpr int ROWS = gram_rows(M), PS = gram_row_words(M), ENT = gram_entries(M);
    static constexpr int PARTS = kGramThreads / ROWS;  // threads per row in the gather
    // column tiles: a real and an imaginary one per 8 pairs; of the REM pairs
    // left, up to four share one tile (real parts, then imaginary ones)
    static constexpr int FULL = P / 8, REM = P % 8;
    static constexpr bool MIXED = REM > 0 && REM <= 4;
    static constexpr int TILES = 2 * FULL + (REM == 0 ? 0 : MIXED ? 1 : 2);
    static constexpr int PRODS = TILES * (TILES + 1) / 2;
    static constexpr int SPLIT = M == 8 ? 4 : M >= 6 ? 2 : 1;  // warps sharing the rows
    static constexpr int GROUPS = kGramThreads / 32 / SPLIT;      // row groups
    static constexpr int NACC = (PRODS + SPLIT - 1) / SPLIT;
    static_assert(PRODS * 64 * 8 <= ROWS * PS * 16, "the reduction reuses the A tile");
    // column of S of the real (c = 0) or imaginary (c = 1) part of pair p
    __host__ __device__ static constexpr int col(int p, int c) {
        return p < 8 * FULL ? (2 * (p / 8) + c) * 8 + p % 8
               : MIXED      ? 2 * FULL * 8 + (p - 8 * FULL) + 4 * c
                            : (2 * FULL + c) * 8 + (p - 8 * FULL);
    }
    // index of the product of the column tiles i <= j
    __host__ __device__ static constexpr int prod(int i, int j) {
        return i * TILES - i * (i - 1) / 2 + (j - i);
    }
    // place of S[x][y] among the products (64 entries each)
    __host__ __device__ static constexpr int at(int x, int y) {
        return x / 8 <= y / 8 ? prod(x / 8, y / 8) * 64 + x % 8 * 8 + y % 8
                              : prod(y / 8, x / 8) * 64 + y % 8 * 8 + x % 8;
    }
};

// Gather tile `tr` (ROWS rows of the (N-2)-boson space, Dp rows in all):
// thread t fills the values p = part, part + PARTS, ... of row t % ROWS.
template <int M>
__device__ __forceinline__ void gram_gather(const SpaceView& sp, uint32_t Dp,
                                            const double2* __restrict__ C, uint32_t tr,
                                            double2* As, int t) {
    using S = GramShape<M>;
    constexpr int P = S::P, PS = S::PS, ROWS = S::ROWS, PARTS = S::PARTS;
    const int N = sp.N;
    const int r = t % ROWS, part = t / ROWS;  // part is warp-uniform
    const uint32_t row = tr * ROWS + r;
    const bool live = row < Dp;
    const uint32_t rr = live ? row : Dp - 1u;
    int n[M];
    uint32_t U1[M], U2[M];
    gram_unrank<M>(sp.T, N, N - 2, Dp, rr, n, U1, U2);
    const uint32_t j0 = sp.dim - Dp + rr;
    // sqrt(n_x + 1), sqrt(n_x + 2) once per orbital; rows past the end are
    // zero through them
    double s1[M], s2[M];
#pragma unroll
    for (int x = 0; x < M; x++) {
        s1[x] = __ldg(sp.sq + n[x] + 1);
        s2[x] = __ldg(sp.sq + n[x] + 2);
    }
    double2* out = As + r * PS;
    const int sw = gram_swz(r);
    // coefficient gathers through L2 only (ld.global.cg), leaving L1 to the
    // rank and square-root tables
    static_for<P>([&](auto pi) {
        constexpr int p = decltype(pi)::value;
        constexpr int q = kPairs<M>.q[p], l = kPairs<M>.l[p];
        if (p % PARTS == part) {
            const uint32_t j = j0 - (U1[q] - U1[l]) - U2[l];
            const double f = q == l ? s1[q] * s2[q] : s1[q] * s1[l];
            const double2 v = cscale(__ldcg(C + j), f);
            out[p ^ sw] = live ? v : make_double2(0.0, 0.0);
        }
    });
}

// FP64 mma.sync m8n8k4: lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4)], D[l/4][2(l%4) + 1]
__device__ __forceinline__ void gram_mma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// acc += the products h, h + SPLIT, ... of S over the rows 4 grp, 4 (grp +
// GROUPS), ... of the tile
template <int M, int H>
__device__ __forceinline__ void gram_products(const double2* As, int grp, int lane,
                                              double (&acc)[GramShape<M>::NACC][2]) {
    using S = GramShape<M>;
    const int g = lane >> 2, t = lane & 3;
    for (int r0 = grp * 4; r0 < S::ROWS; r0 += S::GROUPS * 4) {
        const int r = r0 + t, sw = gram_swz(r);
        const double2* row = As + r * S::PS;
        double x[S::TILES];
#pragma unroll
        for (int a = 0; a < S::FULL; a++) {
            const double2 v = row[(8 * a + g) ^ sw];
            x[2 * a] = v.x;
            x[2 * a + 1] = v.y;
        }
        if constexpr (S::MIXED) {
            const double2 v = row[(8 * S::FULL + (g & 3)) ^ sw];
            x[2 * S::FULL] = (g & 3) >= S::REM ? 0.0 : g < 4 ? v.x : v.y;
        } else if constexpr (S::REM > 0) {
            const double2 v = row[(8 * S::FULL + g) ^ sw];
            x[2 * S::FULL] = g >= S::REM ? 0.0 : v.x;
            x[2 * S::FULL + 1] = g >= S::REM ? 0.0 : v.y;
        }
#pragma unroll
        for (int i = 0; i < S::TILES; i++)
#pragma unroll
            for (int j = i; j < S::TILES; j++)
                if (S::prod(i, j) % S::SPLIT == H)
                    gram_mma(acc[S::prod(i, j) / S::SPLIT], x[i], x[j]);
    }
}

// accumulators of one thread over the tiles of a block, and the block's sum
template <int M>
struct GramAcc {
    using S = GramShape<M>;
    double acc[S::NACC][2];
    int grp, half, lane;
    __device__ explicit GramAcc(int t) {
        lane = t & 31;
        half = (t >> 5) % S::SPLIT;
        grp = (t >> 5) / S::SPLIT;
        clear();
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < S::NACC; i++) acc[i][0] = acc[i][1] = 0.0;
    }
    __device__ __forceinline__ void add(const double2* As) {
        static_for<S::SPLIT>([&](auto h) {
            if (half == decltype(h)::value)
                gram_products<M, decltype(h)::value>(As, grp, lane, acc);
        });
    }
    // row groups added in order 0, 1, ... in shared memory (the A tile), the
    // complex upper triangle stored to out[0 .. ENT); every thread calls it
    __device__ __forceinline__ void store(double2* As, double2* __restrict__ out) {
        double* sum = (double*)As;
        for (int g = 0; g < S::GROUPS; g++) {
            if (grp == g) {
#pragma unroll
                for (int i = 0; i < S::NACC; i++) {
                    const int p = i * S::SPLIT + half;
                    if (p >= S::PRODS) continue;
                    double* d = sum + p * 64 + (lane >> 2) * 8 + 2 * (lane & 3);
                    d[0] = g == 0 ? acc[i][0] : d[0] + acc[i][0];
                    d[1] = g == 0 ? acc[i][1] : d[1] + acc[i][1];
                }
            }
            __syncthreads();
        }
        for (int e = threadIdx.x; e < S::ENT; e += blockDim.x) {
            int a = 0, b = e;
            while (b >= S::P - a) b -= S::P - a++;
            b += a;
            const int ra = S::col(a, 0), ia = S::col(a, 1), rb = S::col(b, 0), ib = S::col(b, 1);
            out[e] = make_double2(sum[S::at(ra, rb)] + sum[S::at(ia, ib)],
                                  sum[S::at(ra, ib)] - sum[S::at(ia, rb)]);
        }
        __syncthreads();
    }
};

// Summed Gram entry `e` of the upper triangle written to rho2 (M^4, (k,s,q,l)
// at k + sM + qM^2 + lM^3): every ordering of a pair reads the same entry, the
// lower triangle is the conjugate of the upper, diagonal entries are real.
template <int M>
__device__ inline void gram_fill(int e, double2 v, double2* __restrict__ rho2) {
    constexpr int P = gram_p(M), M2 = M * M, M3 = M2 * M;
    int pa = 0, pb = e;
    while (pb >= P - pa) pb -= P - pa++;
    pb += pa;
    if (pa == pb) v.y = 0.0;
    const double2 vc = make_double2(v.x, -v.y);
    int k = 0, s = pa, q = 0, l = pb;
    while (s >= M - k) s -= M - k++;
    while (l >= M - q) l -= M - q++;
    s += k;
    l += q;
    const int ks[2][2] = {{k, s}, {s, k}}, ql[2][2] = {{q, l}, {l, q}};
    for (int u = 0; u < (k == s ? 1 : 2); u++)
        for (int w = 0; w < (q == l ? 1 : 2); w++) {
            rho2[ks[u][0] + ks[u][1] * M + ql[w][0] * M2 + ql[w][1] * M3] = v;
            rho2[ql[w][0] + ql[w][1] * M + ks[u][0] * M2 + ks[u][1] * M3] = vc;
        }
}

// Sum of `n` partials of one entry (`stride` apart) by a block of 8 warps: lane
// = entry, each warp an eighth of the partials in order, the eighths in order.
// Warp 0 gets the sum.  (One thread an entry took 77 us for 296 partials at
// N=30 M=8, 3 us so.)
__device__ __forceinline__ double2 gram_sum_parts(const double2* part, int n, size_t stride,
                                                  bool live) {
    __shared__ double2 piece[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int per = (n + 7) / 8, b0 = w * per, b1 = min(b0 + per, n);
    double2 v = make_double2(0.0, 0.0);
    if (live) {
#pragma unroll 4
        for (int b = b0; b < b1; b++) v = cadd(v, part[b * stride]);
    }
    piece[w][lane] = v;
    __syncthreads();
    if (w == 0)
        for (int u = 1; u < 8; u++) v = cadd(v, piece[u][lane]);
    return v;
}

// rho1 from the filled rho2 (N >= 2 bosons): sum_s a+_s a_s counts the N - 1
// bosons left after a_l, so rho1[k][l] = sum_s rho2[k,s,s,l] / (N - 1).  The
// sum runs over s in order; rho2[l,s,s,k] is the exact conjugate of
// rho2[k,s,s,l] (gram_fill), so rho1 comes out exactly Hermitian with a
// real diagonal.  Threads t, t + nt, ... take one entry each.  rho2 may have
// been written earlier in the same kernel, so it is read through a plain
// pointer: no read-only (non-coherent) cache path.
__device__ __forceinline__ void rho1_from_rho2(int N, int M, const double2* rho2, double2* rho1,
                                               int t, int nt) {
    const int M2 = M * M, M3 = M2 * M;
    const double d = (double)(N - 1);
    for (int e = t; e < M2; e += nt) {
        const int k = e / M, l = e % M;
        double2 v = make_double2(0.0, 0.0);
        for (int s = 0; s < M; s++) v = cadd(v, rho2[k + s * M + s * M2 + l * M3]);
        rho1[e] = make_double2(v.x / d, v.y / d);
    }
}

// ---------------------------------------------------------------------------
// single-system kernels
// ---------------------------------------------------------------------------
// One block's share of the Gram matrix of the two-boson-annihilated states of
// C: tiles blockIdx.x, blockIdx.x + gridDim.x, ...; partial: gridDim.x x ENT.
template <int M>
__global__ void __launch_bounds__(kGramThreads, 2)
    gram_kernel(SpaceView sp, uint32_t Dp, const double2* __restrict__ C,
                double2* __restrict__ partial) {
    using S = GramShape<M>;
    extern __shared__ double2 As[];
    GramAcc<M> acc(threadIdx.x);
    const uint32_t ntile_rows = (Dp + S::ROWS - 1) / S::ROWS;
    for (uint32_t tr = blockIdx.x; tr < ntile_rows; tr += gridDim.x) {
        gram_gather<M>(sp, Dp, C, tr, As, threadIdx.x);
        __syncthreads();
        acc.add(As);
        __syncthreads();
    }
    acc.store(As, partial + (size_t)blockIdx.x * S::ENT);
}

// Sum of the block partials and the fill of rho2, 32 entries a block
template <int M>
__global__ void __launch_bounds__(256)
    gram_finalize_kernel(int blocks, const double2* __restrict__ part,
                         double2* __restrict__ rho2) {
    constexpr int ENT = gram_entries(M);
    const int e = blockIdx.x * 32 + (threadIdx.x & 31);
    const double2 v = gram_sum_parts(part + e, blocks, ENT, e < ENT);
    if (threadIdx.x < 32 && e < ENT) gram_fill<M>(e, v, rho2);
}

template <int M>
__global__ void __launch_bounds__(64) gram_rho1_kernel(int N, const double2* __restrict__ rho2,
                                                      double2* __restrict__ rho1) {
    rho1_from_rho2(N, M, rho2, rho1, threadIdx.x, blockDim.x);
}

// one boson: rho1[k][l] = conj(C_k) C_l (the configuration of rank l has its
// boson in orbital l), rho2 = 0
template <int M>
__global__ void __launch_bounds__(256)
    gram_one_kernel(const double2* __restrict__ C, double2* __restrict__ rho1,
                    double2* __restrict__ rho2) {
    for (int e = threadIdx.x; e < M * M * M * M; e += blockDim.x)
        rho2[e] = make_double2(0.0, 0.0);
    for (int e = threadIdx.x; e < M * M; e += blockDim.x) {
        const double2 v = cfma_conj(C[e / M], C[e % M], make_double2(0.0, 0.0));
        rho1[e] = make_double2(v.x, e / M == e % M ? 0.0 : v.y);
    }
}

// launch attributes (dynamic shared memory beyond 48 KB), before any capture
template <int M>
int gram_prepare_tmpl() {
    static std::atomic<uint64_t> done{0};
    return set_attributes_once(done, []() -> int {
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(
            gram_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, gram_smem(M)));
        return 0;
    });
}

template <int M>
int gram_apply_tmpl(const SpaceView& sp, uint32_t D2, const double2* C, double2* partial,
                    double2* rho1, double2* rho2, cudaStream_t st) {
    if (sp.N < 2) {
        gram_one_kernel<M><<<1, 256, 0, st>>>(C, rho1, rho2);
        MCTDHB_CUDA_TRY(cudaGetLastError());
        return 0;
    }
    const int blocks = gram_blocks(M, D2);
    gram_kernel<M><<<blocks, kGramThreads, gram_smem(M), st>>>(sp, D2, C, partial);
    gram_finalize_kernel<M><<<(gram_entries(M) + 31) / 32, 256, 0, st>>>(blocks, partial, rho2);
    gram_rho1_kernel<M><<<1, 64, 0, st>>>(sp.N, rho2, rho1);
    MCTDHB_CUDA_TRY(cudaGetLastError());
    return 0;
}

}  // namespace mctdhb
