// pairhc_tmpl.cuh -- H.C through the two-boson-annihilated space, for
// 2 <= M <= 8 orbitals and N >= 2 bosons (explicit instantiations in
// hc_m*.cu).
//
// The Hamiltonian of hamiltonian.c:7-406 is a pair operator.  On the N-boson
// space a+_k a_q = (1/(N-1)) sum_x a+_k a+_x a_x a_q (sum_x a+_x a_x counts
// the N-1 bosons left after a_q), so
//     H = sum_{P,Q} W[P][Q] a+_P a_Q,     P = {k <= s}, Q = {q <= l},
// with a+_P = a+_k a+_s, a_Q = a_q a_l and W built from h and g with the
// same g elements and combinatorial factors as the reference's rules
// (hcp_w_kernel).  With A_m(Q) = <m|a_Q|C> over the D(N-2, M) configurations
// m of N-2 bosons,
//     Y_m(P) = sum_Q W[P][Q] A_m(Q)                 (hcp_y_kernel)
//     (HC)_i = sum_{P in i} <i|a+_P|i-P> Y_{i-P}(P)  (hcp_g_kernel)
// At N=30, M=8 this is 6.7 M x 36 gathers, a 36 x 36 complex matrix-vector
// product per m (FP64 tensor cores, W staged in shared memory; gather and
// contraction overlapped by warp specialisation) and 10.3 M x 36
// coalesced reads of Y, instead of ~576 scattered coefficient gathers per
// row.  Y (D(N-2, M) x P complex, pair-major so that both kernels access it
// with consecutive lanes on consecutive m) is scratch owned by the Fock
// space.  Every value is computed by one thread in a fixed order, so the
// result does not depend on the launch geometry.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "gram_tmpl.cuh"
#include "kernels.h"
#include "movelist.cuh"

namespace mctdhb {

// shared memory for the producers' rank and square-root tables
constexpr int kPairTabBytes = 8192;

// Launch variants of the pair contraction (the autotuner's choices, tune.cu):
// every variant computes each Y value with the same instructions in the
// same order, so a choice changes speed, never results.
//   0  tiles of 256 rows (128 at 7 and 8 orbitals), one block barrier a tile
//   1  tiles of half as many rows (up to 6 orbitals): twice the tiles, for
//      spaces with fewer tiles than SMs
//   2  variant 0 with two output tiles at a time (from 6 orbitals)
//   3  32 rows at a time handed from one producer warp to its own consumer
//      warp (two at 7 and 8 orbitals) through mbarriers: no barrier joins the
//      block, so a consumer's loads, sums and stores run beside another's
//      products.  What a per-tile barrier costs: eight consumer warps on
//      staged tiles alone took 988 us at N=60 M=6 with it, 704 us without
//      (549 us is the tensor cores' time)
// pair_variant_ok says which exist for M; the batched engine, whose tile
// lists fix the rows per tile, takes 0, 2 and 3.
// (pair_variant_ok and kPairVariants: kernels.h)

template <int M, int V = 0>
struct PairHcShape {
    static constexpr int P = M * (M + 1) / 2;
    static constexpr int CONSUMERS = 256;  // 8 warps: the contraction on the tensor cores
    // Rows of A per tile, one producer thread per row (unrank and gather).
    // Up to 6 orbitals a row carries little contraction, so a tile must
    // keep 256 rows of gathers in flight for the tensor cores; at 7 and 8
    // orbitals 128 rows do.
    static constexpr bool WIDE = P <= 21;
    static constexpr int ROWS = (WIDE ? 256 : 128) / (V == 1 ? 2 : 1);
    static constexpr int PRODUCERS = ROWS;
    static constexpr int THREADS = CONSUMERS + PRODUCERS;
    // contraction depth on the tensor cores: P rounded up to 4, in KS steps of
    // 4 taken two at a time (mma m16n8k8, m16n8k4 for an odd last one);
    // 8-wide output tiles.  When P is one above a multiple of 4 (21 pairs,
    // six orbitals) the last input pair is added by FP64 FMAs on the
    // accumulator fragments (KTAIL) instead of a padded step: 20 columns on
    // the tensor cores instead of 24.
    static constexpr bool KTAIL = P % 4 == 1 && P > 4;
    static constexpr int KP = KTAIL ? P - 1 : (P + 3) / 4 * 4;
    static constexpr int KS = KP / 4;
    static constexpr int NN = (P + 7) / 8;
    // Two forms of the complex product (pair_strip): up to seven orbitals the
    // A fragments of a strip stay in registers; at eight they would take 72
    // registers and their sums 36, and the form that reads them once per pass
    // over NG output tiles is 2 % faster (N=30 M=8: H.C 3,027 against 2,974 us)
    static constexpr bool HELD = M < 8;
    // output tiles at a time
    static constexpr int NG = HELD ? (V == 2 ? 2 : 1) : V == 2 ? 2 : 3;
    static constexpr bool PIPE = V == 3;
    static constexpr int PW = PRODUCERS / 32;  // producer warps
    static constexpr int CPP = 8 / PW;         // consumer warps of a producer warp (PIPE)
    // PIPE: registers a thread after the split (setmaxnreg; 0: no split).  A
    // block's registers at launch are 512 x 128 and the two roles' shares are
    // that.  A consumer holds the A fragments of a strip and their sums beside
    // the accumulators, and 128 registers leave it no loads in flight (N=60
    // M=6, H.C: 1,431 us without the split, 1,349 us with 152, 1,328 us with
    // 168 registers).
    static constexpr int CREG = PIPE && (M == 5 || M == 6) ? 168 : 0, PREG = 88;
    static_assert(CREG == 0 || CONSUMERS * CREG + PRODUCERS * PREG <= THREADS * 128,
                  "the split draws on the registers of the launch");
    // Shared memory, in 16-byte words.  A row of the A tile takes PS words (KP,
    // or P with a tail, rounded up to 8), and element q of row r sits at
    // r * PS + (q ^ swz(r)): the 8 rows stored by 8 consecutive producer
    // lanes fall in 8 different bank groups, and so do the 8 lanes (rows g,
    // g + 1, columns t = 0..3) of each phase of a fragment load.  Columns P ..
    // KP-1 hold zeros.
    static constexpr int PS = ((KTAIL ? P : KP) + 7) / 8 * 8;
    // W in the order of its fragments: word (k * NN + n) * 32 + lane holds the
    // output pair 8n + lane / 4, input pair 4k + lane % 4, zero past the end;
    // then the NN * 8 words of the tail column; then, up to six orbitals, the
    // plane Wr + Wi of the same words (beyond, where two W buffers leave no
    // room, it is formed per fragment).
    static constexpr int WF = KS * NN * 32, WT = KTAIL ? NN * 8 : 0;
    static constexpr bool W3 = M <= 6;
    static constexpr int WWORDS = (WF + WT) + (W3 ? (WF + WT + 1) / 2 : 0);
    static constexpr size_t SMEM =
        (2 * (size_t)ROWS * PS + WWORDS) * sizeof(double2) + kPairTabBytes;
    __host__ __device__ static constexpr int swz(int r) { return ((r & 1) << 2) | ((r >> 1) & 3); }
    __host__ __device__ static constexpr int at(int r, int q) { return r * PS + (q ^ swz(r)); }
};

// mbarriers in shared memory (CTA scope): init by one thread before a block
// barrier; arrive (release) by every thread of a role; a wait (acquire)
// that gives up after about two seconds of clock cycles and returns false,
// so a handover that never comes cannot hold the GPU
__device__ __forceinline__ unsigned mbar_addr(const uint64_t* bar) {
    return (unsigned)__cvta_generic_to_shared(bar);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(mbar_addr(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(
                     mbar_addr(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
// Waits about 2 s at most; NOWAIT: what is not ready is lost at once.  The
// lanes of a warp may disagree at the limit, so the callers take a vote before
// they act on a loss.  A warp that lost a wait takes no further part: it arrives
// on nothing that it has not waited for, so nobody takes a buffer for full or
// empty that is not, and whoever depends on it runs out as well.
constexpr long long kMbarWaitCycles = 4000000000LL;
template <bool NOWAIT>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    if constexpr (NOWAIT) return mbar_test(bar, parity);
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(bar, parity))
        if (clock64() - t0 > kMbarWaitCycles) return false;
    return true;
}

// the register split of the two roles (whole warpgroups call it): producers
// give registers back, consumers wait for theirs
template <int CREG, int PREG>
__device__ __forceinline__ void pair_regs_dec() {
    if constexpr (CREG > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(PREG));
}
template <int CREG>
__device__ __forceinline__ void pair_regs_inc() {
    if constexpr (CREG > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(CREG));
}

// barrier 1 over the block's NT threads (producer and consumer loops meet
// here from their own code paths)
template <int NT>
__device__ __forceinline__ void pair_tile_barrier() {
    asm volatile("bar.sync 1, %0;\n" ::"n"(NT) : "memory");
}

// barrier 2 over the NP producer threads (table staging in the batched
// kernel)
template <int NP>
__device__ __forceinline__ void pair_producer_barrier() {
    asm volatile("bar.sync 2, %0;\n" ::"n"(NP) : "memory");
}

// FP64 mma.sync m16n8k8: D(16x8) += A(16x8) B(8x8).  With g = lane / 4 and
// t = lane % 4, lane l holds A[g][t], A[g+8][t], A[g][t+4], A[g+8][t+4];
// B[t][g], B[t+4][g]; D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1]
__device__ __forceinline__ void dmma1688(double (&d)[4], double a0, double a1, double a2,
                                         double a3, double b0, double b1) {
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// m16n8k4: lane l holds A[g][t], A[g+8][t]; B[t][g]; D as m16n8k8
__device__ __forceinline__ void dmma1684(double (&d)[4], double a0, double a1, double b0) {
    asm(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
        "{%0, %1, %2, %3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

// The rank table (M - 1 rows of N + 1) and the square-root table (N + 3)
// of a space staged in shared memory for the producers' unranking, when
// they fit kPairTabBytes (else the view keeps the global tables): the
// unrank is a chain of dependent table reads, and the L1 left beside the
// contraction's shared memory does not hold them against the gathers.
__host__ __device__ constexpr bool pair_tab_fits(int N, int M) {
    return (N + 3) * 8 + (M - 1) * (N + 1) * 4 <= kPairTabBytes;
}
// tab: kPairTabBytes of shared memory (8-byte aligned); threads t, t + nt, ...
// copy; the caller synchronises its threads before the view is used
__device__ __forceinline__ SpaceView pair_stage_tab(const SpaceView& sp, void* tab, int t,
                                                    int nt) {
    SpaceView v = sp;
    if (!pair_tab_fits(sp.N, sp.M)) return v;
    double* sq = (double*)tab;
    uint32_t* T = (uint32_t*)(sq + sp.N + 3);
    const int nsq = sp.N + 3, nT = (sp.M - 1) * (sp.N + 1);
    for (int i = t; i < nsq; i += nt) sq[i] = sp.sq[i];
    for (int i = t; i < nT; i += nt) T[i] = sp.T[i];
    v.sq = sq;
    v.T = T;
    return v;
}

// W (P x P, global) staged into Ws (PairHcShape's layout) by threads t,
// t + nt, ...
template <int M, int V = 0>
__device__ __forceinline__ void pair_stage_w(const double2* __restrict__ W, double2* Ws, int t,
                                             int nt) {
    using S = PairHcShape<M, V>;
    constexpr int P = S::P;
    double* w3 = (double*)(Ws + S::WF + S::WT);
    for (int i = t; i < S::WF + S::WT; i += nt) {
        const int lane = i & 31, kn = i >> 5, c = i - S::WF;
        const int p = i < S::WF ? kn % S::NN * 8 + (lane >> 2) : c;
        const int q = i < S::WF ? kn / S::NN * 4 + (lane & 3) : P - 1;
        const double2 w = p < P && q < P ? W[p * P + q] : make_double2(0.0, 0.0);
        Ws[i] = w;
        if constexpr (S::W3) w3[i] = w.x + w.y;
    }
}

// ---------------------------------------------------------------------------
// building blocks (shared with the batched engine, batch_tmpl.cuh)
// ---------------------------------------------------------------------------
// `row` of the (N-2)-boson space (the last one past the end) into row r of the
// A tile As: A_m(Q) = sqrt((m_q+1)(m_l+1+[q=l])) C[m + e_q + e_l]
template <int M, int V = 0>
__device__ __forceinline__ void pair_gather_row(const SpaceView& sp,
                                                const double2* __restrict__ C, uint32_t row,
                                                double2* As, int r) {
    using S = PairHcShape<M, V>;
    constexpr int P = S::P;
    const uint32_t D2 = sp.dim2;
    row = min(row, D2 - 1u);
    int n[M];
    uint32_t U1[M], U2[M];
    gram_unrank<M, true>(sp.T, sp.N, sp.N - 2, D2, row, n, U1, U2);
    const uint32_t j0 = sp.dim - D2 + row;
    // sqrt(n_x + 1), sqrt(n_x + 2) once per orbital
    double s1[M], s2[M];
#pragma unroll
    for (int x = 0; x < M; x++) {
        s1[x] = sp.sq[n[x] + 1];
        s2[x] = sp.sq[n[x] + 2];
    }
    static_for<P>([&](auto pi) {
        constexpr int p = decltype(pi)::value;
        constexpr int q = kPairs<M>.q[p], l = kPairs<M>.l[p];
        const uint32_t j = j0 - (U1[q] - U1[l]) - U2[l];
        const double f = q == l ? s1[q] * s2[q] : s1[q] * s1[l];
        As[S::at(r, p)] = cscale(__ldg(C + j), f);
    });
#pragma unroll
    for (int q = P; q < S::KP; q++) As[S::at(r, q)] = make_double2(0.0, 0.0);
}

// Rows r = r0, r0 + rstep, ... < ROWS of tile `tr` into As
template <int M, int V = 0>
__device__ __forceinline__ void pair_gather(const SpaceView& sp, const double2* __restrict__ C,
                                            uint32_t tr, double2* As, int r0, int rstep) {
    constexpr int ROWS = PairHcShape<M, V>::ROWS;
    for (int r = r0; r < ROWS; r += rstep) pair_gather_row<M, V>(sp, C, tr * ROWS + r, As, r);
}

// part F of W word i: 0 Wr, 1 Wi, 2 Wr + Wi
template <int M, int V, int F>
__device__ __forceinline__ double pair_w_part(const double2* Ws, int i) {
    using S = PairHcShape<M, V>;
    if constexpr (F == 0) {
        return Ws[i].x;
    } else if constexpr (F == 1) {
        return Ws[i].y;
    } else if constexpr (S::W3) {
        return ((const double*)(Ws + S::WF + S::WT))[i];
    } else {
        const double2 w = Ws[i];
        return w.x + w.y;
    }
}

// the last input pair by FMAs where P has a tail: D[g][2t + j] += e0
// W[2t + j][P - 1] (rows g + 8 alike), output tiles n0 .. n0 + NG - 1
template <int M, int V, int F>
__device__ __forceinline__ void pair_tail(double e0, double e1, const double2* Ws, int lane, int n0,
                                          double (&acc)[PairHcShape<M, V>::NG][4]) {
    using S = PairHcShape<M, V>;
    if constexpr (S::KTAIL) {
#pragma unroll
        for (int n = 0; n < S::NG; n++) {
            if (n0 + n >= S::NN) continue;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const double w =
                    pair_w_part<M, V, F>(Ws, S::WF + (n0 + n) * 8 + 2 * (lane & 3) + j);
                acc[n][j] = fma(e0, w, acc[n][j]);
                acc[n][j + 2] = fma(e1, w, acc[n][j + 2]);
            }
        }
    }
}

// Y_m(P) = sum_Q W[P][Q] A_m(Q) of a 16-row strip (rows at As, swizzled by the
// row of the strip; m its first row in the (N-2)-space) by one warp on the FP64
// tensor cores, with three real products per complex product:
//     T1 = Ar Wr, T2 = Ai Wi, Yr = T1 - T2, Yi = (Ar + Ai)(Wr + Wi) - T1 - T2.
// The third product continues from -(T1 + T2), Ar + Ai is formed once a strip
// and Wr + Wi once a W: an FP64 addition takes 2.6 cycles of the tensor pipe it
// shares, and 107 of them a strip against 1,440 cycles of products at six
// orbitals are now 72.  (T = (Ar + Ai) Wr continued into both results would
// leave 48, but its longer chains round more: error of H.C 2.4e-16 against
// 2.1e-16.)  When W is real (REAL: real orbitals and coefficients) two products
// do: Yr = Ar Wr, Yi = Ai Wr.  A fragments hold the real and imaginary part of
// an element in one 16-byte load and stay in registers for all output tiles.
// Outputs p >= P and rows m >= D2 are not stored.
template <int M, int V, bool REAL>
__device__ __forceinline__ void pair_strip(const double2* As, const double2* Ws, int lane,
                                           uint32_t m, uint32_t D2, uint32_t ld,
                                           double2* __restrict__ Y) {
    using S = PairHcShape<M, V>;
    constexpr int P = S::P, KS = S::KS, NN = S::NN, NG = S::NG;
    const int g = lane >> 2, t = lane & 3;
    const int sw = S::swz(g);  // rows g and g + 8
    const double2 *r0 = As + g * S::PS, *r1 = r0 + 8 * S::PS;
    double2 a0[KS], a1[KS], e0 = make_double2(0.0, 0.0), e1 = e0;
    double s0[REAL ? 1 : KS], s1[REAL ? 1 : KS];
#pragma unroll
    for (int k = 0; k < KS; k++) {
        a0[k] = r0[(4 * k + t) ^ sw];
        a1[k] = r1[(4 * k + t) ^ sw];
        if constexpr (!REAL) {
            s0[k] = a0[k].x + a0[k].y;
            s1[k] = a1[k].x + a1[k].y;
        }
    }
    if constexpr (S::KTAIL) {
        e0 = r0[(P - 1) ^ sw];
        e1 = r1[(P - 1) ^ sw];
    }
    const double es0 = e0.x + e0.y, es1 = e1.x + e1.y;
#pragma unroll 1
    for (int n0 = 0; n0 < NN; n0 += NG) {
        double T[NG][4], Z[NG][4];
#pragma unroll
        for (int n = 0; n < NG; n++)
#pragma unroll
            for (int j = 0; j < 4; j++) T[n][j] = Z[n][j] = 0.0;
        // T1 and T2 side by side: one 16-byte load serves both
#pragma unroll
        for (int k = 0; k < KS; k += 2)
#pragma unroll
            for (int n = 0; n < NG; n++) {
                if (n0 + n >= NN) continue;
                const int i = (k * NN + n0 + n) * 32 + lane;
                const double2 w0 = Ws[i];
                if (k + 1 < KS) {
                    const double2 w1 = Ws[i + NN * 32];
                    dmma1688(T[n], a0[k].x, a1[k].x, a0[k + 1].x, a1[k + 1].x, w0.x, w1.x);
                    dmma1688(Z[n], a0[k].y, a1[k].y, a0[k + 1].y, a1[k + 1].y,
                             REAL ? w0.x : w0.y, REAL ? w1.x : w1.y);
                } else {
                    dmma1684(T[n], a0[k].x, a1[k].x, w0.x);
                    dmma1684(Z[n], a0[k].y, a1[k].y, REAL ? w0.x : w0.y);
                }
            }
        pair_tail<M, V, 0>(e0.x, e1.x, Ws, lane, n0, T);
        pair_tail<M, V, REAL ? 0 : 1>(e0.y, e1.y, Ws, lane, n0, Z);
        if constexpr (!REAL) {
#pragma unroll
            for (int n = 0; n < NG; n++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const double t1 = T[n][j], t2 = Z[n][j];
                    T[n][j] = t1 - t2;
                    Z[n][j] = -t1 - t2;
                }
#pragma unroll
            for (int k = 0; k < KS; k += 2)
#pragma unroll
                for (int n = 0; n < NG; n++) {
                    if (n0 + n >= NN) continue;
                    const int i = (k * NN + n0 + n) * 32 + lane;
                    const double w0 = pair_w_part<M, V, 2>(Ws, i);
                    if (k + 1 < KS)
                        dmma1688(Z[n], s0[k], s1[k], s0[k + 1], s1[k + 1], w0,
                                 pair_w_part<M, V, 2>(Ws, i + NN * 32));
                    else
                        dmma1684(Z[n], s0[k], s1[k], w0);
                }
            pair_tail<M, V, 2>(es0, es1, Ws, lane, n0, Z);
        }
#pragma unroll
        for (int n = 0; n < NG; n++) {
            if (n0 + n >= NN) continue;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int p = (n0 + n) * 8 + 2 * t + j;
                if (p >= P) continue;
                double2* y = Y + (size_t)p * ld + m + g;
                if (m + g < D2) y[0] = make_double2(T[n][j], Z[n][j]);
                if (m + g + 8 < D2) y[8] = make_double2(T[n][j + 2], Z[n][j + 2]);
            }
        }
    }
}

// The same strip with the A fragments read once per pass over NG output tiles
// (eight orbitals) and three sums: T1 = Ar Wr, T2 = Ai Wi, T3 = (Ar + Ai)
// (Wr + Wi), Yr = T1 - T2, Yi = T3 - T1 - T2.
template <int M, int V, bool REAL>
__device__ __forceinline__ void pair_strip_passes(const double2* As, const double2* Ws, int lane,
                                                  uint32_t m, uint32_t D2, uint32_t ld,
                                                  double2* __restrict__ Y) {
    using S = PairHcShape<M, V>;
    constexpr int P = S::P, KS = S::KS, NN = S::NN, NG = S::NG;
    static_assert(!S::KTAIL, "no tail column");
    const int g = lane >> 2, t = lane & 3;
    const int sw = S::swz(g);  // rows g and g + 8
    const double2 *r0 = As + g * S::PS, *r1 = r0 + 8 * S::PS;
#pragma unroll
    for (int n0 = 0; n0 < NN; n0 += NG) {
        double t1[NG][4], t2[NG][4], t3[REAL ? 1 : NG][4];
#pragma unroll
        for (int n = 0; n < NG; n++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                t1[n][j] = t2[n][j] = 0.0;
                if constexpr (!REAL) t3[n][j] = 0.0;
            }
#pragma unroll
        for (int k = 0; k < KS; k += 2) {
            const bool deep = k + 1 < KS;  // an 8-deep step (else the last 4)
            const int q = 4 * k + t;
            const double2 zero = make_double2(0.0, 0.0);
            const double2 a0 = r0[q ^ sw], a1 = r1[q ^ sw];
            const double2 a2 = deep ? r0[(q + 4) ^ sw] : zero, a3 = deep ? r1[(q + 4) ^ sw] : zero;
#pragma unroll
            for (int n = 0; n < NG; n++) {
                if (n0 + n >= NN) continue;
                const int i = (k * NN + n0 + n) * 32 + lane;
                const double2 b0 = Ws[i], b1 = deep ? Ws[i + NN * 32] : zero;
                if (deep) {
                    dmma1688(t1[n], a0.x, a1.x, a2.x, a3.x, b0.x, b1.x);
                    if constexpr (REAL) {
                        dmma1688(t2[n], a0.y, a1.y, a2.y, a3.y, b0.x, b1.x);
                    } else {
                        dmma1688(t2[n], a0.y, a1.y, a2.y, a3.y, b0.y, b1.y);
                        dmma1688(t3[n], a0.x + a0.y, a1.x + a1.y, a2.x + a2.y, a3.x + a3.y,
                                 b0.x + b0.y, b1.x + b1.y);
                    }
                } else {
                    dmma1684(t1[n], a0.x, a1.x, b0.x);
                    if constexpr (REAL) {
                        dmma1684(t2[n], a0.y, a1.y, b0.x);
                    } else {
                        dmma1684(t2[n], a0.y, a1.y, b0.y);
                        dmma1684(t3[n], a0.x + a0.y, a1.x + a1.y, b0.x + b0.y);
                    }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NG; n++) {
            if (n0 + n >= NN) continue;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int p = (n0 + n) * 8 + 2 * t + (j & 1);
                const uint32_t row = m + g + (j >> 1) * 8;
                if (p >= P || row >= D2) continue;
                if constexpr (REAL)
                    Y[(size_t)p * ld + row] = make_double2(t1[n][j], t2[n][j]);
                else
                    Y[(size_t)p * ld + row] =
                        make_double2(t1[n][j] - t2[n][j], t3[n][j] - t1[n][j] - t2[n][j]);
            }
        }
    }
}

// strips st = s0, s0 + step, ... < ns of the rows at As; `real`: the flag
// stored after the P x P entries of W
template <int M, int V = 0>
__device__ __forceinline__ void pair_strips(const double2* As, const double2* Ws, int s0, int step,
                                            int ns, int lane, uint32_t row0, uint32_t D2,
                                            uint32_t ld, double2* __restrict__ Y, bool real) {
    using S = PairHcShape<M, V>;
    constexpr int W16 = 16 * S::PS;
    auto strip = [&](auto re, int st) {
        constexpr bool REAL = decltype(re)::value;
        if constexpr (S::HELD)
            pair_strip<M, V, REAL>(As + st * W16, Ws, lane, row0 + st * 16, D2, ld, Y);
        else
            pair_strip_passes<M, V, REAL>(As + st * W16, Ws, lane, row0 + st * 16, D2, ld, Y);
    };
    if (real) {
        for (int st = s0; st < ns; st += step) strip(std::true_type{}, st);
    } else {
        for (int st = s0; st < ns; st += step) strip(std::false_type{}, st);
    }
}

// consumer thread t (0 .. CONSUMERS-1) of a tile whose first row is row0
template <int M, int V = 0>
__device__ __forceinline__ void pair_consume(const double2* As, const double2* Ws, int t,
                                             uint32_t row0, uint32_t D2, uint32_t ld,
                                             double2* __restrict__ Y, bool real) {
    using S = PairHcShape<M, V>;
    pair_strips<M, V>(As, Ws, t >> 5, S::CONSUMERS / 32, S::ROWS / 16, t & 31, row0, D2, ld, Y,
                      real);
}

// NaN into all planes of the chunks of 32 rows c, c + step, ... < nchunk: they
// were not handed over
template <int M>
__device__ __forceinline__ void pair_poison(uint32_t c, uint32_t step, uint32_t nchunk, int lane,
                                            const SpaceView& sp, double2* __restrict__ Y) {
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    constexpr int UNROLL = M == 7 ? M * (M + 1) / 2 : 1;  // hcp_y_kernel, IN_LOOP
    for (; c < nchunk; c += step) {
        const uint32_t m = c * 32 + lane;
        if (m >= sp.dim2) continue;
#pragma unroll UNROLL
        for (int p = 0; p < M * (M + 1) / 2; p++)
            Y[(size_t)p * sp.ldy + m] = make_double2(nan, nan);
    }
}

// (HC)_row = sum over pairs P = {k <= s} present in the row of
// sqrt(n_k (n_s - [k=s])) Y_{row - e_k - e_s}(P)
template <int M>
__device__ __forceinline__ double2 pair_gather_back(const SpaceView& sp,
                                                    const double2* __restrict__ Y,
                                                    uint32_t row) {
    constexpr int P = M * (M + 1) / 2;
    const int N = sp.N;
    const uint32_t D2 = sp.dim2;
    // occupations and the suffix sums of the rank offsets of removing one /
    // two bosons: V_d[x] = sum_{y >= x} T_y(L_y) - T_y(L_y - d)
    int n[M];
    uint32_t V1[M], V2[M];
    {
        uint32_t S = sp.dim - 1u - row;
        int Lnext = N;
        int L[M - 1];
#pragma unroll
        for (int x = M - 2; x >= 0; x--) {
            const uint32_t* Tx = sp.T + x * (N + 1);
            const int lo = cns_level(Tx, x, Lnext, S);
            S -= __ldg(Tx + lo);
            n[x + 1] = Lnext - lo;
            L[x] = lo;
            Lnext = lo;
        }
        n[0] = Lnext;
        V1[M - 1] = 0u;
        V2[M - 1] = 0u;
        // an L_y below d only occurs for y below the orbitals of a pair that
        // cannot be removed; those sums are never used
#pragma unroll
        for (int x = M - 2; x >= 0; x--) {
            const uint32_t* Tx = sp.T + x * (N + 1);
            const uint32_t t0 = __ldg(Tx + L[x]);
            V1[x] = V1[x + 1] + (t0 - __ldg(Tx + (L[x] >= 1 ? L[x] - 1 : 0)));
            V2[x] = V2[x + 1] + (t0 - __ldg(Tx + (L[x] >= 2 ? L[x] - 2 : 0)));
        }
    }
    const uint32_t base = D2 - sp.dim + row;
    double2 acc = make_double2(0.0, 0.0);
    // every pair is loaded (row 0 of its plane where the pair is absent, with
    // weight f = 0), so the loads do not wait on branches
    static_for<P>([&](auto pi) {
        constexpr int p = decltype(pi)::value;
        constexpr int k = kPairs<M>.q[p], s = kPairs<M>.l[p];
        bool valid;
        double f;
        if constexpr (k == s) {
            valid = n[k] >= 2;
            f = __ldg(sp.sq + n[k]) * __ldg(sp.sq + (n[k] >= 1 ? n[k] - 1 : 0));
        } else {
            valid = n[k] >= 1 && n[s] >= 1;
            f = __ldg(sp.sq + n[k]) * __ldg(sp.sq + n[s]);
        }
        const uint32_t m = valid ? base + (V1[k] - V1[s]) + V2[s] : 0u;
        const double2 y = __ldg(Y + (size_t)p * sp.ldy + m);
        acc.x = fma(f, y.x, acc.x);
        acc.y = fma(f, y.y, acc.y);
    });
    return acc;
}

// ---------------------------------------------------------------------------
// single-system kernels
// ---------------------------------------------------------------------------
// Y = A W^T for the rows m of the (N-2)-boson space; Y[p * ldy + m] (planes an
// odd number of rows apart, pair_ld).  Warp-specialised and
// double-buffered: while the consumer warps contract rows from one A buffer,
// the producer warps unrank and gather the next ones into the other.
template <int M, int V, bool NOWAIT = false>
__global__ void __launch_bounds__(PairHcShape<M, V>::THREADS, 1)
    hcp_y_kernel(SpaceView sp, const double2* __restrict__ C, const double2* __restrict__ W,
                 double2* __restrict__ Y, HcEpilogue ep) {
    using S = PairHcShape<M, V>;
    constexpr int P = S::P, PS = S::PS, ROWS = S::ROWS;
    extern __shared__ double2 smem[];
    double2* Ab = smem;  // two buffers of ROWS x PS
    double2* Ws = smem + 2 * ROWS * PS;
    if (ep.flag != nullptr && *ep.flag != 0) return;  // Lanczos breakdown: no-op
    const int t = threadIdx.x;
    pair_stage_w<M, V>(W, Ws, t, S::THREADS);
    const SpaceView tv = pair_stage_tab(sp, Ws + S::WWORDS, t, S::THREADS);
    const bool real = W[P * P].x != 0.0;
    const bool producer = t >= S::CONSUMERS;
    const int pt = t - S::CONSUMERS, lane = t & 31;
    if constexpr (S::PIPE) {
        __shared__ uint64_t full[S::PW][2], empty[S::PW][2];
        if (t < 2 * S::PW) {
            mbar_init(&full[t >> 1][t & 1], 32);
            mbar_init(&empty[t >> 1][t & 1], 32 * S::CPP);
        }
        __syncthreads();
        // pair w of this block takes the chunks of 32 rows blockIdx.x +
        // w gridDim.x, ...: a small space spreads over the SMs first.  A
        // consumer that lost a wait leaves NaN in that chunk and all it still
        // has to do: every row of H.C that reads one of them is NaN, and with it
        // the dots of a Lanczos step and all that follows.  A producer that
        // lost one stops, and its consumers run out.
        const int w = producer ? pt >> 5 : (t >> 5) / S::CPP;
        const uint32_t nchunk = (sp.dim2 + 31) / 32, step = gridDim.x * S::PW;
        double2* ring = Ab + w * 2 * 32 * PS;
        const uint32_t c0 = blockIdx.x + w * gridDim.x;
        if constexpr (S::CREG > 0) {
            // Five and six orbitals: with a real W the consumers need neither
            // the A sums nor the third product and the producers set the pace,
            // so the registers stay as launched (N=60 M=6, H.C with a real W:
            // 1,222 us with the split, 1,168 us without).
            auto run = [&](auto real_w) {
                constexpr bool RE = decltype(real_w)::value;
                int i = 0;
                bool ok = true;
                if (producer) {
                    if constexpr (!RE) pair_regs_dec<S::CREG, S::PREG>();
                    for (uint32_t c = c0; c < nchunk && ok; c += step, i++) {
                        const int buf = i & 1;
                        if (i >= 2) ok = mbar_wait<NOWAIT>(&empty[w][buf], ((i >> 1) - 1) & 1);
                        if (!ok) return;
                        pair_gather_row<M, V>(tv, C, c * 32 + lane, ring + buf * 32 * PS, lane);
                        mbar_arrive(&full[w][buf]);
                    }
                } else {
                    if constexpr (!RE) pair_regs_inc<S::CREG>();
                    for (uint32_t c = c0; c < nchunk && ok; c += step, i++) {
                        const int buf = i & 1;
                        ok = mbar_wait<NOWAIT>(&full[w][buf], (i >> 1) & 1);
                        pair_strips<M, V>(ring + buf * 32 * PS, Ws, (t >> 5) % S::CPP, S::CPP, 2,
                                          lane, c * 32, sp.dim2, sp.ldy, Y, RE);
                        mbar_arrive(&empty[w][buf]);
                        ok = __all_sync(0xffffffffu, ok);
                    }
                    if (!ok) pair_poison<M>(c0 + (i - 1) * step, step, nchunk, lane, sp, Y);
                }
            };
            if (real)
                run(std::true_type{});
            else
                run(std::false_type{});
            return;
        }
        // Where the loss is dealt with changes the code the compiler makes of
        // the consumers' loop: at 7 orbitals in the loop and unrolled (N=25 M=7:
        // 165.6 us of H.C, 169 us not unrolled, 170 us after the loop; 165.2 us
        // with no NaN and no vote at all), else after it (N=30 M=8: 2,952 us,
        // 3,018 us unrolled, 3,048 us in the loop, 3,030 us in a lambda as
        // above; 2,936 us with neither).
        constexpr bool IN_LOOP = M == 7;
        int i = 0;
        bool ok = true;
        if (producer) {
            for (uint32_t c = c0; c < nchunk && ok; c += step, i++) {
                const int buf = i & 1;
                if (i >= 2) ok = mbar_wait<NOWAIT>(&empty[w][buf], ((i >> 1) - 1) & 1);
                if (!ok) return;
                pair_gather_row<M, V>(tv, C, c * 32 + lane, ring + buf * 32 * PS, lane);
                mbar_arrive(&full[w][buf]);
            }
        } else {
            for (uint32_t c = c0; c < nchunk && ok; c += step, i++) {
                const int buf = i & 1;
                ok = mbar_wait<NOWAIT>(&full[w][buf], (i >> 1) & 1);
                pair_strips<M, V>(ring + buf * 32 * PS, Ws, (t >> 5) % S::CPP, S::CPP, 2, lane,
                                  c * 32, sp.dim2, sp.ldy, Y, real);
                mbar_arrive(&empty[w][buf]);
                if constexpr (IN_LOOP) {
                    if (__any_sync(0xffffffffu, !ok)) {
                        pair_poison<M>(c, step, nchunk, lane, sp, Y);
                        return;
                    }
                } else {
                    ok = __all_sync(0xffffffffu, ok);
                }
            }
        }
        if (!IN_LOOP && !ok && !producer)
            pair_poison<M>(c0 + (i - 1) * step, step, nchunk, lane, sp, Y);
        return;
    }
    __syncthreads();
    const uint32_t ntiles = (sp.dim2 + ROWS - 1) / ROWS;
    if (producer && blockIdx.x < ntiles)
        pair_gather<M, V>(tv, C, blockIdx.x, Ab, pt, S::PRODUCERS);
    __syncthreads();
    int buf = 0;
    for (uint32_t tr = blockIdx.x; tr < ntiles; tr += gridDim.x, buf ^= 1) {
        if (producer) {
            const uint32_t nx = tr + gridDim.x;
            if (nx < ntiles)
                pair_gather<M, V>(tv, C, nx, Ab + (size_t)(buf ^ 1) * ROWS * PS, pt,
                                  S::PRODUCERS);
        } else {
            pair_consume<M, V>(Ab + (size_t)buf * ROWS * PS, Ws, t, tr * ROWS, sp.dim2, sp.ldy, Y,
                               real);
        }
        __syncthreads();
    }
}

// (HC)_i gathered back from Y, then the Lanczos epilogue
template <int M, bool LZ>
__global__ void __launch_bounds__(256, M < 8 ? 5 : 4)
    hcp_g_kernel(SpaceView sp, const double2* __restrict__ Y, double2* __restrict__ HC,
                 HcEpilogue ep) {
    if (ep.flag != nullptr && *ep.flag != 0) return;
    double2 alpha = make_double2(0.0, 0.0);
#pragma unroll 1
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < sp.dim;
         row += gridDim.x * blockDim.x) {
        const double2 h = pair_gather_back<M>(sp, Y, row);
        if constexpr (LZ)
            hc_row_epilogue(ep, row, h, HC, alpha);
        else
            HC[row] = h;
    }
    if constexpr (LZ) hc_alpha_epilogue(ep, alpha);
}

template <int M, int V>
int hcp_set_attr() {
    static_assert(PairHcShape<M, V>::SMEM <= 227 * 1024, "shared memory of one block (227 KB)");
    if constexpr (pair_variant_ok(M, V))
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(hcp_y_kernel<M, V>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)PairHcShape<M, V>::SMEM));
    return 0;
}

// the instance without waits, loaded only where it is asked for
template <int M>
int hcp_prepare_nowait_tmpl() {
    MCTDHB_CUDA_TRY(cudaFuncSetAttribute(hcp_y_kernel<M, 3, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)PairHcShape<M, 3>::SMEM));
    return 0;
}

template <int M>
int hcp_prepare_tmpl() {
    static std::atomic<uint64_t> done{0};
    return set_attributes_once(done, []() -> int {
        return hcp_set_attr<M, 0>() || hcp_set_attr<M, 1>() || hcp_set_attr<M, 2>() ||
               hcp_set_attr<M, 3>();
    });
}

// parts & 1: the contraction; parts & 2: the gather-back (with the epilogue)
template <int M, int V>
int hcp_launch_v(const SpaceView& sp, const double2* C, double2* HC, const HcEpilogue& ep,
                 int parts, cudaStream_t st) {
    if constexpr (!pair_variant_ok(M, V)) {
        set_error("pair contraction variant %d does not exist for %d orbitals", V, M);
        return -1;
    } else {
        using S = PairHcShape<M, V>;
        if (parts & 1) {
            const uint32_t rows = S::PIPE ? 32 : S::ROWS, ntiles = (sp.dim2 + rows - 1) / rows;
            const int gy = (int)std::min<uint32_t>(ntiles, (uint32_t)num_sms());
            if (gy > 0) {
                auto* kernel = hcp_y_kernel<M, V>;
                if constexpr (S::PIPE)
                    if (ep.nowait) kernel = hcp_y_kernel<M, V, true>;
                kernel<<<gy, S::THREADS, S::SMEM, st>>>(sp, C, sp.pair_w, sp.pair_y, ep);
                MCTDHB_CUDA_TRY(cudaGetLastError());
            }
        }
        if (parts & 2) {
            const uint32_t need = (sp.dim + 255) / 256;
            const int gg =
                (int)std::max<uint32_t>(1u, std::min<uint32_t>(need, (uint32_t)num_sms() * 8));
            if (ep.part != nullptr)
                hcp_g_kernel<M, true><<<gg, 256, 0, st>>>(sp, sp.pair_y, HC, ep);
            else
                hcp_g_kernel<M, false><<<gg, 256, 0, st>>>(sp, sp.pair_y, HC, ep);
            MCTDHB_CUDA_TRY(cudaGetLastError());
        }
        return 0;
    }
}

template <int M>
int hcp_apply_tmpl(const SpaceView& sp, const double2* C, double2* HC, const HcEpilogue& ep,
                   int variant, int parts, cudaStream_t st) {
    switch (variant) {
        case 1: return hcp_launch_v<M, 1>(sp, C, HC, ep, parts, st);
        case 2: return hcp_launch_v<M, 2>(sp, C, HC, ep, parts, st);
        case 3: return hcp_launch_v<M, 3>(sp, C, HC, ep, parts, st);
        default: return hcp_launch_v<M, 0>(sp, C, HC, ep, parts, st);
    }
}

}  // namespace mctdhb
