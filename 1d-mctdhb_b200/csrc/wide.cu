// wide.cu -- H.C and densities through the two-boson-annihilated space for
// more than 8 orbitals and N >= 2 bosons (M <= 30, P = M(M+1)/2 <= 465
// pairs): the pair operator and the Gram matrix of pairhc_tmpl.cuh and
// gram_tmpl.cuh with the orbital count at run time.
//
//   Y_m(P)   = sum_Q W[P][Q] A_m(Q)               wide_y_kernel
//   (HC)_i   = sum_{P in i} <i|a+_P|i-P> Y_{i-P}(P)  wide_g_kernel
//   rho2     = sum_m conj(A_m(P)) A_m(Q)           wide_gram_kernel
//
// What bounds them.  Spaces of this many orbitals hold few bosons (N=8 M=10:
// 24,310 configurations, 5,005 rows of the (N-2)-space), so the kernels are
// sized for latency: 32 rows a block, every block's rows unranked once into
// shared memory and the pairs of a row spread over all its threads.  The
// products run on the FP64 tensor cores.  Against the per-row kernels, which
// visit every move of every row with occupations in local memory (N=8 M=10,
// one B200): H.C 1,462 us -> 27 us, densities 17,400 us -> 31 us.
//
// Every value is computed by one thread, or summed in a fixed order over a
// grid that depends on (N, M) only.
#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "kernels.h"
#include "moves.cuh"
#include "pairhc_tmpl.cuh"
#include "wide.h"

namespace mctdhb {

namespace {

constexpr int kWideRows = 32;      // rows of the (N-2)-space a Gram block holds
constexpr int kWideThreads = 256;  // 8 warps
constexpr int kWideGRows = 64;     // H.C rows of a gather-back block (4 threads a row)
constexpr int kSuper = 64;         // pairs of a Gram super-tile side
constexpr int kGramPS = kSuper * 2 + 2;  // words of a Gram row: 2 (mod 8), fragments conflict-free

__host__ __device__ constexpr int wide_pairs(int M) { return M * (M + 1) / 2; }
// words of a row of the contraction's A tile: a multiple of 8, element q of
// row r at r * PS + (q ^ swz(r)) (PairHcShape's swizzle)
__host__ __device__ constexpr int wide_ps(int P) { return (P + 7) / 8 * 8; }
__host__ __device__ constexpr int wide_swz(int r) { return ((r & 1) << 2) | ((r >> 1) & 3); }

// pair p <-> (q, l), q <= l, in row-major order of the upper triangle, as
// q << 8 | l
__device__ __forceinline__ unsigned short wide_pair(int M, int p) {
    int q = 0;
    while (p >= M - q) {
        p -= M - q;
        q++;
    }
    return (unsigned short)(q << 8 | (q + p));
}

// Unrank `row` of the space of Np bosons (dimension Dp) with the rank table
// of a space of N >= Np bosons: occupations to n[x * st], cumulative ones in
// L (identical to set_config, space.c:138)
__device__ __forceinline__ void wide_unrank(const SpaceView& sp, int Np, uint32_t Dp,
                                            uint32_t row, int* n, int st, int (&L)[kMaxOrb]) {
    const int M = sp.M, N = sp.N;
    uint32_t S = Dp - 1u - row;
    int Lnext = Np;
    for (int x = M - 2; x >= 0; x--) {
        const uint32_t* Tx = sp.T + x * (N + 1);
        int lo = 0, hi = Lnext;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(Tx + mid) <= S)
                lo = mid;
            else
                hi = mid - 1;
        }
        S -= __ldg(Tx + lo);
        n[(x + 1) * st] = Lnext - lo;
        L[x] = lo;
        Lnext = lo;
    }
    n[0] = Lnext;
}

// shared-memory tables of RB rows: occupations and the suffix sums U1, U2 of
// the rank offsets of one and two bosons more (sign +1) or fewer (sign -1),
// element x of row r at x * RB + r
struct WideRows {
    int* n;
    uint32_t *U1, *U2;
};
__host__ __device__ constexpr size_t wide_rows_bytes(int M, int rb) {
    return (size_t)rb * M * 3 * sizeof(int);
}
__device__ __forceinline__ WideRows wide_rows_at(void* mem, int M, int rb) {
    int* n = (int*)mem;
    return WideRows{n, (uint32_t*)(n + M * rb), (uint32_t*)(n + 2 * M * rb)};
}

// the offsets of row r of the (N-2)-space with one and two bosons more
__device__ __forceinline__ void wide_fill_up(const SpaceView& sp, const WideRows& w, int rb, int r,
                                             uint32_t row) {
    const int M = sp.M, N = sp.N;
    int L[kMaxOrb];
    wide_unrank(sp, N - 2, sp.dim2, row, w.n + r, rb, L);
    uint32_t u1 = 0, u2 = 0;
    w.U1[(M - 1) * rb + r] = 0u;
    w.U2[(M - 1) * rb + r] = 0u;
    for (int x = M - 2; x >= 0; x--) {
        const uint32_t* Tx = sp.T + x * (N + 1) + L[x];
        const uint32_t t0 = __ldg(Tx);
        u1 += __ldg(Tx + 1) - t0;
        u2 += __ldg(Tx + 2) - t0;
        w.U1[x * rb + r] = u1;
        w.U2[x * rb + r] = u2;
    }
}

// A_m(q, l) of row r: sqrt((n_q + 1)(n_l + 1 + [q = l])) C[rank(m + e_q + e_l)]
__device__ __forceinline__ double2 wide_amp(const SpaceView& sp, const WideRows& w, int rb, int r,
                                            uint32_t row, unsigned short ql,
                                            const double2* __restrict__ C) {
    const int q = ql >> 8, l = ql & 255;
    const uint32_t j = sp.dim - sp.dim2 + row - (w.U1[q * rb + r] - w.U1[l * rb + r]) -
                       w.U2[l * rb + r];
    const double f = __ldg(sp.sq + w.n[q * rb + r] + 1) *
                     __ldg(sp.sq + w.n[l * rb + r] + 1 + (q == l ? 1 : 0));
    return cscale(__ldg(C + j), f);
}

}  // namespace

// the pair matrix W[P][Q] of H (pair_w_entry), one thread per entry; the
// real-W flag stays 0 (no two-product path here)
__global__ void __launch_bounds__(256)
    wide_w_kernel(int N, int M, const double2* __restrict__ hob, const double2* __restrict__ hint,
                  double2* __restrict__ W) {
    const int P = wide_pairs(M);
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < P * P) W[e] = pair_w_entry(N, M, hob, hint, e);
    if (e == P * P) W[e] = make_double2(0.0, 0.0);
}

// Y[p * D2 + m]: ST strips of 16 rows a block (two up to 20 orbitals: two blocks
// fit an SM up to 19; one beyond, where the A tile of two strips takes over
// 118 KB and at 29 orbitals no longer fits).  Warps take the output tiles of
// 8 pairs; a tile's W fragments come from L2 and serve every strip, with four
// real products per complex one (the kernel waits on its gathers and W, not on
// the tensor cores: the three-product form is no faster here).
template <int ST>
__global__ void __launch_bounds__(kWideThreads)
    wide_y_kernel(SpaceView sp, const double2* __restrict__ C, const double2* __restrict__ W,
                  double2* __restrict__ Y, HcEpilogue ep) {
    constexpr int ROWS = 16 * ST;
    extern __shared__ double2 smem[];
    if (ep.flag != nullptr && *ep.flag != 0) return;  // Lanczos breakdown: no-op
    const int M = sp.M, P = wide_pairs(M), PS = wide_ps(P), t = threadIdx.x;
    double2* As = smem;
    const WideRows rows = wide_rows_at(As + ROWS * PS, M, ROWS);
    const uint32_t D2 = sp.dim2, row0 = blockIdx.x * ROWS;
    if (t < ROWS) wide_fill_up(sp, rows, ROWS, t, min(row0 + t, D2 - 1u));
    __syncthreads();
    const int lane = t & 31, warp = t >> 5;
    const int r = t % ROWS;
    for (int p = t / ROWS; p < PS; p += kWideThreads / ROWS)
        As[r * PS + (p ^ wide_swz(r))] =
            p < P ? wide_amp(sp, rows, ROWS, r, min(row0 + r, D2 - 1u), wide_pair(M, p), C)
                  : make_double2(0.0, 0.0);
    __syncthreads();
    const int g = lane >> 2, tq = lane & 3, sw = wide_swz(g);
    const double2 zero = make_double2(0.0, 0.0);
    for (int n = warp; n * 8 < P; n += kWideThreads / 32) {
        double re[ST][4] = {}, im[ST][4] = {};
        const double2* w = W + (size_t)min(n * 8 + g, P - 1) * P;
        const bool pv = n * 8 + g < P;
        for (int k = 0; k < PS; k += 8) {
            const int q = k + tq;
            const double2 b0 = pv && q < P ? __ldg(w + q) : zero;
            const double2 b1 = pv && q + 4 < P ? __ldg(w + q + 4) : zero;
#pragma unroll
            for (int s = 0; s < ST; s++) {
                const double2* r0 = As + (s * 16 + g) * PS;
                const double2* r1 = r0 + 8 * PS;
                const double2 a0 = r0[q ^ sw], a1 = r1[q ^ sw];
                const double2 a2 = r0[(q + 4) ^ sw], a3 = r1[(q + 4) ^ sw];
                dmma1688(re[s], a0.x, a1.x, a2.x, a3.x, b0.x, b1.x);
                dmma1688(im[s], a0.x, a1.x, a2.x, a3.x, b0.y, b1.y);
                dmma1688(re[s], -a0.y, -a1.y, -a2.y, -a3.y, b0.y, b1.y);
                dmma1688(im[s], a0.y, a1.y, a2.y, a3.y, b0.x, b1.x);
            }
        }
#pragma unroll
        for (int s = 0; s < ST; s++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int p = n * 8 + 2 * tq + (j & 1);
                const uint32_t m = row0 + s * 16 + g + (j >> 1) * 8;
                if (p < P && m < D2) Y[(size_t)p * D2 + m] = make_double2(re[s][j], im[s][j]);
            }
    }
}

// (HC)_i gathered back from Y: 64 rows a block, four threads a row (each a
// quarter of the pairs, added in order), then the Lanczos epilogue
__global__ void __launch_bounds__(kWideThreads)
    wide_g_kernel(SpaceView sp, const double2* __restrict__ Y, double2* HC, HcEpilogue ep) {
    extern __shared__ double2 smem[];
    if (ep.flag != nullptr && *ep.flag != 0) return;
    const int M = sp.M, N = sp.N, P = wide_pairs(M), t = threadIdx.x;
    double2* part = smem;  // 4 x kWideGRows
    const WideRows rows = wide_rows_at(part + 4 * kWideGRows, M, kWideGRows);
    const int r = t % kWideGRows, sub = t / kWideGRows;
    double2 alpha = make_double2(0.0, 0.0);
    for (uint32_t row0 = blockIdx.x * kWideGRows; row0 < sp.dim; row0 += gridDim.x * kWideGRows) {
        const uint32_t row = min(row0 + r, sp.dim - 1u);
        if (sub == 0) {
            int L[kMaxOrb];
            wide_unrank(sp, N, sp.dim, row, rows.n + r, kWideGRows, L);
            // suffix sums of T_y(L_y) - T_y(L_y - d); an L_y below d only occurs
            // for y below the orbitals of a pair that cannot be removed
            uint32_t v1 = 0, v2 = 0;
            rows.U1[(M - 1) * kWideGRows + r] = 0u;
            rows.U2[(M - 1) * kWideGRows + r] = 0u;
            for (int x = M - 2; x >= 0; x--) {
                const uint32_t* Tx = sp.T + x * (N + 1);
                const uint32_t t0 = __ldg(Tx + L[x]);
                v1 += t0 - __ldg(Tx + max(L[x] - 1, 0));
                v2 += t0 - __ldg(Tx + max(L[x] - 2, 0));
                rows.U1[x * kWideGRows + r] = v1;
                rows.U2[x * kWideGRows + r] = v2;
            }
        }
        __syncthreads();
        const uint32_t D2 = sp.dim2, base = D2 - sp.dim + row;
        double2 acc = make_double2(0.0, 0.0);
        const int per = (P + 3) / 4, p0 = sub * per, p1 = min(p0 + per, P);
        unsigned short ks = wide_pair(M, min(p0, P - 1));
        int k = ks >> 8, s = ks & 255;
        for (int p = p0; p < p1; p++) {
            const int nk = rows.n[k * kWideGRows + r], ns = rows.n[s * kWideGRows + r] - (k == s);
            if (nk >= 1 && ns >= 1) {
                const double f = __ldg(sp.sq + nk) * __ldg(sp.sq + ns);
                const uint32_t m = base +
                                   (rows.U1[k * kWideGRows + r] - rows.U1[s * kWideGRows + r]) +
                                   rows.U2[s * kWideGRows + r];
                const double2 y = __ldg(Y + (size_t)p * D2 + m);
                acc.x = fma(f, y.x, acc.x);
                acc.y = fma(f, y.y, acc.y);
            }
            if (++s == M) s = ++k;
        }
        part[sub * kWideGRows + r] = acc;
        __syncthreads();
        if (sub == 0 && row0 + r < sp.dim) {
            for (int u = 1; u < 4; u++) acc = cadd(acc, part[u * kWideGRows + r]);
            hc_row_epilogue(ep, row, acc, HC, alpha);
        }
        __syncthreads();
    }
    hc_alpha_epilogue(ep, alpha);
}

// One block's share of a 64 x 64 super-tile (si <= sj) of the Gram matrix:
// row tiles blockIdx.x, blockIdx.x + gridDim.x, ...; warp ti holds the tile
// row ti, eight 8 x 8 complex tiles of four real m8n8k4 products each.
// partial: [super-tile][block][64 x 64]
__global__ void __launch_bounds__(kWideThreads)
    wide_gram_kernel(SpaceView sp, const double2* __restrict__ C, double2* __restrict__ partial) {
    extern __shared__ double2 smem[];
    const int M = sp.M, P = wide_pairs(M), t = threadIdx.x, lane = t & 31, ti = t >> 5;
    double2* As = smem;  // kWideRows x kGramPS: columns of si, then those of sj
    const WideRows rows = wide_rows_at(As + kWideRows * kGramPS, M, kWideRows);
    int si = 0, sj = blockIdx.y;
    const int ns = (P + kSuper - 1) / kSuper;
    while (sj >= ns - si) {
        sj -= ns - si;
        si++;
    }
    sj += si;
    const int off = si == sj ? 0 : kSuper;  // where the columns of sj are
    const uint32_t D2 = sp.dim2, nt = (D2 + kWideRows - 1) / kWideRows;
    const int g = lane >> 2, tq = lane & 3;
    double re[8][2] = {}, im[8][2] = {};
    for (uint32_t tr = blockIdx.x; tr < nt; tr += gridDim.x) {
        const uint32_t row = tr * kWideRows + lane;
        if (t < kWideRows) wide_fill_up(sp, rows, kWideRows, t, min(row, D2 - 1u));
        __syncthreads();
        for (int c = ti; c < kSuper + off; c += kWideThreads / 32) {
            const int p = c < kSuper ? si * kSuper + c : sj * kSuper + c - kSuper;
            As[lane * kGramPS + c] =
                p < P && row < D2 ? wide_amp(sp, rows, kWideRows, lane, row, wide_pair(M, p), C)
                                  : make_double2(0.0, 0.0);
        }
        __syncthreads();
        for (int r0 = 0; r0 < kWideRows; r0 += 4) {
            const double2* x = As + (r0 + tq) * kGramPS;
            const double2 a = x[ti * 8 + g];
            const double na = -a.y;
#pragma unroll
            for (int tj = 0; tj < 8; tj++) {
                const double2 b = x[off + tj * 8 + g];
                wide_dmma884(re[tj], a.x, b.x);
                wide_dmma884(re[tj], a.y, b.y);
                wide_dmma884(im[tj], a.x, b.y);
                wide_dmma884(im[tj], na, b.x);
            }
        }
        __syncthreads();
    }
    double2* out = partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kSuper * kSuper;
#pragma unroll
    for (int tj = 0; tj < 8; tj++)
#pragma unroll
        for (int j = 0; j < 2; j++)
            out[(ti * 8 + g) * kSuper + tj * 8 + 2 * tq + j] = make_double2(re[tj][j], im[tj][j]);
}

// Gram entry (pa <= pb) summed over the block partials, and its fill of rho2
// (as gram_fill): every ordering of a pair reads the same entry, the lower
// triangle is the conjugate, diagonal entries are real.  Eight warps take an
// eighth of the partials of 32 entries each, added in order (one thread an
// entry took 18.8 us at N=8 M=10, 157 partials, against 5.7 us).
__global__ void __launch_bounds__(256)
    wide_fill_kernel(int M, int blocks, const double2* __restrict__ partial,
                     double2* __restrict__ rho2) {
    __shared__ double2 sum[8][32];
    const int P = wide_pairs(M), lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane, pa = min(e, P * P - 1) / P, pb = min(e, P * P - 1) % P;
    const int ns = (P + kSuper - 1) / kSuper, si = pa / kSuper, sj = pb / kSuper;
    double2 v = make_double2(0.0, 0.0);
    if (pa <= pb) {
        const int st = si * ns - si * (si - 1) / 2 + (sj - si);
        const double2* src = partial + (size_t)st * blocks * kSuper * kSuper +
                             (pa % kSuper) * kSuper + pb % kSuper;
        const int per = (blocks + 7) / 8, b1 = min((part + 1) * per, blocks);
        for (int b = part * per; b < b1; b++) v = cadd(v, __ldg(src + (size_t)b * kSuper * kSuper));
    }
    sum[part][lane] = v;
    __syncthreads();
    if (part != 0 || e >= P * P || pa > pb) return;
    for (int u = 1; u < 8; u++) v = cadd(v, sum[u][lane]);
    if (pa == pb) v.y = 0.0;
    const double2 vc = make_double2(v.x, -v.y);
    const unsigned short u = wide_pair(M, pa), w = wide_pair(M, pb);
    const int M2 = M * M, M3 = M2 * M;
    const int ks[2] = {u >> 8, u & 255}, ql[2] = {w >> 8, w & 255};
    for (int a = 0; a < (ks[0] == ks[1] ? 1 : 2); a++)
        for (int b = 0; b < (ql[0] == ql[1] ? 1 : 2); b++) {
            const int k = ks[a], s = ks[1 - a], q = ql[b], l = ql[1 - b];
            rho2[k + s * M + q * M2 + l * M3] = v;
            rho2[q + l * M + k * M2 + s * M3] = vc;
        }
}

// rho1[k][l] = sum_s rho2[k,s,s,l] / (N - 1), s in order (rho1_from_rho2)
__global__ void __launch_bounds__(128)
    wide_rho1_kernel(int N, int M, const double2* __restrict__ rho2, double2* __restrict__ rho1) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x, M2 = M * M;
    if (e >= M2) return;
    const int k = e / M, l = e % M;
    double2 v = make_double2(0.0, 0.0);
    for (int s = 0; s < M; s++) v = cadd(v, __ldg(rho2 + k + s * M + s * M2 + (size_t)l * M2 * M));
    const double d = (double)(N - 1);
    rho1[e] = make_double2(v.x / d, v.y / d);
}

bool wide_eligible(int N, int M) { return N >= 2 && M > kMaxTemplOrb && M <= kMaxOrb; }

constexpr int wide_strips(int M) { return M <= 20 ? 2 : 1; }
static size_t wide_y_smem(int M) {
    const int rows = 16 * wide_strips(M);
    return (size_t)rows * wide_ps(wide_pairs(M)) * sizeof(double2) + wide_rows_bytes(M, rows);
}
static size_t wide_g_smem(int M) {
    return 4 * kWideGRows * sizeof(double2) + wide_rows_bytes(M, kWideGRows);
}
static size_t wide_gram_smem(int M) {
    return (size_t)kWideRows * kGramPS * sizeof(double2) + wide_rows_bytes(M, kWideRows);
}

int wide_prepare() {
    static std::atomic<uint64_t> done{0};
    return set_attributes_once(done, []() -> int {
        const auto kind = cudaFuncAttributeMaxDynamicSharedMemorySize;
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(wide_y_kernel<2>, kind, (int)wide_y_smem(20)));
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(wide_y_kernel<1>, kind, (int)wide_y_smem(kMaxOrb)));
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(wide_g_kernel, kind, (int)wide_g_smem(kMaxOrb)));
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(wide_gram_kernel, kind, (int)wide_gram_smem(kMaxOrb)));
        return 0;
    });
}

int wide_prep(const SpaceView& sp, const double2* hob, const double2* hint, cudaStream_t st) {
    const int P = wide_pairs(sp.M);
    wide_w_kernel<<<(P * P) / 256 + 1, 256, 0, st>>>(sp.N, sp.M, hob, hint, sp.pair_w);
    MCTDHB_CUDA_TRY(cudaGetLastError());
    return 0;
}

int wide_hc(const SpaceView& sp, const double2* C, double2* HC, const HcEpilogue& ep,
            cudaStream_t st) {
    const int rows = 16 * wide_strips(sp.M), gy = (int)((sp.dim2 + rows - 1) / rows);
    const size_t sm = wide_y_smem(sp.M);
    if (rows == 32)
        wide_y_kernel<2><<<gy, kWideThreads, sm, st>>>(sp, C, sp.pair_w, sp.pair_y, ep);
    else
        wide_y_kernel<1><<<gy, kWideThreads, sm, st>>>(sp, C, sp.pair_w, sp.pair_y, ep);
    const int gg = (int)std::min<uint32_t>((sp.dim + kWideGRows - 1) / kWideGRows,
                                           (uint32_t)num_sms() * 8);
    wide_g_kernel<<<gg, kWideThreads, wide_g_smem(sp.M), st>>>(sp, sp.pair_y, HC, ep);
    MCTDHB_CUDA_TRY(cudaGetLastError());
    return 0;
}

// row blocks of a super-tile: a function of (N, M) only, about two blocks an
// SM in all
static int wide_gram_blocks(int M, uint32_t D2) {
    const int ns = (wide_pairs(M) + kSuper - 1) / kSuper, nst = ns * (ns + 1) / 2;
    const uint32_t nt = (D2 + kWideRows - 1) / kWideRows;
    return (int)std::max<uint32_t>(1u, std::min<uint32_t>(nt, (uint32_t)(296 / nst)));
}

size_t wide_gram_elems(int M, uint32_t D2) {
    const int ns = (wide_pairs(M) + kSuper - 1) / kSuper;
    return (size_t)(ns * (ns + 1) / 2) * wide_gram_blocks(M, D2) * kSuper * kSuper;
}

int wide_dens(const SpaceView& sp, uint32_t D2, const double2* C, double2* partial, double2* rho1,
              double2* rho2, cudaStream_t st) {
    const int M = sp.M, P = wide_pairs(M), ns = (P + kSuper - 1) / kSuper;
    SpaceView v = sp;
    v.dim2 = D2;
    const dim3 grid(wide_gram_blocks(M, D2), ns * (ns + 1) / 2);
    wide_gram_kernel<<<grid, kWideThreads, wide_gram_smem(M), st>>>(v, C, partial);
    wide_fill_kernel<<<(P * P + 31) / 32, 256, 0, st>>>(M, grid.x, partial, rho2);
    wide_rho1_kernel<<<(M * M + 127) / 128, 128, 0, st>>>(sp.N, M, rho2, rho1);
    MCTDHB_CUDA_TRY(cudaGetLastError());
    return 0;
}

}  // namespace mctdhb
