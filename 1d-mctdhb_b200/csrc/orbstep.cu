// orbstep.cu -- the orbital side of a step, one cluster of blocks per system
// (orbstep.cuh): eight for one system, 8, 4, 2 or 1 for a slot of the batch
// (batch.h, cluster_blocks).
//
// What bounds it.  The work of a system is small (M=6 on 1024 points: 6 stages
// of 3.6 M FP64 FMAs) and every stage needs the whole previous one, so the
// time is latency: barriers, dependent sums, too few threads.  One block per
// system took 1,980 us at M=6 on 1024 points (RK5 step with Gram-Schmidt and
// matrices), this kernel takes 170 us; alone, the solver's chain of 30 small
// launches took 190 us at M=4 on 256 points and takes 75 us.  The blocks share the
// points and meet at cluster barriers; every sum over the grid is cut into
// pieces of 256 points (64 for g_ksql) that one warp adds, and the pieces are
// added in order, so a value depends on the system alone.  Work taken out: the
// interacting part through the symmetric pairs q <= l with the orbital count
// known at compile time (the runtime-M loops kept the orbitals in local
// memory), g_ksql between unordered pairs (21 instead of 36 rows at M=6) and
// one triangle of it.
#include <cooperative_groups.h>

#include "common.cuh"
#include "moves.cuh"
#include "orbital_dev.cuh"
#include "orbstep.cuh"
#include "small_linalg.cuh"

namespace cg = cooperative_groups;

namespace mctdhb {

namespace {

constexpr int kOrbThreads = 256;
constexpr int kOrbPiece = 256;     // grid points of one warp's sum
constexpr int kOrbPieces = (kBatchMaxGrid + kOrbPiece - 1) / kOrbPiece;
constexpr int kHintPiece = 64;     // grid points of one warp's g_ksql sum

struct OrbShared {
    double2 part[kBatchMaxOrb * kBatchMaxOrb * kOrbPieces];  // pieces of sums, in every block
    double2 a[kBatchMaxOrb * kBatchMaxOrb];  // summed overlaps / h + B
    double2 b[kBatchMaxOrb * kBatchMaxOrb];
    double2 red[2][kOrbThreads / 32];
    unsigned char pq[40], pl[40];  // pair p <-> (q, l), q <= l
};

// blocks, threads and warps of the cluster: constants for the single system,
// B = 0 any number for the batch.  The batch has one instance alone: the
// compiler fuses a b - c d into either of two multiply-adds, and two instances
// need not agree.
template <int B>
struct OrbSize {
    static constexpr int blocks = B, threads = B * kOrbThreads, warps = threads / 32;
};
template <>
struct OrbSize<0> {
    int blocks, threads, warps;
};

template <int B>
struct OrbBlock : OrbSize<B> {
    cg::cluster_group cl = cg::this_cluster();
    OrbShared* sh;
    double2* sQ;  // M x M x P
    int rank, gtid, gwarp, lane;
};

// the piece e of a sum, held by a whole warp (v of lane 0 .. 31 equal), into
// every block's table
template <class O>
__device__ __forceinline__ void put_piece(O& o, int e, double2 v) {
    if (o.lane < o.blocks) o.cl.map_shared_rank(o.sh, o.lane)->part[e] = v;
}

// out[e] = sum of the pieces e * np .. e * np + np - 1, e < n (own block)
template <class O>
__device__ __forceinline__ void add_pieces(O& o, int n, int np, double2* out) {
    for (int e = threadIdx.x; e < n; e += kOrbThreads) {
        double2 v = o.sh->part[e * np];
        for (int c = 1; c < np; c++) v = cadd(v, o.sh->part[e * np + c]);
        out[e] = v;
    }
    __syncthreads();
}

// pieces of <a_s|b_k> (Simpson) for all s, k
template <int M, class O>
__device__ __forceinline__ void overlap_pieces(O& o, const OrbView& ov, const double2* a,
                                               const double2* b) {
    const int G = ov.G, np = (G + kOrbPiece - 1) / kOrbPiece;
    for (int e = o.gwarp; e < M * M * np; e += o.warps) {
        const int s = e / np / M, k = e / np % M, x0 = e % np * kOrbPiece;
        const double2 *pa = a + (size_t)s * G, *pb = b + (size_t)k * G;
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < kOrbPiece / 32; i++) {
            const int x = x0 + i * 32 + o.lane;
            if (x < G) {
                const double2 t = cfma_conj(pa[x], pb[x], make_double2(0.0, 0.0));
                acc.x += ov.w[x] * t.x;
                acc.y += ov.w[x] * t.y;
            }
        }
        put_piece(o, e, warp_sum(acc));
    }
    o.cl.sync();
}

// sum_s conj(f_s) sum_{q <= l} Q[k][s][q l] f_q f_l at one point; Q holds both
// orders of a pair (split_nonlinear_orbitals.c:4-61)
template <int M>
__device__ __forceinline__ double2 interacting(const double2* Qk, const double2 (&f)[M]) {
    double2 red = make_double2(0.0, 0.0);
#pragma unroll
    for (int s = 0; s < M; s++) {
        const double2* q0 = Qk + s * (M * (M + 1) / 2);
        double2 ts = make_double2(0.0, 0.0);
        int p = 0;
#pragma unroll
        for (int q = 0; q < M; q++) {
            double2 tl = make_double2(0.0, 0.0);
#pragma unroll
            for (int l = q; l < M; l++, p++) tl = cfma(q0[p], f[l], tl);
            ts = cfma(tl, f[q], ts);
        }
        red = cfma(make_double2(f[s].x, -f[s].y), ts, red);
    }
    return red;
}

// robust projector (orbital_integration.c:22-92): P <- S^{-1} P with the full
// overlap matrix S_sl = <y_s|y_l> of the stage orbitals; a singular S keeps
// the simple projector's P and flags the system (BF_ROBFAIL)
template <int M, class O>
__device__ void robust(O& o, const BatchSlot& S, const double2* y) {
    o.cl.sync();  // every block has added the pieces of P
    overlap_pieces<M>(o, S.ov, y, y);
    add_pieces(o, M * M, (S.ov.G + kOrbPiece - 1) / kOrbPiece, o.sh->b);
    if (threadIdx.x == 0) {
        double2 inv[M * M], t[M * M];
        if (herm_inverse(M, o.sh->b, inv)) {
            if (o.rank == 0) S.flags[BF_ROBFAIL] = 1;
        } else {
            for (int a = 0; a < M; a++)
                for (int k = 0; k < M; k++) {
                    double2 z = make_double2(0.0, 0.0);
                    for (int l = 0; l < M; l++)
                        z = cfma(inv[a * M + l], o.sh->a[l * M + k], z);
                    t[a * M + k] = z;
                }
            for (int i = 0; i < M * M; i++) o.sh->a[i] = t[i];
        }
    }
    __syncthreads();
}

// Runge-Kutta tableaux: Heun (2), classical RK4 (4), Butcher RK5 (5); row j
// gives the input of stage j, the last row the step
struct Tableau {
    int stages;
    double c[7][6];
};
__constant__ Tableau kTableaux[3] = {
    {2, {{0}, {1.0}, {0.5, 0.5}}},
    {4, {{0}, {0.5}, {0, 0.5}, {0, 0, 1.0}, {1.0 / 6, 2.0 / 6, 2.0 / 6, 1.0 / 6}}},
    {6,
     {{0},
      {0.25},
      {0.125, 0.125},
      {0, -0.5, 1.0},
      {3.0 / 16, 0, 0, 9.0 / 16},
      {-3.0 / 7, 2.0 / 7, 12.0 / 7, -12.0 / 7, 8.0 / 7},
      {7.0 / 90, 0, 32.0 / 90, 12.0 / 90, 32.0 / 90, 7.0 / 90}}}};

// Runge-Kutta step of the orbitals in place (orbital_integration.c:284-349;
// split: of the nonlinear part alone, :387-415).  A thread owns points (k, x)
// and with them the stage values there (stage[0..4]; the last is not kept);
// the inputs of the stages alternate between stage[5] and stage[6], H phi is
// in S.H.
template <int M, class O>
__device__ void rk_step(O& o, const BatchSlot& S) {
    const OrbView& ov = S.ov;
    constexpr int P = M * (M + 1) / 2;
    const int G = ov.G, n = M * G, np = (G + kOrbPiece - 1) / kOrbPiece;
    const Tableau& tab = kTableaux[S.rk == 2 ? 0 : S.rk == 4 ? 1 : 2];
    const double2 mi_tf = make_double2(ov.tf.y, -ov.tf.x);
    double2 *y = S.orb, *H = S.H;
    const bool rob = S.flags[BF_ROBUST] != 0;
    const double2* in = y;
    for (int j = 0; j < tab.stages; j++) {
        const double* c = tab.c[j + 1];
        const bool last = j + 1 == tab.stages;
        double2* w = S.stage + (size_t)(5 + (j & 1)) * n;
        // the stage value kv at point t, then the next stage's input there
        auto advance = [&](int t, double2 kv) {
            double2 s = make_double2(0.0, 0.0);
            for (int q = 0; q < j; q++)
                if (c[q] != 0.0) {
                    const double2 v = S.stage[(size_t)q * n + t];
                    s.x += c[q] * v.x;
                    s.y += c[q] * v.y;
                }
            s.x += c[j] * kv.x;
            s.y += c[j] * kv.y;
            const double2 y0 = y[t], r = make_double2(y0.x + S.dt * s.x, y0.y + S.dt * s.y);
            if (!last) {
                S.stage[(size_t)j * n + t] = kv;
                w[t] = r;
            } else {
                y[t] = r;
                if (S.orb_next) S.orb_next[t] = r;
            }
        };
        for (int t = o.gtid; t < n; t += o.threads) {
            const int k = t / G, x = t - k * G;
            const double2* fk = in + (size_t)k * G;
            double2 f[M];
#pragma unroll
            for (int a = 0; a < M; a++) f[a] = in[(size_t)a * G + x];
            double2 red = interacting<M>(o.sQ + k * M * P, f);
            if (S.split) {
#pragma unroll
                for (int a = 0; a < M; a++) {
                    const double2 hb = o.sh->a[k * M + a];  // h[a][k] + B[k][a]
                    red.x -= hb.x * f[a].x - hb.y * f[a].y;
                    red.y -= hb.x * f[a].y + hb.y * f[a].x;
                }
                advance(t, cmul(mi_tf, cadd(red, cscale(fk[x], ov.pot[x]))));
            } else {
                H[t] = cadd(red, ov.lin_t ? toeplitz_at(ov, fk, x) : linear_at(ov, fk, x));
            }
        }
        o.cl.sync();
        if (!S.split) {
            overlap_pieces<M>(o, ov, in, H);
            add_pieces(o, M * M, np, o.sh->a);
            if (rob) robust<M>(o, S, in);
            for (int t = o.gtid; t < n; t += o.threads) {
                const int k = t / G, x = t - k * G;
                double2 proj = make_double2(0.0, 0.0);
#pragma unroll
                for (int s = 0; s < M; s++)
                    proj = cfma(in[(size_t)s * G + x], o.sh->a[s * M + k], proj);
                advance(t, cmul(mi_tf, make_double2(H[t].x - proj.x, H[t].y - proj.y)));
            }
            o.cl.sync();
        }
        in = w;
    }
}

// linear half step of the split step, y <- Op y (orb_operator_kernel), through
// stage[6]
template <class O>
__device__ void half_step(O& o, const BatchSlot& S, double2* y) {
    const int M = S.ov.M, G = S.ov.G, n = M * G;
    const int dense = S.half_dense, nn = dense ? G : G - 1;
    double2* w = S.stage + (size_t)6 * n;
    for (int t = o.gtid; t < n; t += o.threads) {
        const int k = t / G, x = t - k * G;
        const double2* f = y + (size_t)k * G;
        double2 acc = make_double2(0.0, 0.0);
        if (dense) {
            for (int j = 0; j < nn; j++) acc = cfma(S.half[(size_t)j * G + x], f[j], acc);
        } else {
            const double2* tk = S.half + (nn - 1 - (x == nn ? 0 : x));
            for (int j = 0; j < nn; j++) acc = cfma(tk[j], f[j], acc);
        }
        w[t] = acc;
    }
    o.cl.sync();
    for (int t = o.gtid; t < n; t += o.threads) y[t] = w[t];
    o.cl.sync();
}

// h[j][k] + B[k][j] into sh->a[k M + j], B[k][j] = sum_a rinv[k][a]
// sum_{s,q,l} rho2[a + sM + qM^2 + lM^3] hint[j + sM + lM^2 + qM^3]
// (split_nonlinear_orbitals.c:63-160): one warp per (a, j)
template <int M, class O>
__device__ void bmat(O& o, const BatchSlot& S) {
    constexpr int M2 = M * M, M3 = M2 * M;
    for (int e = o.gwarp; e < M2; e += o.warps) {
        const int a = e / M, j = e % M;
        double2 acc = make_double2(0.0, 0.0);
        for (int c = o.lane; c < M3; c += 32) {
            const int s = c % M, q = c / M % M, l = c / M2;
            acc = cfma(S.rho2[a + s * M + q * M2 + l * M3], S.hint[j + s * M + l * M2 + q * M3],
                       acc);
        }
        put_piece(o, e, warp_sum(acc));
    }
    o.cl.sync();
    for (int e = threadIdx.x; e < M2; e += kOrbThreads) {
        const int k = e / M, j = e % M;
        double2 acc = S.hob[j * M + k];
        for (int a = 0; a < M; a++) acc = cfma(S.rinv[k * M + a], o.sh->part[a * M + j], acc);
        o.sh->a[e] = acc;
    }
    __syncthreads();
}

// orthonormalize (calculus.c:171-191) by one block.  The reference
// re-evaluates <F_j|F_i> for every grid point k while F_i is being updated;
// that overlap obeys ov_{k+1} = ov_k (1 - w_k |F_j[k]|^2), so the update is a
// prefix product, which depends on F_j alone: formed once per orbital by a
// block scan and kept in S.H.  A thread owns E consecutive points.
template <int E, class O>
__device__ void gram_schmidt(O& o, const BatchSlot& S) {
    const OrbView& ov = S.ov;
    const int M = ov.M, G = ov.G, x0 = threadIdx.x * E, warp = threadIdx.x >> 5;
    double* scan = (double*)S.H;  // M x G
    int turn = 0;
    auto total = [&](double2 v) {  // every thread gets the block sum
        double2* red = o.sh->red[turn];
        turn ^= 1;
        v = warp_sum(v);
        if (o.lane == 0) red[warp] = v;
        __syncthreads();
        double2 s = red[0];
#pragma unroll
        for (int i = 1; i < kOrbThreads / 32; i++) s = cadd(s, red[i]);
        return s;
    };
    for (int i = 0; i < M; i++) {
        double2 f[E];
        double w[E];
#pragma unroll
        for (int u = 0; u < E; u++) {
            f[u] = x0 + u < G ? S.orb[(size_t)i * G + x0 + u] : make_double2(0.0, 0.0);
            w[u] = x0 + u < G ? ov.w[x0 + u] : 0.0;
        }
        for (int j = 0; j < i; j++) {
            const double2* fj = S.orb + (size_t)j * G + x0;
            const double* sj = scan + (size_t)j * G + x0;
            double2 g[E], acc = make_double2(0.0, 0.0);
            double sc[E];
#pragma unroll
            for (int u = 0; u < E; u++) {
                g[u] = x0 + u < G ? fj[u] : make_double2(0.0, 0.0);
                sc[u] = x0 + u < G ? sj[u] : 0.0;
                const double2 t = cfma_conj(g[u], f[u], make_double2(0.0, 0.0));
                acc.x += w[u] * t.x;
                acc.y += w[u] * t.y;
            }
            const double2 over = total(acc);
#pragma unroll
            for (int u = 0; u < E; u++) {
                const double2 t = cmul(cscale(over, sc[u]), g[u]);
                f[u].x -= t.x;
                f[u].y -= t.y;
            }
        }
        double nrm = 0.0;
#pragma unroll
        for (int u = 0; u < E; u++) nrm += w[u] * (f[u].x * f[u].x + f[u].y * f[u].y);
        const double r = sqrt(1.0 / total(make_double2(nrm, 0.0)).x);
        double run = 1.0, before[E];
#pragma unroll
        for (int u = 0; u < E; u++) {
            f[u] = cscale(f[u], r);
            before[u] = run;
            run *= 1.0 - w[u] * (f[u].x * f[u].x + f[u].y * f[u].y);
        }
        // exclusive prefix product of the threads' factors over the block
        double incl = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, d);
            if (o.lane >= d) incl *= v;
        }
        double excl = __shfl_up_sync(0xffffffffu, incl, 1);
        if (o.lane == 0) excl = 1.0;
        double2* red = o.sh->red[turn];
        turn ^= 1;
        if (o.lane == 31) red[warp].x = incl;
        __syncthreads();
        for (int q = 0; q < warp; q++) excl *= red[q].x;
#pragma unroll
        for (int u = 0; u < E; u++)
            if (x0 + u < G) {
                S.orb[(size_t)i * G + x0 + u] = f[u];
                scan[(size_t)i * G + x0 + u] = excl * before[u];
            }
    }
}

// h_kl (orbital_matrices.c:22-70) and g_ksql (:73-287) of the orbitals
template <int M, class O>
__device__ void matrices(O& o, const BatchSlot& S) {
    constexpr int P = M * (M + 1) / 2, M2 = M * M, NT = (P + 7) / 8, TILES = NT * (NT + 1) / 2;
    const OrbView& ov = S.ov;
    const int G = ov.G, np = (G + kOrbPiece - 1) / kOrbPiece;
    const int hp = (G + kHintPiece - 1) / kHintPiece;
    const double r = 1.0 / (12 * ov.dx), g = *S.g;
    // g_ksql = g sum_x w conj(f_k f_s) f_q f_l between the pairs (k <= s) and
    // (q <= l): 8 x 8 tiles of the upper triangle, m8n8k4 products over one
    // piece of the grid per warp.  More than one piece: into the stage
    // buffers, free outside the Runge-Kutta step.
    auto fill = [&](int pr, int pc, double2 v) {
        if (pr > pc) return;
        v = make_double2(g * v.x, pr == pc ? 0.0 : g * v.y);
        const double2 vc = make_double2(v.x, -v.y);
        const int a[2] = {o.sh->pq[pr], o.sh->pl[pr]}, c[2] = {o.sh->pq[pc], o.sh->pl[pc]};
        for (int u = 0; u < (a[0] == a[1] ? 1 : 2); u++)
            for (int z = 0; z < (c[0] == c[1] ? 1 : 2); z++) {
                const int row = a[u] + a[1 - u] * M, col = c[z] + c[1 - z] * M;
                S.hint[row + M2 * col] = v;
                S.hint[col + M2 * row] = vc;
            }
    };
    const int gr = o.lane >> 2, kk = o.lane & 3;
    for (int task = o.gwarp; task < TILES * hp; task += o.warps) {
        const int tile = task / hp, piece = task % hp;
        int ti = 0, tj = tile;
        while (tj >= NT - ti) {
            tj -= NT - ti;
            ti++;
        }
        tj += ti;
        const int pa = ti * 8 + gr, pb = tj * 8 + gr;
        const bool av = pa < P, bv = pb < P;
        const double2* a1 = S.orb + (size_t)o.sh->pq[av ? pa : 0] * G;
        const double2* a2 = S.orb + (size_t)o.sh->pl[av ? pa : 0] * G;
        const double2* b1 = S.orb + (size_t)o.sh->pq[bv ? pb : 0] * G;
        const double2* b2 = S.orb + (size_t)o.sh->pl[bv ? pb : 0] * G;
        double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
#pragma unroll 4
        for (int i = 0; i < kHintPiece / 4; i++) {
            const int x = piece * kHintPiece + i * 4 + kk;
            const bool in = x < G;
            const int xc = in ? x : 0;
            const double2 pA = cmul(a1[xc], a2[xc]), pB = cmul(b1[xc], b2[xc]);
            const double wx = in ? ov.w[xc] : 0.0, wa = av ? wx : 0.0, wb = bv && in ? 1.0 : 0.0;
            const double ar = wa * pA.x, ai = wa * pA.y, br = wb * pB.x, bi = wb * pB.y;
            dmma(re[0], re[1], ar, br);  // conj(A) B
            dmma(re[0], re[1], ai, bi);
            dmma(im[0], im[1], ar, bi);
            dmma(im[0], im[1], -ai, br);
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int c = 2 * kk + j;
            const double2 v = make_double2(re[j], im[j]);
            if (hp == 1) {
                if (ti * 8 + gr < P && tj * 8 + c < P) fill(ti * 8 + gr, tj * 8 + c, v);
            } else {
                S.stage[(size_t)task * 64 + gr * 8 + c] = v;
            }
        }
    }
    for (int e = o.gwarp; e < P * np; e += o.warps) {
        const int p = e / np, x0 = e % np * kOrbPiece;
        const double2* fk = S.orb + (size_t)o.sh->pq[p] * G;
        const double2* fl = S.orb + (size_t)o.sh->pl[p] * G;
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll 2
        for (int i = 0; i < kOrbPiece / 32; i++) {
            const int x = x0 + i * 32 + o.lane;
            if (x < G) {
                const double2 t = hob_integrand(ov, fk, fl, x, r);
                acc.x += ov.w[x] * t.x;
                acc.y += ov.w[x] * t.y;
            }
        }
        put_piece(o, e, warp_sum(acc));
    }
    o.cl.sync();
    if (hp > 1)
        for (int e = o.gtid; e < TILES * 64; e += o.threads) {
            const int tile = e >> 6, cell = e & 63;
            int ti = 0, tj = tile;
            while (tj >= NT - ti) {
                tj -= NT - ti;
                ti++;
            }
            tj += ti;
            const int pr = ti * 8 + (cell >> 3), pc = tj * 8 + (cell & 7);
            if (pr >= P || pc >= P || pr > pc) continue;
            double2 v = S.stage[(size_t)tile * hp * 64 + cell];
            for (int c = 1; c < hp; c++) v = cadd(v, S.stage[(size_t)(tile * hp + c) * 64 + cell]);
            fill(pr, pc, v);
        }
    if (o.rank == o.blocks - 1)
        for (int p = threadIdx.x; p < P; p += kOrbThreads) {
            double2 v = o.sh->part[p * np];
            for (int c = 1; c < np; c++) v = cadd(v, o.sh->part[p * np + c]);
            const int k = o.sh->pq[p], l = o.sh->pl[p];
            if (k == l) v.y = 0.0;
            S.hob[k * M + l] = v;
            if (k != l) S.hob[l * M + k] = make_double2(v.x, -v.y);
        }
    o.cl.sync();
}

template <int M, class O>
__device__ void run_step(O& o, const BatchSlot& S, int parts) {
    constexpr int P = M * (M + 1) / 2, M2 = M * M, M3 = M2 * M;
    const OrbView& ov = S.ov;
    const int G = ov.G, np = (G + kOrbPiece - 1) / kOrbPiece;
    for (int p = threadIdx.x; p < P; p += kOrbThreads) {
        int q = 0, r = p;
        while (r >= M - q) {
            r -= M - q;
            q++;
        }
        o.sh->pq[p] = q;
        o.sh->pl[p] = q + r;
    }
    __syncthreads();
    auto periodic = [&]() {
        if (ov.periodic && o.rank == 0 && threadIdx.x < M)
            S.orb[(size_t)threadIdx.x * G + G - 1] = S.orb[(size_t)threadIdx.x * G];
        o.cl.sync();
    };
    if (parts & kOrbPeriodic) periodic();
    if (parts & kOrbRk) {
        // Q[k][s][q l] = g sum_a rinv[k][a] (rho2[a, s, q, l] + rho2[a, s, l, q])
        const double g = *S.g;
        for (int e = threadIdx.x; e < M2 * P; e += kOrbThreads) {
            const int k = e / (M * P), s = e / P % M, q = o.sh->pq[e % P], l = o.sh->pl[e % P];
            double2 acc = make_double2(0.0, 0.0);
#pragma unroll
            for (int a = 0; a < M; a++) {
                double2 t = S.rho2[a + s * M + q * M2 + l * M3];
                if (q != l) t = cadd(t, S.rho2[a + s * M + l * M2 + q * M3]);
                acc = cfma(S.rinv[k * M + a], t, acc);
            }
            o.sQ[e] = cscale(acc, g);
        }
        __syncthreads();
        if (S.split) {
            // orbital_integration.c:352-434: half step, h and g of the
            // half-stepped orbitals, B, RK of the nonlinear part, half step
            if (parts & kOrbHalf) half_step(o, S, S.orb);
            matrices<M>(o, S);
            bmat<M>(o, S);
        }
        rk_step<M>(o, S);
        if (S.split && (parts & kOrbHalf)) half_step(o, S, S.orb);
    }
    if ((parts & kOrbGs) && S.imag) {
        if (o.rank == 0) {
            if (G <= kOrbThreads)
                gram_schmidt<1>(o, S);
            else if (G <= 2 * kOrbThreads)
                gram_schmidt<2>(o, S);
            else if (G <= 4 * kOrbThreads)
                gram_schmidt<4>(o, S);
            else if (G <= 8 * kOrbThreads)
                gram_schmidt<8>(o, S);
            else
                gram_schmidt<kBatchMaxGrid / kOrbThreads>(o, S);
        }
        o.cl.sync();
    }
    if (parts & kOrbPost) {
        periodic();
        if (!S.imag) {
            // overlap residual sum_{k<l} |<f_k|f_l>| / M (integrator_monitor.c:
            // 31-42), summed in the reference's (k, l) order, for the monitor
            overlap_pieces<M>(o, ov, S.orb, S.orb);
            add_pieces(o, M2, np, o.sh->b);
            if (o.rank == 0 && threadIdx.x == 0) {
                double sum = 0.0;
                for (int k = 0; k < M; k++)
                    for (int l = k + 1; l < M; l++)
                        sum += hypot(o.sh->b[k * M + l].x, o.sh->b[k * M + l].y);
                S.scal[BS_MISC + 5] = make_double2(sum / M, 0.0);
            }
            o.cl.sync();  // every block has added its pieces
        }
    }
    if (!(parts & kOrbMatrices)) return;
    matrices<M>(o, S);
    if (o.rank != 0 || S.sp.pair_w == nullptr) return;
    // the pair matrix of H.C for the new h and g, and its real flag
    // (pairhc_tmpl.cuh)
    bool real = true;
    for (int e = threadIdx.x; e < P * P; e += kOrbThreads) {
        const int a = e / P, b = e % P;
        const double2 w = pair_w_of(S.N, M, S.hob, S.hint, o.sh->pq[a], o.sh->pl[a], o.sh->pq[b],
                                    o.sh->pl[b]);
        real = real && w.y == 0.0;
        S.sp.pair_w[e] = w;
    }
    real = __syncthreads_and(real);
    if (threadIdx.x == 0) {
        S.sp.pair_w[P * P] = make_double2(real ? 1.0 : 0.0, 0.0);
        // Lanczos set-up of this step (multiconfig_lanczos.c:30-41)
        S.flags[BF_BREAK] = 0;
        S.flags[BF_ITERS] = S.lz;
        S.flags[BF_QL] = 0;
        S.scal[BS_MISC + 0] = make_double2(0.0, 0.0);
        S.scal[BS_OFFD + S.lz - 1] = make_double2(0.0, 0.0);
    }
}

constexpr size_t orb_step_smem() {
    return sizeof(OrbShared) +
           (size_t)kBatchMaxOrb * kBatchMaxOrb * (kBatchMaxOrb * (kBatchMaxOrb + 1) / 2) *
               sizeof(double2);
}

}  // namespace

template <int B>
__global__ void __launch_bounds__(kOrbThreads)
    orb_step_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                    const int* __restrict__ nlist, int parts, int* __restrict__ mon) {
    // a new step: no monitor H.C due yet in any orbital count
    if (mon != nullptr && blockIdx.x == 0 && threadIdx.x < kBatchNumM) mon[threadIdx.x] = 0;
    OrbBlock<B> o;
    if constexpr (B == 0) {
        o.blocks = (int)o.cl.num_blocks();
        o.threads = o.blocks * kOrbThreads;
        o.warps = o.threads / 32;
    }
    const int s = blockIdx.x / o.blocks;
    if (s >= *nlist) return;  // the same in every block of the cluster
    const BatchSlot& S = slots[list[s]];
    if (S.flags[BF_STATE] != SLOT_RUNNING) return;
    extern __shared__ __align__(16) unsigned char mem[];
    o.sh = (OrbShared*)mem;
    o.sQ = (double2*)(mem + sizeof(OrbShared));
    o.rank = (int)o.cl.block_rank();
    o.gtid = o.rank * kOrbThreads + threadIdx.x;
    o.gwarp = o.gtid >> 5;
    o.lane = threadIdx.x & 31;
    o.cl.sync();  // every block of the cluster runs before another writes to its tables
    switch (S.M) {
        case 2: run_step<2>(o, S, parts); break;
        case 3: run_step<3>(o, S, parts); break;
        case 4: run_step<4>(o, S, parts); break;
        case 5: run_step<5>(o, S, parts); break;
        case 6: run_step<6>(o, S, parts); break;
        case 7: run_step<7>(o, S, parts); break;
        case 8: run_step<8>(o, S, parts); break;
    }
}

template <int B>
static int orb_step_attributes() {
    static std::atomic<uint64_t> done{0};
    return set_attributes_once(done, []() -> int {
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(orb_step_kernel<B>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)orb_step_smem()));
        return 0;
    });
}
int orb_step_prepare(bool batch) {
    return batch ? orb_step_attributes<0>() : orb_step_attributes<kClusterMax>();
}

int orb_step_waves(int (&at)[kClusterSizes]) {
    return cluster_waves(orb_step_kernel<0>, kOrbThreads, orb_step_smem(), at);
}

int orb_step_launch(const BatchSlot* slots, const int* list, const int* nlist, int nslots,
                    int parts, int* mon, int blocks, cudaStream_t st) {
    const int size = blocks > 0 ? blocks : kClusterMax;
    ClusterLaunch c(nslots * size, kOrbThreads, orb_step_smem(), size, st);
    auto* kernel = blocks > 0 ? orb_step_kernel<0> : orb_step_kernel<kClusterMax>;
    MCTDHB_CUDA_TRY(cudaLaunchKernelEx(&c.cfg, kernel, slots, list, nlist, parts, mon));
    return 0;
}

}  // namespace mctdhb
