// small_linalg.cuh -- dense M x M complex128 kernels (M <= 30) used by the
// density-matrix synchronisation (synchronize.c:42-57 of the reference,
// which calls LAPACK zheev / zhesv through lapack_interface.c:61-163):
//   * Hermitian eigen-decomposition by cyclic Jacobi rotations,
//   * Hermitian inverse by Gauss-Jordan elimination with partial pivoting,
//   * the regularisation A += x exp(-A / x) (lapack_interface.c:126);
// and the real symmetric tridiagonal eigenproblem of the Lanczos step (in
// place of LAPACK dstev, multiconfig_lanczos.c:143).
// Row-major double2 storage; usable from host code and from one device
// thread.  Results agree with LAPACK to rounding for the well-conditioned
// one-body density matrices these are applied to.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace mctdhb {

__host__ __device__ inline double2 c_mul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ inline double2 c_conj(double2 a) { return make_double2(a.x, -a.y); }
__host__ __device__ inline double c_abs(double2 a) { return hypot(a.x, a.y); }

// Eigenvalues ascending in w[n]; eigenvectors in the columns of v (row-major,
// may be null).  `a` is overwritten.  Returns the sweeps used (<= 100).
__host__ __device__ inline int herm_eig_jacobi(int n, double2* a, double* w, double2* v) {
    if (v)
        for (int i = 0; i < n * n; i++) v[i] = make_double2((i / n == i % n) ? 1.0 : 0.0, 0.0);
    int sweep = 0;
    for (; sweep < 100; sweep++) {
        double off = 0.0, tot = 0.0;
        for (int p = 0; p < n; p++)
            for (int q = 0; q < n; q++) {
                const double m2 = a[p * n + q].x * a[p * n + q].x + a[p * n + q].y * a[p * n + q].y;
                tot += m2;
                if (p != q) off += m2;
            }
        if (off == 0.0 || off <= 1e-30 * tot) break;
        for (int p = 0; p < n - 1; p++)
            for (int q = p + 1; q < n; q++) {
                const double2 apq = a[p * n + q];
                const double mag = c_abs(apq);
                if (mag == 0.0) continue;
                const double2 ph = make_double2(apq.x / mag, apq.y / mag);
                const double theta = 0.5 * atan2(2.0 * mag, a[q * n + q].x - a[p * n + p].x);
                const double c = cos(theta), s = sin(theta);
                // A <- J^H A J, J = [[c, s ph], [-s conj(ph), c]] in the (p, q) plane
                for (int k = 0; k < n; k++) {
                    const double2 akp = a[k * n + p], akq = a[k * n + q];
                    const double2 t1 = c_mul(c_conj(ph), akq), t2 = c_mul(ph, akp);
                    a[k * n + p] = make_double2(c * akp.x - s * t1.x, c * akp.y - s * t1.y);
                    a[k * n + q] = make_double2(s * t2.x + c * akq.x, s * t2.y + c * akq.y);
                }
                for (int k = 0; k < n; k++) {
                    const double2 apk = a[p * n + k], aqk = a[q * n + k];
                    const double2 t1 = c_mul(ph, aqk), t2 = c_mul(c_conj(ph), apk);
                    a[p * n + k] = make_double2(c * apk.x - s * t1.x, c * apk.y - s * t1.y);
                    a[q * n + k] = make_double2(s * t2.x + c * aqk.x, s * t2.y + c * aqk.y);
                }
                if (v)
                    for (int k = 0; k < n; k++) {
                        const double2 vkp = v[k * n + p], vkq = v[k * n + q];
                        const double2 t1 = c_mul(c_conj(ph), vkq), t2 = c_mul(ph, vkp);
                        v[k * n + p] = make_double2(c * vkp.x - s * t1.x, c * vkp.y - s * t1.y);
                        v[k * n + q] = make_double2(s * t2.x + c * vkq.x, s * t2.y + c * vkq.y);
                    }
            }
    }
    // selection sort ascending, permuting eigenvector columns
    for (int i = 0; i < n; i++) w[i] = a[i * n + i].x;
    for (int i = 0; i < n; i++) {
        int best = i;
        for (int j = i + 1; j < n; j++)
            if (w[j] < w[best]) best = j;
        if (best != i) {
            const double t = w[i];
            w[i] = w[best];
            w[best] = t;
            if (v)
                for (int k = 0; k < n; k++) {
                    const double2 u = v[k * n + i];
                    v[k * n + i] = v[k * n + best];
                    v[k * n + best] = u;
                }
        }
    }
    return sweep;
}

// inv = A^{-1}; `a` is overwritten.  Returns 0, or k+1 when column k has no
// non-zero pivot (singular).
__host__ __device__ inline int herm_inverse(int n, double2* a, double2* inv) {
    for (int i = 0; i < n * n; i++) inv[i] = make_double2((i / n == i % n) ? 1.0 : 0.0, 0.0);
    for (int c = 0; c < n; c++) {
        int piv = c;
        double best = c_abs(a[c * n + c]);
        for (int r = c + 1; r < n; r++) {
            const double v = c_abs(a[r * n + c]);
            if (v > best) {
                best = v;
                piv = r;
            }
        }
        if (best == 0.0) return c + 1;
        if (piv != c)
            for (int k = 0; k < n; k++) {
                double2 t = a[c * n + k];
                a[c * n + k] = a[piv * n + k];
                a[piv * n + k] = t;
                t = inv[c * n + k];
                inv[c * n + k] = inv[piv * n + k];
                inv[piv * n + k] = t;
            }
        const double2 d = a[c * n + c];
        const double dd = d.x * d.x + d.y * d.y;
        const double2 r = make_double2(d.x / dd, -d.y / dd);
        for (int k = 0; k < n; k++) {
            a[c * n + k] = c_mul(a[c * n + k], r);
            inv[c * n + k] = c_mul(inv[c * n + k], r);
        }
        for (int row = 0; row < n; row++) {
            if (row == c) continue;
            const double2 f = a[row * n + c];
            if (f.x == 0.0 && f.y == 0.0) continue;
            for (int k = 0; k < n; k++) {
                const double2 t1 = c_mul(f, a[c * n + k]), t2 = c_mul(f, inv[c * n + k]);
                a[row * n + k].x -= t1.x;
                a[row * n + k].y -= t1.y;
                inv[row * n + k].x -= t2.x;
                inv[row * n + k].y -= t2.y;
            }
        }
    }
    return 0;
}

// rho1 <- regularised rho1 and rinv = rho1^{-1} following synchronize.c:42-57:
// if lambda_min / lambda_max < reg_fac, add x exp(-rho1 / x) with
// x = lambda_max reg_fac (lapack_interface.c:126-163).  `work` holds 3 n^2
// double2 and n doubles.  Returns 0, or the inverse's error code.
__host__ __device__ inline int sync_rho1(int n, double2* rho1, double2* rinv, double reg_fac,
                                         double2* work, double* wd) {
    double2* a = work;
    double2* v = work + n * n;
    for (int i = 0; i < n * n; i++) a[i] = rho1[i];
    herm_eig_jacobi(n, a, wd, v);
    if (wd[0] / wd[n - 1] < reg_fac) {
        const double x = wd[n - 1] * reg_fac;
        for (int i = 0; i < n; i++)
            for (int j = 0; j < n; j++) {
                double2 z = make_double2(0.0, 0.0);
                for (int k = 0; k < n; k++) {
                    const double f = x * exp(-wd[k] / x);
                    const double2 t = c_mul(v[i * n + k], c_conj(v[j * n + k]));
                    z.x += f * t.x;
                    z.y += f * t.y;
                }
                rho1[i * n + j].x += z.x;
                rho1[i * n + j].y += z.y;
            }
    }
    for (int i = 0; i < n * n; i++) a[i] = rho1[i];
    return herm_inverse(n, a, rinv);
}

#ifdef __CUDACC__
// The same synchronisation by one warp (all 32 lanes call it; rho1, rinv and
// work, 3 n^2 double2, in shared memory or any memory the warp shares).
//
// One thread spent most of its time in the eigenvalues, which only decide
// whether to regularise.  For a positive definite rho1 (the pivots of its LDL^H
// factors are positive) lambda_min >= 1 / |rho1^{-1}|_F and lambda_max <=
// trace, so where 1 / (|rho1^{-1}|_F trace) is above the threshold with a
// factor of 2 to spare the inverse of rho1 as it is is the answer; only
// otherwise the eigenvalues are formed: the n / 2 disjoint rotations of a
// round-robin Jacobi sweep at once, an element of a rotation or of an
// elimination step per lane.  137 us at n = 4 and 177 us at n = 6 by one
// thread, 12 us by the warp.
__device__ inline double warp_max_f64(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ inline double warp_sum_f64(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Hermitian eigen-decomposition: eigenvalues on the diagonal of a,
// eigenvectors in the columns of v.  rot: n / 2 + 1 rotations.
struct WarpRotation {
    double c, s;
    double2 ph;
};
__device__ inline void herm_eig_warp(int n, double2* a, double2* v, WarpRotation* rot) {
    const int lane = threadIdx.x & 31, ne = n + (n & 1), np = ne / 2;
    for (int i = lane; i < n * n; i += 32) v[i] = make_double2((i / n == i % n) ? 1.0 : 0.0, 0.0);
    __syncwarp();
    if (n < 2) return;
    for (int sweep = 0; sweep < 100; sweep++) {
        double off = 0.0, tot = 0.0;
        for (int i = lane; i < n * n; i += 32) {
            const double m2 = a[i].x * a[i].x + a[i].y * a[i].y;
            tot += m2;
            if (i / n != i % n) off += m2;
        }
        off = warp_sum_f64(off);
        tot = warp_sum_f64(tot);
        if (off == 0.0 || off <= 1e-30 * tot) break;
        for (int r = 0; r < ne - 1; r++) {
            // round-robin pairs: ne - 1 stays, the others turn
            auto pair = [&](int i, int& p, int& q) {
                p = i == 0 ? ne - 1 : (r + i) % (ne - 1);
                q = (r + ne - 1 - i) % (ne - 1);
                if (p > q) {
                    const int t = p;
                    p = q;
                    q = t;
                }
            };
            __syncwarp();
            if (lane < np) {
                int p, q;
                pair(lane, p, q);
                WarpRotation w{1.0, 0.0, make_double2(1.0, 0.0)};
                if (q < n) {
                    const double2 apq = a[p * n + q];
                    const double mag = sqrt(apq.x * apq.x + apq.y * apq.y);
                    if (mag > 0.0) {
                        const double im = 1.0 / mag;
                        w.ph = make_double2(apq.x * im, apq.y * im);
                        const double tau = 0.5 * im * (a[q * n + q].x - a[p * n + p].x);
                        const double t = (tau >= 0.0 ? 1.0 : -1.0) /
                                         (fabs(tau) + sqrt(1.0 + tau * tau));
                        w.c = 1.0 / sqrt(1.0 + t * t);
                        w.s = t * w.c;
                    }
                }
                rot[lane] = w;
            }
            __syncwarp();
            // A <- J^H A J, J = [[c, s ph], [-s conj(ph), c]] in the (p, q)
            // planes: columns of A and V, then rows of A
            for (int e = lane; e < np * n; e += 32) {
                int p, q;
                pair(e / n, p, q);
                if (q >= n) continue;
                const int k = e % n;
                const WarpRotation w = rot[e / n];
                for (int m = 0; m < 2; m++) {
                    double2* x = m == 0 ? a : v;
                    const double2 xp = x[k * n + p], xq = x[k * n + q];
                    const double2 t1 = c_mul(c_conj(w.ph), xq), t2 = c_mul(w.ph, xp);
                    x[k * n + p] = make_double2(w.c * xp.x - w.s * t1.x, w.c * xp.y - w.s * t1.y);
                    x[k * n + q] = make_double2(w.s * t2.x + w.c * xq.x, w.s * t2.y + w.c * xq.y);
                }
            }
            __syncwarp();
            for (int e = lane; e < np * n; e += 32) {
                int p, q;
                pair(e / n, p, q);
                if (q >= n) continue;
                const int k = e % n;
                const WarpRotation w = rot[e / n];
                const double2 xp = a[p * n + k], xq = a[q * n + k];
                const double2 t1 = c_mul(w.ph, xq), t2 = c_mul(c_conj(w.ph), xp);
                a[p * n + k] = make_double2(w.c * xp.x - w.s * t1.x, w.c * xp.y - w.s * t1.y);
                a[q * n + k] = make_double2(w.s * t2.x + w.c * xq.x, w.s * t2.y + w.c * xq.y);
            }
        }
        __syncwarp();
    }
    __syncwarp();
}

// whether the Hermitian matrix a (overwritten) is positive definite: the
// pivots of its LDL^H factors (the lower triangle is updated)
__device__ inline bool herm_positive_warp(int n, double2* a) {
    const int lane = threadIdx.x & 31;
    for (int c = 0; c < n; c++) {
        const double d = a[c * n + c].x;
        if (!(d > 0.0)) return false;
        const double r = 1.0 / d;
        if (lane > c && lane < n) {  // row `lane` less its multiple of row c
            const double2 f = make_double2(a[lane * n + c].x * r, a[lane * n + c].y * r);
            for (int k = c + 1; k <= lane; k++) {
                const double2 t = c_mul(f, c_conj(a[k * n + c]));
                a[lane * n + k].x -= t.x;
                a[lane * n + k].y -= t.y;
            }
        }
        __syncwarp();
    }
    return true;
}

// herm_inverse by one warp: the same pivots (largest magnitude, the first of
// equals; a NaN on the diagonal stays the pivot and spreads)
__device__ inline int herm_inverse_warp(int n, double2* a, double2* inv) {
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < n * n; i += 32) inv[i] = make_double2((i / n == i % n) ? 1.0 : 0.0, 0.0);
    __syncwarp();
    for (int c = 0; c < n; c++) {
        double m2 = -1.0;
        if (lane >= c && lane < n) {
            const double2 x = a[lane * n + c];
            m2 = x.x * x.x + x.y * x.y;
        }
        int piv = c;
        if (!isnan(__shfl_sync(0xffffffffu, m2, c))) {
            const double best = warp_max_f64(m2);  // fmax passes over NaN
            if (best == 0.0) return c + 1;
            piv = __ffs(__ballot_sync(0xffffffffu, m2 == best)) - 1;
        }
        const double2 d = a[piv * n + c];
        const double dd = d.x * d.x + d.y * d.y;
        const double2 r = make_double2(d.x / dd, -d.y / dd);
        __syncwarp();
        if (lane < n) {  // lane k: columns k of the rows c and piv
            const double2 u = a[c * n + lane], w = inv[c * n + lane];
            const double2 pu = a[piv * n + lane], pw = inv[piv * n + lane];
            a[piv * n + lane] = u;
            inv[piv * n + lane] = w;
            a[c * n + lane] = c_mul(pu, r);
            inv[c * n + lane] = c_mul(pw, r);
        }
        __syncwarp();
        // every other row less its multiple of row c; column c of a, the
        // multiples, is not read again and stays
        for (int e = lane; e < n * n; e += 32) {
            const int row = e / n, k = e % n;
            if (row == c) continue;
            const double2 f = a[row * n + c];
            if (k != c) {
                const double2 t = c_mul(f, a[c * n + k]);
                a[e].x -= t.x;
                a[e].y -= t.y;
            }
            const double2 t = c_mul(f, inv[c * n + k]);
            inv[e].x -= t.x;
            inv[e].y -= t.y;
        }
        __syncwarp();
    }
    return 0;
}

// sync_rho1 by one warp; n <= 30, work: 3 n^2 double2
__device__ inline int sync_rho1_warp(int n, double2* rho1, double2* rinv, double reg_fac,
                                     double2* work) {
    const int lane = threadIdx.x & 31;
    double2 *a = work, *v = work + n * n;
    auto copy = [&](double2* x) {
        for (int i = lane; i < n * n; i += 32) x[i] = rho1[i];
        __syncwarp();
    };
    copy(v);
    if (herm_positive_warp(n, v)) {
        copy(a);
        if (herm_inverse_warp(n, a, rinv) == 0) {
            double f2 = 0.0, tr = 0.0;
            for (int i = lane; i < n * n; i += 32) {
                f2 += rinv[i].x * rinv[i].x + rinv[i].y * rinv[i].y;
                if (i / n == i % n) tr += rho1[i].x;
            }
            f2 = warp_sum_f64(f2);
            tr = warp_sum_f64(tr);
            if (sqrt(f2) * tr * 2.0 * reg_fac < 1.0) {
                __syncwarp();
                return 0;
            }
        }
        __syncwarp();
    }
    WarpRotation* rot = (WarpRotation*)(work + 2 * n * n);
    copy(a);
    herm_eig_warp(n, a, v, rot);
    const double w = lane < n ? a[lane * n + lane].x : 0.0;
    const double hi = warp_max_f64(lane < n ? w : -1.7976931348623157e308);
    const double lo = -warp_max_f64(lane < n ? -w : -1.7976931348623157e308);
    if (lo / hi < reg_fac) {
        const double x = hi * reg_fac;
        const double f = lane < n ? x * exp(-w / x) : 0.0;
        for (int base = 0; base < n * n; base += 32) {  // the same trips for every lane
            const int e = base + lane, i = e / n, j = e % n;
            double2 z = make_double2(0.0, 0.0);
            for (int k = 0; k < n; k++) {
                const double fk = __shfl_sync(0xffffffffu, f, k);
                if (e < n * n) {
                    const double2 t = c_mul(v[i * n + k], c_conj(v[j * n + k]));
                    z.x += fk * t.x;
                    z.y += fk * t.y;
                }
            }
            if (e < n * n) {
                rho1[e].x += z.x;
                rho1[e].y += z.y;
            }
        }
    }
    __syncwarp();
    copy(a);
    const int rc = herm_inverse_warp(n, a, rinv);
    __syncwarp();
    return rc;
}

// Implicit QL with Wilkinson shifts for the symmetric tridiagonal matrix (d, e)
// by one warp; eigenvectors accumulate in the columns of row-major z (n x n,
// shared by the warp).  Every lane runs the scalar recurrence on its own copies
// of d and e, lane k rotates row k (k + 32) of z.
// c and s are quotients: as products by a rounded 1 / r they moved c^2 + s^2
// off 1 and the error of a Lanczos step against 80-bit arithmetic was 4.9e-16
// instead of 4.3e-16 (mean of 120 steps of 5,000 to 10,600 configurations).  Even
// lanes divide f, odd ones g: one division's time for the two, same doubles (a
// step of 12 bosons in 5 orbitals with 16 vectors 478 -> 462 us, of 8 in 10 with
// 30 vectors 2,016 -> 1,961 us; both divisions on every lane before).
__device__ inline int tridiag_ql_warp(int n, double* d, double* e, double* z) {
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < n; k += 32)
        for (int i = 0; i < n; i++) z[k * n + i] = i == k ? 1.0 : 0.0;
    if (n < 1) return 0;
    e[n - 1] = 0.0;
    for (int l = 0; l < n; l++) {
        for (int iter = 0;; iter++) {
            int m;
            for (m = l; m < n - 1; m++) {
                const double dd = fabs(d[m]) + fabs(d[m + 1]);
                if (fabs(e[m]) <= 2.220446049250313e-16 * dd) break;
            }
            if (m == l) break;
            if (iter == 60) return l + 1;
            double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
            double r = hypot(g, 1.0);
            g = d[m] - d[l] + e[l] / (g + (g >= 0.0 ? fabs(r) : -fabs(r)));
            double s = 1.0, c = 1.0, p = 0.0;
            bool deflated = false;
            for (int i = m - 1; i >= l; i--) {
                const double f = s * e[i], b = c * e[i];
                r = hypot(f, g);
                e[i + 1] = r;
                if (r == 0.0) {
                    d[i + 1] -= p;
                    e[m] = 0.0;
                    deflated = true;
                    break;
                }
                const double q = (lane & 1 ? g : f) / r;
                s = __shfl_sync(0xffffffffu, q, 0);
                c = __shfl_sync(0xffffffffu, q, 1);
                g = d[i + 1] - p;
                r = (d[i] - g) * s + 2.0 * c * b;
                p = s * r;
                d[i + 1] = g + p;
                g = c * r - b;
                for (int k = lane; k < n; k += 32) {
                    const double zf = z[k * n + i + 1], z0 = z[k * n + i];
                    z[k * n + i + 1] = s * z0 + c * zf;
                    z[k * n + i] = c * z0 - s * zf;
                }
            }
            if (deflated) continue;
            d[l] -= p;
            e[l] = g;
            e[m] = 0.0;
        }
    }
    __syncwarp();
    return 0;
}
#endif

}  // namespace mctdhb
