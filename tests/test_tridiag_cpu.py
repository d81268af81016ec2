"""The tridiagonal eigensolver of the Lanczos step (csrc/small_linalg.cuh,
tridiag_ql_warp) on the host: its rotations are c = g / r, s = f / r.  With the
quotients as products by a rounded 1 / r the cosine and sine carry one more
common rounding, c^2 + s^2 moves off 1 with every rotation, and the error of a
whole Lanczos step grew by a tenth (12 seeds at five sizes, against 80-bit
arithmetic).

The header is compiled as plain C++ with a thread per lane of a warp and
shuffles through a barrier, and the result has to be the same doubles as the
recurrence written out below."""
import ctypes as C
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "1d-mctdhb_b200", "csrc")

STUB = r"""
#pragma once
#include <barrier>
#include <cmath>
#include <thread>
#include <vector>
#define __host__
#define __device__
struct double2 { double x, y; };
static inline double2 make_double2(double x, double y) { return double2{x, y}; }
struct Dim { int x; };
static thread_local Dim threadIdx;
static std::barrier<> warp(32);
static double lanes[32];
static inline void __syncwarp() { warp.arrive_and_wait(); }
static inline double exchange(double v, int from) {
    lanes[threadIdx.x] = v;
    warp.arrive_and_wait();
    const double got = lanes[from];
    warp.arrive_and_wait();
    return got;
}
static inline double __shfl_sync(unsigned, double v, int from) { return exchange(v, from); }
static inline double __shfl_xor_sync(unsigned, double v, int x) {
    return exchange(v, threadIdx.x ^ x);
}
static inline unsigned __ballot_sync(unsigned, bool p) { return p; }
static inline int __ffs(unsigned v) { return __builtin_ffs(v); }
using std::isnan;
"""

MAIN = r"""
#define __CUDACC__
#include "small_linalg.cuh"
extern "C" int ql(int n, double* d, double* e, double* z) {
    int rc = 0;
    std::vector<double> out(n);
    std::vector<std::thread> ts;
    for (int lane = 0; lane < 32; lane++)
        ts.emplace_back([&, lane] {
            double dl[64], el[64];
            for (int i = 0; i < n; i++) dl[i] = d[i], el[i] = e[i];
            threadIdx.x = lane;
            const int r = mctdhb::tridiag_ql_warp(n, dl, el, z);
            if (lane == 0) {
                rc = r;
                for (int i = 0; i < n; i++) out[i] = dl[i];
            }
        });
    for (auto& t : ts) t.join();
    for (int i = 0; i < n; i++) d[i] = out[i];
    return rc;
}
"""


@pytest.fixture(scope="module")
def ql(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("ql")
    (d / "cuda_runtime.h").write_text(STUB)
    (d / "ql.cpp").write_text(MAIN)
    so = str(d / "ql.so")
    subprocess.run([cxx, "-std=c++20", "-O1", "-ffp-contract=off", "-pthread", "-shared", "-fPIC", "-I", str(d),
                    "-I", CSRC, str(d / "ql.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    p = C.POINTER(C.c_double)
    lib.ql.argtypes = [C.c_int, p, p, p]

    def solve(diag, off):
        n = len(diag)
        a, b = np.array(diag, float), np.append(off, 0.0)
        z = np.zeros((n, n))
        ptr = lambda x: x.ctypes.data_as(p)  # noqa: E731
        return lib.ql(n, ptr(a), ptr(b), ptr(z)), a, z

    return solve


def recurrence(diag, off):
    """implicit QL with Wilkinson shifts, eigenvectors in the columns of z"""
    n = len(diag)
    d, e, z = [float(x) for x in diag], [float(x) for x in off] + [0.0], np.eye(n)
    for low in range(n):
        while True:
            m = low
            while m < n - 1 and abs(e[m]) > 2.220446049250313e-16 * (abs(d[m]) + abs(d[m + 1])):
                m += 1
            if m == low:
                break
            g = (d[low + 1] - d[low]) / (2.0 * e[low])
            r = float(np.hypot(g, 1.0))
            g = d[m] - d[low] + e[low] / (g + math.copysign(r, g))
            s = c = 1.0
            p = 0.0
            for i in range(m - 1, low - 1, -1):
                f, b = s * e[i], c * e[i]
                r = float(np.hypot(f, g))
                e[i + 1] = r
                if r == 0.0:
                    d[i + 1] -= p
                    e[m] = 0.0
                    break
                s, c = f / r, g / r
                g = d[i + 1] - p
                r = (d[i] - g) * s + 2.0 * c * b
                p = s * r
                d[i + 1] = g + p
                g = c * r - b
                z[:, i], z[:, i + 1] = c * z[:, i] - s * z[:, i + 1], s * z[:, i] + c * z[:, i + 1]
            else:
                d[low] -= p
                e[low] = g
                e[m] = 0.0
    return np.array(d), z


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 16, 33, 64])
def test_rotations_are_quotients(ql, n):
    rng = np.random.default_rng(n)
    for _ in range(8 if n <= 8 else 1):
        diag, off = rng.normal(size=n) * 3, rng.uniform(0.01, 2.0, size=n - 1)
        rc, d, z = ql(diag, off)
        want, zw = recurrence(diag, off)
        assert rc == 0
        assert np.array_equal(d, want) and np.array_equal(z, zw)


def test_split_matrix(ql):
    """a zero off-diagonal element: blocks of their own"""
    rc, d, z = ql([2.0, 1.0, 5.0], [0.5, 0.0])
    assert rc == 0 and d[2] == 5.0 and np.array_equal(z[2], [0.0, 0.0, 1.0])
