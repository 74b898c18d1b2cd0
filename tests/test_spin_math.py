"""The scalar arithmetic of the spindown kernels (tdf_split.cuh), evaluated on
the host: the functions are the kernels' own, compiled by nvcc for the host,
and consist of IEEE operations that give the same bits there (no contraction).
They are compared with the x87 extended precision of numpy.longdouble."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from tdfstat_b200 import build as B

L = np.longdouble
TWO_PI = L("6.283185307179586476925286766559005768")

SOURCE = r"""
#include <math.h>
#include <string.h>
#include "tdf_kernels.cuh"
using namespace tdf;
extern "C" void spin_phase(double het1, double spnd, int N, long n, const int *i, float *plain, float *big) {
     SpinPhase p;
     const bool past = p.init(het1, spnd, N);
     for (long k = 0; k < n; k++) {
          plain[k] = past ? NAN : p.at<false>((double)i[k]);
          big[k] = p.at<true>((double)i[k]);
     }
}
extern "C" void spin_sincos(long n, const double *x, double *s, double *c) {
     for (long k = 0; k < n; k++) sincos_spin(x[k], s[k], c[k]);
}
extern "C" void fp64_fstat(long n, const double *A, const double *B, const double *aa, const double *bb, double *F) {
     for (long k = 0; k < n; k++) F[k] = FstatSums(aa[k], bb[k]).f(A[k], B[k]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("spin_math")
    src, out = os.path.join(d, "spin_math.cu"), os.path.join(d, "spin_math.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    r = subprocess.run([B.nvcc(), "-std=c++17", "-O2", *B.ARCH, "-Xcompiler", "-fPIC", "-shared",
                        "-I" + os.path.join(B.REPO, "include"), "-I" + B.CSRC, "-o", out, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return C.CDLL(out)


def _p(a, t):
    return a.ctypes.data_as(C.POINTER(t))


# N, spindown phase at the last sample in turns (2^18 turns: the limit of the plain branch)
@pytest.mark.parametrize("N,turns", [(5385, 0.3), (86164, 900.0), (258492, -9000.0), (516985, 2.0 ** 18 * 0.99),
                                     (258492, 2.0 ** 18 * 40)])
def test_split_phase_is_rounded_to_fp32_once(lib, N, turns):
    """The phase in radians is off by the FP32 rounding of a value up to pi
    (half of 2^-22), by the fixed-point fraction (2^-33 turns), and by the FP64
    roundings of h, w and q: 2.5 * 2^-53 of the turns."""
    lib.spin_phase.argtypes = [C.c_double, C.c_double, C.c_int, C.c_long] + [C.c_void_p] * 3
    rng = np.random.default_rng(N)
    i = np.unique(np.concatenate([[0, 1, N - 1], rng.integers(0, N, 6000)])).astype(np.int32)
    het1 = rng.uniform(0, 2 * np.pi / 2 ** 18)
    spnd = turns * 2 * np.pi / float(N) ** 2
    plain, big = np.zeros(len(i), np.float32), np.zeros(len(i), np.float32)
    lib.spin_phase(het1, spnd, N, len(i), i.ctypes.data, plain.ctypes.data, big.ctypes.data)
    t = (L(het1) * i + L(spnd) * i.astype(L) ** 2) / TWO_PI
    f = t - np.rint(t)
    for got in (plain, big):
        if np.isnan(got).all():
            assert abs(turns) > 2 ** 18
            continue
        d = (got.astype(L) / TWO_PI - f)
        d -= np.rint(d)   # fractions near half a turn may carry either sign
        d = np.abs(d * TWO_PI)
        tol = 2.0 ** -23 + 2 * np.pi * (2.0 ** -33 + (abs(turns) + 1) * 2.5 * 2.0 ** -53)
        assert np.max(d) <= tol, (float(np.max(d)), tol)
        # a value rounded once, evenly spread over its interval: the rms error over
        # [-pi, pi] is the root mean square of the half ulps over sqrt(3)
        x = np.linspace(0.001, np.pi, 10000).astype(np.float32)
        once = np.sqrt(np.mean((np.spacing(x) / 2) ** 2) / 3)
        rest = 2 * np.pi * (2.0 ** -33 + (abs(turns) + 1) * 2.5 * 2.0 ** -53)
        if abs(turns) > 100:
            assert float(np.sqrt(np.mean(d * d))) <= 1.05 * once + rest


def test_fp64_fstat_rounds_no_more_than_the_quotients(lib):
    """A/aa + B/bb as the FP64 rows form it: two roundings, each of at most
    half an ulp of F (the quotients and their sum make three); values that are
    not finite as the quotients give them."""
    lib.fp64_fstat.argtypes = [C.c_long] + [C.c_void_p] * 5
    rng = np.random.default_rng(7)
    n = 200000
    A, B, aa, bb = (np.exp(rng.uniform(-20, 20, n)) for _ in range(4))
    F = np.zeros(n)
    lib.fp64_fstat(n, *(v.ctypes.data for v in (A, B, aa, bb, F)))
    want = A.astype(L) / aa + B.astype(L) / bb
    ulps = np.abs(F.astype(L) - want) / np.spacing(want.astype(np.float64))
    # the lower parts' terms are 2^-53 of F and rounded to 2^-53 of that; extended precision has 2^-64
    assert np.max(ulps) <= 1.0 + 2.0 ** -9, float(np.max(ulps))
    odd = np.array([[0., 0., 0., 0.], [1., 1., 0., 2.], [np.inf, 1., 4., 3.], [1., np.inf, 3., 4.],
                    [np.nan, 1., 3., 3.], [0., 0., 5., 7.], [1e308, 1e308, 1e-3, 1.], [1., 1., np.inf, 2.]])
    A, B, aa, bb = (np.ascontiguousarray(odd[:, k]) for k in range(4))
    F = np.zeros(len(odd))
    lib.fp64_fstat(len(odd), *(v.ctypes.data for v in (A, B, aa, bb, F)))
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(F, A / aa + B / bb)


@pytest.mark.parametrize("phases", ["1", "100", "1e5", "1e9", "multiples 1e5", "multiples 1e9"])
def test_fp64_sine_and_cosine(lib, phases):
    """Absolute error of sincos_spin() up to 2^30 rad, near multiples of pi/2
    as well: 2^-54 from each of the two reductions and the last multiply-add
    (values below 1), 7e-17 at most from the series' roundings, together below
    2^-52."""
    lib.spin_sincos.argtypes = [C.c_long] + [C.c_void_p] * 3
    rng = np.random.default_rng(11)
    n = 200000
    R = float(phases.split()[-1])
    if phases.startswith("multiples"):
        k = rng.integers(-int(R / 1.6), int(R / 1.6), n)
        # an offset of up to 1e-3 of random size
        x = (k * (TWO_PI / 4) + rng.choice([-1, 0, 1], n) * np.exp(rng.uniform(-40, -7, n))).astype(np.float64)
    else:
        x = rng.uniform(-R, R, n)
    x = np.concatenate([x, [0.0, np.pi / 4, -np.pi / 4, np.pi / 2]])
    s, c = np.zeros(len(x)), np.zeros(len(x))
    lib.spin_sincos(len(x), x.ctypes.data, s.ctypes.data, c.ctypes.data)
    for got, want in ((s, np.sin(x.astype(L))), (c, np.cos(x.astype(L)))):
        assert np.max(np.abs(got.astype(L) - want)) <= 2.0 ** -52
