"""Rounding of the tabulated SO-coupling exponential in imaginary time.

soc_apply of fortress_b200/csrc/fgpe_device.cuh is compiled for the host and
compared with P A0 diag(exp(-dt L alpha)) A0^H P^H in 80 bits (A0 the
eigenvectors of SX, P = diag(exp(-i (S - m) beta))) on random spinors, at wave
numbers where dt alpha is at most 1/16.

There the operator changes a spinor by at most L alpha = 1/16 (three
components) or 1/8 (five) of its length, so its result should be as good as the
exact one rounded to the type, with no error that comes back on every step.
About ten roundings of the change, 1/8 sqrt(10) units against the sum's one
rounding of 0.4 units per component, add at most 0.16 in quadrature: 10 % is
allowed on the rms.  The mean error of one operator over 256 nearby spinors has
a scatter of 1/16 of that rms; the change's own systematic roundings (table and
operator, 1/8 of half a unit each, three of them) add up to 0.1: together less
than a third of the rms."""
import shutil
import subprocess

import pytest

from tests.host_device import compile_probe

pytestmark = pytest.mark.skipif(not shutil.which("g++"), reason="needs a C++ compiler")

PROBE = r"""
#include "fgpe_device.cuh"
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
using namespace fgpe;
typedef long double L;
typedef std::complex<L> cl;
template <int MS> void eigenvectors(L (&a)[MS][MS]) {
    const L h = sqrtl(0.5L), q = sqrtl(0.375L);
    const L a3[9] = {0.5L, -h, 0.5L, -h, 0, h, 0.5L, h, 0.5L};
    const L a5[25] = {0.25L, -0.5L, q, -0.5L, 0.25L, -0.5L, 0.5L, 0, -0.5L, 0.5L, q, 0, -0.5L, 0, q,
                      -0.5L, -0.5L, 0, 0.5L, 0.5L, 0.25L, 0.5L, q, 0.5L, 0.25L};
    for (int i = 0; i < MS * MS; ++i) a[i / MS][i % MS] = MS == 3 ? a3[i % 9] : a5[i];
}
template <typename T, int MS> void run() {
    constexpr int S = MS / 2, NK = 300, NJ = 256;
    std::mt19937_64 g(11);
    std::normal_distribution<double> nd;
    std::uniform_real_distribution<double> un(0, 1);
    L a[MS][MS];
    eigenvectors<MS>(a);
    double e2 = 0, r2 = 0, b2 = 0;
    for (int k = 0; k < NK; ++k) {
        const L x = exp(-5 * un(g)) / 16, beta = 2 * acosl(-1.0L) * un(g);
        Soc4<T> e;
        e.cb = (T)cosl(beta);
        e.sb = (T)sinl(beta);
        if (MS == 3) {
            e.p = (T)(2 * sinhl(x / 2) * sinhl(x / 2));
            e.q = (T)(-sqrtl(2.0L) * sinhl(x));
        } else {
            e.p = (T)expm1l(-x);
            e.q = (T)expm1l(x);
        }
        cl U[MS][MS];
        for (int i = 0; i < MS; ++i)
            for (int j = 0; j < MS; ++j) {
                U[i][j] = 0;
                for (int q = 0; q < MS; ++q) U[i][j] += a[i][q] * a[j][q] * expl(-(q - S) * x);
                U[i][j] *= std::polar((L)1, -(S - i) * beta) * std::polar((L)1, (S - j) * beta);
            }
        double v0[2 * MS];
        for (double& d : v0) d = nd(g);
        cl mean[MS] = {};
        for (int n = 0; n < NJ; ++n) {
            cx<T> v[MS], w[MS];
            cl want[MS];
            L norm = 0;
            for (int m = 0; m < MS; ++m)
                w[m] = v[m] = mk<T>((T)(v0[2 * m] * (1 + 1e-4 * nd(g))), (T)(v0[2 * m + 1] * (1 + 1e-4 * nd(g))));
            for (int i = 0; i < MS; ++i) {
                want[i] = 0;
                for (int j = 0; j < MS; ++j) want[i] += U[i][j] * cl(v[j].x, v[j].y);
                norm += std::norm(want[i]);
            }
            soc_apply<T, MS>(1, e, w);
            for (int m = 0; m < MS; ++m) {
                const cl d = cl(w[m].x, w[m].y) - want[m];
                const cl r = cl((T)want[m].real(), (T)want[m].imag()) - want[m];
                e2 += (double)(std::norm(d) / norm);
                r2 += (double)(std::norm(r) / norm);
                mean[m] += (d - r) / sqrtl(norm) / (L)NJ;
            }
        }
        for (int m = 0; m < MS; ++m) b2 += (double)std::norm(mean[m]);
    }
    const double unit = sizeof(T) == 4 ? 0x1p-24 : 0x1p-53;
    std::printf("%d %d %.4f %.4f %.4f\n", (int)sizeof(T), MS, sqrt(e2 / NK / NJ) / unit, sqrt(r2 / NK / NJ) / unit,
                sqrt(b2 / NK) / unit);
}
int main() {
    run<float, 3>();
    run<float, 5>();
    run<double, 3>();
    run<double, 5>();
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    exe = compile_probe(tmp_path_factory.mktemp("soc"), PROBE)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return {tuple(int(t) for t in r.split()[:2]): [float(t) for t in r.split()[2:]] for r in out.splitlines()}


@pytest.mark.parametrize("ms", [3, 5])
@pytest.mark.parametrize("size", [8, 4], ids=["fp64", "fp32"])
def test_soc_rounds_as_the_exact_result_rounded(rows, size, ms):
    rms, rounded, systematic = rows[size, ms]
    assert rms <= 1.10 * rounded, (rms, rounded)
    assert systematic <= rms / 3, (systematic, rms)
