"""Rounding of the pointwise operators of a spin-1 step.

se_spin1 of fortress_b200/csrc/fgpe_device.cuh is compiled for the host and
compared with the closed form in 80 bits, on spinors of random direction and
of 1 to 1/20 of the largest amplitude.

SE changes a spinor by a small part of itself, so its result should be as
good as the exact one rounded to the type: where the change is at most 1/16
and carries about eight roundings of its own, they add 8 / 16^2 = 3 % to the
square of the one rounding of the sum; 5 % is allowed on the rms (10 % of the
square)."""
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
#include <cstring>
#include <random>
using namespace fgpe;
typedef long double L;
typedef std::complex<L> cl;
template <typename T> cl wide(cx<T> a) { return cl(a.x, a.y); }
template <typename T> cx<T> narrow(cl a) { return mk<T>((T)a.real(), (T)a.imag()); }

void exact_se(int imag, L dt, L t1, cl* v) {
    const cl A = v[1] * std::conj(v[2]) * t1, B = v[1] * std::conj(v[0]) * t1;
    const L r2 = std::norm(A) + std::norm(B), r = sqrtl(r2), x = dt * r;
    const cl h0 = A * v[1], h1 = std::conj(A) * v[0] + std::conj(B) * v[2], h2 = B * v[1];
    const L s = imag ? sinhl(x / 2) : sinl(x / 2), dc = (imag ? 2 : -2) * s * s / r2;
    const cl kf = imag ? cl(-sinhl(x) / r, 0) : cl(0, -sinl(x) / r);
    v[0] += dc * A * h1 + kf * h0;
    v[1] += dc * r2 * v[1] + kf * h1;
    v[2] += dc * B * h1 + kf * h2;
}
struct Rms {
    L e = 0, s = 0;
    void add(cl got, cl want, L norm) { e += std::norm(got - want) / norm; s += 1; }
    double get(double unit) const { return (double)sqrtl(e / s) / unit; }
};
template <typename T> void run(int imag, double dt, double t0, double t1, double amp) {
    StepConst c;
    memset(&c, 0, sizeof c);
    c.dim = 3; c.spin = 1; c.ms = 3; c.dt = dt; c.imag = imag; c.tau0 = t0; c.tau1 = t1;
    const L ldt = (T)dt, l1 = (T)t1;
    std::mt19937_64 g(7);
    std::normal_distribution<double> nd;
    std::uniform_real_distribution<double> un(0, 1);
    Rms se, se_ref;
    for (int i = 0; i < 60000; ++i) {
        const double a = amp * exp(-3 * un(g));
        cx<T> v[3], w[3];
        cl e[3];
        for (int m = 0; m < 3; ++m) {
            v[m] = w[m] = mk<T>((T)(a * nd(g)), (T)(a * nd(g)));
            e[m] = wide<T>(v[m]);
        }
        exact_se(imag, ldt, l1, e);
        se_spin1<T>(c, w);
        const L n = std::norm(e[0]) + std::norm(e[1]) + std::norm(e[2]);
        for (int m = 0; m < 3; ++m) {
            se.add(wide<T>(w[m]), e[m], n);
            se_ref.add(wide<T>(narrow<T>(e[m])), e[m], n);
        }
    }
    const double unit = sizeof(T) == 4 ? 0x1p-24 : 0x1p-53;
    std::printf("se %d %d %g %.5f %.5f\n", (int)sizeof(T), imag, dt * t1 * amp * amp, se.get(unit), se_ref.get(unit));
}
int main() {
    for (int imag = 0; imag < 2; ++imag) {
        const double p[][4] = {{1e-3, 7000, -30, 0.05}, {1e-3, 400, -15, 0.3}, {5e-4, 1000, 40, 0.1}, {1e-4, 2000, -100, 0.1}};
        for (auto& q : p) {
            run<float>(imag, q[0], q[1], q[2], q[3]);
            run<double>(imag, q[0], q[1], q[2], q[3]);
        }
    }
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    exe = compile_probe(tmp_path_factory.mktemp("pointwise"), PROBE)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [r.split() for r in out.splitlines()]


@pytest.mark.parametrize("imag", ["0", "1"], ids=["real", "imaginary"])
@pytest.mark.parametrize("size", ["8", "4"], ids=["fp64", "fp32"])
def test_se_rounds_as_the_exact_result_rounded(rows, size, imag):
    mine = [r for r in rows if r[:3] == ["se", size, imag]]
    assert len(mine) == 4
    for r in mine:
        assert float(r[4]) <= 1.05 * float(r[5]), r
