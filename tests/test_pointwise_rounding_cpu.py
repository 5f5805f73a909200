"""Rounding of the pointwise operators of a spin-1 step.

se_spin1 and apply_sp of fortress_b200/csrc/fgpe_device.cuh are compiled for
the host and compared with the closed forms in 80 bits, on spinors of random
direction and of 1 to 1/20 of the largest amplitude.

SE changes a spinor by a small part of itself, so its result should be as
good as the exact one rounded to the type: where the change is at most 1/16
and carries about eight roundings of its own, they add 8 / 16^2 = 3 % to the
square of the one rounding of the sum; 5 % is allowed on the rms (10 % of the
square).

SP multiplies a component by exp(-i CDT V) exp(-i CDT (tau0 rho + B_m)).  The
bar is the chain with nothing but necessary roundings: the exponential of the
type's angle rounded once, its product with the tabulated exp(-i CDT V), the
product with the component.  An angle of at most 1/16 split in two rounds once
more, 1/16 of a unit beside the chain's 0.6 or more (1 % of the square); 5 %
is allowed on the rms."""
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
// one factor per component, every step of it rounded once
template <typename T> void chain_sp(int imag, T dt, T t0, T t1, cx<T> eV, cx<T>* v) {
    T a[3], rho = 0;
    for (int m = 0; m < 3; ++m) { a[m] = cabs2(v[m]); rho += a[m]; }
    const T B[3] = {t1 * (a[0] + a[1] - a[2]), t1 * (a[0] + a[2]), t1 * (a[2] + a[1] - a[0])};
    for (int m = 0; m < 3; ++m) {
        const L x = dt * (t0 * rho + B[m]);
        const cx<T> e = narrow<T>(imag ? cl(expl(-x), 0) : cl(cosl(x), -sinl(x)));
        v[m] = fmul(imag, fmul(imag, e, eV), v[m]);
    }
}
void exact_sp(int imag, L dt, L t0, L t1, cl eV, cl* v) {
    L a[3], rho = 0;
    for (int m = 0; m < 3; ++m) { a[m] = std::norm(v[m]); rho += a[m]; }
    const L B[3] = {t1 * (a[0] + a[1] - a[2]), t1 * (a[0] + a[2]), t1 * (a[2] + a[1] - a[0])};
    for (int m = 0; m < 3; ++m) {
        const L x = dt * (t0 * rho + B[m]);
        v[m] *= eV * (imag ? cl(expl(-x), 0) : cl(cosl(x), -sinl(x)));
    }
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
    const L ldt = (T)dt, l0 = (T)t0, l1 = (T)t1;
    std::mt19937_64 g(7);
    std::normal_distribution<double> nd;
    std::uniform_real_distribution<double> un(0, 1);
    Rms se, se_ref, sp, sp_ref;
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
        const L V = 20 * dt * un(g);
        const cx<T> eV = narrow<T>(imag ? cl(expl(-V), 0) : cl(cosl(V), -sinl(V)));
        cx<T> u[3];
        for (int m = 0; m < 3; ++m) { w[m] = u[m] = v[m]; e[m] = wide<T>(v[m]); }
        exact_sp(imag, ldt, l0, l1, wide<T>(eV), e);
        apply_sp<T, 3>(c, eV, w);
        chain_sp<T>(imag, (T)dt, (T)t0, (T)t1, eV, u);
        for (int m = 0; m < 3; ++m) {
            sp.add(wide<T>(w[m]), e[m], std::norm(e[m]));
            sp_ref.add(wide<T>(u[m]), e[m], std::norm(e[m]));
        }
    }
    const double unit = sizeof(T) == 4 ? 0x1p-24 : 0x1p-53;
    std::printf("se %d %d %g %.5f %.5f\n", (int)sizeof(T), imag, dt * t1 * amp * amp, se.get(unit), se_ref.get(unit));
    std::printf("sp %d %d %g %.5f %.5f\n", (int)sizeof(T), imag, dt * t0 * amp * amp, sp.get(unit), sp_ref.get(unit));
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


@pytest.mark.parametrize("imag", ["0", "1"], ids=["real", "imaginary"])
@pytest.mark.parametrize("size", ["8", "4"], ids=["fp64", "fp32"])
def test_sp_rounds_as_one_factor_per_component(rows, size, imag):
    mine = [r for r in rows if r[:3] == ["sp", size, imag]]
    assert len(mine) == 4
    for r in mine:
        assert float(r[4]) <= 1.05 * float(r[5]), r
