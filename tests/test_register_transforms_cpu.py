"""Rounding and frequency order of the register-resident transforms.

The library's own in-register transforms, twiddles and radix plans
(fortress_b200/csrc/fgpe_dft.cuh) are compiled for the host and run pass by
pass on random lines, for every plan the column, row and persistent passes
take.  Position p of the result has to hold the frequency that LPlan::krev
names, and the root-mean-square error against an 80-bit transform may not
exceed that of the passes over a shared tile (fgpe_device.cuh, tw_powers) on
the plans of the same length.

Tolerance: both sides are an rms over 24 lines of N values, which scatters by
less than 1 % (24 N > 3000 values); 2 % is allowed."""
import shutil
import subprocess

import pytest

from tests.host_device import compile_probe

PROBE = r"""
#include "fgpe_dft.cuh"
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>
using namespace fgpe;
typedef std::complex<long double> cl;

template <typename T, int R, bool TILE> void butterfly(std::vector<cx<T>>& s, const cx<T>* tw, int e0, int si, int n2, int step) {
    cx<T> v[1][R];
    for (int r = 0; r < R; ++r) v[0][r] = s[e0 + r * si];
    Dft<T, false, R>::run(v[0]);
    if (n2) {
        if constexpr (TILE) {
            cx<T> w[R];
            tw_powers<T, R>(tw, n2, step, w);
            for (int r = 1; r < R; ++r) v[0][r] = cmul(v[0][r], w[r]);
        } else {
            Twiddles<T, R> w;
            w.load(tw, n2, step);
            w.template apply<false, 1>(v);
        }
    }
    for (int r = 0; r < R; ++r) s[e0 + r * si] = v[0][r];
}
template <typename T, bool TILE, int R, int... Q> void passes(std::vector<cx<T>>& s, const cx<T>* tw, int N, int B) {
    const int si = B / R;
    for (int q = 0; q < N / R; ++q) butterfly<T, R, TILE>(s, tw, q / si * B + q % si, si, q % si, N / B);
    if constexpr (sizeof...(Q) > 0) passes<T, TILE, Q...>(s, tw, N, si);
}
// rms error of the plan, in units of the type's rounding; frequency of position p from f
template <typename T, bool TILE, int... R, class F> double rms(F f) {
    constexpr int N = (R * ... * 1);
    const long double pi = acosl(-1.0L);
    std::vector<cx<T>> tw(N);
    std::vector<cl> W(N);
    for (int t = 0; t < N; ++t) {
        tw[t].x = (T)cosl(2 * pi * t / N);
        tw[t].y = (T)-sinl(2 * pi * t / N);
        W[t] = cl(cosl(2 * pi * t / N), -sinl(2 * pi * t / N));
    }
    std::mt19937_64 g(N);
    std::normal_distribution<double> nd;
    long double e2 = 0, s2 = 0;
    for (int trial = 0; trial < 24; ++trial) {
        std::vector<cx<T>> x(N), s;
        for (auto& v : x) { v.x = (T)nd(g); v.y = (T)nd(g); }
        s = x;
        passes<T, TILE, R...>(s, tw.data(), N, N);
        for (int p = 0; p < N; ++p) {
            cl a = 0;
            for (int i = 0; i < N; ++i) a += cl(x[i].x, x[i].y) * W[(long long)i * f(p) % N];
            e2 += std::norm(cl(s[p].x, s[p].y) - a);
            s2 += std::norm(a);
        }
    }
    return (double)sqrtl(e2 / s2) * (sizeof(T) == 4 ? 0x1p24 : 0x1p53);
}
template <typename T, int... R> void tile() {
    constexpr int N = (R * ... * 1), rr[] = {R...};
    auto f = [&](int p) {
        int k = 0, m = 1, b = N;
        for (int r : rr) { b /= r; k += m * (p / b); p %= b; m *= r; }
        return k;
    };
    std::printf("tile %d %d %.4f", (int)sizeof(T), N, rms<T, true, R...>(f));
    for (int r : rr) std::printf(" %d", r);
    std::printf("\n");
}
template <typename T, class P> void lines(const char* what) {
    auto f = [](int p) { return P::krev(p / P::RL) + p % P::RL * (P::N / P::RL); };
    double e;
    if constexpr (P::three) e = rms<T, false, P::R0, P::R1, P::R2>(f);
    else e = rms<T, false, P::R0, P::R1>(f);
    std::printf("%s %d %d %.4f %d %d %d\n", what, (int)sizeof(T), P::N, e, P::R0, P::R1, P::R2);
}
template <typename T, int N> void all() {
    lines<T, typename ColPlan<3, N, COLK_FWD, true>::P>("single");
    lines<T, typename ColPlan<3, N, COLK_Z3D, true>::P>("z3");
    lines<T, typename ColPlan<5, N, COLK_Z3D, true>::P>("z5");
    lines<T, typename ColPlan<3, N, COLK_Y2D, true>::P>("small");
    lines<T, typename PColPlan<N, 1>::P>("persist1");
    lines<T, typename PColPlan<N, 3>::P>("persist3");
}
// the shared-tile plans (cplan 0 to 3, shortest names)
template <typename T> void tiles() {
    tile<T, 8, 8, 2>(); tile<T, 16, 8>();
    tile<T, 8, 8, 3>();
    tile<T, 8, 8, 4>(); tile<T, 16, 16>();
    tile<T, 8, 8, 2, 3>(); tile<T, 16, 8, 3>();
    tile<T, 8, 8, 8>();
}
int main() {
    tiles<double>(); tiles<float>();
    all<double, 128>(); all<double, 192>(); all<double, 256>(); all<double, 384>(); all<double, 512>();
    all<float, 128>(); all<float, 192>(); all<float, 256>(); all<float, 384>(); all<float, 512>();
}
"""


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    exe = compile_probe(tmp_path_factory.mktemp("transforms"), PROBE)
    tile, lines = {}, {}
    for row in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines():
        what, size, n, e, *radices = row.split()
        key = int(size), int(n)
        if what == "tile":
            tile[key] = max(tile.get(key, 0.0), float(e))
        else:
            lines.setdefault(key, {})[what + "-" + "x".join(radices)] = float(e)
    return tile, lines


@pytest.mark.skipif(not shutil.which("g++"), reason="needs a C++ compiler")
@pytest.mark.parametrize("size", [8, 4], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [128, 192, 256, 384, 512])
def test_register_plans_round_no_worse_than_tile_passes(errors, n, size):
    tile, lines = errors
    assert lines[size, n]
    for plan, e in lines[size, n].items():
        assert e <= 1.02 * tile[size, n], (plan, e, tile[size, n])
