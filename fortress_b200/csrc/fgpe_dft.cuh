// fgpe_dft.cuh -- in-register transforms of composite length and the
// compile-time helpers of the register-resident passes (fgpe_regcol.cuh,
// fgpe_regrow.cuh).
#pragma once
#include <type_traits>

#include "fgpe_device.cuh"

namespace fgpe {

template <int I, int N, class F> __device__ __forceinline__ void static_for(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(static_cast<F&&>(f));
    }
}

// cos and sin of 2 pi num / den at compile time: reduced to an octant, then
// the Taylor series on [0, pi/4] (x^21/21! < 1e-21).
struct Root { double c, s; };
constexpr double octant_sin(double x) {
    double t = x, s = x;
    for (int k = 1; k < 11; ++k) { t *= -x * x / ((2.0 * k) * (2.0 * k + 1.0)); s += t; }
    return s;
}
constexpr double octant_cos(double x) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 11; ++k) { t *= -x * x / ((2.0 * k - 1.0) * (2.0 * k)); s += t; }
    return s;
}
constexpr Root unit_root(int num, int den) {
    const double q = 0.78539816339744830961566084581987572105;   // pi/4
    const int p = 8 * (num % den), o = p / den, r = p - o * den;
    const double x = q * (double)((o & 1) ? den - r : r) / (double)den;
    const double c = octant_cos(x), s = octant_sin(x);
    switch (o) {
        case 0: return {c, s};
        case 1: return {s, c};
        case 2: return {-s, c};
        case 3: return {-c, s};
        case 4: return {-c, -s};
        case 5: return {-s, -c};
        case 6: return {s, -c};
        default: return {c, -s};
    }
}

// a * exp(-+ 2 pi i NUM / DEN) (minus: forward)
template <typename T, bool INV, int NUM, int DEN> __device__ __forceinline__ cx<T> rot_root(cx<T> a) {
    constexpr int n = NUM % DEN;
    if constexpr (n == 0) return a;
    else if constexpr (4 * n == DEN) return cmuli(a, INV ? 1 : -1);
    else if constexpr (2 * n == DEN) return mk<T>(-a.x, -a.y);
    else if constexpr (4 * n == 3 * DEN) return cmuli(a, INV ? -1 : 1);
    else {
        constexpr Root w = unit_root(n, DEN);
        constexpr T c = (T)w.c, s = (T)(INV ? w.s : -w.s);
        if constexpr (8 * n % DEN == 0) {
            constexpr T h = (T)0.70710678118654752440084436210484903928;
            constexpr T sc = w.c > 0 ? (T)1 : (T)-1, ss = (INV ? w.s : -w.s) > 0 ? (T)1 : (T)-1;
            return mk<T>(h * (sc * a.x - ss * a.y), h * (ss * a.x + sc * a.y));
        } else {
            return mk<T>(a.x * c - a.y * s, a.x * s + a.y * c);
        }
    }
}

// A*B points as A x B: x[n1 + A n2] -> B-point transforms over n2, twiddles
// W^(n1 k2), A-point transforms over n1 -> X[B k1 + k2] (natural order out).
template <typename T, bool INV, int A, int B> struct DftAB {
    static __device__ __forceinline__ void run(cx<T>* v) {
        cx<T> y[A][B];
        static_for<0, A>([&](auto n1) {
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) y[n1][n2] = v[n1 + A * n2];
            Dft<T, INV, B>::run(y[n1]);
            static_for<0, B>([&](auto k2) {
                constexpr int N1 = decltype(n1)::value, K2 = decltype(k2)::value;
                y[N1][K2] = rot_root<T, INV, N1 * K2, A * B>(y[N1][K2]);
            });
        });
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) {
            cx<T> z[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) z[n1] = y[n1][k2];
            Dft<T, INV, A>::run(z);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) v[B * k1 + k2] = z[k1];
        }
    }
};
template <typename T, bool INV> struct Dft<T, INV, 6> : DftAB<T, INV, 2, 3> {};
template <typename T, bool INV> struct Dft<T, INV, 12> : DftAB<T, INV, 4, 3> {};
template <typename T, bool INV> struct Dft<T, INV, 24> : DftAB<T, INV, 3, 8> {};
template <typename T, bool INV> struct Dft<T, INV, 32> : DftAB<T, INV, 4, 8> {};

// The twiddles w^1..w^(R-1) a thread applies, w = tw[j * step].  FP32 loads
// every power (the rounding of products would show up there).  FP64 up to
// radix 8 loads w and forms the powers by products; above, it loads w, w^4
// and w^16 and forms w^(r mod 4) w^(4 (r div 4)), so that few powers are live
// at a time and none is far from the table: powers of w alone doubled the rms
// error of a 512-point transform (32 * 16: 6.1 units of 2^-53 against 3.1
// with radix 8; this way 2.2).
template <typename T, int R> struct Twiddles {
    static constexpr int NW = sizeof(T) == 4 ? R : R <= 8 ? 2 : R <= 16 ? 3 : 4;
    cx<T> w[NW];        // FP64: w, w^4, w^16
    __device__ __forceinline__ void load(const cx<T>* __restrict__ tw, int j, int step) {
#pragma unroll
        for (int r = 1; r < NW; ++r) w[r] = tw[j * step * (sizeof(T) == 4 ? r : r == 1 ? 1 : r == 2 ? 4 : 16)];
    }
    // v[m][r] *= w^r (conjugate for the inverse)
    template <bool INV, int CNT> __device__ __forceinline__ void apply(cx<T> (&v)[CNT][R]) const {
        auto mul = [](cx<T> a, cx<T> b) { return INV ? cmulc(a, b) : cmul(a, b); };
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int r = 1; r < R; ++r)
#pragma unroll
                for (int m = 0; m < CNT; ++m) v[m][r] = mul(v[m][r], w[r]);
        } else {
            constexpr int LOW = R <= 8 ? R : 4;
            cx<T> b[LOW];
            b[1] = w[1];
#pragma unroll
            for (int r = 2; r < LOW; ++r) b[r] = (r % 2 == 0) ? cmul(b[r / 2], b[r / 2]) : cmul(b[r - 1], b[1]);
#pragma unroll
            for (int r = 1; r < LOW; ++r)
#pragma unroll
                for (int m = 0; m < CNT; ++m) v[m][r] = mul(v[m][r], b[r]);
            if constexpr (R > 8) {
                cx<T> g = w[2];
#pragma unroll
                for (int h = 4; h < R; h += 4) {
                    if (h == 16) g = w[NW - 1];
                    else if (h > 4) g = cmul(g, w[2]);
#pragma unroll
                    for (int r = h; r < h + 4 && r < R; ++r) {
                        const cx<T> x = r == h ? g : cmul(g, b[r - h]);
#pragma unroll
                        for (int m = 0; m < CNT; ++m) v[m][r] = mul(v[m][r], x);
                    }
                }
            }
        }
    }
};

// -------------------------------------------- radix plans of column lines
// Radix plan of a column line: two passes (R2 = 1) or three.
template <int R0_, int R1_, int R2_ = 1> struct LPlan {
    static constexpr int R0 = R0_, R1 = R1_, R2 = R2_;
    static constexpr int N = R0 * R1 * R2;
    static constexpr bool three = R2 > 1;
    static constexpr int RL = three ? R2 : R1;      // radix of the last pass (contiguous positions)
    // frequency of position q*RL is krev(q); position q*RL + r adds r*N/RL
    static __host__ __device__ __forceinline__ int krev(int q) { return three ? q / R1 + R0 * (q % R1) : q; }
};

// COLK_FWD / COLK_INV: one transform of one component's lines (3D y passes);
// COLK_Y2D: F_y, pending scale + KE + SOC, F_y^-1 (the q2D pass);
// COLK_Z3D: F_z, KE and SOC, F_z^-1, with the SO-coupling numbers of a tile
// column in registers.
enum { COLK_FWD = 0, COLK_INV = 1, COLK_Y2D = 2, COLK_Z3D = 3 };

// Radix plans.  Single-component passes take (N/16, 16): one exchange.  The z
// pass of a grid that fills the GPU holds MS * RL complex values per thread
// between its transforms, so RL = 16 with three components and 8 with five.
// The q2D pass, and the z pass of a small grid, have few tiles and are bound
// by one tile's latency: short last radices and more threads per tile
// (512^2 spin-1 FP32: 16 us with (8, 16, 4) and 256 threads, 27 us with
// (32, 16) and 128).
template <int MS, int N, int KIND, bool BIG> struct ColPlan { using P = LPlan<N / 16, 16>; };
template <int N> struct ColPlan<5, N, COLK_Z3D, true> { using P = LPlan<N / 8, 8>; };
template <> struct ColPlan<5, 384, COLK_Z3D, true> { using P = LPlan<8, 6, 8>; };
template <> struct ColPlan<5, 512, COLK_Z3D, true> { using P = LPlan<8, 8, 8>; };
template <int N> struct SmallPlan { using P = LPlan<8, N / 32, 4>; };
template <> struct SmallPlan<128> { using P = LPlan<8, 8, 2>; };
template <int MS, int N> struct ColPlan<MS, N, COLK_Z3D, false> : SmallPlan<N> {};
template <int N> struct ColPlan<5, N, COLK_Z3D, false> : SmallPlan<N> {};
template <int MS, int N, bool BIG> struct ColPlan<MS, N, COLK_Y2D, BIG> : SmallPlan<N> {};

// Plans of the persistent kernel's variants: 0: radix 8 first and 4 last;
// 1: radix 16 first; 3: other splits of the first two passes.  (Passes over
// the tile take the plans of cplan.)
template <int N, int PV> struct PColPlan : SmallPlan<N> {};
template <int N> struct PColPlan<N, 1> { using P = LPlan<16, N / 64, 4>; };
template <> struct PColPlan<128, 3> { using P = LPlan<8, 4, 4>; };
template <> struct PColPlan<192, 3> { using P = LPlan<12, 4, 4>; };
template <> struct PColPlan<256, 3> { using P = LPlan<4, 16, 4>; };
template <> struct PColPlan<384, 3> { using P = LPlan<12, 8, 4>; };
template <> struct PColPlan<512, 3> { using P = LPlan<16, 8, 4>; };

}  // namespace fgpe
