// fgpe_regcol.cuh -- column passes with their transforms in registers.
//
// A tile is TX adjacent x positions by a whole line of N along y or z.  A
// line is transformed by two or three radix passes (LPlan), and each thread
// keeps whole butterflies in registers: the first pass reads its elements
// straight from global memory (with the operators: from slots of its own that
// an asynchronous copy has filled), the last one of an inverse transform
// writes them straight back, and in the pass that carries KE and SOC the last
// forward pass, the k-space operators and the first inverse pass are one
// visit to registers that hold all MS components of the same spectral
// positions.  Shared memory carries only the exchanges between radix passes:
// two to four trips where passes over a shared tile take up to eight.
//
// Measured on one B200, 256^3 spin-1, against the shared-tile passes:
//   y pass   FP64 0.33 -> 0.30 ms (5.3 TB/s, 0.81 of the measured copy
//            rate), FP32 0.19 -> 0.14 ms (5.8 TB/s): bound by HBM;
//   z pass   FP64 0.65 -> 0.42 ms, FP32 0.37 -> 0.25 ms: bound by latency at
//            8 or 12 warps per SM, the FP64 pipe about half busy.  A thread
//            holds 48 complex values there; (8,4,8) and (32,8) lines with
//            twice the warps took 10 to 40 % longer.
#pragma once
#include "fgpe_async.cuh"
#include "fgpe_dft.cuh"
#include "fgpe_group.cuh"
#include "fgpe_kernels.h"

namespace fgpe {

template <typename T, int TX, int RL> struct RegTile {
    // tile rows narrower than 128 bytes are padded by one row every RL (at
    // least 4), so that the strided butterflies of the last pass fall on
    // distinct banks
    static constexpr bool padded = TX * (int)sizeof(cx<T>) < 128;
    static constexpr int PAD = RL < 4 ? 4 : RL;
    static constexpr __host__ __device__ int rows(int n) { return padded ? n + n / PAD : n; }
    static __device__ __forceinline__ int at(int e, int t) { return (padded ? e + e / PAD : e) * TX + t; }
};

// KEZ: the kz part of KE beside the tile (z pass)
template <typename T, int MS, int N, int TX, class PL, int KIND, bool KEZ> constexpr size_t regcol_smem() {
    return ((size_t)(KIND >= COLK_Y2D ? MS : 1) * RegTile<T, TX, PL::RL>::rows(N) * TX + (KEZ ? MS * N : 0)) * sizeof(cx<T>);
}

template <typename T> __device__ __forceinline__ cx<T> ld_stream(const cx<T>* p) { return __ldcg(p); }

// Where the tiles of a pass come from.  OneGrid: the x tiles of one handle's
// lines, the components one after the other in single-component passes.
template <typename T, int MS, int TX, int KIND> struct OneGrid {
    static constexpr bool many = false, KOP = KIND >= COLK_Y2D;
    const StepConst& k;
    const ColArgs& a;
    int nxt, per;
    __device__ __forceinline__ OneGrid(const StepConst& c, const ColArgs& args) : k(c), a(args) {
        nxt = (c.nx + TX - 1) / TX;
        per = nxt * a.n_other;
    }
    __device__ __forceinline__ int tiles() const { return KOP ? per : per * MS; }
    __device__ __forceinline__ const StepConst& c(int) const { return k; }
    __device__ __forceinline__ const void* tw() const { return a.tw; }
    __device__ __forceinline__ long long stride() const { return a.axis_stride; }
    __device__ __forceinline__ int comp(int tile) const { return KOP ? 0 : tile / per; }
    __device__ __forceinline__ int other(int tile) const { return (KOP ? tile : tile % per) / nxt; }
    __device__ __forceinline__ int x0(int tile) const { return (KOP ? tile : tile % per) % nxt * TX; }
    __device__ __forceinline__ int ky(int tile) const { return a.fother[other(tile)]; }
    __device__ __forceinline__ cx<T>* S(int tile) const {
        return (cx<T>*)a.S + (size_t)comp(tile) * k.npts + (long long)other(tile) * a.other_stride + x0(tile);
    }
    __device__ __forceinline__ T scale(int, int m) const { return (T)(a.info[INFO_SC + m] * a.cfac); }
};
// ManyGrids: the x tiles of every instance of a group of q2D instances of one
// shape (fgpe_group.cuh), one instance after the other.
template <typename T, int TX> struct ManyGrids {
    static constexpr bool many = true;
    const InstDesc* d;
    int ninst, per, nx;
    __device__ __forceinline__ ManyGrids(const GroupArgs& g) : d(g.d), ninst(g.ninst), per(g.tiles), nx(g.d[0].c.nx) {}
    __device__ __forceinline__ int tiles() const { return ninst * per; }
    __device__ __forceinline__ const StepConst& c(int tile) const { return d[tile / per].c; }
    __device__ __forceinline__ const void* tw() const { return d[0].c.twy; }     // one line length: one table
    __device__ __forceinline__ long long stride() const { return nx; }
    __device__ __forceinline__ int comp(int) const { return 0; }
    __device__ __forceinline__ int x0(int tile) const { return tile % per * TX; }
    __device__ __forceinline__ int ky(int) const { return 0; }
    __device__ __forceinline__ cx<T>* S(int tile) const { return (cx<T>*)d[tile / per].S + x0(tile); }
    __device__ __forceinline__ T scale(int tile, int m) const {
        return (T)(d[tile / per].info[INFO_SC + m] * (1.0 / (double)d[0].c.npts));
    }
};

template <typename T, int MS, int N, int TX, int TH, class PL, int KIND, bool KEZ, class Src>
__device__ __forceinline__ void regcol_tiles(const Src& src) {
    static_assert(PL::N == N, "plan length");
    constexpr bool KOP = KIND >= COLK_Y2D;
    constexpr int R0 = PL::R0, RL = PL::RL, S0 = N / R0, NQ = N / RL;
    using TL = RegTile<T, TX, RL>;
    constexpr int LINE = TL::rows(N) * TX;           // one component's tile
    constexpr int T0 = S0 * TX, TF = NQ * TX;        // butterflies of the first / last pass per component
    // components one thread takes through the outer passes together: all of
    // them, on one set of twiddles, where that still occupies every thread
    constexpr int CNT = KOP && T0 % TH == 0 && R0 <= 16 && MS * R0 <= 48 ? MS : 1;
    constexpr int TOT0 = KOP ? MS / CNT * T0 : T0;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T>* sm = (cx<T>*)smraw;
    const StepConst& c0 = src.c(0);
    // z pass: exp(-i CDT (kz^2 - 2 L GAMMAZ kz)) per component
    const cx<T>* kez = KEZ ? sm + MS * LINE : (const cx<T>*)c0.kez;
    const long long np = c0.npts;
    const int nx = c0.nx;
    const cx<T>* tw = (const cx<T>*)src.tw();
    const long long st = src.stride();
    const int ntiles = src.tiles();
    constexpr bool SCALED = KIND == COLK_FWD || KIND == COLK_Y2D;
    T fac[MS];
#pragma unroll
    for (int m = 0; m < MS; ++m) fac[m] = SCALED && !Src::many ? src.scale(0, m) : (T)1;

    // where a thread's butterfly is the same in every tile, its twiddles stay
    // in registers
    constexpr bool KEEPW = T0 == TH;
    Twiddles<T, R0> wq;
    if constexpr (KEEPW) wq.load(tw, (threadIdx.x / TX) % S0, 1);
    if constexpr (KEZ) {
        for (int i = threadIdx.x; i < MS * N; i += TH) sm[MS * LINE + i] = ((const cx<T>*)c0.kez)[i];
    }
    // passes with the operators: a butterfly's slots of the first forward and
    // of the last inverse pass belong to one thread, which refills them with
    // the next tile's elements as soon as it has read the last pass's, so the
    // copies overlap that pass's arithmetic and stores
    auto fetch = [&](int tile, int m, int q, int t) {
        if (t > nx - 1 - src.x0(tile)) return;
        const cx<T>* g = src.S(tile) + (size_t)m * np + t + (long long)q * st;
#pragma unroll
        for (int r = 0; r < R0; ++r) cp_elem<T>(sm + m * LINE + TL::at(q + r * S0, t), g + (long long)(r * S0) * st);
    };
    if constexpr (KOP) {
        if (blockIdx.x < ntiles) {
#pragma unroll 1
            for (int b = threadIdx.x; b < MS * T0; b += TH) fetch(blockIdx.x, b / T0, (b / TX) % S0, b % TX);
        }
        cp_commit();
    }
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const StepConst& c = src.c(tile);
        const int imag = c.imag;
        const int x0 = src.x0(tile);
        cx<T>* S = src.S(tile);
        const int last = nx - 1 - x0;              // tile columns past it are absent (nx not a multiple of TX)
        if constexpr (SCALED && Src::many) {
#pragma unroll
            for (int m = 0; m < MS; ++m) fac[m] = src.scale(tile, m);
        }
        T fc = (T)1;
        if constexpr (KIND == COLK_FWD) {
#pragma unroll
            for (int m = 0; m < MS; ++m) fc = src.comp(tile) == m ? fac[m] : fc;
        }
        // a thread keeps its line (TH is a multiple of TX), so the line's kx part
        // of KE, and on z lines, where (kx, ky) is fixed, its ky part and its
        // SO-coupling numbers come once per tile, ahead of their use
        static_assert(TH % TX == 0, "threads per tile row");
        const int xt = x0 + min((int)threadIdx.x % TX, last);
        const Soc4<T>* soc = (const Soc4<T>*)c.soc;
        cx<T> ke;
        Soc4<T> so;
        if constexpr (KOP) ke = ((const cx<T>*)c.kex)[c.fx[xt]];
        if constexpr (KIND == COLK_Z3D) {
            const int iy = src.ky(tile);
            ke = fmul(imag, ke, ((const cx<T>*)c.key)[iy]);
            if (soc) so = soc[(size_t)iy * nx + xt];
        }
        if constexpr (KIND != COLK_INV) {
            // first forward pass; without the operators from global memory
            if constexpr (KOP) cp_wait<0>();
#pragma unroll 1
            for (int b = threadIdx.x; b < TOT0; b += TH) {
                const int t = b % TX, w = b / TX, q = w % S0, m0 = w / S0;
                cx<T>* d = sm + m0 * LINE;
                cx<T> v[CNT][R0];
#pragma unroll
                for (int m = 0; m < CNT; ++m) {
                    if constexpr (KOP) {
#pragma unroll
                        for (int r = 0; r < R0; ++r) v[m][r] = d[m * LINE + TL::at(q + r * S0, t)];
                    } else {
                        const cx<T>* g = S + (long long)q * st + t;
#pragma unroll
                        for (int r = 0; r < R0; ++r) v[0][r] = t <= last ? ld_stream<T>(g + (long long)(r * S0) * st) : mk<T>(0, 0);
#pragma unroll
                        for (int r = 0; r < R0; ++r) v[0][r] = cscale(v[0][r], fc);
                    }
                    Dft<T, false, R0>::run(v[m]);
                }
                if constexpr (!KEEPW) wq.load(tw, q, 1);
                if (q) wq.template apply<false, CNT>(v);
#pragma unroll
                for (int m = 0; m < CNT; ++m)
#pragma unroll
                    for (int r = 0; r < R0; ++r) d[m * LINE + TL::at(q + r * S0, t)] = v[m][r];
            }
            __syncthreads();
            if constexpr (PL::three) {
                constexpr int R1 = PL::R1, S1 = S0 / R1, NB = N / R1;
                constexpr int TOT1 = (KOP ? MS : 1) * NB * TX;
#pragma unroll 1
                for (int b = threadIdx.x; b < TOT1; b += TH) {
                    const int t = b % TX, w = b / TX, q = w % NB, m = w / NB;
                    const int blk = q / S1, n2 = q - blk * S1, e0 = blk * S0 + n2;
                    cx<T>* d = sm + m * LINE;
                    cx<T> v[1][R1];
#pragma unroll
                    for (int r = 0; r < R1; ++r) v[0][r] = d[TL::at(e0 + r * S1, t)];
                    Dft<T, false, R1>::run(v[0]);
                    Twiddles<T, R1> w1;
                    w1.load(tw, n2, R0);
                    if (n2) w1.template apply<false, 1>(v);
#pragma unroll
                    for (int r = 0; r < R1; ++r) d[TL::at(e0 + r * S1, t)] = v[0][r];
                }
                __syncthreads();
            }
        }
        if constexpr (KOP) {
            // last forward pass, k-space operators, first inverse pass
            auto operators = [&](auto time) {
            const int im = time;
#pragma unroll 1
            for (int b = threadIdx.x; b < TF; b += TH) {
                const int t = b % TX, q = b / TX;
                cx<T> v[MS][RL];
#pragma unroll
                for (int m = 0; m < MS; ++m) {
#pragma unroll
                    for (int r = 0; r < RL; ++r) v[m][r] = sm[m * LINE + TL::at(q * RL + r, t)];
                    Dft<T, false, RL>::run(v[m]);
                }
                const int kq = PL::krev(q);
                if constexpr (KIND == COLK_Z3D) {
#pragma unroll
                    for (int r = 0; r < RL; ++r) {
                        cx<T> u[MS];
#pragma unroll
                        for (int m = 0; m < MS; ++m) u[m] = fmul(im, fmul(im, ke, kez[m * N + kq + r * NQ]), v[m][r]);
                        if (soc) soc_apply<T, MS>(im, so, u);
#pragma unroll
                        for (int m = 0; m < MS; ++m) v[m][r] = u[m];
                    }
                } else {
                    const cx<T>* key = (const cx<T>*)c.key;
#pragma unroll
                    for (int r = 0; r < RL; ++r) {
                        const int iy = kq + r * NQ;
                        const cx<T> f = fmul(im, ke, key[iy]);
                        cx<T> u[MS];
#pragma unroll
                        for (int m = 0; m < MS; ++m) u[m] = fmul(im, f, cscale(v[m][r], fac[m]));
                        if (soc) soc_apply<T, MS>(im, soc[(size_t)iy * nx + xt], u);
#pragma unroll
                        for (int m = 0; m < MS; ++m) v[m][r] = u[m];
                    }
                }
#pragma unroll
                for (int m = 0; m < MS; ++m) {
                    Dft<T, true, RL>::run(v[m]);
#pragma unroll
                    for (int r = 0; r < RL; ++r) sm[m * LINE + TL::at(q * RL + r, t)] = v[m][r];
                }
            }
            };
            // one body per time direction (the factors of imaginary time are
            // real), except where two spill: 256^3 FP64 spin-1 z pass in real
            // time 447 us with one, 529 with two; elsewhere two are faster (FP32
            // 260 -> 248, q2D 512^2 FP64 20.7 -> 18.9)
            if constexpr (sizeof(T) == 8 && MS == 3 && KIND == COLK_Z3D) operators(imag);
            else if (imag) operators(std::integral_constant<int, 1>{});
            else operators(std::integral_constant<int, 0>{});
            __syncthreads();
        } else if constexpr (KIND == COLK_FWD) {
            // last forward pass, to global memory in position order
#pragma unroll 1
            for (int b = threadIdx.x; b < TF; b += TH) {
                const int t = b % TX, q = b / TX;
                cx<T> v[RL];
#pragma unroll
                for (int r = 0; r < RL; ++r) v[r] = sm[TL::at(q * RL + r, t)];
                Dft<T, false, RL>::run(v);
                cx<T>* g = S + (long long)(q * RL) * st + t;
                if (t <= last) {
#pragma unroll
                    for (int r = 0; r < RL; ++r) g[(long long)r * st] = v[r];
                }
            }
            __syncthreads();
        } else {
            // first inverse pass, from global memory
#pragma unroll 1
            for (int b = threadIdx.x; b < TF; b += TH) {
                const int t = b % TX, q = b / TX;
                const cx<T>* g = S + (long long)(q * RL) * st + t;
                cx<T> v[RL];
#pragma unroll
                for (int r = 0; r < RL; ++r) v[r] = t <= last ? ld_stream<T>(g + (long long)r * st) : mk<T>(0, 0);
                Dft<T, true, RL>::run(v);
#pragma unroll
                for (int r = 0; r < RL; ++r) sm[TL::at(q * RL + r, t)] = v[r];
            }
            __syncthreads();
        }
        if constexpr (KIND != COLK_FWD) {
            if constexpr (PL::three) {
                constexpr int R1 = PL::R1, S1 = S0 / R1, NB = N / R1;
                constexpr int TOT1 = (KOP ? MS : 1) * NB * TX;
#pragma unroll 1
                for (int b = threadIdx.x; b < TOT1; b += TH) {
                    const int t = b % TX, w = b / TX, q = w % NB, m = w / NB;
                    const int blk = q / S1, n2 = q - blk * S1, e0 = blk * S0 + n2;
                    cx<T>* d = sm + m * LINE;
                    cx<T> v[1][R1];
#pragma unroll
                    for (int r = 0; r < R1; ++r) v[0][r] = d[TL::at(e0 + r * S1, t)];
                    Twiddles<T, R1> w1;
                    w1.load(tw, n2, R0);
                    if (n2) w1.template apply<true, 1>(v);
                    Dft<T, true, R1>::run(v[0]);
#pragma unroll
                    for (int r = 0; r < R1; ++r) d[TL::at(e0 + r * S1, t)] = v[0][r];
                }
                __syncthreads();
            }
            // last inverse pass, to global memory
#pragma unroll 1
            for (int b = threadIdx.x; b < TOT0; b += TH) {
                const int t = b % TX, w = b / TX, q = w % S0, m0 = w / S0;
                const cx<T>* d = sm + m0 * LINE;
                cx<T> v[CNT][R0];
#pragma unroll
                for (int m = 0; m < CNT; ++m)
#pragma unroll
                    for (int r = 0; r < R0; ++r) v[m][r] = d[m * LINE + TL::at(q + r * S0, t)];
                if constexpr (KOP) {
                    if (tile + (int)gridDim.x < ntiles)
#pragma unroll
                        for (int m = 0; m < CNT; ++m) fetch(tile + gridDim.x, m0 + m, q, t);
                }
                if constexpr (!KEEPW) wq.load(tw, q, 1);
                if (q) wq.template apply<true, CNT>(v);
#pragma unroll
                for (int m = 0; m < CNT; ++m) {
                    Dft<T, true, R0>::run(v[m]);
                    cx<T>* g = S + (size_t)(m0 + m) * np + (long long)q * st + t;
                    if (t <= last) {
#pragma unroll
                        for (int r = 0; r < R0; ++r) g[(long long)(r * S0) * st] = v[m][r];
                    }
                }
            }
            if constexpr (KOP) cp_commit();
            else __syncthreads();
        }
    }
}

template <typename T, int MS, int N, int TX, int TH, int MINB, class PL, int KIND, bool KEZ>
__global__ void __launch_bounds__(TH, MINB) k_regcol(const __grid_constant__ StepConst c, const __grid_constant__ ColArgs a) {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const OneGrid<T, MS, TX, KIND> src(c, a);
    regcol_tiles<T, MS, N, TX, TH, PL, KIND, KEZ>(src);
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// The q2D pass of every instance of a group.
template <typename T, int MS, int N, int TX, int TH, int MINB, class PL>
__global__ void __launch_bounds__(TH, MINB) k_regcol_group(const __grid_constant__ GroupArgs g) {
    const ManyGrids<T, TX> src(g);
    regcol_tiles<T, MS, N, TX, TH, PL, COLK_Y2D, false>(src);
}

// ------------------------------------------------------- launch shapes
template <typename T, int MS, int N, int KIND, bool BIG> struct ColShape {
    using P = typename ColPlan<MS, N, KIND, BIG>::P;
    static constexpr bool KOP = KIND >= COLK_Y2D, F64 = sizeof(T) == 8;
    static constexpr bool SMALL = KIND == COLK_Y2D || (KIND == COLK_Z3D && !BIG);
    // x positions per tile.  Single-component passes: 128 bytes.  Big z
    // tiles: the widest that leaves room for two (FP64) or three (FP32)
    // blocks per SM.  Small tiles: 2 positions, 4 where FP32 lines are long.
    static constexpr int ROOM = F64 ? 108 * 1024 : 74 * 1024;
    static constexpr int TXB = !KOP || MS * N * 128 <= ROOM ? 128 : MS * N * 64 <= ROOM ? 64 : 32;
    // q2D, five components, 192 and 256 points: one block of 256 threads takes
    // an SM's registers, so grids of more than two x positions per SM (BIG)
    // would run a second, nearly empty wave.  They take half the threads and
    // two blocks (FP64), or four positions a tile (FP32): 512 x 256, us a step,
    // one form / this one: FP64 36.6 / 33.0, FP32 30.8 / 24.7
    static constexpr bool MANY = KIND == COLK_Y2D && BIG && MS == 5 && (N == 192 || N == 256);
    static constexpr int TX = SMALL ? (!F64 && (N >= 384 || MANY) ? 4 : 2) : TXB / (int)sizeof(cx<T>);
    // threads: one butterfly of the operator pass (or of the wider pass of a
    // single-component kernel) each
    static constexpr int TASKS = TX * (KOP ? N / P::RL : 16);
    static constexpr int TH = SMALL ? (N == 128 || (F64 && (N >= 384 || MANY)) ? 128 : 256) : TASKS < 64 ? 64 : (TASKS + 31) / 32 * 32;
    // threads per SM that share the register file
    static constexpr int PER_SM = SMALL ? (F64 || MS == 5 ? 256 : 512)
                                  : KOP ? (F64 ? 256 : 384)
                                        : (F64 ? (P::R0 > 16 ? 256 : 512) : (P::R0 > 16 ? 512 : 768));
    static constexpr int MINB0 = PER_SM / TH < 1 ? 1 : PER_SM / TH;
    static constexpr int fit(size_t smem) {
        const int f = (int)((226 * 1024) / (smem + 1024));
        return f < 1 ? 1 : f < MINB0 ? f : MINB0;
    }
    // the z pass keeps the kz part of KE in shared memory, except where that
    // costs a resident block (512-point FP64 lines: one block of 128 threads
    // per SM, spin-2 z pass of 3072 lines 162 us against 121)
    static constexpr bool KEZ = KIND == COLK_Z3D && fit(regcol_smem<T, MS, N, TX, P, KIND, true>()) ==
                                                        fit(regcol_smem<T, MS, N, TX, P, KIND, false>());
    static constexpr size_t SMEM = regcol_smem<T, MS, N, TX, P, KIND, KEZ>();
    static constexpr int MINB = fit(SMEM);
    static constexpr auto kernel() { return k_regcol<T, MS, N, TX, TH, MINB, P, KIND, KEZ>; }
};

}  // namespace fgpe
