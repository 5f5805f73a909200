// fgpe_regrow.cuh -- the row pass with its transforms in registers.
//
// An x line of N = 8 M points is a radix-8 pass over elements M apart and
// eight transforms of M adjacent positions (the handle's spectral order: the
// frequencies k = d mod 8 fill the d-th block of M).  One warp takes RW rows
// through the pass.  The block transforms run whole in a thread's registers
// (FP32) or as radix 8 and radix M/8 (FP64, and 512-point lines); between the
// inverse and the forward transform a thread holds all MS components of eight
// points, so the radix-8 passes share one set of twiddles and SE, SP and the
// NORMC terms see the points in slots that are the thread's own.  The last
// pass stores 32-byte pieces from registers.  Shared memory is private to
// the warp: after it has read its rows for the last time it starts the copy
// of its next ones and transforms and stores the old ones meanwhile.  Nothing
// but __syncwarp orders these steps.
//
// Bound by FP64 issue (256^3 spin-1: about 300 FP64 operations a point, that
// pipe half busy) or, in FP32, by issue and latency.  One B200, 65536 rows of
// 256 spin-1 points: FP64 0.72 (k_row_warp) -> 0.55 ms, of which the shorter
// SE and SP are 0.1; FP32 0.57 (k_row_fast) -> 0.32 ms.  Unrolling the point
// loop (two or more points in flight, or all eight in registers) spilled and
// was slower.
#pragma once
#include "fgpe_async.cuh"
#include "fgpe_dft.cuh"
#include "fgpe_group.cuh"
#include "fgpe_kernels.cuh"

namespace fgpe {

template <typename T, bool INV> struct Dft<T, INV, 48> : DftAB<T, INV, 3, 16> {};

// Position p of an M-point block in the handle's order (cplan of 8 M without
// its first radix) -> frequency within the block.
template <int M> constexpr int block_freq(int p) {
    // remaining radices: 16 = 8*2, 24 = 8*3, 32 = 8*4, 48 = 8*2*3
    if (M == 48) return p / 6 + 8 * ((p / 3) % 2) + 16 * (p % 3);
    constexpr int r = M / 8;
    return p / r + 8 * (p % r);
}
// Position within the last radix (6 = 2*3) -> frequency.
template <int R> constexpr int last_freq(int p) { return R == 6 ? p / 3 + 2 * (p % 3) : p; }

template <typename T, int N> struct RegRow {
    static constexpr int M = N / 8;
    // M-point transforms: whole in one thread's registers (FP32 up to 48
    // points), or as a radix-8 pass over elements M/8 apart and M/8-point
    // transforms, with an exchange between them
    static constexpr bool two = sizeof(T) == 8 || M > 48;
    // block stride in shared memory.  Whole blocks: an odd number of 16-byte
    // units, so that threads reading their own blocks fall on distinct banks;
    // two passes: one spare slot every eight does that for both
    static constexpr int SL = two ? M + M / 8 : M + 2;
    static __host__ __device__ constexpr int at(int i) { return two ? i + i / 8 : i; }
};
template <typename T, int MS, int N, int RW> constexpr size_t regrow_warp_smem() {
    return (size_t)RW * MS * 8 * RegRow<T, N>::SL * sizeof(cx<T>);
}

// 32 bytes of a row: two complex doubles or four complex floats
__device__ __forceinline__ void st32(double2* p, const double2* v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "d"(v[0].x), "d"(v[0].y), "d"(v[1].x), "d"(v[1].y) : "memory");
}
__device__ __forceinline__ void st32(float2* p, const float2* v) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(p), "f"(v[0].x), "f"(v[0].y), "f"(v[1].x),
                 "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y) : "memory");
}

// a thread's own block: 16-byte accesses
template <int M> __device__ __forceinline__ void ld_block(double2 (&v)[M], const double2* s) {
    static_for<0, M>([&](auto p) { v[block_freq<M>(p)] = s[p]; });
}
template <int M> __device__ __forceinline__ void ld_block(float2 (&v)[M], const float2* s) {
    static_for<0, M / 2>([&](auto p) {
        const float4 q = *(const float4*)(s + 2 * p);
        v[block_freq<M>(2 * p)] = make_float2(q.x, q.y);
        v[block_freq<M>(2 * p + 1)] = make_float2(q.z, q.w);
    });
}
// natural order: the points between the radix-8 pass and the block transforms
template <int M> __device__ __forceinline__ void ld_points(double2 (&v)[M], const double2* s) {
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = s[i];
}
template <int M> __device__ __forceinline__ void ld_points(float2 (&v)[M], const float2* s) {
#pragma unroll
    for (int i = 0; i < M; i += 2) {
        const float4 q = *(const float4*)(s + i);
        v[i] = make_float2(q.x, q.y);
        v[i + 1] = make_float2(q.z, q.w);
    }
}
template <int M> __device__ __forceinline__ void st_points(const double2 (&v)[M], double2* s) {
#pragma unroll
    for (int i = 0; i < M; ++i) s[i] = v[i];
}
template <int M> __device__ __forceinline__ void st_points(const float2 (&v)[M], float2* s) {
#pragma unroll
    for (int i = 0; i < M; i += 2) *(float4*)(s + i) = make_float4(v[i].x, v[i].y, v[i + 1].x, v[i + 1].y);
}

// Where a pass's rows come from: batches of RW rows.  OneSpinor: the rows of
// one handle; its NORMC terms are summed over the grid at the end.
template <typename T> struct OneSpinor {
    static constexpr bool many = false;
    const StepConst& k;
    const RowArgs& a;
    int nrows;
    __device__ __forceinline__ OneSpinor(const StepConst& c, const RowArgs& args) : k(c), a(args), nrows(c.ny * c.nz) {}
    __device__ __forceinline__ int batches(int rw) const { return (nrows + rw - 1) / rw; }
    __device__ __forceinline__ int next(int batch, int nw) const { return batch + nw; }
    __device__ __forceinline__ int first(int warp) const { return warp; }
    __device__ __forceinline__ const StepConst& c(int) const { return k; }
    __device__ __forceinline__ cx<T>* S(int) const { return (cx<T>*)a.S; }
    __device__ __forceinline__ cx<T>* snap(int) const { return (cx<T>*)a.snap; }
    __device__ __forceinline__ int row0(int batch, int rw) const { return batch * rw; }
};
// ManySpinors: the rows of every instance of a group, in chunks of
// consecutive batches of one instance; the warp that ends a chunk leaves its
// NORMC terms in the instance's slot for it.
template <typename T> struct ManySpinors {
    static constexpr bool many = true;
    const GroupArgs& g;
    int nrows, per;             // rows and batches of an instance
    __device__ __forceinline__ ManySpinors(const GroupArgs& a) : g(a), nrows(a.d[0].c.ny), per(a.tiles) {}
    __device__ __forceinline__ int batches(int) const { return g.ninst * per; }
    __device__ __forceinline__ int next(int batch, int nw) const {
        return (batch + 1) % g.chunk ? batch + 1 : batch + 1 + (nw - 1) * g.chunk;
    }
    __device__ __forceinline__ int first(int warp) const { return warp * g.chunk; }
    __device__ __forceinline__ const InstDesc& inst(int batch) const { return g.d[batch / per]; }
    __device__ __forceinline__ const StepConst& c(int batch) const { return inst(batch).c; }
    __device__ __forceinline__ cx<T>* S(int batch) const { return (cx<T>*)inst(batch).S; }
    __device__ __forceinline__ cx<T>* snap(int batch) const {
        return g.snap == 1 ? (cx<T>*)inst(batch).psi : g.snap == 2 ? (cx<T>*)inst(batch).prev : nullptr;
    }
    __device__ __forceinline__ int row0(int batch, int rw) const { return batch % per * rw; }
    // the chunk that ends with this batch is done
    template <int MS> __device__ __forceinline__ void flush(int batch, double (&acc)[MS]) const {
        if ((batch + 1) % g.chunk) return;
        warp_finish_norms<MS>(inst(batch), batch % per / g.chunk, per / g.chunk, g.snap == 2, acc);
    }
};

template <typename T, int MS, int N, int RW, int WPB, class Src>
__device__ __forceinline__ void regrow_rows(const Src& src, double (&acc)[MS]) {
    constexpr int M = RegRow<T, N>::M, SL = RegRow<T, N>::SL;
    using L = RegRow<T, N>;
    constexpr int NSUB = RW * MS * 8, NPT = RW * M;   // block transforms, radix-8 butterflies (of MS components)
    constexpr int RB = M / 8;                         // last radix of a block in two passes
    constexpr int V = 32 / (int)sizeof(cx<T>);        // elements per 32-byte store
    extern __shared__ __align__(16) unsigned char smraw[];
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    cx<T>* s = (cx<T>*)smraw + (size_t)warp * RW * MS * 8 * SL;
    const StepConst& c0 = src.c(0);
    const long long np = c0.npts;
    const int nrows = src.nrows, nw = (int)gridDim.x * WPB, nb = src.batches(RW);
    const cx<T>* tw = (const cx<T>*)c0.twx;

    // a batch's rows into this warp's blocks
    auto fetch = [&](int batch) {
        constexpr int E = L::two ? 1 : 16 / (int)sizeof(cx<T>), PER = N / E;
        static_assert(M % E == 0, "16-byte chunks stay inside a block");
#pragma unroll
        for (int q = 0; q < RW * MS; ++q) {
            const int rr = q / MS, m = q - rr * MS;
            const int row = src.row0(batch, RW) + rr;
            // (axes are even, so batches of two rows are whole: the checks on
            // nrows hold for any RW)
            if (RW > 1 && row >= nrows) break;
            const cx<T>* g = src.S(batch) + (size_t)m * np + (size_t)row * N;
#pragma unroll
            for (int i = 0; i < (PER + 31) / 32; ++i) {
                const int x = (lane + 32 * i) * E;
                if (PER % 32 == 0 || x < N) {
                    cx<T>* d = s + (q * 8 + x / M) * SL + L::at(x % M);
                    if constexpr (L::two) cp_elem<T>(d, g + x);
                    else cp16(d, g + x);
                }
            }
        }
    };
    // a thread keeps its points from row to row, and their twiddles
    constexpr bool KEEPW = NPT <= 32;
    Twiddles<T, 8> wq;
    if constexpr (KEEPW) wq.load(tw, lane % M, 1);

    int batch = src.first((int)blockIdx.x * WPB + warp);
    if (batch < nb) fetch(batch);
    cp_commit();
    while (batch < nb) {
        // a group's constants come from memory once per batch, one handle's are
        // the kernel's parameters
        std::conditional_t<Src::many, const StepConst, const StepConst&> c = src.c(batch);
        cx<T>* S = src.S(batch);
        cx<T>* snap = src.snap(batch);
        const int row0 = src.row0(batch, RW), nxt = src.next(batch, nw);
        cp_wait<0>();
        __syncwarp();
        if constexpr (!L::two) {
#pragma unroll 1
            for (int b = lane; b < NSUB; b += 32) {
                cx<T> v[M];
                ld_block<M>(v, s + b * SL);
                Dft<T, true, M>::run(v);
                st_points<M>(v, s + b * SL);
            }
        } else {
#pragma unroll 2
            for (int b = lane; b < NSUB * 8; b += 32) {
                cx<T>* d = s + (b / 8) * SL;
                const int e = (b % 8) * RB;
                cx<T> v[RB];
#pragma unroll
                for (int r = 0; r < RB; ++r) v[last_freq<RB>(r)] = d[L::at(e + r)];
                Dft<T, true, RB>::run(v);
#pragma unroll
                for (int r = 0; r < RB; ++r) d[L::at(e + r)] = v[r];
            }
            __syncwarp();
#pragma unroll 1
            for (int b = lane; b < NSUB * RB; b += 32) {
                cx<T>* d = s + (b / RB) * SL;
                const int e = b % RB;
                cx<T> v[1][8];
#pragma unroll
                for (int r = 0; r < 8; ++r) v[0][r] = d[L::at(e + r * RB)];
                Twiddles<T, 8> w;
                w.load(tw, e, 8);
                if (e) w.template apply<true, 1>(v);
                Dft<T, true, 8>::run(v[0]);
#pragma unroll
                for (int r = 0; r < 8; ++r) d[L::at(e + r * RB)] = v[0][r];
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int b = lane; b < NPT; b += 32) {
            const int rr = RW == 1 ? 0 : b / M, x0 = RW == 1 ? b : b - rr * M;
            const int row = row0 + rr;
            if (RW > 1 && row >= nrows) break;
            cx<T>* d = s + rr * MS * 8 * SL + L::at(x0);
            if constexpr (!KEEPW) wq.load(tw, x0, 1);
            cx<T> v[MS][8];
#pragma unroll
            for (int m = 0; m < MS; ++m)
#pragma unroll
                for (int r = 0; r < 8; ++r) v[m][r] = d[(m * 8 + r) * SL];
            if (x0) wq.template apply<true, MS>(v);
#pragma unroll
            for (int m = 0; m < MS; ++m) Dft<T, true, 8>::run(v[m]);
            const int j = row % c.ny, k = row / c.ny;
            double wr = 1.0;
            cx<T> pr = mk<T>((T)1, (T)0);
            if (c.dim >= 2) { wr = c.wy[j]; pr = ((const cx<T>*)c.pvy)[j]; }
            if (c.dim >= 3) { wr *= c.wz[k]; pr = fmul(c.imag, pr, ((const cx<T>*)c.pvz)[k]); }
            // the points go back to their slots, which only this thread
            // reads and writes, for a rolled loop
#pragma unroll
            for (int m = 0; m < MS; ++m)
#pragma unroll
                for (int r = 0; r < 8; ++r) d[(m * 8 + r) * SL] = v[m][r];
#pragma unroll 1
            for (int r = 0; r < 8; ++r) {
                const int x = x0 + r * M;
                cx<T> u[MS];
#pragma unroll
                for (int m = 0; m < MS; ++m) u[m] = d[(m * 8 + r) * SL];
                apply_se<T, MS>(c, u);
                apply_sp<T, MS>(c, fmul(c.imag, ((const cx<T>*)c.pvx)[x], pr), u);
                const double w = c.wx[x] * wr;
#pragma unroll
                for (int m = 0; m < MS; ++m) {
                    acc[m] += w * ((double)u[m].x * (double)u[m].x + (double)u[m].y * (double)u[m].y);
                    d[(m * 8 + r) * SL] = u[m];
                    if (snap) snap[(size_t)m * np + (size_t)row * N + x] = u[m];
                }
            }
#pragma unroll
            for (int m = 0; m < MS; ++m)
#pragma unroll
                for (int r = 0; r < 8; ++r) v[m][r] = d[(m * 8 + r) * SL];
#pragma unroll
            for (int m = 0; m < MS; ++m) Dft<T, false, 8>::run(v[m]);
            if (x0) wq.template apply<false, MS>(v);
#pragma unroll
            for (int m = 0; m < MS; ++m)
#pragma unroll
                for (int r = 0; r < 8; ++r) d[(m * 8 + r) * SL] = v[m][r];
        }
        if constexpr (L::two) {
            __syncwarp();
#pragma unroll 1
            for (int b = lane; b < NSUB * RB; b += 32) {
                cx<T>* d = s + (b / RB) * SL;
                const int e = b % RB;
                cx<T> v[1][8];
#pragma unroll
                for (int r = 0; r < 8; ++r) v[0][r] = d[L::at(e + r * RB)];
                Dft<T, false, 8>::run(v[0]);
                Twiddles<T, 8> w;
                w.load(tw, e, 8);
                if (e) w.template apply<false, 1>(v);
#pragma unroll
                for (int r = 0; r < 8; ++r) d[L::at(e + r * RB)] = v[0][r];
            }
            __syncwarp();
            // the last pass: a row's blocks are read RB values per thread
            constexpr int IT = NSUB * 8 / 32;
            static_assert(NSUB * 8 % 32 == 0, "whole warps of last-radix butterflies");
            constexpr int STEP = RB <= 4 ? 2 : 1;
#pragma unroll 1
            for (int i0 = 0; i0 < IT; i0 += STEP) {
                cx<T> v[STEP][RB];
#pragma unroll
                for (int k = 0; k < STEP; ++k) {
                    const int b = lane + (i0 + k) * 32;
#pragma unroll
                    for (int r = 0; r < RB; ++r) v[k][r] = s[(b / 8) * SL + L::at((b % 8) * RB + r)];
                }
                if (i0 + STEP >= IT) {
                    // every block has been read: the next rows may come in
                    __syncwarp();
                    if (nxt < nb) fetch(nxt);
                    cp_commit();
                }
#pragma unroll
                for (int k = 0; k < STEP; ++k) {
                    const int b = lane + (i0 + k) * 32;
                    const int q = b / 64, rr = q / MS, m = q - rr * MS, row = row0 + rr;
                    Dft<T, false, RB>::run(v[k]);
                    if (RW == 1 || row < nrows) {
                        cx<T>* g = S + (size_t)m * np + (size_t)row * N + (b % 64) * RB;
                        if constexpr (RB % V == 0) {
                            static_for<0, RB / V>([&](auto i) {
                                cx<T> o[V];
#pragma unroll
                                for (int e = 0; e < V; ++e) o[e] = v[k][last_freq<RB>(i * V + e)];
                                st32(g + i * V, o);
                            });
                        } else {
                            static_for<0, RB>([&](auto i) { g[i] = v[k][last_freq<RB>(i)]; });
                        }
                    }
                }
            }
        } else {
            __syncwarp();
#pragma unroll 1
            for (int b0 = 0; b0 < NSUB; b0 += 32) {
                const int b = b0 + lane;
                const bool on = b < NSUB;
                cx<T> v[M];
                if (on) ld_points<M>(v, s + b * SL);
                if (b0 + 32 >= NSUB) {
                    // every block has been read: the next rows may come in
                    __syncwarp();
                    if (nxt < nb) fetch(nxt);
                    cp_commit();
                }
                if (on) {
                    Dft<T, false, M>::run(v);
                    const int q = b / 8, rr = q / MS, m = q - rr * MS, row = row0 + rr;
                    if (RW == 1 || row < nrows) {
                        cx<T>* g = S + (size_t)m * np + (size_t)row * N + (b % 8) * M;
                        static_for<0, M / V>([&](auto i) {
                            cx<T> o[V];
#pragma unroll
                            for (int e = 0; e < V; ++e) o[e] = v[block_freq<M>(i * V + e)];
                            st32(g + i * V, o);
                        });
                    }
                }
            }
        }
        if constexpr (Src::many) src.template flush<MS>(batch, acc);
        batch = nxt;
    }
    cp_wait<0>();
}

template <typename T, int MS, int N, int RW, int WPB, int MINB>
__global__ void __launch_bounds__(WPB * 32, MINB) k_regrow(const __grid_constant__ StepConst c, const __grid_constant__ RowArgs a) {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    __shared__ double red[32 * (MS + 1)];
    __shared__ double bsum[MS];
    double acc[MS];
#pragma unroll
    for (int m = 0; m < MS; ++m) acc[m] = 0.0;
    const OneSpinor<T> src(c, a);
    regrow_rows<T, MS, N, RW, WPB>(src, acc);
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    block_sum<MS>(acc, red, bsum);
    if (threadIdx.x < MS) a.part[(size_t)blockIdx.x * MS + threadIdx.x] = bsum[threadIdx.x];
    finish_norms<MS>(c, a.part, a.counter, a.info, red);
}

// The row pass of every instance of a group (g.tiles batches of RW rows each).
template <typename T, int MS, int N, int RW, int WPB, int MINB>
__global__ void __launch_bounds__(WPB * 32, MINB) k_regrow_group(const __grid_constant__ GroupArgs g) {
    double acc[MS];
#pragma unroll
    for (int m = 0; m < MS; ++m) acc[m] = 0.0;
    const ManySpinors<T> src(g);
    regrow_rows<T, MS, N, RW, WPB>(src, acc);
}

// ------------------------------------------------------- launch shapes
// Rows per warp, warps per block, blocks per SM, as measured.  RW = 0: not
// available (FP64 512-point rows take 28 KB a warp, too few per SM: 0.93 ms
// against 0.83 for the block pass on 36864 rows).
template <typename T, int N> struct RowShape {
    static constexpr bool F64 = sizeof(T) == 8;
    static constexpr int RW = F64 && N == 512 ? 0 : N == 128 ? 2 : 1;
    static constexpr int WPB = F64 && N == 384 ? 2 : 4;
    static constexpr int MINB = F64 ? (N == 384 ? 5 : 4) : (N == 256 || N == 384 ? 3 : 4);
};

}  // namespace fgpe
