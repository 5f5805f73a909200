// fgpe_step_impl.cuh -- definitions of the pass launchers of fgpe_step.h,
// included by one translation unit per (precision, spin).
#pragma once
#include "fgpe_fast.cuh"
#include "fgpe_regcol.cuh"
#include "fgpe_regrow.cuh"
#include "fgpe_step.h"

namespace fgpe {

#define FGPE_STEP_SIZES(CALL) CALL(128) CALL(192) CALL(256) CALL(384) CALL(512)

template <typename T, int MS, int N, int KIND> int regcol_grid_n(int nx, int n_other, int* wide) {
    using W = ColShape<T, MS, N, KIND, true>;
    using S = ColShape<T, MS, N, KIND, false>;
    const int ncomp = KIND >= COLK_Y2D ? 1 : MS;
    const long long tw = (long long)((nx + W::TX - 1) / W::TX) * n_other * ncomp;
    const int gw = resident_grid(W::kernel(), W::TH, W::SMEM, tw);
    *wide = 1;
    if constexpr (KIND < COLK_Y2D) {
        return gw;
    } else if constexpr (KIND == COLK_Y2D) {
        // the form for many tiles once the other one's take more than one wave
        // (up to there it has more threads on each tile: 256 x 256 FP64 24.4 us)
        const long long ts = (long long)((nx + S::TX - 1) / S::TX) * n_other;
        const int gs = resident_grid(S::kernel(), S::TH, S::SMEM, ts);
        if (gw > 0 && ts > gs) return gw;
        *wide = 0;
        return gs;
    } else {
        // the big tiles once there is one for every SM; fewer leave SMs idle,
        // where the small ones occupy them (us by lines, small / big: 256-point
        // FP64 spin 1: 512 lines, 64 big tiles, 14.6 / 18.7; 1024, 128, 20.9 /
        // 18.8; 2048 31.1 / 22.9; 128-point FP32 spin 1: 1024 12.6 / 14.6, 1536,
        // 96, 14.7 / 14.7, 2048 16.8 / 14.7)
        if (gw > 0 && tw >= sm_count()) return gw;
        *wide = 0;
        return resident_grid(S::kernel(), S::TH, S::SMEM, (long long)((nx + S::TX - 1) / S::TX) * n_other);
    }
}

template <typename T, int MS> int regcol_grid(int n, int kind, int nx, int n_other, int* wide) {
    *wide = 0;
    switch (n) {
#define G(NN)                                                                            \
    case NN:                                                                             \
        return kind == COLK_FWD   ? regcol_grid_n<T, MS, NN, COLK_FWD>(nx, n_other, wide) \
               : kind == COLK_INV ? regcol_grid_n<T, MS, NN, COLK_INV>(nx, n_other, wide) \
               : kind == COLK_Y2D ? regcol_grid_n<T, MS, NN, COLK_Y2D>(nx, n_other, wide) \
                                  : regcol_grid_n<T, MS, NN, COLK_Z3D>(nx, n_other, wide);
        FGPE_STEP_SIZES(G)
#undef G
        default: return 0;
    }
}

template <typename T, int MS, int N, int KIND>
cudaError_t regcol_launch_n(int wide, int grid, const StepConst& c, const ColArgs& a, cudaStream_t st, bool pdl) {
    using W = ColShape<T, MS, N, KIND, true>;
    using S = ColShape<T, MS, N, KIND, false>;
    if constexpr (KIND < COLK_Y2D) {
        return launch_step_kernel(W::kernel(), grid, W::TH, W::SMEM, c, a, st, pdl);
    } else {
        if (wide) return launch_step_kernel(W::kernel(), grid, W::TH, W::SMEM, c, a, st, pdl);
        return launch_step_kernel(S::kernel(), grid, S::TH, S::SMEM, c, a, st, pdl);
    }
}

template <typename T, int MS>
cudaError_t regcol_launch(int n, int kind, int wide, int grid, const StepConst& c, const ColArgs& a, cudaStream_t st,
                          bool pdl) {
    switch (n) {
#define L(NN)                                                                                          \
    case NN:                                                                                           \
        return kind == COLK_FWD   ? regcol_launch_n<T, MS, NN, COLK_FWD>(wide, grid, c, a, st, pdl)    \
               : kind == COLK_INV ? regcol_launch_n<T, MS, NN, COLK_INV>(wide, grid, c, a, st, pdl)    \
               : kind == COLK_Y2D ? regcol_launch_n<T, MS, NN, COLK_Y2D>(wide, grid, c, a, st, pdl)    \
                                  : regcol_launch_n<T, MS, NN, COLK_Z3D>(wide, grid, c, a, st, pdl);
        FGPE_STEP_SIZES(L)
#undef L
        default: return cudaErrorInvalidValue;
    }
}

// Warp-row kernel: rows of MS lines up to 16 KB (FP64 spin-1 to 256 points,
// spin-2 to 128; FP32 spin-1 to 512, spin-2 to 256); warps per block so that
// two blocks of NBUF rows per warp fit the shared memory.
template <typename T, int MS, int N> constexpr size_t wrow_tile() { return (size_t)MS * cpad(N) * sizeof(cx<T>); }
template <typename T, int MS, int N> constexpr bool wrow_ok() { return wrow_tile<T, MS, N>() <= 16 * 1024; }
template <typename T, int MS, int N> constexpr int wrow_wpb() {
    const int w = (int)((110 * 1024) / (wrow_tile<T, MS, N>() * FGPE_WROW_NBUF));
    return w < 1 ? 1 : (w > 8 ? 8 : w);
}

template <typename T, int MS> int row_grid(int n, bool warp, int rows) {
    switch (n) {
#define G(NN)                                                                                                       \
    case NN: {                                                                                                      \
        constexpr int R = row_r(NN), TH = row_th<T, MS, NN>();                                                      \
        if (!warp) return rows % R ? 0 : resident_grid(k_row_fast<T, MS, NN, R, TH>, TH, row_smem<T, MS, NN>(), rows / R); \
        if constexpr (wrow_ok<T, MS, NN>()) {                                                                       \
            constexpr int W = wrow_wpb<T, MS, NN>();                                                                \
            return resident_grid(k_row_warp<T, MS, NN, W, FGPE_WROW_NBUF>, W * 32,                                  \
                                 (size_t)W * FGPE_WROW_NBUF * wrow_tile<T, MS, NN>(), (rows + W - 1) / W);          \
        }                                                                                                           \
        return 0;                                                                                                   \
    }
        FGPE_STEP_SIZES(G)
#undef G
        default: return 0;
    }
}

template <typename T, int MS>
cudaError_t row_launch(int n, bool warp, int grid, const StepConst& c, const RowArgs& a, cudaStream_t st, bool pdl) {
    switch (n) {
#define L(NN)                                                                                                       \
    case NN: {                                                                                                      \
        constexpr int R = row_r(NN), TH = row_th<T, MS, NN>();                                                      \
        if (!warp) return launch_step_kernel(k_row_fast<T, MS, NN, R, TH>, grid, TH, row_smem<T, MS, NN>(), c, a, st, pdl); \
        if constexpr (wrow_ok<T, MS, NN>()) {                                                                       \
            constexpr int W = wrow_wpb<T, MS, NN>();                                                                \
            return launch_step_kernel(k_row_warp<T, MS, NN, W, FGPE_WROW_NBUF>, grid, W * 32,                       \
                                      (size_t)W * FGPE_WROW_NBUF * wrow_tile<T, MS, NN>(), c, a, st, pdl);          \
        }                                                                                                           \
        return cudaErrorInvalidValue;                                                                               \
    }
        FGPE_STEP_SIZES(L)
#undef L
        default: return cudaErrorInvalidValue;
    }
}

template <typename T> int regrow_grid(int n, int rows) {
    switch (n) {
#define G(NN)                                                                                                       \
    case NN:                                                                                                        \
        if constexpr (RowShape<T, NN>::RW > 0) {                                                                    \
            using H = RowShape<T, NN>;                                                                              \
            constexpr int per = H::RW * H::WPB;                                                                     \
            return resident_grid(k_regrow<T, 3, NN, H::RW, H::WPB, H::MINB>, H::WPB * 32,                           \
                                 H::WPB * regrow_warp_smem<T, 3, NN, H::RW>(), (rows + per - 1) / per);             \
        }                                                                                                           \
        return 0;
        FGPE_STEP_SIZES(G)
#undef G
        default: return 0;
    }
}

template <typename T>
cudaError_t regrow_launch(int n, int grid, const StepConst& c, const RowArgs& a, cudaStream_t st, bool pdl) {
    switch (n) {
#define L(NN)                                                                                                       \
    case NN:                                                                                                        \
        if constexpr (RowShape<T, NN>::RW > 0) {                                                                    \
            using H = RowShape<T, NN>;                                                                              \
            return launch_step_kernel(k_regrow<T, 3, NN, H::RW, H::WPB, H::MINB>, grid, H::WPB * 32,                \
                                      H::WPB * regrow_warp_smem<T, 3, NN, H::RW>(), c, a, st, pdl);                 \
        }                                                                                                           \
        return cudaErrorInvalidValue;
        FGPE_STEP_SIZES(L)
#undef L
        default: return cudaErrorInvalidValue;
    }
}

// ---------------------------------------------------------- grouped passes
// Column tiles take the big z pass's plan and shape: with many instances there
// is a tile for every resident block, and wide rows of x keep whole sectors.
template <typename T, int MS, int N> struct GroupCol {
    using B = ColShape<T, MS, N, COLK_Z3D, true>;
    using P = typename B::P;
    static constexpr int TX = B::TX, TH = B::TH;
    static constexpr size_t SMEM = regcol_smem<T, MS, N, TX, P, COLK_Y2D, false>();
    static constexpr auto kernel() { return k_regcol_group<T, MS, N, TX, TH, B::MINB, P>; }
};
// Rows: k_regrow_group where k_regrow is available, else the block pass.
template <typename T, int MS, int N> struct GroupRow {
    using H = RowShape<T, N>;
    static constexpr bool reg = MS == 3 && H::RW > 0;
    static constexpr int R = row_r(N), TH = row_th<T, MS, N>();
};
constexpr int most_dividing(int tiles, int most) {
    int c = 1;
    for (int d = 1; d <= most; ++d) if (tiles % d == 0) c = d;
    return c;
}

template <typename T, int MS> bool group_shape(int nx, int ny, int members, GroupShape* g) {
    g->col_grid = g->row_grid = 0;
    switch (ny) {
#define C(NN)                                                                                                     \
    case NN: {                                                                                                    \
        using G = GroupCol<T, MS, NN>;                                                                            \
        g->col_tiles = (nx + G::TX - 1) / G::TX;                                                                  \
        g->col_grid = resident_grid(G::kernel(), G::TH, G::SMEM, (long long)members * g->col_tiles);              \
    } break;
        FGPE_STEP_SIZES(C)
#undef C
    }
    switch (nx) {
#define R(NN)                                                                                                     \
    case NN: {                                                                                                    \
        using G = GroupRow<T, MS, NN>;                                                                            \
        if constexpr (G::reg) {                                                                                   \
            using H = typename G::H;                                                                              \
            g->row_tiles = (ny + H::RW - 1) / H::RW;                                                              \
            g->chunk = most_dividing(g->row_tiles, 2);                                                            \
            const long long chunks = (long long)members * (g->row_tiles / g->chunk);                              \
            g->row_grid = resident_grid(k_regrow_group<T, MS, NN, H::RW, H::WPB, H::MINB>, H::WPB * 32,           \
                                        H::WPB * regrow_warp_smem<T, MS, NN, H::RW>(), (chunks + H::WPB - 1) / H::WPB); \
        } else {                                                                                                  \
            if (ny % G::R) return false;                                                                          \
            g->row_tiles = ny / G::R;                                                                             \
            g->chunk = most_dividing(g->row_tiles, 16);                                                           \
            g->row_grid = resident_grid(k_row_group<T, MS, NN, G::R, G::TH>, G::TH, row_smem<T, MS, NN>(),        \
                                        (long long)members * (g->row_tiles / g->chunk));                          \
        }                                                                                                         \
    } break;
        FGPE_STEP_SIZES(R)
#undef R
    }
    return g->col_grid > 0 && g->row_grid > 0;
}

template <typename T, int MS>
cudaError_t group_launch(int nx, int ny, const GroupShape& g, const InstDesc* d, int members, int snap, cudaStream_t st) {
    const GroupArgs ca{d, members, g.col_tiles, 1, 0}, ra{d, members, g.row_tiles, g.chunk, snap};
    switch (ny) {
#define C(NN)                                                                                                     \
    case NN: {                                                                                                    \
        using G = GroupCol<T, MS, NN>;                                                                            \
        G::kernel()<<<g.col_grid, G::TH, G::SMEM, st>>>(ca);                                                      \
    } break;
        FGPE_STEP_SIZES(C)
#undef C
        default: return cudaErrorInvalidValue;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    switch (nx) {
#define R(NN)                                                                                                     \
    case NN: {                                                                                                    \
        using G = GroupRow<T, MS, NN>;                                                                            \
        if constexpr (G::reg) {                                                                                   \
            using H = typename G::H;                                                                              \
            k_regrow_group<T, MS, NN, H::RW, H::WPB, H::MINB>                                                     \
                <<<g.row_grid, H::WPB * 32, H::WPB * regrow_warp_smem<T, MS, NN, H::RW>(), st>>>(ra);             \
        } else {                                                                                                  \
            k_row_group<T, MS, NN, G::R, G::TH><<<g.row_grid, G::TH, row_smem<T, MS, NN>(), st>>>(ra);            \
        }                                                                                                         \
    } break;
        FGPE_STEP_SIZES(R)
#undef R
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

#define FGPE_STEP_ROW_INSTANTIATE(T)            \
    template int regrow_grid<T>(int, int);      \
    template cudaError_t regrow_launch<T>(int, int, const StepConst&, const RowArgs&, cudaStream_t, bool);

#define FGPE_STEP_INSTANTIATE(T, MS)                                                                  \
    template int regcol_grid<T, MS>(int, int, int, int, int*);                                        \
    template cudaError_t regcol_launch<T, MS>(int, int, int, int, const StepConst&, const ColArgs&,   \
                                              cudaStream_t, bool);                                    \
    template int row_grid<T, MS>(int, bool, int);                                                     \
    template cudaError_t row_launch<T, MS>(int, bool, int, const StepConst&, const RowArgs&, cudaStream_t, bool); \
    template bool group_shape<T, MS>(int, int, int, GroupShape*);                                     \
    template cudaError_t group_launch<T, MS>(int, int, const GroupShape&, const InstDesc*, int, int, cudaStream_t);

}  // namespace fgpe
