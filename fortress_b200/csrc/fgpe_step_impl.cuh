// fgpe_step_impl.cuh -- definitions of the pass launchers of fgpe_step.h,
// included by one translation unit per (precision, spin).
#pragma once
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
    if constexpr (KIND != COLK_Z3D) {
        return gw;
    } else {
        // the big tiles once there is one for every SM
        if (gw > 0 && tw >= 148) return gw;
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
    if constexpr (KIND != COLK_Z3D) {
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

#define FGPE_STEP_ROW_INSTANTIATE(T)            \
    template int regrow_grid<T>(int, int);      \
    template cudaError_t regrow_launch<T>(int, int, const StepConst&, const RowArgs&, cudaStream_t, bool);

#define FGPE_STEP_INSTANTIATE(T, MS)                                                                  \
    template int regcol_grid<T, MS>(int, int, int, int, int*);                                        \
    template cudaError_t regcol_launch<T, MS>(int, int, int, int, const StepConst&, const ColArgs&,   \
                                              cudaStream_t, bool);

}  // namespace fgpe
