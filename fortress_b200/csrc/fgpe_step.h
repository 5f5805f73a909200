// fgpe_step.h -- host side of the register-resident passes of a split step:
// set-up and launch per (precision, spin), compiled in
// fgpe_step_<t><spin>.cu.
#pragma once
#include <cuda_runtime.h>

#include "fgpe_group.cuh"
#include "fgpe_kernels.h"

namespace fgpe {

// Column passes of the line lengths 128, 192, 256, 384 and 512 (kinds COLK_*
// of fgpe_regcol.cuh; here 0 forward, 1 inverse, 2 q2D, 3 3D z).
// regcol_grid: resident grid of the pass for an nx * n_other set of lines (0:
// not available); *wide tells which tile form (big or small) it is for.
template <typename T, int MS> int regcol_grid(int n, int kind, int nx, int n_other, int* wide);
template <typename T, int MS>
cudaError_t regcol_launch(int n, int kind, int wide, int grid, const StepConst& c, const ColArgs& a, cudaStream_t st,
                          bool pdl);
// Radices of the single-component passes (kinds 0 and 1), whose spectra the z
// pass reads.
inline int regcol_radices(int n, int* r) { r[0] = n / 16; r[1] = 16; return 2; }

// Row pass over shared tiles of the same lengths, one block per tile of rows or
// (warp) one warp per row (fgpe_fast.cuh): resident grid for the given number
// of rows (0: not available).
template <typename T, int MS> int row_grid(int n, bool warp, int rows);
template <typename T, int MS>
cudaError_t row_launch(int n, bool warp, int grid, const StepConst& c, const RowArgs& a, cudaStream_t st, bool pdl);

// Row pass of spin-1 lines of the same lengths (fgpe_regrow.cuh): resident
// grid for the given number of rows (0: not available).
template <typename T> int regrow_grid(int n, int rows);
template <typename T>
cudaError_t regrow_launch(int n, int grid, const StepConst& c, const RowArgs& a, cudaStream_t st, bool pdl);

// Grouped passes of q2D instances of one nx x ny shape (fgpe_group.cuh): tiles
// per instance, row tiles or batches per chunk, resident grids.
struct GroupShape { int col_tiles = 0, col_grid = 0, row_tiles = 0, chunk = 1, row_grid = 0; };
template <typename T, int MS> bool group_shape(int nx, int ny, int members, GroupShape* g);
// One whole step of every instance: the column pass, then the row pass
// (snap: see GroupArgs).
template <typename T, int MS>
cudaError_t group_launch(int nx, int ny, const GroupShape& g, const InstDesc* d, int members, int snap, cudaStream_t st);

// Launch as a programmatic dependent (pdl): the pass is launched while the
// previous one drains and waits on griddepcontrol.wait before it touches the
// state.  Grids are one wave of resident blocks, so a waiting block never
// keeps the previous pass from finishing.
template <class K, class A>
inline cudaError_t launch_step_kernel(K kern, int grid, int threads, size_t smem, const StepConst& c, const A& a,
                                      cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, c, a);
}

inline int sm_count() {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

// Resident blocks of kern over the device for ntiles tiles (0: it does not fit).
template <class K> inline int resident_grid(K kern, int th, size_t smem, long long ntiles) {
    int per = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, th, smem) != cudaSuccess || per < 1) return 0;
    const long long g = (long long)per * sm_count();
    return (int)(ntiles < g ? ntiles : g);
}

#define FGPE_STEP_EXTERN(T, MS)                                                                              \
    extern template int regcol_grid<T, MS>(int, int, int, int, int*);                                        \
    extern template cudaError_t regcol_launch<T, MS>(int, int, int, int, const StepConst&, const ColArgs&,   \
                                                     cudaStream_t, bool);                                    \
    extern template int row_grid<T, MS>(int, bool, int);                                                     \
    extern template cudaError_t row_launch<T, MS>(int, bool, int, const StepConst&, const RowArgs&,          \
                                                  cudaStream_t, bool);                                       \
    extern template bool group_shape<T, MS>(int, int, int, GroupShape*);                                     \
    extern template cudaError_t group_launch<T, MS>(int, int, const GroupShape&, const InstDesc*, int, int,  \
                                                    cudaStream_t);
#define FGPE_STEP_ROW_EXTERN(T)                                                                              \
    extern template int regrow_grid<T>(int, int);                                                            \
    extern template cudaError_t regrow_launch<T>(int, int, const StepConst&, const RowArgs&, cudaStream_t, bool);
FGPE_STEP_ROW_EXTERN(float)
FGPE_STEP_ROW_EXTERN(double)
#undef FGPE_STEP_ROW_EXTERN
FGPE_STEP_EXTERN(float, 3)
FGPE_STEP_EXTERN(float, 5)
FGPE_STEP_EXTERN(double, 3)
FGPE_STEP_EXTERN(double, 5)
#undef FGPE_STEP_EXTERN

}  // namespace fgpe
