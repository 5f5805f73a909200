// Register-resident step passes, double complex, spin 1 (fgpe_step.h).
#include "fgpe_step_impl.cuh"

namespace fgpe {
FGPE_STEP_INSTANTIATE(double, 3)
FGPE_STEP_ROW_INSTANTIATE(double)
}  // namespace fgpe
