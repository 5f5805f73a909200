// Register-resident step passes, float complex, spin 1 (fgpe_step.h).
#include "fgpe_step_impl.cuh"

namespace fgpe {
FGPE_STEP_INSTANTIATE(float, 3)
FGPE_STEP_ROW_INSTANTIATE(float)
}  // namespace fgpe
