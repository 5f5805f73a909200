// Register-resident step passes, float complex, spin 2 (fgpe_step.h).
#include "fgpe_step_impl.cuh"

namespace fgpe {
FGPE_STEP_INSTANTIATE(float, 5)
}  // namespace fgpe
