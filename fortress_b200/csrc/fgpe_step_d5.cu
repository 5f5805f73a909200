// Register-resident step passes, double complex, spin 2 (fgpe_step.h).
#include "fgpe_step_impl.cuh"

namespace fgpe {
FGPE_STEP_INSTANTIATE(double, 5)
}  // namespace fgpe
