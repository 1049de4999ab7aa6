// Kernels A and C of the local H|psi> for any supported plane (run-time radices).
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_PLANES(, double, 0, 0, 0)
CPWB_PLANES(, float, 0, 0, 0)
}  // namespace cpwb
