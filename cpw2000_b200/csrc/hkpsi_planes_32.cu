// Kernels A and C of the local H|psi> for planes of 32 x 32 points (radix split 4 x 8).
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_PLANES(, double, 4, 8, 32)
CPWB_PLANES(, float, 4, 8, 32)
}  // namespace cpwb
