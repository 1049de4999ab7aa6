// Kernels A and C of the local H|psi> for planes of 96 x 96 points (radix split 8 x 12).
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_PLANES(, double, 8, 12, 32)
CPWB_PLANES(, float, 8, 12, 32)
}  // namespace cpwb
