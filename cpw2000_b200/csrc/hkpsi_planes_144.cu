// Kernels A and C of the local H|psi> for planes of 144 x 144 points (radix split 12 x 12).
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_PLANES(, double, 12, 12, 32)
CPWB_PLANES(, float, 12, 12, 32)
}  // namespace cpwb
