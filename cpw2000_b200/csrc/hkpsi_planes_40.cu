// Kernels A and C of the local H|psi> for planes of 40 x 40 points (radix split 5 x 8).
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_PLANES(, double, 5, 8, 40)
CPWB_PLANES(, float, 5, 8, 40)
}  // namespace cpwb
