// Kernel B of the local H|psi> for z lines of 96 to 128 points.
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_LINES(, double, 8, 12)
CPWB_LINES(, float, 8, 12)
CPWB_LINES(, double, 10, 10)
CPWB_LINES(, float, 10, 10)
CPWB_LINES(, double, 9, 12)
CPWB_LINES(, float, 9, 12)
CPWB_LINES(, double, 8, 16)
CPWB_LINES(, float, 8, 16)
}  // namespace cpwb
