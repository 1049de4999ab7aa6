// Kernel B of the local H|psi>, its spinor form and the density's, for z lines of 96 to 128 points.
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_LINES(, double, 8, 12)
CPWB_LINES(, float, 8, 12)
CPWB_DENSITY(, 8, 12)
CPWB_LINES(, double, 10, 10)
CPWB_LINES(, float, 10, 10)
CPWB_DENSITY(, 10, 10)
CPWB_LINES(, double, 9, 12)
CPWB_LINES(, float, 9, 12)
CPWB_DENSITY(, 9, 12)
CPWB_LINES(, double, 8, 16)
CPWB_LINES(, float, 8, 16)
CPWB_DENSITY(, 8, 16)
}  // namespace cpwb
