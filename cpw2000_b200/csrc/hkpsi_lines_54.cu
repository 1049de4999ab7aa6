// Kernel B of the local H|psi>, its spinor form and the density's, for z lines of 54 to 80 points.
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_LINES(, double, 6, 9)
CPWB_LINES(, float, 6, 9)
CPWB_DENSITY(, 6, 9)
CPWB_LINES(, double, 8, 8)
CPWB_LINES(, float, 8, 8)
CPWB_DENSITY(, 8, 8)
CPWB_LINES(, double, 8, 9)
CPWB_LINES(, float, 8, 9)
CPWB_DENSITY(, 8, 9)
CPWB_LINES(, double, 8, 10)
CPWB_LINES(, float, 8, 10)
CPWB_DENSITY(, 8, 10)
}  // namespace cpwb
