// Kernel B of the local H|psi>, its spinor form and the density's, for z lines of 144 to 256 points.
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_LINES(, double, 12, 12)
CPWB_LINES(, float, 12, 12)
CPWB_DENSITY(, 12, 12)
CPWB_LINES(, double, 10, 16)
CPWB_LINES(, float, 10, 16)
CPWB_DENSITY(, 10, 16)
CPWB_LINES(, double, 12, 16)
CPWB_LINES(, float, 12, 16)
CPWB_DENSITY(, 12, 16)
CPWB_LINES(, double, 16, 16)
CPWB_LINES(, float, 16, 16)
CPWB_DENSITY(, 16, 16)
}  // namespace cpwb
