// Kernel B of the local H|psi> for z lines of 16 to 50 points.
#include "hkpsi_kernels.cuh"

namespace cpwb {
CPWB_LINES(, double, 4, 4)
CPWB_LINES(, float, 4, 4)
CPWB_LINES(, double, 3, 6)
CPWB_LINES(, float, 3, 6)
CPWB_LINES(, double, 4, 5)
CPWB_LINES(, float, 4, 5)
CPWB_LINES(, double, 4, 6)
CPWB_LINES(, float, 4, 6)
CPWB_LINES(, double, 4, 8)
CPWB_LINES(, float, 4, 8)
CPWB_LINES(, double, 6, 6)
CPWB_LINES(, float, 6, 6)
CPWB_LINES(, double, 5, 8)
CPWB_LINES(, float, 5, 8)
CPWB_LINES(, double, 6, 8)
CPWB_LINES(, float, 6, 8)
CPWB_LINES(, double, 5, 10)
CPWB_LINES(, float, 5, 10)
}  // namespace cpwb
