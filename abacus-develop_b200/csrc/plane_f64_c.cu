// Plane pass kernels with compiled lines (f64), edges 100 to 160.
#include "plane_launch.cuh"

namespace b200 {
namespace line {

template <>
bool plane_fixed_c<double2, double>(const PWGrid& g, const PlaneShape& sh, int n, const double* v, double2* sb, cudaStream_t s) {
    switch (g.nx) {
        case 100: return plane_fixed<double2, double, 100>(g, sh, n, v, sb, s);
        case 108: return plane_fixed<double2, double, 108>(g, sh, n, v, sb, s);
        case 120: return plane_fixed<double2, double, 120>(g, sh, n, v, sb, s);
        case 125: return plane_fixed<double2, double, 125>(g, sh, n, v, sb, s);
        case 128: return plane_fixed<double2, double, 128>(g, sh, n, v, sb, s);
        case 135: return plane_fixed<double2, double, 135>(g, sh, n, v, sb, s);
        case 144: return plane_fixed<double2, double, 144>(g, sh, n, v, sb, s);
        case 150: return plane_fixed<double2, double, 150>(g, sh, n, v, sb, s);
        case 160: return plane_fixed<double2, double, 160>(g, sh, n, v, sb, s);
        default: return false;
    }
}

}  // namespace line
}  // namespace b200
