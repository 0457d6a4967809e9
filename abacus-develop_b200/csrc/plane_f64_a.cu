// Plane pass kernels with compiled lines (f64), edges 18 to 48.
#include "plane_launch.cuh"

namespace b200 {
namespace line {

template <>
bool plane_fixed_a<double2, double>(const PWGrid& g, const PlaneShape& sh, int n, const double* v, double2* sb, cudaStream_t s) {
    switch (g.nx) {
        case 18: return plane_fixed<double2, double, 18>(g, sh, n, v, sb, s);
        case 20: return plane_fixed<double2, double, 20>(g, sh, n, v, sb, s);
        case 24: return plane_fixed<double2, double, 24>(g, sh, n, v, sb, s);
        case 27: return plane_fixed<double2, double, 27>(g, sh, n, v, sb, s);
        case 30: return plane_fixed<double2, double, 30>(g, sh, n, v, sb, s);
        case 32: return plane_fixed<double2, double, 32>(g, sh, n, v, sb, s);
        case 36: return plane_fixed<double2, double, 36>(g, sh, n, v, sb, s);
        case 40: return plane_fixed<double2, double, 40>(g, sh, n, v, sb, s);
        case 45: return plane_fixed<double2, double, 45>(g, sh, n, v, sb, s);
        case 48: return plane_fixed<double2, double, 48>(g, sh, n, v, sb, s);
        default: return false;
    }
}

}  // namespace line
}  // namespace b200
