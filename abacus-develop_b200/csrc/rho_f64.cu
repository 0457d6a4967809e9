// psi -> rho kernels of square planes with compiled lines (f64).
#include "plane_launch.cuh"

namespace b200 {
namespace line {

template <> bool rho_fixed<double2, double>(const PWGrid& g, const RhoArgs<double2, double>& a) {
    if (g.nx != g.ny) return false;
    switch (g.nx) {
        case 18: return rho_fixed_n<double2, double, 18>(g, a);
        case 20: return rho_fixed_n<double2, double, 20>(g, a);
        case 24: return rho_fixed_n<double2, double, 24>(g, a);
        case 27: return rho_fixed_n<double2, double, 27>(g, a);
        case 30: return rho_fixed_n<double2, double, 30>(g, a);
        case 32: return rho_fixed_n<double2, double, 32>(g, a);
        case 36: return rho_fixed_n<double2, double, 36>(g, a);
        case 40: return rho_fixed_n<double2, double, 40>(g, a);
        case 45: return rho_fixed_n<double2, double, 45>(g, a);
        case 48: return rho_fixed_n<double2, double, 48>(g, a);
        case 50: return rho_fixed_n<double2, double, 50>(g, a);
        case 54: return rho_fixed_n<double2, double, 54>(g, a);
        case 60: return rho_fixed_n<double2, double, 60>(g, a);
        case 64: return rho_fixed_n<double2, double, 64>(g, a);
        case 72: return rho_fixed_n<double2, double, 72>(g, a);
        case 75: return rho_fixed_n<double2, double, 75>(g, a);
        case 80: return rho_fixed_n<double2, double, 80>(g, a);
        case 81: return rho_fixed_n<double2, double, 81>(g, a);
        case 90: return rho_fixed_n<double2, double, 90>(g, a);
        case 96: return rho_fixed_n<double2, double, 96>(g, a);
        case 100: return rho_fixed_n<double2, double, 100>(g, a);
        case 108: return rho_fixed_n<double2, double, 108>(g, a);
        case 120: return rho_fixed_n<double2, double, 120>(g, a);
        case 125: return rho_fixed_n<double2, double, 125>(g, a);
        case 128: return rho_fixed_n<double2, double, 128>(g, a);
        case 135: return rho_fixed_n<double2, double, 135>(g, a);
        case 144: return rho_fixed_n<double2, double, 144>(g, a);
        case 150: return rho_fixed_n<double2, double, 150>(g, a);
        case 160: return rho_fixed_n<double2, double, 160>(g, a);
        default: return false;
    }
}

}  // namespace line
}  // namespace b200
