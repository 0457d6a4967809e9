// psi -> rho kernels of square planes with compiled lines (f32).
#include "plane_launch.cuh"

namespace b200 {
namespace line {

template <> bool rho_fixed<float2, float>(const PWGrid& g, const RhoArgs<float2, float>& a) {
    if (g.nx != g.ny) return false;
    switch (g.nx) {
        case 18: return rho_fixed_n<float2, float, 18>(g, a);
        case 20: return rho_fixed_n<float2, float, 20>(g, a);
        case 24: return rho_fixed_n<float2, float, 24>(g, a);
        case 27: return rho_fixed_n<float2, float, 27>(g, a);
        case 30: return rho_fixed_n<float2, float, 30>(g, a);
        case 32: return rho_fixed_n<float2, float, 32>(g, a);
        case 36: return rho_fixed_n<float2, float, 36>(g, a);
        case 40: return rho_fixed_n<float2, float, 40>(g, a);
        case 45: return rho_fixed_n<float2, float, 45>(g, a);
        case 48: return rho_fixed_n<float2, float, 48>(g, a);
        case 50: return rho_fixed_n<float2, float, 50>(g, a);
        case 54: return rho_fixed_n<float2, float, 54>(g, a);
        case 60: return rho_fixed_n<float2, float, 60>(g, a);
        case 64: return rho_fixed_n<float2, float, 64>(g, a);
        case 72: return rho_fixed_n<float2, float, 72>(g, a);
        case 75: return rho_fixed_n<float2, float, 75>(g, a);
        case 80: return rho_fixed_n<float2, float, 80>(g, a);
        case 81: return rho_fixed_n<float2, float, 81>(g, a);
        case 90: return rho_fixed_n<float2, float, 90>(g, a);
        case 96: return rho_fixed_n<float2, float, 96>(g, a);
        case 100: return rho_fixed_n<float2, float, 100>(g, a);
        case 108: return rho_fixed_n<float2, float, 108>(g, a);
        case 120: return rho_fixed_n<float2, float, 120>(g, a);
        case 125: return rho_fixed_n<float2, float, 125>(g, a);
        case 128: return rho_fixed_n<float2, float, 128>(g, a);
        case 135: return rho_fixed_n<float2, float, 135>(g, a);
        case 144: return rho_fixed_n<float2, float, 144>(g, a);
        case 150: return rho_fixed_n<float2, float, 150>(g, a);
        case 160: return rho_fixed_n<float2, float, 160>(g, a);
        default: return false;
    }
}

}  // namespace line
}  // namespace b200
