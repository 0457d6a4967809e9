// Plane pass kernels with compiled lines (f32), edges 50 to 96.
#include "plane_launch.cuh"

namespace b200 {
namespace line {

template <>
bool plane_fixed_b<float2, float>(const PWGrid& g, const PlaneShape& sh, int n, const float* v, float2* sb, cudaStream_t s) {
    switch (g.nx) {
        case 50: return plane_fixed<float2, float, 50>(g, sh, n, v, sb, s);
        case 54: return plane_fixed<float2, float, 54>(g, sh, n, v, sb, s);
        case 60: return plane_fixed<float2, float, 60>(g, sh, n, v, sb, s);
        case 64: return plane_fixed<float2, float, 64>(g, sh, n, v, sb, s);
        case 72: return plane_fixed<float2, float, 72>(g, sh, n, v, sb, s);
        case 75: return plane_fixed<float2, float, 75>(g, sh, n, v, sb, s);
        case 80: return plane_fixed<float2, float, 80>(g, sh, n, v, sb, s);
        case 81: return plane_fixed<float2, float, 81>(g, sh, n, v, sb, s);
        case 90: return plane_fixed<float2, float, 90>(g, sh, n, v, sb, s);
        case 96: return plane_fixed<float2, float, 96>(g, sh, n, v, sb, s);
        default: return false;
    }
}

}  // namespace line
}  // namespace b200
