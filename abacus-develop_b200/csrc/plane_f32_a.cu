// Plane pass kernels with compiled lines (f32), edges 18 to 48.
#include "plane_launch.cuh"

namespace b200 {
namespace line {

template <>
bool plane_fixed_a<float2, float>(const PWGrid& g, const PlaneShape& sh, int n, const float* v, float2* sb, cudaStream_t s) {
    switch (g.nx) {
        case 18: return plane_fixed<float2, float, 18>(g, sh, n, v, sb, s);
        case 20: return plane_fixed<float2, float, 20>(g, sh, n, v, sb, s);
        case 24: return plane_fixed<float2, float, 24>(g, sh, n, v, sb, s);
        case 27: return plane_fixed<float2, float, 27>(g, sh, n, v, sb, s);
        case 30: return plane_fixed<float2, float, 30>(g, sh, n, v, sb, s);
        case 32: return plane_fixed<float2, float, 32>(g, sh, n, v, sb, s);
        case 36: return plane_fixed<float2, float, 36>(g, sh, n, v, sb, s);
        case 40: return plane_fixed<float2, float, 40>(g, sh, n, v, sb, s);
        case 45: return plane_fixed<float2, float, 45>(g, sh, n, v, sb, s);
        case 48: return plane_fixed<float2, float, 48>(g, sh, n, v, sb, s);
        default: return false;
    }
}

}  // namespace line
}  // namespace b200
