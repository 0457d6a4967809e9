// Small DFTs in registers and the radix dispatch of the two-pass line transforms (plane_g.cuh, box_lines.cu).
//
// dft<T, DIR, Q>: Q-point DFT of u[0..Q) in place, natural order in and out (DIR +1: exp(+i), -1: exp(-i)).
// Q = 2, 3, 4, 5 direct; 6, 10, 12, 15 by the prime-factor (Good-Thomas) map, which needs no twiddles
// (12 = 3 x 4: 96 real operations against 120 with W_12 twiddles); 8, 9, 16, 25 as A x B with the twiddles
// W_Q^j as exact constants (cos / sin of multiples of 2 pi / Q), the trivial ones folded at compile time.
#pragma once
#include "fft_core.cuh"
#include "line_plan.h"

namespace b200 {
namespace line {

// cos(2 pi j / Q) for the twiddled sizes
constexpr double kCos16[5] = {1.0, 0.92387953251128675612818318939679, 0.70710678118654752440084436210485,
                              0.38268343236508977172845998403040, 0.0};
constexpr double cos16(int j) {  // j in [0, 16)
    return j <= 4 ? kCos16[j] : j <= 8 ? -kCos16[8 - j] : j <= 12 ? -kCos16[j - 8] : kCos16[16 - j];
}
constexpr double kCos9[5] = {1.0, 0.7660444431189780352024, 0.1736481776669303488517, -0.5000000000000000000000,
                             -0.9396926207859083840541};
constexpr double kSin9[5] = {0.0, 0.6427876096865393263226, 0.9848077530122080593667, 0.8660254037844386467637,
                             0.3420201433256687330441};
constexpr double kCos25[17] = {1.0, 0.9685831611286311194902, 0.8763066800438635873081, 0.7289686274214115231467,
                               0.5358267949789966182713, 0.3090169943749474241023, 0.0627905195293133760762,
                               -0.1873813145857246305426, -0.4257792915650726488625, -0.6374239897486897101767,
                               -0.8090169943749474241023, -0.9297764858882514036609, -0.9921147013144778310498,
                               -0.9921147013144778310498, -0.9297764858882514036609, -0.8090169943749474241023,
                               -0.6374239897486897101767};
constexpr double kSin25[17] = {0.0, 0.2486898871648547882423, 0.4817536741017152749872, 0.6845471059286886737323,
                               0.8443279255020150785486, 0.9510565162951535721164, 0.9980267284282715619523,
                               0.9822872507286886810856, 0.9048270524660195277137, 0.7705132427757892308030,
                               0.5877852522924731291687, 0.3681245526846779591569, 0.1253332335643042453731,
                               -0.1253332335643042453731, -0.3681245526846779591569, -0.5877852522924731291687,
                               -0.7705132427757892308030};
constexpr double cosq(int Q, int j) {
    return Q == 25 ? kCos25[j] : Q == 9 ? kCos9[j] : cos16(j * (16 / Q));
}
constexpr double sinq(int Q, int j) {
    return Q == 25 ? kSin25[j] : Q == 9 ? kSin9[j] : cos16((j * (16 / Q) + 12) % 16);
}

// u * W_Q^j (DIR < 0) or its conjugate, W_Q = exp(-2 pi i / Q); quarter and eighth turns folded
template <typename T, int DIR, int Q, int J> __device__ __forceinline__ T twc(T u) {
    using R = typename RealOf<T>::type;
    if constexpr (J == 0) {
        return u;
    } else if constexpr (4 * J == Q) {  // -+i
        return cmul_si<T, DIR>(u);
    } else {
        constexpr double c = cosq(Q, J), s = DIR * sinq(Q, J);  // c + i s
        if constexpr (8 * J == Q) {                               // (1 +- i) / sqrt 2
            return DIR > 0 ? cmake<T>((u.x - u.y) * R(c), (u.x + u.y) * R(c))
                           : cmake<T>((u.x + u.y) * R(c), (u.y - u.x) * R(c));
        } else if constexpr (8 * J == 3 * Q) {                    // (-1 +- i) / sqrt 2
            return DIR > 0 ? cmake<T>((u.x + u.y) * R(c), (u.y - u.x) * R(c))
                           : cmake<T>((u.x - u.y) * R(c), (u.x + u.y) * R(c));
        } else {
            return cmake<T>(fma(u.x, R(c), -u.y * R(s)), fma(u.x, R(s), u.y * R(c)));
        }
    }
}
template <typename T, int DIR, int Q, int A, int B, int I> __device__ __forceinline__ void tw_all(T (*y)[A]) {
    if constexpr (I < A * B) {
        y[I / A][I % A] = twc<T, DIR, Q, (I / A) * (I % A)>(y[I / A][I % A]);
        tw_all<T, DIR, Q, A, B, I + 1>(y);
    }
}

constexpr int inv_mod(int a, int m) {
    for (int i = 1; i < m; ++i)
        if ((a * i) % m == 1) return i;
    return 1;
}

template <typename T, int DIR, int Q> __device__ __forceinline__ void dft(T* u) {
    if constexpr (Q <= 5) {
        dftR<T, DIR, Q>(u);
    } else {
        constexpr bool pfa = Q == 6 || Q == 10 || Q == 12 || Q == 15;
        constexpr int A = Q == 6 ? 3 : Q == 10 || Q == 15 || Q == 25 ? 5 : Q == 9 ? 3 : 4;
        constexpr int B = Q / A;
        static_assert(A * B == Q && B >= 2 && B <= 5, "unsupported DFT size");
        T y[B][A];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = u[pfa ? (B * n1 + A * n2) % Q : B * n1 + n2];
            dftR<T, DIR, A>(y[n2]);
        }
        if constexpr (!pfa) tw_all<T, DIR, Q, A, B, 0>(y);
        constexpr int eA = B * inv_mod(B % A, A), eB = A * inv_mod(A % B, B);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            T z[B];
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
            dftR<T, DIR, B>(z);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) u[pfa ? (eA * k1 + eB * k2) % Q : k1 + A * k2] = z[k2];
        }
    }
}

// Geometry of a line known at compile time: LineGeom's names, so that the kernels take either.
template <int N, int R1, int R2, int RS, int LD> struct FixedGeom {
    static constexpr int n = N, r1 = R1, r2 = R2, rs = RS, ld = LD;
};

// f(integral constant of the line's r1, or r2); for a run-time geometry the branch is uniform over the launch
// (RMAX: the largest r1 compiled in)
template <int V> struct IC { static constexpr int value = V; };
template <int RMAX, typename F> __device__ __forceinline__ void with_radix(int r, F&& f) {
    switch (r) {
        case 2: f(IC<2>()); break;
        case 3: f(IC<3>()); break;
        case 4: f(IC<4>()); break;
        case 5: f(IC<5>()); break;
        case 6: f(IC<6>()); break;
        case 8: f(IC<8>()); break;
        case 9: f(IC<9>()); break;
        case 10: f(IC<10>()); break;
        case 12: if constexpr (RMAX >= 12) f(IC<12>()); break;
        case 15: if constexpr (RMAX >= 15) f(IC<15>()); break;
        case 16: if constexpr (RMAX >= 16) f(IC<16>()); break;
        case 25: if constexpr (RMAX >= 25) f(IC<25>()); break;
    }
}
template <int RMAX, typename F> __device__ __forceinline__ void with_r1(const LineGeom& g, F&& f) { with_radix<RMAX>(g.r1, f); }
template <int RMAX, typename F> __device__ __forceinline__ void with_r2(const LineGeom& g, F&& f) { with_radix<10>(g.r2, f); }
template <int RMAX, typename F, int N, int R1, int R2, int RS, int LD>
__device__ __forceinline__ void with_r1(const FixedGeom<N, R1, R2, RS, LD>&, F&& f) { f(IC<R1>()); }
template <int RMAX, typename F, int N, int R1, int R2, int RS, int LD>
__device__ __forceinline__ void with_r2(const FixedGeom<N, R1, R2, RS, LD>&, F&& f) { f(IC<R2>()); }

// twiddles a thread keeps for pass B
template <typename G> struct MaxR2 { static constexpr int value = G::r2; };
template <> struct MaxR2<LineGeom> { static constexpr int value = 10; };
// values a thread holds in pass A
template <typename G, int RMAX> struct MaxR1 {
    static constexpr int value = G::r1;
    static constexpr bool fixed = true;
};
template <int RMAX> struct MaxR1<LineGeom, RMAX> {
    static constexpr int value = RMAX;
    static constexpr bool fixed = false;
};
// two compiled lines of one length share their twiddles
template <typename GX, typename GY> struct SameLine { static constexpr bool value = GX::n == GY::n; };
template <typename GY> struct SameLine<LineGeom, GY> { static constexpr bool value = false; };
template <typename GX> struct SameLine<GX, LineGeom> { static constexpr bool value = false; };
template <> struct SameLine<LineGeom, LineGeom> { static constexpr bool value = false; };

}  // namespace line
}  // namespace b200
