// Launch of the plane pass on line transforms (plane_g.cuh): run-time geometry, or the x line (and on square planes
// the y line) compiled in.  Compiled lines take about half the instructions of run-time ones (no index arithmetic, no
// dispatch), and their code stays in the instruction cache.
#pragma once
#include "plane_g.cuh"

namespace b200 {
namespace line {

// threads of a CTA, and resident threads of an SM, by the registers the transforms need: FP64 lines of 12 points and
// more in pass A take 168 a thread, the others 128.  Plane pass with fewer and more: 96^2 FP64 (12 x 8) 12 warps of 168
// 1.17 ms, 16 of 128 1.20; 72 x 36 FP64 16 of 128 284 us, 20 of 96 365, 12 of 168 339; 36^2 FP64 16 of 128 658 us,
// 24 of 80 730, 12 of 168 657; 96^2 FP32 16 of 128 580 us, 20 of 96 610, 12 of 168 614.
constexpr int plane_threads(size_t elem, int r1) { return elem == 8 || r1 <= 10 ? 512 : r1 <= 16 ? 384 : 256; }

template <typename T> const T* roots_of(const FftAxis& a) {
    if constexpr (sizeof(T) == 16) return a.rt64.ptr;
    else return a.rt32.ptr;
}

template <typename T, typename R, int RMAX, int NPOL, typename GX, typename GY>
void plane_launch(const PWGrid& g, const PlaneShape& sh, int nplanes, GX gx, GY gy, const R* v, T* sb, cudaStream_t s) {
    constexpr auto kern = k_plane_g<T, R, RMAX, NPOL, plane_threads(sizeof(T), RMAX), GX, GY>;
    allow_smem<kern>(sh.smem);
    kern<<<dim3(nplanes, g.nz), sh.nw * 32, sh.smem, s>>>(g.plane_view(), gx, gy, sh.L, g.nz, roots_of<T>(g.ax),
                                                          roots_of<T>(g.ay), v, size_t(g.nxyz()), sb);
    note_launch();
    B200_CUDA(cudaGetLastError());
}

// the plane pass with x lines of N compiled in; false for other grids
template <typename T, typename R, int N>
bool plane_fixed(const PWGrid& g, const PlaneShape& sh, int nplanes, const R* v, T* sb, cudaStream_t s) {
    if (g.nx != N) return false;
    constexpr int elem = sizeof(T);
    constexpr LineGeom x = x_geom(N, elem), y = y_geom(N, elem, x.r2);
    using GX = FixedGeom<N, x.r1, x.r2, x.rs, x.ld>;
    using GY = FixedGeom<N, y.r1, y.r2, y.rs, y.ld>;
    constexpr int rmax = x.r1;
    if (g.ny == N) {
        plane_launch<T, R, rmax, 1>(g, sh, nplanes, GX(), GY(), v, sb, s);
        return true;
    }
    const LineGeom& yd = g.lines.y[elem == 8];
    if (yd.r1 > 16) return false;
    if (rmax <= 10 && yd.r1 <= 10) plane_launch<T, R, (rmax <= 10 ? 10 : 16), 1>(g, sh, nplanes, GX(), yd, v, sb, s);
    else plane_launch<T, R, (rmax > 16 ? rmax : 16), 1>(g, sh, nplanes, GX(), yd, v, sb, s);
    return true;
}

// launch of psi -> rho for the bands of one stick-buffer chunk (shape: rho_shape)
template <typename T, typename R> struct RhoArgs {
    const RhoShape& shape;
    const T* sb;
    int nbc;
    const double* w;
    R* ws;
    int first;
    cudaStream_t s;
};
template <typename T, typename R, int RMAX, typename GX, typename GY>
void rho_launch(const PWGrid& g, GX gx, GY gy, const RhoArgs<T, R>& a) {
    constexpr auto kern = k_rho_g<T, R, RMAX, plane_threads(sizeof(T), RMAX), GX, GY>;
    const PlaneShape& sh = a.shape.plane;
    allow_smem<kern>(sh.smem);
    kern<<<dim3(g.nz, a.shape.nsplit), sh.nw * 32, sh.smem, a.s>>>(g.plane_view(), gx, gy, sh.L, g.nz, roots_of<T>(g.ax),
                                                                  roots_of<T>(g.ay), a.sb, a.nbc, a.w, a.shape.nsplit,
                                                                  a.shape.sums, a.ws, a.first);
    note_launch();
    B200_CUDA(cudaGetLastError());
}
template <typename T, typename R, int N> bool rho_fixed_n(const PWGrid& g, const RhoArgs<T, R>& a) {
    constexpr int elem = sizeof(T);
    constexpr LineGeom x = x_geom(N, elem), y = y_geom(N, elem, x.r2);
    rho_launch<T, R, x.r1>(g, FixedGeom<N, x.r1, x.r2, x.rs, x.ld>(), FixedGeom<N, y.r1, y.r2, y.rs, y.ld>(), a);
    return true;
}
// square planes with compiled lines; false for other grids (rho_f64.cu, rho_f32.cu)
template <typename T, typename R> bool rho_fixed(const PWGrid& g, const RhoArgs<T, R>& a);

// the z passes take one k-point (OneK) or a batch indexed by blockIdx.z (ManyK)
struct OneK {
    KBatchEntry e;
    __device__ __forceinline__ const KBatchEntry& get(int) const { return e; }
};
struct ManyK {
    KBatchArgs a;
    __device__ __forceinline__ const KBatchEntry& get(int q) const { return a.e[q]; }
};
template <typename T, typename Src> struct ZArgs {
    bool inv;
    const Src& src;
    int nk, b0, nbc;
    T* sb;
    double tpiba2;
    int accumulate;
    cudaStream_t s;
};
template <typename T> constexpr int z_tile() { return sizeof(T) == 16 ? 16 : 32; }  // 256 bytes of a plane row

template <typename T, typename R, int RMAX, int ZT, typename Src, typename GZ>
void z_launch(const PWGrid& g, GZ gz, const ZArgs<T, Src>& a) {
    constexpr int TS = z_tile<T>();
    const size_t smem = size_t(TS) * gz.ld * sizeof(T);
    const dim3 grid(ceil_div(g.nst, TS), a.nbc, a.nk);
    if (a.inv) {
        constexpr auto kern = k_zinv_g<T, RMAX, TS, ZT, Src, GZ>;
        allow_smem<kern>(smem);
        kern<<<grid, ZT, smem, a.s>>>(a.src, gz, a.b0, a.nbc, roots_of<T>(g.az), a.sb);
    } else {
        constexpr auto kern = k_zfwd_g<T, R, RMAX, TS, ZT, Src, GZ>;
        allow_smem<kern>(smem);
        kern<<<grid, ZT, smem, a.s>>>(a.src, gz, a.b0, a.nbc, roots_of<T>(g.az), a.sb, R(a.tpiba2),
                                       R(1.0 / double(g.nxyz())), a.accumulate);
    }
    note_launch();
    B200_CUDA(cudaGetLastError());
}
template <typename T, typename R, int N, typename Src> bool z_fixed_n(const PWGrid& g, const ZArgs<T, Src>& a) {
    constexpr LineGeom z = z_geom(N, sizeof(T));
    z_launch<T, R, z.r1, z_threads(z.r2)>(g, FixedGeom<N, z.r1, z.r2, z.rs, z.ld>(), a);
    return true;
}
// the z passes with lines of nz compiled in; false for other grids (zpass_f64.cu, zpass_f32.cu, and *_many)
template <typename T, typename R, typename Src> bool z_fixed(const PWGrid& g, const ZArgs<T, Src>& a);

// the compiled edges (2-, 3-, 5-smooth, 18 to 160 except 25), split over translation units
template <typename T, typename R>
bool plane_fixed_a(const PWGrid& g, const PlaneShape& sh, int nplanes, const R* v, T* sb, cudaStream_t s);
template <typename T, typename R>
bool plane_fixed_b(const PWGrid& g, const PlaneShape& sh, int nplanes, const R* v, T* sb, cudaStream_t s);
template <typename T, typename R>
bool plane_fixed_c(const PWGrid& g, const PlaneShape& sh, int nplanes, const R* v, T* sb, cudaStream_t s);

}  // namespace line
}  // namespace b200
