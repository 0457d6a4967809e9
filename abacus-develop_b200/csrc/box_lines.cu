// The drop-in box transforms (PW_Basis_K::recip_to_real / real_to_recip, pw_transform_k.cpp:336-476) on the two-pass line
// transforms of plane_g.cuh, one band: three kernels each way.
//
//   recip -> real:  z of the occupied sticks, straight from psi, into sticks[stick][z]; y of the occupied columns,
//                   from the sticks, into cols[column][y][z]; x into the box r = (x ny + y) nz + z.
//   real -> recip:  the same backwards; x stores only the occupied columns, y only the sticks, z only the sphere.
// The box is not zeroed first and no column without a stick is moved.  Along y and x a CTA takes a tile of 128 bytes
// of z, so every load and store is a whole line; along z the threads are neighbours in z.  One band is a few
// hundred short CTAs, so a kernel is bound by latency: of the Stockham kernels before (up to six block barriers and
// passes through shared memory a line, a memset of the box) each took 6 to 9 us at 90 x 90 x 45 in FP64.
#include <algorithm>

#include "plane_launch.cuh"

namespace b200 {
namespace line {

constexpr int kBoxThreads = 128;

// Transforms of nl lines by one CTA.  ALONG: neighbouring threads take neighbouring points of a line, otherwise
// neighbouring lines (NL lines a tile).  ld(l, i) and st(l, i, v): point i of line l.
template <typename T, int RMAX, int DIR, bool ALONG, int NL, typename Ld, typename St>
__device__ __forceinline__ void box_tile(const LineGeom& g, int nl, T* sm, const T* __restrict__ roots, const Ld& ld,
                                         const St& st) {
    const int tid = threadIdx.x;
    auto pass_a = [&](auto&& body) {  // (line, t)
        const int la = ALONG ? tid / g.r2 : tid % NL, ta = ALONG ? tid % g.r2 : tid / NL;
        const int dl = ALONG ? kBoxThreads / g.r2 : NL, dt = ALONG ? g.r2 : kBoxThreads / NL;
        if (ALONG && la >= dl) return;
        for (int l = la; l < nl; l += dl)
            for (int t = ta; t < g.r2; t += dt) body(l, t);
    };
    auto pass_b = [&](auto&& body) {  // (line, k1)
        const int lb = ALONG ? tid / g.r1 : tid % NL, kb = ALONG ? tid % g.r1 : tid / NL;
        const int dl = ALONG ? kBoxThreads / g.r1 : NL, dk = ALONG ? g.r1 : kBoxThreads / NL;
        if (ALONG && lb >= dl) return;
        for (int l = lb; l < nl; l += dl)
            for (int k1 = kb; k1 < g.r1; k1 += dk) body(l, k1);
    };
    if constexpr (DIR > 0) {
        pass_a([&](int l, int t) {
            with_radix<RMAX>(g.r1, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T u[Q];
#pragma unroll
                for (int n1 = 0; n1 < Q; ++n1) u[n1] = ld(l, n1 * g.r2 + t);
                dft<T, +1, Q>(u);
#pragma unroll
                for (int k1 = 0; k1 < Q; ++k1) sm[l * g.ld + k1 * g.rs + t] = u[k1];
            });
        });
        __syncthreads();
        pass_b([&](int l, int k1) {
            const T* b = sm + l * g.ld + k1 * g.rs;
            with_radix<10>(g.r2, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T w[Q];
                w[0] = b[0];
#pragma unroll
                for (int t = 1; t < Q; ++t) w[t] = cmulc(b[t], __ldg(roots + t * k1));
                dft<T, +1, Q>(w);
#pragma unroll
                for (int k2 = 0; k2 < Q; ++k2) st(l, k1 + g.r1 * k2, w[k2]);
            });
        });
    } else {
        pass_b([&](int l, int k1) {
            T* b = sm + l * g.ld + k1 * g.rs;
            with_radix<10>(g.r2, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T w[Q];
#pragma unroll
                for (int k2 = 0; k2 < Q; ++k2) w[k2] = ld(l, k1 + g.r1 * k2);
                dft<T, -1, Q>(w);
                b[0] = w[0];
#pragma unroll
                for (int t = 1; t < Q; ++t) b[t] = cmul(w[t], __ldg(roots + t * k1));
            });
        });
        __syncthreads();
        pass_a([&](int l, int t) {
            with_radix<RMAX>(g.r1, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T u[Q];
#pragma unroll
                for (int k1 = 0; k1 < Q; ++k1) u[k1] = sm[l * g.ld + k1 * g.rs + t];
                dft<T, -1, Q>(u);
#pragma unroll
                for (int n1 = 0; n1 < Q; ++n1) st(l, n1 * g.r2 + t, u[n1]);
            });
        });
    }
}

constexpr int kBoxSticks = 8;                                                     // sticks of a CTA along z
template <typename T> constexpr int box_z() { return 128 / int(sizeof(T)); }      // z of a CTA along y and x

// z: psi -> sticks (DIR +1), sticks -> psi (DIR -1: out (+)= scale v)
template <typename T, typename R, int RMAX, int DIR>
__global__ void __launch_bounds__(kBoxThreads) k_box_lines_z(StickMapView sm, LineGeom g, const T* __restrict__ roots,
                                                             const T* __restrict__ in, T* __restrict__ out, int add, R scale) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    const int s0 = blockIdx.x * kBoxSticks, nl = min(kBoxSticks, sm.nst - s0);
    // position in psi of point z of stick s0 + l, or -1
    auto sphere = [&](int l, int z) {
        const int2 d = __ldg(sm.sd + s0 + l);
        int dz = z - (d.y & 0xffff);
        if (dz < 0) dz += g.n;
        return dz < d.y >> 16 ? d.x + dz : -1;
    };
    if constexpr (DIR > 0)
        box_tile<T, RMAX, +1, true, 1>(
            g, nl, buf, roots,
            [&](int l, int z) {
                const int i = sphere(l, z);
                return i >= 0 ? in[i] : zero_of<T>();
            },
            [&](int l, int z, T v) { out[size_t(s0 + l) * g.n + z] = v; });
    else
        box_tile<T, RMAX, -1, true, 1>(
            g, nl, buf, roots, [&](int l, int z) { return in[size_t(s0 + l) * g.n + z]; },
            [&](int l, int z, T v) {
                const int i = sphere(l, z);
                if (i >= 0) out[i] = add ? cfma(v, scale, out[i]) : cscale(v, scale);
            });
}

// y of column blockIdx.x, a tile of z: sticks -> cols (DIR +1) or cols -> sticks (DIR -1)
template <typename T, int RMAX, int DIR>
__global__ void __launch_bounds__(kBoxThreads) k_box_lines_y(PlaneMapView pm, LineGeom g, int nz, const T* __restrict__ roots,
                                                             const T* __restrict__ in, T* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    const int c = blockIdx.x, z0 = blockIdx.y * box_z<T>(), nl = min(box_z<T>(), nz - z0);
    const int4 d = __ldg(pm.cd + c);
    auto stick = [&](int y) { return y < d.y ? d.x + y : y >= d.z && y < d.w ? d.x + d.y + y - d.z : -1; };
    if constexpr (DIR > 0)
        box_tile<T, RMAX, +1, false, box_z<T>()>(
            g, nl, buf, roots,
            [&](int l, int y) {
                const int s = stick(y);
                return s >= 0 ? in[size_t(s) * nz + z0 + l] : zero_of<T>();
            },
            [&](int l, int y, T v) { out[(size_t(c) * g.n + y) * nz + z0 + l] = v; });
    else
        box_tile<T, RMAX, -1, false, box_z<T>()>(
            g, nl, buf, roots, [&](int l, int y) { return in[(size_t(c) * g.n + y) * nz + z0 + l]; },
            [&](int l, int y, T v) {
                const int s = stick(y);
                if (s >= 0) out[size_t(s) * nz + z0 + l] = v;
            });
}

// x of row y = blockIdx.x, a tile of z: cols -> box (DIR +1: box = v, or += factor v) or box -> cols (DIR -1)
template <typename T, typename R, int RMAX, int DIR>
__global__ void __launch_bounds__(kBoxThreads) k_box_lines_x(PlaneMapView pm, LineGeom g, int ny, int nz,
                                                             const T* __restrict__ roots, const T* __restrict__ in,
                                                             T* __restrict__ out, int add, R factor) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    const int y = blockIdx.x, z0 = blockIdx.y * box_z<T>(), nl = min(box_z<T>(), nz - z0);
    auto column = [&](int x) { return x < pm.xm ? x : x >= pm.xh ? x - pm.xoff : -1; };
    if constexpr (DIR > 0)
        box_tile<T, RMAX, +1, false, box_z<T>()>(
            g, nl, buf, roots,
            [&](int l, int x) {
                const int c = column(x);
                return c >= 0 ? in[(size_t(c) * ny + y) * nz + z0 + l] : zero_of<T>();
            },
            [&](int l, int x, T v) {
                T* o = out + (size_t(x) * ny + y) * nz + z0 + l;
                *o = add ? cfma(v, factor, *o) : v;
            });
    else
        box_tile<T, RMAX, -1, false, box_z<T>()>(
            g, nl, buf, roots, [&](int l, int x) { return in[(size_t(x) * ny + y) * nz + z0 + l]; },
            [&](int l, int x, T v) {
                const int c = column(x);
                if (c >= 0) out[(size_t(c) * ny + y) * nz + z0 + l] = v;
            });
}

}  // namespace line

namespace {

template <auto Kernel, typename... A> void box_launch(dim3 grid, size_t smem, cudaStream_t s, A... a) {
    allow_smem<Kernel>(smem);
    Kernel<<<grid, line::kBoxThreads, smem, s>>>(a...);
    note_launch();
    B200_CUDA(cudaGetLastError());
}

template <typename T, int RMAX>
void box_both(const PWGrid& g, int ik, bool inverse, const T* in, T* out, T* aux, int add, double factor, cudaStream_t s) {
    using R = typename RealOf<T>::type;
    constexpr int pi = sizeof(T) == 8, TZ = line::box_z<T>();
    const LineGeom &x = g.lines.xbox[pi], &y = g.lines.ybox[pi], &z = g.lines.z[pi];
    T *sticks = aux, *cols = aux + size_t(g.nst) * g.nz;
    const dim3 gz(ceil_div(g.nst, line::kBoxSticks)), gy(g.nxc, ceil_div(g.nz, TZ)), gx(g.ny, ceil_div(g.nz, TZ));
    const size_t sz = size_t(line::kBoxSticks) * z.ld * sizeof(T), sy = size_t(TZ) * y.ld * sizeof(T),
                 sx = size_t(TZ) * x.ld * sizeof(T);
    const T *rx = line::roots_of<T>(g.ax), *ry = line::roots_of<T>(g.ay), *rz = line::roots_of<T>(g.az);
    const PlaneMapView pm = g.plane_view();
    if (inverse) {
        box_launch<line::k_box_lines_z<T, R, RMAX, +1>>(gz, sz, s, g.stick_view(ik), z, rz, in, sticks, 0, R(1));
        box_launch<line::k_box_lines_y<T, RMAX, +1>>(gy, sy, s, pm, y, g.nz, ry, (const T*)sticks, cols);
        box_launch<line::k_box_lines_x<T, R, RMAX, +1>>(gx, sx, s, pm, x, g.ny, g.nz, rx, (const T*)cols, out, add, R(factor));
    } else {
        // set_real_to_recip_output_op: out (+)= factor / nxyz * box (pw_op.cpp:46-66)
        const double scale = (add ? factor : 1.0) / double(g.nxyz());
        box_launch<line::k_box_lines_x<T, R, RMAX, -1>>(gx, sx, s, pm, x, g.ny, g.nz, rx, in, cols, 0, R(1));
        box_launch<line::k_box_lines_y<T, RMAX, -1>>(gy, sy, s, pm, y, g.nz, ry, (const T*)cols, sticks);
        box_launch<line::k_box_lines_z<T, R, RMAX, -1>>(gz, sz, s, g.stick_view(ik), z, rz, (const T*)sticks, out, add, R(scale));
    }
}

}  // namespace

template <typename T>
bool launch_box_lines(const PWGrid& g, int ik, bool inverse, const T* in, T* out, T* aux, int add, double factor,
                      cudaStream_t s) {
    if (!g.lines.ok) return false;
    // sticks and columns share the auxiliary box
    if (size_t(g.nst + g.nxc * g.ny) * g.nz > size_t(g.nxyz())) return false;
    constexpr int pi = sizeof(T) == 8;
    if (std::max({g.lines.x[pi].r1, g.lines.y[pi].r1, g.lines.z[pi].r1}) <= 16)
        box_both<T, 16>(g, ik, inverse, in, out, aux, add, factor, s);
    else
        box_both<T, 25>(g, ik, inverse, in, out, aux, add, factor, s);
    return true;
}

template bool launch_box_lines<double2>(const PWGrid&, int, bool, const double2*, double2*, double2*, int, double, cudaStream_t);
template bool launch_box_lines<float2>(const PWGrid&, int, bool, const float2*, float2*, float2*, int, double, cudaStream_t);

}  // namespace b200
