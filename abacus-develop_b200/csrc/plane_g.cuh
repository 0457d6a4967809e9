// The three passes of the local H|psi> on two-pass line transforms, for any grid whose edges factor as R1 * R2
// (LineGeom; every 2-, 3-, 5-smooth edge from 4 to 160 except 5).
//
// A line of n = R1 R2 points is transformed in two register passes with one exchange through shared memory:
//   pass A  (R2 threads a line)  thread t: the R1-point DFT of f[R2 n1 + t] over n1;
//   pass B  (R1 threads a line)  thread k1: its R2 values times W_n^(t k1), then their R2-point DFT, which gives
//                                X[k1 + R1 k2], k2 < R2.
// The forward transform runs the same factorisation backwards, with the same R2 - 1 twiddles of thread k1, so a
// thread keeps one set for both directions.  In shared memory element (k1, t) of a line lies at k1 rs + t, lines
// at a pitch ld; rs and ld are chosen on the host for the fewest bank conflicts over all access patterns.
//
// Plane pass: one CTA per (band, z).  The sticks of an occupied x column are read straight from the stick
// buffer by pass A of the inverse y transform (a column's occupied y are at most two runs, ColumnDesc) and
// written straight back by pass A of the forward one, so the plane enters and leaves shared memory in
// transformed form only.  Lines are independent, so a warp owns its columns, and later its rows with a private
// row buffer: the passes of a line are ordered by __syncwarp and the CTA meets at two barriers a plane in
// all.  The occupied x are the runs [0, xm) and [xh, nx).  Pass B's threads of a row are neighbours in x for
// each k2, so V_eff is read in its natural (z, y, x) order.
//
// What bounds the plane pass: latency at the 12 to 16 warps an SM's registers hold (128 to 168 a thread: a line's
// R1 complex values, R2 - 1 twiddles, R2 values of V_eff).  Every point crosses shared memory eight times (128 bytes,
// one cycle a point and SM): at 96^2 in FP64 that is 0.49 ms of 1.11 ms per 160 bands, and the FP64 pipe is 46 % busy.
// Before it, edges without 32 as a factor ran one warp a line with up to six passes through shared memory, or the
// Stockham kernels with a block barrier a pass.  FP64, B200, plane pass alone: 36^2 (2048 bands of 36 planes) 4.03 ->
// 0.67 ms, 45^2 (61 x 90) 562 -> 82 us, 72 x 36 (120 x 108) 1966 -> 284 us; with its z passes the k batch's local
// part went from 4.64 to 0.87 ms.  A compiled line takes half the time of a run-time one (36^2 1.36 ms, 45^2 144 us).
#pragma once
#include "line_dft.cuh"
#include "pw_grid.h"

namespace b200 {
namespace line {

template <typename T> __device__ __forceinline__ T zero_of() { return cmake<T>(0, 0); }

// inverse y transform of the columns [c0, c1) of a warp: pass A straight from the sticks, pass B in place
template <typename T, int RMAX, int NPOL, typename GY, typename Tw>
__device__ __forceinline__ void inverse_y(const PlaneMapView& pm, const GY& gy, int lane, int c0, int c1,
                                          const T* __restrict__ plane, size_t pcomp, T* A, const Tw& twy) {
    const int nxc = pm.nxc;
    const int la = lane / gy.r2, ta = lane - la * gy.r2, na = 32 / gy.r2;
    for (int c = c0 + la; c < c1; c += na) {
        if (la >= na) break;
        const int cc = NPOL == 1 ? c : (c >= nxc ? c - nxc : c);
        const int4 d = __ldg(pm.cd + cc);
        const T* src = plane + (NPOL == 2 && c >= nxc ? pcomp : 0) + d.x;
        T* col = A + c * gy.ld + ta;
        with_r1<RMAX>(gy, [&](auto q) {
            constexpr int Q = decltype(q)::value;
            T u[Q];
#pragma unroll
            for (int n1 = 0; n1 < Q; ++n1) {
                const int y = n1 * gy.r2 + ta;
                const bool lo = y < d.y, hi = y >= d.z && y < d.w;
                u[n1] = (lo || hi) ? src[lo ? y : d.y + y - d.z] : zero_of<T>();
            }
            dft<T, +1, Q>(u);
#pragma unroll
            for (int k1 = 0; k1 < Q; ++k1) col[k1 * gy.rs] = u[k1];
        });
    }
    __syncwarp();
    const int lb = lane / gy.r1, k1 = lane - lb * gy.r1, nb = 32 / gy.r1;
    for (int c = c0 + lb; c < c1; c += nb) {
        if (lb >= nb) break;
        T* blk = A + c * gy.ld + k1 * gy.rs;
        with_r2<RMAX>(gy, [&](auto q) {
            constexpr int Q = decltype(q)::value;
            T w[Q];
            w[0] = blk[0];
#pragma unroll
            for (int t = 1; t < Q; ++t) w[t] = cmulc(blk[t], twy(t, k1));
            dft<T, +1, Q>(w);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) blk[k2] = w[k2];
        });
    }
}
// inverse x transform, pass A, of rows [y0, y0 + nl) (of each component) into the row buffer
template <typename T, int RMAX, int NPOL, typename GX, typename GY>
__device__ __forceinline__ void inverse_x_rows(const PlaneMapView& pm, const GX& gx, const GY& gy, int lane, int y0, int nl,
                                               const T* A, T* buf) {
    const int nxc = pm.nxc;
    const int la = lane / gx.r2, ta = lane - la * gx.r2, na = 32 / gx.r2;
    for (int l = la; l < NPOL * nl; l += na) {
        if (la >= na) break;
        const int lr = NPOL == 1 ? l : (l >= nl ? l - nl : l);
        const int y = y0 + lr;
        const int yq = y / gy.r1;
        const T* row = A + (y - yq * gy.r1) * gy.rs + yq + (NPOL == 2 && l >= nl ? nxc * gy.ld : 0);
        T* b = buf + l * gx.ld + ta;
        with_r1<RMAX>(gx, [&](auto q) {
            constexpr int Q = decltype(q)::value;
            T u[Q];
#pragma unroll
            for (int n1 = 0; n1 < Q; ++n1) {
                const int x = n1 * gx.r2 + ta;
                const bool lo = x < pm.xm, hi = x >= pm.xh;
                u[n1] = (lo || hi) ? row[(lo ? x : x - pm.xoff) * gy.ld] : zero_of<T>();
            }
            dft<T, +1, Q>(u);
#pragma unroll
            for (int j = 0; j < Q; ++j) b[j * gx.rs] = u[j];
        });
    }
}

// ---- plane pass ----
// NPOL = 1: v = V_eff (z, y, x).  NPOL = 2: columns 2b and 2b + 1 of the stick buffer are the components of band
// b = blockIdx.x, v the four components of V_eff (pitch vstride), applied as veff_pw_op's 2 x 2 form.
// Shared memory: NPOL * nxc columns of gy.ld, then per warp NPOL * L rows of gx.ld.
// GX, GY: LineGeom (any size, RMAX bounding r1) or FixedGeom.  CTAs of up to MAXT threads, MAXT of them resident.
template <typename T, typename R, int RMAX, int NPOL, int MAXT, typename GX, typename GY>
__global__ void __launch_bounds__(MAXT, 1) k_plane_g(PlaneMapView pm, GX gx, GY gy, int L, int nz,
                                                     const T* __restrict__ rootx, const T* __restrict__ rooty,
                                                     const R* __restrict__ v, size_t vstride, T* __restrict__ sb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* A = reinterpret_cast<T*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nxc = pm.nxc, ncols = NPOL * nxc;
    const int z = blockIdx.y;
    T* plane = sb + (size_t(blockIdx.x) * NPOL * nz + z) * pm.nst;  // component c: + c * nz * nst
    const size_t pcomp = size_t(nz) * pm.nst;
    const int cper = (ncols + nw - 1) / nw;
    const int c0 = warp * cper, c1 = min(ncols, c0 + cper);  // this warp's columns
    // pass B's twiddles W_nx^(t k1), t < r2, for the whole kernel (and the y lines' too where they are the same)
    constexpr int kTw = MaxR2<GX>::value;
    constexpr bool kSame = SameLine<GX, GY>::value;
    T tw[kTw];
    {
        const int k1 = lane % gx.r1;
#pragma unroll
        for (int t = 1; t < kTw; ++t) tw[t] = t < gx.r2 ? __ldg(rootx + t * k1) : zero_of<T>();
    }
    auto twy = [&](int t, int k1) {
        if constexpr (kSame) return tw[t];
        else return __ldg(rooty + t * k1);
    };
    inverse_y<T, RMAX, NPOL>(pm, gy, lane, c0, c1, plane, pcomp, A, twy);
    __syncthreads();
    // ---- rows: inverse x, V_eff, forward x ----
    {
        T* buf = A + ncols * gy.ld + warp * (NPOL * L) * gx.ld;
        const int la = lane / gx.r2, ta = lane - la * gx.r2, na = 32 / gx.r2;
        const int lb = lane / gx.r1, k1 = lane - lb * gx.r1, nb = 32 / gx.r1;
        // V_eff of this thread's next pass-B line, loaded a pass ahead of its use
        R vr[kTw];
        auto load_v = [&](int y) {
            const R* vp = v + (size_t(z) * gy.n + y) * gx.n + k1;
#pragma unroll
            for (int k2 = 0; k2 < kTw; ++k2)
                if (k2 < gx.r2) vr[k2] = __ldg(vp + k2 * gx.r1);
        };
        for (int y0 = warp * L; y0 < gy.n; y0 += nw * L) {
            const int nl = min(L, gy.n - y0);
            if (NPOL == 1 && lb < nb && lb < nl) load_v(y0 + lb);
            inverse_x_rows<T, RMAX, NPOL>(pm, gx, gy, lane, y0, nl, A, buf);
            __syncwarp();
            for (int l = lb; l < nl; l += nb) {
                if (lb >= nb) break;
                const size_t vi = (size_t(z) * gy.n + y0 + l) * gx.n + k1;
                T* b = buf + l * gx.ld + k1 * gx.rs;
                with_r2<RMAX>(gx, [&](auto q) {
                    constexpr int Q = decltype(q)::value;
                    if constexpr (NPOL == 1) {
                        T w[Q];
                        w[0] = b[0];
#pragma unroll
                        for (int t = 1; t < Q; ++t) w[t] = cmulc(b[t], tw[t]);
                        dft<T, +1, Q>(w);
#pragma unroll
                        for (int k2 = 0; k2 < Q; ++k2) w[k2] = cscale(w[k2], vr[k2]);
                        if (l + nb < nl) load_v(y0 + l + nb);
                        dft<T, -1, Q>(w);
                        b[0] = w[0];
#pragma unroll
                        for (int t = 1; t < Q; ++t) b[t] = cmul(w[t], tw[t]);
                    } else {
                        T* bd = b + nl * gx.ld;
                        T up[Q], dn[Q];
                        up[0] = b[0];
                        dn[0] = bd[0];
#pragma unroll
                        for (int t = 1; t < Q; ++t) {
                            up[t] = cmulc(b[t], tw[t]);
                            dn[t] = cmulc(bd[t], tw[t]);
                        }
                        dft<T, +1, Q>(up);
                        dft<T, +1, Q>(dn);
#pragma unroll
                        for (int k2 = 0; k2 < Q; ++k2) {
                            // up' = up (V0 + V3) + dn (V1 - i V2), dn' = dn (V0 - V3) + up (V1 + i V2)
                            const R* vp = v + vi + k2 * gx.r1;
                            const R v0 = __ldg(vp), v1 = __ldg(vp + vstride), v2 = __ldg(vp + 2 * vstride),
                                    v3 = __ldg(vp + 3 * vstride);
                            const T a = up[k2], d = dn[k2];
                            const R dp = v0 + v3, dm = v0 - v3;
                            up[k2] = cmake<T>(dp * a.x + v1 * d.x + v2 * d.y, dp * a.y + v1 * d.y - v2 * d.x);
                            dn[k2] = cmake<T>(dm * d.x + v1 * a.x - v2 * a.y, dm * d.y + v1 * a.y + v2 * a.x);
                        }
                        dft<T, -1, Q>(up);
                        dft<T, -1, Q>(dn);
                        b[0] = up[0];
                        bd[0] = dn[0];
#pragma unroll
                        for (int t = 1; t < Q; ++t) {
                            b[t] = cmul(up[t], tw[t]);
                            bd[t] = cmul(dn[t], tw[t]);
                        }
                    }
                });
            }
            __syncwarp();
            // forward pass A back into the occupied columns; the next rows' pass A of a thread overwrites only
            // what the same thread reads here
            for (int l = la; l < NPOL * nl; l += na) {
                if (la >= na) break;
                const int lr = NPOL == 1 ? l : (l >= nl ? l - nl : l);
                const int y = y0 + lr;
                const int yq = y / gy.r1;
                T* row = A + (y - yq * gy.r1) * gy.rs + yq + (NPOL == 2 && l >= nl ? nxc * gy.ld : 0);
                const T* b = buf + l * gx.ld + ta;
                with_r1<RMAX>(gx, [&](auto q) {
                    constexpr int Q = decltype(q)::value;
                    T u[Q];
#pragma unroll
                    for (int j = 0; j < Q; ++j) u[j] = b[j * gx.rs];
                    dft<T, -1, Q>(u);
#pragma unroll
                    for (int n1 = 0; n1 < Q; ++n1) {
                        const int x = n1 * gx.r2 + ta;
                        const bool lo = x < pm.xm, hi = x >= pm.xh;
                        if (lo || hi) row[(lo ? x : x - pm.xoff) * gy.ld] = u[n1];
                    }
                });
            }
        }
    }
    __syncthreads();
    {
        const int lb = lane / gy.r1, k1 = lane - lb * gy.r1, nb = 32 / gy.r1;
        for (int c = c0 + lb; c < c1; c += nb) {
            if (lb >= nb) break;
            T* blk = A + c * gy.ld + k1 * gy.rs;
            with_r2<RMAX>(gy, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T w[Q];
#pragma unroll
                for (int k2 = 0; k2 < Q; ++k2) w[k2] = blk[k2];
                dft<T, -1, Q>(w);
                blk[0] = w[0];
#pragma unroll
                for (int t = 1; t < Q; ++t) blk[t] = cmul(w[t], twy(t, k1));
            });
        }
        __syncwarp();
        const int la = lane / gy.r2, ta = lane - la * gy.r2, na = 32 / gy.r2;
        for (int c = c0 + la; c < c1; c += na) {
            if (la >= na) break;
            const int cc = NPOL == 1 ? c : (c >= nxc ? c - nxc : c);
            const int4 d = __ldg(pm.cd + cc);
            T* dst = plane + (NPOL == 2 && c >= nxc ? pcomp : 0) + d.x;
            const T* col = A + c * gy.ld + ta;
            with_r1<RMAX>(gy, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T u[Q];
#pragma unroll
                for (int k = 0; k < Q; ++k) u[k] = col[k * gy.rs];
                dft<T, -1, Q>(u);
#pragma unroll
                for (int n1 = 0; n1 < Q; ++n1) {
                    const int y = n1 * gy.r2 + ta;
                    const bool lo = y < d.y, hi = y >= d.z && y < d.w;
                    if (lo || hi) dst[lo ? y : d.y + y - d.z] = u[n1];
                }
            });
        }
    }
}

// ---- psi -> rho: w_b |psi_b(r)|^2 summed over bands g, g + nsplit, ... of the stick buffer, at plane z ----
// One CTA per (z, g = blockIdx.y).  The sums of a CTA's plane live in shared memory after the row buffers, or, where
// that does not fit (sums = false), in its own plane of ws (in L2).  A point is always added to by the same thread,
// so nothing orders the sums but the band loop, and they are deterministic.  ws[g] is overwritten on the first chunk
// of bands and added to afterwards.
template <typename T, typename R, int RMAX, int MAXT, typename GX, typename GY>
__global__ void __launch_bounds__(MAXT, 1) k_rho_g(PlaneMapView pm, GX gx, GY gy, int L, int nz,
                                                   const T* __restrict__ rootx, const T* __restrict__ rooty,
                                                   const T* __restrict__ sb, int nbc, const double* __restrict__ w,
                                                   int nsplit, bool sums, R* __restrict__ ws, int first) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* A = reinterpret_cast<T*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nxc = pm.nxc, z = blockIdx.x, g = blockIdx.y;
    const size_t plane_n = size_t(gy.n) * gx.n;
    R* out = ws + (size_t(g) * nz + z) * plane_n;
    R* acc = sums ? reinterpret_cast<R*>(A + nxc * gy.ld + nw * L * gx.ld) : out;
    const int cper = (nxc + nw - 1) / nw;
    const int c0 = warp * cper, c1 = min(nxc, c0 + cper);
    constexpr int kTw = MaxR2<GX>::value;
    constexpr bool kSame = SameLine<GX, GY>::value;
    const int lb = lane / gx.r1, k1 = lane - lb * gx.r1, nb = 32 / gx.r1;
    T tw[kTw];
#pragma unroll
    for (int t = 1; t < kTw; ++t) tw[t] = t < gx.r2 ? __ldg(rootx + t * k1) : zero_of<T>();
    auto twy = [&](int t, int ky) {
        if constexpr (kSame) return tw[t];
        else return __ldg(rooty + t * ky);
    };
    T* buf = A + nxc * gy.ld + warp * L * gx.ld;
    for (int b = g; b < nbc; b += nsplit) {
        const R wb = R(w[b]);
        const bool init = b == g && (sums || first);
        inverse_y<T, RMAX, 1>(pm, gy, lane, c0, c1, sb + (size_t(b) * nz + z) * pm.nst, 0, A, twy);
        __syncthreads();
        for (int y0 = warp * L; y0 < gy.n; y0 += nw * L) {
            const int nl = min(L, gy.n - y0);
            inverse_x_rows<T, RMAX, 1>(pm, gx, gy, lane, y0, nl, A, buf);
            __syncwarp();
            for (int l = lb; l < nl; l += nb) {
                if (lb >= nb) break;
                const T* bl = buf + l * gx.ld + k1 * gx.rs;
                R* a = acc + size_t(y0 + l) * gx.n + k1;
                with_r2<RMAX>(gx, [&](auto q) {
                    constexpr int Q = decltype(q)::value;
                    T v[Q];
                    v[0] = bl[0];
#pragma unroll
                    for (int t = 1; t < Q; ++t) v[t] = cmulc(bl[t], tw[t]);
                    dft<T, +1, Q>(v);
#pragma unroll
                    for (int k2 = 0; k2 < Q; ++k2) {
                        const R n2 = fma(v[k2].x, v[k2].x, v[k2].y * v[k2].y);
                        a[k2 * gx.r1] = init ? wb * n2 : fma(wb, n2, a[k2 * gx.r1]);
                    }
                });
            }
            __syncwarp();
        }
        __syncthreads();  // the columns are read
    }
    if (g >= nbc) {
        if (first)
            for (size_t i = threadIdx.x; i < plane_n; i += blockDim.x) out[i] = R(0);
    } else if (sums) {
        for (size_t i = threadIdx.x; i < plane_n; i += blockDim.x) out[i] = first ? acc[i] : out[i] + acc[i];
    }
}

// ---- z passes: TS sticks per CTA, ZT threads ----
// Lines of 9 or 10 threads take 160, so that the 16 FP64 sticks of a CTA go through pass A in one round (with 128
// threads the second round held 2 of 16 lines: forward pass at nz = 108, 120 bands, 78 us, now 65); lines of 5 or 6 take
// 96, all of them busy and more CTAs resident (nz = 36, 2048 bands: 151 us, now 124).
constexpr int z_threads(int r2) { return r2 >= 9 ? 160 : r2 >= 7 || r2 <= 4 ? 128 : 96; }
// A stick's occupied z are one run modulo nz and its values consecutive in psi (stick descriptor: first value,
// first z, count), so pass A reads psi, and writes H psi, directly.  Pass B's threads are neighbours in the
// stick index, so the plane-major stick buffer is written and read in whole rows of TS sticks.
template <typename T, int RMAX, int TS, int ZT, typename Src, typename GZ>
__global__ void __launch_bounds__(ZT, RMAX > 16 ? 2 : 512 / ZT)
    k_zinv_g(Src src, GZ gz, int b0, int nbc, const T* __restrict__ roots, T* __restrict__ sb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* A = reinterpret_cast<T*>(smem_raw);
    const KBatchEntry& e = src.get(blockIdx.z);
    const StickMapView sm = e.sm;
    const int tid = threadIdx.x;
    const int s0 = blockIdx.x * TS;
    const int ns = min(TS, sm.nst - s0);
    const int band = blockIdx.y;
    const T* p = reinterpret_cast<const T*>(e.psi) + size_t(b0 + band) * e.ld;
    {
        const int na = ZT / gz.r2, la = tid / gz.r2, ta = tid - la * gz.r2;
        for (int sl = la; sl < ns; sl += na) {
            if (la >= na) break;
            const int2 d = __ldg(sm.sd + s0 + sl);
            const int z0 = d.y & 0xffff, len = d.y >> 16;
            T* st = A + sl * gz.ld + ta;
            with_r1<RMAX>(gz, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T u[Q];
#pragma unroll
                for (int n1 = 0; n1 < Q; ++n1) {
                    int dz = n1 * gz.r2 + ta - z0;
                    if (dz < 0) dz += gz.n;
                    u[n1] = dz < len ? p[d.x + dz] : zero_of<T>();
                }
                dft<T, +1, Q>(u);
#pragma unroll
                for (int k1 = 0; k1 < Q; ++k1) st[k1 * gz.rs] = u[k1];
            });
        }
    }
    __syncthreads();
    const int sl = tid % TS;
    if (sl >= ns) return;
    T* out = sb + (size_t(blockIdx.z) * nbc + band) * gz.n * sm.nst + s0 + sl;
    for (int k1 = tid / TS; k1 < gz.r1; k1 += ZT / TS) {
        const T* blk = A + sl * gz.ld + k1 * gz.rs;
        with_r2<RMAX>(gz, [&](auto q) {
            constexpr int Q = decltype(q)::value;
            T w[Q];
            w[0] = blk[0];
#pragma unroll
            for (int t = 1; t < Q; ++t) w[t] = cmulc(blk[t], __ldg(roots + t * k1));
            dft<T, +1, Q>(w);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) out[size_t(k1 + gz.r1 * k2) * sm.nst] = w[k2];
        });
    }
}

template <typename T, typename R, int RMAX, int TS, int ZT, typename Src, typename GZ>
__global__ void __launch_bounds__(ZT, RMAX > 16 ? 2 : 512 / ZT)
    k_zfwd_g(Src src, GZ gz, int b0, int nbc, const T* __restrict__ roots, const T* __restrict__ sb, R tpiba2,
             R invn, int accumulate) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* A = reinterpret_cast<T*>(smem_raw);
    const KBatchEntry& e = src.get(blockIdx.z);
    const StickMapView sm = e.sm;
    const int tid = threadIdx.x;
    const int s0 = blockIdx.x * TS;
    const int ns = min(TS, sm.nst - s0);
    const int band = blockIdx.y;
    const T* p = reinterpret_cast<const T*>(e.psi) + size_t(b0 + band) * e.ld;
    T* h = reinterpret_cast<T*>(e.hpsi) + size_t(b0 + band) * e.ld;
    const R* gk2 = reinterpret_cast<const R*>(e.gk2);
    const int na = ZT / gz.r2, la = tid / gz.r2, ta = tid - la * gz.r2;
    // psi and |k+G|^2 of this thread's line of pass A; with compiled lines those of the first line are loaded
    // before the stick buffer is read, so that both latencies overlap
    constexpr int kR1 = MaxR1<GZ, RMAX>::value;
    constexpr bool kAhead = MaxR1<GZ, RMAX>::fixed && kR1 <= (sizeof(T) == 16 ? 12 : 16);
    T pv[kR1];
    R kv[kR1];
    int2 d = make_int2(0, 0);
    auto dz_of = [&](int n1) {
        const int dz = n1 * gz.r2 + ta - (d.y & 0xffff);
        return dz < 0 ? dz + gz.n : dz;
    };
    auto load_kin = [&](int sl) {
        d = __ldg(sm.sd + s0 + sl);
#pragma unroll
        for (int n1 = 0; n1 < kR1; ++n1) {
            const int dz = dz_of(n1);
            pv[n1] = zero_of<T>();
            kv[n1] = R(0);
            if (n1 < gz.r1 && dz < d.y >> 16) {
                pv[n1] = p[d.x + dz];
                kv[n1] = __ldg(gk2 + d.x + dz);
            }
        }
    };
    if constexpr (kAhead)
        if (la < na && la < ns) load_kin(la);
    {
        const int sl = tid % TS;
        const T* in = sb + (size_t(blockIdx.z) * nbc + band) * gz.n * sm.nst + s0 + sl;
        for (int k1 = tid / TS; k1 < gz.r1; k1 += ZT / TS) {
            if (sl >= ns) break;
            T* blk = A + sl * gz.ld + k1 * gz.rs;
            with_r2<RMAX>(gz, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T w[Q];
#pragma unroll
                for (int k2 = 0; k2 < Q; ++k2) w[k2] = in[size_t(k1 + gz.r1 * k2) * sm.nst];
                dft<T, -1, Q>(w);
                blk[0] = w[0];
#pragma unroll
                for (int t = 1; t < Q; ++t) blk[t] = cmul(w[t], __ldg(roots + t * k1));
            });
        }
    }
    __syncthreads();
    if (la < na)
        for (int sl = la; sl < ns; sl += na) {
            const T* st = A + sl * gz.ld + ta;
            with_r1<RMAX>(gz, [&](auto q) {
                constexpr int Q = decltype(q)::value;
                T u[Q];
#pragma unroll
                for (int k1 = 0; k1 < Q; ++k1) u[k1] = st[k1 * gz.rs];
                dft<T, -1, Q>(u);
                if constexpr (!kAhead) load_kin(sl);
                else if (sl != la) load_kin(sl);
                // every load before the first store: psi may be H psi's own buffer
#pragma unroll
                for (int n1 = 0; n1 < Q; ++n1) {
                    u[n1] = cadd(cscale(u[n1], invn), cscale(pv[n1], kv[n1] * tpiba2));
                    if (accumulate) {
                        const int dz = dz_of(n1);
                        if (dz < d.y >> 16) u[n1] = cadd(u[n1], h[d.x + dz]);
                    }
                }
#pragma unroll
                for (int n1 = 0; n1 < Q; ++n1) {
                    const int dz = dz_of(n1);
                    if (dz < d.y >> 16) h[d.x + dz] = u[n1];
                }
            });
        }
    if (!accumulate && blockIdx.x == 0)
        for (int g = e.npw + tid; g < e.ld; g += ZT) h[g] = zero_of<T>();
}

}  // namespace line
}  // namespace b200
