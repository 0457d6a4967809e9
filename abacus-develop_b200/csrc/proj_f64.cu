// FP64 projector products of small blocks (nonlocal_pw.cpp:211-304): becp = vkb^H psi and H psi += vkbd becp, all
// k-points of a batch in one launch each.
//
// Both are built from mma.sync m8n8k4 in FP64 (B200 has no tcgen05 FP64 kind; these instructions reach its FP64
// peak), a complex product as four real ones.  Fragments come straight from global memory: a lane's A or B value is one complex
// number (16 bytes: the real and imaginary parts of the fragment at once), four lanes cover 64 contiguous bytes of a
// row (becp: both operands; H psi: becp) or eight cover 128 (H psi: vkbd), and the next step's values are loaded
// before the current one is used.
//   becp:  a warp owns 8 JT x 8 NT values of becp and a share of the plane waves; the four warps of a CTA and then
//          the `slices` CTAs of a tile are added in a fixed order (the tile's last CTA reads the others' partial sums).
//   H psi: a warp owns 8 NT bands x 8 GT plane waves, all projectors.
#include <algorithm>
#include <cmath>

#include "proj_f64.h"

namespace b200 {

namespace {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// c += a b (CONJ: conj(a) b) for 8 x 8 complex tiles
template <bool CONJ> __device__ __forceinline__ void zmma(double (&re)[2], double (&im)[2], double2 a, double2 b) {
    dmma(re, a.x, b.x);
    dmma(re, CONJ ? a.y : -a.y, b.y);
    dmma(im, a.x, b.y);
    dmma(im, CONJ ? -a.y : a.y, b.x);
}

struct OneProj {
    ProjEntry e;
    __host__ __device__ __forceinline__ const ProjEntry& get(int) const { return e; }
};
struct ManyProj {
    ProjEntry e[kMaxProjBatch];
    __host__ __device__ __forceinline__ const ProjEntry& get(int q) const { return e[q]; }
};

constexpr int kWarps = 4;
constexpr int kWave = 3 * 148;  // CTAs of one wave at three a SM

// grid: x = projector tile + slice * tiles, y = band tile, z = k-point
template <int JT, int NT, typename Src>
__global__ void __launch_bounds__(kWarps * 32) k_proj_becp(Src src, int nkb, int nb, int ld, int jtiles, int slices,
                                                          double2* __restrict__ becp, double2* __restrict__ part,
                                                          unsigned* __restrict__ count) {
    __shared__ double2 red[kWarps - 1][JT * NT * 64];
    __shared__ bool last;
    const ProjEntry& e = src.get(blockIdx.z);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int jt = blockIdx.x % jtiles, sl = blockIdx.x / jtiles;
    const int j0 = jt * 8 * JT, b0 = blockIdx.y * 8 * NT;
    const int r = lane >> 2, q = lane & 3;
    // this warp's plane waves, in steps of 4: warp w of slice sl takes a run of whole steps
    const int steps = (e.npw + 3) / 4, share = slices * kWarps, wi = sl * kWarps + warp;
    const int t0 = int(long(steps) * wi / share), t1 = int(long(steps) * (wi + 1) / share);
    const double2 *pa[JT], *pb[NT];
    bool va[JT], vb[NT];
#pragma unroll
    for (int i = 0; i < JT; ++i) {
        va[i] = j0 + 8 * i + r < nkb;
        pa[i] = e.vkb + size_t(va[i] ? j0 + 8 * i + r : 0) * e.npwx + q;
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        vb[i] = b0 + 8 * i + r < nb;
        pb[i] = e.psi + size_t(vb[i] ? b0 + 8 * i + r : 0) * ld + q;
    }
    double re[JT][NT][2], im[JT][NT][2];
#pragma unroll
    for (int i = 0; i < JT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
    const double2 zero = make_double2(0.0, 0.0);
    double2 a[2][JT], b[2][NT];
    auto load = [&](int t, double2 (&x)[JT], double2 (&y)[NT]) {
        const bool in = t < t1 && 4 * t + q < e.npw;
#pragma unroll
        for (int i = 0; i < JT; ++i) x[i] = in && va[i] ? __ldg(pa[i] + 4 * t) : zero;
#pragma unroll
        for (int i = 0; i < NT; ++i) y[i] = in && vb[i] ? __ldg(pb[i] + 4 * t) : zero;
    };
    auto use = [&](double2 (&x)[JT], double2 (&y)[NT]) {
#pragma unroll
        for (int i = 0; i < JT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) zmma<true>(re[i][j], im[i][j], x[i], y[j]);
    };
    load(t0, a[0], b[0]);
    for (int t = t0; t < t1; t += 2) {
        load(t + 1, a[1], b[1]);
        use(a[0], b[0]);
        load(t + 2, a[0], b[0]);
        use(a[1], b[1]);
    }
    // the warps of the CTA, then the slices of the tile
    auto at = [&](int i, int j, int h) { return (i * NT + j) * 64 + r * 8 + 2 * q + h; };
    if (warp > 0) {
#pragma unroll
        for (int i = 0; i < JT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) red[warp - 1][at(i, j, h)] = make_double2(re[i][j][h], im[i][j][h]);
    }
    __syncthreads();
    constexpr int TILE = JT * NT * 64;
    const size_t tile = (size_t(blockIdx.z) * gridDim.y + blockIdx.y) * jtiles + jt;
    double2* mine = part + (tile * slices + sl) * TILE;
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < JT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    double2 v = make_double2(re[i][j][h], im[i][j][h]);
#pragma unroll
                    for (int w = 0; w < kWarps - 1; ++w) {
                        const double2 o = red[w][at(i, j, h)];
                        v.x += o.x;
                        v.y += o.y;
                    }
                    if (slices > 1) {
                        mine[at(i, j, h)] = v;
                    } else {
                        const int jj = j0 + 8 * i + r, bb = b0 + 8 * j + 2 * q + h;
                        if (jj < nkb && bb < nb) becp[(size_t(blockIdx.z) * nb + bb) * nkb + jj] = v;
                    }
                }
    }
    if (slices == 1) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(count + tile, 1u) == unsigned(slices - 1);
        if (last) count[tile] = 0;  // for the next launch
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < TILE; i += kWarps * 32) {
        const double2* p = part + tile * slices * TILE + i;
        double2 v = __ldcg(p);
#pragma unroll 8
        for (int s = 1; s < slices; ++s) {
            const double2 o = __ldcg(p + size_t(s) * TILE);
            v.x += o.x;
            v.y += o.y;
        }
        const int ij = i >> 6, jj = j0 + 8 * (ij / NT) + ((i >> 3) & 7), bb = b0 + 8 * (ij % NT) + (i & 7);
        if (jj < nkb && bb < nb) becp[(size_t(blockIdx.z) * nb + bb) * nkb + jj] = v;
    }
}

// grid: x = plane-wave tile of 8 GT kWarps, y = band tile, z = k-point
template <int NT, int GT, typename Src>
__global__ void __launch_bounds__(kWarps * 32) k_proj_add(Src src, int nkb, int nb, int ld,
                                                         const double2* __restrict__ becp) {
    const ProjEntry& e = src.get(blockIdx.z);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g0 = (blockIdx.x * kWarps + warp) * 8 * GT, b0 = blockIdx.y * 8 * NT;
    if (g0 >= e.npw) return;
    const int r = lane >> 2, q = lane & 3;
    const double2* pa[NT];
    bool va[NT], vb[GT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        va[i] = b0 + 8 * i + r < nb;
        pa[i] = becp + (size_t(blockIdx.z) * nb + (va[i] ? b0 + 8 * i + r : 0)) * nkb + q;
    }
    const double2* pb = e.vkbd + size_t(q) * e.npwx + g0 + r;
#pragma unroll
    for (int i = 0; i < GT; ++i) vb[i] = g0 + 8 * i + r < e.npw;
    const double2 zero = make_double2(0.0, 0.0);
    // H psi of this tile first: its loads run beside the products
    double2 h[NT][GT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < GT; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int bb = b0 + 8 * i + r, g = g0 + 8 * j + 2 * q + k;
                h[i][j][k] = bb < nb && g < e.npw ? e.hpsi[size_t(bb) * ld + g] : zero;
            }
    double re[NT][GT][2], im[NT][GT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < GT; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
    double2 a[2][NT], b[2][GT];
    const int steps = (nkb + 3) / 4;
    auto load = [&](int t, double2 (&x)[NT], double2 (&y)[GT]) {
        const bool in = 4 * t + q < nkb;
#pragma unroll
        for (int i = 0; i < NT; ++i) x[i] = in && va[i] ? __ldg(pa[i] + 4 * t) : zero;
#pragma unroll
        for (int i = 0; i < GT; ++i) y[i] = in && vb[i] ? __ldg(pb + size_t(4 * t) * e.npwx + 8 * i) : zero;
    };
    auto use = [&](double2 (&x)[NT], double2 (&y)[GT]) {
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < GT; ++j) zmma<false>(re[i][j], im[i][j], x[i], y[j]);
    };
    load(0, a[0], b[0]);
    for (int t = 0; t < steps; t += 2) {
        load(t + 1, a[1], b[1]);
        use(a[0], b[0]);
        load(t + 2, a[0], b[0]);
        use(a[1], b[1]);
    }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < GT; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int bb = b0 + 8 * i + r, g = g0 + 8 * j + 2 * q + k;
                if (bb < nb && g < e.npw)
                    e.hpsi[size_t(bb) * ld + g] = make_double2(h[i][j][k].x + re[i][j][k], h[i][j][k].y + im[i][j][k]);
            }
}

int slices_most(int npw) { return std::max(1, int(std::sqrt(npw / 8.0))); }
// What becp_launch may need of partial sums for a call of this size or any smaller one.  A call's own need is not
// monotone in its bands (8 k-points x 64 projectors: 248 832 values at 24 bands, 212 992 at 32), and an array of just
// that size would be freed by a smaller call under a captured graph that holds its address.  Tiles are at most 4 x 4
// blocks of 8 x 8 and 9 in all, and several slices mean tiles * slices <= kWave.
template <typename Src> size_t part_bound(const Src& src, int nk, int nkb, int nb) {
    int npwx = 0;
    for (int q = 0; q < nk; ++q) npwx = std::max(npwx, src.get(q).npwx);
    const size_t blocks = size_t(nk) * (ceil_div(nkb, 8) + 3) * (ceil_div(nb, 8) + 3);
    return std::min(blocks * slices_most(npwx), size_t(kWave) * 9) * 64;
}

template <int JT, int NT, typename Src>
void becp_launch(const Src& src, int nk, int nkb, int nb, int ld, int npw_max, double2* becp, ProjWorkspace& w,
                 cudaStream_t s) {
    const int jtiles = ceil_div(nkb, 8 * JT), btiles = ceil_div(nb, 8 * NT);
    const long tiles = long(nk) * jtiles * btiles;
    // slices of the plane waves: one wave of three CTAs a SM; a step of a warp (4 plane waves) costs about twice what the
    // last CTA takes to add a slice, so a single tile's time is least near sqrt(steps / 2) slices
    const int slices = std::min(int(std::max<long>(1, kWave / tiles)), slices_most(npw_max));
    static_assert(JT <= 4 && NT <= 4 && JT * NT <= 9, "part_bound");
    if (slices > 1) {
        w.part.resize(part_bound(src, nk, nkb, nb));
        if (!w.count.ptr) {
            w.count.resize(kWave);
            B200_CUDA(cudaMemsetAsync(w.count.ptr, 0, w.count.n * sizeof(unsigned), s));
        }
    }
    k_proj_becp<JT, NT, Src><<<dim3(jtiles * slices, btiles, nk), kWarps * 32, 0, s>>>(src, nkb, nb, ld, jtiles, slices, becp,
                                                                                      w.part.ptr, w.count.ptr);
    note_launch();
    B200_CUDA(cudaGetLastError());
}
template <int NT, int GT, typename Src>
void add_run(const Src& src, dim3 grid, int nkb, int nb, int ld, const double2* becp, cudaStream_t s) {
    k_proj_add<NT, GT, Src><<<grid, kWarps * 32, 0, s>>>(src, nkb, nb, ld, becp);
    note_launch();
    B200_CUDA(cudaGetLastError());
}
template <int NT, typename Src>
void add_launch(const Src& src, int nk, int nkb, int nb, int ld, int npw_max, const double2* becp, cudaStream_t s) {
    // 16 plane waves a warp, or 8 (a seventh more loads a product) where that leaves less of a last wave of three CTAs a
    // SM idle
    const int btiles = ceil_div(nb, 8 * NT);
    auto grid = [&](int gt) { return dim3(ceil_div(npw_max, 8 * gt * kWarps), btiles, nk); };
    auto waves = [&](int gt) { return (long(grid(gt).x) * btiles * nk + kWave - 1) / kWave; };
    if (double(waves(1)) * 1.15 < 2.0 * double(waves(2))) add_run<NT, 1>(src, grid(1), nkb, nb, ld, becp, s);
    else add_run<NT, 2>(src, grid(2), nkb, nb, ld, becp, s);
}

// f(source of the k-points): by value, one or up to kMaxProjBatch
template <typename F> void with_source(const ProjEntry* e, int nk, F&& f) {
    B200_CHECK(nk >= 1 && nk <= kMaxProjBatch, kInvalidArgument, "projector products: 1..128 k-points a call");
    if (nk == 1) {
        OneProj o;
        o.e = e[0];
        f(o);
    } else {
        ManyProj m;
        std::copy(e, e + nk, m.e);
        f(m);
    }
}
int npw_most(const ProjEntry* e, int nk) {
    int m = 0;
    for (int q = 0; q < nk; ++q) m = std::max(m, e[q].npw);
    return m;
}

}  // namespace

// 8-band tiles a warp takes at a time, 1 to 4: the fewest padded bands, then the largest tile
static int band_tiles(int nb) {
    int best = 4, pad = 1 << 30;
    for (int nt = 4; nt >= 1; --nt) {
        const int p = ceil_div(nb, 8 * nt) * nt;
        if (p < pad) {
            pad = p;
            best = nt;
        }
    }
    return best;
}

void proj_becp(const ProjEntry* e, int nk, int nkb, int nb, int ld, double2* becp, ProjWorkspace& w, cudaStream_t s) {
    const int npw = npw_most(e, nk);
    with_source(e, nk, [&](const auto& src) {
        switch (band_tiles(nb)) {
            case 1: becp_launch<4, 1>(src, nk, nkb, nb, ld, npw, becp, w, s); break;
            case 2: becp_launch<4, 2>(src, nk, nkb, nb, ld, npw, becp, w, s); break;
            case 3: becp_launch<3, 3>(src, nk, nkb, nb, ld, npw, becp, w, s); break;
            default: becp_launch<2, 4>(src, nk, nkb, nb, ld, npw, becp, w, s); break;
        }
    });
}
void proj_add(const ProjEntry* e, int nk, int nkb, int nb, int ld, const double2* becp, cudaStream_t s) {
    const int npw = npw_most(e, nk);
    with_source(e, nk, [&](const auto& src) {
        switch (band_tiles(nb)) {
            case 1: add_launch<1>(src, nk, nkb, nb, ld, npw, becp, s); break;
            case 2: add_launch<2>(src, nk, nkb, nb, ld, npw, becp, s); break;
            case 3: add_launch<3>(src, nk, nkb, nb, ld, npw, becp, s); break;
            default: add_launch<4>(src, nk, nkb, nb, ld, npw, becp, s); break;
        }
    });
}

// The rules compare two estimates fitted to whole H|psi> calls of 8 to 512 projectors, 205 to 51 569 plane waves and 1
// to 320 bands (2 623 points on B200, spinors up to 256 projectors; us, the library or the int8 emulation / these):
//   these cost a latency that grows with the projectors (k_proj_add walks all of them; taller band tiles take longer a
//   step) and little else in small blocks; the library's GEMMs cost a flat 10 to 20 us more than that, or, for one band, a
//   matrix-vector product each: 16 projectors x 380 plane waves 1 band 23 / 26, 8 bands 29 / 26; 64 x 3000 2 bands 36 / 31;
//   256 x 380 2 bands 36 / 38, 24 bands 36 / 60; 256 x 3000 2 bands 48 / 43.
// Blocks of more than 3e6 products go to the library, which is level from there on and ahead from some 12 bands: 128 x
// 9240, 8 bands 48 / 44, 12 bands 53 / 53, 24 bands 74 / 83; 256 x 3000, 24 bands 44 / 60.
// A batch saves the library's calls for every k-point: 64 x (64 x 3000), 32 bands 2369 / 1172; only one band of a few
// k-points with many projectors loses: 2 x (256 x 9226) 77 / 99, 2 x (64 x 9226) 51 / 42.
// At 6 of the points accepted the call is more than 10 % slower than with the library or the int8 emulation (with the
// limits on the products alone at 170, up to 2.25 x), at 4 of those given up it would have been faster.
bool proj_small(int nkb, int nb, int npw, int nk) {
    const double products = double(nkb) * nb * npw;
    if (nk > 1) return products <= 2e7 && (nb > 1 || nkb * (1 + 1e-4 * npw) <= 280.0 * nk - 360);
    const int step[5] = {0, 1, 2, 4, 4};  // by band tile
    return products <= 3e6 && nb > 1 && nkb * step[band_tiles(nb)] <= 140 + 0.05 * npw;
}
// Spinors: becp of 2 nb columns, then two products of 2 nkb projectors and nb bands one after the other, so the latency
// counts twice: 16 projectors x 3000 plane waves 1 band 44 / 40, 64 x 3000 45 / 52, 256 x 380 2 bands 51 / 83.
bool proj_small_spinor(int nkb, int nb, int npw) {
    if (double(nkb) * 2 * nb * npw > 3e6) return false;
    return nb == 1 ? nkb <= 16 && npw <= 30000 : nkb * (band_tiles(nb) >= 3 ? 1.5 : 1.0) <= 48 + 0.005 * npw;
}
// Against the int8 emulation, whose residues and recombination cost about 35 us more a call than these and a time that
// grows with plane waves x bands whatever the number of projectors: 128 projectors x 9240, 64 bands 232 / 161; 512 x
// 380, 64 bands 73 / 80; 512 x 3000, 128 bands 171 / 236, 48 bands 123 / 112; 256 x 9240, 96 bands 315 / 286.
bool proj_beats_int8(int nkb, int nb, int npw, int npol) {
    const double values = double(npw) * nb * npol, products = nkb * values;
    if (products > 2.5e8) return false;
    return npol == 2 ? 0.1 * nkb + 0.5e-6 * products <= 25 + 0.9e-4 * values
                     : 0.06 * nkb + 0.28e-6 * products <= 35 + 0.5e-4 * values;
}

}  // namespace b200
