// Host plan and launchers of the local H|psi> on two-pass line transforms (plane_g.cuh).
#include <algorithm>

#include "plane_launch.cuh"

namespace b200 {

namespace {

constexpr int kSMs = 148;
// the class of a run-time r1 (RMAX of the kernels)
int rmax_of(int r) { return r <= 10 ? 10 : r <= 16 ? 16 : 25; }

// instructions of the busiest of nw warps with L rows at a time, from the operation counts (x transforms one way
// only and no V_eff for inverse_only)
struct WarpWork {
    int ny, ncols, npol, na, nb, nya, nyb;
    double ca, cb, cya, cyb;
    WarpWork(const LineGeom& x, const LineGeom& y, int ncols_, int npol_, bool inverse_only)
        : ny(y.n), ncols(ncols_), npol(npol_), na(32 / x.r2), nb(32 / x.r1), nya(32 / y.r2), nyb(32 / y.r1) {
        const int ways = inverse_only ? 1 : 2;
        ca = ways * line::dft_ops(x.r1) + 5 * ways * x.r1 + 40;
        cb = npol * (ways * line::dft_ops(x.r2) + 6 * ways * (x.r2 - 1) + 10 * ways * x.r2);
        cya = ways * line::dft_ops(y.r1) + 15 * ways * y.r1 + 40;
        cyb = ways * line::dft_ops(y.r2) + 6 * ways * y.r2 + 10 * ways * y.r2;
    }
    static int up(int a, int b) { return (a + b - 1) / b; }
    double operator()(int nw, int L) const {
        const int groups = up(up(ny, L), nw), cper = up(ncols, nw);
        return groups * (up(npol * L, na) * ca + up(L, nb) * cb) + up(cper, nya) * cya + up(cper, nyb) * cyb;
    }
};

// the shapes worth choosing from: for every (nw, L) that fits, the work of the busiest warp; a shape is dropped if
// another has no more work and no fewer resident CTAs.  extra: further shared memory of a CTA
std::vector<PlaneShape> plane_shapes(const PWGrid& g, int prec, int npol, bool inverse_only, size_t extra) {
    const LineGeom &x = g.lines.x[prec], &y = g.lines.y[prec];
    const size_t elem = prec ? 8 : 16;
    const int maxw = line::plane_threads(elem, std::max(x.r1, y.r1)) / 32, ncols = npol * g.nxc;
    const WarpWork work(x, y, ncols, npol, inverse_only);
    PlaneShape least[33];  // the least work of each number of resident CTAs (0: none)
    for (int nw = 1; nw <= maxw; ++nw)
        for (int L = 1; L <= 12; ++L) {
            PlaneShape s;
            s.nw = nw;
            s.L = L;
            s.smem = (size_t(ncols) * y.ld + size_t(nw) * npol * L * x.ld) * elem + extra;
            if (s.smem > kSmemMax) break;
            s.ctas = std::min<int>({int(228 * 1024 / (s.smem + 1024)), maxw / nw, 32});
            s.work = work(nw, L);
            if (!least[s.ctas].ctas || s.work < least[s.ctas].work) least[s.ctas] = s;
        }
    std::vector<PlaneShape> out;
    for (int c = 32; c > 0; --c) {
        const PlaneShape& s = least[c];
        if (!s.ctas) continue;
        // of equal work, the one with fewer warps, then fewer rows
        if (out.empty() || s.work < out.back().work ||
            (s.work == out.back().work && (s.nw < out.back().nw || (s.nw == out.back().nw && s.L < out.back().L))))
            out.push_back(s);
    }
    std::reverse(out.begin(), out.end());
    return out;
}

// a CTA's time in instructions: its busiest warp's (up to 16 warps of an SM run latency-bound, each at its own pace)
// plus a start-up of about 700
constexpr double kStartUp = 700;
long waves(long nctas, const PlaneShape& s) { return (nctas + long(kSMs) * s.ctas - 1) / (long(kSMs) * s.ctas); }

// the shape for a launch of nctas planes, by waves of resident CTAs times a CTA's time; variant v > 1: the v-th best
// by that estimate (the autotuner's candidates)
const PlaneShape& pick_shape(const std::vector<PlaneShape>& c, long nctas, int variant) {
    auto time_of = [&](const PlaneShape& s) { return double(waves(nctas, s)) * (s.work + kStartUp); };
    const PlaneShape* best = &c[0];
    double floor = -1;
    for (int v = 0; v < std::max(1, variant); ++v) {
        const PlaneShape* next = nullptr;
        for (const PlaneShape& s : c)
            if (time_of(s) > floor && (!next || time_of(s) < time_of(*next))) next = &s;
        if (!next) break;  // fewer candidates than variants: the last one
        best = next;
        floor = time_of(*next);
    }
    return *best;
}

using line::ManyK;
using line::OneK;

template <typename T, typename R, int NPOL>
void plane_pass(const PWGrid& g, int nplanes, const R* v, T* sb, cudaStream_t s) {
    constexpr int pi = sizeof(T) == 8;
    const PlaneShape& sh = pick_shape(g.lines.shapes[pi][NPOL - 1], long(nplanes) * g.nz,
                                      pi ? g.plane_variant32 : g.plane_variant64);
    if constexpr (NPOL == 1)
        if (line::plane_fixed_a<T, R>(g, sh, nplanes, v, sb, s) || line::plane_fixed_b<T, R>(g, sh, nplanes, v, sb, s) ||
            line::plane_fixed_c<T, R>(g, sh, nplanes, v, sb, s))
            return;
    const LineGeom &x = g.lines.x[pi], &y = g.lines.y[pi];
    switch (rmax_of(std::max(x.r1, y.r1))) {
        case 10: line::plane_launch<T, R, 10, NPOL>(g, sh, nplanes, x, y, v, sb, s); break;
        case 16: line::plane_launch<T, R, 16, NPOL>(g, sh, nplanes, x, y, v, sb, s); break;
        default: line::plane_launch<T, R, 25, NPOL>(g, sh, nplanes, x, y, v, sb, s); break;
    }
}

template <typename T, typename R, typename Src>
void z_pass(bool inv, const PWGrid& g, const Src& src, int nk, int b0, int nbc, T* sb, double tpiba2, int accumulate,
            cudaStream_t s) {
    const line::ZArgs<T, Src> a{inv, src, nk, b0, nbc, sb, tpiba2, accumulate, s};
    if (line::z_fixed<T, R, Src>(g, a)) return;
    const LineGeom& gz = g.lines.z[sizeof(T) == 8];
    switch (rmax_of(gz.r1)) {
        case 10: line::z_launch<T, R, 10, 128>(g, gz, a); break;
        case 16: line::z_launch<T, R, 16, 128>(g, gz, a); break;
        default: line::z_launch<T, R, 25, 128>(g, gz, a); break;
    }
}

template <typename T, typename R> OneK one_k(const PWGrid& g, int ik, int ld, const T* psi, T* hpsi) {
    const KMap& km = g.kmaps[ik];
    OneK src;
    src.e.sm = g.stick_view(ik);
    src.e.psi = psi;
    src.e.hpsi = hpsi;
    src.e.ld = ld;
    src.e.npw = km.npw;
    src.e.gk2 = std::is_same<R, double>::value ? (const void*)km.gk2.ptr : (const void*)km.gk2f.ptr;
    return src;
}

}  // namespace

namespace {

// The geometry of the compiled edges as constants: the search of the pads takes 5 to 20 us of a host core for a line
// (a basis of 18^3 in 0.10 ms, with the searches of its twelve lines 0.30).
struct EdgeGeom {
    int n;
    LineGeom x[2], y[2], z[2];  // y: of a square plane
};
template <int N> constexpr EdgeGeom edge_geom() {
    constexpr LineGeom x0 = line::x_geom(N, 16), x1 = line::x_geom(N, 8);
    constexpr LineGeom y0 = line::y_geom(N, 16, x0.r2), y1 = line::y_geom(N, 8, x1.r2);
    constexpr LineGeom z0 = line::z_geom(N, 16), z1 = line::z_geom(N, 8);
    return EdgeGeom{N, {x0, x1}, {y0, y1}, {z0, z1}};
}
template <int... N> struct EdgeTable { static constexpr EdgeGeom of[sizeof...(N)] = {edge_geom<N>()...}; };
using Edges = EdgeTable<18, 20, 24, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 120, 125, 128,
                        135, 144, 150, 160>;
const EdgeGeom* edge_of(int n) {
    for (const EdgeGeom& e : Edges::of)
        if (e.n == n) return &e;
    return nullptr;
}

}  // namespace

void build_line_plan(PWGrid& g) {
    LinePlan& p = g.lines;
    p = LinePlan{};
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const EdgeGeom *ex = edge_of(nx), *ey = edge_of(ny), *ez = edge_of(nz);
    for (int i = 0; i < 2; ++i) {
        const int elem = i ? 8 : 16;
        p.x[i] = ex ? ex->x[i] : line::x_geom(nx, elem);
        p.y[i] = ex && nx == ny ? ex->y[i] : line::y_geom(ny, elem, p.x[i].r2 ? p.x[i].r2 : 1);
        p.z[i] = ez ? ez->z[i] : line::z_geom(nz, elem);
        p.xbox[i] = ex ? ex->z[i] : line::z_geom(nx, elem);
        p.ybox[i] = ey ? ey->z[i] : line::z_geom(ny, elem);
        if (!p.x[i].r1 || !p.y[i].r1 || !p.z[i].r1) return;
    }
    // occupied x: [0, xm) and [xh, nx)
    int m = 0;
    while (m < g.nxc && g.h_xpos[m] == m) ++m;
    p.xm = m;
    p.xoff = nx - g.nxc;
    p.xh = m < g.nxc ? g.h_xpos[m] : nx;
    for (int c = m; c < g.nxc; ++c)
        if (g.h_xpos[c] != c + p.xoff) return;
    // occupied y of each column: [0, m1) and [yh, ye), sticks consecutive in that order
    g.h_cdesc.assign(g.nxc, int4{0, 0, 0, 0});
    for (int c = 0; c < g.nxc; ++c) {
        const int* sm = &g.h_smap[size_t(c) * ny];
        int y = 0, s0 = -1;
        while (y < ny && sm[y] >= 0) {
            if (s0 < 0) s0 = sm[y];
            if (sm[y] != s0 + y) return;
            ++y;
        }
        const int m1 = y;
        while (y < ny && sm[y] < 0) ++y;
        const int yh = y;
        while (y < ny && sm[y] >= 0) {
            if (s0 < 0) s0 = sm[y];
            if (sm[y] != s0 + m1 + y - yh) return;
            ++y;
        }
        const int ye = y;
        while (y < ny && sm[y] < 0) ++y;
        if (y < ny || s0 < 0) return;
        g.h_cdesc[c] = int4{s0, m1, yh, ye};
    }
    // occupied z of each stick: one run modulo nz, consecutive in psi
    for (KMap& km : g.kmaps) {
        km.h_sd.assign(g.nst, int2{0, 0});
        for (int st = 0; st < g.nst; ++st) {
            const int j0 = km.h_gofs[st], len = km.h_gofs[st + 1] - j0;
            if (len == 0) continue;
            if (len > nz) return;
            const int g0 = km.h_glist[j0], z0 = km.h_gpk[j0] & 1023;
            for (int j = 0; j < len; ++j)
                if (km.h_glist[j0 + j] != g0 + j || (km.h_gpk[j0 + j] & 1023) != (z0 + j) % nz) return;
            km.h_sd[st] = int2{g0, z0 | (len << 16)};
        }
    }
    for (int i = 0; i < 2; ++i)
        for (int npol = 1; npol <= 2; ++npol) p.shapes[i][npol - 1] = plane_shapes(g, i, npol, false, 0);
    p.ok = true;
}

bool lines_supported(const PWGrid& g, size_t elem, int npol) {
    return g.lines.ok && !g.lines.shapes[elem == 8][npol - 1].empty();
}

template <typename T, typename R>
bool launch_hpsi_local_lines(const PWGrid& g, int ik, const R* veff_zyx, int nb, int ld, const T* psi, T* hpsi,
                             T* stickbuf, double tpiba2, int accumulate, cudaStream_t s) {
    if (!lines_supported(g, sizeof(T), 1)) return false;
    const OneK src = one_k<T, R>(g, ik, ld, psi, hpsi);
    z_pass<T, R>(true, g, src, 1, 0, nb, stickbuf, tpiba2, 0, s);
    plane_pass<T, R, 1>(g, nb, veff_zyx, stickbuf, s);
    z_pass<T, R>(false, g, src, 1, 0, nb, stickbuf, tpiba2, accumulate, s);
    return true;
}

template <typename T, typename R>
bool launch_hpsi_local_kbatch_lines(const PWGrid& g, const KBatchArgs& args, int nk, int nb, const R* veff_zyx,
                                    T* stickbuf, int chunk, double tpiba2, cudaStream_t s) {
    if (!lines_supported(g, sizeof(T), 1)) return false;
    ManyK src;
    src.a = args;
    for (int b0 = 0; b0 < nb; b0 += chunk) {
        const int nbc = std::min(chunk, nb - b0);
        z_pass<T, R>(true, g, src, nk, b0, nbc, stickbuf, tpiba2, 0, s);
        plane_pass<T, R, 1>(g, nk * nbc, veff_zyx, stickbuf, s);
        z_pass<T, R>(false, g, src, nk, b0, nbc, stickbuf, tpiba2, 0, s);
    }
    return true;
}

template <typename T, typename R>
bool launch_hpsi_local_nc_lines(const PWGrid& g, int ik, const R* veff4_zyx, int ncols, int ld, const T* psi, T* hpsi,
                                T* stickbuf, double tpiba2, cudaStream_t s) {
    if (!lines_supported(g, sizeof(T), 2)) return false;
    const OneK src = one_k<T, R>(g, ik, ld, psi, hpsi);
    z_pass<T, R>(true, g, src, 1, 0, ncols, stickbuf, tpiba2, 0, s);
    plane_pass<T, R, 2>(g, ncols / 2, veff4_zyx, stickbuf, s);
    z_pass<T, R>(false, g, src, 1, 0, ncols, stickbuf, tpiba2, 0, s);
    return true;
}

// ---- psi -> rho ----
namespace {

// rho[x][y][z] += sum over g < nsplit of ws[g][z][y][x] in a fixed order, a 32 x 32 tile of (x, z) per CTA
template <typename R>
__global__ void __launch_bounds__(256) k_rho_reduce(int nx, int ny, int nz, int nsplit, const R* __restrict__ ws,
                                                    R* __restrict__ rho) {
    __shared__ R tile[32][33];
    const int x0 = blockIdx.x * 32, z0 = blockIdx.y * 32, y = blockIdx.z;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const size_t N = size_t(nx) * ny * nz;
    for (int r = ty; r < 32; r += 8) {
        const int z = z0 + r, x = x0 + tx;
        if (z >= nz || x >= nx) continue;
        const R* p = ws + (size_t(z) * ny + y) * nx + x;
        R sum = p[0];
        for (int g = 1; g < nsplit; ++g) sum += p[size_t(g) * N];
        tile[r][tx] = sum;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int x = x0 + r, z = z0 + tx;
        if (z < nz && x < nx) rho[(size_t(x) * ny + y) * nz + z] += tile[tx][r];
    }
}

}  // namespace

int rho_splits_most(const PWGrid& g, size_t elem, int nbc) {
    const size_t grid_bytes = size_t(g.nxyz()) * (elem / 2);
    return int(std::max<size_t>(1, std::min<size_t>(std::min(nbc, 64), kRhoPartBytes / grid_bytes)));
}

// the launch of psi -> rho for nbc bands: nsplit CTAs a plane share its bands, so that the planes of a small grid
// fill the SMs
RhoShape rho_shape(const PWGrid& g, size_t elem, int nbc) {
    const int prec = elem == 8, most = rho_splits_most(g, elem, nbc);
    const size_t real = elem / 2, plane = size_t(g.nx) * g.ny * real;
    RhoShape best;
    double bt = 1e300;
    for (const bool sums : {true, false}) {
        for (const PlaneShape& s : plane_shapes(g, prec, 1, true, sums ? plane : 0))
            for (int ns = 1; ns <= most; ++ns) {
                // An estimate: sums kept in L2 cost a quarter more than in shared memory, and each split writes and reads
                // a partial plane.  Measured at the best split of each (B200, shared memory / L2): 72 x 36 x 108 FP64, 96
                // bands 246 / 312 us; 36^3 FP64, 64 bands 38.8 / 40.3; 45 x 45 x 90 81 / 84; the other way round where
                // one CTA fills an SM: 96^3 FP64, 128 bands 766 / 675, 128^3 FP32, 160 bands 1026 / 959.  Splits: 96^3
                // 1 1073, 3 766, 4 845, 6 769; 36^3 1 128, 4 51, 16 38.8.
                const double per_band = (s.work + kStartUp / 2) * (sums ? 1.0 : 1.25);
                const double t = double(waves(long(g.nz) * ns, s)) * (ceil_div(nbc, ns) * per_band + kStartUp) +
                                 0.02 * ns * double(g.nxyz()) / kSMs;
                if (t < bt) {
                    bt = t;
                    best.plane = s;
                    best.nsplit = ns;
                    best.sums = sums;
                }
            }
    }
    return best;
}

template <typename T, typename R>
void launch_rho_chunk(const PWGrid& g, const RhoShape& shape, int ik, int b0, int nbc, int ld, const T* psi,
                      const double* w_chunk, T* sb, R* ws, int first, cudaStream_t s) {
    constexpr int pi = sizeof(T) == 8;
    const OneK src = one_k<T, R>(g, ik, ld, psi, nullptr);
    z_pass<T, R>(true, g, src, 1, b0, nbc, sb, 0.0, 0, s);
    const line::RhoArgs<T, R> a{shape, sb, nbc, w_chunk, ws, first, s};
    if (line::rho_fixed<T, R>(g, a)) return;
    const LineGeom &x = g.lines.x[pi], &y = g.lines.y[pi];
    switch (rmax_of(std::max(x.r1, y.r1))) {
        case 10: line::rho_launch<T, R, 10>(g, x, y, a); break;
        case 16: line::rho_launch<T, R, 16>(g, x, y, a); break;
        default: line::rho_launch<T, R, 25>(g, x, y, a); break;
    }
}

template <typename R> void launch_rho_reduce(const PWGrid& g, int nsplit, const R* ws, R* rho, cudaStream_t s) {
    k_rho_reduce<R><<<dim3(ceil_div(g.nx, 32), ceil_div(g.nz, 32), g.ny), 256, 0, s>>>(g.nx, g.ny, g.nz, nsplit, ws, rho);
    note_launch();
    B200_CUDA(cudaGetLastError());
}

#define B200_INST(T, R)                                                                                              \
    template bool launch_hpsi_local_lines<T, R>(const PWGrid&, int, const R*, int, int, const T*, T*, T*, double, int, \
                                                cudaStream_t);                                                       \
    template bool launch_hpsi_local_kbatch_lines<T, R>(const PWGrid&, const KBatchArgs&, int, int, const R*, T*, int,  \
                                                       double, cudaStream_t);                                        \
    template bool launch_hpsi_local_nc_lines<T, R>(const PWGrid&, int, const R*, int, int, const T*, T*, T*, double,   \
                                                   cudaStream_t);                                                    \
    template void launch_rho_chunk<T, R>(const PWGrid&, const RhoShape&, int, int, int, int, const T*, const double*,  \
                                         T*, R*, int, cudaStream_t);                                                 \
    template void launch_rho_reduce<R>(const PWGrid&, int, const R*, R*, cudaStream_t);
B200_INST(double2, double)
B200_INST(float2, float)
#undef B200_INST

}  // namespace b200
