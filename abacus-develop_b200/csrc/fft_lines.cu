// Host plan and launchers of the local H|psi> on two-pass line transforms (plane_g.cuh).
#include <algorithm>

#include "plane_launch.cuh"

namespace b200 {

namespace {

constexpr size_t kSmemMax = 227 * 1024;

constexpr int kSMs = 148;

// the shapes of the plane pass worth choosing from: for every (nw, L) that fits, the work of the busiest warp
// from the operation counts; a shape is dropped if another has no more work and no fewer resident CTAs
std::vector<PlaneShape> plane_shapes(const PWGrid& g, int prec, int npol) {
    const LineGeom &x = g.lines.x[prec], &y = g.lines.y[prec];
    const size_t elem = prec ? 8 : 16;
    const int maxw = line::plane_threads(elem, std::max(x.r1, y.r1)) / 32, ncols = npol * g.nxc;
    const int na = 32 / x.r2, nb = 32 / x.r1, nya = 32 / y.r2, nyb = 32 / y.r1;
    const double ca = 2 * line::dft_ops(x.r1) + 10 * x.r1 + 40;
    const double cb = npol * (2 * line::dft_ops(x.r2) + 12 * (x.r2 - 1) + 20 * x.r2);
    const double cya = 2 * line::dft_ops(y.r1) + 30 * y.r1 + 40;
    const double cyb = 2 * line::dft_ops(y.r2) + 12 * y.r2 + 20 * y.r2;
    std::vector<PlaneShape> all, out;
    for (int nw = 1; nw <= maxw; ++nw)
        for (int L = 1; L <= 12; ++L) {
            PlaneShape s;
            s.nw = nw;
            s.L = L;
            s.smem = (size_t(ncols) * y.ld + size_t(nw) * npol * L * x.ld) * elem;
            if (s.smem > kSmemMax) break;
            s.ctas = std::min<int>({int(228 * 1024 / (s.smem + 1024)), maxw / nw, 32});
            const int groups = ceil_div(ceil_div(y.n, L), nw), cper = ceil_div(ncols, nw);
            s.work = groups * (ceil_div(npol * L, na) * ca + ceil_div(L, nb) * cb) + ceil_div(cper, nya) * cya +
                     ceil_div(cper, nyb) * cyb;
            all.push_back(s);
        }
    std::stable_sort(all.begin(), all.end(), [](const PlaneShape& a, const PlaneShape& b) { return a.work < b.work; });
    int most = 0;
    for (const PlaneShape& s : all)
        if (s.ctas > most) {
            most = s.ctas;
            out.push_back(s);
        }
    return out;
}

// the shape for a launch of nctas planes: waves of resident CTAs times a CTA's time, which is its busiest warp's
// (up to 16 warps of an SM run latency-bound, each at its own pace) plus a start-up of about 700 instructions
const PlaneShape& pick_shape(const std::vector<PlaneShape>& c, long nctas) {
    const PlaneShape* best = &c[0];
    double bt = 1e300;
    for (const PlaneShape& s : c) {
        const double t = double((nctas + long(kSMs) * s.ctas - 1) / (long(kSMs) * s.ctas)) * (s.work + 700);
        if (t < bt) {
            bt = t;
            best = &s;
        }
    }
    return *best;
}

using line::ManyK;
using line::OneK;

int rmax_of(int r) { return r <= 10 ? 10 : r <= 16 ? 16 : 25; }

template <typename T, typename R, int NPOL>
void plane_pass(const PWGrid& g, int nplanes, const R* v, T* sb, cudaStream_t s) {
    constexpr int pi = sizeof(T) == 8;
    const PlaneShape& sh = pick_shape(g.lines.shapes[pi][NPOL - 1], long(nplanes) * g.nz);
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
        case 10: line::z_launch<T, R, 10>(g, gz, a); break;
        case 16: line::z_launch<T, R, 16>(g, gz, a); break;
        default: line::z_launch<T, R, 25>(g, gz, a); break;
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

void build_line_plan(PWGrid& g) {
    LinePlan& p = g.lines;
    p = LinePlan{};
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    for (int i = 0; i < 2; ++i) {
        const int elem = i ? 8 : 16;
        p.x[i] = line::x_geom(nx, elem);
        p.y[i] = line::y_geom(ny, elem, p.x[i].r2 ? p.x[i].r2 : 1);
        p.z[i] = line::z_geom(nz, elem);
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
        for (int npol = 1; npol <= 2; ++npol) p.shapes[i][npol - 1] = plane_shapes(g, i, npol);
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

#define B200_INST(T, R)                                                                                              \
    template bool launch_hpsi_local_lines<T, R>(const PWGrid&, int, const R*, int, int, const T*, T*, T*, double, int, \
                                                cudaStream_t);                                                       \
    template bool launch_hpsi_local_kbatch_lines<T, R>(const PWGrid&, const KBatchArgs&, int, int, const R*, T*, int,  \
                                                       double, cudaStream_t);                                        \
    template bool launch_hpsi_local_nc_lines<T, R>(const PWGrid&, int, const R*, int, int, const T*, T*, T*, double,   \
                                                   cudaStream_t);
B200_INST(double2, double)
B200_INST(float2, float)
#undef B200_INST

}  // namespace b200
