// Host check of the line transforms' plan (test_line_plan.py).  Reads cells from stdin, one a line: name, lat0, nine
// lattice components, ecut, grid (0 0 0: the basis's rule), number of k-points and their direct coordinates; prints a
// line per cell: its name, whether the plan holds, and the number of errors.
#include <cstdio>
#include <iostream>
#include <set>
#include <string>
#include <vector>

#include "plane_launch.cuh"

using namespace b200;

static int errors;
static void expect(bool ok, const char* what) {
    if (ok) return;
    if (++errors <= 5) std::fprintf(stderr, "%s\n", what);
}

// every point of a line has an address of its own inside the line's pitch
static void check_geom(const LineGeom& g) {
    expect(g.r1 * g.r2 == g.n && g.r1 <= 25 && g.r2 <= 10 && line::dft_ops(g.r1) && line::dft_ops(g.r2), "factors");
    std::set<int> at;
    for (int k1 = 0; k1 < g.r1; ++k1)
        for (int t = 0; t < g.r2; ++t) at.insert(k1 * g.rs + t);
    expect(int(at.size()) == g.n && *at.rbegin() < g.ld, "pads");
}

static void check_columns(const PWGrid& g) {
    const LinePlan& p = g.lines;
    for (int x = 0, c = 0; x < g.nx; ++x) {
        const bool in = x < p.xm || x >= p.xh, want = c < g.nxc && g.h_xpos[c] == x;
        expect(in == want, "occupied x");
        if (want) {
            expect((x < p.xm ? x : x - p.xoff) == c, "column of x");
            ++c;
        }
    }
    for (int c = 0; c < g.nxc; ++c) {
        const int4 d = g.h_cdesc[c];
        for (int y = 0; y < g.ny; ++y) {
            const int s = y < d.y ? d.x + y : y >= d.z && y < d.w ? d.x + d.y + y - d.z : -1;
            expect(s == g.h_smap[size_t(c) * g.ny + y], "stick of (column, y)");
        }
    }
}

static void check_sticks(const PWGrid& g) {
    for (const KMap& km : g.kmaps)
        for (int s = 0; s < g.nst; ++s) {
            const int z0 = km.h_sd[s].y & 0xffff, len = km.h_sd[s].y >> 16;
            std::vector<int> at(g.nz, -1);
            for (int j = km.h_gofs[s]; j < km.h_gofs[s + 1]; ++j) at[km.h_gpk[j] & 1023] = km.h_glist[j];
            for (int z = 0; z < g.nz; ++z) {
                const int dz = z < z0 ? z - z0 + g.nz : z - z0;
                expect((dz < len ? km.h_sd[s].x + dz : -1) == at[z], "psi position of (stick, z)");
            }
        }
}

static void check_shapes(const PWGrid& g) {
    for (int prec = 0; prec < 2; ++prec) {
        const size_t elem = prec ? 8 : 16;
        const int threads = line::plane_threads(elem, std::max(g.lines.x[prec].r1, g.lines.y[prec].r1));
        for (int npol = 1; npol <= 2; ++npol)
            for (const PlaneShape& s : g.lines.shapes[prec][npol - 1])
                expect(s.smem <= kSmemMax && s.nw * 32 * s.ctas <= threads && s.L >= 1, "plane shape");
        if (!lines_supported(g, elem, 1)) continue;
        int most = 0;
        for (int nb = 1; nb < 130; ++nb) {
            const RhoShape r = rho_shape(g, elem, nb);
            expect(rho_splits_most(g, elem, nb) >= most, "the bound of the partial densities falls");
            most = rho_splits_most(g, elem, nb);
            expect(r.nsplit >= 1 && r.nsplit <= most && r.plane.smem <= kSmemMax, "rho shape");
        }
    }
}

int main() {
    for (int n = 1; n <= 250; ++n)
        for (const int elem : {8, 16}) {
            const LineGeom x = line::x_geom(n, elem);
            if (!x.r1) continue;
            check_geom(x);
            check_geom(line::z_geom(n, elem));
            for (int xr2 = 1; xr2 <= 10; ++xr2) check_geom(line::y_geom(n, elem, xr2));
        }
    std::printf("geometry 1 %d\n", errors);
    std::string name;
    double lat0, ecut, lat[9];
    int n[3], nk;
    while (std::cin >> name >> lat0) {
        for (double& v : lat) std::cin >> v;
        std::cin >> ecut >> n[0] >> n[1] >> n[2] >> nk;
        std::vector<double> k(3 * nk);
        for (double& v : k) std::cin >> v;
        errors = 0;
        PWBasisK b;
        expect(b.setup(lat0, lat, ecut, 0, n[0], n[1], n[2], nk, k.data()) == 0, "basis");
        PWGrid g;
        g.build(b);
        if (g.lines.ok) {
            for (int i = 0; i < 2; ++i)
                for (const LineGeom& q : {g.lines.x[i], g.lines.y[i], g.lines.z[i], g.lines.xbox[i], g.lines.ybox[i]}) check_geom(q);
            check_columns(g);
            check_sticks(g);
            check_shapes(g);
        }
        std::printf("%s %d %d\n", name.c_str(), int(g.lines.ok), errors);
    }
}
