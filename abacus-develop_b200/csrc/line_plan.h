// Factors and shared-memory pads of the two-pass line transforms (plane_g.cuh): constant expressions, so that the
// compiled sizes and the host's plan of any other size follow one rule.
#pragma once

namespace b200 {

// A line of n = r1 * r2 points: in shared memory, element (k1, t) at k1 * rs + t, lines at a pitch ld.
struct LineGeom {
    int n, r1, r2, rs, ld;
};

namespace line {

// real operations of the register DFTs (adds, multiplies and FMAs; line_dft.cuh); 0: not built
constexpr int dft_ops(int q) {
    return q == 2 ? 4 : q == 3 ? 12 : q == 4 ? 16 : q == 5 ? 36 : q == 6 ? 36 : q == 8 ? 56 : q == 9 ? 88 : q == 10 ? 92
         : q == 12 ? 96 : q == 15 ? 168 : q == 16 ? 168 : q == 25 ? 424 : 0;
}
// lane slots a line takes in a warp whose lines have r threads each (32 / r lines a warp, the rest idle)
constexpr double lane_slots(int r) { return 32.0 / (32 / r); }

// n = r1 * r2 (r1 >= r2, r2 <= 10) with the fewest lane slots x operations: FP64 operations issue at half rate, so
// the idle lanes of a warp cost pipe time.  25 only where nothing else divides n; in FP64, 15 and 16 points (64
// registers of data) count a fifth more: at 96^2 12 x 8 runs the local pass in 1.53 ms, 16 x 6 in 1.60 (160 bands).
// r1 = 0: n has no such factors.
constexpr LineGeom choose_factors(int n, int elem) {
    LineGeom g{n, 0, 0, 0, 0};
    double best = 1e30;
    for (int b = 2; b <= 10; ++b) {
        if (n % b || dft_ops(b) == 0) continue;
        const int a = n / b;
        if (a < b || a > 25 || dft_ops(a) == 0) continue;
        const double c = (lane_slots(b) * (2 * dft_ops(a) + 10 * a) +
                          lane_slots(a) * (2 * dft_ops(b) + 12 * (b - 1) + 20 * b)) *
                             (elem == 16 && a > 12 ? 1.2 : 1.0) + (a == 25 ? 1e9 : 0.0);
        if (c < best) {
            best = c;
            g.r1 = a;
            g.r2 = b;
        }
    }
    return g;
}

// shared-memory wavefronts of one warp access by nl lanes at different addresses, in elements of `elem` bytes: 128 bytes
// a wavefront, so 128 / elem lanes are served together and lanes on one bank take turns
constexpr int wavefronts(const int* addr, int nl, int elem) {
    const int slots = 128 / elem;
    int total = 0;
    for (int g = 0; g < nl; g += slots) {
        int on_bank[32] = {}, worst = 0;
        for (int i = g; i < nl && i < g + slots; ++i) {
            const int n = ++on_bank[addr[i] % slots];
            if (n > worst) worst = n;
        }
        total += worst;
    }
    return total;
}
// the same per lane, for lanes (l, i) at l * lp + i * ip, r lanes a line
constexpr double wave_cost(int r, int lp, int ip, int elem) {
    int a[32] = {};
    const int nl = 32 / r * r;
    for (int n = 0, l = 0; n < nl; ++l)
        for (int i = 0; i < r; ++i) a[n++] = l * lp + i * ip;
    return double(wavefronts(a, nl, elem)) / nl;
}
// its least value (no two lanes on one bank)
constexpr double wave_best(int r, int elem) {
    const int nl = 32 / r * r, slots = 128 / elem;
    return double((nl + slots - 1) / slots) / nl;
}

// pads of a row (xr2 = 0) or of a column read and written by rows of xr2 threads: pass A's threads are neighbours
// in t, pass B's in k1, a row's in the column
constexpr LineGeom choose_pads(LineGeom g, int elem, int xr2) {
    if (!g.r1) return g;
    double best = 1e30;
    LineGeom out = g;
    const double least = 2 * wave_best(g.r2, elem) + 4 * wave_best(g.r1, elem) + (xr2 ? 2 * wave_best(xr2, elem) : 0.0);
    for (int rs = g.r2; rs <= g.r2 + 3; ++rs)
        for (int ld = (g.r1 - 1) * rs + g.r2; ld <= g.r1 * rs + 8; ++ld) {
            if (best < least + 1e-3) return out;  // conflict-free, and every further candidate is larger
            double c = 2 * wave_cost(g.r2, ld, 1, elem);
            if (c < best) c += 4 * wave_cost(g.r1, ld, rs, elem);
            c += 1e-6 * ld;
            if (xr2 && c < best) {
                int a[32] = {};
                const int nl = (32 / xr2 < g.n ? 32 / xr2 : g.n) * xr2;
                for (int n = 0, l = 0; n < nl; ++l)
                    for (int i = 0; i < xr2; ++i) a[n++] = l % g.r1 * rs + l / g.r1 + i * ld;
                c += 2.0 * wavefronts(a, nl, elem) / nl;
            }
            if (c < best) {
                best = c;
                out.rs = rs;
                out.ld = ld;
            }
        }
    return out;
}
// pads of a z line: pass A's threads are neighbours in t, pass B's in the stick
constexpr LineGeom choose_pads_z(LineGeom g, int elem) {
    if (!g.r1) return g;
    double best = 1e30;
    LineGeom out = g;
    const double least = wave_best(g.r2, elem) + wave_best(32, elem);
    for (int rs = g.r2; rs <= g.r2 + 1; ++rs)
        for (int ld = (g.r1 - 1) * rs + g.r2; ld <= g.r1 * rs + 16; ++ld) {
            if (best < least + 1e-3) return out;
            double c = wave_cost(g.r2, ld, 1, elem);
            if (c < best) c += wave_cost(32, 0, ld, elem);
            c += 1e-6 * ld;
            if (c < best) {
                best = c;
                out.rs = rs;
                out.ld = ld;
            }
        }
    return out;
}

constexpr LineGeom x_geom(int n, int elem) { return choose_pads(choose_factors(n, elem), elem, 0); }
constexpr LineGeom y_geom(int n, int elem, int xr2) { return choose_pads(choose_factors(n, elem), elem, xr2); }
constexpr LineGeom z_geom(int n, int elem) { return choose_pads_z(choose_factors(n, elem), elem); }

}  // namespace line
}  // namespace b200
