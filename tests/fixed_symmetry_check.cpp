// What symmetry keeps at exactly 0 along a ray stays 0 in the fixed-point
// geodesic (csrc/fixed_geodesic.cuh): k^3 in a plane through the axis of a hole
// without spin, k^2 and the distance from the equator in the equatorial plane.
// Prints the steps taken, 0 if one of them broke it.
#define main fixed_check_main
#include "fixed_check.cpp"
#undef main

static long follow(double a, double h, bool rk2, const Q* y0, bool plane) {
    FxGeo g{};
    g.a = of(a, 62);
    g.a2 = of((Q)a * a, 62);
    g.tc = of((1 - (Q)h) / (4 * PI), 63);
    g.ph = of(PI * (1 - (Q)h), 60);
    g.th2 = of(-2 * PI * PI * (1 - (Q)h), 58);
    g.eps = of(0.05L, 64);
    g.ok = 1;
    FxState s;
    FxPoint pt;
    encode(y0, s);
    fx_normalise(s, fx_log2r(s.x1));
    fx_point(g, fx_log2r(s.x1) - fx_shl((fx)s.n, 57), s.x2, pt);
    bool handed = false;
    FxNoTangent none;
    auto fallback = [&](FxState& w) {
        handed = true;
        w.raw = 1;
        return 0.0;
    };
    long n = 0;
    for (; n < 400; ++n) {
        const double r = std::exp((double)s.x1 * 0x1p-59);
        if (r < 2.3 || (r > 40 && s.k1 < 0)) break;
        double dl;
        fx_step(g, s, pt, rk2, dl, fallback, none);
        if (handed) break;
        if (plane ? s.k3 != 0 : s.k2 != 0 || s.x2 != fx_one(61)) return 0;
    }
    return n;
}

int main() {
    const double spin[2] = {0.9375, 0.0}, slope[3] = {0.3, 1.0, 1.8};
    for (int rk2 = 0; rk2 < 2; ++rk2)
        for (double h : slope)
            for (double beta : {3.0, 6.5, -9.0}) {
                Q y[6];
                photon(0, h, 60, 0, beta, y);
                y[5] = 0;
                printf("%ld\n", follow(0, h, rk2, y, true));
                for (double a : spin) {
                    photon(a, h, 90, beta, 0, y);
                    y[1] = 0.5L;
                    y[4] = 0;
                    printf("%ld\n", follow(a, h, rk2, y, false));
                }
            }
    return 0;
}
