// CPU check of the fixed-point geodesic (csrc/fixed_geodesic.cuh): rays
// integrated in fixed point and in double, each against the same steps in
// long double (64 or 113 significand bits).  Prints, per state component,
// the root mean square over the rays of the final error in fixed point and in
// double (k components relative to k^t and scaled by r), the largest ratio of
// a ray's two errors, and how many steps the fixed-point arithmetic handed
// back.
//   fixed_check rays eps integrator spin hslope inclination box seed
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../raptor_gb300/csrc/fixed_geodesic.cuh"

using namespace raptor;
typedef long double Q;
static const Q PI = 3.14159265358979323846264338327950288L;

// geodesic right-hand side, y = x1, x2, k^t .. k^phi (metric.c:538-638 with
// lengths in units of r)
template <class R>
static void rhs(const R* y, R a, R h, R* f) {
    const R pi = (R)PI, x1 = y[0], x2 = y[1], k0 = y[2], k1 = y[3], k2 = y[4], k3 = y[5];
    const R r = std::exp(x1), sin2 = std::sin(2 * pi * x2), th = pi * x2 + (1 - h) * sin2 / 2;
    const R s = std::sin(th), c = std::cos(th), dth = pi * (1 + (1 - h) * std::cos(2 * pi * x2));
    const R w = 1 / r, idth = 1 / dth, K1 = r * k1, K2 = r * r * k2, K3 = r * r * k3, w2 = w * w, s2 = s * s;
    const R sc = s * c, cot = c / s, sig = 1 + a * a * c * c * w2, rho = 1 + a * a * w2, dl = rho - 2 * w;
    const R i1 = 1 / sig, i2 = i1 * i1, i3 = i2 * i1, P = a * s2 * w2 * K3, bw = (2 - sig) * i3 * w;
    const R ga = i1 - a * a * s2 * bw * w2, X0 = k0 * (k0 - 2 * P), X1 = 2 * K1 * (k0 - P), H = (k0 + K1) * (k0 + K1);
    const R m = w2 * (i1 * dth * dth * K2 * K2 + ga * s2 * K3 * K3), t = a * a * sc * dth * i1 * w2;
    f[0] = k1;
    f[1] = k2;
    f[2] = w * (2 * w * m + 4 * t * i1 * w2 * K2 * (k0 + K1 - P) -
                bw * (2 * w * X0 + (sig + 2 * w) * X1 + 2 * (sig + w) * K1 * K1));
    f[3] = w2 * (dl * m + 2 * t * w * K1 * K2 - K1 * K1 - 2 * i1 * K1 * P -
                 bw * (dl * X0 + (dl - sig) * X1 - (2 * sig - dl) * K1 * K1));
    f[4] = w2 * w * ((t + 2 * pi * pi * (1 - h) * sin2 * idth) * w * K2 * K2 - 2 * i1 * K1 * K2 -
                     sc * i3 * idth * w * (2 * a * K3 * (2 * rho * w * k0 + (sig * sig + 2 * w * rho) * K1) -
                                           (dl * sig * sig + 2 * w * rho * rho) * K3 * K3 - 2 * a * a * w * H));
    f[5] = w2 * w * (2 * a * cot * dth * i2 * w * K2 * (2 * w * k0 + (sig + 2 * w) * K1) - a * bw * (H - 2 * k0 * P) -
                     ga * K3 * (2 * K1 - P) + a * i1 * dth * dth * w2 * K2 * K2 -
                     2 * (cot * dth + 2 * t * i1 * w) * w * K2 * K3);
}

template <class R>
static R step(R* y, R a, R h, R eps, bool rk2) {
    const R m2 = y[1] < 1 - y[1] ? y[1] : 1 - y[1];
    const R d = -eps / (std::fabs(y[3]) + std::fabs(y[4]) / m2 + std::fabs(y[5]));
    R f[4][6], ys[6];
    rhs(y, a, h, f[0]);
    for (int i = 0; i < 6; ++i) ys[i] = y[i] + d / 2 * f[0][i];
    rhs(ys, a, h, f[1]);
    if (rk2) {
        for (int i = 0; i < 6; ++i) y[i] += d * f[1][i];
        return d;
    }
    for (int i = 0; i < 6; ++i) ys[i] = y[i] + d / 2 * f[1][i];
    rhs(ys, a, h, f[2]);
    for (int i = 0; i < 6; ++i) ys[i] = y[i] + d * f[2][i];
    rhs(ys, a, h, f[3]);
    for (int i = 0; i < 6; ++i) y[i] += d / 6 * (f[0][i] + 2 * f[1][i] + 2 * f[2][i] + f[3][i]);
    return d;
}

static fx of(Q x, int b) { return (fx)std::llrint(std::ldexp(x, b)); }

static void encode(const Q* y, FxState& s) {
    auto il = [](Q v) { int e = -200; if (v != 0) std::frexp(v, &e); return e; };
    s.n = (int)std::floor(y[0] / std::log((Q)2));
    s.m = std::max(il(y[2]), il(y[3]) + s.n);
    const int q2 = il(y[4]) + 2 * s.n - s.m, q3 = il(y[5]) + 2 * s.n - s.m;
    s.p = std::max(std::max(std::min(q3, s.n + 3), q2), 0);
    s.u = std::max(q3 - s.p, 0);
    s.raw = 0;
    s.x1 = of(y[0], 59);
    s.x2 = of(y[1], 62);
    s.k0 = of(y[2], 61 - s.m);
    s.k1 = of(y[3], 61 + s.n - s.m);
    s.k2 = of(y[4], 61 + 2 * s.n - s.m - s.p);
    s.k3 = of(y[5], 61 + 2 * s.n - s.m - s.p - s.u);
}
static void decode(const FxState& s, Q* y) {
    y[0] = std::ldexp((Q)s.x1, -59);
    y[1] = std::ldexp((Q)s.x2, -62);
    y[2] = std::ldexp((Q)s.k0, s.m - 61);
    y[3] = std::ldexp((Q)s.k1, s.m - s.n - 61);
    y[4] = std::ldexp((Q)s.k2, s.m + s.p - 2 * s.n - 61);
    y[5] = std::ldexp((Q)s.k3, s.m + s.p + s.u - 2 * s.n - 61);
}

// the initial photon of a camera at r = 1e4 (metric.c:650-727, GRmath.c:135-184)
static void photon(Q a, Q h, Q incl, Q al, Q be, Q* y) {
    const Q mu = std::cos(incl * PI / 180), st = std::sin(incl * PI / 180), r = 1e4, lz = -al * st;
    const Q q = be * be + mu * mu * (al * al - 1);
    const Q kth = (be > 0 ? 1 : be < 0 ? -1 : 0) * std::sqrt(std::fabs(q - lz * lz * mu * mu / (st * st) + mu * mu));
    const Q sg = r * r + a * a * mu * mu, dl = r * r + a * a - 2 * r;
    const Q A = (r * r + a * a) * (r * r + a * a) - dl * a * a * st * st;
    const Q g00 = -A / (sg * dl), g03 = -2 * a * r / (sg * dl), g33 = (dl - a * a * st * st) / (sg * dl * st * st);
    const Q u0 = -g00 + g03 * lz, u3 = g33 * lz - g03, u2 = kth / sg;
    const Q u1 = std::sqrt((u0 - u2 * kth - u3 * lz) * dl / sg) / r;
    Q x2 = incl / 180;
    for (int i = 0; i < 60; ++i)
        x2 -= (PI * x2 + (1 - h) / 2 * std::sin(2 * PI * x2) - incl * PI / 180) /
              (PI * (1 + (1 - h) * std::cos(2 * PI * x2)));
    const Q dth = PI * (1 + (1 - h) * std::cos(2 * PI * x2));
    const Q y0[6] = {std::log(r), x2, u0 + 2 * r / dl * r * u1, u1, u2 / dth, a / dl * r * u1 + u3};
    for (int i = 0; i < 6; ++i) y[i] = (double)y0[i];
}

int main(int argc, char** argv) {
    if (argc < 9) return 2;
    const int rays = atoi(argv[1]);
    const double eps = atof(argv[2]), a = atof(argv[4]), h = atof(argv[5]), incl = atof(argv[6]), box = atof(argv[7]);
    const bool rk2 = atoi(argv[3]) == 2;
    std::mt19937_64 rng(atoi(argv[8]));
    std::uniform_real_distribution<double> uni(-box / 2, box / 2);
    FxGeo g{};
    g.a = of(a, 62);
    g.a2 = of((Q)a * a, 62);
    g.tc = of((1 - (Q)h) / (4 * PI), 63);
    g.ph = of(PI * (1 - (Q)h), 60);
    g.th2 = of(-2 * PI * PI * (1 - (Q)h), 58);
    g.eps = of(eps, 64);
    g.ok = 1;
    double sf[6] = {}, sd[6] = {}, ratio = 0, worst = 0;
    long steps = 0, slow = 0;
    const double cut = (1 + std::sqrt(1 - a * a)) * 1.1;
    for (int k = 0; k < rays; ++k) {
        Q yq[6], yf[6];
        double yd[6];
        photon(a, h, incl, uni(rng), uni(rng), yq);
        for (int i = 0; i < 6; ++i) yd[i] = (double)yq[i];
        FxState s;
        FxPoint pt;
        encode(yq, s);
        fx_normalise(s, fx_log2r(s.x1));
        fx_point(g, fx_log2r(s.x1) - fx_shl((fx)s.n, 57), s.x2, pt);
        for (int n = 0; n < 3000; ++n) {
            const double r = std::exp((double)yq[0]);
            if (!(r < 10100 && r > cut) || (r > 40 && yq[3] < 0)) break;
            step<Q>(yq, a, h, eps, rk2);
            step<double>(yd, a, h, eps, rk2);
            double dl;
            FxNoTangent none;
            auto fallback = [&](FxState& w) {
                ++slow;
                Q t[6];
                double td[6];
                decode(w, t);
                for (int i = 0; i < 6; ++i) td[i] = (double)t[i];
                const double d = step<double>(td, a, h, eps, rk2);
                for (int i = 0; i < 6; ++i) t[i] = td[i];
                encode(t, w);
                return std::fabs(d);
            };
            fx_step(g, s, pt, rk2, dl, fallback, none);
            ++steps;
        }
        decode(s, yf);
        double ef = 0, ed = 0;
        for (int i = 0; i < 6; ++i) {
            const double sc = i < 2 ? 1.0 : std::fabs((double)yq[2]) / (i == 2 ? 1.0 : std::exp((double)yq[0]));
            const double f = std::fabs((double)(yf[i] - yq[i])) / sc, d = std::fabs((double)(yd[i] - yq[i])) / sc;
            sf[i] += f * f;
            sd[i] += d * d;
            ef = std::max(ef, f);
            ed = std::max(ed, d);
        }
        ratio = std::max(ratio, ef / (ed + 1e-13));
        worst = std::max(worst, ef);
    }
    for (int i = 0; i < 6; ++i) printf("%.6e %.6e\n", std::sqrt(sf[i] / rays), std::sqrt(sd[i] / rays));
    printf("%.6e %.6e %ld %ld\n", ratio, worst, steps, slow);
    return 0;
}
