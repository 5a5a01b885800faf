// The mixed form's adjoint with the geodesic in fixed point (vjp_f32.cuh has
// its body, fixed_geodesic.cuh the arithmetic): the path of the mixed forward
// render (ray_fixed.cuh) with the inclination tangent in FP32.
//
// The tangent of a stage's right-hand side runs on the FP32 pipe, which the
// fixed-point code leaves idle.
#include "ray_fixed.cuh"
#include "vjp_f32.cuh"

namespace raptor {
namespace {

// v 2^e of a fixed-point value of order one in its format, from its leading
// word (30 bits, rounded: cut off, its bias would be the same for every ray),
// as a float; scale = 2^(e + 32)
__device__ __forceinline__ float fx_lead(fx v, float scale) { return (float)fx_hi(v) * scale; }
__device__ __forceinline__ float exp2i(int e) { return __int_as_float((e + 127) << 23); }
__device__ __forceinline__ F1 dual(float v, float d) {
    F1 r(v);
    r.d[0] = d;
    return r;
}

// The point with its tangent, given those of x1 and x2 (the sample's metric
// and the right-hand side read it).
struct FxPointF1 {
    F1 r, w, s, c, thp, ithp, isn;
};
__device__ __forceinline__ FxPointF1 fx_point_f1(const FxGeo& g, const FxPoint& q, int n, float d1, float d2) {
    const float r = fx_lead(q.r, exp2i(n - 29)), w = fx_lead(q.w, exp2i(-n - 30));
    const float s = fx_lead(q.s, 0x1p-30f), c = fx_lead(q.c, 0x1p-30f);
    const float thp = fx_lead(q.thp, 0x1p-28f), ithp = fx_lead(q.ithp, 0x1p-29f);
    const float isn = fx_lead(q.isn, exp2i(q.ks - 29));
    const float dthp = fx_lead(g.th2, 0x1p-26f) * fx_lead(q.s2x, 0x1p-30f);
    const float dth = thp * d2;
    FxPointF1 p;
    p.r = dual(r, r * d1);
    p.w = dual(w, -w * d1);
    p.s = dual(s, c * dth);
    p.c = dual(c, -s * dth);
    p.thp = dual(thp, dthp * d2);
    p.ithp = dual(ithp, -ithp * ithp * dthp * d2);
    p.isn = dual(isn, -isn * isn * c * dth);
    return p;
}

// The inclination tangents of x1, x2, k^mu along a step.  A step works in the
// units of fixed_geodesic.cuh (K0..K3, L): the tangent of a stage's right-hand
// side is the differential of fx_rhs term by term, its coefficients the
// fixed-point terms rounded to FP32.
struct FxTangent {
    const FxGeo& g;
    float a, alo;  // the spin in two parts
    float t[6];    // physical, at the step's start, and of the new state once committed
    float tl[6];   // what t's roundings lost so far (FP32 sums' roundings are alike for
                   // neighbouring rays and would add up over the image)
    float y[6];    // t in the step's units
    float ts[6];   // of the stage
    float acc[6];  // the offsets' sum
    float sc0, sc1, sc2, sc3;  // k^mu in physical units per unit of K
    float ev, pn, pp, pu;      // 2^(p-n), 2^-n, 2^-p, 2^u
    float dl, ddl;             // |d lambda| (physical) and its tangent
    float L, dL;               // the step (negative) in its units
    bool rk2;

    __device__ FxTangent(const DevImage& im, const float (&t0)[6], const float (&l0)[6])
        : g(im.fx), a(im.geo_df.a.hi), alo(im.geo_df.a.lo), rk2(im.integrator == 2) {
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            t[i] = t0[i];
            tl[i] = l0[i];
        }
    }
    __device__ __forceinline__ void begin(const FxState& s, const FxPoint&, fx Lf) {
        sc0 = exp2i(s.m);
        sc1 = exp2i(s.m - s.n);
        sc2 = exp2i(s.m + s.p - 2 * s.n);
        sc3 = exp2i(s.m + s.p + s.u - 2 * s.n);
        ev = exp2i(s.p - s.n);
        pn = exp2i(-s.n);
        pp = exp2i(-s.p);
        pu = exp2i(s.u);
        y[0] = t[0];
        y[1] = t[1];
        y[2] = t[2] * exp2i(-s.m);
        y[3] = t[3] * exp2i(s.n - s.m);
        y[4] = t[4] * exp2i(2 * s.n - s.m - s.p);
        y[5] = t[5] * exp2i(2 * s.n - s.m - s.p - s.u);
        // dl = eps m2 / D, D = m2 (|k1| + |k3|) + |k2| (fx_step_size)
        const float x2 = fx_float(s.x2, -62);
        const bool up = s.x2 > fx_one(61);
        const float m2 = up ? fx_float(fx_one(62) - s.x2, -62) : x2, dm2 = up ? -y[1] : y[1];
        const float k1 = fx_float(s.k1, -61), V2 = fx_float(s.k2, s.p - s.n - 61);
        const float V3 = fx_float(s.k3, s.p + s.u - s.n - 61);
        const float dV2 = y[4] * ev, dV3 = y[5] * ev * pu;
        const float i13 = fabsf(k1) + fabsf(V3);
        const float di13 = (k1 < 0.0f ? -y[3] : y[3]) + (V3 < 0.0f ? -dV3 : dV3);
        const float D = m2 * i13 + fabsf(V2);
        const float dV2a = V2 < 0.0f ? -dV2 : dV2;
        L = -fx_float(Lf, -62);
        dL = L * fdiv(fabsf(V2) * fdiv(dm2, m2) - m2 * di13 - dV2a, D);
        const float un = exp2i(s.n - s.m);
        dl = -L * un;
        ddl = -dL * un;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            ts[i] = y[i];
            acc[i] = 0.0f;
        }
    }
    // stage q: the differentials of the terms o of fx_rhs (those of order one
    // from their leading words, the products that shrink with 1/r or the
    // angular momentum formed in FP32: from the fixed-point terms instead,
    // d_inclination is as far from the FP64 adjoint's, 2.8e-6 in the median
    // view, and the pass 7 % slower), then of the offset h f (h = L/2, L/2, L, L/2; RK2 L/2, L)
    __device__ __forceinline__ void stage(int q, int end, const FxPoint& pt, const FxTerms& o, fx k0f, fx k1f, fx k2f,
                                          fx k3f) {
#define Q(x, f) fx_lead(x, 0x1p32f / (float)(1ull << (f)))
        const float dx1 = ts[0], dx2 = ts[1], d0 = ts[2], d1 = ts[3], d2 = ts[4], d3 = ts[5];
        const float k0 = Q(k0f, 61), k1 = fx_float(k1f, -61), k2 = fx_float(k2f, -61), k3 = fx_float(k3f, -61);
        const float V2 = k2 * ev, V3 = k3 * ev;
        const float dV2 = d2 * ev, dV3 = d3 * ev;
        // the point
        const float r = Q(pt.r, 61), wt = Q(pt.w, 62), s = Q(pt.s, 62), c = Q(pt.c, 62), thp = Q(pt.thp, 60);
        const float ithp = Q(pt.ithp, 61), isn = fx_lead(pt.isn, exp2i(pt.ks - 29));
        const float g2 = Q(o.g2, 59), th2 = g2 * thp;  // theta''/theta', theta''
        const float dth = thp * dx2, ds = c * dth, dthp = th2 * dx2, dithp = -ithp * ithp * dthp;
        const float pt2 = ((thp - 3.14159274f) + 8.74227766e-8f) * dx2;
        const float dth2 = -(39.4784164f * pt2 + 1.16148634e-06f * pt2);  // -4 pi^2 (theta' - pi) dx2
        const float w = wt * pn, dw = -w * dx1, dwt = -wt * dx1;
        const float ww = w * wt, dww = -2.0f * ww * dx1, wt2 = Q(o.wt2, 62), dwt2 = -2.0f * wt2 * dx1;
        const float wt3 = wt2 * wt, dwt3 = -3.0f * wt3 * dx1;
        // metric functions
        const float aw = a * w + alo * w, daw = -aw * dx1;
        const float a2w2 = aw * aw, da2w2 = -2.0f * a2w2 * dx1;
        const float s2 = Q(o.s2, 62), sc = Q(o.sc, 62), ds2 = 2.0f * sc * dth, dsc = (1.0f - 2.0f * s2) * dth;
        const float sg = Q(o.sg, 61), dsg = da2w2 * (1.0f - s2) - a2w2 * ds2;
        const float isg = Q(o.isg, 62), isg2 = Q(o.isg2, 62), isg3 = Q(o.isg3, 62);
        const float disg = -isg2 * dsg, disg2 = 2.0f * isg * disg, disg3 = 3.0f * isg2 * disg;
        const float rho = Q(o.rho, 61), drho = da2w2, dlt = Q(o.dl, 61), ddlt = drho - 2.0f * dw;
        const float beta = Q(o.beta, 62), bw = beta * w;
        const float dbeta = (2.0f - sg) * disg3 - dsg * isg3, dbw = dbeta * w + beta * dw;
        const float gam = Q(o.gam, 62), dgam = disg - (da2w2 * s2 + a2w2 * ds2) * bw - a2w2 * s2 * dbw;
        const float thi = Q(o.thi, 60), dthi = dthp * isg + thp * disg;
        const float tt = a2w2 * sc * thi, dt = (da2w2 * sc + a2w2 * dsc) * thi + a2w2 * sc * dthi;
        const float tw = tt * isg * w, dtw = (dt * isg + tt * disg) * w + tt * isg * dw;
        // wave vector
        const float as2 = a * s2 + alo * s2, P = as2 * V3 * pu * pn, dP = (as2 * dV3 + a * ds2 * V3) * pu * pn;
        const float R1 = Q(o.R1, 60), dR1 = r * d1 + R1 * dx1, S = Q(o.S, 60), dS = d0 + dR1;
        const float H = Q(o.H, 59), dH = 2.0f * S * dS;
        const float X0 = Q(o.X0, 59), dX0 = 2.0f * ((k0 - P) * d0 - k0 * dP);
        const float Y = Q(o.Y, 60), dY = d1 * (k0 - P) + k1 * (d0 - dP);
        const float QQ = k1 * k1, dQ = 2.0f * k1 * d1;
        const float RK = Q(o.RK, 60), dRK = dR1 * k1 + R1 * d1;
        const float kap2 = thp * V2, dkap2 = dthp * V2 + thp * dV2;
        const float kap3 = s * V3 * pu, dkap3 = (ds * V3 + s * dV3) * pu;
        const float mu = isg * kap2 * kap2 + gam * kap3 * kap3;
        const float dmu = (disg * kap2 + 2.0f * isg * dkap2) * kap2 + (dgam * kap3 + 2.0f * gam * dkap3) * kap3;
        const float sg2w = sg + 2.0f * w, dsg2w = dsg + 2.0f * dw;
        // E0, E1
        const float s0 = Q(o.s0, 58), s1 = Q(o.s1, 58), SP = S - P;
        const float ds0 = dww * X0 + ww * dX0 + dsg2w * Y + sg2w * dY + (dsg + dw) * RK + (sg + w) * dRK;
        const float dE0 = -2.0f * (dbw * s0 + bw * ds0) + 2.0f * pn * dmu +
                          4.0f * ((dtw * V2 + tw * dV2) * SP + tw * V2 * (dS - dP));
        const float ds1 = (dwt2 * dlt + wt2 * ddlt) * X0 + wt2 * dlt * dX0 +
                          2.0f * ((dwt * (dlt - sg) + wt * (ddlt - dsg)) * Y + wt * (dlt - sg) * dY) -
                          (2.0f * dsg - ddlt) * QQ - (2.0f * sg - dlt) * dQ;
        const float dE1 = -dbw * s1 - bw * ds1 - dQ -
                          2.0f * ((disg * wt + isg * dwt) * k1 * P + isg * wt * (d1 * P + k1 * dP)) +
                          2.0f * (dt * k1 * V2 + tt * (d1 * V2 + k1 * dV2)) + ddlt * mu + dlt * dmu;
        // E2
        const float sg2 = Q(o.sg2, 60), dsg2 = 2.0f * sg * dsg;
        const float wr2 = 2.0f * w * rho, dwr2 = 2.0f * (dw * rho + w * drho);
        const float rww = 2.0f * rho * ww, drww = 2.0f * (drho * ww + rho * dww);  // 2 rho w w~
        const float F1v = Q(o.F1, 58), dF1 = (dsg2 + dwr2) * k1 + (sg2 + wr2) * d1 + drww * k0 + rww * d0;
        const float F2 = Q(o.F2, 60), dF2 = ddlt * sg2 + dlt * dsg2 + dwr2 * rho + wr2 * drho;
        const float z = Q(o.z, 62), dz = (dsc * isg3 + sc * disg3) * ithp + sc * isg3 * dithp;
        const float A = 2.0f * a2w2 * wt3 * pp, dA = -5.0f * A * dx1;  // 2 a^2 w^2 w~^3 2^-p
        const float dg2 = dth2 * ithp + th2 * dithp;
        const float ipu = __fdividef(1.0f, pu);
        const float G = Q(o.G, 57), dG = dF2 * V3 + F2 * dV3 - 2.0f * ipu * (daw * F1v + aw * dF1);
        const float dE2 = (dz * A + z * dA) * H + z * A * dH - 2.0f * (disg * k1 * k2 + isg * (d1 * k2 + k1 * d2)) -
                          (dg2 - dt) * k2 * V2 - (g2 - tt) * (d2 * V2 + k2 * dV2) +
                          pu * pu * ((dz * k3 + z * d3) * G + z * k3 * dG);
        // E3
        const float B = a * bw * wt3 * pp * ipu;  // a beta w w~^3 2^-(p+u)
        const float dB = a * (dbw * wt3 + bw * dwt3) * pp * ipu, HP = H - 2.0f * k0 * P;
        const float wP = wt * P, dwP = dwt * P + wt * dP;
        const float F3 = Q(o.F3, 60), dF3 = 2.0f * (dww * k0 + ww * d0) + dsg2w * k1 + sg2w * d1;
        const float D = k2 * (V3 - ipu * aw * isg2 * F3);
        const float dD = d2 * V3 + k2 * dV3 -
                         ipu * ((daw * isg2 + aw * disg2) * k2 * F3 + aw * isg2 * (d2 * F3 + k2 * dF3));
        const float cot = c * isn, ct = cot * thp, dct = cot * dthp - isn * isn * thp * dth;
        const float kv23 = k2 * V3, dkv23 = d2 * V3 + k2 * dV3;
        const float dE3 = -dB * HP - B * (dH - 2.0f * (d0 * P + k0 * dP)) -
                          (dgam * k3 + gam * d3) * (2.0f * k1 - wP) - gam * k3 * (2.0f * d1 - dwP) +
                          ipu * ((daw * kap2 + aw * dkap2) * thi * k2 + aw * kap2 * (dthi * k2 + thi * d2)) -
                          4.0f * (dtw * kv23 + tw * dkv23) - 2.0f * (dct * D + ct * dD);
        const float E0 = Q(o.E0, 60), E1 = Q(o.E1, 60);
        const float E2 = Q(o.E2a, 57) + Q(o.E2b, 57) * pu * pu * exp2i(-pt.ks);
        const float E3 = Q(o.E3a, 57) + 2.0f * Q(o.E3b, 58) * exp2i(pt.ks);
#undef Q
        const bool whole = q == end - 2 + (rk2 ? 1 : 0);
        const float h = whole ? L : 0.5f * L, dh = whole ? dL : 0.5f * dL;
        const float f[6] = {k1, V2, E0, E1, E2, E3}, df[6] = {d1, dV2, dE0, dE1, dE2, dE3};
        const float wq = q == 1 ? 2.0f : 1.0f;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const float off = h * df[i] + dh * f[i];
            acc[i] = rk2 ? off : acc[i] + wq * off;
            ts[i] = y[i] + off;
        }
    }
    __device__ __forceinline__ void commit() {
        const float un[6] = {1.0f, 1.0f, sc0, sc1, sc2, sc3};
#pragma unroll
        // a third in two parts: FP32's own is 3e-8 off, the same for every ray and step
        for (int i = 0; i < 6; ++i) {
            // acc: RK4's 3 offsets' worth, or RK2's offset
            const float d = (rk2 ? acc[i] : acc[i] * (1.0f / 3.0f) + acc[i] * -9.934107e-9f) * un[i] + tl[i];
            const float sum = __fadd_rn(t[i], d), b = __fsub_rn(sum, t[i]);
            tl[i] = __fadd_rn(__fsub_rn(t[i], __fsub_rn(sum, b)), __fsub_rn(d, b));
            t[i] = sum;
        }
    }
};

using DT = Dual<1, double, float>;

// A step outside the fixed-point ranges: FP64 with FP32 tangents, as
// FormMixed's (vjp_df.cu).  d: |dl| and its tangent.
__device__ __noinline__ void fx_slow_step_tangent(const DevImage& im, FxState* c, float* t, float* d) {
    double y0[6];
    fx_decode(*c, y0);
    DT y[8];
    y[0] = DT(0.0);
    y[3] = DT(0.0);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const int at = i < 2 ? i + 1 : i + 2;
        y[at] = DT(y0[i]);
        y[at].d[0] = t[i];
    }
    MksPointT<DT> p;
    mks_point(y[1], y[2], im.geo, p);
    const DT dl = step_size(im, y);
    if (im.integrator == 2) rk2_step<DT, Geo, false>(im.geo, y, p, dl);
    else rk4_step_rolled<DT, Geo, false>(im.geo, y, p, dl);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const int at = i < 2 ? i + 1 : i + 2;
        y0[i] = y[at].v;
        t[i] = y[at].d[0];
    }
    fx_encode(im.fx, y0, c);
    const DT ad = fabs(dl);
    d[0] = (float)ad.v;
    d[1] = ad.d[0];
}

// The sample's point of a raw state: the FP64 point with FP32 tangents.
__device__ __noinline__ void fx_slow_point_tangent(const DevImage& im, const FxState* c, const float* t,
                                                   MksPointT<F1>* out) {
    double y[6];
    fx_decode(*c, y);
    DT x1(y[0]), x2(y[1]);
    x1.d[0] = t[0];
    x2.d[0] = t[1];
    MksPointT<DT> p;
    mks_point(x1, x2, im.geo, p);
    out->r = to_f1(p.r);
    out->s = to_f1(p.s);
    out->iS = to_f1(p.iS);
    out->irp = to_f1(p.irp);
    out->ithp = to_f1(p.ithp);
    out->isn = to_f1(p.isn);
    out->thp = to_f1(p.thp);
    out->Sg = to_f1(p.Sg);
}

struct FormFx {
    struct State {
        FxState c;
        FxPoint pt;
        float t[6], tl[6];  // tangents of x1, x2, k^mu, and what their roundings lost
    };
    struct Step {
        float adl, dadl;  // |d lambda| and its tangent
    };
    using Th = int;
    static constexpr bool kMergeReplay = true;  // vjp_f32_body's record replay
    __device__ static void start(const DevImage& im, const D1 (&y0)[8], State& g) {
        double d[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const int at = i < 2 ? i + 1 : i + 2;
            d[i] = y0[at].v;
            g.t[i] = (float)y0[at].d[0];
            g.tl[i] = (float)(y0[at].d[0] - (double)g.t[i]);
        }
        FxState c;
        fx_encode(im.fx, d, &c);
        g.c = c;
        if (!c.raw) {
            FxPoint pt;
            fx_start_point(im.fx, &c, &pt);
            g.pt = pt;
        }
    }
    __device__ static bool alive(const DevImage& im, const State& g, int steps, int stop) {
        return fx_in_range(im, g.c) && steps < (int)kMaxSteps && !stop;
    }
    __device__ static Th theta_rate(const State& g) { return fx_theta_sign(g.c); }
    __device__ static bool turned(Th prev, Th now) { return prev * now < 0; }
    __device__ static bool escaped(const DevImage& im, const State& g) { return fx_escaped(im, g.c); }
    __device__ static bool in_grid(const DevImage& im, const State& g) { return fx_in_grid(im, g.c); }
    __device__ static bool finite(const State& g) {
        return !g.c.raw || (isfinite(__longlong_as_double(g.c.x1)) && isfinite(__longlong_as_double(g.c.k1)));
    }
    __device__ static void advance(const DevImage& im, State& g, Step& step) {
        FxTangent tan(im, g.t, g.tl);
        double dl = 0.0;
        bool fixed = true;
        const auto slow = [&](FxState& st) {
            FxState c = st;
            float t[6], d[2];
#pragma unroll
            for (int i = 0; i < 6; ++i) t[i] = tan.t[i];
            fx_slow_step_tangent(im, &c, t, d);
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                tan.t[i] = t[i];
                tan.tl[i] = 0.0f;
            }
            st = c;
            step.adl = d[0];
            step.dadl = d[1];
            fixed = false;
            return 0.0;
        };
        fx_step(im.fx, g.c, g.pt, tan.rk2, dl, slow, tan);
        if (fixed) {
            step.adl = tan.dl;
            step.dadl = tan.ddl;
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            g.t[i] = tan.t[i];
            g.tl[i] = tan.tl[i];
        }
    }
    template <bool K>
    __device__ static bool sample(const DevImage& im, const State& g, const Step& step, SampleCommonF& out) {
        const FxState& c = g.c;
        MksPointT<F1> p;
        double x[6];
        fx_decode(c, x);
        if (!c.raw) {
            const FxPointF1 q = fx_point_f1(im.fx, g.pt, c.n, g.t[0], g.t[1]);
            fx Sg, iS;
            fx_sigma(im.fx, g.pt, c.n, Sg, iS);
            const float Sgf = fx_float(Sg, 2 * c.n - 60), iSf = fx_float(iS, -62 - 2 * c.n);
            const float dSg = 2.0f * (q.r.v * q.r.d[0] + im.geo_df.a2.hi * q.c.v * q.c.d[0]);
            p.r = q.r;
            p.s = q.s;
            p.Sg = dual(Sgf, dSg);
            p.iS = dual(iSf, -iSf * iSf * dSg);
            p.irp = q.w;
            p.thp = q.thp;
            p.ithp = q.ithp;
            p.isn = q.isn;
        } else {
            FxState cc = c;
            float t[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) t[i] = g.t[i];
            MksPointT<F1> pp;
            fx_slow_point_tangent(im, &cc, t, &pp);
            p = pp;
        }
        const MetricT<F1> m = metric_f1(p, im.geo_df);
        const CellCoef cc = cell_coef(im, x[0], x[1]);
        const int i = cc.base / im.n2, j = cc.base - i * im.n2;
        F1 d1(f32_of(cc.d1)), d2(f32_of(cc.d2));
        const double t1 = (x[0] - im.startx1) * im.idx1 - 0.5;
        const double t2 = (x[1] - im.startx2) * im.idx2 - 0.5;
        if ((int)t1 == i) d1.d[0] = g.t[0] * im.idx1_df.hi;  // not clamped
        if ((int)t2 == j) d2.d[0] = g.t[1] * im.idx2_df.hi;
        const F1 k[4] = {dual(f32_of(x[2]), g.t[2]), dual(f32_of(x[3]), g.t[3]), dual(f32_of(x[4]), g.t[4]),
                         dual(f32_of(x[5]), g.t[5])};
        return sample_common_f<K>(im, m, cc.base, d1, d2, k, dual(step.adl, step.dadl), out);
    }
};

// 2 blocks of 128 per SM (255 registers, no spills); 3 (168 registers) were
// 3 % slower at 512x512 and five frequencies, 4 slower still.
#ifndef RAPTOR_VJP_FX_BLOCKS
#define RAPTOR_VJP_FX_BLOCKS 2
#endif

template <int NF, bool K, bool TAPE>
__global__ void __launch_bounds__(kVjpBlock, RAPTOR_VJP_FX_BLOCKS)
    vjp_kernel_fx(const DevImage* __restrict__ imp, CamT<D1> cam, const double* __restrict__ fwd,
                  const double* __restrict__ dLdO, unsigned long long* __restrict__ counters,
                  double* __restrict__ gscal, double* __restrict__ g_rho, double* __restrict__ g_u,
                  double* __restrict__ g_th, int refill_interval, RayRange rr, VjpTape tape) {
    vjp_f32_body<NF, FormFx, K, TAPE>(*imp, cam, fwd, dLdO, counters, gscal, g_rho, g_u, g_th, refill_interval, rr,
                                      tape);
}

template <int NF, bool K, bool TAPE>
void launch_vjp_fx(int grid, cudaStream_t st, const DevImage* im, const CamT<D1>& cam, const double* fwd,
                   const double* dl, unsigned long long* ctr, double* gs, double* gr, double* gu, double* gt,
                   int refill, double*, RayRange rr, VjpTape tape) {
    vjp_kernel_fx<NF, K, TAPE><<<grid, kVjpBlock, 0, st>>>(im, cam, fwd, dl, ctr, gs, gr, gu, gt, refill, rr, tape);
}

template <bool TAPE>
VjpLaunchFn pick_fx(int nf, const void** fn, bool kappa) {
    if (kappa) {
        *fn = (const void*)vjp_kernel_fx<kMaxFreqs, true, TAPE>;
        return launch_vjp_fx<kMaxFreqs, true, TAPE>;
    }
    if (nf <= 1) {
        *fn = (const void*)vjp_kernel_fx<1, false, TAPE>;
        return launch_vjp_fx<1, false, TAPE>;
    }
    *fn = (const void*)vjp_kernel_fx<kMaxFreqs, false, TAPE>;
    return launch_vjp_fx<kMaxFreqs, false, TAPE>;
}

}  // namespace

VjpLaunchFn pick_vjp_fx(int nf, const void** fn, bool kappa, bool tape) {
    return tape ? pick_fx<true>(nf, fn, kappa) : pick_fx<false>(nf, fn, kappa);
}

}  // namespace raptor
