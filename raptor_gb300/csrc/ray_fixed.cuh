// Rays of the FP64 and mixed forms whose geodesic runs in fixed point
// (fixed_geodesic.cuh): the state type that the kernels of ray_kernel.cuh
// take in place of RayState, for the images that fx.ok marks.
//
// A ray is six 64-bit words.  They hold the fixed-point state, or - while the
// ray is where that arithmetic does not cover it: close to the polar axis,
// with a very large angular wave vector, or not finite - the doubles x1, x2,
// k^mu, which then step in FP64 (fx_slow_step) until they fit again.  On the
// 1024x1024 image of the torus at 60 degrees that is 0.02 % of the steps, at 2
// degrees 0.3 % (30 % where L 2^ks was held below 1 instead of shortened,
// fx_excess: FP64 771 ms against 298).
#pragma once
#include "ray_kernel.cuh"

namespace raptor {

// fx_double's value as a float: the leading 32 bits rounded, then the exponent
__device__ __forceinline__ float fx_float(fx v, int e) {
    const ufx u = (ufx)fx_abs(v);
    const int lz = fx_clz(u);
    const unsigned m = (unsigned)((u << (lz & 63)) >> 32);
    const int b = __float_as_int(__uint2float_rn(m)) + ((32 - lz + e) << 23);
    return __int_as_float(u ? (b | ((int)(v >> 32) & 0x80000000)) : 0);
}
// round(v 2^b)
__device__ __forceinline__ fx fx_of(double v, int b) { return __double2ll_rn(scalbn(v, b)); }

// Doubles x1, x2, k^mu into c: the fixed-point state where fx_step covers it,
// else as they are.
static __device__ __noinline__ void fx_encode(const FxGeo& g, const double* y, FxState* c) {
    const double x1 = y[0], x2 = y[1];
    bool ok = g.ok && x1 > 0.0 && x1 < 9.7 && x2 > 0.0001220703125 && x2 < 0.9998779296875;
#pragma unroll
    for (int i = 2; i < 6; ++i) ok = ok && fabs(y[i]) < 1e30;
    if (ok) {
        const int n = (int)floor(x1 * 1.4426950408889634);
        const double k1 = scalbn(y[3], n);
        const double a = fmax(fabs(y[2]), fabs(k1));
        ok = a > 1e-30;
        const int m = ilogb(a) + 1;
        // the exponents of fx_normalise
        const int q2 = fabs(y[4]) > 1e-30 ? ilogb(y[4]) + 1 + 2 * n - m : -1;
        const int q3 = fabs(y[5]) > 1e-30 ? ilogb(y[5]) + 1 + 2 * n - m : -1;
        const int p = max(max(min(q3, n + 3), q2), 0), u = max(q3 - p, 0);
        ok = ok && p - n <= 3 && u <= 11;
        if (ok) {
            c->n = n;
            c->m = m;
            c->p = p;
            c->u = u;
            c->raw = 0;
            c->x1 = fx_of(x1, 59);
            c->x2 = fx_of(x2, 62);
            c->k0 = fx_of(y[2], 61 - m);
            c->k1 = fx_of(y[3], 61 + n - m);
            c->k2 = fx_of(y[4], 61 + 2 * n - m - p);
            c->k3 = fx_of(y[5], 61 + 2 * n - m - p - u);
            return;
        }
    }
    c->n = c->m = c->p = c->u = 0;
    c->raw = 1;
    c->x1 = __double_as_longlong(y[0]);
    c->x2 = __double_as_longlong(y[1]);
    c->k0 = __double_as_longlong(y[2]);
    c->k1 = __double_as_longlong(y[3]);
    c->k2 = __double_as_longlong(y[4]);
    c->k3 = __double_as_longlong(y[5]);
}

// x1, x2, k^mu as doubles
__device__ __forceinline__ void fx_decode(const FxState& c, double y[6]) {
    if (c.raw) {
        y[0] = __longlong_as_double(c.x1);
        y[1] = __longlong_as_double(c.x2);
        y[2] = __longlong_as_double(c.k0);
        y[3] = __longlong_as_double(c.k1);
        y[4] = __longlong_as_double(c.k2);
        y[5] = __longlong_as_double(c.k3);
        return;
    }
    y[0] = fx_double(c.x1, -59);
    y[1] = fx_double(c.x2, -62);
    y[2] = fx_double(c.k0, c.m - 61);
    y[3] = fx_double(c.k1, c.m - c.n - 61);
    y[4] = fx_double(c.k2, c.m + c.p - 2 * c.n - 61);
    y[5] = fx_double(c.k3, c.m + c.p + c.u - 2 * c.n - 61);
}

// One step in FP64 (step_size and rk4_step or rk2_step of ray_kernel.cuh);
// returns |d lambda|.
static __device__ __noinline__ double fx_slow_step(const DevImage& im, FxState* c) {
    double d[6];
    fx_decode(*c, d);
    double y[8] = {0.0, d[0], d[1], 0.0, d[2], d[3], d[4], d[5]};
    MksPoint p;
    mks_point(y[1], y[2], im.geo, p);
    const double dl = step_size(im, y);
    if (im.integrator == 2) rk2_step<double, Geo, false>(im.geo, y, p, dl);
    else rk4_step<double, Geo, false>(im.geo, y, p, dl);
    d[0] = y[1];
    d[1] = y[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) d[2 + i] = y[4 + i];
    fx_encode(im.fx, d, c);
    return fabs(dl);
}

static __device__ __noinline__ void fx_slow_point(const DevImage& im, double x1, double x2, MksPoint* p) {
    mks_point(x1, x2, im.geo, *p);
}
// the point where a ray starts, once per ray
static __device__ __noinline__ void fx_start_point(const FxGeo& g, const FxState* c, FxPoint* pt) {
    fx_point(g, fx_log2r(c->x1) - fx_shl((fx)c->n, 57), c->x2, *pt);
}

// Sigma and 1/Sigma of a point: Sigma 2^(-2n) in Q60, 2^(2n)/Sigma in Q62
__device__ __forceinline__ void fx_sigma(const FxGeo& g, const FxPoint& q, int n, fx& Sg, fx& iS) {
    fx a2w2, s2, sg;
    const fx isg = fx_isigma(g, q, n, a2w2, s2, sg);
    Sg = mulk<3>(sqrk<2>(q.r), sg);
    iS = mulk<2>(isg, sqrk<2>(q.w));
}

// The FP64 sample's inputs from a state and the point at it: x1, x2, k^mu and
// the point's quantities, each rounded once from fixed point.
__device__ __forceinline__ void fx_sample_inputs(const DevImage& im, const FxState& c, const FxPoint& q, double y[8],
                                                 MksPoint& mp) {
    double d[6];
    fx_decode(c, d);
    y[0] = 0.0;
    y[1] = d[0];
    y[2] = d[1];
    y[3] = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) y[4 + i] = d[2 + i];
    if (c.raw) {
        MksPoint t;
        fx_slow_point(im, d[0], d[1], &t);
        mp = t;
        return;
    }
    fx Sg, iS;
    fx_sigma(im.fx, q, c.n, Sg, iS);
    mp.rp = 0.0;  // the metric does not read rp, s2x, c2x
    mp.s2x = 0.0;
    mp.c2x = 0.0;
    mp.r = fx_double(q.r, c.n - 61);
    mp.s = fx_double(q.s, -62);
    mp.c = fx_double(q.c, -62);
    mp.Sg = fx_double(Sg, 2 * c.n - 60);
    mp.thp = fx_double(q.thp, -60);
    mp.iS = fx_double(iS, -62 - 2 * c.n);
    mp.irp = fx_double(q.w, -62 - c.n);
    mp.ithp = fx_double(q.ithp, -61);
    mp.isn = fx_double(q.isn, q.ks - 61);
}

// The tests of advance_ray (ray_kernel.cuh) on the fixed-point state, on ln r
// where that one compares r: within the cut-off radii, the sign of k^2,
// escaped outward, inside the sampling region.
__device__ __forceinline__ bool fx_in_range(const DevImage& im, const FxState& c) {
    if (!c.raw) return c.x1 < im.fx.ln_outer && c.x1 > im.fx.ln_inner;
    const double r = exp(__longlong_as_double(c.x1));
    return r < kCutoffOuter && r > im.cutoff_inner;
}
__device__ __forceinline__ int fx_theta_sign(const FxState& c) {
    if (!c.raw) return c.k2 > 0 ? 1 : (c.k2 < 0 ? -1 : 0);
    const double k2 = __longlong_as_double(c.k2);
    return k2 > 0.0 ? 1 : (k2 < 0.0 ? -1 : 0);
}
__device__ __forceinline__ bool fx_escaped(const DevImage& im, const FxState& c) {
    if (!c.raw) return c.x1 > im.fx.stopx1 && c.k1 < 0;
    return __longlong_as_double(c.x1) > im.stopx1 && __longlong_as_double(c.k1) < 0.0;
}
__device__ __forceinline__ bool fx_in_grid(const DevImage& im, const FxState& c) {
    if (!c.raw)
        return c.x1 < im.fx.stopx1 && c.x1 > im.fx.startx1 && c.x2 > im.fx.startx2 && c.x2 < im.fx.stopx2;
    const double x1 = __longlong_as_double(c.x1), x2 = __longlong_as_double(c.x2);
    return x1 < im.stopx1 && x1 > im.startx1 && x2 > im.startx2 && x2 < im.stopx2;
}

// Blocks: 128-thread blocks per SM the kernels are compiled for.  They wait on
// instruction fetch and on the multiply-adds' latency, which more warps hide,
// but 4 blocks (128 registers) spill where 3 (168) hardly do and 2 (255) do
// not at all; a launch of few rays per lane lasts as long as its longest rays
// and is better off with fewer, quicker warps.  FP64, one frequency (ms at 4,
// 3, 2 blocks): 1024x1024 195, 205, 229; 800x800 122, 126; 512x512 59.1, 52.6,
// 58.7; 360x360 29.5 at 3, 31.1 at 2; 320x320 25.7, 25.1; 256x256 20.8, 19.4;
// five frequencies 320x320 37.1, 38.4; 256x256 29.7, 27.6: kFxFewRays and
// kFxManyRays rays part them.  Mixed (3, 2 blocks): 1024x1024 120 (127 at 4);
// 512x512 33.9, 36.0; 400x400 22.9, 23.3; 360x360 20.5, 19.8; 256x256 16.7,
// 14.8; 128x128 11.7, 10.7; five frequencies 320x320 24.0, 20.2: kFxFewRaysMixed.
// 5 blocks (96 registers) are slower throughout.
// A barrier per step (kLockstep, which only the pooled kernel reads) keeps the
// four warps of a block on the same code: 1024x1024 214 -> 202 ms.  The lines
// between the kernels are numbers of rays on GB300's 152 SMs.
constexpr long long kFxFewRays = 3ll << 15, kFxManyRays = 1ll << 19;
constexpr long long kFxFewRaysMixed = 1ll << 17;

template <int NF, bool MIXED, int Blocks>
struct FxRay {
    static constexpr int kTicketRows = 15;
    static constexpr int kRayBlocks = Blocks, kPoolBlocks = Blocks;
    static constexpr bool kLockstep = true;
    FxState c;
    FxPoint pt;  // at c's position (not formed while c is raw)
    int bsign;       // sign of the impact parameter beta
    int thdot_prev;  // sign of k^2 at the previous step
    int steps, turns, stop, img, pix;
    double tau[NF], I[NF];
    float tf[NF], tc[NF], If[NF], Ic[NF];
};

template <int NF, bool MIXED, int Blocks>
__device__ __forceinline__ const DevImage* start_ray(const DevImage* __restrict__ imgs, int n_imgs, long long rid,
                                                     FxRay<NF, MIXED, Blocks>& s) {
    s.img = find_image(imgs, n_imgs, rid);
    if (!chk(s.img >= 0 && s.img < n_imgs, imgs[0].check_word, kChkImage, s.img)) return nullptr;
    const DevImage* im = imgs + s.img;
    s.pix = (int)(rid - im->ray_begin);
    if (!chk(rid >= im->ray_begin && rid - im->ray_begin < (long long)im->width * im->height, im->check_word,
             kChkPixel, rid))
        return nullptr;
    double y[8];
    double beta;
    init_photon(*im, camera_of(*im), s.pix % im->width, s.pix / im->width, y, beta);
    s.bsign = beta < 0.0 ? -1 : (beta > 0.0 ? 1 : 0);
    const double d[6] = {y[1], y[2], y[4], y[5], y[6], y[7]};
    FxState c;
    fx_encode(im->fx, d, &c);
    s.c = c;
    if (!c.raw) {
        FxPoint pt;
        fx_start_point(im->fx, &c, &pt);
        s.pt = pt;
    }
    s.steps = 0;
    s.turns = 0;
    s.stop = 0;
    s.thdot_prev = 0;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        s.tau[f] = 0.0; s.I[f] = 0.0;
        s.tf[f] = 0.f; s.tc[f] = 0.f; s.If[f] = 0.f; s.Ic[f] = 0.f;
    }
    return im;
}

template <int NF, bool MIXED, int Blocks>
__device__ __forceinline__ void finish_ray(const DevImage& im, const FxRay<NF, MIXED, Blocks>& s, double* __restrict__ out,
                                           RayCounters& c) {
    RayState<NF, MIXED> r;  // finish_ray reads of it the position, wave vector, sums and step count
    double d[6];
    fx_decode(s.c, d);
    r.y[0] = r.y[3] = 0.0;
    r.y[1] = d[0];
    r.y[2] = d[1];
#pragma unroll
    for (int i = 0; i < 4; ++i) r.y[4 + i] = d[2 + i];
    MksPoint p;
    fx_slow_point(im, d[0], d[1], &p);
    r.p = p;
    r.steps = s.steps;
    r.pix = s.pix;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        r.tau[f] = s.tau[f];
        r.I[f] = s.I[f];
        r.If[f] = s.If[f];
        r.Ic[f] = s.Ic[f];
    }
    finish_ray<NF, MIXED>(im, r, out, c);
}

// advance_ray of ray_kernel.cuh on the fixed-point state.
template <bool TPhi, int NF, bool MIXED, int Blocks>
__device__ __forceinline__ int advance_ray(const DevImage& im, FxRay<NF, MIXED, Blocks>& s, double& dl) {
    static_assert(!TPhi, "t and phi are not integrated in fixed point");
    FxState& c = s.c;
    const int th = fx_theta_sign(c);
    if (!(fx_in_range(im, c) && s.steps < (int)kMaxSteps && !s.stop)) return -1;
    if (s.thdot_prev * th < 0 && s.steps > 2) s.turns += 1;
    s.thdot_prev = th;
    if ((s.bsign < 0 && s.turns > kMaxOrder) || (s.bsign > 0 && s.turns > kMaxOrder + 1)) s.stop = 1;
    FxNoTangent none;
    const auto slow = [&](FxState& st) {
        FxState t = st;
        const double d = fx_slow_step(im, &t);
        st = t;
        return d;
    };
    fx_step(im.fx, c, s.pt, im.integrator == 2, dl, slow, none);
    s.steps += 1;
    if (fx_escaped(im, c)) return 3;
    return fx_in_grid(im, c) ? 1 : 0;
}

template <int NF, bool MIXED, int Blocks>
__device__ __forceinline__ bool sample_ray(const DevImage& im, FxRay<NF, MIXED, Blocks>& s, double dl) {
    double y[8];
    MksPoint mp;
    if constexpr (MIXED) {
        if (!s.c.raw) {
            const FxState& c = s.c;
            const FxPoint& q = s.pt;
            fx Sg, iS;
            fx_sigma(im.fx, q, c.n, Sg, iS);
            const PointF32 pf{fx_float(q.r, c.n - 61),      fx_float(q.s, -62),   fx_float(iS, -62 - 2 * c.n),
                              fx_float(q.thp, -60),         fx_float(Sg, 2 * c.n - 60),
                              fx_float(q.w, -62 - c.n),     fx_float(q.ithp, -61), fx_float(q.isn, q.ks - 61)};
            const float k[4] = {fx_float(c.k0, c.m - 61), fx_float(c.k1, c.m - c.n - 61),
                                fx_float(c.k2, c.m + c.p - 2 * c.n - 61),
                                fx_float(c.k3, c.m + c.p + c.u - 2 * c.n - 61)};
            return rt_sample_fp32_at<NF>(im, pf, fx_double(c.x1, -59), fx_double(c.x2, -62), k, dl, s.tf, s.tc,
                                         s.If, s.Ic);
        }
        fx_sample_inputs(im, s.c, s.pt, y, mp);
        return rt_sample_fp32<NF>(im, y, mp, dl, s.tf, s.tc, s.If, s.Ic);
    } else {
        fx_sample_inputs(im, s.c, s.pt, y, mp);
        return rt_sample_fp64<NF>(im, y, mp, dl, s.tau, s.I);
    }
}

// The sample pool's tickets: rows 1-6 the state's words, row 7 its exponents
// (with the point's ks), rows 8-14 the point.
template <int NF, int Blocks>
__device__ __forceinline__ void put_ticket(const FxRay<NF, false, Blocks>& s, double* e) {
    constexpr int C = kPoolCap;
    const fx w[6] = {s.c.x1, s.c.x2, s.c.k0, s.c.k1, s.c.k2, s.c.k3};
    const fx q[7] = {s.pt.r, s.pt.w, s.pt.s, s.pt.c, s.pt.thp, s.pt.ithp, s.pt.isn};
#pragma unroll
    for (int i = 0; i < 6; ++i) e[(1 + i) * C] = __longlong_as_double(w[i]);
    e[7 * C] = __hiloint2double((s.c.m << 16) | (s.c.u << 8) | s.c.p, (s.pt.ks << 16) | (s.c.raw << 8) | s.c.n);
#pragma unroll
    for (int i = 0; i < 7; ++i) e[(8 + i) * C] = __longlong_as_double(q[i]);
}
template <int NF, int Blocks>
struct TicketReader<FxRay<NF, false, Blocks>> {
    static __device__ __forceinline__ void get(const DevImage& im, const double* e, double y[8], MksPoint& mp) {
        constexpr int C = kPoolCap;
        FxState c;
        FxPoint q;
        const int hi = __double2hiint(e[7 * C]), lo = __double2loint(e[7 * C]);
        c.x1 = __double_as_longlong(e[1 * C]);
        c.x2 = __double_as_longlong(e[2 * C]);
        c.k0 = __double_as_longlong(e[3 * C]);
        c.k1 = __double_as_longlong(e[4 * C]);
        c.k2 = __double_as_longlong(e[5 * C]);
        c.k3 = __double_as_longlong(e[6 * C]);
        c.m = hi >> 16;
        c.p = hi & 0xff;
        c.u = (hi >> 8) & 0xff;
        c.raw = (lo >> 8) & 1;
        c.n = lo & 0xff;
        q.ks = lo >> 16;
        q.r = __double_as_longlong(e[8 * C]);
        q.w = __double_as_longlong(e[9 * C]);
        q.s = __double_as_longlong(e[10 * C]);
        q.c = __double_as_longlong(e[11 * C]);
        q.s2x = 0;
        q.thp = __double_as_longlong(e[12 * C]);
        q.ithp = __double_as_longlong(e[13 * C]);
        q.isn = __double_as_longlong(e[14 * C]);
        fx_sample_inputs(im, c, q, y, mp);
    }
};

}  // namespace raptor
