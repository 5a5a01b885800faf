// The geodesic of the FP64 and mixed forms in 64-bit fixed point.
//
// GB300 issues 2 FP64 lanes per clock per SM and 64 lanes of 32x32+64-bit
// integer multiply-add: an FP64 operation holds its pipe for as long as 32
// integer multiply-adds hold theirs.  A signed 64x64-bit product needs three
// of them (mulk below) and a 64-bit sum two integer adds, so the geodesic -
// bounded arithmetic whose ranges are known - runs on the integer pipes, with
// 56 to 61 fraction bits where FP64 has 53.  What bounds it there is the two
// integer pipes' issue (multiply-adds, and the shifts and adds around them).
//
// Units.  A ray carries four exponents: n with 2^n <= r < 2^(n+1) when a
// step begins, m for the wave vector, p for its angular part and u for what
// k^3 is larger than that close to the polar axis.  With r~ = r 2^-n in
// [1, 2) and w~ = 1/r~ the state is
//   x1 = ln r, x2, K0 = k^0 2^-m, K1 = k^1 2^(n-m), K2 = k^2 2^(2n-m-p), K3 = k^3 2^(2n-m-p-u),
//   max(|K0|, |K1|) in [1/2, 1), |K2|, |K3| < 1 (0 <= p <= n + 3, u >= 0),
// V2, V3 = K2, K3 2^(p-n) (= 2^n k^2, 2^(n-u) k^3) and L = d lambda 2^(m-n), so that
//   x1' = K1, x2' = V2 and K' = E per unit of L.
// The Kerr-Schild connection (metric.c:538-638) in these units has no factor
// larger than 8/th' <= 13 (the axis term of E2 at hslope 1.8): with w = 1/r, sigma = Sigma w^2, delta = Delta w^2,
// rho = 1 + a^2 w^2, s = sin theta, c = cos theta, th' = d theta/d x2,
//   beta = (2 - sigma)/sigma^3 (Christoffel's B r^4), gamma = 1/sigma - a^2 s^2 beta w^3 (C r),
//   P = a s^2 k^3, t = a^2 s c th' w^2/sigma, kap2 = th' V2, kap3 = s V3 2^u,
//   mu = kap2^2/sigma + gamma kap3^2, R1 = r k^1 = r~ K1,
//   X0 = K0 (K0 - 2P), Y = K1 (K0 - P), H = (K0 + R1)^2,
//   E0 = -2 beta w (w w~ X0 + (sigma + 2w) Y + (sigma + w) R1 K1)
//        + 4 t w V2 (K0 + R1 - P)/sigma + 2 mu 2^-n
//   E1 = -beta w (w~^2 delta X0 + 2 w~ (delta - sigma) Y - (2 sigma - delta) K1^2) - K1^2
//        - 2 w~ K1 P/sigma + 2 t K1 V2 + delta mu
//   E2 = 2 z a^2 w^2 w~^3 2^-p H - 2 K1 K2/sigma - (th''/th' - t) K2 V2
//        - z K3 2^(2u) (2 a w F1 2^-u - F2 V3),  z = s c/(sigma^3 th'),
//        F1 = (sigma^2 + 2 w rho) K1 + 2 rho w w~ K0, F2 = delta sigma^2 + 2 w rho^2
//   E3 = -a beta w w~^3 2^-(p+u) (H - 2 K0 P) - gamma K3 (2 K1 - w~ P) + a w kap2 th' K2/sigma 2^-u
//        - 4 t w K2 V3/sigma - 2 cot th' (K2 V3 - a w K2 (2 w w~ K0 + (sigma + 2w) K1)/sigma^2 2^-u)
// Close to the axis sin theta = s~ 2^-ks is small, K3 and V3 2^u grow as its
// reciprocal and L shrinks with it: the last terms of E2 and E3 are formed
// without the factors 2^ks and applied with L 2^ks; where that passes 1 (steps
// along the axis with little angular momentum) the products are shifted after.
//
// A quantity "in Qf" is the integer value times 2^-f.  The ranges are those of
// rays with n in [0, 13], p - n <= 3, x2 in [2^-13, 1 - 2^-13] and a step that
// moves ln r by a tenth at most; others step in FP64 (fx_step's slow).
//
// Plain C++ apart from the intrinsics chosen below, so that the CPU tests
// compile it.
#pragma once

#ifdef __CUDACC__
#define FX_HD __device__ __forceinline__
#define FX_MEMBER __device__ __forceinline__
#define FX_TABLE(name, n) __device__ const longlong2 name[n]
#else
#include <cstdint>
struct longlong2 {
    long long x, y;
};
#define FX_HD static inline
#define FX_MEMBER inline
#define FX_TABLE(name, n) static const longlong2 name[n]
#endif

// FX_KEPT(ok): ok holds where an operation keeps every bit of its value;
// FX_TRACK(code) is what it takes to know.  The CPU range check
// (tests/fixed_kept.h) defines them; nothing is tested here.
#ifndef FX_KEPT
#define FX_KEPT(ok)
#define FX_TRACK(code)
#endif

namespace raptor {

#include "fixed_tables.inc"

using fx = long long;
using ufx = unsigned long long;

// Per-image constants (raptor_gpu.cu fills them in FP64)
struct FxGeo {
    fx a, a2;    // spin and its square, Q62
    fx tc;       // (1 - h) / (4 pi): theta in turns = x2/2 + tc sin(2 pi x2), Q63
    fx ph;       // pi (1 - h), Q60
    fx th2;      // -2 pi^2 (1 - h), Q58
    fx eps;      // step-size parameter, Q64
    fx startx1, stopx1, ln_inner, ln_outer;  // Q59
    fx startx2, stopx2;                      // Q62
    int ok;      // the image is one whose ranges the fixed-point step covers
};

#ifdef __CUDACC__
static __constant__ int kFxOne = 1;  // see fx_add32
#endif
#ifdef __CUDA_ARCH__
FX_HD int fx_clz(ufx x) { return __clzll((long long)x); }
FX_HD float fx_rcp_seed(int x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((float)x));
    return y;
}
FX_HD longlong2 fx_load(const longlong2* t) { return __ldg(t); }
// a b + c with 32-bit factors.  Written out because the compiler, where it
// shares a widened factor between basic blocks, otherwise forms whole 64-bit
// products (twice the instructions of the loop).
FX_HD fx fx_wide(int a, int b) {
    fx r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
FX_HD fx fx_wide(int a, int b, fx c) {
    fx r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
FX_HD ufx fx_wideu(unsigned a, unsigned b) {
    ufx r;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
FX_HD ufx fx_wideu(unsigned a, unsigned b, ufx c) {
    ufx r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
FX_HD unsigned fx_funnel(unsigned lo, unsigned hi, int k) { return __funnelshift_l(lo, hi, k); }
// c + h as one multiply-add by a 1 the compiler cannot see: the sign
// extension and the 64-bit sum cost the other integer pipe three instructions
FX_HD fx fx_add32(int c, fx h) { return fx_wide(c, kFxOne, h); }
#else
FX_HD int fx_clz(ufx x) { return x ? __builtin_clzll(x) : 64; }
FX_HD float fx_rcp_seed(int x) { return 1.0f / (float)x; }
FX_HD longlong2 fx_load(const longlong2* t) { return *t; }
FX_HD fx fx_wide(int a, int b) { return (fx)a * b; }
FX_HD fx fx_wide(int a, int b, fx c) { return (fx)a * b + c; }
FX_HD ufx fx_wideu(unsigned a, unsigned b) { return (ufx)a * b; }
FX_HD ufx fx_wideu(unsigned a, unsigned b, ufx c) { return (ufx)a * b + c; }
FX_HD unsigned fx_funnel(unsigned lo, unsigned hi, int k) { return (unsigned)((((ufx)hi << 32 | lo) << k) >> 32); }
FX_HD fx fx_add32(int c, fx h) { return h + c; }
#endif

FX_HD fx fx_one(int q) { return 1ll << q; }
FX_HD unsigned fx_u0(fx a) { return (unsigned)a; }
FX_HD unsigned fx_u1(fx a) { return (unsigned)((ufx)a >> 32); }
FX_HD fx fx_pair(unsigned lo, unsigned hi) { return (fx)((ufx)hi << 32 | lo); }

// A 64-bit value as high and low 32-bit halves, both signed: a = h 2^32 + l.
FX_HD int fx_hi(fx a) { return (int)(a >> 32) + (int)((unsigned)a >> 31); }
FX_HD int fx_lo(fx a) { return (int)(unsigned)a; }

// Sums of products.  h 2^64 + c 2^32, the products of the low halves left
// out: within 1/4 of 2^64 per product, which is 2^-60 for factors in Q62.
struct FxAcc {
    fx h, c;
    FX_TRACK(double most;)  // of |c|, whatever the low halves
};
FX_HD FxAcc fx_mul(fx a, fx b) {
    const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
    FxAcc r;
    r.c = fx_wide(al, bh, fx_wide(ah, bl));
    r.h = fx_wide(ah, bh);
    FX_TRACK(r.most = fx_most(ah, bh);)
    return r;
}
FX_HD FxAcc fx_mac(FxAcc r, fx a, fx b) {
    const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
    r.c = fx_wide(al, bh, fx_wide(ah, bl, r.c));
    r.h = fx_wide(ah, bh, r.h);
    FX_TRACK(r.most += fx_most(ah, bh);)
    FX_KEPT(r.most < 0x1p63);
    return r;
}
// The same sum with c's upper half moved into h.  A product adds as much as
// half of |a| + |b| to |c|: sums whose factors' magnitudes come to 2^64 or
// more take this on the way.
FX_HD FxAcc fx_carry(FxAcc r) {
    r.h = fx_add32((int)fx_u1(r.c), r.h);
    r.c = (fx)fx_u0(r.c);
    FX_TRACK(r.most = 0x1p32;)
    return r;
}
FX_HD bool fx_fits(fx a, int s) { return s < 64 && (fx)((ufx)a << s) >> s == a; }
// Value of the sum times 2^(K - 64), 1 <= K < 32.  (K = 0, which would leave
// the low half of c unused, is avoided throughout: the compiler then takes
// the multiply-add's high-half form, at less than half the rate.)
FX_HD fx fx_sum(FxAcc r, int K) {
    const fx h = fx_add32((int)fx_u1(r.c), r.h);
    FX_KEPT(fx_fits(h, K));
    return fx_pair(fx_funnel(fx_u0(r.c), fx_u0(h), K), fx_funnel(fx_u0(h), fx_u1(h), K));
}
template <int K>
FX_HD fx fx_sum(FxAcc r) {
    return fx_sum(r, K);
}
// a b 2^(K - 64): factors in Qx and Qy give Q(x + y - 64 + K)
template <int K>
FX_HD fx mulk(fx a, fx b) {
    return fx_sum<K>(fx_mul(a, b));
}
// a^2 2^(K - 64)
template <int K>
FX_HD fx sqrk(fx a) {
    const int ah = fx_hi(a), al = fx_lo(a);
    const fx c = fx_wide(ah, al);
    const fx h = fx_add32((int)fx_funnel(fx_u0(c), fx_u1(c), 1), fx_wide(ah, ah));
    FX_KEPT(fx_fits(h, K));
    return fx_pair(fx_funnel(fx_u0(c) << 1, fx_u0(h), K), fx_funnel(fx_u0(h), fx_u1(h), K));
}
FX_HD fx fx_shl(fx a, int s) {
    FX_KEPT(fx_fits(a, s));
    return (fx)((ufx)a << s);
}
// a 2^s for either sign of s, |s| < 64
FX_HD fx fx_scale(fx a, int s) { return s >= 0 ? fx_shl(a, s) : a >> -s; }
FX_HD fx fx_abs(fx a) { return a < 0 ? -a : a; }
FX_HD fx fx_max(fx a, fx b) { return a > b ? a : b; }
FX_HD fx fx_min(fx a, fx b) { return a < b ? a : b; }

// v 2^e as a double, rounded to nearest, on the integer pipes (the hardware
// conversion of a 64-bit integer issues to the FP64 pipe); v 2^e in the
// normal range or 0.
FX_HD double fx_double(fx v, int e) {
    const ufx u = (ufx)fx_abs(v);
    const int lz = fx_clz(u);
    const ufx m = u << (lz & 63);
    const ufx b = (m >> 11) + ((m >> 10) & 1ull) + ((ufx)(1023 + 63 - 1 - lz + e) << 52);
    const ufx r = u ? (b | ((ufx)v & 0x8000000000000000ull)) : 0ull;
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)r);
#else
    double d;
    __builtin_memcpy(&d, &r, 8);
    return d;
#endif
}

// 1/q in Q61 for q in [1/2, 1) in Q62: the FP32 approximation y0 (22 bits),
// then y0 (1 + e + e^2) with e = 1 - q y0, whose remainder e^3 is below 2^-64.
FX_HD fx fx_recip(fx q) {
    const int qh = (int)(q >> 32);
    const unsigned ql = (unsigned)q;
    const int y0 = (int)(fx_rcp_seed(qh) * 576460752303423488.0f);  // 2^59 / qh: 1/q in Q29
    const ufx p = fx_wideu((unsigned)qh, (unsigned)y0, fx_wideu(ql, (unsigned)y0) >> 32);  // Q59
    const fx e = (fx)(fx_one(59) - (fx)p);
    const fx es = fx_shl(e, 21);  // Q80
    const int eh = (int)(es >> 32);
    const fx co = es + (fx_wide(eh, eh) >> 16);
    const fx t = fx_wide((int)(co >> 32), y0, (fx)(fx_wideu((unsigned)co, (unsigned)y0) >> 32));  // Q77
    return fx_shl((fx)y0, 32) + (t >> 16);
}

// The odd and even parts of e^a (SIGN = 1) or e^(i a) (SIGN = -1) for a in
// Q70, |a| <= 2^-8.3: a (1 +- a^2/6 + a^4/120) and a^2/2 +- a^4/24 in Q63,
// the even part less 1 and of the sign of a^2 for both.  The corrections
// need no more than 32 bits of a^2; with that and the terms left out the
// error is below 2^-57.
template <int SIGN>
FX_HD void fx_series(fx a, fx& odd, fx& even) {
    const int ah = fx_hi(a), al = fx_lo(a);
    const fx c = fx_wide(ah, al);
    const fx z = fx_add32((int)fx_funnel(fx_u0(c), fx_u1(c), 1), fx_wide(ah, ah));  // a^2, Q76
    const int zs = (int)fx_funnel(fx_u0(z), fx_u1(z), 3);                            // Q47
    const fx y = fx_wide(zs, zs);                                                    // Q94
    const fx y24 = fx_wide((int)fx_funnel(fx_u0(y), fx_u1(y), 2), 1431655765);            // a^4/24: Q64 x Q35
    const int v = 1431655765 + SIGN * ((int)fx_u1(fx_wide(zs, 1145324612)) >> 19);             // 1/6 +- a^2/120, Q33
    const fx p = fx_wide(zs, v);                                                     // Q80
    const fx ap = fx_wide(ah, (int)fx_funnel(fx_u0(p), fx_u1(p), 2));                // a^3/6..: Q38 x Q50
    odd = (a >> 7) + SIGN * (ap >> 25);
    even = (z >> 13 >> 1) + SIGN * (y24 >> 36);
}

// sin and cos of u turns, u in Q62 in [0, 1): table entry n/1024 and the
// angle-addition formulas.
FX_HD void fx_sincos(fx u, fx& s, fx& c) {
    const int j = (int)(fx_u1(u) + (1u << 19)) >> 20;
    const fx rem = fx_pair(fx_u0(u), fx_u1(u) - ((unsigned)j << 20));
    const fx a = mulk<1>(fx_shl(rem, 11), 7244019458077122842ll);  // Q73 -> Q70
    fx odd, even;
    fx_series<-1>(a, odd, even);
    const longlong2 t = fx_load(&kFxSinCos[j & 1023]);
    const fx cm = -even;
    s = t.x + fx_sum<1>(fx_mac(fx_mul(t.x, cm), t.y, odd));
    c = t.y + fx_sum<1>(fx_mac(fx_mul(t.y, cm), -t.x, odd));
}

// log2 r in Q57
FX_HD fx fx_log2r(fx x1) { return mulk<1>(x1, 3326628274461080623ll); }

// r~ = 2^f (Q61) and 1/r~ (Q62), f in Q57 in (-1/2, 3/2).
FX_HD void fx_exp2(fx f, fx& r, fx& w) {
    const int j = (int)(fx_u1(f) + (1u << 17)) >> 18;
    const fx rem = fx_pair(fx_u0(f), fx_u1(f) - ((unsigned)j << 18));
    const fx a = mulk<1>(fx_shl(rem, 13), 6393154322601327830ll);  // Q70
    fx odd, even;
    fx_series<1>(a, odd, even);
    const longlong2 t = fx_load(&kFxExp2[(j + 64) & 255]);
    r = t.x + mulk<1>(t.x, even + odd);
    w = t.y + mulk<1>(t.y, even - odd);
}

struct FxPoint {
    fx r, w;        // r~ Q61, w~ Q62
    fx s, c;        // Q62
    fx s2x;         // sin(2 pi x2), Q62
    fx thp, ithp;   // th' Q60, 1/th' Q61
    fx isn;         // 1/sin theta = isn 2^ks, isn in Q61
    int ks;
};

// f = log2 r - n in Q57.  Both sincos take one copy of the code: the stage's
// loop has to stay in the instruction caches.
FX_HD void fx_point(const FxGeo& g, fx f, fx x2, FxPoint& p) {
    fx_exp2(f, p.r, p.w);
    fx u = x2, sv, cv;
#ifdef __CUDACC__
#pragma unroll 1
#endif
    for (int k = 0;; ++k) {
        fx_sincos(u, sv, cv);
        if (k == 1) break;
        p.s2x = sv;
        p.thp = 3622009729038561421ll + mulk<2>(g.ph, cv);
        u = (x2 >> 1) + mulk<1>(g.tc, sv);
    }
    p.s = sv;
    p.c = cv;
    const fx th = p.thp >> 1;
    const int kt = fx_clz((ufx)th) - 2;
    p.ithp = (fx)((ufx)fx_recip(fx_shl(th, kt)) << 1 >> (4 - kt));
    const fx sn = p.s - (p.s >> 62);
    p.ks = fx_clz((ufx)sn) - 2;
    p.isn = fx_recip(fx_shl(sn, p.ks));
}

struct FxState {
    fx x1, x2;          // Q59, Q62
    fx k0, k1, k2, k3;  // Q61
    int n, m, p, u;
    int raw;  // the words are the doubles x1, x2, k^mu
};

// The metric functions that the sample shares with the geodesic: 1/sigma in Q62.
FX_HD fx fx_isigma(const FxGeo& g, const FxPoint& p, int n, fx& a2w2, fx& s2, fx& sg) {
    const fx w = p.w >> n;
    a2w2 = mulk<2>(g.a2, sqrk<2>(w));
    s2 = sqrk<2>(p.s);
    sg = fx_one(61) + mulk<1>(a2w2, fx_one(62) - s2);  // Q61, the integer of sigma/2 in Q62
    return fx_recip(sg);                                // 2/sigma in Q61, the integer of 1/sigma in Q62
}

// The terms of a stage's right-hand side that a tangent of it reads.
struct FxTerms {
    fx wt2, s2, sg, isg, rho, dl, isg2, isg3, beta, gam, sc, thi;
    fx R1, S, H, X0, Y, RK, s0, s1;
    fx sg2, F1, F2, z, g2, G, F3;
    fx E0, E1, E2a, E2b, E3a, E3b;
};

// K' = E: E0, E1 in Q60, E2 = E2a + E2b 2^(2u-ks) and E3 = E3a + 2 E3b 2^ks
// with E2a, E2b, E3a in Q57 and E3b in Q58.  v2, v3 in Q58.
FX_HD void fx_rhs(const FxGeo& g, const FxPoint& q, fx k0, fx k1, fx k2, fx k3, int n, int p, int u, fx v2, fx v3,
                  FxTerms& o) {
    fx a2w2, s2, sg;  // Q62, Q62, Q61
    const fx isg = fx_isigma(g, q, n, a2w2, s2, sg);
    const fx w = q.w >> n;                         // Q62
    const fx ww = mulk<2>(w, q.w);                 // w w~, Q62
    const fx wt2 = sqrk<2>(q.w);                   // w~^2, Q62
    const fx wt3 = mulk<1>(wt2, q.w) >> p;         // w~^3 2^-p, Q61
    const fx rho = fx_one(61) + (a2w2 >> 1);       // Q61
    const fx dl = rho - w;                         // delta, Q61 (2w in Q61 is w's integer)
    const fx isg2 = sqrk<2>(isg);                  // Q62
    const fx isg3 = mulk<2>(isg2, isg);            // Q62
    const fx beta = mulk<3>(fx_one(62) - sg, isg3);  // (2 - sigma) Q61: Q62
    const fx nw = -w;                              // (negative factors, so that the sums below need no negation)
    const fx nbw = mulk<2>(beta, nw);              // -beta w, Q62
    const fx gam = isg + mulk<2>(mulk<2>(a2w2, s2), nbw);  // Q62
    const fx awt = mulk<2>(g.a, q.w), aw = awt >> n;  // a w~, a w, Q62
    const fx sc = mulk<2>(q.s, q.c);               // Q62
    const fx thi = mulk<2>(q.thp, isg);            // th'/sigma, Q60
    const fx t = mulk<2>(mulk<2>(a2w2, sc), thi);  // Q60
    const fx ntw = mulk<4>(mulk<2>(t, isg), nw);   // -t w/sigma, Q62

    const fx as2 = mulk<2>(g.a, s2);               // Q62
    const fx P = fx_shl(mulk<5>(as2, v3) >> n, u);  // Q61
    const fx R1 = mulk<2>(q.r, k1);                // Q60
    const fx S = (k0 >> 1) + R1;                   // K0 + R1, Q60
    const fx H = sqrk<3>(S);                       // Q59
    const fx X0 = mulk<2>(k0, (k0 >> 1) - P);      // Q61 x Q60: Q59 (2P in Q60 is P's integer)
    const fx Y = mulk<2>(k1, k0 - P);              // Q60
    const fx Q = sqrk<2>(k1);                      // Q60
    const fx kap2 = mulk<6>(q.thp, v2);            // Q60
    const fx M2 = mulk<3>(kap2, mulk<6>(thi, v2));  // kap2^2/sigma, Q59
    const fx kap3 = fx_shl(mulk<4>(q.s, v3), u);   // Q60
    const fx mu = M2 + mulk<2>(gam, sqrk<3>(kap3));  // Q59

    const fx sg2w = sg + w;                        // sigma + 2w, Q61
    const fx nigk1 = -mulk<1>(isg, k1);            // Q60
    const fx wP = mulk<2>(q.w, P);                 // Q61
    {
        FxAcc s = fx_mul(ww, X0);
        s = fx_mac(s, sg2w, Y);
        o.RK = mulk<3>(R1, k1);                    // Q60
        s = fx_mac(fx_carry(s), sg + (w >> 1), o.RK);  // Q61 x Q60
        o.s0 = fx_sum<1>(s);                       // Q58
        FxAcc e = fx_mul(mulk<5>(ntw, v2), (P >> 1) - S);  // 2 () in Q60 x Q60
        e = fx_mac(e, nbw, o.s0);                          // Q62 x Q58; both doubled below
        o.E0 = fx_sum<5>(e) + (fx_shl(mu, 2) >> n);
    }
    {
        FxAcc s = fx_mul(wt2, mulk<3>(dl, X0));            // Q62 x Q59
        s = fx_mac(s, mulk<3>(q.w, dl - sg), Y);           // 2 w~ (delta - sigma) in Q61 x Q60
        s = fx_mac(fx_carry(s), dl - fx_shl(sg, 1), Q);    // -(2 sigma - delta) Q61 x Q60
        o.s1 = fx_sum<1>(s);                               // Q58
        FxAcc e = fx_mul(nbw, o.s1);                       // Q62 x Q58
        e = fx_mac(e, nigk1, wP);                          // Q60 x 2 w~ P in Q60
        e = fx_mac(e, t, mulk<6>(k1, v2));                 // Q60 x 2 K1 V2 in Q60
        e = fx_mac(e, dl, mu);                             // Q61 x Q59
        o.E1 = fx_sum<4>(e) - Q;
    }
    const fx sg2 = sqrk<2>(sg);                    // Q60
    const fx wr2 = mulk<2>(w, rho);                // 2 w rho in Q60
    const fx kv23 = mulk<5>(k2, v3);               // Q60
    {
        const fx rww = mulk<2>(rho, ww);                                               // Q61
        const fx F1 = fx_sum<1>(fx_mac(fx_mul(sg2 + wr2, k1), rww, k0));               // Q58
        const fx F2 = fx_sum<3>(fx_mac(fx_mul(dl, sg2), wr2, rho));                    // Q60
        const fx z = mulk<3>(mulk<2>(sc, isg3), q.ithp);                               // Q62
        const fx A = mulk<3>(a2w2, wt3);                            // 2 a^2 w^2 w~^3 2^-p in Q61
        FxAcc e = fx_mul(A, mulk<1>(z, H));                         // x Q58
        const fx g2 = mulk<3>(g.th2, mulk<3>(q.s2x, q.ithp));       // th''/th', Q59
        e = fx_mac(e, (t >> 1) - g2, mulk<5>(k2, v2));              // Q59 x Q60
        e = fx_mac(e, nigk1 >> 1, k2);                              // 2 () in Q58 x Q61
        o.E2a = fx_sum<2>(e);
        o.F1 = F1; o.F2 = F2; o.z = z; o.g2 = g2;
        const fx G = mulk<3>(F2, v3) - (mulk<2>(aw, F1) >> u);      // Q57 (2 a w F1 in Q57)
        o.G = G;
        o.E2b = mulk<2>(fx_shl(z, q.ks), mulk<3>(k3, G));             // Q62 x Q57
    }
    {
        const fx B = mulk<2>(mulk<2>(g.a, nbw), wt3) >> u;                      // Q61
        FxAcc e = fx_mul(B, H - mulk<2>(k0, P));                              // x (H - 2 K0 P) Q59
        e = fx_mac(e, mulk<1>(gam, k3), (wP >> 1) - k1);                        // Q60 x (w~ P - 2 K1) Q60
        e = fx_mac(e, ntw, kv23);                                               // 4 () in Q60 x Q60
        o.E3a = fx_sum<1>(e) + (mulk<1>(awt >> p, M2) >> (u + 1));              // a w kap2 th' K2/sigma: Q62 x Q59
        const fx F3 = fx_sum<2>(fx_mac(fx_mul(ww, k0), sg2w, k1));              // Q60
        const fx D = (mulk<2>(mulk<2>(aw, isg2), mulk<3>(k2, F3)) >> u) - kv23;  // Q60
        o.E3b = mulk<3>(mulk<2>(mulk<2>(q.c, q.isn), q.thp), D);                // -cot th' 2^-ks () Q59 x Q60
        o.F3 = F3;
    }
    // (terms that nothing reads cost nothing: the function is inlined)
    o.wt2 = wt2; o.s2 = s2; o.sg = sg; o.isg = isg; o.rho = rho; o.dl = dl; o.isg2 = isg2; o.isg3 = isg3;
    o.beta = beta; o.gam = gam; o.sc = sc; o.thi = thi; o.R1 = R1; o.S = S; o.H = H; o.X0 = X0; o.Y = Y;
    o.sg2 = sg2;
}

FX_HD fx fx_vshift(fx k, int e) { return k >> (3 - e); }  // K 2^e in Q58, e <= 3

// The exponents of a state whose log2 r (Q57) is lr: n from r, then m and p
// so that the wave vector fills its range.
FX_HD void fx_normalise(FxState& s, fx lr) {
    const int dn = (int)(lr >> 57) - s.n;
    if (dn != 0) {
        s.k1 = fx_scale(s.k1, dn);
        s.p += 2 * dn;
        s.n += dn;
    }
    const int sm = fx_clz((ufx)(fx_abs(s.k0) | fx_abs(s.k1))) - 3;
    if (sm != 0) {
        s.k0 = fx_scale(s.k0, sm);
        s.k1 = fx_scale(s.k1, sm);
        s.m -= sm;
        s.p += sm;
    }
    // the exponents that K2 and K3 would take by themselves
    const int q2 = s.p + 3 - fx_clz((ufx)fx_abs(s.k2)), q3 = s.p + s.u + 3 - fx_clz((ufx)fx_abs(s.k3));
    const int cap = s.n + 3;
    int p = q3 < cap ? q3 : cap;
    p = p > q2 ? p : q2;
    p = p > 0 ? p : 0;
    const int u = q3 > p ? q3 - p : 0;
    if (p != s.p || u != s.u) {
        s.k2 = fx_scale(s.k2, s.p - p);
        s.k3 = fx_scale(s.k3, s.p + s.u - p - u);
        s.p = p;
        s.u = u;
    }
}

// Bits by which L 2^ks is shortened to stay below 1: rays along the axis with
// little angular momentum take steps that do not shrink with sin theta.
FX_HD int fx_excess(int ks, fx L) {
    const int e = ks + 2 - fx_clz((ufx)L);
    return e > 0 ? e : 0;
}

// |d lambda| 2^(m-n) in Q62: L = eps m2 / (m2 (|K1| + |V3| 2^u) + |V2|), the
// reciprocals of integrator.c:109-122 folded (its guards against zero rates
// and steps do not act in this range).  False outside the ranges that the
// step's arithmetic covers.
FX_HD bool fx_step_size(const FxGeo& g, const FxState& s, int ks, fx& L) {
    const int e = s.p - s.n;
    const fx m2 = fx_min(s.x2, fx_one(62) - s.x2);
    if (s.raw || s.n < 0 || s.n > 13 || e > 3 || s.u > 11 || (s.u > 0 && s.u >= ks) || m2 < fx_one(49)) return false;
    if (((m2 >> 1) >> (61 - s.u)) != 0) return false;
    const fx m2u = fx_shl(m2, s.u);
    const fx v2 = fx_abs(fx_vshift(s.k2, e)), v3 = fx_abs(fx_vshift(s.k3, e));
    const fx d = fx_sum<3>(fx_mac(fx_mul(m2, fx_abs(s.k1) >> 3), m2u, v3)) + (v2 << 1);  // Q59
    const int kd = fx_clz((ufx)d) - 2;
    if (kd < 1 || kd > 20) return false;
    const fx y = mulk<1>(mulk<3>(g.eps, m2), fx_recip(fx_shl(d, kd)));  // Q65 x Q61: Q63; L = y 2^(kd-3)
    if (kd > 2 && (y >> (66 - kd)) != 0) return false;                  // L >= 1 (below kd = 3 it cannot be)
    L = kd >= 4 ? fx_shl(y, kd - 4) : y >> (4 - kd);
    return s.u == 0 || 2 * (ks - s.u) >= fx_excess(ks, L) + 2;
}

// One step of integrate_geodesic (integrator.c:109-146, 13-70) backward in
// lambda: the step size, then RK4 or RK2; dl is |d lambda|.  pt is the point
// at the ray's position on entry and on exit (not formed for a raw state).
// slow(s) takes the steps that this arithmetic does not cover, leaves s
// fixed-point again or raw, and returns |d lambda|.  tan follows the steps
// that it does cover (the adjoint's tangents; FxNoTangent): begin with the
// step size, stage with each stage's state, commit when the step holds.
struct FxNoTangent {
    FX_MEMBER void begin(const FxState&, const FxPoint&, fx) {}
    FX_MEMBER void stage(int, int, const FxPoint&, const FxTerms&, fx, fx, fx, fx) {}
    FX_MEMBER void commit() {}
};
template <class Slow, class Tangent>
FX_HD void fx_step(const FxGeo& g, FxState& s, FxPoint& pt, bool rk2, double& dl, Slow slow, Tangent& tan) {
    fx L = 0;
    bool go = fx_step_size(g, s, pt.ks, L);
    if (go) tan.begin(s, pt, L);
    const int e = s.p - s.n;
    const fx full = -L, half = full >> 1;
    fx x1 = s.x1, x2 = s.x2, k0 = s.k0, k1 = s.k1, k2 = s.k2, k3 = s.k3;
    // What symmetry keeps at exactly 0 has no products to round: k^3 of a ray in
    // a plane through the axis of a hole without spin (which ends on the axis,
    // and would pass it at a rounding's distance), k^2 in the equatorial plane.
    const fx spins = (g.a | s.k3) != 0 ? 1 : 0, tilts = (s.k2 | (s.x2 - fx_one(61))) != 0 ? 1 : 0;
    // RK4's sums start at the mean of what the floors of their products lose
    // (p2 has two of them)
    fx a1 = 0, a2 = 4 * tilts, b0 = 4, b1 = 4, b2 = 6 * tilts, b3 = 4 * spins;
    const int end = rk2 ? 2 : 4;
#ifdef __CUDACC__
#pragma unroll 1
#endif
    for (int q = 0;; ++q) {
        if (q == end) {
            if (!rk2) {
                const fx third = 3074457345618258603ll;
                x1 = s.x1 + ((mulk<1>(a1, third) + 2) >> 2);
                x2 = s.x2 + mulk<1>(a2, third);
                k0 = s.k0 + mulk<1>(b0, third);
                k1 = s.k1 + mulk<1>(b1, third);
                k2 = s.k2 + mulk<1>(b2, third);
                k3 = s.k3 + mulk<1>(b3, third);
            } else {
                // RK2's offsets lose half a unit each, which N steps would add
                // up to N/2 units: a unit is given back at every other step
                const fx unit = (s.k0 ^ s.k1) & 1;
                x1 += unit;
                x2 += unit & tilts;
                k0 += unit;
                k1 += unit;
                k2 += tilts;  // two floors
                k3 += unit & spins;
            }
            // a wave vector that doubled within the step may have left its range inside it
            go = go && ((ufx)(fx_abs(k0) | fx_abs(k1) | fx_abs(k2) | fx_abs(k3)) >> 62) == 0;
            if (go) {
                dl = fx_double(L, s.n - s.m - 62);
                s.x1 = x1;
                s.x2 = x2;
                s.k0 = k0;
                s.k1 = k1;
                s.k2 = k2;
                s.k3 = k3;
                tan.commit();
            } else {
                dl = slow(s);
                if (s.raw) break;
                x1 = s.x1;
                x2 = s.x2;
            }
        }
        if (q > 0 && (go || q == end)) {
            const fx lr = fx_log2r(x1);
            if (q == end) fx_normalise(s, lr);
            fx_point(g, lr - fx_shl((fx)s.n, 57), x2, pt);
        }
        if (q == end) break;
        if (go) {
            const fx v2 = fx_vshift(k2, e), v3 = fx_vshift(k3, e);
            FxTerms o;
            fx_rhs(g, pt, k0, k1, k2, k3, s.n, s.p, s.u, v2, v3, o);
            tan.stage(q, end, pt, o, k0, k1, k2, k3);
            // offsets h f1, h f2, d f3, h f4 (h = d/2): y + d (f1 + 2 f2 + 2 f3 + f4)/6
            // is y + (o1 + 2 o2 + o3 + o4)/3; RK2: h f1, then y + d f2
            const fx h = q == end - 2 + (rk2 ? 1 : 0) ? full : half;
            const fx o1 = mulk<2>(h, k1), o2 = mulk<6>(h, v2);  // Q61, Q62
            const int ex = fx_excess(pt.ks, L);
            const fx hk = fx_shl(h, pt.ks - ex);
            const fx p0 = mulk<3>(h, o.E0), p1 = mulk<3>(h, o.E1);  // Q61
            // hk E2b reaches 8/th' along the axis (13 at hslope 1.8): two bits
            // of the shift are left out of the product, where there are two
            const int sh = 2 * (pt.ks - s.u) - ex, up = sh >= 2 ? 2 : 0;
            const fx p2 = mulk<6>(h, o.E2a) + (fx_sum(fx_mul(hk, o.E2b), 6 - up) >> (sh - up));
            const fx p3 = fx_sum<6>(fx_mac(fx_mul(h, o.E3a), hk, fx_shl(o.E3b, ex)));  // 2 E3b in Q57
            const int two = q == 1 ? 1 : 0;
            a1 += fx_shl(o1, two);
            a2 += fx_shl(o2, two);
            b0 += fx_shl(p0, two);
            b1 += fx_shl(p1, two);
            b2 += fx_shl(p2, two);
            b3 += fx_shl(p3, two);
            x1 = s.x1 + (o1 >> 2);
            x2 = s.x2 + o2;
            k0 = s.k0 + p0;
            k1 = s.k1 + p1;
            k2 = s.k2 + p2;
            k3 = s.k3 + p3;
        }
    }
}
}  // namespace raptor
