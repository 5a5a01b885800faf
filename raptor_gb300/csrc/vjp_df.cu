// The adjoint passes of the mixed-DF form and, for the images outside the
// fixed-point geodesic's ranges, of the mixed form (vjp_f32.cuh has their
// body): the geodesic through the same templated code as the forward kernels
// (step size, rolled RK4, point transcendentals, Christoffels):
//  - mixed-DF (vjp_kernel_df): DF values with FP32 inclination tangents
//    (Dual<1, DF, float>);
//  - mixed (vjp_kernel_mixed): FP64 values with FP32 inclination tangents
//    (Dual<1, double, float>): the tangent's arithmetic off the FP64 pipe.
#include "vjp_f32.cuh"

namespace raptor {
namespace {

// ------------------------------------------------------------ the two forms
// Both step the templated geodesic (step size, rolled RK4, point
// transcendentals, Christoffels) on a value with its inclination tangent;
// FormRk is their common part.
template <class S_>
struct RkState {
    S_ y[8];
    MksPointT<S_> p;
};
template <class F, class S_>
struct FormRk {
    using S = S_;
    using State = RkState<S>;
    using Step = S;
    __device__ __forceinline__ static void start(const DevImage& im, const D1 (&y0)[8], State& g) {
#pragma unroll
        for (int i = 0; i < 8; ++i) g.y[i] = F::from_camera(y0[i]);
        mks_point(g.y[1], g.y[2], F::geo(im), g.p);
    }
    __device__ __forceinline__ static void advance(const DevImage& im, State& g, Step& dl) {
        using G = typename std::remove_cv<typename std::remove_reference<decltype(F::geo(im))>::type>::type;
        dl = F::step(im, g.y);
        if (im.integrator == 2) rk2_step<S, G, false>(F::geo(im), g.y, g.p, dl);
        else rk4_step_rolled<S, G, false>(F::geo(im), g.y, g.p, dl);
    }
    __device__ __forceinline__ static bool alive(const DevImage& im, const State& g, int steps, int stop) {
        return F::alive_at(im, g.p, steps, stop);
    }
    __device__ __forceinline__ static auto theta_rate(const State& g) { return F::rate(g.y[6]); }
    __device__ __forceinline__ static bool escaped(const DevImage& im, const State& g) { return F::escaped_at(im, g.y); }
    __device__ __forceinline__ static bool in_grid(const DevImage& im, const State& g) { return F::in_grid_at(im, g.y); }
    __device__ __forceinline__ static bool finite(const State& g) { return F::finite_at(g.p, g.y); }
    template <bool K>
    __device__ __forceinline__ static bool sample(const DevImage& im, const State& g, const Step& dl,
                                                  SampleCommonF& out) {
        return F::template sample_at<K>(im, g.y, g.p, fabs(dl), out);
    }
};

// Mixed-DF: the geodesic of ray_kernel_df.
struct FormDF : FormRk<FormDF, DD1> {
    using S = DD1;
    using Th = float;  // d x2 / d lambda as the theta-turn test reads it
    static constexpr bool kMergeReplay = false;  // vjp_f32_body's record replay
    __device__ static const GeoDF& geo(const DevImage& im) { return im.geo_df; }
    __device__ static S from_camera(const D1& y) {
        S s(df_const(y.v));
        s.d[0] = (float)y.d[0];
        return s;
    }
    // stepsize (integrator.c:109-122) as step_size_df
    __device__ static S step(const DevImage& im, const S y[8]) {
        const DF t = df_const(1.e-40);
        const S m2 = fmin(y[2], 1.0 - y[2]);
        const S i13 = (fabs(y[5]) + t) + (fabs(y[7]) + t);
        const S i2 = fabs(y[6]) + t;
        return -fmax(m2 / ((m2 * i13 + i2) * im.inv_stepsize_df), 1e-12);
    }
    __device__ static bool alive_at(const DevImage& im, const MksPointT<S>& p, int steps, int stop) {
        const DF r = p.rp.v;
        return r < df_const(kCutoffOuter) && r > im.cutoff_inner_df && steps < (int)kMaxSteps && !stop;
    }
    __device__ static Th rate(const S& y6) { return y6.v.hi; }
    __device__ static bool turned(Th prev, Th now) {
        return (prev < 0.0f && now > 0.0f) || (prev > 0.0f && now < 0.0f);
    }
    __device__ static bool escaped_at(const DevImage& im, const S y[8]) {
        return y[1].v > im.stopx1_df && y[5].v.hi < 0.0f;
    }
    // a finite photon state at the ray's end, as finish_ray tests it
    __device__ static bool finite_at(const MksPointT<S>& p, const S y[8]) {
        return p.rp.v.hi == p.rp.v.hi && isfinite(y[5].v.hi);
    }
    __device__ static bool in_grid_at(const DevImage& im, const S y[8]) {
        return y[1].v < im.stopx1_df && y[1].v > im.startx1_df && y[2].v > im.startx2_df && y[2].v < im.stopx2_df;
    }
    // rt_sample_df's inputs: Xtoij (grmhd.c:46-71) from the DF position,
    // the offsets carrying the inclination tangent unless clamped
    template <bool K>
    __device__ static bool sample_at(const DevImage& im, const S y[8], const MksPointT<S>& p, const S& adl,
                                  SampleCommonF& out) {
        const MetricT<F1> g = metric_f1(p, im.geo_df);
        const DF t1 = (y[1].v - im.startx1_df) * im.idx1_df - 0.5;
        const DF t2 = (y[2].v - im.startx2_df) * im.idx2_df - 0.5;
        int i = df_trunc(t1), j = df_trunc(t2);
        F1 d1(0.0f), d2(0.0f);
        if (i < 0) i = 0;
        else if (i > im.n1 - 2) { i = im.n1 - 2; d1 = F1(1.0f); }
        else { d1 = F1(df_value(add_f(t1, (float)-i))); d1.d[0] = y[1].d[0] * im.idx1_df.hi; }
        if (j < 0) j = 0;
        else if (j > im.n2 - 2) { j = im.n2 - 2; d2 = F1(1.0f); }
        else { d2 = F1(df_value(add_f(t2, (float)-j))); d2.d[0] = y[2].d[0] * im.idx2_df.hi; }
        if (!chk(i >= 0 && i <= im.n1 - 2 && j >= 0 && j <= im.n2 - 2, im.check_word, kChkCell,
                 (long long)i * im.n2 + j))
            i = j = 0;
        const F1 k[4] = {to_f1(y[4]), to_f1(y[5]), to_f1(y[6]), to_f1(y[7])};
        return sample_common_f<K>(im, g, i * im.n2 + j, d1, d2, k, to_f1(adl), out);
    }
};

// Mixed: the FP64 geodesic of ray_kernel<NF, true>, with the inclination
// tangent in TD.
template <class TD>
struct FormMixed : FormRk<FormMixed<TD>, Dual<1, double, TD>> {
    using S = Dual<1, double, TD>;
    using Th = double;
    static constexpr bool kMergeReplay = true;  // vjp_f32_body's record replay
    __device__ static const Geo& geo(const DevImage& im) { return im.geo; }
    __device__ static S from_camera(const D1& y) {
        S s(y.v);
        s.d[0] = (TD)y.d[0];
        return s;
    }
    __device__ static S step(const DevImage& im, const S y[8]) { return step_size(im, y); }
    // the while-condition of integrator.c:228-229, as advance_ray
    __device__ static bool alive_at(const DevImage& im, const MksPointT<S>& p, int steps, int stop) {
        const double r = p.rp.v;
        return r < kCutoffOuter && r > im.cutoff_inner && (double)steps < kMaxSteps && !stop;
    }
    __device__ static Th rate(const S& y6) { return y6.v; }
    __device__ static bool turned(Th prev, Th now) { return prev * now < 0.0; }
    __device__ static bool escaped_at(const DevImage& im, const S y[8]) { return y[1].v > im.stopx1 && y[5].v < 0.0; }
    __device__ static bool in_grid_at(const DevImage& im, const S y[8]) {
        return y[1].v < im.stopx1 && y[1].v > im.startx1 && y[2].v > im.startx2 && y[2].v < im.stopx2;
    }
    __device__ static bool finite_at(const MksPointT<S>& p, const S y[8]) {
        return p.rp.v == p.rp.v && isfinite(y[5].v);
    }
    // rt_sample_fp32's inputs: the metric in FP32 from the FP64 point
    // rounded (with its tangent), Xtoij in FP64 (cell_coef), the wave vector
    // rounded to FP32
    template <bool K>
    __device__ static bool sample_at(const DevImage& im, const S y[8], const MksPointT<S>& p, const S& adl,
                                  SampleCommonF& out) {
        const MetricT<F1> g = metric_f1(p, im.geo_df);
        const CellCoef cc = cell_coef(im, y[1].v, y[2].v);
        const int i = cc.base / im.n2, j = cc.base - i * im.n2;
        F1 d1(f32_of(cc.d1)), d2(f32_of(cc.d2));
        const double t1 = (y[1].v - im.startx1) * im.idx1 - 0.5;
        const double t2 = (y[2].v - im.startx2) * im.idx2 - 0.5;
        if ((int)t1 == i) d1.d[0] = y[1].d[0] * im.idx1_df.hi;  // not clamped
        if ((int)t2 == j) d2.d[0] = y[2].d[0] * im.idx2_df.hi;
        const F1 k[4] = {to_f1(y[4]), to_f1(y[5]), to_f1(y[6]), to_f1(y[7])};
        return sample_common_f<K>(im, g, cc.base, d1, d2, k, to_f1(adl), out);
    }
};

#ifndef RAPTOR_VJP_DF_MIN_BLOCKS
#define RAPTOR_VJP_DF_MIN_BLOCKS 2
#endif
#ifndef RAPTOR_VJP_MIXED_MIN_BLOCKS
#define RAPTOR_VJP_MIXED_MIN_BLOCKS 2
#endif
// The mixed adjoint's inclination tangent: FP32 (1), which keeps its
// arithmetic off the FP64 pipe, or FP64 (0).
#ifndef RAPTOR_VJP_MIXED_TANGENT_FP32
#define RAPTOR_VJP_MIXED_TANGENT_FP32 1
#endif
using MixedTangent = std::conditional<RAPTOR_VJP_MIXED_TANGENT_FP32 != 0, float, double>::type;

template <int NF, bool K, bool TAPE>
__global__ void __launch_bounds__(kVjpBlock, RAPTOR_VJP_DF_MIN_BLOCKS)
    vjp_kernel_df(const DevImage* __restrict__ imp, CamT<D1> cam, const double* __restrict__ fwd,
                  const double* __restrict__ dLdO, unsigned long long* __restrict__ counters,
                  double* __restrict__ gscal, double* __restrict__ g_rho, double* __restrict__ g_u,
                  double* __restrict__ g_th, int refill_interval, RayRange rr, VjpTape tape) {
    vjp_f32_body<NF, FormDF, K, TAPE>(*imp, cam, fwd, dLdO, counters, gscal, g_rho, g_u, g_th, refill_interval, rr,
                                      tape);
}

template <int NF, bool K, bool TAPE>
__global__ void __launch_bounds__(kVjpBlock, RAPTOR_VJP_MIXED_MIN_BLOCKS)
    vjp_kernel_mixed(const DevImage* __restrict__ imp, CamT<D1> cam, const double* __restrict__ fwd,
                     const double* __restrict__ dLdO, unsigned long long* __restrict__ counters,
                     double* __restrict__ gscal, double* __restrict__ g_rho, double* __restrict__ g_u,
                     double* __restrict__ g_th, int refill_interval, RayRange rr, VjpTape tape) {
    vjp_f32_body<NF, FormMixed<MixedTangent>, K, TAPE>(*imp, cam, fwd, dLdO, counters, gscal, g_rho, g_u, g_th,
                                                       refill_interval, rr, tape);
}

template <int NF, bool K, bool TAPE>
void launch_vjp_df(int grid, cudaStream_t st, const DevImage* im, const CamT<D1>& cam, const double* fwd,
                   const double* dl, unsigned long long* ctr, double* gs, double* gr, double* gu, double* gt,
                   int refill, double*, RayRange rr, VjpTape tape) {
    vjp_kernel_df<NF, K, TAPE><<<grid, kVjpBlock, 0, st>>>(im, cam, fwd, dl, ctr, gs, gr, gu, gt, refill, rr, tape);
}

template <int NF, bool K, bool TAPE>
void launch_vjp_mixed(int grid, cudaStream_t st, const DevImage* im, const CamT<D1>& cam, const double* fwd,
                      const double* dl, unsigned long long* ctr, double* gs, double* gr, double* gu, double* gt,
                      int refill, double*, RayRange rr, VjpTape tape) {
    vjp_kernel_mixed<NF, K, TAPE><<<grid, kVjpBlock, 0, st>>>(im, cam, fwd, dl, ctr, gs, gr, gu, gt, refill, rr,
                                                              tape);
}

template <bool TAPE>
VjpLaunchFn pick_df(int nf, const void** fn, bool kappa) {
    if (kappa) {
        *fn = (const void*)vjp_kernel_df<kMaxFreqs, true, TAPE>;
        return launch_vjp_df<kMaxFreqs, true, TAPE>;
    }
    if (nf <= 1) {
        *fn = (const void*)vjp_kernel_df<1, false, TAPE>;
        return launch_vjp_df<1, false, TAPE>;
    }
    *fn = (const void*)vjp_kernel_df<kMaxFreqs, false, TAPE>;
    return launch_vjp_df<kMaxFreqs, false, TAPE>;
}

template <bool TAPE>
VjpLaunchFn pick_mixed(int nf, const void** fn, bool kappa) {
    if (kappa) {
        *fn = (const void*)vjp_kernel_mixed<kMaxFreqs, true, TAPE>;
        return launch_vjp_mixed<kMaxFreqs, true, TAPE>;
    }
    if (nf <= 1) {
        *fn = (const void*)vjp_kernel_mixed<1, false, TAPE>;
        return launch_vjp_mixed<1, false, TAPE>;
    }
    *fn = (const void*)vjp_kernel_mixed<kMaxFreqs, false, TAPE>;
    return launch_vjp_mixed<kMaxFreqs, false, TAPE>;
}

}  // namespace

// kappa: the kappa fits' instantiation (any frequency count); tape: the
// one-pass kernel
VjpLaunchFn pick_vjp_df(int nf, const void** fn, bool kappa, bool tape) {
    return tape ? pick_df<true>(nf, fn, kappa) : pick_df<false>(nf, fn, kappa);
}

VjpLaunchFn pick_vjp_mixed(int nf, const void** fn, bool kappa, bool tape) {
    return tape ? pick_mixed<true>(nf, fn, kappa) : pick_mixed<false>(nf, fn, kappa);
}

}  // namespace raptor
