// The render kernels of the FP64 and mixed forms with the geodesic in fixed
// point (ray_fixed.cuh): instantiations of ray_kernel.cuh's kernels.
#include <cuda_runtime.h>

#include "engine_internal.h"
#include "ray_fixed.cuh"

using namespace raptor;

namespace {

template <int NF, bool MIXED, int Blocks>
void launch_ray_fx(const LaunchShape& ls, cudaStream_t st, const DevImage* imgs, int n, long long b, long long e,
                   unsigned long long* ctr, double* out, TraceSpec tr) {
    ray_kernel<NF, MIXED, false, FxRay<NF, MIXED, Blocks>><<<ls.grid, ls.block, 0, st>>>(imgs, n, b, e, ctr, out,
                                                                                        ls.refill, tr);
}
template <int NF, int Blocks>
void launch_ray_pool_fx(const LaunchShape& ls, cudaStream_t st, const DevImage* imgs, int n, long long b, long long e,
                        unsigned long long* ctr, double* out, TraceSpec) {
    ray_kernel_pool<NF, FxRay<NF, false, Blocks>><<<ls.grid, ls.block, 0, st>>>(imgs, n, b, e, ctr, out, ls.refill);
}

template <int NF, bool MIXED, int Blocks>
RayLaunchFn in_place(const void** fn) {
    *fn = (const void*)ray_kernel<NF, MIXED, false, FxRay<NF, MIXED, Blocks>>;
    return launch_ray_fx<NF, MIXED, Blocks>;
}
template <int NF, int Blocks>
RayLaunchFn pooled(const void** fn) {
    *fn = (const void*)ray_kernel_pool<NF, FxRay<NF, false, Blocks>>;
    return launch_ray_pool_fx<NF, Blocks>;
}

template <int NF>
RayLaunchFn pick(bool mixed, const void** fn, bool pool, long long rays) {
    if (mixed) return rays < kFxFewRaysMixed ? in_place<NF, true, 2>(fn) : in_place<NF, true, 3>(fn);
    if (!pool) return in_place<NF, false, 3>(fn);
    if (rays < kFxFewRays) return pooled<NF, 2>(fn);
    return rays < kFxManyRays ? pooled<NF, 3>(fn) : pooled<NF, 4>(fn);
}

}  // namespace

RayLaunchFn pick_ray_kernel_fx(int nf, bool mixed, const void** fn, bool pool, long long rays) {
    if (nf <= 1) return pick<1>(mixed, fn, pool, rays);
    if (nf <= 2) return pick<2>(mixed, fn, pool, rays);
    if (nf <= 4) return pick<4>(mixed, fn, pool, rays);
    return pick<8>(mixed, fn, pool, rays);
}
