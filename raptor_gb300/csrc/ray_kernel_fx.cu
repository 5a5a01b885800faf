// The render kernels of the FP64 and mixed forms with the geodesic in fixed
// point (ray_fixed.cuh): instantiations of ray_kernel.cuh's kernels.
#include <cuda_runtime.h>

#include "engine_internal.h"
#include "ray_fixed.cuh"

using namespace raptor;

namespace {

template <int NF, bool MIXED>
void launch_ray_fx(const LaunchShape& ls, cudaStream_t st, const DevImage* imgs, int n, long long b, long long e,
                   unsigned long long* ctr, double* out, TraceSpec tr) {
    ray_kernel<NF, MIXED, false, FxRay<NF, MIXED, 3>><<<ls.grid, ls.block, 0, st>>>(imgs, n, b, e, ctr, out, ls.refill,
                                                                                   tr);
}
template <int NF, int Blocks>
void launch_ray_pool_fx(const LaunchShape& ls, cudaStream_t st, const DevImage* imgs, int n, long long b, long long e,
                        unsigned long long* ctr, double* out, TraceSpec) {
    ray_kernel_pool<NF, FxRay<NF, false, Blocks>><<<ls.grid, ls.block, 0, st>>>(imgs, n, b, e, ctr, out, ls.refill);
}

template <int NF>
RayLaunchFn pick(bool mixed, const void** fn, bool pool, bool many) {
    if (mixed) {
        *fn = (const void*)ray_kernel<NF, true, false, FxRay<NF, true, 3>>;
        return launch_ray_fx<NF, true>;
    }
    if (pool && many) {
        *fn = (const void*)ray_kernel_pool<NF, FxRay<NF, false, 4>>;
        return launch_ray_pool_fx<NF, 4>;
    }
    if (pool) {
        *fn = (const void*)ray_kernel_pool<NF, FxRay<NF, false, 3>>;
        return launch_ray_pool_fx<NF, 3>;
    }
    *fn = (const void*)ray_kernel<NF, false, false, FxRay<NF, false, 3>>;
    return launch_ray_fx<NF, false>;
}

}  // namespace

RayLaunchFn pick_ray_kernel_fx(int nf, bool mixed, const void** fn, bool pool, long long rays) {
    const bool many = rays >= kFxManyRays;
    if (nf <= 1) return pick<1>(mixed, fn, pool, many);
    if (nf <= 2) return pick<2>(mixed, fn, pool, many);
    if (nf <= 4) return pick<4>(mixed, fn, pool, many);
    return pick<8>(mixed, fn, pool, many);
}
