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
    ray_kernel<NF, MIXED, false, FxRay<NF, MIXED>><<<ls.grid, ls.block, 0, st>>>(imgs, n, b, e, ctr, out, ls.refill,
                                                                                tr);
}
template <int NF>
void launch_ray_pool_fx(const LaunchShape& ls, cudaStream_t st, const DevImage* imgs, int n, long long b, long long e,
                        unsigned long long* ctr, double* out, TraceSpec) {
    ray_kernel_pool<NF, FxRay<NF, false>><<<ls.grid, ls.block, 0, st>>>(imgs, n, b, e, ctr, out, ls.refill);
}

template <int NF>
RayLaunchFn pick(bool mixed, const void** fn, bool pool) {
    if (mixed) {
        *fn = (const void*)ray_kernel<NF, true, false, FxRay<NF, true>>;
        return launch_ray_fx<NF, true>;
    }
    if (pool) {
        *fn = (const void*)ray_kernel_pool<NF, FxRay<NF, false>>;
        return launch_ray_pool_fx<NF>;
    }
    *fn = (const void*)ray_kernel<NF, false, false, FxRay<NF, false>>;
    return launch_ray_fx<NF, false>;
}

}  // namespace

RayLaunchFn pick_ray_kernel_fx(int nf, bool mixed, const void** fn, bool pool) {
    if (nf <= 1) return pick<1>(mixed, fn, pool);
    if (nf <= 2) return pick<2>(mixed, fn, pool);
    if (nf <= 4) return pick<4>(mixed, fn, pool);
    return pick<8>(mixed, fn, pool);
}
