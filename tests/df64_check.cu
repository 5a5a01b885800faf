// The shortened double-float operations of csrc/df64.cuh against its general
// ones, bit for bit, and its comparison against the exact sign (run by
// tests/test_gpu_df_sums.py).  Prints how many results of each differ.
#include <cmath>
#include <cstdio>

#include "dual.cuh"
#include "df64.cuh"

using namespace raptor;

__device__ unsigned next(unsigned& s) { return s = s * 1664525u + 1013904223u; }
// A double-float value with exponent lo..hi, its lo part a few ulp as products leave it
__device__ DF value(unsigned& s, int lo, int hi) {
    const float m = 1.0f + (float)(next(s) >> 9) * 0x1p-23f;
    const float h = ldexpf((next(s) >> 31) ? m : -m, lo + (int)(next(s) >> 8) % (hi - lo));
    return DF{h, h * ((float)(int)next(s) * 0x1p-29f) * 0x1p-24f};
}
__device__ bool same(DF a, DF b) {
    return __float_as_uint(a.hi) == __float_as_uint(b.hi) && __float_as_uint(a.lo) == __float_as_uint(b.lo);
}

__global__ void check(int rounds, unsigned* bad) {
    unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < 8; ++k) next(s);
    for (int k = 0; k < rounds; ++k) {
        DF a = value(s, -3, 14), b = value(s, -3 - (k % 4) * 12, 14 - (k % 4) * 12);
        if (fabsf(a.hi) < fabsf(b.hi)) {
            const DF t = a;
            a = b;
            b = t;
        }
        if (!same(add_ordered(a, b), a + b)) atomicAdd(bad + 0, 1u);
        if (!same(add_ordered(a, b.hi), add_f(a, b.hi))) atomicAdd(bad + 1, 1u);
        const DF f{a.hi, 0.0f};
        if (!same(add_ordered(a.hi, b), add_f(b, a.hi)) && !same(add_ordered(a.hi, b), f + b)) atomicAdd(bad + 2, 1u);
        const DF c = value(s, -3, 14), d = value(s, -3, 14);
        for (float w : {0.5f, 1.0f, 2.0f})
            if (!same(add_scaled(c, d, w), c + stage_scale(d, w))) atomicAdd(bad + 3, 1u);
        const DF p = c * d;
        if (fabsf(p.hi) >= fabsf(b.hi) && !same(fma_large(c, d, b), fma(c, d, b))) atomicAdd(bad + 4, 1u);
        if (fabsf(p.hi) <= fabsf(a.hi) && !same(fma_small(c, d, a), fma(c, d, a))) atomicAdd(bad + 5, 1u);
        if (fabsf(p.hi) <= 1.0f && !same(fma_small(c, d, 1.0), fma(c, d, 1.0))) atomicAdd(bad + 6, 1u);
        // neighbours, equal leading parts, and values of their own
        const DF near{nextafterf(c.hi, k % 2 ? INFINITY : -INFINITY), 0.5f * c.lo};
        const DF twin{c.hi, nextafterf(c.lo, 0.0f)};
        for (const DF e : {near, twin, d, c}) {
            const double diff = ((double)c.hi - (double)e.hi) + ((double)c.lo - (double)e.lo);
            if ((c < e) != (diff < 0.0)) atomicAdd(bad + 7, 1u);
        }
    }
}

int main() {
    unsigned *d = nullptr, h[8];
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 2;
    check<<<64, 128>>>(64, d);
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    for (unsigned x : h) printf("%u\n", x);
    cudaFree(d);
    return 0;
}
