// Launch-shape autotuner for the persistent ray kernel.
//
// The shape of the persistent launch - threads per block (at the resident
// blocks per SM that the kernel's registers allow) and how many geodesic
// steps a lane runs between queue refills ("steps per chunk") - trades
// warp granularity against lane idling at ray ends.  With options.autotune
// set, the first render of a batch
// signature (device, precision, frequency bucket, size class) times each
// candidate on a sample of that batch's rays - a contiguous range from its
// middle, about six rays per lane - and keeps the fastest.  Results live in
// the context and, if RAPTOR_TUNE_CACHE names a file, are appended there and
// read back by later contexts.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "engine_internal.h"
#include "ray_kernel.cuh"

using raptor::kCtrCount;
using raptor::TraceSpec;

namespace {

int occupancy(const void* fn, int block) {
    int occ = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, block, 0);
    return std::max(occ, 1);
}

// What a tuned shape is kept for: the form, the size class, and what the rules
// on the number of rays, whose lines lie inside the classes, make of it: the
// kernel's blocks per SM (its register budget), one block per SM or all that
// fit, and the queue's order.
std::string signature(const raptor_gpu_ctx* ctx, const Batch& b, int form, const void* fnp, const LaunchShape& base,
                      long long rays) {
    char k[384];
    const int size_class = (int)std::log2((double)std::max<long long>(rays, 1));
    const char* name = form == RAPTOR_PREC_MIXED_DF ? "mixed_df"
                       : form == RAPTOR_PREC_MIXED  ? "mixed"
                       : ctx->opt.no_sample_pool    ? "fp64_inplace"
                                                    : "fp64";
    const char* geo = b.fixed && form != RAPTOR_PREC_MIXED_DF ? "_fx" : "";
    const char* grid = base.bps == 1 ? "one" : "full";
    const char* order = raptor::middle_out(rays, (long long)base.grid * base.block) ? "middle" : "rows";
    snprintf(k, sizeof k, "%s|%s%s|b%d|%s|%s|nf%d|2^%d", ctx->device_name, name, geo, occupancy(fnp, raptor::kRayMaxBlock),
             grid, order, b.max_nf, size_class);
    std::string s(k);
    for (char& c : s)
        if (c == ' ') c = '_';
    return s;
}

void load_file_cache(raptor_gpu_ctx* ctx) {
    const char* path = getenv("RAPTOR_TUNE_CACHE");
    if (!path || ctx->tune_file_loaded) return;
    ctx->tune_file_loaded = true;
    FILE* f = fopen(path, "r");
    if (!f) return;
    char key[384];
    LaunchShape ls;
    while (fscanf(f, "%383s %d %d %d", key, &ls.block, &ls.bps, &ls.refill) == 4) ctx->tuned[key] = ls;
    fclose(f);
}

void save_file_cache(const std::string& key, const LaunchShape& ls) {
    const char* path = getenv("RAPTOR_TUNE_CACHE");
    if (!path) return;
    FILE* f = fopen(path, "a");
    if (!f) return;
    fprintf(f, "%s %d %d %d\n", key.c_str(), ls.block, ls.bps, ls.refill);
    fclose(f);
}

}  // namespace

LaunchShape choose_shape(raptor_gpu_ctx* ctx, const Batch& b, int form, RayLaunchFn fn, const void* fnp, long long rays) {
    LaunchShape base = default_shape(ctx, fnp, form, b.fixed, b.rk2, rays);
    if (!ctx->opt.autotune) return base;
    load_file_cache(ctx);
    const std::string key = signature(ctx, b, form, fnp, base, rays);
    auto it = ctx->tuned.find(key);
    if (it != ctx->tuned.end()) {
        LaunchShape ls = it->second;
        ls.bps = std::max(1, std::min(ls.bps, occupancy(fnp, ls.block)));
        ls.grid = ctx->num_sms * ls.bps;
        return ls;
    }
    // Candidates run at full occupancy.  The timed sample has a few rays per
    // lane, where a smaller grid wins by balancing the tail; on whole batches
    // (~100 rays per lane) full occupancy is faster (64 images: 2 blocks of 128
    // per SM 3545 ms, 1 block 3630 ms), so only the block size and the refill
    // interval are tuned.
    std::vector<LaunchShape> cands;
    for (int block : {64, 128}) {
        const int occ = occupancy(fnp, block);
        for (int refill : {1, 4, 8, 16}) {
            LaunchShape ls;
            ls.block = block;
            ls.bps = occ;
            ls.grid = ctx->num_sms * occ;
            ls.refill = refill;
            cands.push_back(ls);
        }
    }
    if (base.bps == 1) cands.push_back(base);  // a launch of all its rays at once (default_blocks)
    // the timed sample: a launch whose rays go in the order of rows is timed on
    // enough of them to be one too, at every candidate's grid
    long long lanes = 0;
    for (const LaunchShape& ls : cands) lanes = std::max(lanes, (long long)ls.grid * ls.block);
    const long long n = std::min<long long>(rays, (raptor::kOrderedLanes + 1) * lanes);
    const long long rb = (b.total_rays - n) / 2, re = rb + n;
    LaunchShape best = base;
    float best_ms = 1e30f;
    const TraceSpec none{-1, nullptr, 0};
    for (size_t k = 0; k <= cands.size(); ++k) {
        // k == 0 is a warm-up of the default shape
        const LaunchShape& ls = k == 0 ? base : cands[k - 1];
        cudaMemsetAsync(ctx->d_counters, 0, kCtrCount * sizeof(unsigned long long), ctx->stream);
        cudaEventRecord(ctx->ev0, ctx->stream);
        fn(ls, ctx->stream, ctx->d_imgs, b.n, rb, re, ctx->d_counters, ctx->d_out, none);
        cudaEventRecord(ctx->ev1, ctx->stream);
        if (cudaEventSynchronize(ctx->ev1) != cudaSuccess) {
            cudaGetLastError();
            return base;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        if (k > 0 && ms < best_ms) {
            best_ms = ms;
            best = ls;
        }
    }
    ctx->tuned[key] = best;
    save_file_cache(key, best);
    return best;
}
