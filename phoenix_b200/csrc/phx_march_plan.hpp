// Row segments and occupancy of the marching-warps kernels (phx_march.cu,
// phx_march_general.cu).
#pragma once

#include <algorithm>

#include "phx_rt.hpp"
#include "phx_step_march.cuh"

namespace phx {

// Rows per segment.  A segment of L rows costs about L + extra full steps (its
// first rows run through some stages only; four stages: 3), and an SM with w
// CTAs takes cost(w) per step of all of them (measured at 1024^2; one CTA
// leaves its schedulers waiting on one warp's latencies).  More CTAs than fit
// at once run in rounds.  4096^2 FP32: 184 us at 64 rows (estimate 189), 196 at
// 32 (199).
template <typename T>
double march_cost(int L, long long items, int per_sm, int sm_count, double extra) {
    const double cost32[4] = {0.0, 0.47, 0.74, 1.05}, cost64[3] = {0.0, 0.92, 1.52};
    auto cost = [&](int w) {
        if (sizeof(T) == 4) return w <= 3 ? cost32[w] : cost32[3] * w / 3;
        return w <= 2 ? cost64[w] : cost64[2] * w / 2;
    };
    const long long ctas = (items + kMarchWarps - 1) / kMarchWarps, w = (ctas + sm_count - 1) / sm_count;
    return (L + extra) * ((double)(w / per_sm) * cost(per_sm) + cost((int)(w % per_sm)));
}
// the cheapest segment length of at most max_rows, items(L) segments in all
template <typename T, typename Items>
int march_seg_rows(int max_rows, const Items& items, int per_sm, int sm_count, double extra = 3.0) {
    int best_L = max_rows;
    double best = -1.0;
    for (int L = std::min(max_rows, 2); L <= std::min(max_rows, 256); ++L) {
        const double t = march_cost<T>(L, items(L), per_sm, sm_count, extra);
        if (best < 0.0 || t < best) best = t, best_L = L;
    }
    return best_L;
}
template <typename K, typename Q>
void march_launch(K kern, const Q& params, int n_items, int bytes, cudaStream_t stream, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((n_items + kMarchWarps - 1) / kMarchWarps));
    cfg.blockDim = dim3(32 * kMarchWarps);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    PHX_CUDA(cudaLaunchKernelEx(&cfg, kern, params));
}
template <typename K>
int march_occupancy(K kern, int bytes) {
    int per_sm = 0;
    PHX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    PHX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kMarchWarps, bytes));
    if (per_sm < 1) fail(PHX_ERR_UNSUPPORTED, "marching iteration kernel does not fit on an SM");
    return per_sm;
}

}  // namespace phx
