// Row segments and occupancy of the marching-warps kernels (phx_march.cu,
// phx_march_general.cu).
#pragma once

#include <algorithm>

#include "phx_rt.hpp"
#include "phx_step_march.cuh"

namespace phx {

// What a launch of a marching kernel takes: base + (L + extra) step(w) for
// segments of L rows with w CTAs on an SM.  A segment runs L + 6 steps, `extra`
// counts them in full ones (its first rows go through some of the stages only);
// one CTA leaves its schedulers waiting on one warp's latencies, so a step of two
// CTAs does not take twice its time.  More CTAs than fit at once run in rounds.
struct MarchCost {
    double base, extra, step[3];  // us; step: with one, two, three CTAs per SM
    double of(int ctas) const { return ctas <= 0 ? 0.0 : (ctas <= 3 ? step[ctas - 1] : step[2] * ctas / 3); }
};
// The plain scalar iteration at 1024^2 (no base: its own segments are all that it
// is used to compare); 4096^2 FP32: 184 us at 64 rows (estimate 189), 196 at 32
// (199).  The adjoint's kernel takes the same figures; its steps last longer and
// its start is nearer four of them.
template <typename T>
constexpr MarchCost kMarchCost = sizeof(T) == 4 ? MarchCost{0.0, 3.0, {0.47, 0.74, 1.05}}
                                                : MarchCost{0.0, 3.0, {0.92, 1.52, 2.28}};

// the cheapest segment length of at most max_rows, items(L) segments in all, and its time
struct MarchSegments {
    int rows;
    double us;
};
template <typename Items>
MarchSegments march_segments(int max_rows, const Items& items, int per_sm, int sm_count, const MarchCost& cost) {
    MarchSegments best{max_rows, -1.0};
    for (int L = std::min(max_rows, 2); L <= std::min(max_rows, 256); ++L) {
        const long long ctas = (items(L) + kMarchWarps - 1) / kMarchWarps, w = (ctas + sm_count - 1) / sm_count;
        const double us =
            cost.base + (L + cost.extra) * ((double)(w / per_sm) * cost.of(per_sm) + cost.of((int)(w % per_sm)));
        if (best.us < 0.0 || us < best.us) best = {L, us};
    }
    return best;
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
