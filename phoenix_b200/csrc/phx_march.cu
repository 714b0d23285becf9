// Host side of the marching-warps RK4 iteration: kernel variant, row segments,
// launch.
#include "phx_march.hpp"

#include "phx_step_march.cuh"

namespace phx {
namespace {

// Rows per segment.  A segment of L rows costs about L + 3 full steps (its
// first rows run through some stages only), and an SM with w CTAs takes
// cost[w] per step of all of them (measured at 1024^2; one CTA leaves its
// schedulers waiting on one warp's latencies).  More CTAs than fit at once
// follow one another without a common end, hence the fractional rounds.
template <typename T>
int march_seg_rows(int N_r, int strips, int per_sm, int sm_count) {
    const double cost32[4] = {0.0, 0.61, 0.86, 1.2}, cost64[3] = {0.0, 0.94, 1.55};
    auto cost = [&](int w) {
        if (sizeof(T) == 4) return w <= 3 ? cost32[w] : cost32[3] * w / 3;
        return w <= 2 ? cost64[w] : cost64[2] * w / 2;
    };
    int best_L = N_r;
    double best = -1.0;
    for (int L = std::min(N_r, 2); L <= std::min(N_r, 256); ++L) {
        const long long items = (long long)strips * ((N_r + L - 1) / L);
        const long long ctas = (items + kMarchWarps - 1) / kMarchWarps;
        const long long w = (ctas + sm_count - 1) / sm_count;
        const double t = (L + 3.0) * (w <= per_sm ? cost((int)w)
                                                  : ((double)ctas / ((double)per_sm * sm_count) + 0.3) * cost(per_sm));
        if (best < 0.0 || t < best) best = t, best_L = L;
    }
    return best_L;
}

}  // namespace

template <typename T>
void MarchLauncher<T>::launch(const FusedParams<T>& F, const MarchOptions& o, int sm_count, cudaStream_t stream) {
    constexpr int MINB = sizeof(T) == 4 ? 3 : 2;  // FP32 150, FP64 250 registers
    using Lay = MarchLayout<T>;
    using K = void (*)(MarchParams<T>);
    bool unit = true;
    for (int s = 0; s < 4; ++s) {
        if (F.pump && F.pump_c[s] != (T)1) unit = false;
        if (F.pot && F.pot_c[s] != (T)1) unit = false;
    }
    // the variant with temporal coefficients always takes the potential's terms
    const bool pot = F.pot != nullptr || !unit;
    K kern = nullptr;
    auto pick = [&](auto res, auto fma, auto store) {
        constexpr bool R = decltype(res)::value, M = decltype(fma)::value, S = decltype(store)::value;
        kern = !pot ? (K)rk4_march_kernel<T, R, false, true, M, S, MINB>
                    : (unit ? (K)rk4_march_kernel<T, R, true, true, M, S, MINB> : (K)rk4_march_kernel<T, R, true, false, M, S, MINB>);
    };
    using std::false_type;
    using std::true_type;
    if (o.store) {
        if (o.fma || !unit) fail(PHX_ERR_UNSUPPORTED, "stage values are stored in the bit-exact arithmetic with constant envelopes");
        if (o.res)
            kern = pot ? (K)rk4_march_kernel<T, true, true, true, false, true, MINB> : (K)rk4_march_kernel<T, true, false, true, false, true, MINB>;
        else
            kern = pot ? (K)rk4_march_kernel<T, false, true, true, false, true, MINB> : (K)rk4_march_kernel<T, false, false, true, false, true, MINB>;
    } else if (o.fma) {
        if constexpr (sizeof(T) == 4) {
            if (o.res) pick(true_type{}, true_type{}, false_type{});
            else pick(false_type{}, true_type{}, false_type{});
        }
    } else {
        if (o.res) pick(true_type{}, false_type{}, false_type{});
        else pick(false_type{}, false_type{}, false_type{});
    }
    if (!kern) fail(PHX_ERR_UNSUPPORTED, "the fused multiply-add arithmetic is FP32 only");
    int& per_sm = per_sm_[reinterpret_cast<const void*>(kern)];
    if (!per_sm) {
        PHX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::bytes));
        PHX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kMarchWarps, Lay::bytes));
        if (per_sm < 1) fail(PHX_ERR_UNSUPPORTED, "marching iteration kernel does not fit on an SM");
    }
    MarchParams<T> Q;
    Q.f = F;
    Q.strips = (F.N_c + kMarchOut - 1) / kMarchOut;
    const std::array<int, 4> plan = {F.N_r, F.N_c, per_sm, sm_count};
    if (plan != plan_) {
        plan_rows_ = march_seg_rows<T>(F.N_r, Q.strips, per_sm, sm_count);
        plan_ = plan;
    }
    Q.seg_rows = plan_rows_;
    Q.n_items = Q.strips * ((F.N_r + Q.seg_rows - 1) / Q.seg_rows);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((Q.n_items + kMarchWarps - 1) / kMarchWarps));
    cfg.blockDim = dim3(32 * kMarchWarps);
    cfg.dynamicSmemBytes = Lay::bytes;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = o.pdl ? 1 : 0;
    PHX_CUDA(cudaLaunchKernelEx(&cfg, kern, Q));
}

template class MarchLauncher<float>;
template class MarchLauncher<double>;

}  // namespace phx
