// Host side of the adjoint's marching-warps kernel: variant, row segments, launch.
#include "phx_adjoint_march.cuh"
#include "phx_march.hpp"
#include "phx_march_plan.hpp"

namespace phx {

template <typename T>
void AdjMarch<T>::launch(const AdjFusedParams<T>& Q, int sm_count, cudaStream_t stream, bool pdl) {
    using K = void (*)(AdjMarchParams<T>);
    using Lay = AdjMarchLayout<T>;
    const bool res = Q.res != 0, pot = Q.pot != nullptr;
    auto pick = [&](auto wrap) -> K {
        constexpr bool W = decltype(wrap)::value;
        return res ? (pot ? (K)adj_march_kernel<T, true, true, W, 2> : (K)adj_march_kernel<T, true, false, W, 2>)
                   : (pot ? (K)adj_march_kernel<T, false, true, W, 2> : (K)adj_march_kernel<T, false, false, W, 2>);
    };
    K kern = nullptr;
    if (wraps(Q.N_c)) {
        kern = pick(std::true_type{});
    } else {
        if constexpr (sizeof(T) == 8) kern = pick(std::false_type{});  // FP32 grids have an even number of columns
    }
    if (!kern) fail(PHX_ERR_UNSUPPORTED, "FP32 grids need an even N_c");
    int& per_sm = per_sm_[reinterpret_cast<const void*>(kern)];
    if (!per_sm) per_sm = march_occupancy(kern, Lay::bytes);
    AdjMarchParams<T> M;
    M.a = Q;
    M.strips = (Q.N_c + kMarchOut - 1) / kMarchOut;
    const std::array<int, 4> plan = {Q.N_r, Q.N_c, per_sm, sm_count};
    if (plan != plan_) {
        plan_rows_ = march_segments(Q.N_r, [&](int L) { return (long long)M.strips * ((Q.N_r + L - 1) / L); }, per_sm,
                                    sm_count, kMarchCost<T>)
                         .rows;
        plan_ = plan;
    }
    M.seg_rows = plan_rows_;
    M.n_items = M.strips * ((Q.N_r + M.seg_rows - 1) / M.seg_rows);
    march_launch(kern, M, M.n_items, Lay::bytes, stream, pdl);
}

template class AdjMarch<float>;
template class AdjMarch<double>;

}  // namespace phx
