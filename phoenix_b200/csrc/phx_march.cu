// Host side of the marching-warps RK4 iteration: kernel variant, row segments,
// launch.
#include "phx_march.hpp"

#include "phx_march_plan.hpp"
#include "phx_step_march.cuh"

namespace phx {
namespace {

// CTAs per SM the registers must leave room for (FP32 155, FP64 250 registers)
template <typename T>
constexpr int kMarchMinB = sizeof(T) == 4 ? 3 : 2;

}  // namespace

template <typename T>
void MarchLauncher<T>::launch(const FusedParams<T>& F, const MarchOptions& o, int sm_count, cudaStream_t stream) {
    constexpr int MINB = kMarchMinB<T>;
    using Lay = MarchLayout<T>;
    using K = void (*)(MarchParams<T>);
    bool unit = true;
    for (int s = 0; s < 4; ++s) {
        if (F.pump && F.pump_c[s] != (T)1) unit = false;
        if (F.pot && F.pot_c[s] != (T)1) unit = false;
    }
    const bool pot = F.pot != nullptr;
    K kern = nullptr;
    using std::false_type;
    using std::true_type;
    auto pick = [&](auto res, auto fma, auto img) {
        constexpr bool R = decltype(res)::value, M = decltype(fma)::value, I = decltype(img)::value;
        kern = pot ? (unit ? (K)rk4_march_kernel<T, R, true, true, M, false, I, MINB>
                           : (K)rk4_march_kernel<T, R, true, false, M, false, I, MINB>)
                   : (unit ? (K)rk4_march_kernel<T, R, false, true, M, false, I, MINB>
                           : (K)rk4_march_kernel<T, R, false, false, M, false, I, MINB>);
    };
    auto pick_store = [&](auto res, auto img) {
        constexpr bool R = decltype(res)::value, I = decltype(img)::value;
        kern = pot ? (K)rk4_march_kernel<T, R, true, true, false, true, I, MINB>
                   : (K)rk4_march_kernel<T, R, false, true, false, true, I, MINB>;
    };
    if (o.store) {
        if (!unit) fail(PHX_ERR_UNSUPPORTED, "stage values are stored with constant envelopes");
        auto pick_img = [&](auto img) { o.res ? pick_store(true_type{}, img) : pick_store(false_type{}, img); };
        if (!o.img) pick_img(false_type{});
        if constexpr (sizeof(T) == 8) {  // odd numbers of columns, and the tile sweep of the adjoint, are FP64's
            if (o.img) pick_img(true_type{});
        }
    } else if (o.fma) {
        if constexpr (sizeof(T) == 4) {
            if (o.res) pick(true_type{}, true_type{}, false_type{});
            else pick(false_type{}, true_type{}, false_type{});
        }
    } else if (o.img) {
        if constexpr (sizeof(T) == 8) {  // odd numbers of columns are FP64's
            if (o.res) pick(true_type{}, false_type{}, true_type{});
            else pick(false_type{}, false_type{}, true_type{});
        }
    } else {
        if (o.res) pick(true_type{}, false_type{}, false_type{});
        else pick(false_type{}, false_type{}, false_type{});
    }
    if (!kern) fail(PHX_ERR_UNSUPPORTED, "no marching variant for these options");
    int& per_sm = per_sm_[reinterpret_cast<const void*>(kern)];
    if (!per_sm) per_sm = march_occupancy(kern, Lay::bytes);
    MarchParams<T> Q;
    Q.f = F;
    Q.strips = (F.N_c + kMarchOut - 1) / kMarchOut;
    const std::array<int, 4> plan = {F.N_r, F.N_c, per_sm, sm_count};
    if (plan != plan_) {
        plan_rows_ = march_segments(F.N_r, [&](int L) { return (long long)Q.strips * ((F.N_r + L - 1) / L); }, per_sm,
                                    sm_count, kMarchCost<T>)
                         .rows;
        plan_ = plan;
    }
    Q.seg_rows = plan_rows_;
    Q.n_items = Q.strips * ((F.N_r + Q.seg_rows - 1) / Q.seg_rows);
    march_launch(kern, Q, Q.n_items, Lay::bytes, stream, o.pdl);
}

template <typename T>
void MarchBatch<T>::build(const std::vector<FusedParams<T>>& f, bool res, bool fma, int sm_count, cudaStream_t stream) {
    using K = void (*)(MarchBatchParams<T>);
    constexpr int MINB = kMarchMinB<T>;
    int with_pot = 0, max_rows = 1;
    const int n = (int)(f.size() / 2);
    for (int i = 0; i < n; ++i) {
        with_pot += f[2 * i].pot != nullptr;
        max_rows = std::max(max_rows, f[2 * i].N_r);
    }
    K kern = nullptr;
    auto pick_pots = [&](auto r, auto m, auto img) {
        constexpr bool R = decltype(r)::value, M = decltype(m)::value, I = decltype(img)::value;
        kern = with_pot == 0   ? (K)rk4_march_batch_kernel<T, R, 0, M, I, MINB>
               : with_pot == n ? (K)rk4_march_batch_kernel<T, R, 1, M, I, MINB>
                               : (K)rk4_march_batch_kernel<T, R, 2, M, I, MINB>;
    };
    auto pick = [&](auto m, auto img) {
        if (res) pick_pots(std::true_type{}, m, img);
        else pick_pots(std::false_type{}, m, img);
    };
    images_ = false;
    for (int i = 0; i < n; ++i) images_ = images_ || march_needs_images(f[2 * i].N_c, f[2 * i].img_x);
    if constexpr (sizeof(T) == 4) {
        if (fma) pick(std::true_type{}, std::false_type{});
    } else {
        if (images_) pick(std::false_type{}, std::true_type{});
    }
    if (!kern) pick(std::false_type{}, std::false_type{});
    const int per_sm = march_occupancy(kern, MarchLayout<T>::bytes);
    auto strips = [&](int i) { return (f[2 * i].N_c + kMarchOut - 1) / kMarchOut; };
    const int L = march_segments(
                      max_rows,
                      [&](int l) {
                          long long items = 0;
                          for (int i = 0; i < n; ++i) items += (long long)strips(i) * ((f[2 * i].N_r + l - 1) / l);
                          return items;
                      },
                      per_sm, sm_count, kMarchCost<T>)
                      .rows;
    std::vector<MarchItem> items;
    for (int i = 0; i < n; ++i) {
        const int rows = f[2 * i].N_r, segs = (rows + L - 1) / L, per = (rows + segs - 1) / segs;
        for (int r = 0; r < rows; r += per)
            for (int s = 0; s < strips(i); ++s) items.push_back({i, s, r, std::min(r + per, rows)});
    }
    f_.alloc(sizeof(FusedParams<T>) * f.size(), stream);
    items_.alloc(sizeof(MarchItem) * items.size(), stream);
    PHX_CUDA(cudaMemcpyAsync(f_.p, f.data(), f_.bytes, cudaMemcpyHostToDevice, stream));
    PHX_CUDA(cudaMemcpyAsync(items_.p, items.data(), items_.bytes, cudaMemcpyHostToDevice, stream));
    PHX_CUDA(cudaStreamSynchronize(stream));  // the host vectors die here
    kern_ = reinterpret_cast<const void*>(kern);
    n_items_ = (int)items.size();
}

template <typename T>
void MarchBatch<T>::launch(int dir, cudaStream_t stream) const {
    MarchBatchParams<T> Q;
    Q.f = static_cast<const FusedParams<T>*>(f_.p);
    Q.items = static_cast<const MarchItem*>(items_.p);
    Q.n_items = n_items_;
    Q.dir = dir;
    void* args[] = {&Q};
    PHX_CUDA(cudaLaunchKernel(kern_, dim3((unsigned)((n_items_ + kMarchWarps - 1) / kMarchWarps)), dim3(32 * kMarchWarps), args,
                              MarchLayout<T>::bytes, stream));
}

template class MarchBatch<float>;
template class MarchBatch<double>;
template class MarchLauncher<float>;
template class MarchLauncher<double>;

}  // namespace phx
