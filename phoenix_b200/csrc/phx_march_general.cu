// Host side of the marching-warps iteration with noise, pulses, a second pump
// group or two polarisations: kernel variant, row segments, launch.
#include "phx_march.hpp"
#include "phx_march_plan.hpp"
#include "phx_step_march_general.cuh"

namespace phx {
namespace {

template <typename T, int COMPS>
using GeneralKernel = void (*)(MarchGeneralParams<T, COMPS>);

struct Variant {
    int np, nv, nq;
    bool noise, img;
};

// kernel and shared memory of a variant; a null kernel when there is none
template <typename T, int COMPS, int NP, int NV, int NQ, bool NOISE>
void take(const Variant& v, GeneralKernel<T, COMPS>& k, int& bytes) {
    if (v.np != NP || v.nv != NV || v.nq != NQ || v.noise != NOISE) return;
    constexpr int MINB = COMPS == 1 && sizeof(T) == 4 ? 3 : 2;
    k = rk4_march_general_kernel<T, COMPS, true, NP, NV, NQ, NOISE, true, false, MINB>;
    if constexpr (sizeof(T) == 8) {  // odd numbers of columns are FP64's
        if (v.img) k = rk4_march_general_kernel<T, COMPS, true, NP, NV, NQ, NOISE, true, true, MINB>;
    }
    bytes = MarchGeneralLayout<T, COMPS, true, NP, NV, NQ, NOISE>::bytes;
}
template <typename T, int COMPS, int NP, int NV, int NQ>
void take_noise(const Variant& v, GeneralKernel<T, COMPS>& k, int& bytes) {
    // the scalar model with one pump group, no pulse and no noise is phx_step_march.cuh's
    if constexpr (COMPS == 2 || NP > 1 || NQ > 0) take<T, COMPS, NP, NV, NQ, false>(v, k, bytes);
    take<T, COMPS, NP, NV, NQ, true>(v, k, bytes);
}
template <typename T, int COMPS, int NP>
void take_rest(const Variant& v, GeneralKernel<T, COMPS>& k, int& bytes) {
    take_noise<T, COMPS, NP, 0, 0>(v, k, bytes);
    take_noise<T, COMPS, NP, 0, 1>(v, k, bytes);
    take_noise<T, COMPS, NP, 1, 0>(v, k, bytes);
    take_noise<T, COMPS, NP, 1, 1>(v, k, bytes);
}

}  // namespace

template <typename T>
template <int COMPS>
bool MarchGeneral<T>::launch_comps(const TetmParams<T> (&st)[4], const cx<T>* const* psi0, const T* const* n0,
                                   cx<T>* const* psi1, T* const* n1, int sm_count, cudaStream_t stream, bool pdl) {
    const StageParams<T>& P = st[0].p;
    const Variant v{P.n_pump, P.n_pot, P.n_pulse, P.noise.on != 0, march_needs_images(P.N_c, P.img_x)};
    GeneralKernel<T, COMPS> kern = nullptr;
    int bytes = 0;
    take_rest<T, COMPS, 1>(v, kern, bytes);
    if constexpr (COMPS == 1) take_rest<T, COMPS, 2>(v, kern, bytes);
    if (!kern) return false;
    int& per_sm = per_sm_[reinterpret_cast<const void*>(kern)];
    if (!per_sm) per_sm = march_occupancy(kern, bytes);
    MarchGeneralParams<T, COMPS> G;
    for (int s = 0; s < 4; ++s) G.st[s] = st[s];
    for (int q = 0; q < COMPS; ++q) {
        G.psi0[q] = psi0[q];
        G.n0[q] = n0[q];
        G.psi1[q] = psi1[q];
        G.n1[q] = n1[q];
    }
    G.strips = (P.N_c + kMarchOut - 1) / kMarchOut;
    const std::array<int, 4> plan = {P.N_r, P.N_c, per_sm, sm_count};
    if (plan != plan_) {
        plan_rows_ = march_seg_rows<T>(
            P.N_r, [&](int L) { return (long long)G.strips * ((P.N_r + L - 1) / L); }, per_sm, sm_count);
        plan_ = plan;
    }
    G.seg_rows = plan_rows_;
    G.n_items = G.strips * ((P.N_r + G.seg_rows - 1) / G.seg_rows);
    march_launch(kern, G, G.n_items, bytes, stream, pdl);
    return true;
}

template <typename T>
bool MarchGeneral<T>::launch(const TetmParams<T> (&st)[4], int comps, bool res, const cx<T>* const* psi0, const T* const* n0,
                             cx<T>* const* psi1, T* const* n1, int sm_count, cudaStream_t stream, bool pdl) {
    const StageParams<T>& P = st[0].p;
    // Small grids give every scheduler less than one warp, whose steps then run at
    // their latency; the tile kernels spread such a grid wider.  us per iteration,
    // tiles against march: FP32 without noise 9.2 / 7.8 at 128^2 already; with
    // noise (long steps) 10.2 / 14.4 at 256^2, 22.7 / 23.3 at 512^2, 68.9 / 46.5 at
    // 1024^2, the spinor 28 / 46 at 384^2, 48 / 46 at 512^2; FP64 9.1 / 14.3 at
    // 256^2, 16.4 / 16.7 at 384^2, 28.6 / 21.8 at 512^2.
    const long long points = (long long)P.N_r * P.N_c;
    if (points < (P.noise.on ? 280000 : (sizeof(T) == 8 ? 150000 : 0))) return false;
    // 32-bit indices over every group's planes; a reservoir with its pump; real
    // potential coefficients
    const int groups = std::max({1, P.n_pump, P.n_pot, P.n_pulse});
    if (!res || P.n_pump < 1 || P.plane * groups >= (1LL << 31)) return false;
    for (int s = 0; s < 4; ++s)
        for (int g = 0; g < P.n_pot; ++g)
            if (st[s].p.pot_c[g].im != (T)0) return false;
    if (comps == 1) return launch_comps<1>(st, psi0, n0, psi1, n1, sm_count, stream, pdl);
    // FP64: two polarisations' rows do not fit the registers
    if constexpr (sizeof(T) == 4) return launch_comps<2>(st, psi0, n0, psi1, n1, sm_count, stream, pdl);
    return false;
}

template class MarchGeneral<float>;
template class MarchGeneral<double>;

}  // namespace phx
