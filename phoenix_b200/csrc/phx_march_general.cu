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
    k = rk4_march_general_kernel<T, COMPS, NP, NV, NQ, NOISE, true, false, MINB>;
    if constexpr (sizeof(T) == 8) {  // odd numbers of columns are FP64's
        if (v.img) k = rk4_march_general_kernel<T, COMPS, NP, NV, NQ, NOISE, true, true, MINB>;
    }
    bytes = MarchGeneralLayout<T, COMPS, NP, NV, NQ, NOISE>::bytes;
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

// Marching or tile kernel?  Small grids give every scheduler of the marching
// kernel less than one warp, whose steps then run at their latency, narrow ones
// fill half a strip, and long steps of noisy spinors hide nothing behind each
// other; tiles spread such grids wider.  Both are estimated in us.  The marching
// kernel: MarchCost as measured on 224 columns with segments of 8 to 32 rows, one
// to three CTAs per SM.  The tile kernels (phx_step_tetm_fused.cuh): first + round n
// for n = ceil(tiles / SMs), within 9 % of 45 grids from n = 2 on, and at least
// `one`.  march_input and tile_input are the shares that a potential or a pulse
// adds.  Over 896 grids and kinds, from 8 to 1024 columns, the choice costs 5 % at
// most against the faster of the two.
// Tile / marching kernel, us: FP32 with a pulse 7.3 / 5.4 at 64^2, 28 / 15 at 768^2;
// with noise 8.7 / 12.5 at 256^2, 20.2 / 19.4 at 544 x 520, 61 / 40 at 1024^2; the
// spinor 11.2 / 11.7 at 256^2, 14.9 / 16.4 at 24 x 4096, 27 / 19 at 512^2, with noise
// 15 / 28 at 256^2, 38 / 45 at 544 x 520, 124 / 74 at 1024^2, with a pulse and a
// potential as well (one CTA per SM) 98 / 108 at 768^2, 176 / 172 at 1024^2; FP64 with
// a pulse 13.9 / 14.5 at 384^2, 24 / 28 at 64 x 4096, 50 / 29 at 768^2.
struct Kind {
    MarchCost march;
    double march_input;
    double one, first, round, tile_input;
};
template <typename T>
const Kind& kind_of(int comps, bool noise) {
    static const Kind f32[4] = {{{2.0, 6.0, {0.456, 0.722, 1.11}}, 0.09, 6.2, 2.4, 2.7, 0.16},
                                {{2.4, 6.0, {1.15, 1.61, 2.17}}, 0.04, 8.7, 3.2, 4.2, 0.13},
                                {{2.0, 6.0, {1.08, 1.77, 2.66}}, 0.12, 11.1, 1.4, 6.6, 0.20},
                                {{3.2, 6.0, {2.73, 3.12, 4.68}}, 0.25, 14.8, 2.5, 8.9, 0.17}};
    static const Kind f64[2] = {{{3.3, 6.0, {0.85, 1.47, 2.21}}, 0.20, 5.7, 1.6, 2.6, 0.19},
                                {{3.3, 6.0, {1.65, 2.45, 3.68}}, 0.07, 8.6, 1.8, 4.4, 0.11}};
    if (sizeof(T) == 4) return f32[(comps - 1) * 2 + noise];
    return f64[noise];
}
constexpr int kTileW = 32;  // the tile kernels' tiles (go_general, go_tetm_fused)
template <typename T>
constexpr int kTileH = sizeof(T) == 4 ? 16 : 8;

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
    const int strips = (P.N_c + kMarchOut - 1) / kMarchOut;
    const std::array<int, 4> plan = {P.N_r, P.N_c, per_sm, sm_count};
    if (plan != plan_) {
        const Kind& k = kind_of<T>(COMPS, v.noise);
        const int inputs = v.nv + v.nq;
        MarchCost cost = k.march;
        // (periodic images, FP64 odd widths: 29.7 us a launch at 64 x 4096, 32.4 at 63)
        for (double& c : cost.step) c *= (1.0 + k.march_input * inputs) * (v.img ? 1.09 : 1.0);
        const MarchSegments seg = march_segments(
            P.N_r, [&](int L) { return (long long)strips * ((P.N_r + L - 1) / L); }, per_sm, sm_count, cost);
        const long long tiles = (long long)((P.N_c + kTileW - 1) / kTileW) * ((P.N_r + kTileH<T> - 1) / kTileH<T>);
        const double tile_us = std::max(k.one, k.first + k.round * (double)((tiles + sm_count - 1) / sm_count));
        plan_rows_ = forced_ == 1 || seg.us < tile_us * (1.0 + k.tile_input * inputs) ? seg.rows : 0;
        plan_ = plan;
    }
    if (!plan_rows_) return false;
    MarchGeneralParams<T, COMPS> G;
    for (int s = 0; s < 4; ++s) G.st[s] = st[s];
    for (int q = 0; q < COMPS; ++q) {
        G.psi0[q] = psi0[q];
        G.n0[q] = n0[q];
        G.psi1[q] = psi1[q];
        G.n1[q] = n1[q];
    }
    G.strips = strips;
    G.seg_rows = plan_rows_;
    G.n_items = G.strips * ((P.N_r + G.seg_rows - 1) / G.seg_rows);
    march_launch(kern, G, G.n_items, bytes, stream, pdl);
    return true;
}

template <typename T>
bool MarchGeneral<T>::launch(const TetmParams<T> (&st)[4], int comps, bool res, const cx<T>* const* psi0, const T* const* n0,
                             cx<T>* const* psi1, T* const* n1, int sm_count, cudaStream_t stream, bool pdl) {
    if (forced_ == 0) return false;
    const StageParams<T>& P = st[0].p;
    // 32-bit indices over every group's planes; a reservoir with its pump; real
    // potential coefficients
    const int groups = std::max({1, P.n_pump, P.n_pot, P.n_pulse});
    bool takes = res && P.n_pump >= 1 && P.plane * groups < (1LL << 31);
    for (int s = 0; s < 4; ++s)
        for (int g = 0; g < P.n_pot; ++g) takes = takes && st[s].p.pot_c[g].im == (T)0;
    bool done = false;
    if (takes && comps == 1) done = launch_comps<1>(st, psi0, n0, psi1, n1, sm_count, stream, pdl);
    // FP64: two polarisations' rows do not fit the registers
    if constexpr (sizeof(T) == 4) {
        if (takes && comps == 2) done = launch_comps<2>(st, psi0, n0, psi1, n1, sm_count, stream, pdl);
    }
    if (!done && forced_ == 1) fail(PHX_ERR_UNSUPPORTED, "no marching kernel takes this iteration (PHX_GENERAL_MARCH=1)");
    return done;
}

template class MarchGeneral<float>;
template class MarchGeneral<double>;

}  // namespace phx
