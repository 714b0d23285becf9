// Launcher of the marching-warps RK4 iteration (phx_step_march.cuh), compiled
// in its own unit (phx_march.cu).
#pragma once

#include <array>
#include <cstdlib>
#include <map>
#include <vector>

#include "phx_adjoint.cuh"
#include "phx_rt.hpp"
#include "phx_stage_tetm.cuh"

namespace phx {

// whether the marching iterations read and write the periodic images in the
// planes' rings: only where column pairs cannot wrap around the grid
inline bool march_needs_images(int N_c, int periodic_x) { return periodic_x && N_c % 2 != 0; }

struct MarchOptions {
    bool res = true;     // reservoir
    bool fma = false;    // fused multiply-add arithmetic (FP32)
    bool store = false;  // also write the stage values (FusedParams::st_psi / st_n)
    bool img = false;    // read and write periodic images (march_needs_images, or another reader needs them)
    bool pdl = true;     // programmatic stream serialization
};

template <typename T>
class MarchLauncher {
public:
    // planes of `plane` points can be indexed in 32 bits
    static bool fits(long long plane) { return plane < (1LL << 31); }
    // one iteration F.psi0, F.n0 -> F.psi1, F.n1 on `stream` of the current device
    void launch(const FusedParams<T>& F, const MarchOptions& o, int sm_count, cudaStream_t stream);

private:
    std::map<const void*, int> per_sm_;  // CTAs per SM of the kernel variants used so far
    std::array<int, 4> plan_{};          // grid, CTAs per SM and SMs of the last row segmentation
    int plan_rows_ = 0;
};

// The same iteration over every instance of a batch, in one launch.
template <typename T>
class MarchBatch {
public:
    // f: two directions per instance (constant envelopes); waits for the copies
    void build(const std::vector<FusedParams<T>>& f, bool res, bool fma, int sm_count, cudaStream_t stream);
    void launch(int dir, cudaStream_t stream) const;
    // whether the launches read and write periodic images (march_needs_images)
    bool images() const { return images_; }

private:
    bool images_ = false;
    DevBuf f_, items_;
    const void* kern_ = nullptr;
    int n_items_ = 0;
};

// The iteration with noise, pulses, a second pump group or two polarisations
// (phx_step_march_general.cuh, compiled in phx_march_general.cu).
template <typename T>
class MarchGeneral {
public:
    // st: the parameters of the four stages (scalar model: .p only); state
    // planes per component.  False when no variant takes this iteration or the
    // tile kernels are the faster ones for the grid.
    bool launch(const TetmParams<T> (&st)[4], int comps, bool res, const cx<T>* const* psi0, const T* const* n0,
                cx<T>* const* psi1, T* const* n1, int sm_count, cudaStream_t stream, bool pdl);

private:
    template <int COMPS>
    bool launch_comps(const TetmParams<T> (&st)[4], const cx<T>* const* psi0, const T* const* n0, cx<T>* const* psi1,
                      T* const* n1, int sm_count, cudaStream_t stream, bool pdl);
    std::map<const void*, int> per_sm_;  // CTAs per SM of the kernel variants used so far
    std::array<int, 4> plan_{};          // grid, CTAs per SM and SMs of the last row segmentation
    int plan_rows_ = 0;                  // 0: the tile kernel
    // PHX_GENERAL_MARCH: 1 the marching kernel on every grid (an error where no
    // variant takes the iteration), 0 never; otherwise the faster of the two
    int forced_ = [] {
        const char* e = std::getenv("PHX_GENERAL_MARCH");
        return e && (e[0] == '0' || e[0] == '1') ? e[0] - '0' : -1;
    }();
};

// The adjoint's four vector-Jacobian stages of one iteration
// (phx_adjoint_march.cuh, compiled in phx_adjoint_march.cu); planes as
// MarchLauncher::fits.
template <typename T>
class AdjMarch {
public:
    // whether the kernel wraps around the grid itself, so that neither the stage
    // values nor lam' need periodic images
    static bool wraps(int N_c) { return N_c % 2 == 0; }
    void launch(const AdjFusedParams<T>& Q, int sm_count, cudaStream_t stream, bool pdl);

private:
    std::map<const void*, int> per_sm_;  // CTAs per SM of the kernel variants used so far
    std::array<int, 4> plan_{};          // grid, CTAs per SM and SMs of the last row segmentation
    int plan_rows_ = 0;
};

extern template class AdjMarch<float>;
extern template class AdjMarch<double>;
extern template class MarchGeneral<float>;
extern template class MarchGeneral<double>;
extern template class MarchBatch<float>;
extern template class MarchBatch<double>;
extern template class MarchLauncher<float>;
extern template class MarchLauncher<double>;

}  // namespace phx
