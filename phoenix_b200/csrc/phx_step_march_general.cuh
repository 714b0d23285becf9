// Marching warps (phx_step_march.cuh) for what the plain scalar iteration does
// not take: the TE/TM spinor, a second pump group, pulses, time-dependent
// envelopes beside them, and noise.  The same walk: stage s of a warp's strip
// on row t - s, windows and accumulators in registers, neighbours (for the
// spinor the diagonal ones too) by shuffles, inputs in a shared ring per warp.
//
// The numbers of groups, the noise and the kind of the potential's coefficient
// are template parameters, so a step is one straight run of instructions; the
// host takes the kernel where a variant and its ring fit and it is the faster one
// (phx_march_general.cu), and the tile kernels (phx_step_tetm_fused.cuh) elsewhere.
//
// The noise value of a point and its scale are drawn once, when the first
// stage meets the row, and kept in the ring for the other three.
//
// Per point the operations are rhs_scalar_src's / rhs_tetm_src's and the kRk4*
// sums of the stage kernels, in the same order: bit-identical results, but for the
// sign of an exact zero and for divisions by dV outside div_known's range (FP32
// dividends below 2^-100: their last bit).  A value that is not finite in the
// stage kernels is not finite here; it may be infinite where theirs is NaN
// (ScalarGlobalSrc::real_pot).
#pragma once

#include "phx_stage_tetm.cuh"
#include "phx_step_march.cuh"

namespace phx {

template <typename T, int COMPS>
struct MarchGeneralParams {
    TetmParams<T> st[4];       // stage s: coefficients, b, dtw, w_sum, input planes (scalar model: .p only)
    const cx<T>* psi0[COMPS];  // state in and out, [component]
    const T* n0[COMPS];
    cx<T>* psi1[COMPS];
    T* n1[COMPS];
    int strips, seg_rows, n_items;
};

// A warp's ring row: per lane 16-byte pieces 512 bytes apart, two points' psi
// and pulses of every component, the noise values, then the reals (pairs; two
// pairs to a piece in FP32): n, pump groups, potential groups, noise scale.
template <typename T, int COMPS, int NP, int NV, int NQ, bool NOISE>
struct MarchGeneralLayout {
    static constexpr int cx_bytes = 4 * (int)sizeof(T) * 32, per = sizeof(T) == 4 ? 2 : 1;
    static constexpr int psi_off(int q) { return q * cx_bytes; }
    static constexpr int pulse_off(int g, int q) { return (COMPS + g * COMPS + q) * cx_bytes; }
    static constexpr int xi_off = COMPS * (1 + NQ) * cx_bytes;
    static constexpr int reals_off = xi_off + (NOISE ? cx_bytes : 0);
    static constexpr int real_off(int slot) { return reals_off + slot / per * 512 + slot % per * 8; }
    static constexpr int n_slot(int q) { return q; }
    static constexpr int pump_slot(int g, int q) { return COMPS * (1 + g) + q; }
    static constexpr int pot_slot(int g, int q) { return COMPS * (1 + NP + g) + q; }
    static constexpr int scale_slot = COMPS * (1 + NP + NV);
    static constexpr int slots = scale_slot + (NOISE ? 1 : 0);
    static constexpr int row_bytes = reals_off + (slots + per - 1) / per * 512;
    static constexpr int warp_bytes = kMarchRing * row_bytes;
    static constexpr int bytes = kMarchWarps * warp_bytes;
};

// the pointwise inputs of one point, from the lane's registers
template <typename T, int COMPS, int NP, int NV, int NQ, bool NOISE, bool REALV>
struct MarchSrc {
    const T (&pu)[NP > 0 ? NP : 1][COMPS][2];
    const T (&po)[NV > 0 ? NV : 1][COMPS][2];
    const cx<T> (&ps)[NQ > 0 ? NQ : 1][COMPS][2];
    int j;
    static __device__ __forceinline__ constexpr int n_pump() { return NP; }
    static __device__ __forceinline__ constexpr int n_pot() { return NV; }
    static __device__ __forceinline__ constexpr int n_pulse() { return NQ; }
    static __device__ __forceinline__ constexpr bool noise() { return NOISE; }
    static __device__ __forceinline__ constexpr bool real_pot() { return REALV; }
    // the drift of an infinite psi is taken from the infinity of its |psi|^2, the
    // reservoir's gain from an infinite n added to the opposite infinity of its
    // loss: NaN whatever the quotient
    static __device__ __forceinline__ T over_dV(const StageParams<T>& S, T x) { return div_known_finite(x, S.dV, S.inv_dV); }
    __device__ __forceinline__ T pump(int c, int g) const { return pu[g][c][j]; }
    __device__ __forceinline__ T pot(int c, int g) const { return po[g][c][j]; }
    __device__ __forceinline__ cx<T> pulse(int c, int g) const { return ps[g][c][j]; }
    __device__ __forceinline__ T pump(int g) const { return pu[g][0][j]; }
    __device__ __forceinline__ T pot(int g) const { return po[g][0][j]; }
    __device__ __forceinline__ cx<T> pulse(int g) const { return ps[g][0][j]; }
};

template <typename T, int COMPS, int NP, int NV, int NQ, bool NOISE, bool REALV, bool IMG, int MINB>
__global__ void __launch_bounds__(32 * kMarchWarps, MINB)
    rk4_march_general_kernel(const __grid_constant__ MarchGeneralParams<T, COMPS> F) {
    using Lay = MarchGeneralLayout<T, COMPS, NP, NV, NQ, NOISE>;
    using C = cx<T>;
    constexpr int CPT = 2;
    constexpr int PB = 4 * (int)sizeof(T), RB = 2 * (int)sizeof(T);
    extern __shared__ __align__(16) unsigned char march_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, item = blockIdx.x * kMarchWarps + warp;
    if (item >= F.n_items) return;
    const StageParams<T>& P0 = F.st[0].p;
    const int N_r = P0.N_r, N_c = P0.N_c, pitch = (int)P0.pitch, plane = (int)P0.plane;
    const int strip = item % F.strips, R0 = item / F.strips * F.seg_rows, R1 = min(R0 + F.seg_rows, N_r);
    const int c = strip * kMarchOut - 4 + CPT * lane;
    unsigned char* const mine = march_smem + warp * Lay::warp_bytes + lane * 16;
    const unsigned s_mine = (unsigned)__cvta_generic_to_shared(mine);

    // rows are counted from k = 0 at R0 - 4: step k evaluates stage s (0-based) on row k - s
    const int last_k = R1 - R0 + 7;
    const bool wrap_x = !IMG && P0.img_x, wrap_y = !IMG && P0.img_y;  // march_segment's IMG
    int next_k = 0, next_r = R0 - 4;
    if (wrap_y && next_r < 0) next_r += N_r;
    int next_g = next_r * pitch + (wrap_x ? (c % N_c + N_c) % N_c : min(c, (N_c + 8 - CPT) & ~(CPT - 1)));
    auto copy_cx = [&](unsigned d, const C* p) __attribute__((always_inline)) {
#pragma unroll
        for (int i = 0; i < PB / 16; ++i) cp_async<16>(d + i * 512, reinterpret_cast<const unsigned char*>(p + next_g) + i * 16);
    };
    auto issue = [&]() __attribute__((always_inline)) {
        const unsigned d = s_mine + (unsigned)(next_k & (kMarchRing - 1)) * Lay::row_bytes;
#pragma unroll
        for (int q = 0; q < COMPS; ++q) {
            copy_cx(d + Lay::psi_off(q), F.psi0[q]);
            cp_async<RB>(d + Lay::real_off(Lay::n_slot(q)), F.n0[q] + next_g);
#pragma unroll
            for (int g = 0; g < NP; ++g)
                cp_async<RB>(d + Lay::real_off(Lay::pump_slot(g, q)), (q ? F.st[0].pump : P0.pump) + next_g + g * plane);
#pragma unroll
            for (int g = 0; g < NV; ++g)
                cp_async<RB>(d + Lay::real_off(Lay::pot_slot(g, q)), (q ? F.st[0].pot : P0.pot) + next_g + g * plane);
#pragma unroll
            for (int g = 0; g < NQ; ++g) copy_cx(d + Lay::pulse_off(g, q), (q ? F.st[0].pulse : P0.pulse) + g * plane);
        }
        cp_async_commit();
        ++next_k;
        ++next_r;
        next_g += pitch;
        if (wrap_y && next_r == N_r) next_r = 0, next_g -= N_r * pitch;
    };
    pdl_wait();  // the previous iteration's kernel has completed
#pragma unroll
    for (int k = 0; k < 5; ++k) issue();

    const bool store_lane = c >= strip * kMarchOut && c < (strip + 1) * kMarchOut && c < N_c;
    const bool store_two = sizeof(T) == 4 || c + 2 <= N_c;
    const bool edge_strip = P0.img_x && (strip == 0 || (strip + 1) * kMarchOut > N_c - kImgDepth);
    auto put = [&](int q, int row, const C* v, const T* nv) __attribute__((always_inline)) {
        C* const out = F.psi1[q];
        T* const out_n = F.n1[q];
        const int g = row * pitch + c;
        auto put_at = [&](int gi) __attribute__((always_inline)) {
            if (store_two) {
                st_two(out + gi, v);
                st_two(out_n + gi, nv);
            } else {
                out[gi] = v[0];
                out_n[gi] = nv[0];
            }
        };
        if (store_lane && row >= R0) put_at(g);
        if constexpr (!IMG) return;
        if (row < R0) return;
        if (edge_strip || (P0.img_y && (row < kImgDepth || row >= N_r - kImgDepth))) {
            const int dy = !P0.img_y ? 0 : (row < kImgDepth ? N_r : (row >= N_r - kImgDepth ? -N_r : 0));
            if (store_lane && dy) put_at(g + dy * pitch);
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                const int dx = !P0.img_x ? 0 : (c + j < kImgDepth ? N_c : (c + j >= N_c - kImgDepth ? -N_c : 0));
                if (store_lane && dx != 0 && c + j < N_c) {
                    const int gi = g + j + dx;
                    out[gi] = v[j];
                    out_n[gi] = nv[j];
                    if (dy) {
                        out[gi + dy * pitch] = v[j];
                        out_n[gi + dy * pitch] = nv[j];
                    }
                }
            }
        }
    };

    C up[4][COMPS][CPT], ce[4][COMPS][CPT];    // stage inputs: the row above, and the row, that the stage evaluates next
    C a[3][COMPS][CPT];                        // stage s to stage s + 1: accumulators of one row,
    T an[3][COMPS][CPT], ns[3][COMPS][CPT];    // the reservoirs', and their stage values
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int q = 0; q < COMPS; ++q)
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                up[s][q][j] = ce[s][q][j] = mk((T)0, (T)0);
                if (s < 3) a[s][q][j] = mk((T)0, (T)0), an[s][q][j] = ns[s][q][j] = (T)0;
            }
    auto row_of = [&](int k) { return mine + (k & (kMarchRing - 1)) * Lay::row_bytes; };
    cp_async_wait<3>();  // rows 0 and 1
#pragma unroll
    for (int q = 0; q < COMPS; ++q) {
        ring_two(row_of(0) + Lay::psi_off(q), up[0][q]);
        ring_two(row_of(1) + Lay::psi_off(q), ce[0][q]);
    }

    // sqrt((R n + gamma_c) / (4 dV)); the reciprocal of 4 dV is that of dV over 4
    auto scale_of = [](const StageParams<T>& P, T n) {
        return rsqrt_rn(div_known(radd(rmul(P.R, n), P.gamma_c), P.four_dV, (T)0.25 * P.inv_dV));
    };
    C dn[COMPS][CPT], pa[COMPS][CPT];  // the row the stage before has just made, and what it hands on with it
    T pan[COMPS][CPT], pn[COMPS][CPT];
    auto stage = [&](auto st, int k) __attribute__((always_inline)) {
        constexpr int s = decltype(st)::value, before = s > 0 ? s - 1 : 0;
        const TetmParams<T>& Q = F.st[s];
        const StageParams<T>& P = Q.p;
        unsigned char* const ro = row_of(k - s);
        C y0[COMPS][CPT], kw[COMPS][CPT], ps[NQ > 0 ? NQ : 1][COMPS][CPT], xi[CPT];
        T n0[COMPS][CPT], kn[COMPS][CPT], pu[NP > 0 ? NP : 1][COMPS][CPT], po[NV > 0 ? NV : 1][COMPS][CPT], sc[CPT];
#pragma unroll
        for (int q = 0; q < COMPS; ++q) {
            if constexpr (s > 0) ring_two(ro + Lay::psi_off(q), y0[q]);
            ring_two(ro + Lay::real_off(Lay::n_slot(q)), n0[q]);
#pragma unroll
            for (int g = 0; g < NP; ++g) ring_two(ro + Lay::real_off(Lay::pump_slot(g, q)), pu[g][q]);
#pragma unroll
            for (int g = 0; g < NV; ++g) ring_two(ro + Lay::real_off(Lay::pot_slot(g, q)), po[g][q]);
#pragma unroll
            for (int g = 0; g < NQ; ++g) ring_two(ro + Lay::pulse_off(g, q), ps[g][q]);
        }
        const int row = R0 - 4 + k - s;
        if constexpr (NOISE) {
            if constexpr (s == 0) {
#pragma unroll
                for (int j = 0; j < CPT; ++j) {
                    xi[j] = stage_xi(P, row, c + j);
                    sc[j] = scale_of(P, n0[0][j]);
                    if constexpr (sizeof(T) == 4) {
                        reinterpret_cast<C*>(ro + Lay::xi_off)[j] = xi[j];
                    } else {
                        *reinterpret_cast<C*>(ro + Lay::xi_off + j * 512) = xi[j];
                    }
                    reinterpret_cast<T*>(ro + Lay::real_off(Lay::scale_slot))[j] = sc[j];
                }
            } else {
                ring_two(ro + Lay::xi_off, xi);
                ring_two(ro + Lay::real_off(Lay::scale_slot), sc);
            }
        }
        C lf[COMPS], rt[COMPS];
#pragma unroll
        for (int q = 0; q < COMPS; ++q) lf[q] = shfl_up1(ce[s][q][1]), rt[q] = shfl_dn1(ce[s][q][0]);
        if constexpr (COMPS == 1) {
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                if constexpr (s == 0) y0[0][j] = ce[0][0][j];
                const T nin = s == 0 ? n0[0][j] : ns[before][0][j];
                kn[0][j] = (T)0;
                const MarchSrc<T, COMPS, NP, NV, NQ, NOISE, REALV> src{pu, po, ps, j};
                rhs_scalar_src<T, true>(P, src, ce[s][0][j], up[s][0][j], dn[0][j], j == 0 ? lf[0] : ce[s][0][0],
                                       j == 0 ? ce[s][0][1] : rt[0], nin, kw[0][j], kn[0][j]);
            }
        } else {
            constexpr int m = COMPS - 1;
            const C ulp = shfl_up1(up[s][0][1]), urp = shfl_dn1(up[s][0][0]), dlp = shfl_up1(dn[0][1]), drp = shfl_dn1(dn[0][0]);
            const C ulm = shfl_up1(up[s][m][1]), urm = shfl_dn1(up[s][m][0]), dlm = shfl_up1(dn[m][1]), drm = shfl_dn1(dn[m][0]);
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                if constexpr (s == 0) y0[0][j] = ce[0][0][j], y0[m][j] = ce[0][m][j];
                const T np = s == 0 ? n0[0][j] : ns[before][0][j], nm = s == 0 ? n0[m][j] : ns[before][m][j];
                const MarchSrc<T, COMPS, NP, NV, NQ, NOISE, REALV> src{pu, po, ps, j};
                rhs_tetm_src<T>(Q, src, ce[s][0][j], up[s][0][j], dn[0][j], j == 0 ? lf[0] : ce[s][0][0],
                                j == 0 ? ce[s][0][1] : rt[0], j == 0 ? ulp : up[s][0][0], j == 0 ? up[s][0][1] : urp,
                                j == 0 ? dlp : dn[0][0], j == 0 ? dn[0][1] : drp, ce[s][m][j], up[s][m][j], dn[m][j],
                                j == 0 ? lf[m] : ce[s][m][0], j == 0 ? ce[s][m][1] : rt[m], j == 0 ? ulm : up[s][m][0],
                                j == 0 ? up[s][m][1] : urm, j == 0 ? dlm : dn[m][0], j == 0 ? dn[m][1] : drm, np, nm, kw[0][j],
                                kn[0][j], kw[m][j], kn[m][j]);
            }
        }
        C o[COMPS][CPT];
        T on[COMPS][CPT];
#pragma unroll
        for (int q = 0; q < COMPS; ++q)
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                up[s][q][j] = ce[s][q][j];
                ce[s][q][j] = dn[q][j];
                C t = mk((T)0, (T)0);
                T tn = (T)0;
                on[q][j] = (T)0;
                // the kRk4First / kRk4Mid / kRk4Last sums of the stage kernels
                if constexpr (s == 0) {
                    t = smul(P.b, kw[q][j]);
                    tn = rmul(P.b, kn[q][j]);
                } else if constexpr (s < 3) {
                    t = cadd(a[before][q][j], smul(P.b, kw[q][j]));
                    tn = radd(an[before][q][j], rmul(P.b, kn[q][j]));
                }
                if constexpr (s < 3) {
                    o[q][j] = cadd(y0[q][j], smul(P.dtw, kw[q][j]));
                    on[q][j] = radd(n0[q][j], rmul(P.dtw, kn[q][j]));
                } else {
                    o[q][j] = cadd(y0[q][j], smul(P.dt, cadd(a[2][q][j], smul(P.b, kw[q][j]))));
                    on[q][j] = radd(n0[q][j], rmul(P.dt, radd(an[2][q][j], rmul(P.b, kn[q][j]))));
                }
                if constexpr (NOISE) {
                    // one noise value for both polarisations, scaled by the plus
                    // reservoir; the last sum sees the updated n+ for psi-
                    const T z = s == 3 && q == 1
                                    ? scale_of(P, on[0][j]) : sc[j];
                    o[q][j] = cadd(o[q][j], mk(rmul(rmul(P.w_sum, xi[j].re), z), rmul(rmul(P.w_sum, xi[j].im), z)));
                }
                if constexpr (s > 0)
                    a[before][q][j] = pa[q][j], an[before][q][j] = pan[q][j], ns[before][q][j] = pn[q][j];
                pa[q][j] = t, pan[q][j] = tn, pn[q][j] = on[q][j];
                dn[q][j] = o[q][j];
            }
        if constexpr (s == 3) {
            // a segment's first steps make no row of its own yet (put)
#pragma unroll
            for (int q = 0; q < COMPS; ++q) put(q, row, o[q], on[q]);
        }
    };
    // Every step runs all four stages: in a segment's first six steps the later
    // ones work on rows that are not there yet and store nothing (4 % more work
    // on segments of 64 rows; separate first steps, as the scalar kernel has
    // them, would double the code, which the instruction cache does not hold).
#pragma unroll 1
    for (int k = 1; k < last_k; ++k) {
        issue();             // row k + 4, into the slot of row k - 4, which step k - 1 read last
        cp_async_wait<3>();  // rows up to k + 1 are there
#pragma unroll
        for (int q = 0; q < COMPS; ++q) ring_two(row_of(k + 1) + Lay::psi_off(q), dn[q]);
        stage(std::integral_constant<int, 0>{}, k);
        stage(std::integral_constant<int, 1>{}, k);
        stage(std::integral_constant<int, 2>{}, k);
        stage(std::integral_constant<int, 3>{}, k);
    }
    cp_async_wait<0>();  // no copy may land after the CTA's shared memory has gone to another
}

}  // namespace phx
