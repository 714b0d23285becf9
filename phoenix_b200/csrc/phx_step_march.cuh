// The whole RK4 iteration (RungeKutta4::step,
// source/cuda_solver/solver/iterator/runge_kutta.cu:74-94) as independent warps
// that march down the grid: no CTA barrier, no shared stencil tile.
//
// A warp owns a strip of 64 columns (two neighbouring points per lane) and a
// segment of rows.  At step t it evaluates stage 1 on row t, stage 2 on
// row t - 1, stage 3 on row t - 2 and stage 4 on row t - 3.  Every stage's
// vertical neighbours are the two rows it saw before, kept in registers, and
// the row the stage before it has just made; horizontal neighbours come from
// the lanes beside it by shuffles.  The accumulators and stage reservoirs
// pass from stage to stage in registers as well.  Only the inputs (psi, n,
// pump, potential of the last five rows) go through shared memory: a ring of
// eight rows per warp, filled by cp.async four rows ahead, in which every lane
// reads nothing but what it copied itself.
//
// The strip loses one column a side and stage, so 56 of its columns are stored;
// a segment of L rows evaluates L + 6, L + 4, L + 2 and L rows.
// (FP32 155, FP64 250 registers; four points per lane lost to the longer code.)
//
// Why: the tile kernels spend their time on stage barriers, on the stencil's
// shared-memory traffic (70 % of that pipe) and on idle lanes in the
// shrinking stage regions.  Here a stage of one row costs its arithmetic, 4
// shuffles and 4 shared-memory reads, and consecutive stages hang together
// only by the row just made, so one warp alone has enough independent
// instructions to keep a scheduler busy.
//
// The arithmetic of a point is rhs_iter's and the RK4 sums' of
// rk4_fused_kernel, in the same order (bit-identical results).
#pragma once

#include <type_traits>

#include "phx_step_fused.cuh"

namespace phx {

template <typename T>
struct MarchParams {
    FusedParams<T> f;
    int strips, seg_rows, n_items;  // n_items = strips * segments
};

constexpr int kMarchWarps = 4;  // warps per CTA: one per scheduler of the SM
constexpr int kMarchRing = 8;   // rows t - 3 .. t + 4
constexpr int kMarchCols = 64;  // columns a warp evaluates, two per lane
constexpr int kMarchOut = kMarchCols - 8;  // columns it stores

// One ring row of a warp, in pieces of 512 bytes of which every lane owns 16 (so
// that one address serves all of a lane's values, and its accesses and its
// neighbours' fall on consecutive banks): psi, then n, pump and potential; in
// FP32 n and pump share a piece.
template <typename T>
struct MarchLayout {
    static constexpr int PB = 4 * (int)sizeof(T), RB = 2 * (int)sizeof(T);  // a lane's bytes of psi / of a real
    static constexpr int n_off = PB * 32;
    static constexpr int pump_off = n_off + (RB == 8 ? 8 : 512);
    static constexpr int pot_off = n_off + (RB == 8 ? 512 : 1024);
    static constexpr int row_bytes = pot_off + 512;
    static constexpr int warp_bytes = kMarchRing * row_bytes;
    static constexpr int bytes = kMarchWarps * warp_bytes;
};

template <int N>
__device__ __forceinline__ void cp_async(unsigned dst, const void* src) {
    if constexpr (N == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// a lane's two points / reals into global memory (aligned to their size, at
// most 16 bytes a store), and from its pieces of the ring
__device__ __forceinline__ void st_two(cx<float>* p, const cx<float>* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0].re, v[0].im, v[1].re, v[1].im);
}
__device__ __forceinline__ void st_two(cx<double>* p, const cx<double>* v) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0].re, v[0].im);
    *reinterpret_cast<double2*>(p + 1) = make_double2(v[1].re, v[1].im);
}
__device__ __forceinline__ void st_two(float* p, const float* v) { *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]); }
__device__ __forceinline__ void st_two(double* p, const double* v) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void ring_two(const unsigned char* p, cx<float>* v) {
    const float4 u = *reinterpret_cast<const float4*>(p);
    v[0] = mk(u.x, u.y), v[1] = mk(u.z, u.w);
}
__device__ __forceinline__ void ring_two(const unsigned char* p, cx<double>* v) {
    const double2 u = *reinterpret_cast<const double2*>(p), w = *reinterpret_cast<const double2*>(p + 512);
    v[0] = mk(u.x, u.y), v[1] = mk(w.x, w.y);
}
__device__ __forceinline__ void ring_two(const unsigned char* p, float* v) {
    const float2 u = *reinterpret_cast<const float2*>(p);
    v[0] = u.x, v[1] = u.y;
}
__device__ __forceinline__ void ring_two(const unsigned char* p, double* v) {
    const double2 u = *reinterpret_cast<const double2*>(p);
    v[0] = u.x, v[1] = u.y;
}

// One warp's segment: rows [R0, R1) of strip `strip`; `ring` is the warp's
// shared memory.
// POT: there is a potential (where there is none its terms are not evaluated: 0
// times an infinite psi would not be zero).
// UNIT: every temporal coefficient is exactly 1 (constant envelopes); the
// products with it, which change nothing, are left out.  STORE: also write
// the stage values Y2..Y4 of the stored points, which the adjoint's backward
// sweep reads.  IMG: read the periodic images in the planes' rings and write
// them for what is stored.  Without it (an even number of columns, or walls in
// x) rows and column pairs wrap as they are copied, no image is read or
// written, and a step has no branch left (FP32, us per iteration at 1024^2 /
// 4096^2: 18.6 / 216 with, 16.2 / 184 without).  Plane indices are 32-bit (the
// host takes this kernel for planes of fewer than 2^31 points only).
template <typename T, bool RES, bool POT, bool UNIT, bool FMA, bool STORE, bool IMG>
__device__ __forceinline__ void march_segment(const FusedParams<T>& P, int strip, int R0, int R1, unsigned char* ring) {
    using Lay = MarchLayout<T>;
    using C = cx<T>;
    constexpr int CPT = 2;
    // the RK4 weights (FusedParams::b)
    constexpr T wb[4] = {(T)(1.0 / 6.0), (T)(1.0 / 3.0), (T)(1.0 / 3.0), (T)(1.0 / 6.0)};
    const int lane = threadIdx.x & 31;
    const int c = strip * kMarchOut - 4 + CPT * lane;
    const int pitch = (int)P.pitch;
    const bool has_pump = RES && P.pump != nullptr;
    unsigned char* const mine = ring + lane * 16;
    if (RES && !has_pump) {  // an absent pump counts as zero
        for (int k = 0; k < kMarchRing; ++k)
#pragma unroll
            for (int j = 0; j < CPT; ++j) reinterpret_cast<T*>(mine + k * Lay::row_bytes + Lay::pump_off)[j] = (T)0;
    }

    // rows are counted from k = 0 at R0 - 4: step k evaluates stage s (0-based)
    // on row k - s.  Copies run ahead to row R1 + 6, within the planes' rings of
    // 8.  Lanes past the ring read its last columns: columns beyond N_c + 3 go
    // wrong, which nothing stored depends on
    const int last_k = R1 - R0 + 7;
    const bool wrap_x = !IMG && P.img_x, wrap_y = !IMG && P.img_y;
    int next_k = 0, next_r = R0 - 4;  // the next row to copy
    if (wrap_y && next_r < 0) next_r += P.N_r;
    int next_g = next_r * pitch + (wrap_x ? (c % P.N_c + P.N_c) % P.N_c : min(c, (P.N_c + 8 - CPT) & ~(CPT - 1)));
    const unsigned s_mine = (unsigned)__cvta_generic_to_shared(mine);
    auto issue = [&]() __attribute__((always_inline)) {
        const unsigned d = s_mine + (unsigned)(next_k & (kMarchRing - 1)) * Lay::row_bytes;
#pragma unroll
        for (int i = 0; i < Lay::PB / 16; ++i)
            cp_async<16>(d + i * 512, reinterpret_cast<const unsigned char*>(P.psi0 + next_g) + i * 16);
        if constexpr (RES) {
            cp_async<Lay::RB>(d + Lay::n_off, P.n0 + next_g);
            if (has_pump) cp_async<Lay::RB>(d + Lay::pump_off, P.pump + next_g);
        }
        if constexpr (POT) cp_async<Lay::RB>(d + Lay::pot_off, P.pot + next_g);
        cp_async_commit();
        ++next_k;
        ++next_r;
        next_g += pitch;
        if (wrap_y && next_r == P.N_r) next_r = 0, next_g -= P.N_r * pitch;
    };
#pragma unroll
    for (int k = 0; k < 5; ++k) issue();

    const bool store_lane = c >= strip * kMarchOut && c < (strip + 1) * kMarchOut && c < P.N_c;
    const bool store_two = sizeof(T) == 4 || c + 2 <= P.N_c;  // FP32 grids have an even number of columns
    auto put_at = [&](C* out, T* out_n, int g, const C* v, const T* nv) __attribute__((always_inline)) {
        if (store_two) {
            st_two(out + g, v);
            if constexpr (RES) st_two(out_n + g, nv);
        } else {
            out[g] = v[0];
            if constexpr (RES) out_n[g] = nv[0];
        }
    };
    const bool edge_strip = P.img_x && (strip == 0 || (strip + 1) * kMarchOut > P.N_c - kImg);
    auto put = [&](C* out, T* out_n, int row, const C* v, const T* nv) __attribute__((always_inline)) {
        const int g = row * pitch + c;
        if (store_lane) put_at(out, out_n, g, v, nv);
        if constexpr (!IMG) return;
        if (edge_strip || (P.img_y && (row < kImg || row >= P.N_r - kImg))) {
            const int dy = !P.img_y ? 0 : (row < kImg ? P.N_r : (row >= P.N_r - kImg ? -P.N_r : 0));
            if (store_lane && dy) put_at(out, out_n, g + dy * pitch, v, nv);
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                const int dx = !P.img_x ? 0 : (c + j < kImg ? P.N_c : (c + j >= P.N_c - kImg ? -P.N_c : 0));
                if (store_lane && dx != 0 && c + j < P.N_c) {
                    const int gi = g + j + dx;
                    out[gi] = v[j];
                    if constexpr (RES) out_n[gi] = nv[j];
                    if (dy) {
                        out[gi + dy * pitch] = v[j];
                        if constexpr (RES) out_n[gi + dy * pitch] = nv[j];
                    }
                }
            }
        }
    };

    C up[4][CPT], ce[4][CPT];  // stage inputs: the row above, and the row, that the stage evaluates next
    C a[3][CPT];               // stage s to stage s + 1: accumulators of one row,
    T an[3][CPT], ns[3][CPT];  // the reservoir's, and its stage value
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int j = 0; j < CPT; ++j) {
            up[s][j] = ce[s][j] = mk((T)0, (T)0);
            if (s < 3) a[s][j] = mk((T)0, (T)0), an[s][j] = ns[s][j] = (T)0;
        }
    auto row_of = [&](int k) { return mine + (k & (kMarchRing - 1)) * Lay::row_bytes; };
    cp_async_wait<3>();  // rows 0 and 1
    ring_two(row_of(0), up[0]);
    ring_two(row_of(1), ce[0]);

    C dn[CPT], pa[CPT];  // the row the stage before has just made, and what it hands on with it
    T pan[CPT], pn[CPT];
    auto stage = [&](auto st, int k) __attribute__((always_inline)) {
        constexpr int s = decltype(st)::value, before = s > 0 ? s - 1 : 0, own = s < 3 ? s : 0;
        const unsigned char* const ro = row_of(k - s);
        C y0[CPT], kw[CPT], o[CPT];
        T n0[CPT], pu[CPT], po[CPT], kn[CPT], on[CPT];
        if constexpr (s > 0) ring_two(ro, y0);
        if constexpr (RES) {
            ring_two(ro + Lay::n_off, n0);
            ring_two(ro + Lay::pump_off, pu);
        }
        if constexpr (POT) ring_two(ro + Lay::pot_off, po);
        const C lft = shfl_up1(ce[s][CPT - 1]), rgt = shfl_dn1(ce[s][0]);
#pragma unroll
        for (int j = 0; j < CPT; ++j) {
            if constexpr (s == 0) y0[j] = ce[0][j];
            const T nin = !RES ? (T)0 : (s == 0 ? n0[j] : ns[before][j]);
            kn[j] = (T)0;
            rhs_iter<T, RES, FMA, UNIT>(P, s, ce[s][j], up[s][j], dn[j], j == 0 ? lft : ce[s][j > 0 ? j - 1 : 0],
                                        j == CPT - 1 ? rgt : ce[s][j < CPT - 1 ? j + 1 : j], nin, RES ? pu[j] : (T)0,
                                        POT ? po[j] : (T)0, RES, POT, kw[j], kn[j]);
        }
#pragma unroll
        for (int j = 0; j < CPT; ++j) {
            up[s][j] = ce[s][j];
            ce[s][j] = dn[j];
            C t = mk((T)0, (T)0);
            T tn = (T)0;
            on[j] = (T)0;
            if constexpr (s == 0) {
                t = smul(wb[0], kw[j]);
                tn = rmul(wb[0], kn[j]);
            } else if constexpr (s < 3) {
                t = axpy<FMA>(wb[s], kw[j], a[before][j]);
                tn = raxpy<FMA>(wb[s], kn[j], an[before][j]);
            }
            if constexpr (s < 3) {
                o[j] = axpy<FMA>(P.dtw[own], kw[j], y0[j]);
                if constexpr (RES) on[j] = raxpy<FMA>(P.dtw[own], kn[j], n0[j]);
            } else {
                o[j] = final_update<FMA>(P.dt, wb[3], a[2][j], kw[j], y0[j]);
                if constexpr (RES) on[j] = rfinal_update<FMA>(P.dt, wb[3], an[2][j], kn[j], n0[j]);
            }
            // what stage s - 1 handed on for this row is used up: the next row's takes its place
            if constexpr (s > 0) a[before][j] = pa[j], an[before][j] = pan[j], ns[before][j] = pn[j];
            pa[j] = t, pan[j] = tn, pn[j] = on[j];
            dn[j] = o[j];
        }
        const int row = R0 - 4 + k - s;
        if constexpr (STORE && s < 3) {
            if constexpr (IMG) {
                if (row >= R0 && row < R1) put(P.st_psi[own], P.st_n[own], row, o, on);
            } else {
                if (store_lane && row >= R0 && row < R1) put_at(P.st_psi[own], P.st_n[own], row * pitch + c, o, on);
            }
        }
        if constexpr (s == 3) put(P.psi1, P.n1, row, o, on);
    };
    // step k with the first NS stages; the row that the last of them makes goes
    // into the next stage's window
    auto step = [&](auto ns_, int k) __attribute__((always_inline)) {
        constexpr int NS = decltype(ns_)::value, nx = NS < 4 ? NS : 3;
        issue();             // row k + 4, into the slot of row k - 4, which step k - 1 read last
        cp_async_wait<3>();  // rows up to k + 1 are there
        ring_two(row_of(k + 1), dn);
        stage(std::integral_constant<int, 0>{}, k);
        if constexpr (NS > 1) stage(std::integral_constant<int, 1>{}, k);
        if constexpr (NS > 2) stage(std::integral_constant<int, 2>{}, k);
        if constexpr (NS > 3) stage(std::integral_constant<int, 3>{}, k);
        if constexpr (NS < 4) {
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                up[nx][j] = ce[nx][j];
                ce[nx][j] = dn[j];
                a[nx - 1][j] = pa[j], an[nx - 1][j] = pan[j], ns[nx - 1][j] = pn[j];
            }
        }
    };
    // a segment's first rows are there for the first stages only
    int k = 1;
#pragma unroll 1
    for (; k < 3; ++k) step(std::integral_constant<int, 1>{}, k);
#pragma unroll 1
    for (; k < 5; ++k) step(std::integral_constant<int, 2>{}, k);
#pragma unroll 1
    for (; k < 7; ++k) step(std::integral_constant<int, 3>{}, k);
    // two steps a round: fewer register moves between the windows' rows, and a
    // loop that still comes from the instruction cache (FP32, us per iteration
    // at 1024^2 / 4096^2: one step 16.8 / 196, two 16.2 / 184)
#pragma unroll 1
    while (k < last_k) {
        step(std::integral_constant<int, 4>{}, k);
        if (++k >= last_k) break;
        step(std::integral_constant<int, 4>{}, k);
        ++k;
    }
    // the last rows' copies may still be on their way: they must land before
    // the CTA's shared memory can belong to another kernel's
    cp_async_wait<0>();
}

template <typename T, bool RES, bool POT, bool UNIT, bool FMA, bool STORE, bool IMG, int MINB>
__global__ void __launch_bounds__(32 * kMarchWarps, MINB) rk4_march_kernel(const __grid_constant__ MarchParams<T> Q) {
    extern __shared__ __align__(16) unsigned char march_smem[];
    const int warp = threadIdx.x >> 5, item = blockIdx.x * kMarchWarps + warp;
    if (item >= Q.n_items) return;
    const int R0 = item / Q.strips * Q.seg_rows;
    // The previous iteration's kernel has completed.  The next one's is
    // scheduled when this one's CTAs are done, not earlier: CTAs that wait in
    // free slots leave the next grid unevenly spread over the SMs (25.4 against
    // 18.6 us at 1024^2 FP32, two CTAs per SM).
    pdl_wait();
    march_segment<T, RES, POT, UNIT, FMA, STORE, IMG>(Q.f, item % Q.strips, R0, min(R0 + Q.seg_rows, Q.f.N_r),
                                                 march_smem + warp * MarchLayout<T>::warp_bytes);
}

// ---------------------------------------------------------------- batches
// The segments of every instance of a batch, one warp each.  An instance's
// constants are loaded into registers once per segment.
struct MarchItem {
    int inst, strip, r0, r1;
};

template <typename T>
struct MarchBatchParams {
    const FusedParams<T>* f;  // [instance][direction]
    const MarchItem* items;
    int n_items, dir;
};

// POTS: no instance has a potential (0), all have one (1), or some (2)
template <typename T, bool RES, int POTS, bool FMA, bool IMG, int MINB>
__global__ void __launch_bounds__(32 * kMarchWarps, MINB) rk4_march_batch_kernel(const __grid_constant__ MarchBatchParams<T> Q) {
    extern __shared__ __align__(16) unsigned char march_smem[];
    const int warp = threadIdx.x >> 5, item = blockIdx.x * kMarchWarps + warp;
    if (item >= Q.n_items) return;
    const MarchItem it = Q.items[item];
    const FusedParams<T> P = Q.f[2 * it.inst + Q.dir];
    unsigned char* const ring = march_smem + warp * MarchLayout<T>::warp_bytes;
    if constexpr (POTS != 0) {
        if (POTS == 1 || P.pot != nullptr) {
            march_segment<T, RES, true, true, FMA, false, IMG>(P, it.strip, it.r0, it.r1, ring);
            return;
        }
    }
    if constexpr (POTS != 1) march_segment<T, RES, false, true, FMA, false, IMG>(P, it.strip, it.r0, it.r1, ring);
}

}  // namespace phx
