// The vector-Jacobian product of one RK4 iteration (the four stages of
// adj_stage_kernel, phx_adjoint.cuh) as marching warps, the walk of
// phx_step_march.cuh run through the stages backwards: at step k a warp forms
// Ybar_4 on row k, Ybar_3 on row k - 1, Ybar_2 on row k - 2 and Ybar_1 on row
// k - 3.  The stencil input of a stage is kbar_s = dt b_s lam' + a_s dt
// Ybar_{s+1}: its rows stay in registers, its horizontal neighbours come by
// shuffles.  lam' and the potential (needed by all four stages) go through a
// ring of eight rows per warp, the stage values Y_s (needed by one stage each)
// through rings of four rows that run behind by the stage's lag.
//
// The grid is periodic on both axes.  With WRAP (an even number of columns) the
// copies wrap rows and column pairs themselves, and neither lam' nor the Y_s
// need periodic images; without it both carry them, four deep.
//
// us a launch at 512^2 / 1024^2 FP32: 9.6 / 22.9 (a kernel of 64 x 16 tiles,
// which waited for its global loads and recomputed every tile's halo, took 16.4
// / 51.3); FP64 at 512^2 26.0 (32.9).
#pragma once

#include "phx_adjoint.cuh"
#include "phx_step_march.cuh"

namespace phx {

template <typename T>
struct AdjMarchParams {
    AdjFusedParams<T> a;
    int strips, seg_rows, n_items;
};

// Ring rows in 16-byte pieces per lane, 512 bytes apart: lam' psi, then (lam_n,
// potential), which share a piece in FP32; the rings of Y_4..Y_1 (psi, n) after
// them.
template <typename T>
struct AdjMarchLayout {
    static constexpr int PB = 4 * (int)sizeof(T), RB = 2 * (int)sizeof(T);
    static constexpr int n_off = PB * 32, pot_off = n_off + (RB == 8 ? 8 : 512);
    static constexpr int lam_row = n_off + (RB == 8 ? 512 : 1024);
    static constexpr int y_row = PB * 32 + 512, y_rows = 4;
    static constexpr int y_off(int u) { return kMarchRing * lam_row + u * y_rows * y_row; }
    static constexpr int warp_bytes = kMarchRing * lam_row + 4 * y_rows * y_row;
    static constexpr int bytes = kMarchWarps * warp_bytes;
};

template <typename T, bool RES, bool POT, bool WRAP, int MINB>
__global__ void __launch_bounds__(32 * kMarchWarps, MINB) adj_march_kernel(const __grid_constant__ AdjMarchParams<T> M) {
    using Lay = AdjMarchLayout<T>;
    using C = cx<T>;
    extern __shared__ __align__(16) unsigned char march_smem[];
    const AdjFusedParams<T>& Q = M.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, item = blockIdx.x * kMarchWarps + warp;
    if (item >= M.n_items) return;
    const int strip = item % M.strips, R0 = item / M.strips * M.seg_rows, R1 = min(R0 + M.seg_rows, Q.N_r);
    const int c = strip * kMarchOut - 4 + 2 * lane;
    const int pitch = (int)Q.pitch;
    unsigned char* const mine = march_smem + warp * Lay::warp_bytes + lane * 16;
    const unsigned s_mine = (unsigned)__cvta_generic_to_shared(mine);

    // rows are counted from k = 0 at R0 - 4.  Without WRAP the rows copied ahead
    // end at R1 + 6 and begin at R0 - 8, within the planes' rings of 8, and lanes
    // past the ring read its last columns, which nothing stored depends on
    const int N_r = Q.N_r, N_c = Q.N_c;
    const int cl = WRAP ? (c % N_c + N_c) % N_c : min(c, (N_c + 6) & ~1);
    int next_r = WRAP ? ((R0 - 4) % N_r + N_r) % N_r : R0 - 4;  // the row that lam' is copied from next
    auto copy = [&](unsigned d, const auto* p, int g) __attribute__((always_inline)) {
        constexpr int bytes = 2 * (int)sizeof(*p);
#pragma unroll
        for (int i = 0; i < bytes; i += 16)
            cp_async<(bytes < 16 ? bytes : 16)>(d + i * 32, reinterpret_cast<const unsigned char*>(p + g) + i);
    };
    // what step k copies: lam' and the potential of row k + 4, Y_{4-u} of row k + 3 - u
    auto issue = [&](int k, bool y) __attribute__((always_inline)) {
        const int g = next_r * pitch + cl;
        const unsigned d = s_mine + (unsigned)((k + 4) & (kMarchRing - 1)) * Lay::lam_row;
        copy(d, Q.lam_psi, g);
        if constexpr (RES) copy(d + Lay::n_off, Q.lam_n, g);
        if constexpr (POT) copy(d + Lay::pot_off, Q.pot, g);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (!y) break;
            int r = next_r - (1 + u);
            if (WRAP && r < 0) r += N_r;
            const int gy = r * pitch + cl;
            const unsigned dy = s_mine + Lay::y_off(u) + (unsigned)((k + 3 - u) & (Lay::y_rows - 1)) * Lay::y_row;
            copy(dy, Q.Ypsi[3 - u], gy);
            if constexpr (RES) copy(dy + Lay::PB * 32, Q.Yn[3 - u], gy);
        }
        cp_async_commit();
        ++next_r;
        if (WRAP && next_r == N_r) next_r = 0;
    };
    pdl_wait();  // what the kernel before wrote is there
    // Y_{4-u} from row 1 - u on, its first use: earlier rows would fall into
    // slots whose next rows are on their way at the same time
#pragma unroll
    for (int k = -4; k < 1; ++k) issue(k, k >= -2);

    const bool store_lane = c >= strip * kMarchOut && c < (strip + 1) * kMarchOut && c < Q.N_c;
    const bool store_two = sizeof(T) == 4 || c + 2 <= Q.N_c;
    const bool edge_strip = strip == 0 || (strip + 1) * kMarchOut > N_c - 4;
    auto put = [&](int row, bool live, const C* v, const T* nv) __attribute__((always_inline)) {
        auto put_at = [&](int gi) __attribute__((always_inline)) {
            if (store_two) {
                st_two(Q.out_psi + gi, v);
                if constexpr (RES) st_two(Q.out_n + gi, nv);
            } else {
                Q.out_psi[gi] = v[0];
                if constexpr (RES) Q.out_n[gi] = nv[0];
            }
        };
        const int g = row * pitch + c;
        if (live) put_at(g);
        if constexpr (!WRAP) {
            if (edge_strip || row < 4 || row >= N_r - 4) {
                // 4-deep periodic images: the next iteration reads lam with a 4-cell halo
                const int dy = row < 4 ? N_r : (row >= N_r - 4 ? -N_r : 0);
                if (live && dy) put_at(g + dy * pitch);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int dx = c + j < 4 ? N_c : (c + j >= N_c - 4 ? -N_c : 0);
                    if (live && dx != 0 && c + j < N_c) {
                        const int gi = g + j + dx;
                        Q.out_psi[gi] = v[j];
                        if constexpr (RES) Q.out_n[gi] = nv[j];
                        if (dy) {
                            Q.out_psi[gi + dy * pitch] = v[j];
                            if constexpr (RES) Q.out_n[gi + dy * pitch] = nv[j];
                        }
                    }
                }
            }
        }
    };

    C up[4][2], ce[4][2];  // kbar of the row above, and of the row, that stage u (s = 4 - u) evaluates next
    C acc[3][2];           // stage u to u + 1, of one row: the sum of Ybar, its n part,
    T accn[3][2], ybn[3][2], pb[3][2], vb[3][2];  // Ybar's n part, dL/dP, dL/dV
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            up[u][j] = ce[u][j] = mk((T)0, (T)0);
            if (u < 3) acc[u][j] = mk((T)0, (T)0), accn[u][j] = ybn[u][j] = pb[u][j] = vb[u][j] = (T)0;
        }
    auto lam_row = [&](int k) { return mine + (k & (kMarchRing - 1)) * Lay::lam_row; };
    auto scaled_row = [&](int k, C* v) {
        ring_two(lam_row(k), v);
#pragma unroll
        for (int j = 0; j < 2; ++j) v[j].re *= Q.dt_b[3], v[j].im *= Q.dt_b[3];
    };
    cp_async_wait<3>();  // lam' of rows 0 and 1
    scaled_row(0, up[0]);
    scaled_row(1, ce[0]);

    T pb_old[2], vb_old[2];  // dL/dP, dL/dV so far of the row that the last stage works on
    C dn[2], pacc[2];  // kbar of the row the stage before has just made, and what it hands on with it
    T paccn[2], pybn[2], ppb[2], pvb[2];
    auto stage = [&](auto ut, int k) __attribute__((always_inline)) {
        constexpr int u = decltype(ut)::value, s = 4 - u, before = u > 0 ? u - 1 : 0;
        const unsigned char* const ro = lam_row(k - u);
        const unsigned char* const yo = mine + Lay::y_off(u) + ((k - u) & (Lay::y_rows - 1)) * Lay::y_row;
        C psi[2], lam[2];
        T n[2], lamn[2], pot[2];
        ring_two(yo, psi);
        ring_two(ro, lam);
        if constexpr (RES) {
            ring_two(yo + Lay::PB * 32, n);
            ring_two(ro + Lay::n_off, lamn);
        }
        if constexpr (POT) ring_two(ro + Lay::pot_off, pot);
        const C lft = shfl_up1(ce[u][1]), rgt = shfl_dn1(ce[u][0]);
        const T dtb = Q.dt_b[s - 1];
        C out[2];
        T outn[2];
        const int row = R0 - 4 + k - u;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const C mu = ce[u][j], mu_u = up[u][j], mu_d = dn[j], mu_l = j == 0 ? lft : ce[u][0], mu_r = j == 0 ? ce[u][1] : rgt;
            T m = (T)0;
            if constexpr (RES) m = u == 0 ? dtb * lamn[j] : dtb * lamn[j] + Q.a_dt[s - 1] * ybn[before][j];
            const T nn = RES ? n[j] : (T)0;
            const T norm = psi[j].re * psi[j].re + psi[j].im * psi[j].im;
            C lap;
            lap.re = Q.m2 * mu.re + Q.ody2 * (mu_u.re + mu_d.re) + Q.odx2 * (mu_l.re + mu_r.re);
            lap.im = Q.m2 * mu.im + Q.ody2 * (mu_u.im + mu_d.im) + Q.odx2 * (mu_l.im + mu_r.im);
            T W = Q.ohb_gc * norm;
            T B = -Q.half_gamma_c;
            if constexpr (RES) {
                W += Q.ohb_gr * nn;
                B += Q.half_R * nn;
            }
            if constexpr (POT) W += Q.ohb * (pot[j] * Q.c_pot[s - 1]);
            // h = A lap(mu) + W mu; i h = (-h.im, h.re)
            const T hre = Q.A * lap.re + W * mu.re, him = Q.A * lap.im + W * mu.im;
            const T im_mbar_psi = mu.re * psi[j].im - mu.im * psi[j].re;  // Im(conj(mu) psi)
            const T re_mbar_psi = mu.re * psi[j].re + mu.im * psi[j].im;  // Re(conj(mu) psi)
            const T sp = (T)2 * Q.ohb_gc * im_mbar_psi - (RES ? (T)2 * Q.R * nn * m : (T)0);
            C g;
            g.re = -him + B * mu.re + sp * psi[j].re;
            g.im = hre + B * mu.im + sp * psi[j].im;
            const T gn = RES ? Q.ohb_gr * im_mbar_psi + Q.half_R * re_mbar_psi - (Q.gamma_r + Q.R * norm) * m : (T)0;
            const T dp = Q.c_pump[s - 1] * m, dv = Q.ohb * Q.c_pot[s - 1] * im_mbar_psi;
            C t;
            T tn, tp, tv;
            if constexpr (u == 0) {
                t = g, tn = gn, tp = dp, tv = dv;
            } else {
                t = mk(acc[before][j].re + g.re, acc[before][j].im + g.im);
                tn = accn[before][j] + gn, tp = pb[before][j] + dp, tv = vb[before][j] + dv;
                // used up: the next row's take their place
                acc[before][j] = pacc[j], accn[before][j] = paccn[j], ybn[before][j] = pybn[j], pb[before][j] = ppb[j],
                vb[before][j] = pvb[j];
            }
            if constexpr (u < 3) {
                // kbar of the next stage on this row
                const T db = Q.dt_b[s - 2], ad = Q.a_dt[s - 2];
                out[j] = mk(db * lam[j].re + ad * g.re, db * lam[j].im + ad * g.im);
                pacc[j] = t, paccn[j] = tn, pybn[j] = gn, ppb[j] = tp, pvb[j] = tv;
            } else {
                out[j] = mk(lam[j].re + t.re, lam[j].im + t.im);
                outn[j] = RES ? lamn[j] + tn : (T)0;
                pb_old[j] += tp;
                vb_old[j] += tv;
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) up[u][j] = ce[u][j], ce[u][j] = dn[j];
        if constexpr (u == 3) {
            const bool live = row >= R0 && store_lane;
            put(row, live, out, outn);
            if (live) {
                const int g = row * pitch + c;
                if (RES && Q.pbar) {
                    if (store_two) st_two(Q.pbar + g, pb_old);
                    else Q.pbar[g] = pb_old[0];
                }
                if (Q.vbar) {
                    if (store_two) st_two(Q.vbar + g, vb_old);
                    else Q.vbar[g] = vb_old[0];
                }
            }
        } else {
            dn[0] = out[0], dn[1] = out[1];
        }
    };
    const int last_k = R1 - R0 + 7;
    auto open = [&](int k) __attribute__((always_inline)) {
        issue(k, true);
        cp_async_wait<3>();  // what step k - 3 copied: lam' of row k + 1, Y_{4-u} of row k - u
        scaled_row(k + 1, dn);
    };
    // stage u has its first row at step 1 + 2 u: the first four steps run two
    // stages, the others all of them (the later ones work on rows that are not
    // there yet and store nothing)
    int k = 1;
#pragma unroll 1
    for (; k < 5; ++k) {
        open(k);
        stage(std::integral_constant<int, 0>{}, k);
        stage(std::integral_constant<int, 1>{}, k);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            up[2][j] = ce[2][j];
            ce[2][j] = dn[j];
            acc[1][j] = pacc[j], accn[1][j] = paccn[j], ybn[1][j] = pybn[j], pb[1][j] = ppb[j], vb[1][j] = pvb[j];
        }
    }
#pragma unroll 1
    for (; k < last_k; ++k) {
        // asked for now, added to in the last stage
        const int row = R0 - 7 + k, g = row * pitch + c;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const bool live = row >= R0 && store_lane && (store_two || j == 0);
            pb_old[j] = RES && Q.pbar && live ? Q.pbar[g + j] : (T)0;
            vb_old[j] = Q.vbar && live ? Q.vbar[g + j] : (T)0;
        }
        open(k);
        stage(std::integral_constant<int, 0>{}, k);
        stage(std::integral_constant<int, 1>{}, k);
        stage(std::integral_constant<int, 2>{}, k);
        stage(std::integral_constant<int, 3>{}, k);
    }
    cp_async_wait<0>();  // no copy may land after the CTA's shared memory has gone to another
}

}  // namespace phx
