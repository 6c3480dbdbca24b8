/* RKN4 stage kernels of FP32 levels (the precision form on levels and AMR
 * hierarchies) for the axion-string projects of this library
 * (AxionStringsLap1 / AxionStringsLap2):
 *   Psi' = Pi,
 *   Pi'  = -2 Pi / eta + lap_N(Psi) - lambda Psi [eta^2 (|Psi|^2 - 1) + c]
 * with lambda = params[0], c = params[1], written against the equations in
 * FP32 (the plugin hooks compute in FP64, which runs at 1/64 of the FP32
 * rate on GB300).
 *
 * Same schedule as the FP64 stage kernel (sh_stage.cuh) with the RKN4
 * tableau of source/integrators/rkn.cpp:130-139 (c = {0, 1/2, 1},
 * a_21 = 1/8, a_32 = 1/2, a_31 = 0, bbar = {1/6, 1/3, 0},
 * b = {1/6, 2/3, 1/6}; every stage uses the step's initial momenta,
 * rkn.cpp:55-117):
 *   STAGE 0: K0 = accel(y0);  Y1 = y0 + h/2 y0' + h^2/8 K0
 *   STAGE 1: K1 = accel(Y1);  Y2 = y0 + h y0' + h^2/2 K1
 *   STAGE 2: K2 = accel(Y2);  y1 = y0 + h y0' + h^2 (K0/6 + K1/3),
 *                             y1' = y0' + h ((K0 + K2)/6 + 2 K1/3)
 * The stage buffers hold the positions Y_i only (every stage reads the
 * momenta y0' of the step's initial state), and only their two position
 * components get ghost cells at the stage times.  The last stage adds the
 * increments with Kahan compensation (the value y and its compensation c
 * stand for y - c; the compensations of the new state are written beside
 * it).
 *
 * The arithmetic is the explicitly rounded FP32 of the ensemble kernels
 * (sh_f32.cuh): Laplacian, potential, acceleration, stage positions and
 * increments round exactly as there.
 */
#ifndef SH_STAGE32_CUH_
#define SH_STAGE32_CUH_

#include "sh_f32.cuh"
#include "sh_internal.h"

namespace sh {

struct Stage32Args {
    const TileDev *tiles;
    const BoxDev *boxes;
    const float *state; /* Y_i, positions with filled ghost cells (stage 0: y0) */
    const float *y0;    /* the step's initial state (positions and momenta) */
    float *out;         /* stages 0, 1: Y_{i+1} (positions); stage 2: y1 */
    const float *k0, *k1; /* K buffers, two components each (box layout) */
    float *kout;
    const float *c_old;   /* compensations of y0 */
    float *c_new;         /* compensations of y1 */
    float h, cm, ck;      /* dt; stage position coefficients of y0' and K */
    float h2;             /* dt^2 */
    float inv;            /* 1/dx^2 (7 points) or 1/(12 dx^2) (13 points) */
    float lam, cst;       /* params[0], params[1] */
    float friction, eta2; /* -2/eta and eta^2 at the stage time */
};

/* V neighbouring cells along x at p + o */
template <int V>
__device__ __forceinline__ void ld_cells(float (&x)[V], const float *__restrict__ p, int o) {
    if constexpr (V == 2) {
        const float2 v = *reinterpret_cast<const float2 *>(p + o);
        x[0] = v.x;
        x[1] = v.y;
    } else {
        x[0] = p[o];
    }
}
template <int V>
__device__ __forceinline__ void st_cells(float *p, int o, const float (&x)[V]) {
    if constexpr (V == 2) *reinterpret_cast<float2 *>(p + o) = make_float2(x[0], x[1]);
    else p[o] = x[0];
}

/* Each thread walks the z-column of V neighbouring cells along x, keeping the
 * 2 ORDER + 1 values of the two position components along z in registers (one
 * new plane value per step instead of 2 ORDER + 1 loads), with
 * restrict-qualified pointers (every buffer of a stage is distinct).  The sums
 * are formed in the order of the ensemble kernels (x+, x-, y+, y-, z+, z-).
 *
 * Memory bounds the stages (8, 10 and 22 words per cell; DRAM moves 11-12%
 * more, for the ghost cells), through the loads that wait and the sectors that
 * a 128-byte row 8 bytes off its boundary touches twice.  V = 2 reads pairs as
 * 8-byte words, 7 loads per component and pair instead of 18 with 13 points,
 * and 200 instructions per cell row become 90; it needs rows of an even number
 * of cells behind an even number of ghost cells in all boxes (L->x_pairs, so
 * that every pair lies on an 8-byte boundary), and V = 1 takes the others, the
 * 7-point levels of one ghost cell among them.
 * 64 boxes of 64^3, 13 points, stages 0, 1, 2: V = 1 with the next plane's
 * words prefetched 158, 178, 340 us; V = 2 in 32-cell rows and 8 planes 143,
 * 159, 302 us, in 64-cell rows and 4 planes 133, 147, 275 us (floors at
 * 6.78 TB/s: 79, 99, 218).  Prefetches cost V = 2 time (281 against 289-309
 * us in stage 2), as do 10 or more blocks per SM in stage 2 (293 us) and fewer
 * than 16 in the others (stage 1: 154 us with 10). */
template <int ORDER, int STAGE, int V>
__global__ void __launch_bounds__(kThreads / V, V == 1 ? (STAGE == 2 ? 10 : 16)
                                                       : (STAGE == 2 ? 8 : 16))
    stage32_axion_kernel(const __grid_constant__ Stage32Args a) {
    constexpr int R = ORDER; /* stencil reach */
    const TileDev t = a.tiles[blockIdx.x];
    const BoxDev b = a.boxes[t.box];
    const int tid = threadIdx.x;
    const int ty = tid * V / t.nx;
    const int i = t.x0 + (tid * V - ty * t.nx);
    const int j = t.y0 + ty;
    if (ty >= kThreads / t.nx || i > b.hi[0] || j > b.hi[1]) return;
    const int kend = min(t.z0 + t.nz - 1, b.hi[2]);
    const long long gvol = b.gvol;
    const int gx = (int)b.gdim[0], gxy = gx * (int)b.gdim[1];
    /* the tile's first cell in each buffer (the same for all threads), and
     * 32-bit offsets from there */
    const long long corner = (t.x0 - b.glo[0]) + (long long)(t.y0 - b.glo[1]) * gx +
                             (long long)(t.z0 - b.glo[2]) * gxy;
    const long long s4 = b.off * 4 + corner, s2 = b.off * 2 + corner;
    const float *__restrict__ st = a.state + s4;
    const float *__restrict__ y0 = a.y0 + s4;
    const float *__restrict__ k0 = a.k0 + s2;
    const float *__restrict__ k1 = a.k1 + s2;
    const float *__restrict__ c_old = a.c_old + s4;
    float *__restrict__ out = a.out + s4;
    float *__restrict__ kout = a.kout + s2;
    float *__restrict__ c_new = a.c_new + s4;
    int o = (i - t.x0) + (j - t.y0) * gx;
    /* z-window of the two positions: w[c][d] = values at plane k - R + d */
    float w[2][2 * R + 1][V];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int d = 0; d < 2 * R; ++d) ld_cells<V>(w[c][d], st + c * gvol, o + (d - R) * gxy);
    for (int n = kend - t.z0; n >= 0; --n, o += gxy) {
        /* the next cell's y0 asked into L1 while this one is computed, in the
         * form that gains by it on large levels: a step of one 192^3 level of
         * three ghost cells 319 us against 325, of 27 boxes of 63^3 405
         * against 407, of 96^3 63.4 against 62.5; in every form of V = 1 the
         * 7-point steps of 160^3 and more take 4 % longer */
        if constexpr (V == 1 && ORDER == 2 && STAGE == 1) {
            if (n > 0) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(y0 + c * gvol + (o + gxy)));
            }
        }
        float lap[2][V];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float *__restrict__ s = st + c * gvol;
            float yp[R][V], ym[R][V], x[V + 2 * R];
            ld_cells<V>(w[c][2 * R], s, o + R * gxy);
#pragma unroll
            for (int r = 1; r <= R; ++r) {
                ld_cells<V>(yp[r - 1], s, o + r * gx);
                ld_cells<V>(ym[r - 1], s, o - r * gx);
            }
            if constexpr (V == 2 && R == 2) {
                float l[2], h[2];
                ld_cells<2>(l, s, o - 2);
                ld_cells<2>(h, s, o + 2);
                x[0] = l[0], x[1] = l[1], x[4] = h[0], x[5] = h[1];
            } else {
#pragma unroll
                for (int r = 1; r <= R; ++r) {
                    x[R - r] = s[o - r];
                    x[R + V - 1 + r] = s[o + V - 1 + r];
                }
            }
#pragma unroll
            for (int v = 0; v < V; ++v) x[R + v] = w[c][R][v];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if constexpr (ORDER == 1) {
                    lap[c][v] = f32::lap7(x[v + 1], x[v + 2], x[v], yp[0][v], ym[0][v], w[c][2][v],
                                          w[c][0][v], a.inv);
                } else {
                    const float s1 = f32::ring(x[v + 3], x[v + 1], yp[0][v], ym[0][v], w[c][3][v],
                                               w[c][1][v]);
                    const float s2 = f32::ring(x[v + 4], x[v], yp[1][v], ym[1][v], w[c][4][v],
                                               w[c][0][v]);
                    lap[c][v] = f32::lap13(x[v + 2], s1, s2, a.inv);
                }
            }
        }
        float q[2][V], kq[2][V];
#pragma unroll
        for (int c = 0; c < 2; ++c) ld_cells<V>(q[c], y0 + (2 + c) * gvol, o);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const float p0 = w[0][R][v], p1 = w[1][R][v];
            const float pot = f32::potential(p0, p1, a.lam, a.eta2, a.cst);
            kq[0][v] = f32::accel(q[0][v], lap[0][v], p0, pot, a.friction);
            kq[1][v] = f32::accel(q[1][v], lap[1][v], p1, pot, a.friction);
        }
        if constexpr (STAGE < 2) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                st_cells<V>(kout + c * gvol, o, kq[c]);
                float y[V];
                /* (stage 0 reads the initial state itself) */
                if constexpr (STAGE == 0) {
#pragma unroll
                    for (int v = 0; v < V; ++v) y[v] = w[c][R][v];
                } else {
                    ld_cells<V>(y, y0 + c * gvol, o);
                }
#pragma unroll
                for (int v = 0; v < V; ++v)
                    y[v] = f32::stage_pos(y[v], q[c][v], kq[c][v], a.cm, a.ck);
                st_cells<V>(out + c * gvol, o, y);
            }
        } else {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float ka[V], kb[V], y[V], cy[V], cm[V];
                ld_cells<V>(ka, k0 + c * gvol, o);
                ld_cells<V>(kb, k1 + c * gvol, o);
                ld_cells<V>(y, y0 + c * gvol, o);
                ld_cells<V>(cy, c_old + c * gvol, o);
                ld_cells<V>(cm, c_old + (2 + c) * gvol, o);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    f32::kahan(y[v], f32::dpos(q[c][v], ka[v], kb[v], a.h, a.h2), cy[v]);
                    f32::kahan(q[c][v], f32::dmom(ka[v], kb[v], kq[c][v], a.h), cm[v]);
                }
                st_cells<V>(out + c * gvol, o, y);
                st_cells<V>(out + (2 + c) * gvol, o, q[c]);
                st_cells<V>(c_new + c * gvol, o, cy);
                st_cells<V>(c_new + (2 + c) * gvol, o, cm);
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int d = 0; d < 2 * R; ++d)
#pragma unroll
                for (int v = 0; v < V; ++v) w[c][d][v] = w[c][d + 1][v];
    }
}

/* Kick-drift-kick leapfrog stages of FP32 levels of FirstOrderPhaseTransition
 * with the pure potential (params[0] = 0), with or without the GW tensor:
 *   Phi'' = lap Phi + q2 Phi + q3 Phi^2 + q4 Phi^3,
 *   u_ij'' = lap u_ij + d_i Phi d_j Phi
 * (4th-order Laplacian and gradient; projects/FirstOrderPhaseTransition/
 * kernels_rhs.h:20-109), the schedule of source/integrators/leapfrog.cpp:13-57
 * (both kicks with the acceleration of the positions they see):
 *   STAGE 0: a = f(x0);  vh = v0 + dt/2 a;  x1 = x0 + dt vh
 *   STAGE 1: a = f(x1);  v1 = vh + dt/2 a
 * with Kahan-compensated updates: vh and its compensation go to the K
 * buffer, x1 and v1 with theirs to the new state.  The arithmetic is that of
 * the FP32 ensemble kernel of the same equations (sh_fast.cu). */
struct Stage32FoptArgs {
    const TileDev *tiles;
    const BoxDev *boxes;
    const float *state; /* positions read by the stencils (stage 0: x0, 1: x1) */
    const float *y0;    /* the step's initial state */
    const float *c_old; /* its compensations */
    float *out;         /* the new state */
    float *c_new;       /* its compensations */
    float *kv, *kc;     /* vh and its compensation (np components each) */
    float inv12dx2, inv12dx, hdt, dt, q2, q3, q4;
};

template <int STAGE, bool GW>
__global__ void __launch_bounds__(kThreads)
    stage32_fopt_kernel(const __grid_constant__ Stage32FoptArgs a) {
    constexpr int NP = GW ? 7 : 1, NC = 2 * NP;
    const TileDev t = a.tiles[blockIdx.x];
    const BoxDev b = a.boxes[t.box];
    const int tid = threadIdx.x + kTileX * threadIdx.y;
    const int ty = tid / t.nx;
    const int i = t.x0 + (tid - ty * t.nx);
    const int j = t.y0 + ty;
    if (ty >= kThreads / t.nx || i > b.hi[0] || j > b.hi[1]) return;
    const int kend = min(t.z0 + t.nz - 1, b.hi[2]);
    const long long gx = b.gdim[0], gxy = gx * b.gdim[1], gvol = b.gvol;
    /* position q: Phi, u_xx, u_yy, u_zz, u_xy, u_xz, u_yz; momentum: dPhi,
     * du_xx, ... (the level's component order) */
    auto pos = [](int q) { return q == 0 ? 0 : 1 + q; };
    auto mom = [](int q) { return q == 0 ? 1 : NP + q; };
    for (int k = t.z0; k <= kend; ++k) {
        const long long lc =
            (i - b.glo[0]) + (long long)(j - b.glo[1]) * gx + (long long)(k - b.glo[2]) * gxy;
        const long long sb = b.off * NC + lc;
        const long long kb = b.off * NP + lc;
        float acc[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const float *s = a.state + sb + pos(q) * gvol;
            float s1 = s[1] + s[-1];
            s1 += s[gx] + s[-gx];
            s1 += s[gxy] + s[-gxy];
            float s2 = s[2] + s[-2];
            s2 += s[2 * gx] + s[-2 * gx];
            s2 += s[2 * gxy] + s[-2 * gxy];
            acc[q] = (16.f * s1 - s2 - 90.f * s[0]) * a.inv12dx2;
        }
        const float *ph = a.state + sb;
        const float phi = ph[0];
        acc[0] += phi * (a.q2 + phi * (a.q3 + phi * a.q4));
        if constexpr (GW) {
            float g[3];
            g[0] = (8.f * (ph[1] - ph[-1]) - (ph[2] - ph[-2])) * a.inv12dx;
            g[1] = (8.f * (ph[gx] - ph[-gx]) - (ph[2 * gx] - ph[-2 * gx])) * a.inv12dx;
            g[2] = (8.f * (ph[gxy] - ph[-gxy]) - (ph[2 * gxy] - ph[-2 * gxy])) * a.inv12dx;
            acc[1] += g[0] * g[0];
            acc[2] += g[1] * g[1];
            acc[3] += g[2] * g[2];
            acc[4] += g[0] * g[1];
            acc[5] += g[0] * g[2];
            acc[6] += g[1] * g[2];
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            if constexpr (STAGE == 0) {
                float v = a.y0[sb + mom(q) * gvol], cv = a.c_old[sb + mom(q) * gvol];
                f32::kahan(v, a.hdt * acc[q], cv);
                a.kv[kb + q * gvol] = v;
                a.kc[kb + q * gvol] = cv;
                float x = a.y0[sb + pos(q) * gvol], cx = a.c_old[sb + pos(q) * gvol];
                f32::kahan(x, a.dt * v, cx);
                a.out[sb + pos(q) * gvol] = x;
                a.c_new[sb + pos(q) * gvol] = cx;
            } else {
                float v = a.kv[kb + q * gvol], cv = a.kc[kb + q * gvol];
                f32::kahan(v, a.hdt * acc[q], cv);
                a.out[sb + mom(q) * gvol] = v;
                a.c_new[sb + mom(q) * gvol] = cv;
            }
        }
    }
}

} // namespace sh

#endif
