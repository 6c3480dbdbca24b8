/* Stage kernels instantiated once per project (included by proj_*.cu after
 * the project's hook headers and SLEDGEHAMR_FINISH_SETUP).
 *
 * One launch evaluates the project's per-cell Rhs (plus the GW source,
 * backreaction and Kreiss-Oliger terms when enabled) on every valid cell of
 * a level and fuses the linear combination that the reference performs
 * afterwards as separate MultiFab passes:
 *
 *   RKN stage i    K_i = accel(Y_i); Y_{i+1} = y0 + c h y0' + h^2 sum a K_j
 *                  (source/integrators/rkn.cpp:57-95)
 *   RKN final      y1 = y0 + h y0' + h^2 sum bbar K; y1' = y0' + h sum b K
 *                  (rkn.cpp:97-117)
 *   SSPRK3 stages  K = f(u) + w K; u' = y0 + c K   (lsssprk3.cpp:14-31,
 *                  FillAddRhs macros.h:392-485)
 *   leapfrog       vh = v0 + dt/2 a, x1 = x0 + dt vh; v1 = vh + dt/2 a
 *                  (leapfrog.cpp:13-57)
 *
 * Thread mapping: a block of kThreads = 128 threads owns a tile of one box,
 * nx <= 32 cells wide in x (the box width when the box is narrower, so that
 * the small boxes of refined levels keep every thread busy), kThreads / nx
 * rows in y and t.nz planes in z; each thread walks its z-column, so that
 * per-thread set-up (the reciprocals of dx^2 and of the time in the hooks)
 * is paid once per column.  Hooks read the stage state
 * straight from HBM through an Array4 view of the ghost-grown box; the
 * reuse of neighbour values comes from L1.  The per-cell Rhs output is an
 * Array4 over a register array (all strides zero), which the compiler keeps
 * in registers because every component index is a compile-time constant.
 */
#ifndef SH_STAGE_CUH_
#define SH_STAGE_CUH_

#include <sledgehamr.h>

#include "sh_internal.h"

namespace sh {

static_assert(sledgehamr::kStageParams == kMaxParams, "parameter array of StageArgs");

/* Position/momentum pairing of the reference (rkn.cpp:32-44): user fields
 * [0, uN) pair with [uN, 2uN); with GW the tensor block [Nf, Nf+6) pairs
 * with [Nf+6, Nf+12). */
template <int NSCAL, bool GW>
struct Pairs {
    static constexpr int kUN = NSCAL / 2;
    static constexpr int kNP = kUN + (GW ? 6 : 0);
    static constexpr int kNC = NSCAL + (GW ? 12 : 0);
    __host__ __device__ static constexpr int pos(int q) {
        return q < kUN ? q : NSCAL + (q - kUN);
    }
    __host__ __device__ static constexpr int mom(int q) {
        return q < kUN ? kUN + q : NSCAL + 6 + (q - kUN);
    }
};

/* Resident blocks per SM (of kThreads threads; caps the registers).  The
 * integer and the FP64 work of a warp overlap only with other warps', so the
 * occupancy counts until the spills cost more.  Device time per launch, us:
 * 7-point axion level 128^3, blocks 6 / 7 / 8: 74.9 / 70.8 / 72.3; 13-point
 * 256^3 in 32^3 boxes: 650 / 623 / 602 (9: 599); 13-point with tensor, 160^3:
 * 3 / 4 / 5 / 6 / 7 / 8: 880 / 763 / 736 / 701 / 700 / 681; dissipation, 99^3:
 * uncapped / 4 / 5 / 6: 202 / 129 / 124 / 125. */
template <bool GW, int KO, int REACH>
constexpr int stage_min_blocks() {
    return KO != 0 && !GW ? 5 : (GW || REACH >= 2 ? 8 : 7);
}

/* EPI: the epilogue, or kEpiAny where it is taken from the arguments at run
 * time.  The instantiations for the RKN4 and leapfrog stages leave out the
 * switch and the loops over the earlier K; an intermediate RKN4 stage of the
 * 7-point kernel issues 597 warp instructions per 32 cells. */
template <class H, bool GW, int KO, bool SP = false, int EPI = kEpiAny>
__global__ void __launch_bounds__(kTileX *kTileY, (stage_min_blocks<GW, KO, H::kReach>()))
    stage_kernel(const __grid_constant__ StageArgs a) {
    using PR = Pairs<H::kNScalars, GW>;
    constexpr int NC = PR::kNC;
    constexpr int NP = PR::kNP;

    const TileDev t = a.tiles[blockIdx.x];
    const BoxDev b = a.boxes[t.box];
    const int tid = threadIdx.x + kTileX * threadIdx.y;
    const int ty = tid / t.nx;
    const int i = t.x0 + (tid - ty * t.nx);
    const int j = t.y0 + ty;
    if (ty >= kThreads / t.nx || i > b.hi[0] || j > b.hi[1]) return;
    const int kend = min(t.z0 + t.nz - 1, b.hi[2]);

    const long long gx = b.gdim[0];
    const long long gxy = gx * b.gdim[1];
    const long long gvol = b.gvol;
    const amrex::Dim3 glo{b.glo[0], b.glo[1], b.glo[2]};
    const amrex::Dim3 ghi{b.glo[0] + b.gdim[0], b.glo[1] + b.gdim[1], b.glo[2] + b.gdim[2]};
    const amrex::Array4<const double> st(a.state + b.off * NC, gx, gxy, gvol, glo, ghi, NC);
    /* periodic images of a cell in the ghost cells of a self-periodic box:
     * along each axis within ng of a face, the element offset of its image
     * across the domain (0 elsewhere); the cell's images are the non-empty
     * combinations of the non-zero offsets (x and y fixed per thread, z per
     * cell).  SP: the instantiation for such boxes (a.self_periodic set). */
    long long ox = 0, oy = 0;
    if constexpr (SP) {
        if (i < b.lo[0] + a.ng) ox = a.per[0];
        else if (i > b.hi[0] - a.ng) ox = -a.per[0];
        if (j < b.lo[1] + a.ng) oy = a.per[1] * gx;
        else if (j > b.hi[1] - a.ng) oy = -a.per[1] * gx;
    }

    for (int k = t.z0; k <= kend; ++k) {
        /* the epilogue's inputs of the next cell (y0 and the earlier K) asked
         * into L1 while this cell's stencil runs; the stencil's own loads
         * are left to the cache (prefetching them too measured no better) */
        if (k < kend) {
            const long long next = (i - glo.x) + (j - glo.y) * gx + (k + 1 - glo.z) * gxy;
            if (EPI != kEpiLf1 && a.y0) {
#pragma unroll
                for (int n = 0; n < NC; ++n)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(a.y0 + b.off * NC + next +
                                                                 n * gvol));
            }
            /* the K buffers hold every component in the SSPRK3 stages and
             * the momenta of the pairs otherwise */
            if (EPI == kEpiRknStage || EPI == kEpiLf0) {
                /* no earlier K */
            } else if (EPI == kEpiAny && (a.epi == kEpiSsp0 || a.epi == kEpiSspAdd)) {
                for (int s = 0; s < a.nkin; ++s)
#pragma unroll
                    for (int n = 0; n < NC; ++n)
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(
                            a.kin[s] + b.off * NC + next + n * gvol));
            } else {
                const int nk = EPI == kEpiRknFinal ? 2 : (EPI == kEpiLf1 ? 1 : a.nkin);
#pragma unroll 2
                for (int s = 0; s < nk; ++s)
#pragma unroll
                    for (int q = 0; q < NP; ++q)
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(
                            a.kin[s] + b.off * NP + next + q * gvol));
            }
        }
        double r[NC];
#pragma unroll
        for (int n = 0; n < NC; ++n) r[n] = 0.;
        const amrex::Array4<double> rhs(r, 0, 0, 1, amrex::Dim3{i, j, k},
                                        amrex::Dim3{i + 1, j + 1, k + 1}, NC);
        H::rhs(rhs, st, i, j, k, a.lev, a.time, a.dt, a.dx, a.params);
        if constexpr (GW) {
            H::gw_rhs(rhs, st, i, j, k, a.lev, a.time, a.dt, a.dx, a.gw_params);
            H::gw_backreaction(rhs, st, i, j, k, a.lev, a.time, a.dt, a.dx, a.params,
                               a.gw_params);
        }
        if constexpr (KO == 2 || KO == 3) {
            /* the RKN and leapfrog epilogues take the momenta's rates alone */
            const bool all =
                a.epi == kEpiPlainRhs || a.epi == kEpiSsp0 || a.epi == kEpiSspAdd;
            sledgehamr::utils::constexpr_for<0, NP, 1>([&](auto q) {
                constexpr int m = PR::mom(q), n = PR::pos(q);
                r[m] += sledgehamr::kernels::KreissOligerDissipation<KO>(st, i, j, k, m, a.dx,
                                                                        a.ko_strength[m]);
                if (all)
                    r[n] += sledgehamr::kernels::KreissOligerDissipation<KO>(
                        st, i, j, k, n, a.dx, a.ko_strength[n]);
            });
            if constexpr (H::kNScalars % 2 == 1) { /* a field without a partner */
                constexpr int n = H::kNScalars - 1;
                r[n] += sledgehamr::kernels::KreissOligerDissipation<KO>(st, i, j, k, n, a.dx,
                                                                        a.ko_strength[n]);
            }
        }

        const long long lc = (i - glo.x) + (j - glo.y) * gx + (k - glo.z) * gxy;
        const long long sbase = b.off * NC + lc; /* state-layout element of comp 0 */
        long long oz = 0;
        if constexpr (SP) {
            if (k < b.lo[2] + a.ng) oz = a.per[2] * gxy;
            else if (k > b.hi[2] - a.ng) oz = -a.per[2] * gxy;
        }
        switch (EPI == kEpiAny ? a.epi : EPI) {
        case kEpiPlainRhs: {
#pragma unroll
            for (int n = 0; n < NC; ++n) a.out[sbase + n * gvol] = r[n];
            break;
        }
        case kEpiRknStage: {
            const long long kb = b.off * NP + lc;
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const double kq = r[PR::mom(q)];
                a.kout[kb + q * gvol] = kq;
                double y = a.y0[sbase + PR::pos(q) * gvol];
                const double m = a.y0[sbase + PR::mom(q) * gvol];
                y += a.c_mom * m;
                if constexpr (EPI == kEpiRknStage) {
                    y += a.c_k[0] * kq; /* no earlier K */
                } else {
                    for (int s = 0; s < a.nkin; ++s) y += a.c_k[s] * a.kin[s][kb + q * gvol];
                    y += a.c_k[a.nkin] * kq;
                }
                a.out[sbase + PR::pos(q) * gvol] = y;
                a.out[sbase + PR::mom(q) * gvol] = m;
            }
            break;
        }
        case kEpiRknFinal: {
            /* y1 = y0 + dt g and y1' = g + sum_s c_k2 K_s with the common
             * g = y0' + sum_s c_k K_s, c_k = dt bbar, c_k2 = dt (b - bbar):
             * a K_s with b = bbar (K_0 of RKN4) enters once, five FP64
             * instructions a pair instead of six.  The masks name the K_s
             * with a non-zero coefficient; bit nkin is the current stage's. */
            const long long kb = b.off * NP + lc;
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const double y = a.y0[sbase + PR::pos(q) * gvol];
                double g = a.y0[sbase + PR::mom(q) * gvol];
                if constexpr (EPI == kEpiRknFinal) { /* RKN4 */
                    const double k0 = a.kin[0][kb + q * gvol], k1 = a.kin[1][kb + q * gvol];
                    g += a.c_k[0] * k0;
                    g += a.c_k[1] * k1;
                    a.out[sbase + PR::pos(q) * gvol] = y + a.dt * g;
                    g += a.c_k2[1] * k1;
                    a.out[sbase + PR::mom(q) * gvol] = g + a.c_k2[2] * r[PR::mom(q)];
                    continue;
                }
                double d = a.c_k2[a.nkin] * r[PR::mom(q)];
                for (int s = 0; s < a.nkin; ++s) {
                    const double ks = a.kin[s][kb + q * gvol];
                    if (a.kmask >> s & 1u) g += a.c_k[s] * ks;
                    if (a.kmask2 >> s & 1u) d += a.c_k2[s] * ks;
                }
                if (a.kmask >> a.nkin & 1u) g += a.c_k[a.nkin] * r[PR::mom(q)];
                a.out[sbase + PR::pos(q) * gvol] = y + a.dt * g;
                a.out[sbase + PR::mom(q) * gvol] = g + d;
            }
            break;
        }
        case kEpiSsp0:
        case kEpiSspAdd: {
            const long long kb = b.off * NC + lc;
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                double kn = r[n];
                if (a.epi == kEpiSspAdd) kn += a.weight * a.kin[0][kb + n * gvol];
                if (a.kout) a.kout[kb + n * gvol] = kn;
                a.out[sbase + n * gvol] = 1. * a.y0[sbase + n * gvol] + a.c_out * kn;
            }
            break;
        }
        case kEpiLf0: {
            const long long kb = b.off * NP + lc;
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const double vh =
                    1. * a.y0[sbase + PR::mom(q) * gvol] + (a.dt / 2.) * r[PR::mom(q)];
                a.kout[kb + q * gvol] = vh;
                a.out[sbase + PR::pos(q) * gvol] = 1. * a.y0[sbase + PR::pos(q) * gvol] + a.dt * vh;
            }
            break;
        }
        case kEpiLf1: {
            const long long kb = b.off * NP + lc;
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                a.out[sbase + PR::mom(q) * gvol] =
                    1. * a.kin[0][kb + q * gvol] + (a.dt / 2.) * r[PR::mom(q)];
                a.out[sbase + PR::pos(q) * gvol] = a.state[sbase + PR::pos(q) * gvol];
            }
            break;
        }
        default:
            break;
        }
        /* a cell within ng of a face of a self-periodic box: its stored
         * values (every component, as a fill copies them) read back and
         * written to its periodic images, out of the epilogue so that no
         * value stays live across the image stores */
        if constexpr (SP) {
            if (((ox | oy | oz) != 0) && (EPI != kEpiAny || a.epi != kEpiPlainRhs)) {
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    const long long e = sbase + n * gvol;
                    const double v = a.out[e];
                    if (ox != 0) a.out[e + ox] = v;
                    if (oy != 0) {
                        a.out[e + oy] = v;
                        if (ox != 0) a.out[e + ox + oy] = v;
                    }
                    if (oz != 0) {
                        a.out[e + oz] = v;
                        if (ox != 0) a.out[e + ox + oz] = v;
                        if (oy != 0) {
                            a.out[e + oy + oz] = v;
                            if (ox != 0) a.out[e + ox + oy + oz] = v;
                        }
                    }
                }
            }
        }
    }
}

/* Tagging with the CPU semantics of SLEDGEHAMR_PRJ_TAG_WITH_TRUNCATION_CPU
 * (macros.h:489-566): mask(c) = user(c) OR (c has all-even indices AND some
 * component's TruncationModifier<n>(te) >= te_crit[n]).  The sequential
 * reference loop sets the 2x2x2 block of such an even cell and then clears
 * the seven odd cells again when it reaches them, so only the even cell
 * keeps the truncation-error tag; this kernel computes that end state
 * directly, without the racy block writes of the reference's GPU variant.
 * The counters follow the CPU statistics: total += user, and for every
 * even truncation-error cell total += 8 - user; trunc[n] += 8. */
template <class H, int NC>
__global__ void __launch_bounds__(kTileX *kTileY) tag_kernel(const __grid_constant__ TagArgs a) {
    const TileDev t = a.tiles[blockIdx.x];
    const BoxDev b = a.boxes[t.box];
    const int tid = threadIdx.x + kTileX * threadIdx.y;
    const int ty = tid / t.nx;
    const int i = t.x0 + (tid - ty * t.nx);
    const int j = t.y0 + ty;
    const bool inside = (ty < kThreads / t.nx && i <= b.hi[0] && j <= b.hi[1]);
    const int kend = min(t.z0 + t.nz - 1, b.hi[2]);
    const long long gx = b.gdim[0], gxy = gx * b.gdim[1];
    const amrex::Dim3 glo{b.glo[0], b.glo[1], b.glo[2]};
    const amrex::Dim3 ghi{b.glo[0] + b.gdim[0], b.glo[1] + b.gdim[1], b.glo[2] + b.gdim[2]};
    const amrex::Array4<const double> st(a.state + b.off * a.ncomp, gx, gxy, b.gvol, glo, ghi,
                                         a.ncomp);
    const amrex::Array4<const double> te(a.te ? a.te + b.off * a.ncomp : nullptr, gx, gxy,
                                         b.gvol, glo, ghi, a.ncomp);
    const int vx = b.hi[0] - b.lo[0] + 1, vy = b.hi[1] - b.lo[1] + 1;
    unsigned long long n_user = 0, n_total = 0;
    unsigned long long n_trunc[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n) n_trunc[n] = 0;
    if (inside) {
        for (int k = t.z0; k <= kend; ++k) {
            const bool user = H::tag(st, i, j, k, a.lev, a.time, a.dt, a.dx, a.params_tag);
            bool te_res = false;
            if (a.te && (i % 2 == 0) && (j % 2 == 0) && (k % 2 == 0)) {
                sledgehamr::utils::constexpr_for<0, NC, 1>([&](auto n) {
                    const double mte = H::template te_modifier<n>(
                        st, i, j, k, a.lev, a.time, a.dt, a.dx, te(i, j, k, n), a.params_mod);
                    if (mte >= a.te_crit[n]) {
                        te_res = true;
                        n_trunc[n] += 8;
                    }
                });
            }
            n_user += user;
            n_total += user;
            if (te_res) n_total += 8 - (int)user;
            const long long m = a.mask_off[t.box] + (i - b.lo[0]) +
                                (long long)vx * ((j - b.lo[1]) + (long long)vy * (k - b.lo[2]));
            a.mask[m] = (user || te_res) ? 1 : 0;
        }
    }
    /* warp sums, one atomic per warp and counter */
    const unsigned full = 0xffffffffu;
    for (int o = 16; o > 0; o >>= 1) {
        n_user += __shfl_down_sync(full, n_user, o);
        n_total += __shfl_down_sync(full, n_total, o);
#pragma unroll
        for (int n = 0; n < NC; ++n) n_trunc[n] += __shfl_down_sync(full, n_trunc[n], o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (n_total) atomicAdd(&a.counts[0], n_total);
        if (n_user) atomicAdd(&a.counts[1], n_user);
#pragma unroll
        for (int n = 0; n < NC; ++n)
            if (n_trunc[n]) atomicAdd(&a.counts[2 + n], n_trunc[n]);
    }
}

template <class H, bool GW, int KO, bool SP>
void launch_stage_epi(const StageLaunch &L, cudaStream_t s) {
    const dim3 block(kTileX, kTileY, 1), grid(L.ntiles, 1, 1);
    const StageArgs &a = L.args;
    /* instantiations of the RKN4 stages, both intermediate ones (no earlier
     * K with a non-zero coefficient) and the final one, and of the leapfrog's
     * with the tensor components */
    if constexpr (GW && KO == 0) {
        if (a.epi == kEpiLf0) {
            stage_kernel<H, GW, KO, SP, kEpiLf0><<<grid, block, 0, s>>>(a);
            return;
        }
        if (a.epi == kEpiLf1) {
            stage_kernel<H, GW, KO, SP, kEpiLf1><<<grid, block, 0, s>>>(a);
            return;
        }
    }
    if constexpr (!GW && KO == 0) {
        if (a.epi == kEpiRknStage && a.nkin == 0) {
            stage_kernel<H, GW, KO, SP, kEpiRknStage><<<grid, block, 0, s>>>(a);
            return;
        }
        if (a.epi == kEpiRknFinal && a.nkin == 2 && a.kmask == 3u && a.kmask2 == 6u) {
            stage_kernel<H, GW, KO, SP, kEpiRknFinal><<<grid, block, 0, s>>>(a);
            return;
        }
    }
    stage_kernel<H, GW, KO, SP><<<grid, block, 0, s>>>(a);
}

template <class H, bool GW>
void launch_stage_variant(const StageLaunch &L, cudaStream_t s) {
    switch (L.ko_order) {
    case 2: launch_stage_epi<H, GW, 2, false>(L, s); break;
    case 3: launch_stage_epi<H, GW, 3, false>(L, s); break;
    default:
        if (L.args.self_periodic) launch_stage_epi<H, GW, 0, true>(L, s);
        else launch_stage_epi<H, GW, 0, false>(L, s);
        break;
    }
}

template <class H>
cudaError_t launch_stage_impl(const StageLaunch &L, cudaStream_t s) {
    if (L.ntiles <= 0) return cudaSuccess;
    if (!L.with_gw) {
        launch_stage_variant<H, false>(L, s);
    } else {
        if constexpr (H::kHasGw) launch_stage_variant<H, true>(L, s);
        else return cudaErrorNotSupported;
    }
    return cudaGetLastError();
}

template <class H>
cudaError_t launch_tag_impl(const TagArgs &a, int ntiles, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    dim3 block(kTileX, kTileY, 1);
    if (a.ncomp == H::kNScalars) {
        tag_kernel<H, H::kNScalars><<<ntiles, block, 0, s>>>(a);
    } else if (a.ncomp == H::kNScalars + 12) {
        tag_kernel<H, H::kNScalars + 12><<<ntiles, block, 0, s>>>(a);
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

} // namespace sh

/* Defines the ProjectOps table `sh::project_<NAME>` for the project namespace
 * NS (after its hooks and SLEDGEHAMR_FINISH_SETUP) and registers it with the
 * library when it loads.  HAS_GW: the project
 * specialises GravitationalWavesRhs<true>; REACH: the largest neighbour
 * offset its hooks read (levels need at least that many ghost cells).
 * SH_DEFINE_PROJECT_OPTIONS also says whether the Rhs hooks read neighbours
 * of positions alone (POS; the momenta's ghost cells are then not filled
 * between stages), and names a host function
 * void fn(double *params, double time) that writes per-launch constants
 * behind the project's own parameters, for its hooks to read. */
#define SH_DEFINE_PROJECT(NAME, NS, HAS_GW, REACH)                              \
    SH_DEFINE_PROJECT_OPTIONS(NAME, NS, HAS_GW, REACH, false, nullptr)
#define SH_DEFINE_PROJECT_OPTIONS(NAME, NS, HAS_GW, REACH, POS, FN)             \
    namespace sh {                                                             \
    struct Hooks_##NAME : NS::ShHooks {                                        \
        static constexpr bool kHasGw = HAS_GW;                                 \
        static constexpr int kReach = REACH;                                   \
    };                                                                         \
    static const char *field_name_##NAME(int c) {                              \
        const auto &f = NS::ShHooks::fields();                                 \
        return c >= 0 && c < (int)f.size() ? f[c]->name.c_str() : nullptr;    \
    }                                                                          \
    extern const ProjectOps project_##NAME;                                    \
    const ProjectOps project_##NAME = {                                        \
        #NAME,                                                                 \
        NS::ShHooks::kNScalars,                                                \
        NS::ShHooks::kNFields,                                                 \
        HAS_GW,                                                                \
        REACH,                                                                 \
        &field_name_##NAME,                                                    \
        &launch_stage_impl<Hooks_##NAME>,                                      \
        &launch_tag_impl<Hooks_##NAME>,                                        \
        FN,                                                                    \
        POS};                                                                  \
    static const ProjectRegistrar registrar_##NAME(&project_##NAME);          \
    }

#endif // SH_STAGE_CUH_
