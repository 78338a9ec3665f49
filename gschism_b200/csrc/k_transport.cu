// Tracer transport, first-order upwind (computeTransport, schism_step.py:78-93; kernels
// meshdata.cu:6493-6665, 6739-6774, 6842-6863).
//
// The sub-cycling loop runs inside one cooperative launch: every member keeps its own
// remaining time and sub-step on the device (the reference reads minTransportDt back to the
// host once per sub-step).  The minimum admissible sub-step of a member is reduced with an
// integer atomicMin on the bit pattern of non-negative doubles, which is order-independent.
//
// The reference copies every element's tracers into a snapshot before each sub-step and reads
// the neighbours from it.  Here the two tracer arrays alternate instead: sub-step s reads one
// (etr for even s, prev for odd s) and writes the other, so no copy is made; after a member's
// last sub-step its result sits in prev when it took an odd number of sub-steps.  The implicit
// vertical advection runs after every member has finished sub-cycling, reads the result from
// where it sits and writes etr.
//
// Horizontal passes.  Levels are independent there, so a thread owns kRun consecutive levels of one
// element: enough threads for small meshes, and the element's side table is read once per run.  The
// admissible sub-step is a minimum over the member that nearly always allows the whole remaining time,
// so the pass that finds it also makes the update with that time; the update is made again, with the
// shorter sub-step, only for members whose minimum falls below it.
//
// Vertical pass.  A Thomas sweep per column; its coefficients are the same for
// every tracer, but on meshes too small to fill the GPU with columns a thread owns one tracer's column
// instead and forms them again.
//
// TVD (itr_met = 3; the reference has only upwind): flux-limited horizontal advection restated
// from Casulli & Zanolli (2005).  On a face between the upwind prism U and the downwind prism D
// the face value is C_U + psi(r)/2 (C_D - C_U), r = S_U / (|Q| (C_U - C_D)), S_U = sum over U's
// interior inflow faces g of |Q_g| (C_g - C_U).  A sub-step needs the inflow sums of
// the snapshot, the admissible sub-step (every update coefficient non-negative:
// dt <= V / sum_in |Q| (1 - psi/2 + sum_out psi/(2r))), and the update
// C_P += dt/V [sum_in |Q| (1 - psi/2)(C_U - C_P) + sum_out |Q| psi/2 (C_P - C_D)].  Limiter 0
// (psi = 0) reproduces the upwind scheme bit for bit.  The vertical solve optionally adds a
// constant diffusivity between prism centres.  This file is compiled with -fmad=false so that
// the limiter's branches see the same rounding as the FP64 CPU restatement.
//
// Vertical FCT (itr_met = 4: the TVD horizontal passes plus a flux-corrected vertical step; no
// counterpart in the reference either): Zalesak's (1979) flux-corrected transport with the
// implicit upwind solve as the low-order scheme.  After the Thomas sweep gives C^L, interior
// interface j of a column carries the anti-diffusive transfer a_j = dt |Qv| (C^L_{j+1} - C^L_j)/2
// (central minus upwind flux), scaled by min(R+ of the receiver, R- of the giver), R+/- =
// min(1, Q+/-/P+/-) from the prism's incoming / outgoing transfers P and its room to the bounds Q
// = V (C_max/min - C^L) over the prism and its column neighbours, of C^L and of the field before
// the vertical step.  The transfers are antisymmetric, so the column's tracer mass is unchanged,
// and no new extremum appears whatever the vertical Courant number.  The field before the step is
// kept in prev.
#include "dev_common.cuh"
#include "kernels.h"

namespace gs {

constexpr double kHuge = 1.79e+308;

struct TrArgs {
    double* rem;                 // [2][nmem] remaining time by parity
    unsigned long long* mindt;   // [2][nmem]
    int32_t* nsub;               // [nmem]
    unsigned* active;            // members still sub-cycling
    double dt;
    int maxsub;
};

__device__ __forceinline__ double evol(const Dev& d, int e, int k) {
    return d.area[e] * (d.ez[(size_t)(k + 1) * d.NE + e] - d.ez[(size_t)k * d.NE + e]);
}

// flux limiter psi(r): 0 none, 1 minmod, 2 Osher (beta = 2), 3 van Leer, 4 superbee; 0 for r <= 0,
// the limit value for r beyond 1e300
__device__ __forceinline__ double tvd_psi(int lim, double r) {
    if (!(r > 0.0)) return 0.0;
    if (!(r < 1.0e300)) return lim == 0 ? 0.0 : (lim == 1 ? 1.0 : 2.0);
    switch (lim) {
    case 1: return fmin(r, 1.0);
    case 2: return fmin(r, 2.0);
    case 3: return (r + r) / (1.0 + r);
    case 4: return fmax(fmin(2.0 * r, 1.0), fmin(r, 2.0));
    default: return 0.0;
    }
}

// psi of a face with upwind value cu, downwind value cd, flux magnitude aq and upwind inflow sum
// su; psir = psi / (2 r) (0 when psi = 0)
__device__ __forceinline__ double tvd_face(int lim, double su, double aq, double cu, double cd, double& psir) {
    const double dd = cu - cd;
    if (dd == 0.0) { psir = 0.0; return 0.0; }
    const double r = su / (aq * dd);
    const double psi = tvd_psi(lim, r);
    psir = (psi > 0.0) ? psi / (2.0 * r) : 0.0;
    return psi;
}

// Minimum of non-negative doubles (compared as their bit patterns) into slot[m] for each lane's
// member m (m < 0: none): a warp whose lanes share one member reduces with shuffles and issues
// one atomic, instead of one per element on the same word.  All 32 lanes must call it.
__device__ __forceinline__ void warp_min_to_member(unsigned long long* slot, int m, double v) {
    const unsigned full = 0xffffffffu;
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int m0 = __shfl_sync(full, m, 0);
    if (__all_sync(full, m == m0 || m < 0)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long w = __shfl_xor_sync(full, b, o);
            b = w < b ? w : b;
        }
        if ((threadIdx.x & 31) == 0 && m0 >= 0) atomicMin(slot + m0, b);
    } else if (m >= 0) {
        atomicMin(slot + m, b);
    }
}

// The three sides of element e as the horizontal update needs them (loaded once per element).
struct ElemSides {
    int s[3], kbs[3], nb[3];
    double sg[3];
    bool nbwet[3];
    int8_t bt[3];
};

__device__ __forceinline__ ElemSides elem_sides(const Dev& d, int e) {
    ElemSides q;
    const int NE = d.NE, NS = d.NS;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int s = d.es[j * NE + e];
        q.s[j] = s;
        q.kbs[j] = d.kbs[s];
        const int e0 = d.se[s], e1 = d.se[NS + s];
        const int nb = (e0 == e) ? e1 : e0;
        q.nb[j] = nb;
        q.nbwet[j] = nb >= 0 && !d.edry[nb];
        q.sg[j] = (double)d.ssgn[j * NE + e];
        q.bt[j] = d.sbt[s];
    }
    return q;
}

// Flux-corrected vertical step of one tracer of element e's column (FCT above): cl holds C^L and co the
// field before the vertical step; streamed from the bed up with a window of three prisms, each prism's
// corrected value written two levels behind the read.  The expression order is the CPU restatement's.
__device__ void vertical_fct(const Dev& d, const Phys& P, int e, double dt, const double* co, double* cl) {
    const int NE = d.NE, nvrt = P.nvrt;
    const int k0 = d.kbe[e] + 1;
    const int n = nvrt - k0;
    if (n < 2) return;
    // prisms i-2 (m2) and i-1 (m1); raw transfer of face (i-2, i-1); scaled transfer of face
    // (i-3, i-2); limiter factors of prism i-2
    double cl_m2 = 0.0, cl_m1 = 0.0, co_m2 = 0.0, co_m1 = 0.0, v_m2 = 1.0, v_m1 = 1.0;
    double a_m2 = 0.0, fa_m3 = 0.0, rp_m2 = 1.0, rm_m2 = 1.0;
    for (int i = 0; i <= n + 1; i++) {
        double cl_i = 0.0, co_i = 0.0, v_i = 1.0, a_m1 = 0.0;
        if (i < n) {
            const size_t ix = (size_t)(k0 + i) * NE + e;
            cl_i = cl[ix]; co_i = co[ix]; v_i = evol(d, e, k0 + i - 1);
            if (i >= 1) a_m1 = 0.5 * dt * fabs(d.Qv[(size_t)(k0 + i - 1) * NE + e]) * (cl_i - cl_m1);
        }
        double rp_m1 = 1.0, rm_m1 = 1.0, fa_m2 = 0.0;
        if (i >= 1 && i <= n) {
            // limiter factors of prism i-1: transfers a_m2 (below) and a_m1 (above)
            double cmax = fmax(cl_m1, co_m1), cmin = fmin(cl_m1, co_m1);
            if (i >= 2) { cmax = fmax(cmax, fmax(cl_m2, co_m2)); cmin = fmin(cmin, fmin(cl_m2, co_m2)); }
            if (i < n) { cmax = fmax(cmax, fmax(cl_i, co_i)); cmin = fmin(cmin, fmin(cl_i, co_i)); }
            const double pp = fmax(0.0, a_m2) + fmax(0.0, -a_m1);
            const double pm = fmin(0.0, a_m2) + fmin(0.0, -a_m1);
            const double qp = v_m1 * (cmax - cl_m1), qm = v_m1 * (cmin - cl_m1);
            rp_m1 = pp > 0.0 ? fmin(1.0, qp / pp) : 1.0;
            rm_m1 = pm < 0.0 ? fmin(1.0, qm / pm) : 1.0;
            if (i >= 2) fa_m2 = a_m2 * (a_m2 > 0.0 ? fmin(rp_m1, rm_m2) : fmin(rm_m1, rp_m2));
        }
        if (i >= 2) cl[(size_t)(k0 + i - 2) * NE + e] = cl_m2 + (fa_m3 - fa_m2) / v_m2;
        fa_m3 = fa_m2; a_m2 = a_m1; rp_m2 = rp_m1; rm_m2 = rm_m1;
        cl_m2 = cl_m1; co_m2 = co_m1; v_m2 = v_m1;
        cl_m1 = cl_i; co_m1 = co_i; v_m1 = v_i;
    }
}

// Vertical step of every wet element once its member has finished sub-cycling: after n sub-steps the
// horizontal result is in prev when n is odd, in etr when it is even; the step's result goes to etr.  A
// thread owns NT tracers of one column, tracer group in blockIdx.y.
//   verticalAdvectionUpdate, meshdata.cu:6611-6665 (upwind: phi = 0), with the arithmetic of the
// reference's tridag_sch<1> (meshdata.cu:3664-3716) row by row; with FCT the flux correction follows.
//
// The eliminated super-diagonal goes to the group's own scratch slice: prev's where upwind leaves it
// free (its values are read before they are overwritten), the inflow sums' with TVD.  The next level's
// inputs are loaded ahead of a level's two dependent divisions.  720k columns of 30 levels, 2 tracers:
// 386 us for 2.0 GB of loads and stores, some of which the L2 serves (318k columns: DRAM at 0.43 of the measured
// copy rate, a third of the warps, waiting for loads); with the column in shared memory, which moves half of
// that, 531 us (too few threads fit).
template <int NT, bool TVD, bool FCT>
__global__ void __launch_bounds__(128) k_vertical(Dev d, Phys P, const int32_t* nsub, double dt) {
    const int NE = d.NE, nvrt = P.nvrt;
    const size_t trs = (size_t)nvrt * NE, at = (size_t)blockIdx.y * NT * trs;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < NE; e += gridDim.x * blockDim.x) {
        if (d.edry[e]) continue;
        const int kb = d.kbe[e], k0 = kb + 1;
        if (k0 >= nvrt) continue;        // a wet element has at least one layer
        const double* src = ((nsub[d.elem_member[e]] & 1) ? d.prev : d.etr) + at;
        double* dst = d.etr + at;
        double* scr = (TVD ? d.tvds : d.prev) + at;
        double* keep = d.prev + at;      // FCT: the field before the step
        const double ar = d.area[e];
        double bet = 0.0, cprev = 0.0, up[NT], c[NT];
        // heights of levels k - 2 .. k, fluxes of k - 1 and k, tracers of k
        double zmm = 0.0, zm = d.ez[(size_t)kb * NE + e], zc = d.ez[(size_t)k0 * NE + e];
        double qm = d.Qv[(size_t)kb * NE + e], qk = d.Qv[(size_t)k0 * NE + e];
#pragma unroll
        for (int t = 0; t < NT; t++) c[t] = src[t * trs + (size_t)k0 * NE + e];
        for (int k = k0; k < nvrt; k++) {
            const bool top = k == nvrt - 1;
            const size_t ix = (size_t)k * NE + e;
            double zp = 0.0, qp = 0.0, cn[NT];
            if (!top) { zp = d.ez[ix + NE]; qp = d.Qv[ix + NE]; }
#pragma unroll
            for (int t = 0; t < NT; t++) cn[t] = top ? 0.0 : src[t * trs + ix + NE];
            double alow = 0.0, cupp = 0.0, bdia = 0.0;
            const double dbv = dt / (ar * (zc - zm));
            bdia += 1.0;
            if (!top && qk < 0.0) { const double tmp = dbv * fabs(qk); cupp -= tmp; bdia += tmp; }
            if (k - 1 != kb && qm > 0.0) { const double tmp = dbv * fabs(qm); alow -= tmp; bdia += tmp; }
            if (P.dfh0 > 0.0) {
                // diffusion across the interfaces with the prisms above and below, over the distance
                // between prism centres
                if (!top) {
                    const double tmp = dbv * (P.dfh0 * ar / (0.5 * (zp - zm)));
                    cupp -= tmp; bdia += tmp;
                }
                if (k - 1 != kb) {
                    const double tmp = dbv * (P.dfh0 * ar / (0.5 * (zc - zmm)));
                    alow -= tmp; bdia += tmp;
                }
            }
            double gam = 0.0;
            if (k == k0) {
                bet = bdia;
            } else {
                gam = cprev / bet;
                bet = bdia - alow * gam;
            }
#pragma unroll
            for (int t = 0; t < NT; t++) {
                if (FCT) keep[t * trs + ix] = c[t];
                up[t] = k == k0 ? (c[t] * 1.0) / bet : (c[t] * 1.0 - alow * up[t]) / bet;
                dst[t * trs + ix] = up[t];
            }
            if (k != k0) scr[ix] = gam;
            cprev = cupp;
            zmm = zm; zm = zc; zc = zp; qm = qk; qk = qp;
#pragma unroll
            for (int t = 0; t < NT; t++) c[t] = cn[t];
        }
        // back substitution: u_j -= gam_{j+1} u_{j+1}; up holds the top level's value
        for (int k = nvrt - 2; k >= k0; k--) {
            const double gam = scr[(size_t)(k + 1) * NE + e];
            const size_t ix = (size_t)k * NE + e;
#pragma unroll
            for (int t = 0; t < NT; t++) {
                up[t] = dst[t * trs + ix] - gam * up[t];
                dst[t * trs + ix] = up[t];
            }
        }
        if (FCT) {
#pragma unroll
            for (int t = 0; t < NT; t++) {
                vertical_fct(d, P, e, dt, keep + t * trs, dst + t * trs);
                up[t] = dst[t * trs + (size_t)k0 * NE + e];
            }
        }
        // levels at and below the bed take the bottom prism's value
        for (int k = 0; k <= kb; k++)
#pragma unroll
            for (int t = 0; t < NT; t++) dst[t * trs + (size_t)k * NE + e] = up[t];
    }
}

// Levels of a horizontal work item: 160k nodes of 30 levels, 2 tracers, upwind 258 us with 6, 245 with 8,
// 240 with 10; 40k nodes of 40 levels, 5 tracers, TVD 716, 684 and 701 us.  (One thread per column and
// separate passes for the sub-step and the update: 540 us of 719 with the vertical sweep, and 3.5 ms.)
constexpr int kRun = 8;

// Horizontal update of the levels [ka, ke) of element e over dtb, and the smallest admissible sub-step
// of those levels (both from one read of the faces).  UPDATE: write the result to dst.  Neighbours are
// read whatever the flux's direction, so that their loads do not wait for it.
// NT tracers from slice at on.
//   upwind: horizontalAdvectionPrepare and horizontalAdvectionUpdate, meshdata.cu:6493-6609
template <int NT, bool TVD, bool UPDATE>
__device__ __forceinline__ double horizontal_run(const Dev& d, const Phys& P, int e, int ka, int ke, size_t at,
                                                 const double* src, double* dst, double dtb) {
    const int NE = d.NE, NS = d.NS, lim = P.tvd_limiter;
    const size_t trs = (size_t)P.nvrt * NE;
    const double* tv = d.tvds + at;
    src += at;
    dst += at;
    const ElemSides q = elem_sides(d, e);
    const double ar = d.area[e];
    double md = kHuge, zlo = d.ez[(size_t)(ka - 1) * NE + e];
    for (int k = ka; k < ke; k++) {
        const size_t ix = (size_t)k * NE + e;
        const double zhi = d.ez[ix];
        const double vol = ar * (zhi - zlo), dbv = dtb / vol;
        zlo = zhi;
        double fq[3], sQ[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            fq[j] = k > q.kbs[j] ? d.Qh[(size_t)k * NS + q.s[j]] : 0.0;
            sQ[j] = k > q.kbs[j] ? q.sg[j] * fq[j] : 0.0;
            fq[j] = fabs(fq[j]);
        }
        if constexpr (!TVD) {
            double in = 0.0;
#pragma unroll
            for (int j = 0; j < 3; j++)
                if (sQ[j] < 0.0 && q.nbwet[j] && q.bt[j] != 1) in += fq[j];
            const double pd = (in == 0.0) ? kHuge : vol / in * (1.0 - 1.0e-6);
            md = fmin(md, pd);
        }
        if (TVD || UPDATE) {
#pragma unroll
            for (int t = 0; t < NT; t++) {
                const double own = src[t * trs + ix];
                double cn[3];
#pragma unroll
                for (int j = 0; j < 3; j++)
                    cn[j] = q.nbwet[j] ? src[t * trs + (size_t)k * NE + q.nb[j]] : 0.0;
                double psi[3];
                if constexpr (TVD) {
                    const double so_own = tv[t * trs + ix];
                    double sn[3], so = 0.0, den = 0.0;
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        sn[j] = q.nbwet[j] ? tv[t * trs + (size_t)k * NE + q.nb[j]] : 0.0;
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        psi[j] = 0.0;
                        if (!q.nbwet[j]) continue;
                        double psir;
                        if (sQ[j] > 0.0) {
                            psi[j] = tvd_face(lim, so_own, fq[j], own, cn[j], psir);
                            so += psir;
                        } else if (sQ[j] < 0.0) {
                            psi[j] = tvd_face(lim, sn[j], fq[j], cn[j], own, psir);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        if (q.nbwet[j] && sQ[j] < 0.0) den += fq[j] * (1.0 - 0.5 * psi[j] + so);
                    const double pd = (den == 0.0) ? kHuge : vol / den * (1.0 - 1.0e-6);
                    md = fmin(md, pd);
                }
                if (UPDATE) {
                    double adv = own;
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        const double coef = dbv * fq[j];
                        if (sQ[j] < 0.0) {
                            if (q.nbwet[j]) {
                                if (TVD) adv += coef * (1.0 - 0.5 * psi[j]) * (cn[j] - own);
                                else adv += coef * (cn[j] - own);
                            } else if (q.bt[j] == 2) {
                                // the reference's open-boundary inflow: the running value
                                adv += coef * (adv - own);
                            }
                        } else if (TVD && sQ[j] > 0.0 && q.nbwet[j]) {
                            adv += coef * (0.5 * psi[j]) * (own - cn[j]);
                        }
                    }
                    dst[t * trs + ix] = adv;
                }
            }
        }
    }
    return md;
}

// TVD inflow sums of the levels [ka, ke): S = sum over interior inflow faces of |Q| (C_nb - C), side order
template <int NTR>
__device__ __forceinline__ void inflow_run(const Dev& d, const Phys& P, int e, int ka, int ke, const double* src) {
    const int NE = d.NE, NS = d.NS;
    const size_t trs = (size_t)P.nvrt * NE;
    const ElemSides q = elem_sides(d, e);
    for (int k = ka; k < ke; k++) {
        const size_t ix = (size_t)k * NE + e;
        double own[NTR], su[NTR];
#pragma unroll
        for (int t = 0; t < NTR; t++) { own[t] = src[t * trs + ix]; su[t] = 0.0; }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (k <= q.kbs[j] || !q.nbwet[j]) continue;
            const double fq = d.Qh[(size_t)k * NS + q.s[j]];
            const size_t nx = (size_t)k * NE + q.nb[j];
#pragma unroll
            for (int t = 0; t < NTR; t++) {
                const double cn = src[t * trs + nx];
                if (q.sg[j] * fq < 0.0) su[t] += fabs(fq) * (cn - own[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < NTR; t++) d.tvds[t * trs + ix] = su[t];
    }
}

// f(element or -1, member, group, first level, end level) over the work items (tracer group, level run,
// element) of the grid; every lane of a warp calls it together
template <typename F>
__device__ __forceinline__ void for_runs(const Dev& d, int nvrt, int groups, F f) {
    const int lane = threadIdx.x & 31, NE = d.NE, nblk = (NE + 31) / 32, runs = (nvrt - 1 + kRun - 1) / kRun;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (long long w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < (long long)nblk * runs * groups; w += nw) {
        const int gr = (int)(w / nblk), g = gr / runs, r = gr - g * runs, e = 32 * (int)(w - (long long)gr * nblk) + lane;
        const bool ok = e < NE && !d.edry[e];
        const int m = ok ? d.elem_member[e] : -1;
        const int ka = ok ? max(d.kbe[e] + 1, 1 + r * kRun) : 0, ke = ok ? min(nvrt, 1 + (r + 1) * kRun) : 0;
        f(ka < ke ? e : -1, m, g, ka, ke);
    }
}

// Upwind shares the faces' fluxes between the tracers; with TVD the limiters dominate, and a work item
// takes one tracer (more threads).  At 64 registers both spill (upwind 56 to 200 bytes of stores, TVD 396 to
// 460), and four blocks per SM are still the best split: the transport step of 40k nodes, 40 levels, 5
// tracers, TVD takes 970 us at four, 1,028 at three and 1,196 at two; of 250k nodes, 30 levels, upwind 637, 695
// and 826.
template <int NTR, bool TVD>
__global__ void __launch_bounds__(256, 4) k_transport(Dev d, Phys P, TrArgs T) {
    constexpr int NT = TVD ? 1 : NTR, groups = NTR / NT;
    const size_t gs = (size_t)NT * P.nvrt * d.NE;
    const int nvrt = P.nvrt, nmem = d.nmem;
    const int G = gridDim.x * blockDim.x;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long seed = (unsigned long long)__double_as_longlong(1e34);
    for (int m = gid; m < nmem; m += G) {
        T.rem[m] = T.dt; T.rem[nmem + m] = T.dt;
        T.mindt[m] = seed; T.mindt[nmem + m] = seed;
        T.nsub[m] = 0;
    }
    if (gid == 0) *T.active = (unsigned)nmem;
    if (!grid_sync(d.bar, d.err, d.wait_polls)) return;
    for (int sub = 0; sub < T.maxsub; sub++) {
        if (*((volatile unsigned*)T.active) == 0u) break;
        const int par = sub & 1, nxt = par ^ 1;
        const double* src = par ? d.prev : d.etr;     // the sub-step's snapshot
        double* dst = par ? d.etr : d.prev;
        const volatile double* rem = T.rem + par * nmem;
        const volatile unsigned long long* mind = T.mindt + par * nmem;
        if (TVD) {
            for_runs(d, nvrt, 1, [&](int e, int m, int, int ka, int ke) {
                if (e >= 0 && rem[m] > 0.0) inflow_run<NTR>(d, P, e, ka, ke, src);
            });
            if (!grid_sync(d.bar, d.err, d.wait_polls)) return;
        }
        // admissible sub-step, and on the first sub-step the update over the whole time (later ones
        // follow a minimum that was shorter than the time left, so it is not tried again)
        for_runs(d, nvrt, groups, [&](int e, int m, int g, int ka, int ke) {
            double md = kHuge;
            const double left = m >= 0 ? rem[m] : 0.0;
            int mm = -1;
            if (e >= 0 && left > 0.0) {
                mm = m;
                md = sub == 0 ? horizontal_run<NT, TVD, true>(d, P, e, ka, ke, g * gs, src, dst, left)
                              : horizontal_run<NT, TVD, false>(d, P, e, ka, ke, g * gs, src, dst, left);
            }
            warp_min_to_member(T.mindt + par * nmem, mm, md);
        });
        if (!grid_sync(d.bar, d.err, d.wait_polls)) return;
        // the update with dtb = min(remaining, min maxDt) where it has not been made with it
        for_runs(d, nvrt, groups, [&](int e, int m, int g, int ka, int ke) {
            if (e < 0) return;
            const double left = rem[m];
            if (!(left > 0.0)) return;
            const double mdt = __longlong_as_double((long long)mind[m]);
            if (sub == 0 && mdt >= left) return;
            horizontal_run<NT, TVD, true>(d, P, e, ka, ke, g * gs, src, dst, fmin(left, mdt));
        });
        // member bookkeeping; a finished member stays finished (its remaining time moves to the next
        // parity slot, which still holds the value from before its last sub-step)
        for (int m = gid; m < nmem; m += G) {
            const double left = rem[m];
            if (!(left > 0.0)) { T.rem[nxt * nmem + m] = left; continue; }
            const double mdt = __longlong_as_double((long long)mind[m]);
            const double dtb = fmin(left, mdt);
            T.rem[nxt * nmem + m] = left - dtb;
            T.mindt[nxt * nmem + m] = seed;
            T.nsub[m] = sub + 1;
            if (!((left - dtb) > 0.0)) atomicSub(T.active, 1u);
        }
        if (!grid_sync(d.bar, d.err, d.wait_polls)) return;
    }
}

// Tracer mass budget of one member (elements [e0, e1)): per tracer, the sum over wet prisms of
// volume x concentration in FP64 with Neumaier's compensated summation.  Every thread sums its
// prisms, the block merges its threads in a fixed tree and a final one-thread pass merges the
// blocks in order: the grid is fixed (kMassBlocks), so the result does not depend on the GPU.
__device__ __forceinline__ void neumaier_add(double& s, double& c, double v) {
    const double t = s + v;
    if (fabs(s) >= fabs(v)) c += (s - t) + v;
    else c += (v - t) + s;
    s = t;
}

__global__ void __launch_bounds__(256) k_tracer_mass(Dev d, int nvrt, int ntr, int e0, int e1, double* part) {
    __shared__ double sh_s[256], sh_c[256];
    const int tid = threadIdx.x, NE = d.NE;
    for (int t = 0; t < ntr; t++) {
        double s = 0.0, c = 0.0;
        for (int e = e0 + blockIdx.x * blockDim.x + tid; e < e1; e += gridDim.x * blockDim.x) {
            if (d.edry[e]) continue;
            for (int k = d.kbe[e] + 1; k < nvrt; k++)
                neumaier_add(s, c, evol(d, e, k - 1) * d.etr[((size_t)t * nvrt + k) * NE + e]);
        }
        sh_s[tid] = s; sh_c[tid] = c;
        __syncthreads();
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if (tid < w) {
                double a = sh_s[tid], ca = sh_c[tid];
                neumaier_add(a, ca, sh_s[tid + w]);
                sh_s[tid] = a; sh_c[tid] = ca + sh_c[tid + w];
            }
            __syncthreads();
        }
        if (tid == 0) {
            part[((size_t)blockIdx.x * ntr + t) * 2] = sh_s[0];
            part[((size_t)blockIdx.x * ntr + t) * 2 + 1] = sh_c[0];
        }
        __syncthreads();
    }
}

__global__ void k_tracer_mass_final(int nblk, int ntr, const double* part, double* out) {
    const int t = threadIdx.x;
    if (t >= ntr) return;
    double s = 0.0, c = 0.0;
    for (int b = 0; b < nblk; b++) {
        neumaier_add(s, c, part[((size_t)b * ntr + t) * 2]);
        c += part[((size_t)b * ntr + t) * 2 + 1];
    }
    out[t] = s + c;
}

cudaError_t launch_tracer_mass(const Dev& d, const Phys& P, int e0, int e1, double* part, double* out,
                               cudaStream_t st) {
    k_tracer_mass<<<kMassBlocks, 256, 0, st>>>(d, P.nvrt, P.ntr, e0, e1, part);
    k_tracer_mass_final<<<1, 32, 0, st>>>(kMassBlocks, P.ntr, part, out);
    return cudaGetLastError();
}

// levels of a node that one thread sums
template <int NTR>
constexpr int nodal_run() { return NTR <= 4 ? 3 : 2; }

// nodalTracerUpdate, meshdata.cu:6739-6774 (node-centred gather, no atomics).  A thread owns a run of
// levels of one node, run in blockIdx.y: an element's index, wetness, area and bed are looked up once
// for the run, and the loads of all its levels are in flight together.  Each (node, level) sums its
// elements in the same order as a node-by-node loop.  (160k nodes, 30 levels, 2 tracers: 239 us with one
// level per thread, 167 with runs of 3, 174 with runs of 5.)
template <int NTR>
__global__ void __launch_bounds__(kGatherThreads) k_nodal_tracer(Dev d, Phys P) {
    constexpr int R = nodal_run<NTR>();
    const int NP = d.NP, NE = d.NE, nvrt = P.nvrt, ivrt = nvrt - 1, ka = blockIdx.y * R;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NP; i += gridDim.x * blockDim.x) {
        if (d.ndry[i]) continue;
        const int q0 = d.nne_s[i], q1 = d.nne_s[i + 1];
        double sum[NTR][R];
#pragma unroll
        for (int t = 0; t < NTR; t++)
#pragma unroll
            for (int r = 0; r < R; r++) sum[t][r] = 0.0;
        double sumA = 0.0;
        for (int q = q0; q < q1; q++) {
            const int e = d.nne[q];
            if (d.edry[e]) continue;
            const int kb = d.kbe[e];
            const double A = d.area[e];
            // heights of levels ka - 1 .. ka + R and tracers of ka .. ka + R, held inside the column
            double z[R + 2], c[NTR][R + 1];
#pragma unroll
            for (int r = 0; r < R + 2; r++) z[r] = d.ez[(size_t)min(max(ka - 1 + r, kb), ivrt) * NE + e];
#pragma unroll
            for (int t = 0; t < NTR; t++) {
                const double* tr = d.etr + (size_t)t * nvrt * NE;
#pragma unroll
                for (int r = 0; r < R + 1; r++) c[t][r] = tr[(size_t)min(max(ka + r, kb + 1), ivrt) * NE + e];
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int k = ka + r;
                // the top level, and levels at or below the bed, take one prism's value
                const bool one = k >= ivrt || k <= kb;
                const double zrat = one ? 0.0 : (z[r + 2] - z[r + 1]) / (z[r + 2] - z[r]);
#pragma unroll
                for (int t = 0; t < NTR; t++)
                    sum[t][r] += A * ((1.0 - zrat) * (one ? c[t][r] : c[t][r + 1]) + zrat * c[t][r]);
            }
            sumA += A;
        }
        if (sumA == 0.0) continue;
        const double inv = 1.0 / sumA;
#pragma unroll
        for (int t = 0; t < NTR; t++)
#pragma unroll
            for (int r = 0; r < R; r++)
                if (ka + r < nvrt) d.tr[((size_t)t * nvrt + ka + r) * NP + i] = inv * sum[t][r];
    }
}

// All tracers of a column in one thread when there are columns enough to keep the SMs busy (heights and fluxes
// are then read once), one tracer per thread below that.  The whole transport step, one tracer and all per
// thread, us: 10k elements of 40 levels, 5 tracers, TVD 200 and 253; 20k elements of 23 levels, 3 tracers, FCT
// 191 and 236; 51k elements of 30 levels, 2 tracers, upwind 135 and 141, of 40 levels, 5 tracers, TVD 647 and
// 660; 79k elements, the same two, 205 and 195, 970 and 946; 179k elements 389 and 369, 2,190 and 2,077.
constexpr int kColumnsPerSM = 448;

template <int NTR, bool TVD, bool FCT>
static void launch_vertical(const Dev& d, const Phys& P, double dt, cudaStream_t st, int nsm) {
    const int b = 128, g = std::max(1, std::min((d.NE + b - 1) / b, nsm * 16));
    if (NTR > 1 && d.NE < nsm * kColumnsPerSM)
        k_vertical<1, TVD, FCT><<<dim3(g, NTR), b, 0, st>>>(d, P, d.mem_nsub, dt);
    else
        k_vertical<NTR, TVD, FCT><<<dim3(g, 1), b, 0, st>>>(d, P, d.mem_nsub, dt);
}

template <int NTR>
static cudaError_t launch_ntr(const Dev& d, const Phys& P, TrArgs& T, cudaStream_t st, int nsm, const LaunchShape& nt) {
    // the TVD passes live in their own instantiation, so the upwind one keeps its smaller
    // register budget and its occupancy
    const void* fn = P.tvd ? (const void*)k_transport<NTR, true> : (const void*)k_transport<NTR, false>;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, 0);
    if (per_sm < 1) per_sm = 1;
    if (per_sm > 4) per_sm = 4;
    const long long items = (long long)((d.NE + 31) / 32) * ((P.nvrt - 1 + kRun - 1) / kRun) * (P.tvd ? NTR : 1);
    const int grid = (int)std::max(1LL, std::min((long long)nsm * per_sm, (items + 7) / 8));
    Dev dd = d;
    Phys pp = P;
    void* args[] = {&dd, &pp, &T};
    cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(256), args, 0, st);
    if (e != cudaSuccess) return e;
    if (P.tvd_vert) launch_vertical<NTR, true, true>(d, P, T.dt, st, nsm);
    else if (P.tvd) launch_vertical<NTR, true, false>(d, P, T.dt, st, nsm);
    else launch_vertical<NTR, false, false>(d, P, T.dt, st, nsm);
    k_nodal_tracer<NTR><<<dim3(grid_of(d.NP, nt, nsm), (P.nvrt + nodal_run<NTR>() - 1) / nodal_run<NTR>()),
                          nt.block, 0, st>>>(d, P);
    return cudaGetLastError();
}

// k_nodal_tracer (shapes above kGatherThreads are entered as that)
int transport_max_threads(int) { return 1024; }

cudaError_t launch_transport(const Dev& d, const Phys& P, double dt, cudaStream_t st, int nsm, const LaunchTable& L) {
    if (P.ntr <= 0) return cudaSuccess;
    TrArgs T;
    T.rem = d.mem_rem; T.mindt = d.mem_mindt; T.nsub = d.mem_nsub; T.active = (unsigned*)(d.mem_mindt + 2 * d.nmem);
    T.dt = dt; T.maxsub = 100000;
    static_assert(kMaxTracers == 8, "one instantiation per tracer count");
    switch (P.ntr) {
    case 1: return launch_ntr<1>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    case 2: return launch_ntr<2>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    case 3: return launch_ntr<3>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    case 4: return launch_ntr<4>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    case 5: return launch_ntr<5>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    case 6: return launch_ntr<6>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    case 7: return launch_ntr<7>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    default: return launch_ntr<8>(d, P, T, st, nsm, L.k[LK_NODAL_TRACER]);
    }
}

}  // namespace gs
