// Mixed-precision Jacobi-PCG on a caller's CSR matrix (gs_jcg with GS_FP32_IR): FP64 refinement sweeps
// r = b - A x, x += d around an FP32 solve of A d = r, one persistent cooperative launch.  (A context's
// refinement solve, whose rows have a spatial order, is jcg_mg.cu.)
//
// The inner solve is the single-reduction form of Jacobi-PCG (Chronopoulos and Gear, 1989): with
// u = D^-1 r and w = A u the recurrences
//   s_i = w_i + beta_i s_{i-1},   p_i = u_i + beta_i p_{i-1},   d += alpha_i p_i,
//   r_{i+1} = r_i - alpha_i s_i,  w_{i+1} = A u_{i+1},
//   gamma = (r, u), delta = (w, u),  beta_i = gamma_i / gamma_{i-1},
//   alpha_i = gamma_i / (delta_i - beta_i gamma_i / alpha_{i-1})
// need one grid-wide reduction per iteration.  The vectors are kept scaled by D^-1 and the FP32 matrix
// copy holds D^-1 A; a row's (u, w, s, p) travel together, double-buffered by iteration parity.
//
// An iteration is bound by the latency between two barriers.  The matrix of a block's rows stays in
// shared memory for the whole solve, and w_{i+1} = A u - alpha (A w + beta A s) is formed from three
// products that are gathered while alpha and beta are still being added up, so the reduction and the
// gathers overlap.
#include <algorithm>

#include "jcg_share.cuh"
#include "jcg_work.h"
#include "kernels.h"

namespace gs {

namespace {

struct View32 : SolveView {
    int n;
    const int32_t *indptr, *indices;
    const double *A, *b, *invD;
    const float *A32, *diag;                 // D^-1 A, D
    double* x;
    float4* uw[2];                           // (u, w, s, p) by parity
    float* d;
    int32_t *mdone, *mouter, *status;
    int stall_member;
    int cache_entries;                       // matrix entries a block can hold (8 bytes each)
    double rtol, inner_rtol;
    int inner_maxiter, check_every;
};

constexpr int kNone = 0x7fffffff;            // shift of a block whose entries are not cached
struct RowState {
    float4 o;                                // (u, w, s, p) of the row
    float au, aw, as;                        // D^-1 A (u, w, s)
    float d, D;
};

template <bool HELD>
__device__ __forceinline__ RowState row_state(const View32& J, const float* cv, const int32_t* ci, int shift, int i,
                                              const float4* uw) {
    RowState R;
    R.au = R.aw = R.as = 0.0f;
    const int a = __ldg(J.indptr + i), n = __ldg(J.indptr + i + 1) - a;
    R.o = uw[i]; R.d = J.d[i]; R.D = __ldg(J.diag + i);
    for (int k0 = 0; k0 < n; k0 += 4) {
        int c[4];
        float v[4];
        float4 y[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool ok = k0 + k < n;
            const int at = a + k0 + k;
            if (HELD && shift != kNone) {
                c[k] = ok ? ci[at - shift] : i;
                v[k] = ok ? cv[at - shift] : 0.0f;
            } else {
                c[k] = ok ? __ldg(J.indices + at) : i;
                v[k] = ok ? __ldg(J.A32 + at) : 0.0f;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) y[k] = uw[c[k]];
#pragma unroll
        for (int k = 0; k < 4; k++) { R.au += v[k] * y[k].x; R.aw += v[k] * y[k].y; R.as += v[k] * y[k].z; }
    }
    return R;
}

// f(row, tile sums) over the block's rows, slice j by warp j % 16; one partial per tile and kind
template <int NV, typename F>
__device__ __forceinline__ void rows_sum(const View32& J, const Part& q, TileSums& ts, int k0, F f) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, per = q.tr / 32;
    for (int a = q.a; a < q.e; a += kTileRun) {
        const int e = min(q.e, a + kTileRun);
        const int s0 = a * per, s1 = min(e * per, (q.rows + 31) / 32);
        clear_tiles<NV>(ts, e - a);
        double v[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = 0.0;
        int tile = -1;
        for (int s = s0 + ((w - s0) & (kT / 32 - 1)); s < s1; s += kT / 32) {
            if (s / per != tile) {
                if (tile >= 0) put_warp<NV>(ts, tile - a, v);
                tile = s / per;
            }
            const int o = 32 * s + lane;
            if (o < q.rows) f(q.row0 + o, s, v);
        }
        if (tile >= 0) put_warp<NV>(ts, tile - a, v);
        put_tiles<NV>(J, q, a, e, ts, k0);
    }
}

#define SYNC32() do { if (!bar.sync(J, stall)) return; } while (0)

// HELD: one block per SM, the matrix in shared memory, the products of a thread's first four rows
// gathered before the totals are known.  Otherwise (a matrix larger than the chip's shared memory) two
// blocks per SM and one row ahead: such a solve is bound by the gathers in flight.
template <bool HELD>
__global__ void __launch_bounds__(kT, HELD ? 1 : 2) k_jcg_ir(View32 J) {
    constexpr int kEarly = HELD ? 4 : 1;
    __shared__ TileSums ts;
    __shared__ Share S;
    __shared__ double tot[3];
    extern __shared__ __align__(16) unsigned char dyn[];
    Part* const part = reinterpret_cast<Part*>(dyn);
    float* const cv = reinterpret_cast<float*>(part + J.max_parts);
    int32_t* const ci = reinterpret_cast<int32_t*>(cv + J.cache_entries);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const bool stall = J.stall_member >= 0 && blockIdx.x == 0;
    GridBarrier bar;
    make_share(J, 0, S, part, [](Part&) {});
    const bool mine = S.n > 0;
    Part q{};
    if (mine) q = part[0];
    const int per = mine ? q.tr / 32 : 1;
    const int first = q.a * per + ((w - q.a * per) & (kT / 32 - 1)), last = mine ? min(q.e * per, (q.rows + 31) / 32) : 0;
    // the block's matrix entries, when they fit
    int shift = kNone;
    if (mine) {
        const int ra = q.row0 + q.a * q.tr, rb = q.row0 + min(q.e * q.tr, q.rows);
        const int from = J.indptr[ra], n = J.indptr[rb] - from;
        if (n <= J.cache_entries) {
            for (int j = tid; j < n; j += kT) { cv[j] = J.A32[from + j]; ci[j] = J.indices[from + j]; }
            shift = from;
        }
        rows_sum<1>(J, q, ts, 0, [&](int i, int, double (&v)[1]) { v[0] += J.b[i] * J.b[i]; });
    }
    SYNC32();
    double v1[1];
    totals<1>(J, 0, J.ntiles, 0, v1, tot);
    const double atol = J.rtol * sqrt(v1[0]), atol2 = atol * atol;
    if (atol == 0.0) {
        // a zero right-hand side (every block decides alike)
        if (mine) part_rows(q, [&](int i, bool ok) { if (ok) J.x[i] = 0.0; });
        if (blockIdx.x == 0 && tid == 0) *J.mdone = 0;
        return;
    }
    SYNC32();
    int inner = 0, par = 0;                  // iterations so far; parity that holds the last (u, w, s, p)
    double ac = 0.0, gc = 0.0, rc = 0.0, target = 0.0;
    for (int sweep = 0; sweep < 64; sweep++) {
        // O1: r = b - A x; u_0 = D^-1 r in FP32 replaces the recursive residual, d = 0
        if (mine)
            rows_sum<1>(J, q, ts, 0, [&](int i, int, double (&v)[1]) {
                double ax = 0.0;
                for (int k = __ldg(J.indptr + i); k < __ldg(J.indptr + i + 1); k += 8) {
                    int c[8];
                    double h[8];
                    const int end = __ldg(J.indptr + i + 1);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        c[j] = k + j < end ? __ldg(J.indices + k + j) : i;
                        h[j] = k + j < end ? __ldg(J.A + k + j) : 0.0;
                    }
#pragma unroll
                    for (int j = 0; j < 8; j++) ax += h[j] * J.x[c[j]];
                }
                const double ri = J.b[i] - ax;
                float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (sweep > 0) o = J.uw[par][i];
                J.uw[0][i] = make_float4((float)(J.invD[i] * ri), 0.0f, o.z, o.w);
                J.d[i] = 0.0f;
                v[0] += ri * ri;
            });
        SYNC32();
        // O2: outer test, inner target, w_0 = D^-1 A u_0
        totals<1>(J, 0, J.ntiles, 0, v1, tot);
        if (v1[0] <= atol2) {
            if (blockIdx.x == 0 && tid == 0) { *J.mdone = inner; *J.mouter = sweep; }
            return;
        }
        // a sweep that did not halve the FP64 residual restarts the next one's recurrence
        if (sweep > 0 && !(v1[0] <= 0.25 * target / (J.inner_rtol * J.inner_rtol))) rc = 0.0;
        target = J.inner_rtol * J.inner_rtol * v1[0];
        if (mine)
            rows_sum<3>(J, q, ts, 3, [&](int i, int, double (&v)[3]) {
                const int a = __ldg(J.indptr + i), n = __ldg(J.indptr + i + 1) - a;
                float s = 0.0f;
                for (int k = 0; k < n; k++) {
                    const int at = a + k;
                    const int c = shift != kNone ? ci[at - shift] : __ldg(J.indices + at);
                    s += (shift != kNone ? cv[at - shift] : __ldg(J.A32 + at)) * J.uw[0][c].x;
                }
                // (neighbours read only the u component, this row writes only its w component)
                J.uw[0][i].y = s;
                const double ui = J.uw[0][i].x, D = __ldg(J.diag + i), Du = D * ui;
                v[0] += Du * ui; v[1] += D * (double)s * ui; v[2] += Du * Du;
            });
        SYNC32();
        // the recurrence goes on from the last sweep (residual replacement, which keeps the FP32
        // recursion accurate when inner_rtol >= 1e-2) unless the replaced residual is more than 4x the
        // recursive one
        double ap = 0.0, gp = 0.0;
        for (int it = 0;; it++) {
            const float4* uc = J.uw[it & 1];
            float4* un = J.uw[(it & 1) ^ 1];
            RowState R[kEarly];
#pragma unroll
            for (int j = 0; j < kEarly; j++) {
                const int s = first + j * (kT / 32), o = 32 * s + lane;
                if (s < last && o < q.rows) R[j] = row_state<HELD>(J, cv, ci, shift, q.row0 + o, uc);
            }
            double v[3];
            totals<3>(J, 0, J.ntiles, 3 * ((it & 1) ^ 1), v, tot);
            par = it & 1;
            if (it == 0 && sweep > 0 && J.inner_rtol >= 1e-2 && v[2] <= 16.0 * rc) { ap = ac; gp = gc; }
            const double beta = (ap != 0.0 && gp != 0.0) ? v[0] / gp : 0.0;
            const double den = v[1] - (beta != 0.0 ? beta * v[0] / ap : 0.0);
            const double alpha = den != 0.0 ? v[0] / den : 0.0;
            const bool capped = it == J.inner_maxiter;
            if ((it > 0 && it % J.check_every == 0 && v[2] <= target) || capped) {
                // (a sweep stopped by the cap leaves r.r = 0: the next one restarts)
                ac = ap; gc = gp; rc = capped ? 0.0 : v[2];
                inner += it;
                break;
            }
            ap = alpha; gp = v[0];
            const float al = (float)alpha, bt = (float)beta;
            // (slower blocks may still be reading this iteration's partials: the new ones go to the other
            // three kinds)
            if (mine)
                rows_sum<3>(J, q, ts, 3 * (it & 1), [&](int i, int s, double (&u)[3]) {
                    RowState r;
                    const int j = (s - first) / (kT / 32);
                    if (j == 0) r = R[0];
                    else if (kEarly > 1 && j == 1) r = R[kEarly > 1 ? 1 : 0];
                    else if (kEarly > 2 && j == 2) r = R[kEarly > 2 ? 2 : 0];
                    else if (kEarly > 3 && j == 3) r = R[kEarly > 3 ? 3 : 0];
                    else r = row_state<HELD>(J, cv, ci, shift, i, uc);
                    const float snew = r.o.y + bt * r.o.z, pnew = r.o.x + bt * r.o.w;
                    const float unew = r.o.x - al * snew, wnew = r.au - al * (r.aw + bt * r.as);
                    J.d[i] = r.d + al * pnew;
                    un[i] = make_float4(unew, wnew, snew, pnew);
                    const double D = r.D, Du = D * unew;
                    u[0] += Du * unew; u[1] += D * (double)wnew * unew; u[2] += Du * Du;
                });
            SYNC32();
        }
        if (mine) part_rows(q, [&](int i, bool ok) { if (ok) J.x[i] += (double)J.d[i]; });
        if (blockIdx.x == 0 && tid == 0) *J.mouter = sweep + 1;
        SYNC32();
    }
    if (blockIdx.x == 0 && tid == 0) { *J.mdone = inner; atomicOr(J.status, ERR_JCG_NOT_CONVERGED); }
}

}  // namespace

cudaError_t jcg_ir_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st, int nsm) {
    View32 J{};
    J.nmem = 1; J.ntiles = w->ntiles;
    J.row0 = w->mem_row0; J.rows = w->mem_rows; J.tile_rows = w->mem_tr; J.t0 = w->mem_t0;
    J.part = w->tile_part; J.mfin = w->mgen; J.bar = w->bar; J.err = a.err;
    J.polls = a.wait_polls > 0 ? a.wait_polls : kWaitPolls;
    J.n = a.n; J.indptr = a.indptr; J.indices = a.indices; J.A = a.A; J.b = a.b; J.invD = a.invD;
    J.A32 = a.A32; J.diag = a.diag32; J.x = a.x;
    J.uw[0] = reinterpret_cast<float4*>(a.ir32); J.uw[1] = J.uw[0] + a.n; J.d = a.ir32 + 8 * (size_t)a.n;
    J.mdone = w->mdone; J.mouter = w->mouter; J.status = w->status;
    J.stall_member = a.stall_member < 1 ? a.stall_member : -1;
    J.rtol = a.rtol; J.inner_rtol = a.inner_rtol; J.inner_maxiter = a.inner_maxiter;
    J.check_every = a.check_every > 0 ? a.check_every : 1;
    // a row of a triangular mesh has about seven entries: the matrix is held when that many fit (a block
    // whose rows turn out to have more reads them from global memory)
    const void* fn = (const void*)k_jcg_ir<true>;
    long long room = 0;
    cudaError_t e = grant_shared(fn, room);
    if (e != cudaSuccess) return e;
    int grid = std::max(1, std::min(w->ntiles, nsm));
    J.max_parts = share_parts(1, grid);
    size_t shared = sizeof(Part) * J.max_parts;
    J.cache_entries = (int)((room - (long long)shared) / 8);
    if (7LL * a.n <= (long long)J.cache_entries * grid) {
        shared += 8 * (size_t)J.cache_entries;
    } else {
        fn = (const void*)k_jcg_ir<false>;
        grid = std::max(1, std::min(w->ntiles, 2 * nsm));
        J.cache_entries = 0;
    }
    e = jcg_clear(w, st);
    if (e != cudaSuccess) return e;
    void* args[] = {&J};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kT), args, shared, st);
}

}  // namespace gs
