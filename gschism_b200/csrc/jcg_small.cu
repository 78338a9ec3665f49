// The mixed-precision solve of a context's small members (below kMgMinRows rows; the larger ones are
// jcg_mg.cu's): FP64 refinement sweeps around FP32 Jacobi-PCG, one block per member.  (Replaces
// PCGSolverMultiGPU.solve, src/solver/pcg_solver.py:1075-1124, whose stopping test r.r <= (rtol |b|)^2 it
// keeps in FP64.)
//
// Such a member is bound by the latency of its 100 to 400 iterations, not by work: in a block of its own an
// iteration needs no grid barrier (1.5 us at 400 rows, 4.6 at 4,000), its vectors stay in registers and the
// gathered one in shared memory, and members do not wait for one another.  400 rows 0.20 ms a solve, 0.93 as
// plain Jacobi between the grid barriers of jcg_mg.cu; 256 members of 400 rows 0.37 and 4.7 ms.
//
// The recurrence is that of jcg_mg.cu (Chronopoulos and Gear, 1989) with z = u = D^-1 r.  Sums are taken in
// a fixed order that depends on the member's row count alone, so a member gets the same bits alone and in
// any batch, whatever the solver's tiling.
#include "jcg_share.cuh"
#include "jcg_work.h"
#include "kernels.h"

namespace gs {

namespace {

struct SmallView {
    const int32_t *row0, *rows;
    const int2* sell;                        // FP64 matrix (SELL-32, batch slices)
    const int32_t* indices;
    const double *A, *b, *invD;
    const float* diag;
    double* x;
    MgMatrix F;                              // D^-1 A off the diagonal, slices relative to the member's first row
    const int32_t* mem_s;
    int32_t *mdone, *mouter, *mfin, *status, *err;
    long long polls;
    int stall_member;
    double rtol, inner_rtol;
    int inner_maxiter;
};

// kOwn: rows of a thread (tid, tid + 512, ...), enough for the context's largest small member; a thread's rows
// beyond a member's end add zeros, so a member gets the same bits in every form.
template <int kOwn>
__global__ void __launch_bounds__(kT) k_jcg_small(SmallView J) {
    const int m = blockIdx.x, n = J.rows[m], r0 = J.row0[m], tid = threadIdx.x;
    if (n >= kMgMinRows) return;
    __shared__ double sh[3][kT / 32];
    __shared__ float us[kOwn * kT];
    if (tid == 0) J.mfin[m] = -1;            // not among the members that iterate together
    if (__syncthreads_or(timed_out(J.err))) return;
    if (m == J.stall_member) {
        // recovery tests: a wait that runs out
        if (tid == 0) {
            long long spins = 0;
            while (++spins <= J.polls && !(*((volatile int32_t*)J.err) & ERR_BARRIER_TIMEOUT))
                if (spins > 4096) __nanosleep(128);
            atomicOr(J.err, ERR_BARRIER_TIMEOUT);
        }
        return;
    }
    double v1[1] = {0.0};
    for (int i = tid; i < n; i += kT) v1[0] += J.b[r0 + i] * J.b[r0 + i];
    block_sum<1>(v1, sh);
    const double atol = J.rtol * sqrt(v1[0]), atol2 = atol * atol;
    if (atol == 0.0) {
        // a zero right-hand side is solved by x = 0
        for (int i = tid; i < n; i += kT) J.x[r0 + i] = 0.0;
        if (tid == 0) J.mdone[m] = 0;
        return;
    }
    float u[kOwn], p[kOwn], s[kOwn], d[kOwn], w[kOwn], D[kOwn];
    int2 row[kOwn];                          // first entry and entries of the row's slice in F
#pragma unroll
    for (int j = 0; j < kOwn; j++) {
        const int i = tid + j * kT;
        u[j] = p[j] = s[j] = d[j] = w[j] = D[j] = 0.0f;
        row[j] = make_int2(0, 0);
        if (i < n) {
            D[j] = J.diag[r0 + i];
            const int2 sl = J.F.sl[J.mem_s[m] + i / 32];
            row[j] = make_int2(sl.x + (i & 31), sl.y);
        }
    }
    int inner = 0;
    double ap = 0.0, gp = 0.0, rc = 0.0, target = 0.0;
    for (int sweep = 0; sweep < 64; sweep++) {
        // r = b - A x; u = D^-1 r in FP32 replaces the recursive residual, d = 0
        v1[0] = 0.0;
#pragma unroll
        for (int j = 0; j < kOwn; j++) {
            const int i = r0 + tid + j * kT;
            if (tid + j * kT >= n) continue;
            const int2 sw = J.sell[i >> 5];
            double a = 0.0;
            for (int k0 = 0; k0 < sw.y; k0 += 8) {
                int c[8];
                double h[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const bool in = k0 + k < sw.y;
                    const size_t at = (size_t)sw.x + 32 * (size_t)(k0 + k) + (i & 31);
                    c[k] = in ? J.indices[at] : i;
                    h[k] = in ? J.A[at] : 0.0;
                }
#pragma unroll
                for (int k = 0; k < 8; k++) a += h[k] * J.x[c[k]];
            }
            const double r = J.b[i] - a;
            u[j] = (float)(J.invD[i] * r);
            d[j] = 0.0f;
            v1[0] += r * r;
        }
        block_sum<1>(v1, sh);
        if (v1[0] <= atol2) {
            if (tid == 0) { J.mdone[m] = inner; J.mouter[m] = sweep; }
            return;
        }
        // a sweep that did not halve the FP64 residual restarts the recurrence
        if (sweep > 0 && !(v1[0] <= 0.25 * target / (J.inner_rtol * J.inner_rtol))) rc = 0.0;
        target = J.inner_rtol * J.inner_rtol * v1[0];
        for (int it = 0;; it++) {
#pragma unroll
            for (int j = 0; j < kOwn; j++)
                if (tid + j * kT < n) us[tid + j * kT] = u[j];
            __syncthreads();
            double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int j = 0; j < kOwn; j++) {
                float a = 0.0f;
                for (int k0 = 0; k0 < row[j].y; k0 += 8) {
                    int c[8];
                    float h[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const bool in = k0 + k < row[j].y;
                        const size_t at = (size_t)row[j].x + 32 * (size_t)(k0 + k);
                        c[k] = in ? J.F.idx[at] - r0 : 0;
                        h[k] = in ? J.F.val[at] : 0.0f;
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++) a = fmaf(h[k], us[c[k]], a);
                }
                w[j] = u[j] + a;
                const double Du = (double)D[j] * u[j];
                v[0] += Du * u[j];
                v[1] += Du * w[j];
                v[2] += Du * Du;
            }
            block_sum<3>(v, sh);             // (every thread has read us behind the barriers inside)
            // the first iteration of a sweep goes on from the last sweep unless the FP64 residual is more
            // than 4x the recursive one it replaces, or the inner tolerance is too tight for that
            if (it == 0 && !(sweep > 0 && J.inner_rtol >= 1e-2 && v[2] <= 16.0 * rc)) ap = gp = 0.0;
            const double beta = (ap != 0.0 && gp != 0.0) ? v[0] / gp : 0.0;
            const double den = v[1] - (beta != 0.0 ? beta * v[0] / ap : 0.0);
            const double alpha = den != 0.0 ? v[0] / den : 0.0;
            const bool broken = !(fabs(alpha) < 1e300 && fabs(beta) < 1e300);
            if ((it > 0 && v[2] <= target) || broken || it == J.inner_maxiter) {
                rc = (broken || it == J.inner_maxiter) ? 0.0 : v[2];
                inner += it;
                break;
            }
            ap = alpha; gp = v[0];
            const float al = (float)alpha, bt = (float)beta;
#pragma unroll
            for (int j = 0; j < kOwn; j++) {
                p[j] = bt != 0.0f ? u[j] + bt * p[j] : u[j];
                s[j] = bt != 0.0f ? w[j] + bt * s[j] : w[j];
                d[j] += al * p[j];
                u[j] -= al * s[j];
            }
        }
#pragma unroll
        for (int j = 0; j < kOwn; j++)
            if (tid + j * kT < n) J.x[r0 + tid + j * kT] += (double)d[j];
        if (tid == 0) J.mouter[m] = sweep + 1;
        __syncthreads();
    }
    if (tid == 0) { J.mdone[m] = inner; atomicOr(J.status, ERR_JCG_NOT_CONVERGED); }
}

}  // namespace

cudaError_t jcg_small_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st) {
    SmallView J{};
    J.row0 = w->mem_row0; J.rows = w->mem_rows;
    J.sell = a.sell; J.indices = a.indices; J.A = a.A; J.b = a.b; J.invD = a.invD; J.diag = a.diag32; J.x = a.x;
    J.F = a.mg->A; J.mem_s = a.mg->mem_s;
    J.mdone = w->mdone; J.mouter = w->mouter; J.mfin = w->mgen; J.status = w->status; J.err = a.err;
    J.polls = a.wait_polls > 0 ? a.wait_polls : kWaitPolls;
    J.stall_member = a.stall_member;
    J.rtol = a.rtol; J.inner_rtol = a.inner_rtol; J.inner_maxiter = a.inner_maxiter;
    // the fewest rows a thread that hold the largest small member (400 rows: 0.19 ms with two, 0.24 with eight)
    static_assert(kMgMinRows <= 8 * kT, "rows of a thread");
    if (w->small_rows <= 2 * kT) k_jcg_small<2><<<w->nmem, kT, 0, st>>>(J);
    else if (w->small_rows <= 4 * kT) k_jcg_small<4><<<w->nmem, kT, 0, st>>>(J);
    else k_jcg_small<8><<<w->nmem, kT, 0, st>>>(J);
    return cudaGetLastError();
}

}  // namespace gs
