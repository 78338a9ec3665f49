// The mixed-precision elevation solve of a context (GS_FP32_IR): FP64 refinement sweeps
// r = b - A x, x += d around an FP32 conjugate-gradient solve of A d = r, one persistent
// cooperative launch for every member of a batch (replaces PCGSolverMultiGPU.solve,
// src/solver/pcg_solver.py:1075-1124, whose stopping test r.r <= (rtol |b|)^2 it keeps in FP64).
//
// Why a hierarchy.  The system is mass + (theta dt)^2 g H stiffness: a disturbance spreads over
// theta dt sqrt(gH), some 30 cells of a 500 m mesh in deep water, so Jacobi-PCG needs 620-780
// iterations, each bounded by its matrix traffic and its reduction.  Here the preconditioner adds a
// coarse correction: z = w0 D^-1 r + c P V(P^T r), with P piecewise constant over four consecutive
// rows (rows follow a Hilbert curve, so an aggregate is compact) and V one V(1,1) cycle with damped
// Jacobi over kMgLevels levels of four-fold aggregation whose matrices are Galerkin sums.  Members
// below kMgMinRows rows are solved apart (jcg_small.cu); a member whose coarse rows are too wide for the
// hierarchy, or whose sweeps twice failed to halve the residual, iterates with plain Jacobi (z = D^-1 r).
//
// The preconditioner is symmetric positive definite for any weights because every smoother is
// convergent: a row-scaled element matrix of a triangle is semi-definite with trace 3 (2 or 1 when an
// aggregate holds two or three of its corners), so the eigenvalues of D^-1 A stay below 3 on every
// level and 2/3 is the limit of the damping; the coarsest polynomial has odd degree 3, which is
// positive on the whole half-line.
//
// Single-reduction form of the recurrence (Chronopoulos and Gear, 1989), in vectors scaled by D^-1
// (u = D^-1 r; the FP32 matrix holds D^-1 A):
//   z = M r, w = D^-1 A z, gamma = (r, z), delta = (A z, z), beta = gamma / gamma_old,
//   alpha = gamma / (delta - beta gamma / alpha_old),
//   p = z + beta p, s = w + beta s, d += alpha p, u -= alpha s.
// An iteration is a vector pass (F2: update and restriction to level 1), the cycle over the coarse
// levels (one matrix product per level and direction; the last one, level_up<0>, writes z for every fine row)
// and one fine matrix product (F1) that gathers z.  Phases are separated by a grid barrier.
//
// Sums are deterministic and batch independent: a phase writes one partial per tile (fixed block
// tree) and every block adds a member's tile partials in tile order after the barrier, so all blocks
// take the same decisions and no scalar has to be published.
#include <algorithm>

#include "jcg_share.cuh"
#include "jcg_work.h"
#include "kernels.h"

namespace gs {

namespace {

constexpr int kFlags = 16384;               // members that get a flag in shared memory
constexpr float kW0 = 0.7f;                 // fine-level Jacobi weight of the additive part
constexpr float kOmega = 0.66f;             // damping of the coarse levels' smoother (limit 2/3)
constexpr float kOver = 1.5f;               // over-correction of piecewise-constant interpolation
// Chebyshev polynomial of degree 3 on [0.3, 2.2], coarsest level
constexpr double kChTheta = 1.25, kChDelta = 0.95, kChSigma = kChTheta / kChDelta;
constexpr double kChR0 = 1.0 / kChSigma, kChR1 = 1.0 / (2.0 * kChSigma - kChR0), kChR2 = 1.0 / (2.0 * kChSigma - kChR1);

struct MgView : SolveView {
    int n, max_on;
    const int2* sell;                        // FP64 matrix (SELL-32, batch slices)
    const int32_t* indices;
    const double *A, *b, *invD;
    const float* diag;
    double* x;
    float *u, *z, *w, *p, *s, *d;
    MgDev g;
    double* atol2;                           // [nmem] (rtol |b|)^2
    double* carry;                           // [2][4][nmem] by sweep parity: the alpha, gamma and r.r a sweep
                                             // ended with, its inner target
    int32_t *mdone, *mouter, *minner;        // results: iterations (-1: not converged), sweeps, iterations
    int32_t* mbad[2];                        // by sweep parity: sweeps that did not halve the residual
    unsigned* nstop;                         // members not iterating in this sweep
    unsigned* nlev;                          // members that iterate with the coarse correction in this sweep
    int32_t* status;
    int stall_member;
    double rtol, inner_rtol;
    int inner_maxiter;
};

// a sweep's share, and a flag per member for the coarse slices
__device__ __forceinline__ void mg_share(const MgView& J, int sweep, Share& S, Part* part, uint8_t* member_on) {
    __syncthreads();
    for (int m = threadIdx.x; m < J.max_on; m += kT) member_on[m] = active(J, m, sweep);
    make_share(J, sweep, S, part, [&](Part& q) { q.cb = J.g.mem_c[q.m]; q.sl = J.g.mem_s[q.m]; });
}

// Matrix entries pass through the SM once per product: they are read around the L1, which then
// keeps the gathered vectors.  The structure is constant; the coarse levels' values are written earlier
// in the same launch by other SMs, so values are never read through the non-coherent path.
__device__ __forceinline__ int32_t ld_stream(const int32_t* p) {
    int32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// Every warp streams the matrix slices that it works on through a ring of its own in shared memory
// (16-byte asynchronous copies, kDepth slices in flight).  The matrix does not change during a solve,
// so a phase's first slices are requested before the barrier that opens it: what follows the barrier
// is one gather, not a chain of header, index and value loads.  Slices wider than kWide entries are
// read directly, entry by entry behind the barrier: none of a lattice's fine slices (six entries), but 37 to
// 54% of those on level 1 and up to 29% on the higher levels (30k to 1M rows; the widest have 12 entries).
constexpr int kDepth = 3, kWide = 8;
struct __align__(16) Ring {
    int32_t idx[kDepth][kWide * 32];
    float val[kDepth][kWide * 32];
    int4 head[kDepth];        // slice offset and width (kOff: skip, kEnd: no more slices), two words of the phase
};
constexpr int kOff = -1, kEnd = -2;

__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void ring_request(Ring& R, int q, const MgMatrix& A, int4 h) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) R.head[q] = h;
    if (h.y > 0 && h.y <= kWide) {
        // 8 lanes move one entry of the slice's 32 rows (128 bytes)
#pragma unroll
        for (int k = 0; k < kWide; k += 4) {
            if (k + (lane >> 3) < h.y) {
                cp16(&R.idx[q][32 * k + 4 * lane], A.idx + h.x + 32 * k + 4 * lane);
                cp16(&R.val[q][32 * k + 4 * lane], A.val + h.x + 32 * k + 4 * lane);
            }
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void ring_drain() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// The warp's walk over a phase's slices: at(n) is the header of its n-th one.
template <typename At>
__device__ __forceinline__ void ring_open(Ring& R, const MgMatrix& A, At at) {
    int4 h[kDepth];
#pragma unroll
    for (int q = 0; q < kDepth; q++) h[q] = at(q);
    // (copies of a walk that was opened and not run)
    ring_drain();
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kDepth; q++) ring_request(R, q, A, h[q]);
}

// f(ring slot, header, n) for every slice that is on
template <typename At, typename F>
__device__ __forceinline__ void ring_run(Ring& R, const MgMatrix& A, At at, F f) {
    int q = 0;
    int4 next = at(kDepth);
    for (int n = 0;; n++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
        __syncwarp();
        const int4 h = R.head[q];
        if (h.y == kEnd) break;
        if (h.y != kOff) f(q, h, n);
        __syncwarp();
        ring_request(R, q, A, next);
        next = at(n + 1 + kDepth);
        if (++q == kDepth) q = 0;
    }
}

// sum_k val[k] g(idx[k]) over the entries of this lane's row in the slice of ring slot q, rounded the
// same way whatever the slice's width (on the coarsest levels a slice may hold rows of two members)
template <typename G>
__device__ __forceinline__ float row_sum(const Ring& R, int q, int4 h, const MgMatrix& A, G g) {
    const int lane = threadIdx.x & 31;
    float s = 0.0f;
    if (h.y <= kWide) {
        float y[kWide];
#pragma unroll
        for (int k = 0; k < kWide; k++) y[k] = k < h.y ? g(R.idx[q][32 * k + lane]) : 0.0f;
#pragma unroll
        for (int k = 0; k < kWide; k++) s = fmaf(k < h.y ? R.val[q][32 * k + lane] : 0.0f, y[k], s);
    } else {
        for (int k = 0; k < h.y; k++) {
            const size_t at = (size_t)h.x + 32 * (size_t)k + lane;
            s = fmaf(ld_stream(A.val + at), g(ld_stream(A.idx + at)), s);
        }
    }
    return s;
}

__device__ __forceinline__ float sum4(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}

// --- coarse matrices: A_{k+1}[I][J] = sum of A_k[i][j] over i in I, j in J -----------------------
// One thread per coarse row adds the entries of its four rows into 16 slots held in shared memory
// (wider rows take several passes).
constexpr int kAcc = 16;

template <typename Row>
__device__ __forceinline__ void galerkin_row(const MgLevel& L, int I, float* acc, Row row) {
    const int2 sw = L.A.sl[I >> 5];
    const int lane = I & 31;
    float D = 0.0f, inv = 1.0f;
    for (int base = 0; base == 0 || base < sw.y; base += kAcc) {
#pragma unroll
        for (int k = 0; k < kAcc; k++) acc[k * kT] = 0.0f;
        for (int j = 0; j < 4; j++)
            row(j, [&](int slot, float a) {
                if (slot == kMgDiag) { if (base == 0) D += a; }
                else if (slot >= base && slot < base + kAcc) acc[(slot - base) * kT] += a;
            });
        // a row without a positive diagonal (padding, or a matrix that is not positive definite)
        // is decoupled
        if (base == 0) { if (D > 0.0f && D < 3.0e38f) inv = 1.0f / D; else { D = 0.0f; inv = 0.0f; } }
        for (int k = base; k < min(sw.y, base + kAcc); k++)
            L.A.val[(size_t)sw.x + 32 * (size_t)k + lane] = acc[(k - base) * kT] * inv;
    }
    L.D[I] = D;
    L.Dinv[I] = inv;
}

__device__ void galerkin_fine(const MgView& J, float* acc) {
    const MgLevel& L = J.g.lv[0];
    for (int I = blockIdx.x * kT + threadIdx.x; I < L.n; I += gridDim.x * kT) {
        const int m = J.g.chunk_mem[I / kMgChunk];
        const int a = m < 0 ? 0 : 4 * (I - J.g.mem_c[m]);
        galerkin_row(L, I, acc + threadIdx.x, [&](int j, auto add) {
            if (m < 0 || a + j >= J.rows[m]) return;
            const int i = J.row0[m] + a + j;
            const int2 sw = J.g.A.sl[J.g.mem_s[m] + (a + j) / 32];
            const float D = J.diag[i];
            add((int)kMgDiag, D);
            for (int k = 0; k < sw.y; k++) {
                const size_t at = (size_t)sw.x + 32 * (size_t)k + ((a + j) & 31);
                add((int)J.g.A.map[at], J.g.A.val[at] * D);
            }
        });
    }
}

__device__ void galerkin_level(const MgLevel& F, const MgLevel& L, float* acc) {
    for (int I = blockIdx.x * kT + threadIdx.x; I < L.n; I += gridDim.x * kT)
        galerkin_row(L, I, acc + threadIdx.x, [&](int j, auto add) {
            const int i = 4 * I + j;
            const int2 sw = F.A.sl[i >> 5];
            const float D = F.D[i];
            add((int)kMgDiag, D);
            for (int k = 0; k < sw.y; k++) {
                const size_t at = (size_t)sw.x + 32 * (size_t)k + (i & 31);
                add((int)F.A.map[at], F.A.val[at] * D);
            }
        });
}

// --- the cycle over the coarse levels --------------------------------------------------------

// Slices s = warp, warp + warps of the grid, ... of level K (0 = level 1).  On the two finest levels a
// slice belongs to one member and is skipped once that member has converged.
template <int K>
struct Slices {
    const MgView& J;
    const uint8_t* member_on;
    __device__ __forceinline__ int slice(int n) const {
        return (int)blockIdx.x + (int)gridDim.x * ((int)(threadIdx.x >> 5) + n * (kT / 32));
    }
    __device__ __forceinline__ int4 operator()(int n) const {
        const int s = slice(n);
        if (s >= J.g.lv[K].n / 32) return make_int4(0, kEnd, 0, 0);
        const int2 sw = __ldg(J.g.lv[K].A.sl + s);
        int4 h = make_int4(sw.x, sw.y, 0, 0);
        if constexpr (K < 2) {
            constexpr int per = kMgChunk >> (5 + 2 * K);
            const int m = __ldg(J.g.chunk_mem + s / per);
            if constexpr (K == 0) {
                // the fine rows under the slice, for the interpolation
                const int2 f = __ldg(J.g.chunk_fine + s / per);
                h.z = f.x + 128 * (s % per);
                h.w = f.y - 128 * (s % per);
            }
            if (m < 0 || (m < J.max_on && !member_on[m])) h.y = kOff;
        }
        return h;
    }
};

template <int K>
__device__ __forceinline__ void level_open(const MgView& J, const uint8_t* member_on, Ring& R) {
    ring_open(R, J.g.lv[K].A, Slices<K>{J, member_on});
}

// f(ring slot, header, row)
template <int K, typename F>
__device__ __forceinline__ void level_run(const MgView& J, const uint8_t* member_on, Ring& R, F f) {
    const Slices<K> at{J, member_on};
    ring_run(R, J.g.lv[K].A, at, [&](int q, int4 h, int n) { f(q, h, 32 * at.slice(n) + (int)(threadIdx.x & 31)); });
}

template <int K>
__device__ __forceinline__ void level_down(const MgView& J, const uint8_t* member_on, Ring& R) {
    const MgLevel &L = J.g.lv[K], &C = J.g.lv[K + 1];
    level_run<K>(J, member_on, R, [&](int q, int4 h, int I) {
        const float own = L.rh[I], D = __ldcg(L.D + I), Di = __ldcg(C.Dinv + (I >> 2));
        const float a = row_sum(R, q, h, L.A, [&](int c) { return L.rh[c]; });
        const float t = sum4(D * (own - kOmega * (own + a)));
        if ((I & 3) == 0) C.rh[I >> 2] = t * Di;
    });
}

// On level 1 the correction goes straight to the fine rows: z = w0 u + c P e.
template <int K>
__device__ __forceinline__ void level_up(const MgView& J, const uint8_t* member_on, Ring& R) {
    const MgLevel &L = J.g.lv[K], &C = J.g.lv[K + 1];
    const int lane = threadIdx.x & 31;
    level_run<K>(J, member_on, R, [&](int q, int4 h, int I) {
        float u[4];
        if constexpr (K == 0) {
#pragma unroll
            for (int j = 0; j < 4; j++) u[j] = 32 * j + lane < h.w ? J.u[h.z + 32 * j + lane] : 0.0f;
        }
        const float own = L.rh[I], y = kOmega * own + kOver * C.e[I >> 2];
        const float a = row_sum(R, q, h, L.A, [&](int c) { return kOmega * L.rh[c] + kOver * C.e[c >> 2]; });
        const float e = y + kOmega * (own - (y + a));
        if constexpr (K == 0) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float ej = __shfl_sync(0xffffffffu, e, 8 * j + (lane >> 2));
                if (32 * j + lane < h.w) J.z[h.z + 32 * j + lane] = kW0 * u[j] + kOver * ej;
            }
        } else {
            L.e[I] = e;
        }
    });
}

__device__ __forceinline__ void coarsest_1(const MgView& J, const uint8_t* member_on, Ring& R) {
    constexpr int K = kMgLevels - 1;
    const MgLevel& L = J.g.lv[K];
    constexpr float i0 = (float)(1.0 / kChTheta), c1 = (float)(kChR1 * kChR0), c2 = (float)(2.0 * kChR1 / kChDelta);
    level_run<K>(J, member_on, R, [&](int q, int4 h, int I) {
        const float own = L.rh[I], d0 = i0 * own;
        const float a = row_sum(R, q, h, L.A, [&](int c) { return i0 * L.rh[c]; });
        const float r = own - (d0 + a), d1 = c1 * d0 + c2 * r;
        J.g.cr[I] = r;
        J.g.cd[I] = d1;
        L.e[I] = d0 + d1;
    });
}

__device__ __forceinline__ void coarsest_2(const MgView& J, const uint8_t* member_on, Ring& R) {
    constexpr int K = kMgLevels - 1;
    const MgLevel& L = J.g.lv[K];
    constexpr float c1 = (float)(kChR2 * kChR1), c2 = (float)(2.0 * kChR2 / kChDelta);
    level_run<K>(J, member_on, R, [&](int q, int4 h, int I) {
        const float d1 = J.g.cd[I], r = J.g.cr[I], x = L.e[I];
        const float a = row_sum(R, q, h, L.A, [&](int c) { return J.g.cd[c]; });
        L.e[I] = x + c1 * d1 + c2 * (r - (d1 + a));
    });
}

// restriction of D u to level 1 (all lanes; rows past the member's end contribute nothing)
__device__ __forceinline__ void restrict_row(const MgView& J, const Part& q, int i, float Du) {
    const float t = sum4(Du);
    const int o = i - q.row0;
    if ((o & 3) == 0 && o < q.rows) {
        const int I = q.cb + (o >> 2);
        J.g.lv[0].rh[I] = t * __ldcg(J.g.lv[0].Dinv + I);
    }
}

// --- the fine product ---------------------------------------------------------------------------

struct FineSlices {
    const MgView& J;
    int sl, s0, s1;           // first slice of the member, the run's slices [s0, s1)
    __device__ __forceinline__ FineSlices(const MgView& J_, const Part& q, int a, int e) : J(J_), sl(q.sl) {
        s0 = a * (q.tr / 32);
        s1 = min(e * (q.tr / 32), (q.rows + 31) / 32);
    }
    __device__ __forceinline__ int slice(int n) const {
        const int w = threadIdx.x >> 5;
        return s0 + ((w - s0) & (kT / 32 - 1)) + n * (kT / 32);
    }
    __device__ __forceinline__ int4 operator()(int n) const {
        const int s = slice(n);
        if (s >= s1) return make_int4(0, kEnd, 0, 0);
        const int2 sw = __ldg(J.g.A.sl + sl + s);
        return make_int4(sw.x, sw.y, s, 0);
    }
};

__device__ __forceinline__ void fine_open(const MgView& J, const Part& q, int a, Ring& R) {
    ring_open(R, J.g.A, FineSlices(J, q, a, min(q.e, a + kTileRun)));
}

// w = D^-1 A z and the partials of gamma = (r, z), delta = (A z, z) and r.r of a part's tiles; z = u
// without the coarse correction.  `opened`: the ring already holds the part's first slices.
__device__ __forceinline__ void fine_part(const MgView& J, const Part& q, Ring& R, TileSums& ts, bool opened) {
    const int lane = threadIdx.x & 31, per = q.tr / 32;
    const float* z = q.lev ? J.z : J.u;
    for (int a = q.a; a < q.e; a += kTileRun) {
        const int e = min(q.e, a + kTileRun);
        const FineSlices at(J, q, a, e);
        if (!opened) ring_open(R, J.g.A, at);
        opened = false;
        clear_tiles<3>(ts, e - a);
        double v[3] = {0.0, 0.0, 0.0};
        int tile = -1;
        ring_run(R, J.g.A, at, [&](int b, int4 h, int) {
            const int t = h.z / per;
            if (t != tile) {
                if (tile >= 0) put_warp<3>(ts, tile - a, v);
                tile = t;
            }
            const int o = 32 * h.z + lane, i = q.row0 + o;
            const bool ok = o < q.rows;
            const float zi = ok ? z[i] : 0.0f, ui = ok ? J.u[i] : 0.0f, Di = ok ? __ldcg(J.diag + i) : 0.0f;
            const float wi = zi + row_sum(R, b, h, J.g.A, [&](int c) { return z[c]; });
            if (ok) {
                J.w[i] = wi;
                const double D = Di, Du = D * ui, Dz = D * zi;
                v[0] += Du * zi;
                v[1] += Dz * wi;
                v[2] += Du * Du;
            }
        });
        if (tile >= 0) put_warp<3>(ts, tile - a, v);
        put_tiles<3>(J, q, a, e, ts);
    }
}

// own values of a row for the vector update
struct RowVec {
    float z, w, p, s, d, u, D;
};
__device__ __forceinline__ RowVec row_vec(const MgView& J, const Part& q, int i) {
    return {q.lev ? J.z[i] : J.u[i], J.w[i], J.p[i], J.s[i], J.d[i], J.u[i], __ldcg(J.diag + i)};
}

// A failed wait ends the kernel; no thread leaves with copies of its own in flight.  (Predicated in PTX: as a
// branch of its own behind each of the fourteen barriers it costs registers, and 3% of the solve.)
__device__ __forceinline__ void leave_unless(bool ok) {
    asm volatile("{ .reg .pred p; setp.eq.s32 p, %0, 0; @p cp.async.wait_all; @p exit; }" ::"r"((int)ok) : "memory");
}
#define MG_SYNC() leave_unless(bar.sync(J, stall))

__global__ void __launch_bounds__(kT, 2) k_jcg_mg(MgView J, int with_levels) {
    __shared__ double sh[3][kT / 32];
    __shared__ TileSums ts;
    __shared__ Share S;
    // rings of the warps (the Galerkin sums' slots before the first sweep), parts, flags per member
    extern __shared__ __align__(16) unsigned char dyn[];
    Ring& R = reinterpret_cast<Ring*>(dyn)[threadIdx.x >> 5];
    float* const acc = reinterpret_cast<float*>(dyn);
    static_assert(sizeof(Ring) * (kT / 32) >= sizeof(float) * kAcc * kT, "Galerkin slots");
    Part* const part = reinterpret_cast<Part*>(dyn + sizeof(Ring) * (kT / 32));
    uint8_t* const member_on = reinterpret_cast<uint8_t*>(part + J.max_parts);
    const int tid = threadIdx.x, nmem = J.nmem;
    const bool stall = J.stall_member >= 0 && blockIdx.x == 0;
    if (__syncthreads_or(timed_out(J.err))) return;
    GridBarrier bar;
    // |b|^2 partials; coarse matrices of this step's A
    mg_share(J, 0, S, part, member_on);
    for (int k = 0; k < S.n; k++) {
        part_sum(J, part[k], ts, [&](int i, bool ok) {
            const double bi = ok ? J.b[i] : 0.0;
            return bi * bi;
        });
    }
    if (with_levels) galerkin_fine(J, acc);
    MG_SYNC();
    // (rtol |b|)^2; a zero right-hand side is solved by x = 0
    for (int k = 0; k < S.n; k++) {
        const Part& q = part[k];
        double v[1];
        member_total<1>(J, q, v, sh);
        const double atol = J.rtol * sqrt(v[0]);
        if (q.a == 0 && tid == 0) {
            J.atol2[q.m] = atol * atol;
            if (atol == 0.0) J.mdone[q.m] = 0;
        }
        if (atol == 0.0) part_rows(q, [&](int i, bool ok) { if (ok) J.x[i] = 0.0; });
    }
    for (int k = 1; k < kMgLevels; k++) {
        if (with_levels) galerkin_level(J.g.lv[k - 1], J.g.lv[k], acc);
        MG_SYNC();
        // every block has made its share of sweep 0 by now
        if (k == 1)
            for (int m = blockIdx.x * kT + tid; m < nmem; m += gridDim.x * kT)
                if (*((volatile int32_t*)&J.mdone[m]) == 0) J.mfin[m] = -1;
    }
    for (int sweep = 0; sweep < 64; sweep++) {
        const int par = sweep & 1;
        mg_share(J, sweep, S, part, member_on);
        if (S.none) { ring_drain(); break; }
        // O1: r = b - A x; u = D^-1 r in FP32 replaces the recursive residual, d = 0
        for (int k = 0; k < S.n; k++) {
            const Part& q = part[k];
            part_sum(J, q, ts, [&](int i, bool ok) {
                float Du = 0.0f;
                double r = 0.0;
                if (ok) {
                    const int2 sw = __ldg(J.sell + (i >> 5));
                    double a = 0.0;
                    for (int k0 = 0; k0 < sw.y; k0 += 8) {
                        int c[8];
                        double h[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const bool in = k0 + k < sw.y;
                            const size_t at = (size_t)sw.x + 32 * (size_t)(k0 + k) + (i & 31);
                            c[k] = in ? __ldg(J.indices + at) : i;
                            h[k] = in ? __ldg(J.A + at) : 0.0;
                        }
#pragma unroll
                        for (int k = 0; k < 8; k++) a += h[k] * J.x[c[k]];
                    }
                    r = J.b[i] - a;
                    const float ui = (float)(J.invD[i] * r);
                    J.u[i] = ui;
                    J.d[i] = 0.0f;
                    Du = J.diag[i] * ui;
                }
                if (q.cb >= 0) restrict_row(J, q, i, Du);
                return r * r;
            });
        }
        if (blockIdx.x == 0) {
            double c[1] = {0.0};
            for (int m = tid; m < nmem; m += kT) c[0] += active(J, m, sweep) ? 0.0 : 1.0;
            block_sum<1>(c, sh);
            if (tid == 0) { *J.nstop = (unsigned)c[0]; *J.nlev = 0u; }
        }
        if (with_levels) level_open<0>(J, member_on, R);
        MG_SYNC();
        // O2: outer test; the inner target; whether the recurrence continues from the last sweep.  Every
        // block that holds tiles of a member decides alike; the one that holds its first tile records it.
        for (int k = 0; k < S.n; k++) {
            Part& q = part[k];
            const int m = q.m;
            double v[1];
            member_total<1>(J, q, v, sh);
            if (tid != 0) continue;
            const bool own = q.a == 0;
            if (v[0] <= J.atol2[m]) {
                q.on = 0;
                if (own) {
                    J.mdone[m] = J.minner[m];
                    J.mouter[m] = sweep;
                    J.mfin[m] = sweep;
                    __threadfence();
                    atomicAdd(J.nstop, 1u);
                }
                continue;
            }
            const double* C = J.carry + (size_t)4 * (par ^ 1) * nmem + m;
            int bad = 0;
            if (sweep > 0) {
                bad = J.mbad[par ^ 1][m];
                q.ap = C[0]; q.gp = C[nmem]; q.rc = C[2 * (size_t)nmem];
                // a sweep that did not halve the FP64 residual restarts the recurrence (its search
                // directions have gone stale); a second one leaves the hierarchy out
                if (!(v[0] <= 0.25 * C[3 * (size_t)nmem] / (J.inner_rtol * J.inner_rtol))) { q.rc = 0.0; bad++; }
            }
            q.target = J.inner_rtol * J.inner_rtol * v[0];
            q.lev = q.cb >= 0 && bad < 2;
            if (own) {
                J.carry[(size_t)(4 * par + 3) * nmem + m] = q.target;
                J.mbad[par][m] = bad;
                J.mouter[m] = sweep + 1;
                if (q.lev) atomicAdd(J.nlev, 1u);
            }
        }
        __syncthreads();
        // The cycle runs in a sweep in which a member iterates with it; one in which none does goes on without its
        // eight barriers (a plain iteration takes 7 to 10 us, one with the cycle 30 to 40).  The cycle's first phase
        // stands at the end of the iteration before, and the loop is skipped by its counter: in this form the
        // kernel's 64 registers suffice (-Xptxas -v: no spills; 160k rows 2.70 ms a solve), with the phase at the
        // start or a break instead it spills 120 bytes (2.79 to 2.90).  nstop and nlev are read behind a barrier
        // after O2 or F2, which alone change them, so every block reads the same values.
        if (with_levels) {
            level_down<0>(J, member_on, R);
            level_open<1>(J, member_on, R);
        }
        MG_SYNC();
        const bool cycle = *((volatile unsigned*)J.nlev) > 0u;
        int it = 0;
        if (*((volatile unsigned*)J.nstop) >= (unsigned)nmem) it = J.inner_maxiter + 1;      // every member has converged
        for (; it <= J.inner_maxiter; it++) {
            if (cycle) {
                level_down<1>(J, member_on, R);
                level_open<2>(J, member_on, R);
                MG_SYNC();
                level_down<2>(J, member_on, R);
                level_open<3>(J, member_on, R);
                MG_SYNC();
                coarsest_1(J, member_on, R);
                level_open<3>(J, member_on, R);
                MG_SYNC();
                coarsest_2(J, member_on, R);
                level_open<2>(J, member_on, R);
                MG_SYNC();
                level_up<2>(J, member_on, R);
                level_open<1>(J, member_on, R);
                MG_SYNC();
                level_up<1>(J, member_on, R);
                level_open<0>(J, member_on, R);
                MG_SYNC();
                level_up<0>(J, member_on, R);
                if (S.n > 0) fine_open(J, part[0], part[0].a, R);
                MG_SYNC();
            }
            // F1: w = D^-1 A z; gamma, delta and r.r
            for (int k = 0; k < S.n; k++) {
                const Part& q = part[k];
                if (q.on) fine_part(J, q, R, ts, cycle && k == 0);
            }
            // F2: scalars and the stopping test, the vector update, restriction of the new residual.
            // A thread's first row was written by itself in F1, so it is loaded before the barrier.
            RowVec first{};
            int fi = -1;
            if (S.n > 0) {
                const Part& q = part[0];
                const int s0 = q.a * (q.tr / 32), o = 32 * (s0 + (((tid >> 5) - s0) & (kT / 32 - 1))) + (tid & 31);
                if (o < min(q.e * q.tr, q.rows)) { fi = q.row0 + o; first = row_vec(J, q, fi); }
            }
            MG_SYNC();
            for (int k = 0; k < S.n; k++) {
                Part& q = part[k];
                if (!q.on) continue;
                const int m = q.m;
                const double rc = q.rc, target = q.target;
                double ap = q.ap, gp = q.gp;
                double v[3];
                member_total<3>(J, q, v, sh);
                // the first iteration of a sweep replaces the residual: the recurrence goes on from the
                // last sweep unless the FP64 residual is more than 4x the recursive one it replaces, or
                // the inner tolerance is too tight for that
                if (it == 0 && !(sweep > 0 && J.inner_rtol >= 1e-2 && v[2] <= 16.0 * rc)) ap = gp = 0.0;
                const double beta = (ap != 0.0 && gp != 0.0) ? v[0] / gp : 0.0;
                const double den = v[1] - (beta != 0.0 ? beta * v[0] / ap : 0.0);
                const double alpha = den != 0.0 ? v[0] / den : 0.0;
                const bool broken = !(fabs(alpha) < 1e300 && fabs(beta) < 1e300);
                const bool done = (it > 0 && v[2] <= target) || broken || it == J.inner_maxiter;
                if (tid == 0) {
                    if (done) {
                        q.on = 0;
                        if (q.a == 0) {
                            // what the next sweep continues from (r.r = 0: it restarts)
                            double* C = J.carry + (size_t)4 * par * nmem + m;
                            C[0] = ap; C[nmem] = gp;
                            C[2 * (size_t)nmem] = (broken || it == J.inner_maxiter) ? 0.0 : v[2];
                            if (broken) J.mbad[par][m] = 2;
                            J.minner[m] += it;
                            __threadfence();
                            atomicAdd(J.nstop, 1u);
                        }
                    } else {
                        q.ap = alpha; q.gp = v[0];
                    }
                }
                if (done) continue;
                const float al = (float)alpha, bt = (float)beta;
                part_rows(q, [&](int i, bool ok) {
                    float Du = 0.0f;
                    if (ok) {
                        const RowVec o = i == fi ? first : row_vec(J, q, i);
                        const float p = bt != 0.0f ? o.z + bt * o.p : o.z;
                        const float s = bt != 0.0f ? o.w + bt * o.s : o.w;
                        const float ui = o.u - al * s;
                        J.p[i] = p;
                        J.s[i] = s;
                        J.d[i] = o.d + al * p;
                        J.u[i] = ui;
                        Du = o.D * ui;
                    }
                    if (q.cb >= 0) restrict_row(J, q, i, Du);
                });
            }
            if (cycle) level_open<0>(J, member_on, R);
            MG_SYNC();
            if (*((volatile unsigned*)J.nstop) >= (unsigned)nmem) break;
            if (cycle) {
                level_down<0>(J, member_on, R);
                level_open<1>(J, member_on, R);
                MG_SYNC();
            }
        }
        // x += d for the members that iterated in this sweep
        for (int k = 0; k < S.n; k++) {
            const Part& q = part[k];
            if (q.target == 0.0) continue;
            part_rows(q, [&](int i, bool ok) { if (ok) J.x[i] += (double)J.d[i]; });
        }
        MG_SYNC();
    }
    for (int m = blockIdx.x * kT + tid; m < nmem; m += gridDim.x * kT)
        if (*((volatile int32_t*)&J.mdone[m]) < 0) {
            J.mdone[m] = J.minner[m];
            atomicOr(J.status, ERR_JCG_NOT_CONVERGED);
        }
}

}  // namespace

static size_t mg_shared(int nmem, int grid) {
    return sizeof(Ring) * (kT / 32) + sizeof(Part) * share_parts(nmem, grid) + std::min(nmem, kFlags);
}

// Two blocks per SM; one where the parts of very many members leave no room for two.
static int mg_grid(int ntiles, int nmem, int nsm) {
    long long room = 0;
    grant_shared((const void*)k_jcg_mg, room);
    const int grid = std::max(1, std::min(ntiles, 2 * nsm));
    int fit = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_jcg_mg, kT, mg_shared(nmem, grid));
    return fit >= 2 ? grid : std::max(1, std::min(ntiles, nsm));
}

cudaError_t jcg_mg_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st, int nsm) {
    MgView J{};
    const size_t n = a.n;
    const int grid = mg_grid(w->ntiles, w->nmem, nsm);
    J.n = a.n; J.nmem = w->nmem; J.ntiles = w->ntiles;
    J.sell = a.sell; J.indices = a.indices; J.A = a.A; J.b = a.b; J.invD = a.invD; J.diag = a.diag32; J.x = a.x;
    J.u = a.ir32; J.z = a.ir32 + n; J.w = a.ir32 + 2 * n; J.p = a.ir32 + 3 * n; J.s = a.ir32 + 4 * n; J.d = a.ir32 + 5 * n;
    J.g = *a.mg;
    J.row0 = w->mem_row0; J.rows = w->mem_rows; J.tile_rows = w->mem_tr; J.t0 = w->mem_t0;
    J.part = w->tile_part; J.atol2 = w->mem_atol2; J.carry = w->mem_ab;
    J.mdone = w->mdone; J.mouter = w->mouter; J.minner = w->minner;
    J.mfin = w->mgen; J.mbad[0] = w->mbad[0]; J.mbad[1] = w->mbad[1];
    J.nstop = w->ndone; J.nlev = w->nlev; J.status = w->status; J.bar = w->bar;
    J.err = a.err;
    J.polls = a.wait_polls > 0 ? a.wait_polls : kWaitPolls;
    J.stall_member = a.stall_member < w->nmem ? a.stall_member : -1;
    J.rtol = a.rtol; J.inner_rtol = a.inner_rtol; J.inner_maxiter = a.inner_maxiter;
    // parts of a block, and a flag per member for the coarse slices (beyond kFlags members theirs
    // are always worked on)
    J.max_parts = share_parts(w->nmem, grid);
    J.max_on = std::min(w->nmem, kFlags);
    cudaError_t e = jcg_clear(w, st);
    if (e == cudaSuccess && w->nsmall > 0) e = jcg_small_launch(a, w, st);
    if (e != cudaSuccess || w->nsmall == w->nmem) return e;
    int lev = a.mg->lv[0].n > 0 ? 1 : 0;
    void* args[] = {&J, &lev};
    return cudaLaunchCooperativeKernel((const void*)k_jcg_mg, dim3(grid), dim3(kT), args,
                                       mg_shared(w->nmem, grid), st);
}

}  // namespace gs
