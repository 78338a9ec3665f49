// Jacobi-preconditioned CG in FP64 (GS_FP64), one persistent cooperative launch per solve for every
// member of a batch (replaces PCGSolverMultiGPU.solve / NativePCG, src/solver/pcg_solver.py:1075-1124
// and src/solver/pcg_loop.cpp:334-416): the reference's iteration, with its two reductions.
//   A: beta = rz / rz_old; p_new = z + beta p; q = A p_new; p.q partials
//   B: alpha = rz / p.q; x += alpha p; r -= alpha q; z = invD r; r.r and r.z partials
// Members retire at the reference's checkpoints ((it + 1) % check_every == 0 or the last iteration,
// r.r <= (rtol |b|)^2, pcg_loop.cpp:405-412).
//
// What bounds it.  Up to some 300k rows an iteration is short: its time is the latency of two
// reductions and of the loads between them, not bandwidth.  So the chain behind each barrier is kept
// to one round trip: the matrix of a block's rows stays in shared memory for the whole solve (it does
// not change; blocks whose rows do not fit read it from global memory), the products A z and A p are
// gathered while beta is still being added up (q = A z + beta A p), a thread's own values for phase B
// are loaded before the barrier that opens it, and every block adds the partials itself instead of
// waiting for one block to publish the scalar.
#include <algorithm>
#include <mutex>

#include "jcg_share.cuh"
#include "jcg_work.h"
#include "kernels.h"

namespace gs {

namespace {

struct View64 : SolveView {
    const int32_t *indptr, *indices;         // CSR rows (indptr), or SELL-32 slices when sell is set
    const int2* sell;
    const double *A, *b, *invD;
    double *x, *r, *z, *q, *p0, *p1;
    int32_t* mdone;                          // iterations at convergence
    unsigned* nstop;                         // members done
    int32_t* status;
    int stall_member;
    int cache_entries;                       // matrix entries a block can hold
    double rtol;
    int maxiter, check_every;
};

// Where the entries of a block's rows are: entry k of a row at off + k * stride.
template <bool SELL>
struct Rows {
    static constexpr int stride = SELL ? 32 : 1;
    __device__ __forceinline__ static int2 at(const View64& J, int i) {
        if constexpr (SELL) {
            const int2 sw = __ldg(J.sell + (i >> 5));
            return make_int2(sw.x + (i & 31), sw.y);
        } else {
            const int a = __ldg(J.indptr + i);
            return make_int2(a, __ldg(J.indptr + i + 1) - a);
        }
    }
    // the entries of rows [ra, rb) lie in [from, to)
    __device__ __forceinline__ static int from(const View64& J, int ra) { return SELL ? J.sell[ra >> 5].x : J.indptr[ra]; }
    __device__ __forceinline__ static int to(const View64& J, int rb) {
        if constexpr (SELL) {
            const int2 sw = J.sell[(rb - 1) >> 5];
            return sw.x + 32 * sw.y;
        } else {
            return J.indptr[rb];
        }
    }
};

// first entry of a part's cached run minus its place in the cache (kNotCached: read from global memory)
constexpr int kNotCached = 0x7fffffff;

// s1 = sum v f[c] over a row's entries and, with NV = 2, s2 = sum v g[c]; eight gathers of each are in
// flight.  The multiply-adds here and below are written out, so that every form of the kernel rounds
// alike and a member gets the same bits in each.
template <bool SELL, bool HELD, int NV>
__device__ __forceinline__ void row_products(const View64& J, const double* cv, const int32_t* ci, int shift, int i,
                                             const double* f, const double* g, double& s1, double& s2) {
    constexpr int st = Rows<SELL>::stride;
    const int2 o = Rows<SELL>::at(J, i);
    s1 = 0.0; s2 = 0.0;
    for (int k0 = 0; k0 < o.y; k0 += 8) {
        int c[8];
        double v[8], a[8], b[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const bool ok = k0 + k < o.y;
            const int at = o.x + (k0 + k) * st;
            if (HELD && shift != kNotCached) {
                c[k] = ok ? ci[at - shift] : i;
                v[k] = ok ? cv[at - shift] : 0.0;
            } else {
                c[k] = ok ? __ldg(J.indices + at) : i;
                v[k] = ok ? __ldg(J.A + at) : 0.0;
            }
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            a[k] = f[c[k]];
            if (NV == 2) b[k] = g[c[k]];
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            s1 = fma(v[k], a[k], s1);
            if (NV == 2) s2 = fma(v[k], b[k], s2);
        }
    }
}

// f(part, totals of kinds [k0, k0 + NV)), by one thread, for every part of the block that still iterates.  A
// warp adds a part's partials, so a block waits for one round trip, not for one per part.
template <int NV, typename F>
__device__ __forceinline__ void part_totals(const View64& J, const Share& S, Part* part, int k0, F f) {
    __syncthreads();
    for (int k = threadIdx.x >> 5; k < S.n; k += kT / 32) {
        Part& q = part[k];
        if (!q.on) continue;
        double v[NV];
        lane_totals<NV>(J, q.t0, tiles_of(q), k0, v);
        if ((threadIdx.x & 31) == 0) f(q, v);
    }
    __syncthreads();
}

#define SYNC64() do { if (!bar.sync(J, stall)) return; } while (0)

// partial kinds: a phase never writes the kinds it reads, since a slower block may not have read yet
enum { K_PQ = 0, K_RR = 1, K_RZ = 2 };
// HELD: one block per SM, the matrix in shared memory, the products of a thread's first two rows gathered
// before the totals are known (200k rows: 13.4 us an iteration, 20.0 before with one block publishing
// each scalar).  Otherwise, for a matrix larger than the chip's shared memory, two blocks per SM and
// nothing ahead: such a solve is bound by the gathers in flight (1M rows: 55 us in the first form,
// 39.7 in the second, 43.0 before).
//
// MANY: a batch whose blocks hold tiles of several members (more tiles than blocks).  A block takes the totals
// of all its parts at once and no products ahead of them: 16 members of 8,100 rows 5.6 ms a solve, 6.3 part by
// part; 64 members of 8,100 rows 8.9 and 9.5.  A block of one part keeps what it needs of it in registers over
// the barriers, which that form does not (30k rows: 4.3 ms, 4.5 in it).
template <bool SELL, bool HELD, bool MANY>
__global__ void __launch_bounds__(kT, HELD ? 1 : 2) k_jcg64(View64 J) {
    constexpr int kEarly = 2;
    constexpr bool kAhead = HELD && !MANY;   // products gathered before the totals are known
    __shared__ TileSums ts;
    __shared__ Share S;
    __shared__ double tot[3];
    __shared__ int cached;
    extern __shared__ __align__(16) unsigned char dyn[];
    Part* const part = reinterpret_cast<Part*>(dyn);
    double* const cv = reinterpret_cast<double*>(part + J.max_parts);
    int32_t* const ci = reinterpret_cast<int32_t*>(cv + J.cache_entries);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, nmem = J.nmem;
    const bool stall = J.stall_member >= 0 && blockIdx.x == 0;
    if (__syncthreads_or(timed_out(J.err))) return;
    GridBarrier bar;
    make_share(J, 0, S, part, [](Part&) {});
    // the matrix entries of the block's parts, as many parts as fit (Part::sl: their shift)
    if (tid == 0) cached = 0;
    __syncthreads();
    for (int k = 0; k < S.n; k++) {
        Part& q = part[k];
        const int ra = q.row0 + q.a * q.tr, rb = q.row0 + min(q.e * q.tr, q.rows);
        const int from = Rows<SELL>::from(J, ra), n = Rows<SELL>::to(J, rb) - from, at = cached;
        const bool fits = n <= J.cache_entries - at;
        if (fits)
            for (int j = tid; j < n; j += kT) { cv[at + j] = J.A[from + j]; ci[at + j] = J.indices[from + j]; }
        __syncthreads();
        if (tid == 0) {
            q.sl = fits ? from - at : kNotCached;
            if (fits) cached = at + n;
        }
        __syncthreads();
    }
    // |b|^2
    for (int k = 0; k < S.n; k++)
        part_sum(J, part[k], ts, [&](int i, bool ok) {
            const double bi = ok ? J.b[i] : 0.0;
            return __dmul_rn(bi, bi);
        });
    SYNC64();
    for (int k = 0; k < S.n; k++) {
        Part& q = part[k];
        double v[1];
        totals<1>(J, q.t0, tiles_of(q), 0, v, tot);
        const double atol = J.rtol * sqrt(v[0]);
        if (tid == 0) {
            q.target = atol * atol;
            q.gp = 0.0;
            if (atol == 0.0) {
                // a zero right-hand side: solved by x = 0, before the first iteration
                q.on = 0;
                if (q.a == 0) { J.mdone[q.m] = 0; __threadfence(); atomicAdd(J.nstop, 1u); }
            }
        }
        if (atol == 0.0) part_rows(q, [&](int i, bool ok) { if (ok) { J.x[i] = 0.0; J.r[i] = 0.0; J.z[i] = 0.0; } });
    }
    SYNC64();
    // r = b - A x; z = invD r; p = 0; the products of the rows below read only x
    for (int k = 0; k < S.n; k++) {
        const Part& q = part[k];
        if (!q.on) continue;
        for (int a = q.a; a < q.e; a += kTileRun) {
            const int e = min(q.e, a + kTileRun);
            const int per = q.tr / 32, s0 = a * per, s1 = min(e * per, (q.rows + 31) / 32);
            clear_tiles<2>(ts, e - a);
            double v[2] = {0.0, 0.0};
            int tile = -1;
            for (int s = s0 + ((w - s0) & (kT / 32 - 1)); s < s1; s += kT / 32) {
                if (s / per != tile) {
                    if (tile >= 0) put_warp<2>(ts, tile - a, v);
                    tile = s / per;
                }
                const int o = 32 * s + lane, i = q.row0 + o;
                if (o < q.rows) {
                    double ax, no;
                    row_products<SELL, HELD, 1>(J, cv, ci, q.sl, i, J.x, nullptr, ax, no);
                    const double ri = J.b[i] - ax, zi = J.invD[i] * ri;
                    J.r[i] = ri; J.z[i] = zi; J.p0[i] = 0.0; J.p1[i] = 0.0;
                    v[0] = fma(ri, ri, v[0]); v[1] = fma(ri, zi, v[1]);
                }
            }
            if (tile >= 0) put_warp<2>(ts, tile - a, v);
            put_tiles<2>(J, q, a, e, ts, K_RR);
        }
    }
    SYNC64();
    // whether the block's first part still iterates, a copy of every thread's own: Part::on is cleared by one
    // thread in phase A and read by the others only behind a barrier
    bool first_on = S.n > 0 && part[0].on;
    for (int it = 0;; it++) {
        const double* pc = (it & 1) ? J.p1 : J.p0;
        double* pn = (it & 1) ? J.p0 : J.p1;
        // ---- A
        if constexpr (MANY) {
            part_totals<2>(J, S, part, K_RR, [&](Part& q, const double (&v)[2]) {
                // the test of iteration it - 1
                const bool conv = it > 0 && (it % J.check_every == 0 || it == J.maxiter) && v[0] <= q.target;
                if (conv || it == J.maxiter) {
                    q.on = 0;
                    if (q.a == 0) {
                        J.mdone[q.m] = it;
                        if (!conv) atomicOr(J.status, ERR_JCG_NOT_CONVERGED);
                        __threadfence();
                        atomicAdd(J.nstop, 1u);
                    }
                } else {
                    q.ap = (it == 0 || q.gp == 0.0) ? 0.0 : v[1] / q.gp;
                    q.gp = v[1];
                }
            });
            first_on = S.n > 0 && part[0].on;
        }
        for (int k = 0; k < S.n; k++) {
            Part& q = part[k];
            if (!q.on) continue;
            const int per = q.tr / 32, first = q.a * per + ((w - q.a * per) & (kT / 32 - 1));
            const int last = min(q.e * per, (q.rows + 31) / 32);
            double az[kEarly], ap[kEarly], zi[kEarly], pi[kEarly];
#pragma unroll
            for (int j = 0; kAhead && j < kEarly; j++) {
                const int s = first + j * (kT / 32), o = 32 * s + lane, i = q.row0 + o;
                az[j] = ap[j] = zi[j] = pi[j] = 0.0;
                if (s < last && o < q.rows) {
                    row_products<SELL, HELD, 2>(J, cv, ci, q.sl, i, J.z, pc, az[j], ap[j]);
                    zi[j] = J.z[i]; pi[j] = pc[i];
                }
            }
            double beta;
            if constexpr (MANY) {
                beta = q.ap;
            } else {
                const double rz_old = q.gp;
                double v[2];
                totals<2>(J, q.t0, tiles_of(q), K_RR, v, tot);
                const bool conv = it > 0 && (it % J.check_every == 0 || it == J.maxiter) && v[0] <= q.target;
                const bool done = conv || it == J.maxiter;
                if (k == 0 && done) first_on = false;
                if (tid == 0) {
                    if (done) {
                        q.on = 0;
                        if (q.a == 0) {
                            J.mdone[q.m] = it;
                            if (!conv) atomicOr(J.status, ERR_JCG_NOT_CONVERGED);
                            __threadfence();
                            atomicAdd(J.nstop, 1u);
                        }
                    } else {
                        q.gp = v[1];
                    }
                }
                if (done) continue;
                beta = (it == 0 || rz_old == 0.0) ? 0.0 : v[1] / rz_old;
            }
            for (int a = q.a; a < q.e; a += kTileRun) {
                const int e = min(q.e, a + kTileRun);
                const int s0 = a * per, s1 = min(e * per, last);
                clear_tiles<1>(ts, e - a);
                double pq[1] = {0.0};
                int tile = -1;
                for (int s = s0 + ((w - s0) & (kT / 32 - 1)); s < s1; s += kT / 32) {
                    if (s / per != tile) {
                        if (tile >= 0) put_warp<1>(ts, tile - a, pq);
                        tile = s / per;
                    }
                    const int o = 32 * s + lane, i = q.row0 + o;
                    if (o < q.rows) {
                        double s1_, s2_, z_, p_;
                        const int j = (s - first) / (kT / 32);
                        if (kAhead && j < kEarly) {
                            s1_ = j ? az[1] : az[0]; s2_ = j ? ap[1] : ap[0];
                            z_ = j ? zi[1] : zi[0]; p_ = j ? pi[1] : pi[0];
                        } else {
                            row_products<SELL, HELD, 2>(J, cv, ci, q.sl, i, J.z, pc, s1_, s2_);
                            z_ = J.z[i]; p_ = pc[i];
                        }
                        const double p = fma(beta, p_, z_), ax = fma(beta, s2_, s1_);
                        pn[i] = p; J.q[i] = ax;
                        pq[0] = fma(p, ax, pq[0]);
                    }
                }
                if (tile >= 0) put_warp<1>(ts, tile - a, pq);
                put_tiles<1>(J, q, a, e, ts);
            }
        }
        // ---- B: a thread's rows are those it wrote in A, so the first ones of the block's first part
        // are loaded before the barrier
        double fx[kEarly], fr[kEarly], fq[kEarly], fp[kEarly], fd[kEarly];
        int fs = -1;
        if (HELD && first_on) {
            const Part& q = part[0];
            const int per = q.tr / 32, last = min(q.e * per, (q.rows + 31) / 32);
            fs = q.a * per + ((w - q.a * per) & (kT / 32 - 1));
#pragma unroll
            for (int j = 0; j < kEarly; j++) {
                const int s = fs + j * (kT / 32), o = 32 * s + lane, i = q.row0 + o;
                fx[j] = fr[j] = fq[j] = fp[j] = fd[j] = 0.0;
                if (s < last && o < q.rows) { fx[j] = J.x[i]; fr[j] = J.r[i]; fq[j] = J.q[i]; fp[j] = pn[i]; fd[j] = J.invD[i]; }
            }
        }
        SYNC64();
        // (uniform: nstop only changes in the set-up and in phase A, each with a barrier behind it)
        if (*((volatile unsigned*)J.nstop) >= (unsigned)nmem) break;
        if constexpr (MANY)
            part_totals<1>(J, S, part, K_PQ, [&](Part& q, const double (&v)[1]) { q.ap = v[0] != 0.0 ? q.gp / v[0] : 0.0; });
        for (int k = 0; k < S.n; k++) {
            const Part& q = part[k];
            if (!q.on) continue;
            const int per = q.tr / 32;
            double alpha;
            if constexpr (MANY) {
                alpha = q.ap;
            } else {
                double v[1];
                totals<1>(J, q.t0, tiles_of(q), K_PQ, v, tot);
                alpha = v[0] != 0.0 ? q.gp / v[0] : 0.0;
            }
            for (int a = q.a; a < q.e; a += kTileRun) {
                const int e = min(q.e, a + kTileRun);
                const int s0 = a * per, s1 = min(e * per, (q.rows + 31) / 32);
                clear_tiles<2>(ts, e - a);
                double u[2] = {0.0, 0.0};
                int tile = -1;
                for (int s = s0 + ((w - s0) & (kT / 32 - 1)); s < s1; s += kT / 32) {
                    if (s / per != tile) {
                        if (tile >= 0) put_warp<2>(ts, tile - a, u);
                        tile = s / per;
                    }
                    const int o = 32 * s + lane, i = q.row0 + o;
                    if (o < q.rows) {
                        double x, r, ax, p, d;
                        if (HELD && k == 0 && s == fs) { x = fx[0]; r = fr[0]; ax = fq[0]; p = fp[0]; d = fd[0]; }
                        else if (HELD && k == 0 && fs >= 0 && s == fs + kT / 32) { x = fx[1]; r = fr[1]; ax = fq[1]; p = fp[1]; d = fd[1]; }
                        else { x = J.x[i]; r = J.r[i]; ax = J.q[i]; p = pn[i]; d = J.invD[i]; }
                        const double ri = fma(-alpha, ax, r), z = d * ri;
                        J.x[i] = fma(alpha, p, x);
                        J.r[i] = ri; J.z[i] = z;
                        u[0] = fma(ri, ri, u[0]); u[1] = fma(ri, z, u[1]);
                    }
                }
                if (tile >= 0) put_warp<2>(ts, tile - a, u);
                put_tiles<2>(J, q, a, e, ts, K_RR);
            }
        }
        SYNC64();
    }
}

}  // namespace

// Kernel, grid and shared memory of a solve of `rows` rows.  A row of a triangular mesh has about seven
// entries; the matrix is held when that many fit the blocks' shared memory (a block whose rows turn out
// to have more reads them from global memory).  Batches of members below 1,024 rows on average are not held:
// what bounds them is a block's chain of parts, which two blocks per SM halve (256 members of 400 rows 1.56 ms,
// 1.70 held; 64 of 1,600 rows 2.74 and 2.67; 32 of 8,100 rows 6.98 and 6.76).
struct Shape64 {
    const void* fn;
    int grid, entries;
    size_t shared;
};
template <bool HELD>
static const void* kernel64(bool sell, bool many) {
    if (!sell) return (const void*)k_jcg64<false, HELD, false>;       // a caller's matrix is one member
    return many ? (const void*)k_jcg64<true, HELD, true> : (const void*)k_jcg64<true, HELD, false>;
}
static cudaError_t jcg64_shape(bool sell, long long rows, int ntiles, int nmem, int nsm, Shape64& S) {
    S.grid = std::max(1, std::min(ntiles, nsm));
    const bool many = nmem > 1 && ntiles > S.grid;
    S.fn = kernel64<true>(sell, many);
    long long room = 0;
    cudaError_t e = grant_shared(S.fn, room);
    if (e != cudaSuccess) return e;
    long long parts = (long long)(sizeof(Part) * share_parts(nmem, S.grid));
    if (parts > room) return cudaErrorInvalidConfiguration;
    S.entries = (int)((room - parts) / 12) & ~1;
    if (!(many && rows < 1024LL * nmem) && rows * 7 <= (long long)S.entries * S.grid) {
        S.shared = (size_t)parts + 12 * (size_t)S.entries;
    } else {
        const int grid = std::max(1, std::min(ntiles, 2 * nsm));
        const void* fn = kernel64<false>(sell, nmem > 1 && ntiles > grid);
        const size_t shared = sizeof(Part) * share_parts(nmem, grid);
        int fit = 0;
        long long room2 = 0;
        e = grant_shared(fn, room2);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, fn, kT, shared);
        if (e != cudaSuccess) return e;
        if (fit >= 2) { S.fn = fn; S.grid = grid; S.entries = 0; S.shared = shared; return cudaSuccess; }
        S.shared = (size_t)parts + 12 * (size_t)S.entries;
    }
    return cudaSuccess;
}

cudaError_t jcg64_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st, int nsm) {
    View64 J{};
    J.nmem = w->nmem; J.ntiles = w->ntiles;
    J.row0 = w->mem_row0; J.rows = w->mem_rows; J.tile_rows = w->mem_tr; J.t0 = w->mem_t0;
    J.part = w->tile_part; J.mfin = w->mgen; J.bar = w->bar; J.err = a.err;
    J.polls = a.wait_polls > 0 ? a.wait_polls : kWaitPolls;
    J.indptr = a.indptr; J.indices = a.indices; J.sell = a.sell; J.A = a.A; J.b = a.b; J.invD = a.invD;
    J.x = a.x; J.r = a.r; J.z = a.z; J.q = a.q; J.p0 = a.p0; J.p1 = a.p1;
    J.mdone = w->mdone; J.nstop = w->ndone; J.status = w->status;
    J.stall_member = a.stall_member < w->nmem ? a.stall_member : -1;
    J.rtol = a.rtol; J.maxiter = a.maxiter; J.check_every = a.check_every > 0 ? a.check_every : 1;
    Shape64 S{};
    cudaError_t e = jcg64_shape(w->sell, a.n, w->ntiles, w->nmem, nsm, S);
    if (e != cudaSuccess) return e;
    J.cache_entries = S.entries;
    J.max_parts = share_parts(w->nmem, S.grid);
    e = jcg_clear(w, st);
    if (e != cudaSuccess) return e;
    void* args[] = {&J};
    return cudaLaunchCooperativeKernel(S.fn, dim3(S.grid), dim3(kT), args, S.shared, st);
}

// ------------------------------------------------------------- solve without allocating ----
//
// gs_jcg_solve_csr_noalloc: the FP64 solve on a caller CSR for callers that cannot allocate device
// memory.  Its scratch (residual, search directions, inverse diagonal, tile partials and control
// words) lives in the file-scope array below; every GPU that loads the library holds it until the
// process exits.

constexpr int kNoAllocMaxRows = 65536;
constexpr int kNoAllocTileRows = 256;
constexpr int kNoAllocMaxTiles = kNoAllocMaxRows / kNoAllocTileRows;     // 256
// byte offsets inside the scratch array (all 256-byte aligned)
constexpr size_t kNaVec = sizeof(double) * kNoAllocMaxRows;              // one FP64 vector
constexpr size_t kNaOffPart = 6 * kNaVec;
constexpr size_t kNaOffCtl = kNaOffPart + sizeof(double) * 6 * kNoAllocMaxTiles;
constexpr size_t kNaCtlBytes = 256;
constexpr size_t kNoAllocBytes = kNaOffCtl + kNaCtlBytes;                // about 3 MiB

static __device__ __align__(256) unsigned char gs_noalloc_scratch[kNoAllocBytes];

// control words at kNaOffCtl
enum { NA_ROW0 = 0, NA_ROWS, NA_TILE, NA_T0, NA_MDONE, NA_MFIN, NA_NSTOP, NA_BAR, NA_STATUS, NA_ERR, NA_COUNT };

__global__ void k_noalloc_setup(unsigned char* base, int n, const int32_t* indptr, const int32_t* indices,
                                const double* A) {
    // control words of one member, inverse diagonal
    int32_t* ctl = (int32_t*)(base + kNaOffCtl);
    double* invD = (double*)(base + 5 * kNaVec);
    const int gid = blockIdx.x * blockDim.x + threadIdx.x, G = gridDim.x * blockDim.x;
    if (gid < NA_COUNT)
        ctl[gid] = gid == NA_ROWS ? n : gid == NA_TILE ? kNoAllocTileRows : gid == NA_MDONE ? -1 : gid == NA_MFIN ? 0x7f7f7f7f : 0;
    for (int i = gid; i < n; i += G) {
        double dg = 0.0;
        for (int a = indptr[i]; a < indptr[i + 1]; a++)
            if (indices[a] == i) dg = A[a];
        invD[i] = 1.0 / dg;
    }
}

static std::mutex g_noalloc_mu;
static unsigned char* g_noalloc_ptr[64] = {nullptr};

// Device address of the scratch array on the current device, looked up once per device.
static cudaError_t noalloc_base(unsigned char** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, gs_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[dev] = (unsigned char*)p;
    }
    *out = g_noalloc_ptr[dev];
    return cudaSuccess;
}

}  // namespace gs

extern "C" gs_status gs_jcg_solve_csr_noalloc(int n, const int32_t* indptr, const int32_t* indices,
                                              const double* data, const double* b, double* x, double rtol,
                                              int maxiter, int check_every, void* stream, int* iters) {
    using namespace gs;
    if (n <= 0 || n > kNoAllocMaxRows || !indptr || !indices || !data || !b || !x || maxiter < 1)
        return GS_ERR_ARG;
    unsigned char* base = nullptr;
    if (noalloc_base(&base) != cudaSuccess) return GS_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int ntiles = (n + kNoAllocTileRows - 1) / kNoAllocTileRows;
    k_noalloc_setup<<<std::max(1, std::min(64, (n + 255) / 256)), 256, 0, st>>>(base, n, indptr, indices, data);
    int32_t* ctl = (int32_t*)(base + kNaOffCtl);
    View64 J{};
    J.nmem = 1; J.ntiles = ntiles;
    J.row0 = ctl + NA_ROW0; J.rows = ctl + NA_ROWS; J.tile_rows = ctl + NA_TILE; J.t0 = ctl + NA_T0;
    J.part = (double*)(base + kNaOffPart);
    J.mfin = ctl + NA_MFIN; J.bar = (unsigned*)(ctl + NA_BAR); J.err = ctl + NA_ERR; J.polls = kWaitPolls;
    J.indptr = indptr; J.indices = indices; J.A = data; J.b = b; J.x = x;
    J.r = (double*)(base + 0 * kNaVec); J.z = (double*)(base + 1 * kNaVec); J.q = (double*)(base + 2 * kNaVec);
    J.p0 = (double*)(base + 3 * kNaVec); J.p1 = (double*)(base + 4 * kNaVec);
    J.invD = (const double*)(base + 5 * kNaVec);
    J.mdone = ctl + NA_MDONE; J.nstop = (unsigned*)(ctl + NA_NSTOP); J.status = ctl + NA_STATUS;
    J.stall_member = -1;
    J.rtol = rtol; J.maxiter = maxiter; J.check_every = check_every > 0 ? check_every : 1;
    Shape64 S{};
    if (jcg64_shape(false, n, ntiles, 1, nsm, S) != cudaSuccess) return GS_ERR_CUDA;
    J.cache_entries = S.entries;
    J.max_parts = share_parts(1, S.grid);
    void* args[] = {&J};
    cudaError_t e = cudaLaunchCooperativeKernel(S.fn, dim3(S.grid), dim3(kT), args, S.shared, st);
    if (e != cudaSuccess) return GS_ERR_CUDA;
    int32_t h[NA_COUNT] = {0};
    e = cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return GS_ERR_CUDA;
    if (iters) *iters = h[NA_MDONE];
    if (h[NA_ERR] & ERR_BARRIER_TIMEOUT) return GS_ERR_TIMEOUT;
    return GS_OK;
}
