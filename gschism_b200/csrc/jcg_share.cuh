// What the persistent solves share: the grid barrier, the dealing of a member's tiles to the blocks and
// the deterministic sums over them.
//
// A phase writes one partial per tile (a fixed tree over the tile's rows); after the barrier every block
// that holds tiles of a member adds the member's partials in tile order, so all blocks take the same
// decisions, no scalar has to be published, and a member gets the same bits alone and in any batch.
#pragma once
#include <algorithm>

#include "dev_common.cuh"

namespace gs {

constexpr int kT = 512;                     // threads per block, two blocks per SM

struct SolveView {
    int nmem, ntiles, max_parts;
    const int32_t *row0, *rows, *tile_rows, *t0;   // per member: first row, rows, rows per tile, first tile
    double* part;                            // [6][ntiles]
    int32_t* mfin;                           // sweep (refinement) after which a member is left out
    unsigned* bar;
    int32_t* err;
    long long polls;
};

// Grid barrier on a word that only grows within a launch (cleared by the host before it): one
// release-add per block, then an acquire poll.  Bounded like every device wait: after `polls` polls,
// or when another block has given up, the kernel leaves (false in every thread of the block).
struct GridBarrier {
    unsigned target = 0;
    __device__ __forceinline__ bool sync(const SolveView& J, bool skip_arrival = false) {
        __syncthreads();
        int bad = 0;
        if (threadIdx.x == 0) {
            target += gridDim.x;
            if (!skip_arrival) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(J.bar) : "memory");
            long long spins = 0;
            while ((int)(ld_acquire_u32(J.bar) - target) < 0) {
                if (++spins > 4096) __nanosleep(128);
                if (spins > J.polls) { atomicOr(J.err, ERR_BARRIER_TIMEOUT); bad = 1; break; }
                if ((spins & 255) == 0 && (*((volatile int32_t*)J.err) & ERR_BARRIER_TIMEOUT)) { bad = 1; break; }
            }
        }
        return __syncthreads_or(bad) == 0;
    }
};

// A launch that starts after a wait ran out in an earlier one (the host has not reported and cleared it yet)
// leaves at once: its inputs are those of an unfinished step.
__device__ __forceinline__ bool timed_out(const int32_t* err) {
    return (*((const volatile int32_t*)err) & ERR_BARRIER_TIMEOUT) != 0;
}

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (*sh)[kT / 32]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) sh[k][w] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = lane < kT / 32 ? sh[k][lane] : 0.0;
#pragma unroll
    for (int o = kT / 64; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = __shfl_sync(0xffffffffu, v[k], 0);
}

// A member's tiles [a, e) of one block (tile numbers count from the member's first), what the phases
// need to know about the member, and its scalars (every block that holds tiles of a member computes
// the same ones).
struct Part {
    int m, a, e;
    int row0, rows, tr, t0, cb, sl;
    int on, lev;              // still iterating in this sweep; with the coarse correction
    double ap, gp, rc, target;
};

// The tiles of a sweep are dealt to the blocks over the members still active, so that the blocks stay
// evenly loaded as members converge.  A member counts as its rows plus one eighth of a block's share:
// that bounds the members of a block (share_parts), whose parts are found once per
// sweep and kept in shared memory; looking them up in every phase would cost a chain of dependent
// loads each time.
struct Share {
    int n;                    // parts held
    bool none;                // no member is active
};

__device__ __forceinline__ bool active(const SolveView& J, int m, int sweep) {
    return *((volatile int32_t*)&J.mfin[m]) >= sweep;
}

// Tiles of a member (rows rows in tiles of tr) whose middle row lies before row x of the member.
__device__ __forceinline__ int tiles_before(long long x, int rows, int tr) {
    const int nt = (rows + tr - 1) / tr;
    if (x <= 0) return 0;
    if (x > rows - 1) return nt;
    const long long h = tr / 2;
    return x <= h ? 0 : (int)min((long long)nt, (x - h + tr - 1) / tr);
}

template <typename F>
__device__ void make_share(const SolveView& J, int sweep, Share& S, Part* part, F more) {
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        long long rows = 0;
        int cnt = 0;
        for (int b = 0; b < J.nmem; b += 32) {
            const int m = b + lane;
            const bool on = m < J.nmem && active(J, m, sweep);
            long long r = on ? J.rows[m] : 0;
            for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
            rows += r;
            cnt += __popc(__ballot_sync(0xffffffffu, on));
        }
        const long long extra = rows / (8 * gridDim.x) + 1, tot = rows + extra * cnt;
        const long long lo = tot * blockIdx.x / gridDim.x, hi = tot * (blockIdx.x + 1) / gridDim.x;
        long long cum = 0;
        int n = 0;
        for (int b = 0; b < J.nmem && cum < hi; b += 32) {
            const int m = b + lane;
            Part q;
            const bool on = m < J.nmem && active(J, m, sweep);
            q.rows = on ? J.rows[m] : 0;
            const long long own = on ? q.rows + extra : 0;
            long long inc = own;
            for (int o = 1; o < 32; o <<= 1) {
                const long long up = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += up;
            }
            q.a = q.e = 0;
            if (on) {
                const long long c0 = cum + inc - own;
                q.tr = J.tile_rows[m];
                q.a = tiles_before(lo - c0, q.rows, q.tr);
                q.e = tiles_before(hi - c0, q.rows, q.tr);
            }
            const unsigned hit = __ballot_sync(0xffffffffu, q.a < q.e);
            const int at = n + __popc(hit & ((1u << lane) - 1u));
            if (q.a < q.e && at < J.max_parts) {
                q.m = m; q.row0 = J.row0[m]; q.t0 = J.t0[m];
                q.on = 1; q.lev = 0; q.cb = -1; q.sl = 0;
                q.ap = q.gp = q.rc = q.target = 0.0;
                more(q);
                part[at] = q;
            }
            n += __popc(hit);
            cum += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) { S.n = min(n, J.max_parts); S.none = cnt == 0; }
    }
    __syncthreads();
}

// A member's totals: its tile partials in a fixed tree, the same in every block.
template <int NV>
__device__ __forceinline__ void member_total(const SolveView& J, const Part& q, double (&v)[NV], double (*sh)[kT / 32]) {
    const int a = q.t0, n = (q.rows + q.tr - 1) / q.tr;
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = 0.0;
    for (int t = threadIdx.x; t < n; t += kT)
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] += __ldcg(J.part + (size_t)k * J.ntiles + a + t);
    block_sum<NV>(v, sh);
}

// A part's rows are one contiguous run of 32-row slices.  Slice j of a member (counted from its first row) is
// always worked on by warp j % 16 of the block that holds its tile, so a tile's sums do not depend on
// where the block's run begins; a warp's sums of a tile wait in shared memory until the block has done
// kTileRun tiles.
constexpr int kTileRun = 16;
typedef double TileSums[kTileRun][3][kT / 32];

// the block's sums of tiles [a, e): one partial per tile, warps added in order
template <int NV>
__device__ __forceinline__ void put_tiles(const SolveView& J, const Part& q, int a, int e, const TileSums& ts, int k0 = 0) {
    __syncthreads();
    for (int k = threadIdx.x; k < NV * (e - a); k += kT) {
        const int t = k / NV, v = k - NV * t;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kT / 32; w++) s += ts[t][v][w];
        J.part[(size_t)(k0 + v) * J.ntiles + q.t0 + a + t] = s;
    }
    __syncthreads();
}

template <int NV>
__device__ __forceinline__ void put_warp(TileSums& ts, int t, double (&v)[NV]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) ts[t][k][threadIdx.x >> 5] = v[k];
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = 0.0;
}

template <int NV>
__device__ __forceinline__ void clear_tiles(TileSums& ts, int n) {
    for (int t = threadIdx.x & 31; t < n; t += 32)
#pragma unroll
        for (int k = 0; k < NV; k++) ts[t][k][threadIdx.x >> 5] = 0.0;
    __syncwarp();
}

// f(row, ok) over a part's rows, slice j by warp j % 16: every thread of a warp calls it together,
// ok is false past the member's last row
template <typename F>
__device__ __forceinline__ void part_rows(const Part& q, F f) {
    const int w = threadIdx.x >> 5, s0 = q.a * (q.tr / 32), s1 = min(q.e * (q.tr / 32), (q.rows + 31) / 32);
    for (int s = s0 + ((w - s0) & (kT / 32 - 1)); s < s1; s += kT / 32) {
        const int o = 32 * s + (threadIdx.x & 31);
        f(q.row0 + o, o < q.rows);
    }
}

// sum over a part's tiles of the values f(row, ok) returns, one partial per tile
template <typename F>
__device__ __forceinline__ void part_sum(const SolveView& J, const Part& q, TileSums& ts, F f) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, per = q.tr / 32;
    for (int a = q.a; a < q.e; a += kTileRun) {
        const int e = min(q.e, a + kTileRun);
        const int s0 = a * per, s1 = min(e * per, (q.rows + 31) / 32);
        clear_tiles<1>(ts, e - a);
        double v[1] = {0.0};
        int tile = -1;
        for (int s = s0 + ((w - s0) & (kT / 32 - 1)); s < s1; s += kT / 32) {
            if (s / per != tile) {
                if (tile >= 0) put_warp<1>(ts, tile - a, v);
                tile = s / per;
            }
            const int o = 32 * s + lane;
            v[0] += f(q.row0 + o, o < q.rows);
        }
        if (tile >= 0) put_warp<1>(ts, tile - a, v);
        put_tiles<1>(J, q, a, e, ts);
    }
}

// Totals of kinds [k0, k0 + NV) of the n tiles from t0 in one warp: the partials are added lane by lane and
// then over the lanes.
template <int NV>
__device__ __forceinline__ void lane_totals(const SolveView& J, int t0, int n, int k0, double (&s)[NV]) {
#pragma unroll
    for (int k = 0; k < NV; k++) s[k] = 0.0;
    for (int t = threadIdx.x & 31; t < n; t += 128) {
        double u[NV][4];
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int k = 0; k < NV; k++)
                u[k][j] = t + 32 * j < n ? __ldcg(J.part + (size_t)(k0 + k) * J.ntiles + t0 + t + 32 * j) : 0.0;
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int k = 0; k < NV; k++) s[k] += u[k][j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
}

// The same totals in every thread: the first warp adds them while the other warps go on to the barrier inside.
template <int NV>
__device__ __forceinline__ void totals(const SolveView& J, int t0, int n, int k0, double (&v)[NV], double* sh) {
    __syncthreads();
    if (threadIdx.x < 32) {
        double s[NV];
        lane_totals<NV>(J, t0, n, k0, s);
        if (threadIdx.x == 0)
#pragma unroll
            for (int k = 0; k < NV; k++) sh[k] = s[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = sh[k];
}

__device__ __forceinline__ int tiles_of(const Part& q) { return (q.rows + q.tr - 1) / q.tr; }

// Largest number of members a block holds parts of (Share): the members inside a share of
// (rows + extra members) / grid, each counting at least extra = rows / (8 grid), and two at its ends.
inline int share_parts(int nmem, int grid) { return 12 + nmem / grid; }

// Dynamic shared memory that a block of fn can have: all that the device grants beside fn's static part.
// The limit is a property of the function on the device, shared by every context and host thread, so it is
// always set to this one value; a launch asks for what it needs.
inline cudaError_t grant_shared(const void* fn, long long& room) {
    int dev = 0, optin = 0;
    cudaFuncAttributes fa{};
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return e;
    room = (long long)optin - (long long)fa.sharedSizeBytes;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room);
}

}  // namespace gs
