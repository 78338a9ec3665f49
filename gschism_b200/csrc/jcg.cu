// Work list of the elevation solves and their dispatch (jcg64.cu: FP64; jcg_mg.cu and, for small members,
// jcg_small.cu: mixed precision of a context; jcg_ir.cu: mixed precision of a caller's CSR matrix).
//
// A member's rows are cut into tiles whose size depends only on that member's row count; every grid-wide
// reduction adds one partial per tile in tile order.  Sums are therefore deterministic and independent of the
// batch composition: a member gives bit-identical results alone and inside any batch.  Scalars stay on
// the device; convergence is tested on the device, so a solve never returns to the host.
#include <algorithm>

#include "dev_common.cuh"
#include "jcg_work.h"
#include "kernels.h"

namespace gs {

constexpr int kPartialKinds = 6;

// Tile rows of a member: a function of the member's own size and the tiling only (batch
// independence).  By default a large member is cut into 296 tiles (two per SM), so its rows spread
// evenly over the SMs, and tiles never go below 256 rows.  The autotuner may choose other values
// (JcgTiling).
static int tile_rows_for(int rows, const JcgTiling& tl) {
    const long long per = ((long long)rows + tl.tiles - 1) / tl.tiles;
    return (int)std::max((long long)tl.min_rows, (per + 31) / 32 * 32);
}

cudaError_t jcg_work_alloc(JcgWork*& w, const std::vector<int>& row0, const std::vector<int>& rows, bool sell,
                           cudaStream_t st, const JcgTiling& tiling) {
    w = new JcgWork();
    const int nmem = (int)rows.size();
    std::vector<int32_t> mt0(nmem), mtr(nmem);
    int T = 0;
    for (int m = 0; m < nmem; m++) {
        if (rows[m] < kMgMinRows) { w->nsmall++; w->small_rows = std::max(w->small_rows, rows[m]); }
        mtr[m] = tile_rows_for(rows[m], tiling);
        mt0[m] = T;
        T += (rows[m] + mtr[m] - 1) / mtr[m];
    }
    w->nmem = nmem;
    w->ntiles = T;
    w->sell = sell;
    cudaError_t e = cudaSuccess;
    auto A = [&](void** p, size_t bytes) { if (e == cudaSuccess) e = cudaMalloc(p, bytes ? bytes : 8); };
    const size_t nm = nmem;
    A((void**)&w->mem_t0, 4 * nm); A((void**)&w->mem_row0, 4 * nm); A((void**)&w->mem_rows, 4 * nm);
    A((void**)&w->mem_tr, 4 * nm);
    A((void**)&w->tile_part, 8 * (size_t)kPartialKinds * T);
    A((void**)&w->mem_atol2, 8 * nm);
    A((void**)&w->mem_ab, 64 * nm);
    A((void**)&w->mctl, 4 * (6 * nm + 4));
    if (e != cudaSuccess) return e;
    w->mdone = w->mctl; w->mouter = w->mctl + nm; w->minner = w->mctl + 2 * nm; w->mbad[0] = w->mctl + 3 * nm;
    w->mgen = w->mctl + 4 * nm; w->mbad[1] = w->mctl + 5 * nm;
    w->ndone = (unsigned*)(w->mctl + 6 * nm);
    w->status = w->mctl + 6 * nm + 1;
    w->bar = (unsigned*)(w->mctl + 6 * nm + 2);
    w->nlev = (unsigned*)(w->mctl + 6 * nm + 3);
    // uploads on the caller's stream, never the legacy default stream (pageable sources are
    // staged before each call returns)
    cudaMemcpyAsync(w->mem_t0, mt0.data(), 4 * nm, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(w->mem_row0, row0.data(), 4 * nm, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(w->mem_rows, rows.data(), 4 * nm, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(w->mem_tr, mtr.data(), 4 * nm, cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(w->tile_part, 0, 8 * (size_t)kPartialKinds * T, st);
    cudaMemsetAsync(w->mem_ab, 0, 64 * nm, st);
    cudaMemsetAsync(w->mctl, 0, 4 * (6 * nm + 4), st);
    cudaStreamSynchronize(st);
    return cudaGetLastError();
}

void jcg_work_free(JcgWork* w) {
    if (!w) return;
    void* ps[] = {w->mem_t0, w->mem_row0, w->mem_rows, w->mem_tr, w->tile_part, w->mem_atol2, w->mem_ab, w->mctl};
    for (void* p : ps) cudaFree(p);
    delete w;
}

cudaError_t jcg_clear(JcgWork* w, cudaStream_t st) {
    const size_t nm = w->nmem;
    cudaError_t e = cudaMemsetAsync(w->mdone, 0xFF, 4 * nm, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(w->mouter, 0, 4 * (5 * nm + 4), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(w->mgen, 0x7F, 4 * nm, st);
    return e;
}

cudaError_t jcg_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st, int nsm) {
    if ((a.sell != nullptr) != w->sell) return cudaErrorInvalidValue;
    if (a.precision != GS_FP32_IR) return jcg64_launch(a, w, st, nsm);
    return w->sell ? jcg_mg_launch(a, w, st, nsm) : jcg_ir_launch(a, w, st, nsm);
}

cudaError_t jcg_read_iters(JcgWork* w, std::vector<int>& iters, std::vector<int>& outer, cudaStream_t st) {
    iters.resize(w->nmem);
    outer.resize(w->nmem);
    cudaMemcpyAsync(iters.data(), w->mdone, 4 * (size_t)w->nmem, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(outer.data(), w->mouter, 4 * (size_t)w->nmem, cudaMemcpyDeviceToHost, st);
    return cudaStreamSynchronize(st);
}

int32_t* jcg_iters_device(JcgWork* w) { return w->mdone; }

cudaError_t jcg_read_status(JcgWork* w, int32_t* flags, cudaStream_t st) {
    cudaMemcpyAsync(flags, w->status, 4, cudaMemcpyDeviceToHost, st);
    return cudaStreamSynchronize(st);
}

}  // namespace gs
