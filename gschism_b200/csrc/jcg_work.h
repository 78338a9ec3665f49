// Work list and per-member control words of a solve.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace gs {

struct JcgArgs;

struct JcgWork {
    int nmem = 0, ntiles = 0;
    int nsmall = 0, small_rows = 0;  // members below kMgMinRows rows, rows of the largest of them
    bool sell = false;               // rows in the SELL-32 layout of a context, else a caller's CSR
    // per member: first tile, first row, rows, rows per tile
    int32_t *mem_t0 = nullptr, *mem_row0 = nullptr, *mem_rows = nullptr, *mem_tr = nullptr;
    double *tile_part = nullptr, *mem_atol2 = nullptr, *mem_ab = nullptr;
    // per-member control words in one array: mdone, mouter, minner, mbad[0], mgen, mbad[1] ([nmem] each),
    // ndone, status (ERR_JCG_NOT_CONVERGED of the last solve), bar (grid barrier), nlev (members
    // that iterate with the coarse correction in a sweep)
    int32_t* mctl = nullptr;
    int32_t* status = nullptr;
    int32_t *mdone = nullptr, *mouter = nullptr, *minner = nullptr, *mgen = nullptr;
    int32_t* mbad[2] = {nullptr, nullptr};
    unsigned *ndone = nullptr, *bar = nullptr, *nlev = nullptr;
};

// Control words at the start of a solve: mdone = -1, mgen = 0x7f7f7f7f, the others 0.
cudaError_t jcg_clear(JcgWork* w, cudaStream_t st);
// jcg64.cu: the FP64 solve
cudaError_t jcg64_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st, int nsm);
// jcg_mg.cu: the refinement solve of a context (a.mg set); jcg_small.cu: its members below kMgMinRows rows
cudaError_t jcg_mg_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st, int nsm);
cudaError_t jcg_small_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st);
// jcg_ir.cu: the refinement solve of a caller's CSR matrix
cudaError_t jcg_ir_launch(const JcgArgs& a, JcgWork* w, cudaStream_t st, int nsm);

}  // namespace gs
