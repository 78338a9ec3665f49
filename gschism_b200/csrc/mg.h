// Multilevel hierarchy of the FP32 refinement solve (jcg_mg.cu): layout, host construction
// (mg_setup.cpp) and launch.
#pragma once
#include <cstdint>
#include <vector>

#include <vector_types.h>

namespace gs {

constexpr int kMgLevels = 4;          // coarse levels; level k joins 4^k consecutive rows of a member
constexpr int kMgChunk = 256;         // a member's coarse rows start at a multiple of this on level 1
constexpr int kMgPad = 2048;          // level-1 rows of the batch, so that every level has whole slices
constexpr uint8_t kMgDiag = 255;      // Galerkin map: the entry falls inside its own aggregate
constexpr int kMgMaxSlots = 255;      // widest coarse row

// FP32 matrices without their (unit) diagonal in SELL-32: entry k of row l of slice s sits at
// sl[s].x + 32 k + l for k < sl[s].y; padding entries hold the row itself and a zero value.
struct MgMatrix {
    int2* sl = nullptr;
    int32_t* idx = nullptr;
    float* val = nullptr;             // D^-1 A off the diagonal
    uint8_t* map = nullptr;           // slot of the entry in its aggregate's row one level up
};
struct MgLevel {
    int n = 0;                        // rows (a multiple of 32; rows of no aggregate stay zero)
    MgMatrix A;
    float *D = nullptr, *Dinv = nullptr;
    float *rh = nullptr;              // D^-1 (restricted residual)
    float *e = nullptr;               // correction
};
struct MgDev {
    MgMatrix A;                       // fine matrix, slices relative to the member's first row
    MgLevel lv[kMgLevels];
    float *cr = nullptr, *cd = nullptr;   // coarsest level: residual and last step of the polynomial
    int32_t *mem_s = nullptr;         // [nmem] a member's first fine slice
    int32_t *mem_c = nullptr;         // [nmem] a member's first row on level 1, -1: no hierarchy
    int32_t *chunk_mem = nullptr;     // [level-1 rows / kMgChunk] member, -1 padding
    int2 *chunk_fine = nullptr;       // first fine row of the chunk and the number of fine rows under it
    int32_t *row_at = nullptr;        // [rows] position of a row's entry 0 in A
};

// Host side: structure of every level of a batch.
struct MgHostMatrix {
    std::vector<int2> sl;
    std::vector<int32_t> idx;
    std::vector<uint8_t> map;
};
struct MgHost {
    MgHostMatrix A, lv[kMgLevels];
    int n[kMgLevels] = {0};
    std::vector<int32_t> mem_s, mem_c, chunk_mem, row_at;
    std::vector<int2> chunk_fine;
};
// Members with fewer rows have no hierarchy and are solved by one block each (jcg_small.cu).  A solve alone, by
// one block and with the hierarchy: 961 rows 0.37 and 1.46 ms, 2,025 rows 0.72 and 1.77, 3,969 rows 1.43 and
// 1.92; on short channels the gap is larger (63 x 20 nodes, 6 steps 3.4 and 14.1 ms).  64 members of 3,969 rows
// 2.0 and 3.4 ms.  Beside a 40,000-row member the block's time adds to the solve's (2,025 rows: 3.0 ms, 2.3 with the
// hierarchy).  The line is where a block's threads hold eight rows each; there the two are close.
constexpr int kMgMinRows = 4096;
// nnp_s/nnp: node -> nodes of the batch (global rows, ball order); row0/rows per member.
// A member has a hierarchy from kMgMinRows rows on, unless one of its coarse rows has more neighbours than
// a map byte can name: a property of the member alone.  Returns false when a matrix needs more than 32-bit
// offsets.
bool mg_build(const std::vector<int>& row0, const std::vector<int>& rows, const std::vector<int32_t>& nnp_s,
              const std::vector<int32_t>& nnp, MgHost& H);

}  // namespace gs
