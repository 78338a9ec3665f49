// Structure of the multilevel hierarchy of the FP32 refinement solve.  Rows are numbered along a
// Hilbert curve, so four consecutive rows are neighbours in space: level 1 joins rows 4I .. 4I+3 of
// a member, level k + 1 joins four consecutive rows of level k.  The coarse matrices are the sums of
// the fine entries over pairs of aggregates; only their structure is built here, with one byte per
// entry that says to which slot of the aggregate's row it is added.
#include <algorithm>

#include "mg.h"

namespace gs {

namespace {

// Neighbour lists of one level: row i has cols[ptr[i]] .. cols[ptr[i + 1] - 1].
struct Graph {
    std::vector<int32_t> ptr, cols;
};

// What build() found: everything built, offsets beyond 32 bits, or (>= 0) the member with a coarse row
// wider than a map byte can name.
enum { kBuilt = -1, kTooLarge = -2 };

// `on`: members with a hierarchy
int build(const std::vector<int>& row0, const std::vector<int>& rows, const std::vector<int32_t>& nnp_s,
          const std::vector<int32_t>& nnp, const std::vector<uint8_t>& on, MgHost& H) {
    H = MgHost();
    const int nmem = (int)rows.size();
    // fine slices, relative to each member's first row
    H.mem_s.resize(nmem);
    H.mem_c.assign(nmem, -1);
    const int N = nmem ? row0.back() + rows.back() : 0;
    H.row_at.resize(N);
    int64_t off = 0;
    for (int m = 0; m < nmem; m++) {
        H.mem_s[m] = (int)H.A.sl.size();
        for (int b = 0; b < rows[m]; b += 32) {
            int w = 0;
            for (int i = row0[m] + b; i < row0[m] + std::min(rows[m], b + 32); i++) w = std::max(w, nnp_s[i + 1] - nnp_s[i]);
            H.A.sl.push_back(int2{(int)off, w});
            off += 32LL * w;
        }
    }
    if (off > 0x7fffffffLL) return kTooLarge;
    H.A.idx.resize((size_t)off);
    H.A.map.assign((size_t)off, kMgDiag);
    for (int m = 0; m < nmem; m++)
        for (int b = 0; b < rows[m]; b += 32) {
            const int2 s = H.A.sl[H.mem_s[m] + b / 32];
            for (int l = 0; l < 32; l++) {
                const int i = row0[m] + b + l;
                const int deg = b + l < rows[m] ? nnp_s[i + 1] - nnp_s[i] : 0;
                const int self = std::min(i, row0[m] + rows[m] - 1);
                for (int k = 0; k < s.y; k++)
                    H.A.idx[(size_t)s.x + 32 * (size_t)k + l] = k < deg ? nnp[nnp_s[i] + k] : self;
                if (b + l < rows[m]) H.row_at[i] = s.x + l;
            }
        }
    // level 1: a member's rows start at a multiple of kMgChunk, so that on every level four rows
    // share one parent and a member's first row has a whole number of ancestors
    int n1 = 0;
    for (int m = 0; m < nmem; m++) {
        if (!on[m]) continue;
        H.mem_c[m] = n1;
        const int c = ((rows[m] + 3) / 4 + kMgChunk - 1) / kMgChunk;
        n1 += c * kMgChunk;
        H.chunk_mem.insert(H.chunk_mem.end(), c, m);
        for (int k = 0; k < c; k++)
            H.chunk_fine.push_back(int2{row0[m] + 4 * kMgChunk * k, std::min(4 * kMgChunk, rows[m] - 4 * kMgChunk * k)});
    }
    n1 = (n1 + kMgPad - 1) / kMgPad * kMgPad;
    H.chunk_mem.resize(n1 / kMgChunk, -1);
    H.chunk_fine.resize(n1 / kMgChunk, int2{0, 0});
    Graph g;                      // of the level just built
    g.ptr.reserve(n1 + 1);
    g.ptr.push_back(0);
    std::vector<int32_t> own;
    for (int m = 0; m < nmem; m++) {
        const int cb = H.mem_c[m];
        if (cb < 0) continue;
        g.ptr.resize(cb + 1, (int)g.cols.size());
        for (int a = 0; a < rows[m]; a += 4) {
            const int I = cb + a / 4;
            own.clear();
            for (int j = a; j < std::min(rows[m], a + 4); j++) {
                const int i = row0[m] + j;
                for (int k = 0; k < nnp_s[i + 1] - nnp_s[i]; k++) {
                    const int J = cb + (nnp[nnp_s[i] + k] - row0[m]) / 4;
                    if (J == I) continue;
                    const size_t slot = std::find(own.begin(), own.end(), J) - own.begin();
                    if (slot == own.size()) own.push_back(J);
                    if (slot >= (size_t)kMgMaxSlots) return m;
                    H.A.map[(size_t)H.row_at[i] + 32 * (size_t)k] = (uint8_t)slot;
                }
            }
            g.cols.insert(g.cols.end(), own.begin(), own.end());
            g.ptr.push_back((int)g.cols.size());
        }
    }
    g.ptr.resize(n1 + 1, (int)g.cols.size());
    for (int lev = 0, n = n1; lev < kMgLevels; lev++, n /= 4) {
        H.n[lev] = n;
        MgHostMatrix& A = H.lv[lev];
        A.sl.resize(n / 32);
        off = 0;
        for (int s = 0; s < n / 32; s++) {
            int w = 0;
            for (int i = 32 * s; i < 32 * s + 32; i++) w = std::max(w, g.ptr[i + 1] - g.ptr[i]);
            A.sl[s] = int2{(int)off, w};
            off += 32LL * w;
        }
        if (off > 0x7fffffffLL) return kTooLarge;
        A.idx.resize((size_t)off);
        for (int s = 0; s < n / 32; s++)
            for (int l = 0; l < 32; l++) {
                const int i = 32 * s + l, deg = g.ptr[i + 1] - g.ptr[i];
                for (int k = 0; k < A.sl[s].y; k++)
                    A.idx[(size_t)A.sl[s].x + 32 * (size_t)k + l] = k < deg ? g.cols[g.ptr[i] + k] : i;
            }
        if (lev + 1 == kMgLevels) break;
        A.map.assign((size_t)off, kMgDiag);
        Graph c;
        c.ptr.reserve(n / 4 + 1);
        c.ptr.push_back(0);
        for (int I = 0; I < n / 4; I++) {
            own.clear();
            for (int i = 4 * I; i < 4 * I + 4; i++)
                for (int k = 0; k < g.ptr[i + 1] - g.ptr[i]; k++) {
                    const int J = g.cols[g.ptr[i] + k] / 4;
                    if (J == I) continue;
                    const size_t slot = std::find(own.begin(), own.end(), J) - own.begin();
                    if (slot == own.size()) own.push_back(J);
                    if (slot >= (size_t)kMgMaxSlots) return H.chunk_mem[((size_t)I << (2 * (lev + 1))) / kMgChunk];
                    A.map[(size_t)A.sl[i / 32].x + 32 * (size_t)k + i % 32] = (uint8_t)slot;
                }
            c.cols.insert(c.cols.end(), own.begin(), own.end());
            c.ptr.push_back((int)c.cols.size());
        }
        g = std::move(c);
    }
    return kBuilt;
}

}  // namespace

bool mg_build(const std::vector<int>& row0, const std::vector<int>& rows, const std::vector<int32_t>& nnp_s,
              const std::vector<int32_t>& nnp, MgHost& H) {
    // a member with too wide a coarse row goes without the hierarchy, the others keep theirs
    std::vector<uint8_t> on(rows.size());
    for (size_t m = 0; m < rows.size(); m++) on[m] = rows[m] >= kMgMinRows;
    for (;;) {
        const int r = build(row0, rows, nnp_s, nnp, on, H);
        if (r < 0) return r == kBuilt;
        on[r] = 0;
    }
}

}  // namespace gs
