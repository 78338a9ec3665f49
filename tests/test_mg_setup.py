"""Structure of the refinement solve's hierarchy (mg_setup.cpp) on the CPU: which members of a batch
get one.  The choice depends on the member alone, so that a member gives the same bits alone and in
any batch."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "gschism_b200", "csrc")

HARNESS = r"""
#include "mg.h"
// mem_c of every member (its first row on level 1, -1: no hierarchy); returns -1 where mg_build refuses
extern "C" int mg_members(int nmem, const int* rows, const int32_t* nnp_s, const int32_t* nnp, int32_t* mem_c) {
    std::vector<int> row0(nmem), rw(rows, rows + nmem);
    int n = 0;
    for (int m = 0; m < nmem; m++) { row0[m] = n; n += rw[m]; }
    std::vector<int32_t> s(nnp_s, nnp_s + n + 1), c(nnp, nnp + nnp_s[n]);
    gs::MgHost H;
    if (!gs::mg_build(row0, rw, s, c, H)) return -1;
    for (int m = 0; m < nmem; m++) mem_c[m] = H.mem_c[m];
    return 0;
}
"""


@pytest.fixture(scope="module")
def mg(tmp_path_factory):
    d = tmp_path_factory.mktemp("mg")
    src, lib = d / "harness.cpp", d / "libmg.so"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-I/usr/local/cuda/include", str(src),
                    os.path.join(CSRC, "mg_setup.cpp"), "-o", str(lib)], check=True)
    return ctypes.CDLL(str(lib))


def _lattice(nx, ny):
    """Neighbour lists of a lattice with one diagonal (six neighbours inside)."""
    out = []
    for j in range(ny):
        for i in range(nx):
            out.append([(j + b) * nx + i + a for a, b in ((-1, 0), (1, 0), (0, -1), (0, 1), (1, 1), (-1, -1))
                        if 0 <= i + a < nx and 0 <= j + b < ny])
    return out


def _members(mg, graphs):
    rows = np.array([len(g) for g in graphs], dtype=np.int32)
    flat, ptr, r0 = [], [0], 0
    for g in graphs:
        for nb in g:
            flat.extend(r0 + c for c in nb)
            ptr.append(len(flat))
        r0 += len(g)
    a = [np.array(v, dtype=np.int32) for v in (ptr, flat)]
    mem_c = np.full(len(graphs), -7, dtype=np.int32)
    p = [v.ctypes.data_as(ctypes.c_void_p) for v in (rows, a[0], a[1], mem_c)]
    assert mg.mg_members(len(graphs), *p) == 0
    return mem_c


@pytest.mark.parametrize("nx,ny,on", [(20, 20, False), (63, 65, False), (64, 64, True), (80, 90, True)])
def test_line_between_plain_and_hierarchy(mg, nx, ny, on):
    """4,095 rows and fewer have no hierarchy, alone and beside a large member."""
    g, big = _lattice(nx, ny), _lattice(110, 90)
    assert (_members(mg, [g])[0] >= 0) == on
    c = _members(mg, [g, big])
    assert (c[0] >= 0) == on and c[1] >= 0


def _hub(n, spokes):
    """A path of n rows whose first row is also a neighbour of every eighth one, `spokes` times."""
    g = [[j for j in (i - 1, i + 1) if 0 <= j < n] for i in range(n)]
    for k in range(1, spokes + 1):
        g[0].append(8 * k)
        g[8 * k].append(0)
    return g


@pytest.mark.parametrize("spokes,on", [(200, True), (300, False)])
def test_wide_coarse_row_drops_only_its_own_member(mg, spokes, on):
    """A coarse row of more than 255 neighbours leaves that member without the hierarchy; its neighbours in
    the batch keep theirs, as they would alone."""
    hub, other = _hub(8 * 600, spokes), _lattice(70, 70)
    assert (_members(mg, [hub])[0] >= 0) == on
    for batch, k in (([other, hub, other], 1), ([hub, other], 0)):
        c = _members(mg, batch)
        assert (c[k] >= 0) == on
        assert all(v >= 0 for i, v in enumerate(c) if i != k)


def test_wide_row_on_a_higher_level(mg):
    """300 neighbours of the sixteen rows of one level-2 aggregate, at most 80 of any four of them."""
    n = 16 * 400
    g = [[j for j in (i - 1, i + 1) if 0 <= j < n] for i in range(n)]
    for k in range(300):
        a, b = k % 16, 16 * (k + 10)
        g[a].append(b)
        g[b].append(a)
    other = _lattice(70, 70)
    c = _members(mg, [other, g, other])
    assert c[0] >= 0 and c[1] < 0 and c[2] >= 0


def test_values_written_in_the_launch_are_read_coherently():
    """The coarse matrices are written by the launch that reads them: ld.global.nc and __ldg, which need
    data that no thread writes during the kernel, may only read the structure and the constant inputs."""
    text = open(os.path.join(CSRC, "jcg_mg.cu")).read()
    assert re.findall(r"ld\.global\.nc\S*\.(\w+) ", text) == ["s32"]
    for arg in re.findall(r"__ldg\(([^;]*?)\)[;,]? ?", text):
        assert not re.search(r"\.val\b|\bDinv\b|\.D\b|\.rh\b|\.e\b|\bJ\.[uzwpsdx]\b", arg), arg


def test_no_exit_with_copies_in_flight():
    """Every way out of the solve's kernel behind the first barrier waits for the thread's own asynchronous
    copies: slices are requested before the barrier that may end the kernel."""
    text = open(os.path.join(CSRC, "jcg_mg.cu")).read()
    body = text[text.index("__global__"):text.index("static size_t mg_shared")]
    assert "leave_unless(bar.sync(J, stall))" in re.search(r"#define MG_SYNC\(\) (.*)", text).group(1)
    leave = text[text.index("void leave_unless"):]
    assert re.search(r"@p cp\.async\.wait_all; @p exit;", leave[:leave.index("\n}")])
    loop = body[body.index("MG_SYNC"):]
    assert "return;" not in loop                        # a failed wait is the only early exit
    assert re.search(r"if \(S\.none\) \{ ring_drain\(\); break; \}", loop)
