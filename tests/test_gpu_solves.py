"""The elevation solves at the edges of their forms: the mixed-precision solve with its aggregation
hierarchy (jcg_mg.cu) against the FP64 oracle, members alone and in batches (gpu).

Sizes: both sides of the 4,096-row line between plain Jacobi and the hierarchy, and row counts that
are no multiple of an aggregate (4), a slice (32) or a chunk of 1,024 rows.  A Delaunay mesh of random
points has nodes with more than eight neighbours, whose slices are read past the shared-memory ring.

Bound: a solve stops at |b - A x| <= 1e-12 |b|; the mass matrix bounds A from below by the smallest
element areas, and measured against the FP64 oracle the elevations of these meshes differ by less
than 1e-11 of the largest one after a step, so 1e-9 leaves two digits for three steps."""
import numpy as np
import pytest

from gschism_b200 import cases
from tests._parity import relerr

pytestmark = pytest.mark.gpu


def _basin(seed, side):
    c = cases.basin(seed=seed, n=side, nvrt=4, nz=2, ntr=1, length=500.0 * side)
    c.params.dramp = 0.05
    return c


def _delaunay(seed, side):
    """A basin of the same outline on random interior points (node degrees 3 to about 12)."""
    spatial = pytest.importorskip("scipy.spatial")
    c = _basin(seed, side)
    rng = np.random.default_rng(seed)
    length = 500.0 * side
    bnd = np.unique(np.concatenate(c.open_bnd + c.land_bnd))
    inner = np.setdiff1d(np.arange(c.n_nodes), bnd)
    lo, hi = 250.0, length - 250.0
    c.x[inner], c.y[inner] = rng.uniform(lo, hi, inner.size), rng.uniform(lo, hi, inner.size)
    # the outline bulges slightly, so that every boundary node is a corner of the hull
    bx, by = c.x[bnd] / length - 0.5, c.y[bnd] / length - 0.5
    sx, sy = np.abs(bx) >= np.abs(by), np.abs(by) >= np.abs(bx)
    c.x[bnd] += np.where(sx, np.sign(bx) * 100.0 * (0.25 - by ** 2), 0.0)
    c.y[bnd] += np.where(sy, np.sign(by) * 100.0 * (0.25 - bx ** 2), 0.0)
    tri = spatial.Delaunay(np.stack([c.x, c.y], 1)).simplices
    a, b, d = (np.stack([c.x[tri[:, k]], c.y[tri[:, k]]], 1) for k in range(3))
    ccw = (b[:, 0] - a[:, 0]) * (d[:, 1] - a[:, 1]) - (d[:, 0] - a[:, 0]) * (b[:, 1] - a[:, 1]) > 0
    tri = np.where(ccw[:, None], tri, tri[:, ::-1])
    c.elnode = np.ascontiguousarray(tri, dtype=np.int32)
    deg = np.bincount(c.elnode.ravel(), minlength=c.n_nodes)
    assert deg.max() > 8
    return c


@pytest.mark.parametrize("make", [lambda: _basin(11, 63), lambda: _basin(12, 64), lambda: _basin(13, 65),
                                  lambda: _basin(14, 101), lambda: _delaunay(15, 80)],
                         ids=["3969", "4096", "4225", "10201", "delaunay6400"])
def test_elevation_against_oracle(native, oracle_lib, make):
    from gschism_b200.model import Model
    from oracle.step_api import OracleModel
    c = make()
    o = OracleModel(c)
    o.run(3)
    g = Model([c], precision="fp32_ir")
    g.step(3)
    st = g.stats(0)
    assert st["error_flags"] == 0
    assert relerr(g.get(0, "ETA2"), o.get("ETA2")) <= 1e-9
    g.close()


@pytest.mark.parametrize("tiles", [None, (40, 32)])
def test_members_equal_their_solo_runs(native, tiles):
    """Members on both sides of the line, and one with wide rows, in one context: bit for bit the
    results of each member alone, with the default tiles and with 32-row ones."""
    from gschism_b200.model import Model
    cs = [_basin(21, 40), _delaunay(22, 70), _basin(23, 101), _basin(24, 66)]
    mix = Model(cs, precision="fp32_ir")
    if tiles:
        mix.set_launch("JCG_TILES", *tiles)
    mix.step(3)
    for k, c in enumerate(cs):
        solo = Model([c], precision="fp32_ir")
        if tiles:
            solo.set_launch("JCG_TILES", *tiles)
        solo.step(3)
        assert np.array_equal(mix.get(k, "ETA2"), solo.get(0, "ETA2")), k
        assert mix.stats(k)["jcg_iters"] == solo.stats(0)["jcg_iters"]
        solo.close()
    mix.close()


def test_fp64_member_in_a_batch_beyond_shared_memory(native):
    """The FP64 solve holds the matrix in shared memory while it fits; a batch of more rows reads it
    from global memory with other launch shapes.  A member gets the same bits in both."""
    from gschism_b200.model import Model
    cs = [_basin(31, 45), _basin(32, 640)]
    mix = Model(cs, precision="fp64", maxiter=60)
    solo = Model(cs[:1], precision="fp64", maxiter=60)
    mix.step(2)
    solo.step(2)
    assert np.array_equal(mix.get(0, "ETA2"), solo.get(0, "ETA2"))
    assert mix.stats(0)["jcg_iters"] == solo.stats(0)["jcg_iters"]
    mix.close()
    solo.close()


def _solve_ms(model, first, solves=8):
    """Shortest time of the SOLVE phase over some steps (CUDA events)."""
    import torch
    from gschism_b200.autotune import PhaseTimer
    timer = PhaseTimer(model, first_step=first)
    ts = [timer.step()["SOLVE"] for _ in range(solves)]
    torch.cuda.synchronize()
    return min(ts)


def test_batch_is_no_slower_than_its_members_one_after_another(native):
    """A small member's iterations do not carry a large member's phases: one solve of the batch takes no more
    time than solves of its members in turn (measured 0.91; 1.9 when they did)."""
    from gschism_b200.model import Model
    cs = [_basin(41, 40), _basin(42, 63), _basin(43, 200)]
    times = []
    for group in [cs] + [[c] for c in cs]:
        m = Model(group, precision="fp32_ir")
        m.step(8)
        times.append(_solve_ms(m, 9))
        m.close()
    assert times[0] <= 1.25 * sum(times[1:]), times


@pytest.mark.parametrize("side", [31, 32, 33, 45, 46, 63, 64])
def test_elevation_at_the_lines(native, oracle_lib, side):
    """Both sides of the lines between two, four and eight rows a thread of a block's own solve (1,024 and 2,048
    rows) and between it and the hierarchy (4,096), against the oracle."""
    from gschism_b200.model import Model
    from oracle.step_api import OracleModel
    c = _basin(50 + side, side)
    o = OracleModel(c)
    o.run(3)
    g = Model([c], precision="fp32_ir")
    g.step(3)
    assert g.stats(0)["error_flags"] == 0
    assert relerr(g.get(0, "ETA2"), o.get("ETA2")) <= 1e-9
    g.close()


@pytest.mark.parametrize("inner_maxiter", [1, 2, 400])
def test_small_and_large_members_equal_their_solo_runs(native, inner_maxiter):
    """Members on both sides of the line in one context, bit for bit their solo results; with one or two
    iterations a sweep every member leaves the hierarchy after sweeps that do not halve the residual."""
    from gschism_b200.model import Model
    cs = [_basin(61, 20), _basin(62, 33), _basin(63, 63), _basin(64, 64), _basin(65, 90)]
    mix = Model(cs, precision="fp32_ir", ir_inner_maxiter=inner_maxiter)
    mix.step(2)
    for k, c in enumerate(cs):
        solo = Model([c], precision="fp32_ir", ir_inner_maxiter=inner_maxiter)
        solo.step(2)
        assert np.array_equal(mix.get(k, "ETA2"), solo.get(0, "ETA2")), k
        assert mix.stats(k)["jcg_iters"] == solo.stats(0)["jcg_iters"]
        assert mix.stats(k)["jcg_outer"] == solo.stats(0)["jcg_outer"]
        solo.close()
    mix.close()


@pytest.mark.parametrize("side", [6, 8, 22, 23])
def test_elevation_of_a_block_member(native, oracle_lib, side):
    """Small members solved by one block: fewer rows than two slices, and both sides of one row per thread,
    against the oracle."""
    from gschism_b200.model import Model
    from oracle.step_api import OracleModel
    c = _basin(70 + side, side)
    o = OracleModel(c)
    o.run(3)
    g = Model([c], precision="fp32_ir")
    g.step(3)
    assert g.stats(0)["error_flags"] == 0
    assert relerr(g.get(0, "ETA2"), o.get("ETA2")) <= 1e-9
    g.close()


def test_parked_block_member_is_done_at_once(native):
    """A zero right-hand side: solved by x = 0 without an iteration, beside members that iterate."""
    from gschism_b200.model import Model
    cs = [_basin(81, 20), _basin(82, 25), _basin(83, 70)]
    m = Model(cs, precision="fp32_ir")
    m.park(0, m.member_state(0))
    m.step(2)
    assert m.stats(0)["jcg_iters"] == 0 and m.stats(0)["error_flags"] == 0
    assert np.abs(m.get(0, "ETA2")).max() == 0.0
    for k in (1, 2):
        solo = Model(cs[k:k + 1], precision="fp32_ir")
        solo.step(2)
        assert np.array_equal(m.get(k, "ETA2"), solo.get(0, "ETA2"))
        solo.close()
    m.close()


def test_timed_out_member_is_reported_and_the_context_recovers(native):
    """The recovery path (test_gpu_recovery.py) with a stalled member that one block solves, alone and beside
    a large member, and with the large one stalled: the wait runs out, is reported once, and the context
    steps on bit for bit."""
    from gschism_b200 import _lib as L
    from gschism_b200.model import Model
    both = [_basin(84, 20), _basin(85, 70)]
    for cs, stalled in ((both[:1], 0), (both, 0), (both, 1)):
        ref, m = (Model(cs, precision="fp32_ir") for _ in range(2))
        ref.step(3)
        m.step(2)
        saved = [m.member_state(k) for k in range(len(cs))]
        m.set_wait_limit(1 << 14)
        m.test_stall_solve(stalled)
        m.step(1)
        with pytest.raises(L.GsError) as ei:
            m.sync()
        assert ei.value.status == L.GS_ERR_TIMEOUT
        m.sync()
        m.test_stall_solve(-1)
        m.set_wait_limit(0)
        for k in range(len(cs)):
            m.put_member_state(k, saved[k])
        m.phase("BEGIN", 2)
        m.step(1)
        m.sync()
        for k in range(len(cs)):
            assert np.array_equal(m.get(k, "ETA2"), ref.get(k, "ETA2")), k
            assert m.stats(k)["error_flags"] == 0
        m.close()
        ref.close()


@pytest.mark.parametrize("precision,most", [("fp32_ir", 3.0), ("fp64", 2.4)])
def test_many_small_members_do_not_wait_for_one_another(native, precision, most):
    """256 members of 400 rows take less than `most` times the time of one (measured 2.2 and 2.1; 4.6 and 2.6
    when members waited for one another)."""
    from gschism_b200.model import Model
    times = []
    for n in (1, 256):
        m = Model([_basin(100 + k, 20) for k in range(n)], precision=precision)
        m.step(8)
        times.append(_solve_ms(m, 9))
        m.close()
    assert times[1] <= most * times[0], times


@pytest.mark.parametrize("sides", [[45, 120, 173], [20, 25, 30, 18] * 24], ids=["held", "small"])
def test_fp64_members_of_shared_blocks_equal_their_solo_runs(native, sides):
    """FP64 batches with more tiles than blocks, matrix held and not: bit for bit the solo results."""
    from gschism_b200.model import Model
    cs = [_basin(200 + k, s) for k, s in enumerate(sides)]
    assert sum(max(1, (s * s + 255) // 256) for s in sides) > 148
    mix = Model(cs, precision="fp64")
    mix.step(2)
    for k in range(0, len(cs), max(1, len(cs) // 8)):
        solo = Model(cs[k:k + 1], precision="fp64")
        solo.step(2)
        assert np.array_equal(mix.get(k, "ETA2"), solo.get(0, "ETA2")), k
        assert mix.stats(k)["jcg_iters"] == solo.stats(0)["jcg_iters"]
        solo.close()
    mix.close()


def test_block_member_gets_the_same_bits_in_every_form(native):
    """A thread of a block's solve holds as many rows as the context's largest small member needs; a member's
    bits do not depend on that."""
    from gschism_b200.model import Model
    small = _basin(91, 24)
    solo = Model([small], precision="fp32_ir")
    solo.step(3)
    for side in (40, 60):
        m = Model([_basin(92, side), small], precision="fp32_ir")
        m.step(3)
        assert np.array_equal(m.get(1, "ETA2"), solo.get(0, "ETA2")), side
        m.close()
    solo.close()
