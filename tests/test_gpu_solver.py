"""Stand-alone JCG on a caller CSR (PCGSolverMultiGPU drop-in) against the oracle's JCG (gpu)."""
import numpy as np
import pytest

from gschism_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system(oracle_lib):
    """An elevation system assembled by the oracle after a few channel steps."""
    from oracle.step_api import OracleModel
    c = cases.channel(seed=21)
    o = OracleModel(c)
    o.run(3)
    o.begin_step(4)
    o.btrack()
    o.prepare_elevation(4 * c.params.dt)
    o.assemble(4 * c.params.dt)
    o.essential_bc()
    A = (o.get("CSR_INDPTR"), o.get("CSR_INDICES"), o.get("CSR_DATA"))
    b = o.get("QEL")
    hist = (o.get("JCG_X"), o.get("JCG_X1"), o.get("JCG_X2"))
    its, rel = o.jcg_solve(1e-12, 1500, 10)
    return A, b, hist, its, o.get("JCG_X"), rel


def _fill(s, A, b):
    import torch
    ip, ix, da = A
    s.csr_indptr(0).copy_(torch.as_tensor(ip))
    s.csr_indices(0).copy_(torch.as_tensor(ix))
    s.csr_data(0).copy_(torch.as_tensor(da))
    s.b_m[0].copy_(torch.as_tensor(b))


def test_jcg_csr_matches_oracle(native, system):
    from gschism_b200.solver import PCGSolverMultiGPU
    A, b, hist, its_o, x_o, rel_o = system
    s = PCGSolverMultiGPU(None, [b.size], [A[2].size])
    _fill(s, A, b)
    # a fresh solver starts from x = 0 (empty history), the oracle from its parabolic guess:
    # both solutions meet rtol = 1e-12 and agree to the conditioning of the system
    its = s.solve(rtol=1e-12, maxiter=1500, checkEvery=10)
    assert 0 < its < 1500
    x = s.x_m[0].cpu().numpy()
    assert s.checkSolution() <= 1e-11
    assert rel_o <= 1e-11
    assert np.abs(x - x_o).max() <= 1e-9 * np.abs(x_o).max()
    s.close()


def test_jcg_csr_zero_rhs_returns_zero(native, system):
    from gschism_b200.solver import PCGSolverMultiGPU
    A, b, *_ = system
    s = PCGSolverMultiGPU(None, [b.size], [A[2].size])
    _fill(s, A, np.zeros_like(b))
    assert s.solve(rtol=1e-12, maxiter=100) == 0
    assert np.all(s.x_m[0].cpu().numpy() == 0.0)
    s.close()


def test_jcg_csr_maxiter_cap(native, system):
    from gschism_b200.solver import PCGSolverMultiGPU
    A, b, *_ = system
    s = PCGSolverMultiGPU(None, [b.size], [A[2].size])
    _fill(s, A, b)
    assert s.solve(rtol=1e-14, maxiter=3, checkEvery=10) == 3     # not converged: returns maxiter
    s.close()


def test_jcg_csr_mixed_precision(native, system):
    from gschism_b200.solver import PCGSolverMultiGPU
    A, b, hist, its_o, x_o, rel_o = system
    s = PCGSolverMultiGPU(None, [b.size], [A[2].size], precision="fp32_ir")
    _fill(s, A, b)
    s.solve(rtol=1e-12, maxiter=1500, checkEvery=10)
    assert s.checkSolution() <= 1e-11
    s.close()


def _tridiagonal(n):
    """CSR of a diagonally dominant tridiagonal matrix."""
    r = np.repeat(np.arange(n), 3)
    c = r + np.tile([-1, 0, 1], n)
    keep = (c >= 0) & (c < n)
    r, c = r[keep], c[keep]
    ptr = np.zeros(n + 1, dtype=np.int32)
    ptr[1:] = np.cumsum(np.bincount(r, minlength=n))
    return ptr, c.astype(np.int32), np.where(r == c, 2.5, -1.0)


def test_solvers_of_two_threads_do_not_disturb_each_other(native):
    """Solvers whose launches need different amounts of shared memory (one block, and several), solving at
    the same time from two host threads: a kernel's limit is shared by both."""
    import threading
    from gschism_b200.solver import PCGSolverMultiGPU
    rng = np.random.default_rng(5)
    solvers, results = [], [None, None]
    for n in (100, 3000):
        A = _tridiagonal(n)
        s = PCGSolverMultiGPU(None, [n], [A[2].size])
        _fill(s, A, rng.standard_normal(n))
        solvers.append(s)

    def work(k):
        try:
            results[k] = [solvers[k].solve(rtol=1e-10, maxiter=200, checkEvery=5) for _ in range(1500)]
        except Exception as e:       # reported by the main thread
            results[k] = e

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, s in enumerate(solvers):
        assert isinstance(results[k], list), results[k]
        assert s.checkSolution() <= 1e-9
        s.close()


def _banded(n, offsets):
    """CSR of a symmetric diagonally dominant matrix: -1 at the offsets (both sides), rows summing to 0.5, so
    its eigenvalues lie in [0.5, 4 len(offsets) + 0.5]."""
    off = np.array(sorted([-o for o in offsets] + [0] + list(offsets)))
    c = np.arange(n)[:, None] + off
    keep = (c >= 0) & (c < n)
    deg = keep.sum(1)
    ptr = np.zeros(n + 1, dtype=np.int32)
    ptr[1:] = np.cumsum(deg)
    v = np.where(off == 0, (deg - 1)[:, None] + 0.5, -1.0)
    return ptr, c[keep].astype(np.int32), v[keep]


_NEIGHBOURS = (1, 389)                                      # a lattice of 389 columns
_DENSE = tuple(range(1, 16))                                # 31 entries a row


@pytest.mark.parametrize("n,offsets,precision", [
    (151321, _NEIGHBOURS, "fp64"), (151321, _NEIGHBOURS, "fp32_ir"),      # several tiles and rows a thread
    (40001, _NEIGHBOURS, "fp64"), (40001, _NEIGHBOURS, "fp32_ir"),        # one slice a warp, ragged end
    (409601, _NEIGHBOURS, "fp64"), (640001, _NEIGHBOURS, "fp32_ir"),      # beyond the chip's shared memory
    (151321, _DENSE, "fp64"), (151321, _DENSE, "fp32_ir"),                # a block's rows do not fit its cache
    (1, (1,), "fp64"), (1, (1,), "fp32_ir"), (33, (1,), "fp64"), (33, (1,), "fp32_ir")])
def test_csr_forms_against_known_solution(native, n, offsets, precision):
    """Every form of the stand-alone solves against the solution the right-hand side was made from.  The solve
    stops at |r| <= 1e-12 |b|, so |x - x*| <= 1e-12 |b| / 0.5 <= 1e-12 (4 len(offsets) + 0.5) / 0.5 |x*|; the
    right-hand side is exact to rounding (1e-15 of the same factor)."""
    from gschism_b200.solver import PCGSolverMultiGPU
    ptr, idx, val = _banded(n, offsets)
    truth = np.random.default_rng(n).standard_normal(n)
    rows = np.repeat(np.arange(n), np.diff(ptr))
    b = np.bincount(rows, weights=val * truth[idx], minlength=n)
    s = PCGSolverMultiGPU(None, [n], [val.size], precision=precision)
    _fill(s, (ptr, idx, val), b)
    bound = 1.1e-12 * (4 * len(offsets) + 0.5) / 0.5
    for check in (10, 7):                                   # the second solve starts from its own history
        its = s.solve(rtol=1e-12, maxiter=600, checkEvery=check)
        assert 0 < its < 600 or check == 7
        x = s.x_m[0].cpu().numpy()
        assert np.linalg.norm(x - truth) <= bound * np.linalg.norm(truth)
        assert s.checkSolution() <= 1.01e-12
    s.close()


@pytest.mark.parametrize("n", [33, 40001])
def test_csr_zero_rhs_mixed_precision(native, n):
    """A zero right-hand side is answered with x = 0 and no iteration, also after a solve."""
    from gschism_b200.solver import PCGSolverMultiGPU
    A = _banded(n, _NEIGHBOURS)
    s = PCGSolverMultiGPU(None, [n], [A[2].size], precision="fp32_ir")
    for b in (np.zeros(n), np.ones(n), np.zeros(n)):
        _fill(s, A, b)
        its = s.solve(rtol=1e-12, maxiter=600)
        assert (its == 0) == (not b.any())
        assert b.any() or np.all(s.x_m[0].cpu().numpy() == 0.0)
    s.close()
