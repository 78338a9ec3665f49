"""Autotuner on the GPU (gpu): every chosen shape is accepted by the library, stream-kernel
shapes leave the results bit-identical, and a different solver tiling stays within the solver's
tolerance."""
import numpy as np
import pytest

from gschism_b200 import autotune, cases

pytestmark = pytest.mark.gpu


def test_tuned_shapes_valid_and_results_unchanged(native, tmp_path):
    from gschism_b200.model import Model
    c = cases.basin(n=120, nvrt=12, nz=4, nsteps=20)
    shapes = autotune.tuned_shapes([c], precision="fp64", warmup=2, rounds=1, path=str(tmp_path / "t.json"))
    assert set(shapes) == set(autotune.TUNE_ORDER)
    # the cache answers the second call
    assert autotune.tuned_shapes([c], precision="fp64", path=str(tmp_path / "t.json")) == shapes

    ref = Model([c], precision="fp64")
    ref.step(6)
    streams = Model([c], precision="fp64")
    autotune.apply(streams, {k: v for k, v in shapes.items() if k != "JCG_TILES"})
    assert all(streams.get_launch(k) == v for k, v in shapes.items() if k != "JCG_TILES")
    streams.step(6)
    for f in ("ETA2", "SIDE_U2", "ELEM_TR", "SIDE_BTU"):
        assert np.array_equal(streams.get(0, f), ref.get(0, f)), f

    tiled = Model([c], precision="fp64")
    tiled.set_launch("JCG_TILES", 37, 64)           # a tiling far from the default
    assert tiled.get_launch("JCG_TILES") == (37, 64)
    tiled.step(6)
    eta, eta_ref = tiled.get(0, "ETA2"), ref.get(0, "ETA2")
    assert np.abs(eta - eta_ref).max() <= 1e-10 * np.abs(eta_ref).max()


def test_invalid_shapes_rejected(native):
    from gschism_b200._lib import GsError
    from gschism_b200.model import Model
    m = Model([cases.channel()])
    for k, a, b in (("BTRACK", 256, 16), ("GHAT", 48, 16), ("GHAT", 128, 0), ("JCG_TILES", 100, 100)):
        with pytest.raises(GsError):
            m.set_launch(k, a, b)
    assert m.get_launch("BTRACK") == (128, 32)


def test_reported_shape_is_the_one_that_runs(native):
    """The node gathers take shapes of up to 1,024 threads and run with 256 at most; gs_get_launch says so,
    and the results do not depend on it."""
    from gschism_b200.model import Model
    c = cases.channel()
    ref, m = Model([c]), Model([c])
    for k in ("NODAL_VEL", "NODAL_TRACER"):
        for block in (512, 1024):
            m.set_launch(k, block, 8)
            assert m.get_launch(k) == (256, 8)
        m.set_launch(k, 64, 8)
        assert m.get_launch(k) == (64, 8)
        m.set_launch(k, 512, 1)
    ref.step(3)
    m.step(3)
    for f in ("NODE_U2", "NODE_W2", "NODE_TR"):
        assert np.array_equal(m.get(0, f), ref.get(0, f)), f
    ref.close()
    m.close()
