"""The momentum solve's two forms (gpu): a batch of many sides with few levels runs without the loads ahead.
A member gets the same bits alone and in such a batch."""
import numpy as np
import pytest

from gschism_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvrt", [3, 5, 8, 9])
def test_member_beside_a_large_one_equals_its_solo_run(native, nvrt):
    from gschism_b200.model import Model
    cs = [cases.basin(seed=3 + k, n=n, nvrt=nvrt, nz=2, ntr=1, length=500.0 * n, tau=(1e-4, 5e-5), dt=60.0)
          for k, n in enumerate((30, 170))]
    for c in cs:
        c.params.dramp = 0.05
    mix, solo = Model(cs), Model(cs[:1])
    assert sum(s["ns"] for s in mix.sizes) > 148 * 512 >= solo.sizes[0]["ns"]
    mix.step(4)
    solo.step(4)
    for f in ("SIDE_U2", "SIDE_QH", "ETA2", "ELEM_W"):
        assert np.array_equal(mix.get(0, f), solo.get(0, f)), f
    assert np.abs(solo.get(0, "SIDE_U2")).max() > 0.0
    mix.close()
    solo.close()
