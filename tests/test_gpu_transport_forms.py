"""The transport step's forms (gpu): a member's tracers are the same bits whatever form its batch takes.

The vertical sweep takes one tracer per thread below about 66,000 elements and all tracers of a column
above; the horizontal update made with the whole remaining time is made again for members whose
admissible sub-step is shorter.  Both depend on the batch, the arithmetic does not."""
import numpy as np
import pytest

from gschism_b200 import cases

pytestmark = pytest.mark.gpu


def _case(seed, n, itr_met, levels=7):
    c = cases.transport_stress(seed=seed, n=n, nvrt=levels, ntr=3, tau_mag=0.3, limiter=3, dfh0=1e-4)
    c.params.itr_met = itr_met
    c.params.maxiter = 40
    return c


def _transport(model, scale):
    """One transport step on fluxes `scale` times those of the second step, member by member."""
    model.step(2)
    for m, s in enumerate(scale):
        qh = model.get(m, "SIDE_QH")
        model.put(m, "SIDE_QH", np.where(qh > -1e30, s * qh, qh))
    model.phase("TRANSPORT", 3)
    model.sync()


@pytest.mark.parametrize("itr_met", [1, 3, 4])
def test_small_member_beside_a_large_one(native, itr_met):
    from gschism_b200.model import Model
    small = [_case(1, 33, itr_met), _case(2, 50, itr_met)]
    large = _case(3, 400, itr_met)
    assert 2 * 399 * 399 > 148 * 2048
    scale = [1.0, 4000.0]                      # the second member needs several sub-steps
    mix = Model(small + [large])
    _transport(mix, scale + [1.0])
    assert mix.stats(0)["transport_substeps"] == 1
    assert mix.stats(1)["transport_substeps"] > 1
    for k, c in enumerate(small):
        solo = Model([c])
        _transport(solo, scale[k:k + 1])
        assert solo.stats(0)["transport_substeps"] == mix.stats(k)["transport_substeps"]
        for f in ("ELEM_TR", "NODE_TR"):
            assert np.array_equal(mix.get(k, f), solo.get(0, f)), (k, f)
        solo.close()
    mix.close()
