"""A pinned kernel shape is the one that runs, at every size; without a pin small problems run the default
shape with fewer sources per thread, and the autotuner times them that way."""
import numpy as np
import pytest

from dugma_b200 import api, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

CALLS = [lambda h, P: api.energy_grad(h, P.R_G, P.t_G, 0.05)[:2], lambda h, P: (api.energy(h, P.R_G, P.t_G, 0.05),)]


@pytest.mark.parametrize("what", [0, 1])
@pytest.mark.parametrize("D", [2, 3])
def test_pinned_shape_runs(D, what):
    P = synth.workload5(trial=4, n=1500) if D == 2 else synth.workload0(trial=4, n=1500)
    _, h = api.init(P.X, P.X_C, P.Y, P.Y_C)
    Eo, go = orc.State(P.X, P.X_C, P.Y, P.Y_C).energy(P.R_G, P.t_G, 0.05)[:2]
    want = CALLS[what](h, P)
    assert api.last_pass(h)[:2] == (0, 1)
    default = api.get_shape(h, what)
    for shape in api.shapes(what):
        api.set_shape(h, what, shape)
        got = CALLS[what](h, P)
        assert api.last_pass(h)[:2] == (0, shape[0]), shape
        assert abs(got[0] - Eo) <= 1e-6 * Eo
        if what == 0:
            assert np.linalg.norm(got[1] - go) <= 1e-5 * np.linalg.norm(go)
    api.set_shape(h, what, default)   # the same tiles and chunks: FP64 additions regroup
    got = CALLS[what](h, P)
    assert default[0] == 4 and api.last_pass(h)[1] == 4
    assert all(np.linalg.norm(np.subtract(u, v)) <= 1e-12 * np.linalg.norm(v) for u, v in zip(got, want))
    api.fr_m(h)


def test_autotune_times_what_runs():
    P = synth.workload0(trial=4, n=1500)
    _, h = api.init(P.X, P.X_C, P.Y, P.Y_C)
    last = api.shapes(0)[-1]
    assert last == (4, 64, 64, 2)
    api.set_shape(h, 0, last)
    api.autotune(h, 0)
    assert api.last_pass(h)[:2] == (0, 1)        # the last candidate, the default shape, as a call runs it
    best = api.get_shape(h, 0)
    CALLS[0](h, P)
    assert api.last_pass(h)[1] == (1 if best == last else best[0])
    api.fr_m(h)
