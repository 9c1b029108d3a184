"""Very uneven sizes and clouds with most points in one place: the way of an evaluation follows from how far the
points reach, not from the clouds' mean variance and radius."""
import numpy as np
import pytest

from dugma_b200 import api
from tests.test_sparse_pairs import _problem

pytestmark = pytest.mark.gpu


def _cluster(P, share, radius, rng):
    k = int(share * len(P))
    P[:k] = P[0] + radius * rng.standard_normal((k, P.shape[1]))


@pytest.mark.parametrize("call", ["grad", "energy", "conv", "compi"])
def test_way_of_uneven_clouds(call):
    """The same covariances and sigma: sparse on an even surface; all pairs where the sources are few, where
    most points lie in one place, and where one far point stretches both clouds' radii."""
    run = {"grad": lambda h, R, t, s: api.energy_grad(h, R, t, s), "energy": lambda h, R, t, s: api.energy(h, R, t, s),
           "conv": lambda h, R, t, s: api.energy_grad(h, R, t, s, model=1),
           "compi": lambda h, R, t, s: api.compi(h, R, t, sig=s)}[call]
    rng = np.random.default_rng(1)

    def way(X, XC, Y, YC, R, t, sig):
        _, h = api.init(X, XC, Y, YC)
        run(h, R, t, sig)
        took = api.last_pass(h)[0]
        api.fr_m(h)
        return took

    X, XC, Y, YC, R, t = _problem("sphere", 8001, 7001, 1)
    assert way(X, XC, Y, YC, R, t, 1e-3) == 1
    A, B = X.copy(), Y.copy()
    _cluster(A, 0.95, 0.003, rng)
    _cluster(B, 0.95, 0.003, rng)
    assert way(A, XC, B, YC, R, t, 1e-3) == 0
    A, B = X.copy(), Y.copy()
    A[3], B[5] = 1e4, -1e4
    assert way(A, XC, B, YC, R, t, 1e-3) == 1 and way(A, XC, B, YC, R, t, 3.0) == 0
    X, XC, Y, YC, R, t = _problem("sphere", 64, 300000, 2)
    assert way(X, XC, Y, YC, R, t, 1e-3) == 0


def test_line_is_the_same_in_every_init():
    """The samples behind the choice are taken by index: a sigma on either side of the line goes the same way in
    every init of the data, although the spatial order inside a grid cell may differ."""
    X, XC, Y, YC, R, t = _problem("outliers", 8001, 7001, 1)

    def way(sig):
        _, h = api.init(X, XC, Y, YC)
        api.energy(h, R, t, sig)
        took = api.last_pass(h)[0]
        api.fr_m(h)
        return took

    lo, hi = 1e-5, 10.0
    assert way(lo) == 1 and way(hi) == 0
    while hi / lo > 1 + 1e-9:
        mid = np.sqrt(lo * hi)
        lo, hi = (mid, hi) if way(mid) else (lo, mid)
    assert all(way(lo) == 1 and way(hi) == 0 for _ in range(20))
