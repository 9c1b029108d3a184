"""Very uneven sizes and clouds with most points in one place: what a rule made for even surfaces sends the
slow way.  The searches give the bits of all pairs whichever way they go; the way of an evaluation follows
from how far the points reach, not from the clouds' mean variance and radius."""
import numpy as np
import pytest

from dugma_b200 import api
from tests.test_sparse_pairs import _problem

pytestmark = pytest.mark.gpu


def _cluster(P, share, radius, rng):
    k = int(share * len(P))
    P[:k] = P[0] + radius * rng.standard_normal((k, P.shape[1]))


@pytest.mark.parametrize("cluster", [False, True])
@pytest.mark.parametrize("n,m,pruned", [(32, 16383, (1, 1)), (32, 16384, (0, 0)), (257, 20000, (1, 0)), (300, 240000, (0, 0)),
                                        (3999, 16384, (1, 0)), (4000, 16384, (1, 1)), (262144, 256, (0, 0)),
                                        (262144, 257, (1, 1))])
def test_search_of_uneven_clouds(n, m, pruned, cluster):
    rng = np.random.default_rng(n + m)
    X, Y = rng.uniform(-1, 1, (n, 3)), rng.uniform(-1, 1, (m, 3))
    if cluster:
        _cluster(X, 0.9, 0.003, rng)
        _cluster(Y, 0.9, 0.003, rng)
    eye = lambda k: np.broadcast_to(np.eye(3), (k, 3, 3))  # noqa: E731
    R, t = np.eye(3), np.array([0.01, -0.02, 0.0])
    _, h = api.init(X, eye(n), Y, eye(m))
    got = [api.update_sig(h, R, t), api.sigma(h, R, t)]
    assert api.last_pass(h)[2] == pruned[cluster]
    got += list(api.nn(h, R, t, 1))
    assert api.last_pass(h)[2] == pruned[cluster]
    got += list(api.nn(h, R, t, 5))
    assert api.last_pass(h)[2] == 1
    got.append(api.update_sig(h, R, t))
    api.set_shape(h, 2, api.shapes(2)[0])
    want = [api.update_sig(h, R, t), api.sigma(h, R, t), *api.nn(h, R, t, 1), *api.nn(h, R, t, 5), api.update_sig(h, R, t)]
    assert api.last_pass(h)[2] == 0
    assert all(np.array_equal(u, v) for u, v in zip(got, want))
    api.fr_m(h)


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
