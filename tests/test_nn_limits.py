"""The pruned search where FP32 ends: distances that overflow, points that are not finite, distances below
the smallest normal number.  Against the all-pairs kernels (a pinned shape): the same bits, also the mark
of a neighbour that does not exist."""
import numpy as np
import pytest

from dugma_b200 import api

pytestmark = pytest.mark.gpu


def _pinned(X, Y, R, t, ks):
    D = X.shape[1]
    eye = lambda n: np.broadcast_to(np.eye(D), (n, D, D))  # noqa: E731
    _, h = api.init(X, eye(len(X)), Y, eye(len(Y)))
    got = [api.nn(h, R, t, k) for k in ks], api.update_sig(h, R, t)
    assert api.last_pass(h)[2] == 1
    api.set_shape(h, 2, api.shapes(2)[0])
    want = [api.nn(h, R, t, k) for k in ks], api.update_sig(h, R, t)
    assert api.last_pass(h)[2] == 0
    api.fr_m(h)
    return got, want


def _same(got, want):
    for (i, d), (i0, d0) in zip(got[0], want[0]):
        assert np.array_equal(d, d0) and np.array_equal(i, i0)
    assert got[1] == want[1]


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("n,m", [(5, 40), (1500, 1300)])
@pytest.mark.parametrize("far", [1e20, 3e38, np.inf, np.nan])
def test_infinite_distances_are_no_neighbours(far, n, m, D):
    rng = np.random.default_rng(3)
    X, Y = rng.uniform(-1, 1, (n, D)), rng.uniform(-1, 1, (m, D))
    Y[3:] += 0.5 * far        # fewer targets in reach of a distance than neighbours asked for
    X[n // 2] = far
    _same(*_pinned(X, Y, np.eye(D), np.zeros(D), (1, 5, 16)))


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("scale", [1e-18, 1e-19, 1e-20, 1e-21, 3e-22, 1e-24])
def test_distances_below_the_normal_numbers(scale, D):
    rng = np.random.default_rng(4)
    X, Y = scale * rng.uniform(-1, 1, (2100, D)), scale * rng.uniform(-1, 1, (3000, D))
    _same(*_pinned(X, Y, np.eye(D), 0.1 * scale * np.ones(D), (1, 8)))


@pytest.mark.parametrize("n", [40, 3000])
def test_covariances_of_points_without_neighbours(n):
    """A point with no finite distance to another has no neighbours: the others' covariances are what they
    are without it, its own is the least one, or not finite like its coordinates."""
    rng = np.random.default_rng(5)
    P = rng.uniform(-1, 1, (n, 3))
    Q = np.concatenate([P, [[1e39, 0.0, 0.0], [np.nan, 0.0, 0.0], [0.0, -1e39, 1.0]]])
    got = api.knn_covariance(Q, 8, 1e-6, 1e-2)
    assert np.array_equal(got[:n], api.knn_covariance(P, 8, 1e-6, 1e-2))
    for k in (n, n + 2):
        assert np.array_equal(got[k], 1e-6 * np.eye(3))
