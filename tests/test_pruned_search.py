"""The pruned nearest-neighbour search (spatial order, spheres) against the all-pairs kernels, which
a pinned shape (distances and indices) or a row range (sigma's sums) runs: the same bits on every
form of input, among them ties, coincident and non-finite points, a far outlier, clouds that do
not overlap, and poses that are no rotation."""
import numpy as np
import pytest

from dugma_b200 import api, synth

pytestmark = pytest.mark.gpu


def _clouds(kind, n, m, D, rng):
    X, Y = rng.uniform(-1, 1, (n, D)), rng.uniform(-1, 1, (m, D))
    if kind == "surface" and D == 3:
        X, Y = synth.bumpy_sphere(rng, n), synth.bumpy_sphere(rng, m)
    elif kind == "lattice":      # many equal distances
        X, Y = np.round(4 * X) / 4, np.round(4 * Y) / 4
    elif kind == "one_point":
        X[:], Y[:] = 0.25, -0.5
    elif kind == "outlier":
        Y[m // 2] = 1e4
        X[0] = -3e3
    elif kind == "apart":
        Y += 50.0
    elif kind == "not_finite":
        X[n // 2, 0] = np.nan
        Y[m // 3] = np.inf
        Y[m // 2, D - 1] = np.nan
    return X, Y


def _pose(kind, D, rng):
    if D == 2:
        c, s = np.cos(0.4), np.sin(0.4)
        R = np.array([[c, -s], [s, c]])
    else:
        R = synth.random_rotation(rng, 60.0)
    return (R @ np.diag([1.6, 0.4, 2.0][:D]) if kind == "stretch" else R), 0.1 * rng.standard_normal(D)


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("n,m", [(1, 1), (31, 40), (32, 32), (33, 129), (1000, 37), (65, 2100), (4097, 3000)])
@pytest.mark.parametrize("kind", ["surface", "lattice", "one_point", "outlier", "apart", "not_finite"])
def test_same_bits_as_all_pairs(kind, n, m, D):
    rng = np.random.default_rng(n * 31 + m * 7 + D)
    X, Y = _clouds(kind, n, m, D, rng)
    eye = lambda k: np.broadcast_to(np.eye(D), (k, D, D))  # noqa: E731
    _, h = api.init(X, eye(n), Y, eye(m))
    try:
        for pose in ("rotation", "stretch"):
            R, t = _pose(pose, D, rng)
            parts = sum(api.sigma_range(h, R, t, a, b) for a, b in ((0, n // 2), (n // 2, n)) if b - a < n) \
                if n > 1 else None
            got = {k: api.nn(h, R, t, k) for k in (1, 5, 16) if k <= m}
            sig = api.update_sig(h, R, t)
            if parts is not None:
                assert sig == float(np.float32(parts[1] / 1e6 / n))
            _, b = api.init(X, eye(n), Y, eye(m))
            api.set_shape(b, 2, api.shapes(2)[0])
            assert np.array_equal(sig, api.update_sig(b, R, t))
            for k, (idx, d2) in got.items():
                i0, d0 = api.nn(b, R, t, k)
                assert np.array_equal(d2, d0, equal_nan=True)
                assert np.array_equal(idx, i0)
            api.fr_m(b)
    finally:
        api.fr_m(h)
