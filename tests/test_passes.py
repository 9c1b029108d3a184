"""Which way an evaluation goes (api.last_pass): the comparisons of the sparse passes with all pairs do
compare two different passes, and inputs on which they can differ -- points that overflow FP32 beside
finite statistics, batches of several slabs -- against all pairs (DUGMA_ALL_PAIRS=1 at init) to the
rounding of FP64 additions, 1e-12."""
import numpy as np
import pytest

from dugma_b200 import api
from tests.test_sparse_pairs import COEF, CONV, ENERGY, _problem

pytestmark = pytest.mark.gpu


def _run(monkeypatch, calls, prob, R, t, sig, all_pairs):
    """{name: (the pass taken, outputs or error code)}"""
    if all_pairs:
        monkeypatch.setenv("DUGMA_ALL_PAIRS", "1")
    else:
        monkeypatch.delenv("DUGMA_ALL_PAIRS", raising=False)
    _, h = api.init(*prob[:4])
    out = {}
    try:
        for name, fn in calls.items():
            try:
                got = [np.asarray(v) for v in fn(h, R, t, sig)]
            except api.DugmaError as e:
                got = e.code
            out[name] = (api.last_pass(h)[0], got)
    finally:
        api.fr_m(h)
    return out


def _same(a, b, name):
    if isinstance(a, int) or isinstance(b, int):
        assert isinstance(a, int) and isinstance(b, int) and a == b, (name, a, b)
        return
    for u, v in zip(a, b):
        assert np.array_equal(np.isfinite(u), np.isfinite(v)), name
        u, v = u[np.isfinite(u)], v[np.isfinite(v)]
        assert np.linalg.norm(u - v) <= 1e-12 * np.linalg.norm(v), (name, u, v)


SPARSE = [(ENERGY, 6001, 5100), (ENERGY, 20001, 4001), (CONV, 7001, 6301), (CONV, 20001, 5025), (COEF, 6001, 5901)]


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("calls,n,m", SPARSE)
@pytest.mark.parametrize("kind", ["sphere", "outliers", "harmonic", "curve"])
def test_sparse_pass_is_taken(kind, calls, n, m, monkeypatch):
    prob = _problem(kind, n, m, 3)
    R, t = prob[4], prob[5] + 0.01
    for all_pairs in (False, True):
        for name, (took, _) in _run(monkeypatch, calls, prob, R, t, 2e-5, all_pairs).items():
            assert took == (0 if all_pairs else 1), (name, took)


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("calls,n,m", SPARSE)
@pytest.mark.parametrize("what", ["inf_target", "inf_source", "inf_corner"])
def test_points_beyond_fp32(what, calls, n, m, monkeypatch):
    """A coordinate that is finite in FP64 and infinite in FP32: the other cloud's radius keeps the
    evaluation sparse."""
    X, XC, Y, YC, R, t = _problem("harmonic", n, m, 4)
    if what == "inf_target":
        Y[3, 0] = 1e39
    elif what == "inf_source":
        X[n // 2, 1] = -1e39
    else:
        Y[m - 1] = 1e39
    prob = (X, XC, Y, YC)
    for sig in (2e-5, 2e-3):
        a = _run(monkeypatch, calls, prob, R, t + 0.01, sig, False)
        b = _run(monkeypatch, calls, prob, R, t + 0.01, sig, True)
        for name in b:
            assert b[name][0] == 0 and (sig > 1e-4 or a[name][0] == 1), (name, a[name][0])
            _same(a[name][1], b[name][1], name)


def test_batch_of_several_slabs(monkeypatch):
    """More source rows than one sparse launch takes (4M), among sparse and dense poses."""
    probs = [_problem(k, 20001, 1301, s) for s, k in enumerate(("sphere", "harmonic", "sphere", "outliers", "sphere"))]
    Q = 48
    R = np.array([[p[4]] * Q for p in probs])
    t = np.array([[p[5] + 0.001 * q for q in range(Q)] for p in probs])
    sig = np.array([[1e-4] * (Q - 1) + [10.0]] * len(probs))
    out = []
    for all_pairs in (False, True):
        if all_pairs:
            monkeypatch.setenv("DUGMA_ALL_PAIRS", "1")
        b = api.Batch([p[:4] for p in probs])
        out.append(b.energy_grad(R, t, sig))
        took = b.last_pass()
        assert took[:2] == ((0, 0) if all_pairs else (len(probs) * (Q - 1), 2)), took
        b.close()
    for u, v in zip(*out):
        for p in range(len(probs)):
            for q in range(Q):
                _same([u[p, q]], [v[p, q]], (p, q))


def _needles(n, m, seed):
    """Half of each cloud on a line with needle covariances along it (condition 5e4: their pairs fail the
    FP32 path's test, yet have a bound on their reach), the sources' on one side and the targets' on the
    other, half beside the whole line with round ones."""
    rng = np.random.default_rng(seed)
    u = np.array([0.48, -0.6, 0.64])

    def cloud(k, side):
        s, needle = rng.uniform(-1, 1, k), rng.uniform(size=k) < 0.5
        P = np.outer(np.where(needle, side * (0.1 + 0.9 * np.abs(s)), s), u)
        P += np.where(needle, 1e-4, 0.02)[:, None] * rng.standard_normal((k, 3))
        v = u + 1e-3 * rng.standard_normal((k, 3))
        v *= rng.uniform(0.9, 1.1, (k, 1)) / np.linalg.norm(v, axis=1)[:, None]
        flat = 1e-3 * v[:, :, None] * v[:, None, :] + 2e-8 * np.eye(3)
        return P, np.where(needle[:, None, None], flat, 1e-3 * np.eye(3))

    return (*cloud(n, -1.0), *cloud(m, 1.0), np.eye(3), np.zeros(3))


@pytest.mark.parametrize("n,m", [(7001, 6301), (12001, 5001)])
def test_conv_of_needles(n, m, monkeypatch):
    """A pair that fails the FP32 path's test is evaluated in FP64; what the FP32 path made of it has no
    say in which term is the largest, whether or not the pass comes upon that pair."""
    prob = _needles(n, m, 5)
    for sig in (5e-5, 1e-4, 2e-4):
        a = _run(monkeypatch, CONV, prob, prob[4], prob[5] + 1e-3, sig, False)
        b = _run(monkeypatch, CONV, prob, prob[4], prob[5] + 1e-3, sig, True)
        for name in b:
            assert (a[name][0], b[name][0]) == (1, 0), (name, a[name][0])
            _same(a[name][1], b[name][1], name)


def test_conv_with_a_boundless_covariance(monkeypatch):
    """A covariance so large that its weight is 0 in FP32 (but its determinant positive): the CONV model still
    has its pairs, and the sparse pass does not take it for a point without variance."""
    X, XC, Y, YC, R, t = _problem("harmonic", 7001, 6301, 3)
    XC[5] = YC[9] = 1e31 * np.eye(3)
    a = _run(monkeypatch, CONV, (X, XC, Y, YC), R, t + 0.01, 1e-5, False)
    b = _run(monkeypatch, CONV, (X, XC, Y, YC), R, t + 0.01, 1e-5, True)
    for name in b:
        assert (a[name][0], b[name][0]) == (1, 0) and b[name][1][0] > 0, (name, a[name][0], b[name][1][0])
        _same(a[name][1], b[name][1], name)
