"""Evaluations over the pairs above the FP32 flush against all pairs (DUGMA_ALL_PAIRS=1 at init):
the same FP32 terms and sums, so equal to the rounding of FP64 additions (1e-12 of the result; a
gradient's sums cancel by less than 1e3 here), on clouds whose covariances follow the spacing, with
outliers, ill-conditioned and neglected covariances, coincident and far points, poses that are no
rotation, and points that are not finite or near overflow."""
import numpy as np
import pytest

from dugma_b200 import api, synth

pytestmark = pytest.mark.gpu


def _problem(kind, n, m, seed):
    rng = np.random.default_rng(seed)
    k = max(n, m)
    if kind == "curve":
        P = synth.workload5(trial=seed, n=k)
    elif kind == "outliers":
        P = synth.workload1(trial=seed, n=k)
    elif kind == "harmonic":
        P = synth.workload2(trial=seed, n=k)
    else:
        P = synth.workload0(trial=seed, n=k)
    i, j = rng.permutation(k)[:n], rng.permutation(k)[:m]
    X, XC, Y, YC = P.X[i].copy(), P.X_C[i].copy(), P.Y[j].copy(), P.Y_C[j].copy()
    D = X.shape[1]
    if kind == "neglected":
        XC[::7] = 0.0
        YC[::5, 0, 0] *= -1.0
    elif kind == "coincident":
        X[: n // 2] = X[0]
        Y[: m // 3] = (X[0] - P.t_G) @ P.R_G      # R_G^T (x - t)
    elif kind == "far":
        Y[m // 2:] += 1e3
        X[0] = -1e4
    elif kind == "mixed_scales":
        XC *= np.exp(rng.uniform(-4, 4, n))[:, None, None]
        YC *= np.exp(rng.uniform(-4, 4, m))[:, None, None]
    elif kind == "nearly_singular":   # flat covariances, some along the same plane: the FP64 path
        flat = np.diag([1e-3, 1e-3, 1e-11][:D])
        XC[::2], YC[::3] = flat, P.R_G.T @ flat @ P.R_G
    elif kind == "not_finite":
        Y[3, 0] = np.inf
    elif kind == "huge":
        Y[5] = 3e18
        XC[0] = 1e-18 * np.eye(D)
    return X, XC, Y, YC, P.R_G, P.t_G


ENERGY = {"grad": lambda h, R, t, sig: api.energy_grad(h, R, t, sig)[:2],
          "grad_dx": lambda h, R, t, sig: api.energy_grad(h, R, t, sig, with_dx=True),
          "energy": lambda h, R, t, sig: (api.energy(h, R, t, sig),),
          "fd": lambda h, R, t, sig: (api.energy_fd_grad(h, R, t, sig)[0],)}
CONV = {"conv_grad": lambda h, R, t, sig: api.energy_grad(h, R, t, sig, model=1, with_dx=True),
        "conv_energy": lambda h, R, t, sig: (api.energy(h, R, t, sig, model=1),)}
COEF = {"compi": lambda h, R, t, sig: (api.compi(h, R, t, sig=sig),)}


def _evaluate(monkeypatch, calls, prob, R, t, sig, all_pairs):
    if all_pairs:
        monkeypatch.setenv("DUGMA_ALL_PAIRS", "1")
    else:
        monkeypatch.delenv("DUGMA_ALL_PAIRS", raising=False)
    _, h = api.init(*prob[:4])
    out = {}
    try:
        for name, fn in calls.items():
            try:
                out[name] = [np.asarray(v) for v in fn(h, R, t, sig)]
            except api.DugmaError as e:
                out[name] = e.code
    finally:
        api.fr_m(h)
    return out


KINDS = ["sphere", "outliers", "harmonic", "curve", "neglected", "coincident", "far", "mixed_scales", "not_finite",
         "huge"]


def _compare(monkeypatch, calls, kind, n, m, sigs):
    prob = _problem(kind, n, m, 3)
    R, t = prob[4], prob[5]
    for scale in (1.0, 1.05):        # a rotation, and a matrix that stretches
        for sig in sigs:
            a = _evaluate(monkeypatch, calls, prob, scale * R, t + 0.01, sig, False)
            b = _evaluate(monkeypatch, calls, prob, scale * R, t + 0.01, sig, True)
            for name in b:
                if isinstance(b[name], int) or isinstance(a[name], int):
                    assert isinstance(b[name], int) and a[name] == b[name], (name, a[name], b[name])
                    continue
                for u, v in zip(a[name], b[name]):
                    assert np.all(np.isfinite(u) == np.isfinite(v)), name
                    u, v = u[np.isfinite(u)], v[np.isfinite(v)]
                    assert np.linalg.norm(u - v) <= 1e-12 * np.linalg.norm(v), (name, sig, u, v)


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("n,m", [(4001, 3100), (20001, 1025), (1001, 20033)])
@pytest.mark.parametrize("kind", KINDS)
def test_energy_same_sums_as_all_pairs(kind, n, m, monkeypatch):
    _compare(monkeypatch, ENERGY, kind, n, m, (2e-4, 4e-3, 3e-2))


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("n,m", [(6401, 6301), (40001, 1025), (1001, 40033)])
@pytest.mark.parametrize("kind", KINDS + ["nearly_singular"])
def test_conv_same_sums_as_all_pairs(kind, n, m, monkeypatch):
    _compare(monkeypatch, CONV, kind, n, m, (2e-4, 2e-3, 8e-3))


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("n,m", [(5001, 4901), (40001, 1025), (1001, 40033)])
@pytest.mark.parametrize("kind", KINDS)
def test_compi_same_sums_as_all_pairs(kind, n, m, monkeypatch):
    _compare(monkeypatch, COEF, kind, n, m, (4e-4, 2e-2))


@pytest.mark.parametrize("widen", [1.0, 1e4])   # (1e4: sigma beyond the rule, all pairs run)
def test_em_step_is_update_sig_and_compi(widen):
    """An EM step decides on the device what compi decides on the host: the same bits either way."""
    X, XC, Y, YC, R, t = _problem("sphere", 5001, 4999, 1)
    _, h = api.init(X, XC * widen, Y, YC * widen)
    em = api.EMGraph(h)
    sig, A = em(R, t + 0.01)
    assert sig == api.update_sig(h, R, t + 0.01)
    assert np.array_equal(A, api.compi(h, R, t + 0.01, sig=sig))
    em.close()
    api.fr_m(h)


def test_batch_same_sums_as_all_pairs(monkeypatch):
    """Problems of uneven sizes, sparse and dense poses mixed, every tile shape."""
    probs = [_problem(k, n, m, 5) for k, n, m in (("sphere", 2500, 3001), ("outliers", 5000, 1999), ("sphere", 300, 280),
                                                  ("harmonic", 3333, 2222))]
    R = np.array([[p[4], p[4] @ p[4], np.eye(3)] for p in probs])
    t = np.array([[p[5] + 0.01, p[5], p[5]] for p in probs])
    sig = np.array([[2e-3, 1e-2, 3.0]] * len(probs))
    out = []
    for all_pairs in (False, True):
        if all_pairs:
            monkeypatch.setenv("DUGMA_ALL_PAIRS", "1")
        b = api.Batch([p[:4] for p in probs])
        got = []
        for shape in api.Batch.shapes():
            b.set_shape(shape)
            got += list(b.energy_grad(R, t, sig))
        again = b.energy_grad(R, t, sig)
        assert all(np.array_equal(u, v) for u, v in zip(got[-2:], again))
        b.close()
        out.append(got)
    for u, v in zip(*out):
        assert np.all(np.linalg.norm((u - v).reshape(len(probs), 3, -1), axis=2)
                      <= 1e-12 * np.linalg.norm(v.reshape(len(probs), 3, -1), axis=2))


@pytest.mark.parametrize("model", [0, 1])
def test_device_pose_is_host_pose(model):
    """Where only the device knows sigma (a pose in device memory) a flag picks the pass that a host pose
    picks on the host: the same bits, below the rule's line (3e-4) and above it (1)."""
    import torch
    from dugma_b200 import _lib
    X, XC, Y, YC, R, t = _problem("sphere", 16385, 16001, 2)
    _, h = api.init(X, XC, Y, YC)
    s = torch.cuda.Stream()
    pose, out = torch.zeros(16, dtype=torch.float64, device="cuda"), torch.zeros(8, dtype=torch.float64, device="cuda")
    dx = torch.zeros(len(X), 3, dtype=torch.float64, device="cuda")
    for sig in (3e-4, 1.0, 3e-4):
        pose[:9] = torch.tensor(np.asarray(R).T.reshape(-1))
        pose[9:12] = torch.tensor(t + 0.01)
        pose[12] = sig
        torch.cuda.synchronize()
        assert _lib.load().dugma_energy_grad_async(h.arr, pose.data_ptr(), model, out.data_ptr(), dx.data_ptr(),
                                                   s.cuda_stream) == 0
        torch.cuda.synchronize()
        E, g, d = api.energy_grad(h, R, t + 0.01, sig, model=model, with_dx=True)
        got = out.cpu().numpy()
        assert got[0] == E and np.array_equal(got[1:7], np.asarray(g).reshape(-1))
        assert np.array_equal(dx.cpu().numpy().reshape(-1), np.asarray(d).reshape(-1))
    api.fr_m(h)


@pytest.mark.parametrize("kind,m", [("sphere", 70001), ("sphere", 300001), ("not_finite", 270000)])
def test_many_super_tiles(kind, m, monkeypatch):
    """Targets beyond 64 super tiles (65536 points), whose tests the block shares, and beyond the 128 or 256
    that it tests together: the same sums as all pairs."""
    _compare(monkeypatch, {**ENERGY, **CONV, **COEF}, kind, 501, m, (2e-4, 4e-3))
