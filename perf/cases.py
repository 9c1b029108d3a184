"""The calls whose speed is kept under watch, at the sizes, covariances and poses their users meet.

A case is one call of the public Python interface (dugma_b200.api) on one kind of cloud:

    call      api.energy_grad (REF or CONV model, with or without dE/dx), api.energy, the plain form
              api.energy_fd_grad, the plugin calls api.update_sig and api.compi, one EM iteration
              (api.EMGraph), api.nn, api.knn_covariance, api.Batch and the whole loop api.DUGMA
    cloud     sphere    bumpy sphere, covariances from the point spacing
              outliers  the same with 10 % outliers and 8-neighbour sample covariances
              harmonic  harmonic surface, 8-neighbour sample covariances (condition up to 1e4)
              depth     two depth-camera views, the sensor's depth-dependent noise
              curve     2D closed curve, covariances along the tangent
              sensor    3D surface with the wide isotropic covariances (1.3 .. 7.9 on a cloud of
                        unit radius) of the reference's Kinect scenes: every pair counts
    angle, shift   how far the pose is from the true one (degrees, length)
    widen     the energy's sigma over the one update_sig gives at that pose (annealing starts wide)
"""
import math

import numpy as np
import torch

from dugma_b200 import api, prep, synth
from dugma_b200.pose import expmap, rot2d

CONV = 1


def _case(name, call, cloud, N, M, angle=3.0, shift=0.02, widen=1.0, **more):
    return dict(name=name, call=call, cloud=cloud, N=N, M=M, angle=angle, shift=shift, widen=widen, **more)


def listed():
    return [
        # the fused adjoint (energy and pose gradient), what a pose optimiser calls: a small cloud, where
        # latency and launches count; one with outliers and the per-point gradient; the benchmark's size
        _case("grad_1k", "grad", "sphere", 1000, 1000, angle=10.0),
        _case("grad_dx_6k", "grad_dx", "outliers", 6000, 5501, angle=10.0, shift=0.05),
        _case("grad_64k", "grad", "harmonic", 65536, 65536),
        # two whole depth views, the largest clouds of the configured workloads
        _case("grad_depth_240k", "grad", "depth", 240000, 239999, angle=1.0),
        # the 2D path
        _case("grad_2d_20k", "grad", "curve", 20011, 17003),
        # each pair's own combined covariance
        _case("conv_16k", "conv_grad", "harmonic", 16000, 16384),
        # the reference's plugin calls: sigma, and the surrogate's coefficients
        _case("update_sig_64k", "update_sig", "harmonic", 65536, 65536, angle=10.0, shift=0.05),
        _case("compi_16k", "compi", "harmonic", 16384, 15000),
        # one iteration of the registration loop, and the whole loop, at the size and with the
        # covariances of a Kinect scene
        _case("em_step_4k", "em", "sensor", 4501, 3907, angle=10.0),
        _case("register_4k", "register", "sensor", 4203, 3400, angle=15.0, shift=0.1),
        # nearest neighbours with their indices (data preparation)
        _case("knn8_30k", "nn", "sphere", 30000, 28001, k=8),
        # many problems with several start poses each
        _case("batch_24x8", "batch", "sphere", 8000, 500, angle=20.0, problems=24, poses=8),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["grad", "grad", "grad", "grad_dx", "energy", "fd", "conv_grad", "update_sig", "compi", "compi",
                       "em", "nn", "knn_cov", "batch"])
    cloud = rng.choice(["sphere", "outliers", "harmonic", "depth", "curve", "sensor"])
    if call == "knn_cov" and cloud in ("sensor", "depth"):
        cloud = "harmonic"
    if call == "batch":
        hi = log(1000, 8000)
        return dict(call=call, cloud=rng.choice(["sphere", "sensor", "curve"]), N=hi, M=max(400, hi // 8),
                    angle=rng.uniform(0.5, 30.0), shift=rng.uniform(0.0, 0.1), widen=1.0, problems=rng.randint(4, 32),
                    poses=rng.randint(1, 8))
    N = log(500, 65536)
    if cloud == "depth":   # dense range maps, seen from nearly the same place: their noise is small
        N = max(N, log(20000, 65536))
    M = min(65536, max(500, int(N * math.exp(rng.uniform(-1.0, 0.7)))))
    c = dict(call=call, cloud=cloud, N=N, M=M, angle=math.exp(rng.uniform(math.log(0.3), math.log(45.0))),
             shift=rng.uniform(0.0, 0.2), widen=rng.choice([1.0, 1.0, math.exp(rng.uniform(0.0, math.log(16.0)))]))
    if cloud == "depth":
        c["angle"], c["shift"] = min(c["angle"], 3.0), 0.15 * c["shift"]
    if call in ("nn", "knn_cov"):
        c["k"] = rng.randint(1, 15)
    return c


# ------------------------------------------------------------------------------------------------
# clouds
# ------------------------------------------------------------------------------------------------
def _problem(cloud, N, M, trial):
    """(X, X_C, Y, Y_C, R_G, t_G) with N and M points in random order."""
    n = max(N, M)
    rng = np.random.Generator(np.random.PCG64([7, trial]))
    if cloud == "sensor":
        X, S = synth.bumpy_sphere(rng, N), synth.bumpy_sphere(rng, M)
        Rm, tm = synth.random_rotation(rng, 45.0), rng.uniform(-0.3, 0.3, 3)
        Y = (S + 0.005 * rng.standard_normal(S.shape)) @ Rm.T + tm
        X, Y, norm = prep.normalize(X, Y)
        cov = lambda P: (1.3 * (7.9 / 1.3) ** ((P[:, 2] + 1.0) / 3.0).clip(0.0, 1.0))[:, None, None] * np.eye(3)  # noqa: E731
        t_G = (Rm.T @ (norm.yd - tm) - norm.xd) / norm.scale
        return X, cov(X), Y, cov(Y), Rm.T, t_G
    make = {"sphere": synth.workload0, "outliers": synth.workload1, "harmonic": synth.workload2,
            "depth": synth.workload4, "curve": synth.workload5}[cloud]
    P = make(trial=trial, n=n)
    for k in range(1, 40):   # a camera that stands inside a box or too near one sees too little
        if P.N >= N and P.M >= M:
            break
        P = make(trial=40 * trial + k, n=n)
    i = rng.permutation(P.N)[:N]
    j = rng.permutation(P.M)[:M]
    return P.X[i], P.X_C[i], P.Y[j], P.Y_C[j], P.R_G, P.t_G


def _pose(case, R_G, t_G, rng):
    """The true pose turned by `angle` degrees about a random axis and moved by `shift`."""
    D = len(t_G)
    ax, sh = rng.standard_normal(3), rng.standard_normal(D)
    a = math.radians(case["angle"])
    Q = expmap(a * ax / np.linalg.norm(ax)) if D == 3 else rot2d(a * math.copysign(1.0, ax[0]))
    return Q @ R_G, t_G + case["shift"] * sh / np.linalg.norm(sh)


class _State:
    """What a program keeps between calls; the handles are released with it."""

    def __init__(self):
        self.close = []

    def __del__(self):
        for fn in reversed(self.close):
            fn()


def _inputs(case, seed):
    """The clouds and poses of a case: a list of (X, X_C, Y, Y_C) and, per problem, its (R, t) poses."""
    rng = np.random.Generator(np.random.PCG64([11, seed]))
    if case["call"] != "batch":
        X, XC, Y, YC, R_G, t_G = _problem(case["cloud"], case["N"], case["M"], seed)
        return [(X, XC, Y, YC)], [[_pose(case, R_G, t_G, rng)]]
    probs, poses = [], []
    for p in range(case["problems"]):   # sizes iid uniform in [M, N]
        n, m = (int(v) for v in rng.integers(case["M"], case["N"] + 1, 2))
        X, XC, Y, YC, R_G, t_G = _problem(case["cloud"], n, m, (seed << 8) + p)
        probs.append((X, XC, Y, YC))
        poses.append([_pose(case, R_G, t_G, rng) for _ in range(case["poses"])])
    return probs, poses


def prepare(case, seed):
    st = _State()
    st.case = case
    probs, poses = _inputs(case, seed)
    X, XC, Y, YC = probs[0]
    st.R, st.t = poses[0][0]
    call = case["call"]
    if call == "register":
        # the loop starts from the identity; the case's pose is how far that is from the truth
        R, t = poses[0][0]
        Y, YC = Y @ R.T + t, np.einsum("ab,nbc,dc->nad", R, YC, R)
        st.args = (X, Y, XC, YC, np.eye(X.shape[1]), np.zeros(X.shape[1]))
    elif call == "knn_cov":
        st.X = X
    elif call == "batch":
        st.R = np.array([[R for R, _ in q] for q in poses])
        st.t = np.array([[t for _, t in q] for q in poses])
        st.sig = np.zeros(st.R.shape[:2])
        for k, (X, XC, Y, YC) in enumerate(probs):
            h = api.init(X, XC, Y, YC)[1]
            st.sig[k] = case["widen"] * api.update_sig(h, st.R[k, 0], st.t[k, 0])
            api.fr_m(h)
        st.b = api.Batch(probs)
        st.close.append(st.b.close)
    else:
        st.h = api.init(X, XC, Y, YC)[1]
        st.close.append(lambda h=st.h: api.fr_m(h))
        if call == "em":
            st.g = api.EMGraph(st.h)
            st.close.append(st.g.close)
        elif call not in ("nn", "update_sig"):
            st.sig = case["widen"] * api.update_sig(st.h, st.R, st.t)
    return st


def run(st):
    call = st.case["call"]
    if call == "grad":
        return api.energy_grad(st.h, st.R, st.t, st.sig)[:2]
    if call == "grad_dx":
        return api.energy_grad(st.h, st.R, st.t, st.sig, with_dx=True)
    if call == "conv_grad":
        return api.energy_grad(st.h, st.R, st.t, st.sig, model=CONV)[:2]
    if call == "energy":
        return api.energy(st.h, st.R, st.t, st.sig)
    if call == "fd":
        return api.energy_fd_grad(st.h, st.R, st.t, st.sig)
    if call == "update_sig":
        return api.update_sig(st.h, st.R, st.t)
    if call == "compi":
        return api.compi(st.h, st.R, st.t, sig=st.sig)
    if call == "em":
        return st.g(st.R, st.t)
    if call == "nn":
        return api.nn(st.h, st.R, st.t, k=st.case["k"])
    if call == "knn_cov":
        return api.knn_covariance(st.X, k=st.case["k"])
    if call == "batch":
        return st.b.energy_grad(st.R, st.t, st.sig)
    assert call == "register", call
    R, t, stats = api.DUGMA(*st.args, Max_Iteration=300, accuracy_rotation=1e-4, accuracy_translation=1e-8,
                            accuracy_sig=1e-9)
    return R, t, float(stats[1]), int(stats[0])


# Gaussians that reach a point: nearly all other pairs are below the smallest FP32 number where the
# covariances follow the point spacing; the sensor clouds' covariances reach every point.
NEAR = 32


def work(case):
    """Inputs read once, outputs written once; per point its per-pose arithmetic (rotated covariance,
    record, contraction: about 200 operations) and the operations of the pairs that can count."""
    D = 2 if case["cloud"] == "curve" else 3
    call = case["call"]
    n, m, reps = case["N"], case["M"], 1
    if call == "batch":
        n = m = (case["N"] + case["M"]) // 2
        reps = case["problems"] * case["poses"]
    elif call == "register":
        reps = 30   # EM iterations, about
    elif call == "fd":
        reps = 13 if D == 3 else 7
    elif call == "knn_cov":
        m = n
    point = 4 * (D + D * D + 1)
    near = max(n, m) * (min(n, m) if case["cloud"] == "sensor" else NEAR)
    if call in ("nn", "knn_cov", "update_sig"):
        point, near, per = 4 * D, max(n, m) * NEAR, 12
    else:
        per = {"energy": 30, "fd": 30, "conv_grad": 72, "compi": 50, "em": 50, "register": 50}.get(call, 48)
    out = {"grad_dx": 8 * n * D, "nn": 8 * n * case.get("k", 1), "knn_cov": 8 * n * D * D, "compi": 5096, "em": 5104}
    return {"bytes": float(reps * (n + m) * point + out.get(call, 64 * reps)),
            "flops": float(reps * (200 * (n + m) + 2 * per * near))}


# ------------------------------------------------------------------------------------------------
# the same outputs in plain FP64 torch, from the FP32 state init leaves on the device (coordinates,
# inverse covariances, |Sigma|^-1/2; the covariances themselves for the CONV model)
# ------------------------------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f32(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float32), device=_dev()).double()


def _sym(A):
    return 0.5 * (A + A.transpose(1, 2))


def _cross(a, b):
    """a x b over the last axis (a scalar in 2D)."""
    if a.shape[-1] == 2:
        return (a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0])[..., None]
    return torch.linalg.cross(a.expand_as(b) if a.dim() == b.dim() else a, b, dim=-1)


def _rows(N, M):
    step = max(1, min(N, (1 << 24) // M))
    return [(i, min(N, i + step)) for i in range(0, N, step)]


def _exact_ref(P, R, t, sig, grad=True):
    X, XC, Y, YC = (_f32(a) for a in P)
    D, s = X.shape[1], 1.0 / sig
    R, t = (torch.as_tensor(np.asarray(a, np.float64), device=X.device) for a in (R, t))
    inv = lambda C: torch.linalg.inv(C).float().double()  # noqa: E731
    wgt = lambda C: torch.sqrt(1.0 / torch.linalg.det(C)).float().double()  # noqa: E731
    B = s * _sym(inv(XC))
    C = s * (R @ _sym(inv(YC)) @ R.T)
    w, v, Yp = wgt(XC), wgt(YC), Y @ R.T + t
    E, g, dx = 0.0, 0.0, []
    for i0, i1 in _rows(len(X), len(Y)):
        x, b = X[i0:i1], B[i0:i1]
        d = [x[:, None, a] - Yp[None, :, a] for a in range(D)]
        u = [sum(C[None, :, a, c] * d[c] for c in range(D)) for a in range(D)]
        z = [sum(b[:, None, a, c] * d[c] for c in range(D)) for a in range(D)]
        e1 = v * torch.exp(-0.5 * sum(d[a] * u[a] for a in range(D)))
        e2 = v * torch.exp(-0.5 * sum(d[a] * z[a] for a in range(D)))
        wi = w[i0:i1] * s ** D
        E = E + (wi * (e1.sum(1) + e2.sum(1))).sum()
        if not grad:
            continue
        f = torch.stack([(e1 * u[a] + e2 * z[a]).sum(1) for a in range(D)], 1)      # sum e1 C'd + e2 Bd
        pairs = ((0, 1),) if D == 2 else ((1, 2), (2, 0), (0, 1))
        dxz = torch.stack([(e2 * (d[a] * z[c] - d[c] * z[a])).sum(1) for a, c in pairs], 1)   # sum e2 d x Bd
        rot = _cross(x - t, f) - dxz
        g = g + torch.cat([(wi[:, None] * rot).sum(0), (wi[:, None] * f).sum(0)])
        dx.append(-wi[:, None] * f)
    return (E, g, torch.cat(dx)) if grad else (E, None, None)


def _exact_conv(P, R, t, sig):
    X, XC, Y, YC = (_f32(a) for a in P)
    D = X.shape[1]
    R, t = (torch.as_tensor(np.asarray(a, np.float64), device=X.device) for a in (R, t))
    Sx, Sy, Yp = sig * _sym(XC), sig * (R @ _sym(YC) @ R.T), Y @ R.T + t
    E, g = 0.0, 0.0
    for i0, i1 in _rows(len(X), 8 * len(Y)):
        d = X[i0:i1, None] - Yp[None]
        inv = torch.linalg.inv(Sx[i0:i1, None] + Sy[None])
        u = (inv @ d[..., None])[..., 0]
        n = torch.sqrt(torch.linalg.det(inv)) * torch.exp(-0.5 * (d * u).sum(-1)) * (2 * math.pi) ** (-D / 2)
        A = Sx[i0:i1, None] @ inv
        Su = (Sx[i0:i1, None] @ u[..., None])[..., 0]
        ax = (A[..., 0, 1] - A[..., 1, 0])[..., None] if D == 2 else torch.stack(
            [A[..., 1, 2] - A[..., 2, 1], A[..., 2, 0] - A[..., 0, 2], A[..., 0, 1] - A[..., 1, 0]], -1)
        rot = _cross((X[i0:i1] - t)[:, None].expand_as(u), u) - _cross(Su, u) + ax
        E = E + n.sum()
        g = g + torch.cat([(n[..., None] * rot).sum((0, 1)), (n[..., None] * u).sum((0, 1))])
    return E, g


def _exact_nn(X, Yp, k):
    X, Yp = X.double(), Yp.double()
    out = []
    for i0, i1 in _rows(len(X), len(Yp)):
        d2 = sum((X[i0:i1, None, a] - Yp[None, :, a]) ** 2 for a in range(X.shape[1]))
        out.append(torch.topk(d2, k, largest=False, sorted=True).values)
    return torch.cat(out)


def exact(case, seed):
    call = case["call"]
    # no independent 64-bit form here: the 637 coefficients (their FP64 check is the oracle's), the loop,
    # and the largest clouds (minutes in FP64)
    if call in ("compi", "em", "register") or case["N"] * case["M"] > 5e9:
        return None
    probs, poses = _inputs(case, seed)
    num = lambda *v: tuple(x if x is None else float(x) if x.dim() == 0 else x.cpu().numpy() for x in v)  # noqa: E731
    if call == "batch":
        E, G = [], []
        st = prepare(case, seed)   # for the sigmas, an input of this call
        for p, P in enumerate(probs):
            got = [_exact_ref(P, R, t, st.sig[p, q]) for q, (R, t) in enumerate(poses[p])]
            E.append([float(e) for e, _, _ in got])
            G.append([g.cpu().numpy() for _, g, _ in got])
        return np.array(E), np.array(G)
    P = probs[0]
    R, t = poses[0][0]
    if call in ("nn", "update_sig"):
        # the searched positions are FP32: y' = float(R y + t)
        Yp = torch.as_tensor((np.float32(P[2]).astype(np.float64) @ R.T + t).astype(np.float32), device=_dev())
        d2 = _exact_nn(_f32(P[0]), Yp, case.get("k", 1))
        return (None, d2.cpu().numpy()) if call == "nn" else float(d2.mean() / P[0].shape[1])
    if call == "knn_cov":
        X = _f32(P[0])
        idx = []
        for i0, i1 in _rows(len(X), len(X)):
            d2 = sum((X[i0:i1, None, a] - X[None, :, a]) ** 2 for a in range(X.shape[1]))
            d2[torch.arange(i1 - i0), torch.arange(i0, i1)] = -1.0   # the point itself first
            idx.append(torch.topk(d2, case["k"] + 1, largest=False).indices)
        Q = torch.as_tensor(P[0], device=X.device)[torch.cat(idx)]
        Q = Q - Q.mean(1, keepdim=True)
        lam, V = torch.linalg.eigh((Q.transpose(1, 2) @ Q / case["k"]).cpu())
        return (V * lam.clamp(1e-6, 1e-2)[:, None, :] @ V.transpose(1, 2)).numpy()
    st = prepare(case, seed)
    if call == "conv_grad":
        return num(*_exact_conv(P, R, t, st.sig))
    if call in ("energy", "fd"):
        E = float(_exact_ref(P, R, t, st.sig, grad=False)[0])
        return E if call == "energy" else (E, None)   # the differences' step is part of their value
    E, g, dx = _exact_ref(P, R, t, st.sig)
    return num(E, g, dx) if call == "grad_dx" else num(E, g)
