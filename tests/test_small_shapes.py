"""The REF kernels of small problems (fewer sources per thread) against the FP64 oracle at the edges of
their blocks of 64 sources and tiles of 128 targets and on both sides of the pair counts where the
shapes change, in the Cholesky and the Horner form, and against the default shape's sums: a row
range of all but one row of a problem on the other side of the line adds up with that row's."""
import numpy as np
import pytest

from dugma_b200 import api, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _clouds(n, m, D, indefinite):
    P = synth.workload5(trial=2, n=max(n, m)) if D == 2 else synth.workload0(trial=2, n=max(n, m))
    X, XC, Y, YC = P.X[:n], P.X_C[:n].copy(), P.Y[:m], P.Y_C[:m].copy()
    if indefinite:   # a source with det > 0 but no Cholesky factor, and small exponents
        XC[0] = np.diag([-100.0, -100.0] if D == 2 else [-100.0, -100.0, 0.01])
    return X, XC, Y, YC, P.R_G, P.t_G


@pytest.mark.parametrize("indefinite", [False, True])
@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("n,m", [(1, 1), (63, 127), (64, 128), (65, 129), (1, 300), (1581, 1580), (1583, 1582),
                                 (3400, 3200), (3300, 3400)])
def test_against_oracle(n, m, D, indefinite):
    X, XC, Y, YC, R, t = _clouds(n, m, D, indefinite)
    sig = 0.05 if D == 3 else 1.0
    _, h = api.init(X, XC, Y, YC)
    st = orc.State(X, XC, Y, YC)
    try:
        E, g, dx = api.energy_grad(h, R, t, sig, with_dx=True)
        Eo, go, dxo = st.energy(R, t, sig, with_dx=True)
        assert abs(E - Eo) <= 1e-6 * abs(Eo)
        assert np.linalg.norm(g - go) <= 1e-5 * np.linalg.norm(go)
        assert np.linalg.norm(dx - dxo) <= 1e-5 * np.linalg.norm(dxo)
        assert abs(api.energy(h, R, t, sig) - Eo) <= 1e-6 * abs(Eo)
    finally:
        api.fr_m(h)


def test_same_sums_across_the_line():
    n, m = 9100, 9050   # all rows: past the line; the range without the last rows: before it
    X, XC, Y, YC, R, t = _clouds(n, m, 3, False)
    _, h = api.init(X, 1e4 * XC, Y, 1e4 * YC)   # (wide covariances: all pairs on both sides)
    E, g, _ = api.energy_grad(h, R, t, 0.05)
    parts = [api.energy_grad_range(h, R, t, 0.05, a, b) for a, b in ((0, 9000), (9000, n))]
    assert abs(E - sum(p[0] for p in parts)) <= 1e-6 * E
    assert np.linalg.norm(g - sum(p[1] for p in parts)) <= 1e-5 * np.linalg.norm(g)
    api.fr_m(h)
