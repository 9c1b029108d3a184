"""Batches beside one another and problems of very different sizes in one batch: every batch that can be
evaluated alone can be evaluated while others are, and beside a problem of any other size."""
import threading

import numpy as np
import pytest

from dugma_b200 import _lib, api
from tests.test_sparse_pairs import _problem

pytestmark = pytest.mark.gpu


def _poses(probs, Q, sig):
    R = np.array([[p[4]] * Q for p in probs])
    t = np.array([[p[5] + 0.001 * q for q in range(Q)] for p in probs])
    return R, t, np.full((len(probs), Q), sig)


def test_batches_in_threads():
    """Sparse batches whose largest problems differ, from a thread each: their launches need different
    amounts of shared memory, and none takes another's."""
    L = _lib.load()
    work = []
    for s, (n, m) in enumerate([(1001, 900), (5001, 60000)] * 3):
        probs = [_problem("sphere", n, m, s)]
        b = api.Batch([p[:4] for p in probs])
        pose = _poses(probs, 1, 1e-4)
        E, g = b.energy_grad(*pose)
        assert b.last_pass() == (1, 1, 8)
        work.append((b, b._poses(*pose)[0], np.concatenate([E.ravel(), g.ravel()]), np.zeros(7)))
    failed, start = [], threading.Barrier(len(work))

    def run(b, rec, want, out):
        start.wait(60)
        for _ in range(4000):
            if L.dugma_batch_energy_grad(b.b, 1, api._ptr(rec), 0, api._ptr(out)):
                failed.append(L.dugma_last_error().decode())
            elif not np.array_equal(out, want):
                failed.append("another result")

    threads = [threading.Thread(target=run, args=w) for w in work]
    for th in threads:
        th.start()
    for th in threads:
        th.join(600)
    for w in work:
        w[0].close()
    assert not failed, (len(failed), failed[0])


def test_sparse_problem_beside_a_huge_one():
    """A problem of more targets than the sparse pass takes: it is evaluated over all pairs, and the
    launch of the sparse one beside it does not grow with it."""
    n, m = 16, 3700000
    rng = np.random.default_rng(8)
    small = _problem("sphere", 3001, 3000, 2)
    eye = lambda k: np.broadcast_to(1e-3 * np.eye(3), (k, 3, 3))  # noqa: E731
    big = (rng.uniform(-1, 1, (n, 3)), eye(n), rng.uniform(-1, 1, (m, 3)), eye(m), np.eye(3), np.zeros(3))
    out = []
    for k, probs in enumerate(([small], [small, big], [big])):
        b = api.Batch([p[:4] for p in probs])
        out.append(b.energy_grad(*_poses(probs, 2, 1e-4)))
        assert b.last_pass()[0] == (0 if k == 2 else 2), b.last_pass()
        b.close()
    for k in range(2):
        assert np.allclose(out[1][k][0], out[0][k][0], rtol=1e-12, atol=0)
        assert np.allclose(out[1][k][1], out[2][k][0], rtol=1e-12, atol=0)


def test_rows_only_where_something_is_sparse():
    """The sparse pass's rows (64 bytes a source and pose) are allocated by the first evaluation that has a
    sparse pose, whatever came before it."""
    import torch
    probs = [_problem("sphere", 20001, 1301, s) for s in range(4)]
    rows = 4 * 24 * 20001 * 64
    out, used = [], []
    for sigs in ((30.0, 1e-4), (1e-4, 30.0)):
        b = api.Batch([p[:4] for p in probs])
        got = []
        for sig in sigs + sigs:
            free = torch.cuda.mem_get_info()[0]
            got.append(b.energy_grad(*_poses(probs, 24, sig)))
            assert b.last_pass()[0] == (0 if sig > 1 else 96)
            used.append(free - torch.cuda.mem_get_info()[0])
        b.close()
        assert all(np.array_equal(u, v) for k in range(2) for u, v in zip(got[k], got[k + 2]))
        out.append(got)
    assert all(np.array_equal(u, v) for k in range(2) for u, v in zip(out[0][k], out[1][1 - k]))
    assert 0.9 * rows <= used[1] <= rows + (8 << 20) and used[4] >= used[0] + 0.9 * rows, (rows, used)
    assert max(used[2:4] + used[5:]) <= 8 << 20, used
