"""A call that failed leaves no error behind for the next one."""
import ctypes

import numpy as np
import pytest

from dugma_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu


def test_call_after_a_failed_one():
    """Timing events recorded into a captured graph cannot be waited for: that query fails, on the host, and
    the evaluation after it does not."""
    import torch
    P = synth.workload0(trial=1, n=500)
    _, h = api.init(P.X, P.X_C, P.Y, P.Y_C)
    want = api.energy_grad(h, P.R_G, P.t_G, 0.05)[:2]
    pose = torch.zeros(16, dtype=torch.float64, device="cuda")
    pose[:9] = torch.tensor(np.asarray(P.R_G).T.reshape(-1))
    pose[9:12] = torch.tensor(P.t_G)
    pose[12] = 0.05
    out = torch.zeros(8, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    L = _lib.load()
    assert L.dugma_timing(h.arr, 1, None, None) == 0
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        assert L.dugma_energy_grad_async(h.arr, pose.data_ptr(), 0, out.data_ptr(), None, s.cuda_stream) == 0
    assert L.dugma_timing(h.arr, 0, None, None) == 0
    assert L.dugma_timing(h.arr, 2, ctypes.byref(ctypes.c_double()), ctypes.byref(ctypes.c_int())) == _lib.ERR_CUDA
    got = api.energy_grad(h, P.R_G, P.t_G, 0.05)[:2]
    assert got[0] == want[0] and np.array_equal(got[1], want[1])
    g.replay()
    torch.cuda.synchronize()
    assert out.cpu().numpy()[0] == want[0]
    del g
    api.fr_m(h)
