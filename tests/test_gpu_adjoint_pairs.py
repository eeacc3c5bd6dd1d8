"""Adjoint of float states (node sums in float pairs within a warp's runs) against the float64 adjoint of
the same inputs, which sums every contribution in float64: one particle, the edges of a warp and a CTA, all
particles in one cell, in cell order and in no order."""
import ctypes

import numpy as np
import pytest
import torch

from gpu_helpers import n, t
from femflow_gb300 import _native as N
from femflow_gb300 import engine as E

pytestmark = pytest.mark.gpu


def _adjoint(dtype, res, state, adj, vol, mu, lam, dt):
    cnt = state[0].shape[0]
    col = lambda a: t(a.reshape(cnt, -1).T, dtype).contiguous()
    dev, ad = [col(a) for a in state], [col(a) for a in adj]
    Jp = torch.ones(cnt, dtype=dtype, device="cuda")
    p = E.make_params(3, res, dtype, 1 / res, float(res), dt, -9.8, vol, 1.0, vol, mu, lam, model="fixed_corotated")
    P = E.particles_struct(*dev, Jp, stride=cnt, n=cnt)
    A = N.Adjoint()
    A.x, A.v, A.F, A.C = (a.data_ptr() for a in ad)
    mb, lb = torch.zeros(cnt, dtype=torch.float64, device="cuda"), torch.zeros(cnt, dtype=torch.float64, device="cuda")
    A.mu_0, A.lambda_0 = mb.data_ptr(), lb.data_ptr()
    size = ctypes.c_size_t(0)
    N.call("ffmpm_adjoint_workspace_size", ctypes.byref(p), cnt, ctypes.byref(size))
    ws = torch.zeros(size.value + 256, dtype=torch.uint8, device="cuda")
    at = (ws.data_ptr() + 255) // 256 * 256
    N.call("ffmpm_substep_adjoint", ctypes.byref(p), ctypes.byref(P), ctypes.byref(A), ctypes.c_void_p(at),
           ctypes.c_size_t(size.value), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return [n(a.T) for a in ad] + [n(mb), n(lb)]


@pytest.mark.parametrize("layout", ["random", "one_cell", "ordered"])
@pytest.mark.parametrize("count", [1, 31, 33, 127, 129, 3001])
def test_float_adjoint_against_the_float64_one(count, layout):
    res, dt = 32, 1e-4
    rng = np.random.default_rng(count)
    r32 = lambda a: np.asarray(a).astype(np.float32).astype(np.float64)
    x = (rng.uniform(15.6, 16.4, (count, 3)) + 0.5) / res if layout == "one_cell" else rng.uniform(0.3, 0.6, (count, 3))
    x = r32(x)
    if layout == "ordered":
        b = np.floor(x * res - 0.5).astype(np.int64)
        x = x[np.argsort((b[:, 0] * 64 + b[:, 1]) * 64 + b[:, 2], kind="stable")]
    state = [x, r32(rng.normal(0, 0.3, (count, 3))), r32(np.eye(3) + rng.normal(0, 0.01, (count, 3, 3))),
             r32(rng.normal(0, 1, (count, 3, 3)))]
    adj = [r32(rng.normal(0, 1, s.shape)) for s in state]
    vol, mu, lam = 0.3 ** 3 / count, 1500.0, 2300.0
    got = _adjoint(torch.float32, res, state, adj, vol, mu, lam, dt)
    want = _adjoint(torch.float64, res, state, adj, vol, mu, lam, dt)
    for k, (a, b) in enumerate(zip(got, want)):
        # the bound the float adjoint has against the float64 oracle
        assert np.abs(a - b).max() <= 2e-3 * max(np.abs(b).max(), 1e-30), (k, np.abs(a - b).max(), np.abs(b).max())
