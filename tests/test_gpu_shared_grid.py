"""Two streams, each with its own workspace and particles, add into one caller's grid at the same time: nothing
is lost (the phase adds to the grid; both bodies lie over the same nodes)."""
import ctypes

import pytest
import torch

from femflow_gb300 import _native as N
from femflow_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dim", [2, 3])
def test_two_streams_add_into_one_grid(dim, dtype):
    n, res, m = 20_000, (96 if dim == 3 else 700), 1e-5
    R = res + 1
    g = torch.Generator(device="cuda").manual_seed(dim)
    prm = E.make_params(dim, res, dtype, 1 / res, float(res), 1e-4, 0.0, 1e-6, 1.0, m, 0.0, 0.0)
    parts, keep = [], []
    for _ in range(2):
        x = 0.1 + 0.8 * torch.rand((n, dim), generator=g, device="cuda", dtype=torch.float64).to(dtype)
        v = torch.ones((n, dim), dtype=dtype, device="cuda")
        F = torch.eye(dim, dtype=dtype, device="cuda").repeat(n, 1, 1).contiguous()
        C, J = torch.zeros_like(F), torch.ones(n, dtype=dtype, device="cuda")
        keep.append((x, v, F, C, J))
        parts.append((E.particles_struct(x, v, F, C, J), E.Workspace(prm, n, "cuda"), torch.cuda.Stream()))
    gv, gm = torch.zeros((R ** dim, dim), dtype=dtype, device="cuda"), torch.zeros(R ** dim, dtype=dtype, device="cuda")
    G = E.grid_struct(gv, gm)
    torch.cuda.synchronize()
    rounds = 50
    for _ in range(rounds):
        for P, ws, s in parts:
            N.call("ffmpm_p2g", ctypes.byref(prm), ctypes.byref(P), ctypes.byref(G), ctypes.c_void_p(ws.ptr),
                   ctypes.c_size_t(ws.bytes), ctypes.c_void_p(s.cuda_stream))
    torch.cuda.synchronize()
    total = 2 * n * m * rounds
    # every particle's weights sum to one: only rounding is missing (a node takes 100 adds and the sums under them)
    tol = 1e-5 if dtype == torch.float32 else 1e-12
    assert abs(float(gm.double().sum()) - total) <= tol * total
    assert float((gv.double().sum(0) - total).abs().max()) <= tol * total
