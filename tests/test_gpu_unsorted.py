"""In-place substeps without a block sort, at the sizes where their warps, stretches and counting sort
have edges, against the float64 oracle: particles in no order, all in one cell (long runs), and in cell
order with the caller's hint; row-major and component-major arrays."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from gpu_helpers import TOL, close, n, t
from femflow_gb300 import _native as N
from femflow_gb300 import engine as E

pytestmark = pytest.mark.gpu
DT, G = 1e-4, -9.8


def _scene(dim, count, layout, res):
    rng = np.random.default_rng(count + dim)
    if layout == "one_cell":
        x = (np.array([res // 2] * dim) + 1.0 + rng.uniform(-0.45, 0.45, (count, dim))) / res
    else:
        x = rng.uniform(0.3, 0.6, (count, dim))
    x = x.astype(np.float32).astype(np.float64)
    if layout == "ordered":
        b = np.floor(x * res - 0.5).astype(np.int64)
        key = b[:, 0]
        for a in range(1, dim):
            key = key * (res + 1) + b[:, a]
        x = np.ascontiguousarray(x[np.argsort(key, kind="stable")])
    r32 = lambda a: a.astype(np.float32).astype(np.float64)
    v = r32(1.0 + 0.1 * rng.standard_normal((count, dim)))
    F = r32(np.eye(dim) + 0.01 * rng.standard_normal((count, dim, dim)))
    C = r32(rng.standard_normal((count, dim, dim)))
    return x, v, F, C


def _substep(dim, dtype, res, x, v, F, C, vol, mu, lam, variant, soa):
    cnt = x.shape[0]
    lay = lambda a: t(a.reshape(cnt, -1).T if soa else a, dtype).contiguous()
    dev = [lay(a) for a in (x, v, F, C)] + [torch.ones(cnt, dtype=dtype, device="cuda")]
    p = E.make_params(dim, res, dtype, 1 / res, float(res), DT, G, vol, 1.0, vol, mu, lam, variant=variant)
    ps = E.particles_struct(*dev, stride=cnt if soa else 0, n=cnt)
    ws = E.Workspace(p, cnt, "cuda")
    for _ in range(2):  # the second call finds the counters and the grid as the first left them
        N.call("ffmpm_substep", ctypes.byref(p), ctypes.byref(ps), ctypes.c_void_p(ws.ptr), ctypes.c_size_t(ws.bytes),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    ws.raise_on_status()
    back = lambda a, s: n(a.T if soa else a).reshape(s.shape)
    return [back(a, s) for a, s in zip(dev, (x, v, F, C))]


# 31..33: a warp; 95..97, 193: the stretches of a warp and a CTA; 4096 / 4097: scattered as they come /
# by counting sort; 20011: many stretches, and in one cell the longest ones
@pytest.mark.parametrize("layout", ["random", "one_cell", "ordered"])
@pytest.mark.parametrize("count", [1, 31, 33, 97, 4096, 4097, 4193, 20011])
@pytest.mark.parametrize("dim,dtype", [(3, torch.float32), (2, torch.float32), (3, torch.float64), (2, torch.float64)])
def test_in_place_substeps_against_the_oracle(dim, dtype, count, layout):
    res = 40
    x, v, F, C = _scene(dim, count, layout, res)
    vol, mu, lam = 0.3 ** dim / count, 300.0, 500.0
    variant = N.VARIANT_CELL_ORDER if layout == "ordered" else 0
    got = _substep(dim, dtype, res, x, v, F, C, vol, mu, lam, variant, soa=count % 2 == 1)
    Jp = np.ones((count, 1))
    for _ in range(2):
        if dim == 3:
            full = lambda a: np.full(count, a)
            O.substep_3d(res, float(res), 1.0, 1 / res, DT, vol, G, x, full(vol), full(mu), full(lam), v, F, C, Jp)
        else:
            O.substep_2d(res, float(res), 1.0, mu, lam, vol, 1 / res, DT, vol, G, x, v, F, C, Jp)
    tol = TOL[dtype]
    vs = max(1.0, float(np.abs(v).max()))
    close(got[0], x, tol["x"], scale=1.0, what="x")
    close(got[1], v, tol["v"], scale=vs, what="v")
    s = np.sign(np.einsum("nij,nij->n", got[2], F))[:, None, None] if dim == 2 else 1.0
    close(got[2] * s, F, tol["F"], scale=1.0, what="F")
    close(got[3], C, tol["C"], scale=vs * res, what="C")


def test_a_grid_large_against_the_particles_keeps_the_sorted_form():
    """res 256 (17M nodes) with few particles: the same substep through the block sort."""
    res = 256
    x, v, F, C = _scene(3, 5000, "random", res)
    vol, mu, lam = 1e-6, 300.0, 500.0
    got = _substep(3, torch.float32, res, x, v, F, C, vol, mu, lam, 0, soa=False)
    full = lambda a: np.full(5000, a)
    Jp = np.ones((5000, 1))
    for _ in range(2):
        O.substep_3d(res, float(res), 1.0, 1 / res, DT, vol, G, x, full(vol), full(mu), full(lam), v, F, C, Jp)
    close(got[0], x, TOL[torch.float32]["x"], scale=1.0, what="x")
    close(got[1], v, TOL[torch.float32]["v"], scale=float(np.abs(v).max()), what="v")
