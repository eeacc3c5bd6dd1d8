"""In-place operations that put particles of any order in cell order as a permutation (double ones, and 2D float
ones from 2,049 on): particles outside the grid among them, and the rounding of their node sums."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from gpu_helpers import TOL, close, n, t
from femflow_gb300 import _native as N
from femflow_gb300 import engine as E
from femflow_gb300.solvers.mpm import two_d
from test_gpu_unsorted import DT, G, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,dtype,count", [(3, torch.float64, 4097), (3, torch.float64, 4351), (2, torch.float64, 2049),
                                             (2, torch.float32, 2049), (2, torch.float32, 4096)])
def test_particles_outside_the_grid_are_left_and_reported(dim, dtype, count):
    """Twice over one workspace: the counters come back to zero with particles outside."""
    res, vol, mu, lam = 40, 0.3 ** dim / count, 300.0, 500.0
    x, v, F, C = _scene(dim, count, "random", res)
    out = np.arange(count) % 37 == 5
    dev = [t(a.reshape(count, -1), dtype).contiguous() for a in (x, v, F, C)] + [torch.ones(count, dtype=dtype, device="cuda")]
    dev[0][torch.as_tensor(out, device="cuda")] = 1.5
    p = E.make_params(dim, res, dtype, 1 / res, float(res), DT, G, vol, 1.0, vol, mu, lam)
    ps = E.particles_struct(*dev)
    ws = E.Workspace(p, count, "cuda")
    for _ in range(2):
        N.call("ffmpm_substep", ctypes.byref(p), ctypes.byref(ps), ctypes.c_void_p(ws.ptr), ctypes.c_size_t(ws.bytes),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert ws.status()[0] == N.STATUS_OOB
        ws.clear_status()
    got = [n(a).reshape(s.shape) for a, s in zip(dev, (x, v, F, C))]
    k = ~out
    for a, b in zip(got[1:], (v, F, C)):
        assert np.array_equal(a[out], t(b, dtype).double().cpu().numpy()[out])
    assert np.all(got[0][out] == 1.5)
    s = [np.ascontiguousarray(a[k]) for a in (x, v, F, C)]
    cnt = int(k.sum())
    full, Jp = (lambda a: np.full(cnt, a)), np.ones((cnt, 1))
    for _ in range(2):
        if dim == 3:
            O.substep_3d(res, float(res), 1.0, 1 / res, DT, vol, G, s[0], full(vol), full(mu), full(lam), *s[1:], Jp)
        else:
            O.substep_2d(res, float(res), 1.0, mu, lam, vol, 1 / res, DT, vol, G, *s, Jp)
    tol, vs = TOL[dtype], max(1.0, float(np.abs(s[1]).max()))
    close(got[0][k], s[0], tol["x"], scale=1.0, what="x")
    close(got[1][k], s[1], tol["v"], scale=vs, what="v")
    close(got[3][k], s[3], tol["C"], scale=vs * res, what="C")


@pytest.mark.parametrize("dtype,count,res", [(torch.float64, 60_000, 128), (torch.float32, 4000, 33),
                                             (torch.float32, 60_000, 128)])
def test_rounding_of_node_masses(dtype, count, res):
    """12 particles a cell (2D): rms of the relative error of the nodes' masses.  One rounding of a sum is uniform
    within half an ulp, 0.21 eps rms over the binade; K equal parts added in turn come to 0.21 sqrt(K / 3) eps: 1.25
    eps for the 108 particles of a node in no order, and 0.45 eps for the sums of its 9 cells, the part of a warp's
    32 particles each (13 parts).  Bound: 0.8 eps."""
    edge = np.sqrt(count / 12) / res
    rng = np.random.default_rng(count)
    np_dt = np.float64 if dtype == torch.float64 else np.float32
    x = (0.5 + edge * (rng.uniform(size=(count, 2)) - 0.5)).astype(np_dt)
    m = np_dt(1e-4)
    R = res + 1
    gv = torch.zeros((R, R, 2), dtype=dtype, device="cuda")
    gm = torch.zeros((R, R, 1), dtype=dtype, device="cuda")
    z = lambda *s: torch.zeros(s, dtype=dtype, device="cuda")
    F = torch.eye(2, dtype=dtype, device="cuda").repeat(count, 1, 1).contiguous()
    two_d.p2g(float(res), 1.0, 0.0, 0.0, float(m), 1 / res, DT, 1e-4, gv, gm, t(x, dtype), z(count, 2), F, z(count, 2, 2),
              z(count, 1) + 1)
    L = np.longdouble
    xs = (x * np_dt(res)).astype(np_dt)
    base = np.trunc((xs - np_dt(0.5)).astype(np_dt)).astype(np.int64)
    fx = (xs - base.astype(np_dt)).astype(np_dt).astype(L)
    w = [L(0.5) * (L(1.5) - fx) ** 2, L(0.75) - (fx - L(1)) ** 2, L(0.5) * (fx - L(0.5)) ** 2]
    want = np.zeros((R, R), dtype=L)
    for i in range(3):
        for j in range(3):
            np.add.at(want, (base[:, 0] + i, base[:, 1] + j), w[i][:, 0] * w[j][:, 1] * L(m))
    got = gm[..., 0].cpu().numpy().astype(L)
    inner = want > L(0.9) * want.max() * L(0.5)
    rel = ((got - want)[inner] / want[inner]).astype(np.float64)
    rms = float(np.sqrt((rel ** 2).mean())) / float(np.finfo(np_dt).eps)
    assert rms <= 0.8, rms
