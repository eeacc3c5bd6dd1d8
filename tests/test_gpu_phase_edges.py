"""The phases on the caller's grid at the edges of their kernels' tiles, with a mass and a material of each particle
and a grid that holds values already, against the float64 oracle; and in-place substeps replayed from a captured
graph."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from gpu_helpers import TOL, close, n, t
from femflow_gb300 import _native as N
from femflow_gb300 import engine as E
from femflow_gb300.solvers.mpm import three_d, two_d
from femflow_gb300.solvers.mpm.particle import ParticleSet
from test_gpu_unsorted import DT, G, _scene, _substep

pytestmark = pytest.mark.gpu


# 31..33, 97: warps and their thirds; 2049, 4097: the forms of the scatter; 4193: its stretches
@pytest.mark.parametrize("count", [1, 31, 33, 97, 2049, 4097, 4193])
@pytest.mark.parametrize("dim,dtype", [(3, torch.float32), (2, torch.float32), (3, torch.float64), (2, torch.float64)])
def test_p2g_and_g2p_against_the_oracle(dim, dtype, count):
    res = 37  # (res + 1)^dim is no multiple of a CTA
    dx = 1 / res
    rng = np.random.default_rng(count)
    r32 = lambda a: a.astype(np.float32).astype(np.float64)
    x, v, F, C = _scene(dim, count, "random", res)
    vol = 0.3 ** dim / count
    Jp = np.ones((count, 1))
    gv, gm = (r32(0.01 * vol * rng.standard_normal(((res + 1,) * dim) + (k,))) for k in (dim, 1))
    tgv, tgm, tx, tv, tF, tC, tJ = (t(a, dtype).contiguous() for a in (gv, gm, x, v, F, C, Jp))
    mass, mu, lam = (r32(s * rng.uniform(0.5, 2.0, count)) for s in (vol, 300.0, 500.0))
    if dim == 3:
        parts = ParticleSet(tx, *(t(a, dtype) for a in (mass, mu, lam)))
        three_d.p2g(float(res), 1.0, dx, DT, vol, tgv, tgm, parts, tv, tF, tC, tJ)
        O.p2g_3d(float(res), 1.0, dx, DT, vol, gv, gm, x, mass, mu, lam, v, F, C, Jp)
    else:
        two_d.p2g(float(res), 1.0, 300.0, 500.0, vol, dx, DT, vol, tgv, tgm, tx, tv, tF, tC, tJ)
        O.p2g_2d(float(res), 1.0, 300.0, 500.0, vol, dx, DT, vol, gv, gm, x, v, F, C, Jp)
    close(n(tgv), gv, TOL[dtype]["grid"], what="momentum")
    close(n(tgm), gm, TOL[dtype]["grid"], what="mass")
    vel = r32(rng.standard_normal(gv.shape))
    tvel = t(vel, dtype).contiguous()
    if dim == 3:
        three_d.g2p(float(res), DT, tvel, parts, tv, tF, tC, tJ)
        O.g2p_3d(float(res), DT, vel, x, v, F, C, Jp)
    else:
        two_d.g2p(float(res), DT, tvel, tx, tv, tF, tC, tJ)
        O.g2p_2d(float(res), DT, vel, x, v, F, C, Jp)
    tol, vs = TOL[dtype], 3.0
    close(n(parts.pos if dim == 3 else tx), x, tol["x"], scale=1.0, what="x")
    close(n(tv), v, tol["v"], scale=vs, what="v")
    s = np.sign(np.einsum("nij,nij->n", n(tF), F))[:, None, None] if dim == 2 else 1.0
    close(n(tF) * s, F, tol["F"], scale=1.0, what="F")
    close(n(tC), C, tol["C"], scale=vs * res, what="C")


# as they come, as a permutation, as records
@pytest.mark.parametrize("dim,dtype,count", [(3, torch.float32, 1000), (2, torch.float32, 3000), (3, torch.float64, 6000),
                                             (3, torch.float32, 20011)])
def test_in_place_substeps_replayed_from_a_graph(dim, dtype, count):
    res, vol, mu, lam = 40, 0.3 ** dim / count, 300.0, 500.0
    x, v, F, C = _scene(dim, count, "random", res)
    want = _substep(dim, dtype, res, x, v, F, C, vol, mu, lam, 0, soa=False)  # two substeps
    dev = [t(a.reshape(count, -1), dtype).contiguous() for a in (x, v, F, C)] + [torch.ones(count, dtype=dtype, device="cuda")]
    keep = [a.clone() for a in dev]
    p = E.make_params(dim, res, dtype, 1 / res, float(res), DT, G, vol, 1.0, vol, mu, lam)
    ps = E.particles_struct(*dev)
    ws = E.Workspace(p, count, "cuda")

    def step():
        N.call("ffmpm_substep", ctypes.byref(p), ctypes.byref(ps), ctypes.c_void_p(ws.ptr), ctypes.c_size_t(ws.bytes),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))

    step()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        step()
    for a, b in zip(dev, keep):
        a.copy_(b)
    g.replay()
    g.replay()
    ws.raise_on_status()
    tol, vs = TOL[dtype], max(1.0, float(np.abs(want[1]).max()))
    for a, b, k, s in zip(dev, want, ("x", "v", "F", "C"), (1.0, vs, 1.0, vs * res)):
        close(n(a).reshape(b.shape), b, tol[k], scale=s, what=k)
