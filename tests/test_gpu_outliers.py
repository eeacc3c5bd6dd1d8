"""Particles far faster or far lighter than the rest, one at the head of every warp (of the caller's, the
sorted and the batch's order), cost the others no digits: the others, which share no node with them, against the
float64 oracle at the bounds of an ordinary scene."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from gpu_helpers import TOL, close, n, t
from femflow_gb300 import _native as N
from femflow_gb300 import engine as E
from femflow_gb300.batched import Batch2D
from femflow_gb300.solver import MPMSolver
from femflow_gb300.solvers.mpm import mls_mpm
from femflow_gb300.solvers.mpm.particle import ParticleSet

pytestmark = pytest.mark.gpu
RES, DT, G = 32, 1e-4, -9.8
VOL, MU, LAM = 1e-5, 300.0, 500.0
r32 = lambda a: np.asarray(a).astype(np.float32).astype(np.float64)


def _scene(dim, count, kind):
    """Every 32nd particle is an outlier on the grid rows of the body, well before it along the last axis (so in
    cell order too the body's particles follow one)."""
    rng = np.random.default_rng(count + dim)
    x = rng.uniform(0.3, 0.6, (count, dim))
    out = np.arange(count) % 32 == 0
    x[out, -1] = 0.1
    v = 1.0 + 0.1 * rng.standard_normal((count, dim))
    F = np.eye(dim) + 0.01 * rng.standard_normal((count, dim, dim))
    mass = np.full(count, VOL)
    if kind == "fast":
        v[out] = 1e5
    else:  # their stress over their mass is a velocity of about 1e5
        mass[out] *= 1e-6
    return dict(x=r32(x), v=r32(v), F=r32(F), C=np.zeros((count, dim, dim)), mass=r32(mass), out=out)


def _oracle(dim, s, steps):
    x, v, F, C = (s[k].copy() for k in "xvFC")
    count = len(x)
    Jp = np.ones((count, 1))
    for _ in range(steps):
        if dim == 3:
            O.substep_3d(RES, float(RES), 1.0, 1 / RES, DT, VOL, G, x, s["mass"], np.full(count, MU),
                         np.full(count, LAM), v, F, C, Jp)
        else:
            O.substep_2d(RES, float(RES), 1.0, MU, LAM, VOL, 1 / RES, DT, VOL, G, x, v, F, C, Jp)
    return x, v, F, C


def _check(got, want, s, dtype):
    k = ~s["out"]
    tol, vs = TOL[dtype], float(np.abs(want[1][k]).max())
    assert vs < 5.0  # the outliers move none of the others
    close(got[0][k], want[0][k], tol["x"], scale=1.0, what="x")
    close(got[1][k], want[1][k], tol["v"], scale=vs, what="v")
    close(got[2][k], want[2][k], tol["F"], scale=1.0, what="F")
    close(got[3][k], want[3][k], tol["C"], scale=vs * RES, what="C")


# 2048: float32 particles scattered as they come; 6016: by the counting sort
@pytest.mark.parametrize("count", [2048, 6016])
@pytest.mark.parametrize("dim,dtype,kind", [(3, torch.float32, "fast"), (3, torch.float32, "light"),
                                            (2, torch.float32, "fast"), (3, torch.float64, "light")])
def test_in_place_substep(dim, dtype, kind, count):
    s = _scene(dim, count, kind)
    dev = [t(s[k].reshape(count, -1), dtype).contiguous() for k in "xvFC"] + [torch.ones(count, dtype=dtype, device="cuda")]
    mat = [t(a, dtype) for a in (s["mass"], np.full(count, MU), np.full(count, LAM))] if dim == 3 else []
    p = E.make_params(dim, RES, dtype, 1 / RES, float(RES), DT, G, VOL, 1.0, VOL, MU, LAM)
    ps = E.particles_struct(*dev, *mat)
    ws = E.Workspace(p, count, "cuda")
    N.call("ffmpm_substep", ctypes.byref(p), ctypes.byref(ps), ctypes.c_void_p(ws.ptr), ctypes.c_size_t(ws.bytes),
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    ws.raise_on_status()
    _check([n(a).reshape(s[k].shape) for a, k in zip(dev, "xvFC")], _oracle(dim, s, 1), s, dtype)


@pytest.mark.parametrize("kind", ["fast", "light"])
def test_host_arrays(kind):
    s = _scene(3, 6016, kind)
    pin = lambda a: torch.tensor(a, dtype=torch.float32).pin_memory()
    x, v, F, C = (pin(s[k]) for k in "xvFC")
    one = np.ones(6016)
    mls_mpm.solve_mls_mpm_3d(RES, float(RES), 1.0, 1 / RES, DT, VOL, G,
                             ParticleSet(x, pin(s["mass"]), pin(MU * one), pin(LAM * one)), v, F, C, pin(one[:, None]))
    _check([a.double().numpy() for a in (x, v, F, C)], _oracle(3, s, 1), s, torch.float32)


@pytest.mark.parametrize("kind", ["fast", "light"])
def test_resident_solver(kind):
    """Two substeps: the first scatter, then the fused gather and scatter (the grid clamps the outliers' velocities)."""
    s = _scene(3, 6016, kind)
    one = torch.ones(6016)
    sol = MPMSolver(torch.tensor(s["x"]), res=RES, dt=DT, gravity=G, volume=VOL, mass=torch.tensor(s["mass"]), mu_0=MU * one,
                    lambda_0=LAM * one, v=torch.tensor(s["v"]), F=torch.tensor(s["F"]))
    sol.step(2, check=True)
    st = sol.state()
    _check([n(st[k]).reshape(s[k].shape) for k in "xvFC"], _oracle(3, s, 2), s, torch.float32)


def test_batched_scenes():
    s = _scene(2, 6016, "fast")
    b = Batch2D([dict(x=s["x"], v=s["v"], F=s["F"], res=RES, dt=DT, mass=VOL, volume=VOL, mu_0=MU, lambda_0=LAM)])
    b.step(1)
    assert b.status() == 0
    st = b.scene_state(0)
    _check([n(st[k]).reshape(s[k].shape) for k in "xvFC"], _oracle(2, s, 1), s, torch.float32)
