"""In-place substeps over one workspace read no velocity of an earlier call: particles without mass and
stress in a region that a moving body left, and particles at exactly half a cell (stencil weight zero) after a
run on the same workspace has diverged; against the float64 oracle."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from gpu_helpers import TOL, close, n, t
from femflow_gb300 import _native as N
from femflow_gb300 import engine as E

pytestmark = pytest.mark.gpu
RES, DT, G = 32, 1e-4, -9.8
VOL, MU, LAM = 1e-5, 300.0, 500.0


def _params(dim, dtype, mass, mu=MU, lam=LAM):
    return E.make_params(dim, RES, dtype, 1 / RES, float(RES), DT, G, VOL, 1.0, mass, mu, lam)


def _workspace(dim, dtype, cnt):
    return E.Workspace(_params(dim, dtype, VOL), cnt, "cuda")


def _substep(prm, dtype, ws, state, material=None):
    cnt = state[0].shape[0]
    dev = [t(a.reshape(cnt, -1), dtype).contiguous() for a in state] + [torch.ones(cnt, dtype=dtype, device="cuda")]
    mat = [t(a, dtype) for a in material] if material else []
    ps = E.particles_struct(*dev, *mat)
    N.call("ffmpm_substep", ctypes.byref(prm), ctypes.byref(ps), ctypes.c_void_p(ws.ptr), ctypes.c_size_t(ws.bytes),
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    ws.raise_on_status()
    return [n(a).reshape(s.shape) for a, s in zip(dev, state)]


def _oracle(dim, state, mass, mu, lam):
    x, v, F, C = (a.copy() for a in state)
    cnt = len(x)
    Jp = np.ones((cnt, 1))
    if dim == 3:
        O.substep_3d(RES, float(RES), 1.0, 1 / RES, DT, VOL, G, x, mass, mu, lam, v, F, C, Jp)
    else:
        O.substep_2d(RES, float(RES), 1.0, mu, lam, mass, 1 / RES, DT, VOL, G, x, v, F, C, Jp)
    return x, v, F, C


def _check(got, want, dtype):
    tol, vs = TOL[dtype], max(1.0, float(np.abs(want[1]).max()))
    close(got[0], want[0], tol["x"], scale=1.0, what="x")
    close(got[1], want[1], tol["v"], scale=vs, what="v")
    close(got[2], want[2], tol["F"], scale=1.0, what="F")
    close(got[3], want[3], tol["C"], scale=vs * RES, what="C")


def _body(dim, count, lo, speed, seed):
    rng = np.random.default_rng(seed)
    r32 = lambda a: a.astype(np.float32).astype(np.float64)
    return (r32(rng.uniform(lo, lo + 0.2, (count, dim))), r32(speed + 0.1 * rng.standard_normal((count, dim))),
            np.tile(np.eye(dim), (count, 1, 1)), np.zeros((count, dim, dim)))


# 3000: float32 particles scattered as they come; 6000: by the counting sort
@pytest.mark.parametrize("count", [3000, 6000])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dim", [2, 3])
def test_massless_particles_where_a_body_was(dim, dtype, count):
    ws = _workspace(dim, dtype, count)
    _substep(_params(dim, dtype, VOL), dtype, ws, _body(dim, count, 0.3, 5.0, 1))
    if dim == 3:  # half the particles a body elsewhere, half without mass and stress where the first body was
        a, b = _body(dim, count // 2, 0.6, 1.0, 2), _body(dim, count // 2, 0.3, 3.0, 3)
        state = [np.concatenate(p) for p in zip(a, b)]
        has = np.concatenate([np.ones(count // 2), np.zeros(count // 2)])
        mat = [VOL * has, MU * has, LAM * has]
        got = _substep(_params(dim, dtype, 0.0, 0.0, 0.0), dtype, ws, state, mat)
        want = _oracle(dim, state, *mat)
        assert not want[1][count // 2:].any()  # a node without mass has velocity zero
    else:  # one mass for all particles: none
        state = _body(dim, count, 0.3, 3.0, 3)
        got = _substep(_params(dim, dtype, 0.0, 0.0, 0.0), dtype, ws, state)
        want = _oracle(dim, state, 0.0, 0.0, 0.0)
        assert not want[1].any()
    _check(got, want, dtype)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dim", [2, 3])
def test_half_cell_particles_after_a_diverged_run(dim, dtype, variant):
    count = 4000
    ws = _workspace(dim, dtype, count)
    # one block-sorted substep of a body whose velocities are not numbers (its end state is not used)
    x, v, F, C = _body(dim, count, 0.3, 5.0, 1)
    v[:] = np.nan
    prm = _params(dim, dtype, VOL)
    prm.variant = variant
    bufs = []
    for _ in range(2):
        bufs.append([t(a.reshape(count, -1), dtype).contiguous() for a in (x, v, F, C)] +
                    [torch.ones(count, dtype=dtype, device="cuda")])
    a, b = (E.particles_struct(*q) for q in bufs)
    N.call("ffmpm_substeps_sorted", ctypes.byref(prm), ctypes.byref(a), ctypes.byref(b), None, None, 1,
           ctypes.c_void_p(ws.ptr), ctypes.c_size_t(ws.bytes), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert ws.status()[0] & N.STATUS_NONFINITE
    ws.clear_status()
    # a sheet of particles at exactly half a cell along the first axis in that region: node base + 2 has weight zero
    x = _body(dim, count, 0.3, 1.0, 7)[0]
    x[:, 0] = 12.5 / RES
    state = (x, *_body(dim, count, 0.3, 1.0, 5)[1:])
    got = _substep(_params(dim, dtype, VOL), dtype, ws, state)
    _check(got, _oracle(dim, state, *((np.full(count, VOL), np.full(count, MU), np.full(count, LAM)) if dim == 3
                                      else (VOL, MU, LAM))), dtype)
