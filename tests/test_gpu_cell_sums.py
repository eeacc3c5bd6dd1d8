"""Sums over cells of in-place substeps where cells are full, so that the lanes of a warp share each run: runs
that cross stages and stretches, and long runs beside single particles, against the float64 oracle; and the
rounding of a dense body's sums beside that of the block-sorted form."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from gpu_helpers import TOL, close
from femflow_gb300 import _native as N
from femflow_gb300 import engine as E
from test_gpu_unsorted import DT, G, _substep

pytestmark = pytest.mark.gpu


def _scene(dim, count, layout, res):
    rng = np.random.default_rng(count + dim)
    if layout == "lumps":  # nine tenths in three neighbouring cells of a row, the rest over the body
        x = rng.uniform(0.3, 0.6, (count, dim))
        k = count * 9 // 10
        x[:k] = (rng.uniform(-0.45, 0.45, (k, dim)) + 17.0) / res
        x[:k, -1] += rng.integers(0, 3, k) / res
    else:  # a body of about 20 (3D) or 30 (2D) particles a cell
        x = rng.uniform(0.3, 0.45 if dim == 3 else 0.6, (count, dim))
    r32 = lambda a: a.astype(np.float32).astype(np.float64)
    x = x[rng.permutation(count)]
    return (r32(x), r32(1.0 + 0.1 * rng.standard_normal((count, dim))),
            r32(np.eye(dim) + 0.01 * rng.standard_normal((count, dim, dim))), r32(rng.standard_normal((count, dim, dim))))


@pytest.mark.parametrize("layout", ["dense", "lumps"])
@pytest.mark.parametrize("count", [4097, 4193, 8160, 20011])
@pytest.mark.parametrize("dim", [3, 2])
def test_full_cells_against_the_oracle(dim, count, layout):
    res = 40
    x, v, F, C = _scene(dim, count, layout, res)
    vol, mu, lam = 0.2 ** dim / count, 300.0, 500.0
    got = _substep(dim, torch.float32, res, x, v, F, C, vol, mu, lam, 0, soa=count % 2 == 1)
    Jp = np.ones((count, 1))
    full = lambda a: np.full(count, a)
    for _ in range(2):
        if dim == 3:
            O.substep_3d(res, float(res), 1.0, 1 / res, DT, vol, G, x, full(vol), full(mu), full(lam), v, F, C, Jp)
        else:
            O.substep_2d(res, float(res), 1.0, mu, lam, vol, 1 / res, DT, vol, G, x, v, F, C, Jp)
    tol, vs = TOL[torch.float32], max(1.0, float(np.abs(v).max()))
    close(got[0], x, tol["x"], scale=1.0, what="x")
    close(got[1], v, tol["v"], scale=vs, what="v")
    close(got[2], F, tol["F"], scale=1.0, what="F")
    close(got[3], C, tol["C"], scale=vs * res, what="C")


def test_rounding_of_dense_sums_beside_the_block_sorted_form():
    """Float error of C over a large time step (95 particles a cell): at most 1.15 times that of one block-sorted
    substep, whose sums are two-level (cells in shared memory, then chunks).  Parts of a node added one after
    another in no order give 1.25."""
    n, res, dt = 400_000, 64, 4e-4
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    x = (torch.rand((n, 3), generator=g, device="cuda") - 0.5) * 0.2 + 0.5
    side = torch.where(torch.arange(n, device="cuda") < n // 2, -1.0, 1.0)
    x[:, 0] += 0.15 * side
    v = 0.05 * rnd(n, 3)
    v[:, 0] -= side
    state = [x, v, (torch.eye(3, device="cuda") + 0.01 * rnd(n, 3, 3)).reshape(n, 9), rnd(n, 9)]
    vol = float(np.float32(2 * 0.2 ** 3 / n))
    mu, lam = 58.0, 87.0

    def run(dtype, block_sorted):
        prm = E.make_params(3, res, dtype, 1 / res, float(res), dt, G, vol, 1.0, vol, mu, lam, model="fixed_corotated")
        ws = E.Workspace(prm, n, "cuda")
        tail = (ctypes.c_void_p(ws.ptr), ctypes.c_size_t(ws.bytes), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        a = [t.to(dtype).clone().contiguous() for t in state] + [torch.ones(n, dtype=dtype, device="cuda")]
        A = E.particles_struct(*a)
        if not block_sorted:
            N.call("ffmpm_substep", ctypes.byref(prm), ctypes.byref(A), *tail)
            ws.raise_on_status()
            return a[3].double()
        b = [torch.empty_like(t) for t in a]
        B = E.particles_struct(*b)
        ids, out = torch.arange(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        N.call("ffmpm_substeps_sorted", ctypes.byref(prm), ctypes.byref(A), ctypes.byref(B), ctypes.c_void_p(ids.data_ptr()),
               ctypes.c_void_p(out.data_ptr()), 1, *tail)
        ws.raise_on_status()
        C = torch.empty_like(b[3])
        C[out.long()] = b[3]
        return C.double()

    exact = run(torch.float64, False)
    here, there = ((run(torch.float32, s) - exact).norm().item() for s in (False, True))
    assert here <= 1.15 * there, (here, there, here / there)
