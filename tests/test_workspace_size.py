"""What a workspace holds for the in-place operations' counting sort by cell: counters and first slots per node
(8 bytes), a record per float particle (64 bytes in 3D, 48 in 2D); nothing for callers that keep their particles
near cell order, who never sort (the resident solver, the host-array substep)."""
import pytest
import torch

from femflow_gb300 import _native as N
from femflow_gb300 import engine as E


def _bytes(dim, res, n, dtype, variant):
    return E.workspace_bytes(E.make_params(dim, res, dtype, 1 / res, float(res), 1e-4, variant=variant), n)


@pytest.mark.parametrize("dim,res,dtype,record", [(3, 64, torch.float32, 64), (2, 128, torch.float32, 48),
                                                  (3, 64, torch.float64, 0), (2, 128, torch.float64, 0)])
def test_room_for_the_sort_by_cell(dim, res, dtype, record):
    n = 100_000
    with_sort, without = (_bytes(dim, res, n, dtype, v) for v in (0, N.VARIANT_CELL_ORDER))
    nodes = -(-(res + 1) ** dim // 4096) * 4096
    assert record * n + 8 * nodes <= with_sort - without <= record * n + 8 * nodes + 3 * 256


def test_room_does_not_depend_on_the_other_variants():
    assert len({_bytes(3, 64, 100_000, torch.float32, v) for v in (0, 1, 2, 4, 8 << 8)}) == 1


@pytest.mark.gpu
def test_solver_and_host_substep_keep_none():
    from femflow_gb300.solver import MPMSolver
    from femflow_gb300.solvers.mpm import mls_mpm
    from femflow_gb300.solvers.mpm.particle import ParticleSet

    n, res = 50_001, 48
    x = 0.3 + 0.4 * torch.rand(n, 3)
    s = MPMSolver(x, res=res, dt=1e-4, volume=1e-6, mass=1e-6, mu_0=300.0, lambda_0=500.0)
    assert s.ws.bytes == _bytes(3, res, n, torch.float32, N.VARIANT_CELL_ORDER)
    pin = lambda t: t.clone().pin_memory()
    one = torch.ones(n)
    before = set(E._WS_CACHE)
    mls_mpm.solve_mls_mpm_3d(res, float(res), 1.0, 1 / res, 1e-4, 1e-6, -9.8,
                             ParticleSet(pin(x), pin(1e-6 * one), pin(300 * one), pin(500 * one)), pin(0 * x),
                             pin(torch.eye(3).repeat(n, 1, 1)), pin(torch.zeros(n, 3, 3)), pin(one[:, None]))
    (new,) = set(E._WS_CACHE) - before
    assert E._WS_CACHE[new].bytes == _bytes(3, res, n, torch.float32, N.VARIANT_CELL_ORDER)
    assert s.ws.bytes + 64 * n < _bytes(3, res, n, torch.float32, 0)
