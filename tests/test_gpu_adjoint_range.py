"""Adjoint of float states: at masses whose momenta float cannot hold (without stress the gradients do not depend on
the mass, so powers of two of it give those of unit mass: the float64 adjoint, at the float adjoint's bound), and
the sums in float pairs beside float64 terms."""
import numpy as np
import pytest
import torch

from test_gpu_adjoint_pairs import _adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mass", [2.0 ** 124, 2.0 ** 100, 1.0, 2.0 ** -100])
@pytest.mark.parametrize("count", [33, 3001])
def test_gradients_without_stress_do_not_depend_on_the_mass(count, mass):
    res, dt = 32, 1e-4
    rng = np.random.default_rng(count)
    r32 = lambda a: np.asarray(a).astype(np.float32).astype(np.float64)
    # 100 times 2^124 is beyond float; one particle in 40 stands still (a term that is zero)
    v = rng.normal(0, 100, (count, 3))
    v[::40] = 0.0
    state = [r32(rng.uniform(0.3, 0.6, (count, 3))), r32(v), np.tile(np.eye(3), (count, 1, 1)), r32(rng.normal(0, 1, (count, 3, 3)))]
    adj = [r32(rng.normal(0, 1, s.shape)) for s in state]
    got = _adjoint(torch.float32, res, state, adj, mass, 0.0, 0.0, dt)
    want = _adjoint(torch.float64, res, state, adj, 1.0, 0.0, 0.0, dt)
    for k, (a, b) in enumerate(zip(got[:4], want[:4])):  # x, v, F, C
        if k == 0 and mass > 2.0 ** 116:
            continue  # the derivative of the weights takes the momentum m v in float: not finite
        assert np.abs(a - b).max() <= 2e-3 * max(np.abs(b).max(), 1e-30), (k, np.abs(a - b).max(), np.abs(b).max())


@pytest.mark.parametrize("count", [3001, 20000])
def test_pairs_keep_what_float64_terms_keep(count):
    """A large common part in velocities and adjoints, of which the stress derivative sees the variation: the sums in
    float pairs give the gradients of float64 terms to float's rounding (2^-22 in norm; plain float terms give 4e-6).
    The float64 terms: one particle of every warp has values that pairs do not hold, in place of zeros."""
    res, dt = 32, 1e-4
    r32 = lambda a: np.asarray(a).astype(np.float32).astype(np.float64)
    few = np.arange(count) % 32 == 0

    def run(tiny):
        g = np.random.default_rng(count)
        state = [r32(g.uniform(0.4, 0.6, (count, 3))), r32(10 + g.normal(0, 0.1, (count, 3))),
                 r32(np.eye(3) + g.normal(0, 0.01, (count, 3, 3))), r32(g.normal(0, 1, (count, 3, 3)))]
        adj = [np.zeros((count, 3)), r32(10 + g.normal(0, 0.1, (count, 3))), np.zeros((count, 3, 3)), np.zeros((count, 3, 3))]
        state[1][few] = tiny
        adj[3][few] = tiny
        return _adjoint(torch.float32, res, state, adj, 0.2 ** 3 / count, 1500.0, 2300.0, dt)

    for k, (a, b) in enumerate(zip(run(0.0), run(1e-30))):
        assert np.linalg.norm(a - b) <= 2.0 ** -22 * np.linalg.norm(b), (k, np.linalg.norm(a - b) / np.linalg.norm(b))
