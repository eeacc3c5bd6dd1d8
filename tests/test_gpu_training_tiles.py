"""Training kernels of the corrector network at the edges of their tiling, against the numpy oracle with
the GPU's rounding points: one tile of 128 rows, as many tiles as SMs, one more (a CTA with two tiles, whose
weight gradients accumulate), a batch below max_batch, and float buffers that are not 16-byte aligned."""
import numpy as np
import pytest
import torch

from oracle import mlp as M
from femflow_gb300 import _native as N
from femflow_gb300 import learned as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,spare,shift", [(1, 0, 0), (3, 5, 0), (152, 0, 0), (153, 0, 0), (2, 0, 1)])
def test_training_pass_at_tile_edges(tiles, spare, shift):
    rng = np.random.default_rng(tiles)
    B = 128 * tiles
    net = L.Net(max_batch=B + 128 * spare, seed=1)
    net.params[M.OFF["b1"]:M.OFF["b1"] + 192] = torch.tensor(rng.normal(0, 0.1, 192), dtype=torch.float32)
    net.params[M.OFF["b4"]:M.OFF["b4"] + 12] = torch.tensor(rng.normal(0, 0.1, 12), dtype=torch.float32)
    net.repack()
    if shift:
        f32 = lambda *s: torch.zeros(int(np.prod(s)) + shift, device="cuda")[shift:].view(*s)
        for k, s in (("Z1", 64), ("Z2", 64), ("Z3", 64), ("Y", 16)):
            net.buf[k] = f32(net.max_batch, s)
        net.grads = f32(N.MLP_PARAMS)
        assert net.grads.data_ptr() % 16 != 0
    X = rng.normal(0, 1, (B, 128))
    X = torch.from_numpy(X.astype(np.float32)).to(torch.bfloat16).cuda()  # columns 113.. are not zero
    T = torch.tensor(rng.normal(0, 1, (B, 12)), dtype=torch.float32, device="cuda")
    w = torch.tensor(rng.uniform(0.5, 2.0, 12), dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    P = net.params.cpu().numpy().copy()
    P[:64 * 128].reshape(64, 128)[:, N.MLP_FEATURES:] = 0  # weights of unused features start as zero
    Y = net.forward_train(X).cpu().numpy()
    net.backward_train(T, w, loss)
    net.check()
    Xr = X.float().cpu().numpy()
    l_ref, g_ref, Y_ref = M.backward(P, Xr, T.cpu().numpy(), w.cpu().numpy())
    rel = lambda a, b: float(np.linalg.norm(a - b) / np.linalg.norm(b))
    # bf16 operands of the same rounding points: the bounds of the training test at 1,024 rows
    assert rel(Y, Y_ref) < 1e-3
    assert abs(float(loss.item()) - l_ref) <= 1e-3 * l_ref
    g = net.grads.cpu().numpy()
    for k, n in (("W2", 4096), ("W3", 4096), ("W4", 768), ("b1", 64), ("b2", 64), ("b3", 64), ("b4", 12)):
        sl = slice(M.OFF[k], M.OFF[k] + n)
        assert rel(g[sl], g_ref[sl]) < 1e-2, k
    g1, r1 = (a[:64 * 128].reshape(64, 128) for a in (g, g_ref))
    assert rel(g1[:, :N.MLP_FEATURES], r1[:, :N.MLP_FEATURES]) < 1e-2
    assert np.all(g1[:, N.MLP_FEATURES:] == 0)
    assert np.all(g[64 * 128:M.OFF["W2"]] == 0) and np.all(g[M.OFF["W4"] + 768:M.OFF["b1"]] == 0)
    # what the forward pass keeps
    b = net.buf
    for i, t in (("H1", "H1t"), ("H2", "H2t"), ("H3", "H3t")):
        assert torch.equal(b[t].reshape(-1)[:64 * B].view(64, B), b[i][:B].t())
    Xt = b["Xt"].reshape(-1)[:128 * B].view(128, B)
    assert torch.equal(Xt[:N.MLP_FEATURES], X.t()[:N.MLP_FEATURES]) and not bool(Xt[N.MLP_FEATURES:].any())
