"""Fused corrector G2P at the edges of its tiling: counts around a tile of 128 particles, more tiles than the
four groups of every SM take at once, a particle outside the grid among them; against the plain G2P plus the
training forward of the exported features (the same bf16 operands; GELU differs by float rounding)."""
import ctypes

import numpy as np
import pytest
import torch

from femflow_gb300 import _native as N
from femflow_gb300 import engine as E
from femflow_gb300 import learned as L
from femflow_gb300.diff import pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,out", [(1, False), (127, False), (129, True), (1000, False), (128 * 608 + 5, True)])
def test_corrected_g2p_at_tile_edges(count, out):
    res, dt = 32, 4e-4
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(count)
    rnd = lambda *s: torch.randn(s, generator=g, device=dev)
    x = 0.3 + 0.4 * torch.rand((count, 3), generator=g, device=dev)
    if out:
        x[count // 2] = 2.0
    F = torch.eye(3, device=dev) + 0.02 * rnd(count, 3, 3)
    buf = pack(x, rnd(count, 3), F, rnd(count, 3, 3))
    gv = rnd((res + 1) ** 3, 3).contiguous()
    Jp = torch.ones(count, device=dev)
    prm = E.make_params(3, res, torch.float32, 1 / res, float(res), dt, -9.8, 1e-6, 1.0, 1e-6, 60.0, 90.0,
                        model="fixed_corotated")
    net = L.Net(max_batch=(count + 127) // 128 * 128, seed=3)
    net.in_scale.copy_(0.5 + torch.rand(128, generator=g, device=dev))
    net.out_scale[:12] = 1e-3

    def run(net_, feats):
        b = buf.clone()
        P = N.Particles()
        P.n, P.stride = count, count
        P.x, P.v, P.F, P.C = (b.data_ptr() + 4 * count * r for r in (0, 3, 6, 15))
        P.Jp = Jp.data_ptr()
        G = E.grid_struct(gv, None)
        st = torch.zeros(1, dtype=torch.int32, device=dev)
        m = net_.mlp() if net_ is not None else None
        N.call("ffmpm_corrector_g2p", ctypes.byref(prm), ctypes.byref(G), ctypes.byref(P),
               ctypes.byref(m) if m is not None else None, ctypes.c_void_p(feats.data_ptr() if feats is not None else 0),
               None, ctypes.c_void_p(st.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert int(st.item()) == (N.STATUS_OOB if out else 0)
        return b

    X = torch.zeros((net.max_batch, 128), dtype=torch.bfloat16, device=dev)
    plain = run(None, None)
    corr = run(net, X)  # features (scaled) exported beside the correction
    y = net.forward_train(X)[:count] * net.out_scale[:12]
    inside = torch.ones(count, dtype=torch.bool, device=dev)
    if out:
        inside[count // 2] = False
        assert torch.equal(corr[:, count // 2], buf[:, count // 2])  # left as it was
    vs = dt * res
    k = inside
    # a bf16 flip of one hidden unit moves an output by about 1e-2 of its size, 1e-5 after out_scale
    assert float((corr[6:15] - plain[6:15] - y[:, :9].t())[:, k].abs().max() if bool(k.any()) else 0.0) <= 2e-5
    assert float((corr[3:6] - plain[3:6] - y[:, 9:12].t() / vs)[:, k].abs().max()) <= 2e-5 / vs
    assert float((corr[0:3] - plain[0:3] - dt * y[:, 9:12].t() / vs)[:, k].abs().max()) <= 2e-5
    assert torch.equal(corr[15:24], plain[15:24])
    # the grid features against torch: (v_i - u) dt / dx times the input scale, in bf16
    xs = buf[0:3].t() * res
    b = torch.trunc(xs - 0.5).long()
    at = lambda i, j, l: ((b[:, 0] + i) * (res + 1) + b[:, 1] + j) * (res + 1) + b[:, 2] + l
    idx = torch.stack([at(i, j, l) for i in range(3) for j in range(3) for l in range(3)], 1)[k]
    want = ((gv[idx] - gv[idx[:, 13]][:, None]) * vs).reshape(-1, 81) * net.in_scale[21:102]
    got = X[:count][k][:, 21:102].float()
    assert float((got - want).abs().max()) <= 2 ** -8 * float(want.abs().max())
    assert not bool(X[:count][:, 113:].any())
