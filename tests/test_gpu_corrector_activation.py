"""The corrector's activation far from zero: GELU of the third layer's biases, alone through the network (all
other weights zero), at large arguments, infinities and NaN."""
import ctypes
import math

import numpy as np
import pytest
import torch

from femflow_gb300 import _native as N
from femflow_gb300 import engine as E
from femflow_gb300 import learned as L
from femflow_gb300.diff import pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z", [-5.0, 5.0, -6.5, 6.5, -30.0, 30.0, -1e4, -1e8, 1e8, -3e38, 3e38, math.inf, -math.inf, math.nan])
def test_gelu_far_from_zero(z):
    res, count, dev = 16, 130, "cuda"
    net = L.Net(max_batch=256, seed=1)
    for w in net.W.values():
        w.zero_()
    net.W["W4"][3, 7] = 1.0  # output 3 (an entry of F) is unit 7 of the third layer
    net.params[N.MLP_OFF["b1"]:] = 0.0
    net.params[N.MLP_OFF["b3"] + 7] = z
    x = 0.5 + 0.05 * torch.arange(count, device=dev).view(-1, 1) / count * torch.ones(1, 3, device=dev)
    buf = pack(x, torch.zeros(count, 3, device=dev), torch.eye(3, device=dev).repeat(count, 1, 1), torch.zeros(count, 3, 3, device=dev))
    gv = torch.zeros((res + 1) ** 3, 3, device=dev)
    Jp = torch.ones(count, device=dev)
    prm = E.make_params(3, res, torch.float32, 1 / res, float(res), 1e-4, 0.0, 1e-6, 1.0, 1e-6, 60.0, 90.0)
    P = N.Particles()
    P.n, P.stride = count, count
    P.x, P.v, P.F, P.C = (buf.data_ptr() + 4 * count * r for r in (0, 3, 6, 15))
    P.Jp = Jp.data_ptr()
    G, m, st = E.grid_struct(gv, None), net.mlp(), torch.zeros(1, dtype=torch.int32, device=dev)
    N.call("ffmpm_corrector_g2p", ctypes.byref(prm), ctypes.byref(G), ctypes.byref(P), ctypes.byref(m), None, None,
           ctypes.c_void_p(st.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    got = buf[6 + 3].cpu().numpy().astype(np.float64)  # F at rest is the identity: entry 3 is zero
    if math.isnan(z):
        assert np.isnan(got).all()
    elif z == math.inf or abs(z) == 3e38:
        # (a bf16 has float's exponents: 3e38 stays finite)
        assert (got == math.inf).all() if z == math.inf else np.allclose(got, max(z, 0.0), rtol=2 ** -8, atol=1e-7)
    else:
        # within a bf16 rounding of the unit, and 1e-7 for the tail below -6
        want = 0.0 if z < -30.0 else z * 0.5 * math.erfc(-z / math.sqrt(2.0))
        assert np.abs(got - want).max() <= 2 ** -8 * abs(want) + 1e-7, (z, got[0], want)
