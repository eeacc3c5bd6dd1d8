"""Radix sort at the counts where its tiles change size (a quarter, half and the whole of 4,096 keys) and at
their edges: the permutation equals numpy's stable argsort."""
import ctypes

import numpy as np
import pytest
import torch

from femflow_gb300 import _native as N
from femflow_gb300 import engine as E
from test_gpu_sort_and_solver import host_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1023, 1024, 1025, 151_552, 151_553, 303_104, 303_105, 310_001])
def test_sort_at_tile_size_changes(count):
    res = 64
    x = np.random.default_rng(count).uniform(0.05, 0.95, size=(count, 3)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    prm = E.make_params(3, res, torch.float32, 1 / res, float(res), 1e-4)
    ws = E.Workspace(prm, count, "cuda")
    keys = torch.empty(count, dtype=torch.int32, device="cuda")
    perm = torch.empty(count, dtype=torch.int32, device="cuda")
    N.call("ffmpm_sort_by_block", ctypes.byref(prm), ctypes.c_void_p(xd.data_ptr()), count,
           ctypes.c_void_p(keys.data_ptr()), ctypes.c_void_p(perm.data_ptr()), ctypes.c_void_p(ws.ptr),
           ctypes.c_size_t(ws.bytes), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert ws.status()[0] == 0
    hk = host_keys(x, res, 8, False)
    ref = np.argsort(hk, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), ref)
    assert np.array_equal(keys.cpu().numpy().view(np.uint32).astype(np.uint64), hk[ref])
