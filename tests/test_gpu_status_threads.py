"""A thread that has read a status word ends while another thread captures a stream: the capture, which allows
no unsafe call by any thread, goes on."""
import os
import threading
import time

import pytest
import torch

from femflow_gb300 import engine as E

pytestmark = pytest.mark.gpu


def test_a_thread_that_read_a_status_ends_during_a_capture():
    prm = E.make_params(3, 16, torch.float32, 1 / 16, 16.0, 1e-4)
    ws = E.Workspace(prm, 100, "cuda")
    read, go, tid = threading.Event(), threading.Event(), []

    def worker():
        assert ws.status() == (0, 0)
        tid.append(threading.get_native_id())
        read.set()
        go.wait(30)

    t = threading.Thread(target=worker)
    t.start()
    assert read.wait(30)
    x = torch.zeros(16, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        x += 1
        go.set()
        t.join(30)
        end = time.monotonic() + 10
        while os.path.exists(f"/proc/self/task/{tid[0]}") and time.monotonic() < end:
            time.sleep(0.01)  # the thread's own end follows that of its Python part
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert bool((x == 2).all())
