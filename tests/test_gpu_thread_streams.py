"""Weights made on cudaStreamPerThread: one handle, a stream in every thread.

The threads wait for their own work before they end, and the whole runs in a process of its own with a time limit: a stop there
is this test's failure and holds up no other."""
import ctypes
import os
import subprocess
import sys
import threading

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PER_THREAD = 2   # cudaStreamPerThread


def _run(made_in):
    """Two threads run products at the same time: a weight each, made by the thread that runs it or by another; or one weight."""
    import numpy as np
    import torch
    from fuel_b200 import GgmlDType as T, _lib, ops
    L = _lib.lib
    g = torch.Generator(device="cuda").manual_seed(3)
    m, n, k, calls = 5, 512, 8192, 60
    ws = [ops.quantize_weights(T.Q6K, torch.randn(n, k, generator=g, device="cuda")) for _ in range(2)]
    if made_in == "one weight":
        ws[1] = ws[0]
    xs = [torch.randn(m, k, generator=g, device="cuda") for _ in range(2)]
    want = [ops.qmatmul(T.Q6K, w, n, x) for w, x in zip(ws, xs)]
    ys = [torch.zeros(calls, m, n, device="cuda") for _ in range(2)]
    host = [np.ascontiguousarray(w.cpu().numpy()) for w in ws]
    torch.cuda.synchronize()

    def load(i):
        h = ctypes.c_void_p()
        _lib.check(L.fuelq_qtensor_load(0, PER_THREAD, int(T.Q6K), n, k, host[i].ctypes.data, host[i].size, ctypes.byref(h)), "load")
        return h

    handles, errors, start, done = [None, None], [], threading.Barrier(2), threading.Barrier(2)
    if made_in == "one thread":
        handles = [load(0), load(1)]
    elif made_in == "one weight":
        handles = [load(0)] * 2

    def work(i):
        try:
            if handles[i] is None:
                handles[i] = load(i)
            back = np.empty_like(host[i])
            start.wait(60)
            for y in ys[i]:
                _lib.check(L.fuelq_qmatmul_forward(handles[i], xs[i].data_ptr(), m, y.data_ptr()), "forward")
            _lib.check(L.fuelq_qtensor_data(handles[i], back.ctypes.data, back.size), "data")   # waits for this thread's stream
            done.wait(60)
        except Exception as e:   # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,), daemon=True) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(90)
    assert not errors and not any(t.is_alive() for t in threads), errors
    for i in range(2):
        assert torch.equal(ys[i], want[i].expand_as(ys[i])), (made_in, i)
    for h in {h.value: h for h in handles}.values():
        L.fuelq_qtensor_free(h)
    assert ops.device_error() == 0


@pytest.mark.gpu
def test_threads_do_not_share_scratch_between_their_streams():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], cwd=ROOT, capture_output=True, text=True, timeout=240)
    assert r.returncode == 0 and "threads ok" in r.stdout, r.stdout + r.stderr


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    for mode in ("each thread", "one thread", "one weight"):
        _run(mode)
    print("threads ok")
