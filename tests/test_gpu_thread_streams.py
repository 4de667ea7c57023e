"""Weights made on cudaStreamPerThread: one handle, a stream in every thread."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
PER_THREAD = 2   # cudaStreamPerThread


def _load(blocks, t, n, k):
    from fuel_b200 import _lib
    h = ctypes.c_void_p()
    _lib.check(_lib.lib.fuelq_qtensor_load(0, PER_THREAD, int(t), n, k, blocks.ctypes.data, blocks.size, ctypes.byref(h)), "load")
    return h


def _forward(h, x, ys):
    from fuel_b200 import _lib
    for y in ys:
        _lib.check(_lib.lib.fuelq_qmatmul_forward(h, x.data_ptr(), x.shape[0], y.data_ptr()), "forward")


@pytest.mark.parametrize("made_in", ("each thread", "one thread", "one weight"))
@pytest.mark.parametrize("m", (1, 5, 200))
def test_threads_do_not_share_scratch_between_their_streams(m, made_in):
    """Two threads run products at the same time: a weight each, made by the thread that runs it or by another; or one weight."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fuel_b200 import GgmlDType as T, _lib, ops
    g = torch.Generator(device="cuda").manual_seed(m)
    n, k, calls = 512, 8192, 60
    ws = [ops.quantize_weights(T.Q6K, torch.randn(n, k, generator=g, device="cuda")) for _ in range(2)]
    if made_in == "one weight":
        ws[1] = ws[0]
    xs = [torch.randn(m, k, generator=g, device="cuda") for _ in range(2)]
    want = [ops.qmatmul(T.Q6K, w, n, x) for w, x in zip(ws, xs)]
    ys = [torch.zeros(calls, m, n, device="cuda") for _ in range(2)]
    host = [np.ascontiguousarray(w.cpu().numpy()) for w in ws]
    torch.cuda.synchronize()
    handles, errors = [None, None], []
    if made_in != "each thread":
        handles = [_load(b, T.Q6K, n, k) for b in host]
    if made_in == "one weight":
        _lib.lib.fuelq_qtensor_free(handles[1])
        handles[1] = handles[0]
    start = threading.Barrier(2)

    def work(i):
        try:
            if handles[i] is None:
                handles[i] = _load(host[i], T.Q6K, n, k)
            start.wait(60)
            _forward(handles[i], xs[i], ys[i])
        except Exception as e:   # noqa: BLE001 - reported by the test
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for h in {h.value: h for h in handles if h}.values():
        _lib.lib.fuelq_qtensor_free(h)
    assert not errors
    for i in range(2):
        assert torch.equal(ys[i], want[i].expand_as(ys[i])), i
    assert ops.device_error() == 0
