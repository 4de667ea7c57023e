"""Chains of calls that are enqueued without a wait on the host, in the default launch mode: every kernel is put on the SMs
before its predecessor ends, so what it reads must come after its wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def _device():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("name,m", [("Q4K", 1), ("Q4K", 2), ("Q6K", 4), ("Q8_0", 3), ("Q4_0", 1), ("Q3K", 1), ("Q5_1", 2)])
def test_host_results_feed_the_next_host_call(name, m):
    """Pinned activations and results: each call's result is the next call's input, written back and read by kernels."""
    from fuel_b200 import GgmlDType as T, ops
    t, n, steps = getattr(T, name), 2048, 24
    gen = torch.Generator(device="cuda").manual_seed(m)
    ws = [ops.quantize_weights(t, torch.randn(n, n, generator=gen, device="cuda") / n ** 0.5) for _ in range(3)]
    bufs = [torch.empty(m, n).pin_memory() for _ in range(steps + 1)]
    bufs[0].copy_(torch.randn(m, n, generator=torch.Generator().manual_seed(5)))
    scratch = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    for i in range(steps):
        ops.qmatmul_host(t, ws[i % 3], n, bufs[i], bufs[i + 1], scratch)
    torch.cuda.synchronize()
    want = torch.empty(m, n).pin_memory()
    for i in range(steps):
        ops.qmatmul_host(t, ws[i % 3], n, bufs[i], want, scratch)
        torch.cuda.synchronize()
        assert torch.equal(bufs[i + 1], want), i
    assert ops.device_error() == 0
