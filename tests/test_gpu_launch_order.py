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


@pytest.mark.parametrize("name", ["Q4K", "Q6K", "Q8_0", "Q2K", "Q5_0"])
@pytest.mark.parametrize("m", [1, 2, 16, 65, 200])
def test_results_feed_the_next_call(name, m):
    """Each product's result is the next one's input, in one workspace: integer kernels up to the crossover, above it the
    conversion, several slabs (the first dequantized beside the conversion, the next ones over what the GEMM before them reads)
    and the GEMM."""
    from fuel_b200 import GgmlDType as T, _lib, ops
    t, n, steps = getattr(T, name), 1024, 12
    gen = torch.Generator(device="cuda").manual_seed(m)
    ws = [ops.quantize_weights(t, torch.randn(n, n, generator=gen, device="cuda") / n ** 0.5) for _ in range(3)]
    ys = [torch.empty(m, n, device="cuda") for _ in range(steps + 1)]
    ys[0].normal_(generator=gen)
    try:
        _lib.check(_lib.lib.fuelq_set_option(116, 768), "set_option")   # slabs of 384 rows: two whole ones and a rest
        scratch = torch.empty(_lib.lib.fuelq_qmatmul_workspace_bytes(int(t), m, n, n), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        for i in range(steps):
            ops.qmatmul(t, ws[i % 3], n, ys[i], out=ys[i + 1], workspace=scratch)
        torch.cuda.synchronize()
        for i in range(steps):
            want = ops.qmatmul(t, ws[i % 3], n, ys[i], workspace=scratch)
            torch.cuda.synchronize()
            assert torch.equal(ys[i + 1], want), i
    finally:
        _lib.lib.fuelq_set_option(116, 0)
    assert ops.device_error() == 0


@pytest.mark.parametrize("name", ["Q4K", "Q6K", "Q8_0", "Q3K", "Q4_1"])
@pytest.mark.parametrize("m", [1, 3, 40, 100])
def test_weights_quantized_just_before_their_product(name, m):
    """One buffer of blocks, written by the quantizer and read by the product behind it, over and over: a call streams weights
    beside its own kernels, never beside what comes before the call."""
    from fuel_b200 import GgmlDType as T, _lib, ops
    t, n, k, steps = getattr(T, name), 768, 2048, 8
    L, gen = _lib.lib, torch.Generator(device="cuda").manual_seed(m)
    ws = [torch.randn(n, k, generator=gen, device="cuda") for _ in range(steps)]
    x = torch.randn(m, k, generator=gen, device="cuda")
    blocks = torch.zeros(ops.storage_bytes(t, n * k), dtype=torch.uint8, device="cuda")
    scratch = torch.empty(L.fuelq_qmatmul_workspace_bytes(int(t), m, n, k), dtype=torch.uint8, device="cuda")
    ys = [torch.empty(m, n, device="cuda") for _ in range(steps)]
    st = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    for w, y in zip(ws, ys):
        _lib.check(L.fuelq_quantize_weights(int(t), n * k, w.data_ptr(), blocks.data_ptr(), st), "quantize")
        ops.qmatmul(t, blocks, n, x, out=y, workspace=scratch)
    torch.cuda.synchronize()
    for i, (w, y) in enumerate(zip(ws, ys)):
        b = ops.quantize_weights(t, w)
        torch.cuda.synchronize()
        assert torch.equal(y, ops.qmatmul(t, b, n, x)), i
    assert ops.device_error() == 0
