"""Scratch of products recorded into a graph."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_recorded_calls_keep_scratch_of_their_own():
    """A product recorded on a stream and replayed on another, beside eager products of another weight on the first."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fuel_b200 import GgmlDType as T, ops
    from fuel_b200.quantized import QMatMul, QTensor
    gen = torch.Generator(device="cuda").manual_seed(3)
    home, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(home):
        a, b = (QMatMul.from_qtensor(QTensor.quantize(torch.randn(n, 2048, generator=gen, device="cuda"), T.Q4K)) for n in (512, 768))
        xa, xb = torch.randn(5, 2048, generator=gen, device="cuda"), torch.randn(40, 2048, generator=gen, device="cuda")
        want_a, want_b = a.forward(xa), b.forward(xb)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=home):
        out = a.forward(xa)
    torch.cuda.synchronize()
    for _ in range(50):
        with torch.cuda.stream(other):
            graph.replay()
        with torch.cuda.stream(home):
            yb = b.forward(xb)
    torch.cuda.synchronize()
    assert torch.equal(out, want_a) and torch.equal(yb, want_b)
    assert ops.device_error() == 0
