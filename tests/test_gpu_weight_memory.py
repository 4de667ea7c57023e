"""Device memory of weights: whose it is, and when it goes back."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def _device():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _weight(n, k, seed):
    from fuel_b200 import GgmlDType as T
    from fuel_b200.quantized import QMatMul, QTensor
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return QMatMul.from_qtensor(QTensor.quantize(torch.randn(n, k, generator=gen, device="cuda"), T.Q8_0))


def test_a_freed_weight_is_the_drivers_again():
    keep = _weight(256, 256, 0)                      # the library's own set-up is done
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    w = [_weight(8192, 4096, i) for i in range(4)]   # 34 MiB of blocks each
    torch.cuda.empty_cache()
    assert torch.cuda.mem_get_info()[0] < before - (100 << 20)
    del w
    torch.cuda.empty_cache()
    assert torch.cuda.mem_get_info()[0] > before - (16 << 20)
    assert keep is not None


def test_a_weight_freed_during_a_capture_leaves_the_graph_whole():
    from fuel_b200 import ops
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        a, b = _weight(512, 1024, 1), _weight(4096, 4096, 2)
        x = torch.randn(3, 1024, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
        want = a.forward(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        first = a.forward(x)
        del b
        second = a.forward(x)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(first, want) and torch.equal(second, want)
    assert ops.device_error() == 0
