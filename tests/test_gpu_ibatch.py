"""The integer batch kernel at the edges of its tiles, for every weight format, against the CPU oracle.

Rows 2..8 use one 8-row tile, up to 16, 32 and 64 the wider forms, above 64 several passes. Widths: a single row, one ragged
16-row tile, fewer tiles than SMs, more than one tile per thread block with a ragged last one. Lengths: one block, blocks that
do not divide among the warps, and activations that need several chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FORMATS = ("Q4_0", "Q4_1", "Q5_0", "Q5_1", "Q8_0", "Q2K", "Q3K", "Q4K", "Q5K", "Q6K")


@pytest.mark.parametrize("name", FORMATS)
def test_batch_edges_match_the_oracle(oracle, name):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fuel_b200 import GgmlDType as T, _lib, ops
    from test_gpu_kernels import assert_matmul_close
    t, ot = getattr(T, name), getattr(oracle, name)
    g = np.random.Generator(np.random.PCG64(11))
    _lib.check(_lib.lib.fuelq_set_option(_lib.OPT_DECODE_MAX_M, 1 << 20), "set_option")
    try:
        for n, k, ms in ((1, 256, (2, 9)), (37, 768, (2, 8, 9, 16, 17, 33, 64, 65, 130)), (300, 11008, (7, 45, 67)), (4757, 1280, (3, 31))):
            wb = oracle.quantize(ot, g.standard_normal((n, k), dtype=np.float32) * np.float32(0.02))
            x_all = g.standard_normal((max(ms), k), dtype=np.float32)
            x_all[1] = 0.0
            wd = torch.from_numpy(wb).cuda()
            for m in ms:
                got = ops.qmatmul(t, wd, n, torch.from_numpy(x_all[:m]).cuda()).cpu().numpy()
                assert_matmul_close(got, oracle.matmul(ot, x_all[:m], wb, n), (name, n, k, m))
    finally:
        _lib.lib.fuelq_set_option(_lib.OPT_DECODE_MAX_M, 0)
    assert ops.device_error() == 0
