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


@pytest.mark.parametrize("name", ("Q4K", "Q6K"))
@pytest.mark.parametrize("counts,n,k", [
    ([0, 3, 0, 0, 1, 0, 0, 9] + [0] * 56, 293, 768),          # few groups: blocks of their own
    ([1] * 70 + [0] * 5 + [40] + [2] * 52, 37, 512),          # many: blocks that span several, one group in several passes
    ([17, 0, 33, 24, 8, 130, 1, 16] * 5, 165, 2304),          # several passes of 32 rows
    ([26, 31, 12, 0, 25, 18, 32, 20] * 16, 85, 2048),         # some twenty rows each: sixteen warps a block
    ([0, 0, 1, 0], 37, 1280),                                 # a single row: planes, the sums converted as they are staged
])
def test_groups_match_the_oracle(oracle, name, counts, n, k):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fuel_b200 import GgmlDType as T, _lib, ops
    from test_gpu_kernels import assert_matmul_close
    t, ot, L = getattr(T, name), getattr(oracle, name), _lib.lib
    g = np.random.Generator(np.random.PCG64(5))
    e, rows = len(counts), sum(counts)
    wb = oracle.quantize(ot, g.standard_normal((e * n, k), dtype=np.float32) * np.float32(0.02))
    x = g.standard_normal((rows, k), dtype=np.float32)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    order = g.permutation(rows).astype(np.int32)               # where each row's result goes
    xd, wd, od, rd = (torch.from_numpy(a).cuda() for a in (x, wb, off, order))
    ids = torch.arange(rows, dtype=torch.int32, device="cuda")
    packed = torch.empty(L.fuelq_act_packed_bytes(int(T.Q4K), rows, k), dtype=torch.uint8, device="cuda")
    y = torch.full((rows, n), float("nan"), device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(L.fuelq_moe_quantize_rows(xd.data_ptr(), k, ids.data_ptr(), 1, rows, packed.data_ptr(), packed.numel(), st), "quantize")
    _lib.check(L.fuelq_moe_qmatmul(int(t), e, n, k, wd.data_ptr(), packed.data_ptr(), rows, od.data_ptr(), rd.data_ptr(), y.data_ptr(), st), "qmatmul")
    got = y.cpu().numpy()[order]
    per = wb.size // e
    for i, c in enumerate(counts):
        if c:
            r = slice(off[i], off[i] + c)
            assert_matmul_close(got[r], oracle.matmul(ot, x[r], wb.reshape(-1)[i * per:(i + 1) * per], n), (name, i, c))
    assert ops.device_error() == 0


@pytest.mark.parametrize("name", FORMATS)
def test_a_row_that_is_not_finite_stays_by_itself(name):
    """Rows are columns of the MMAs: infinities and NaN in some rows change no bit of the others, in the same call or the next."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fuel_b200 import GgmlDType as T, ops
    t, n, k = getattr(T, name), 83, 1536
    gen = torch.Generator(device="cuda").manual_seed(17)
    w = ops.quantize_weights(t, torch.randn(n, k, generator=gen, device="cuda"))
    for m in (2, 7, 16):
        x = torch.randn(m, k, generator=gen, device="cuda")
        want = ops.qmatmul(t, w, n, x)
        bad = x.clone()
        bad[m // 2, 3], bad[m // 2, 700] = float("inf"), float("nan")
        got = ops.qmatmul(t, w, n, bad)
        rest = [i for i in range(m) if i != m // 2]
        assert torch.equal(got[rest], want[rest]), m
        ops.qmatmul(t, w, n, torch.full((16, k), float("nan"), device="cuda"))
        assert torch.equal(ops.qmatmul(t, w, n, x), want), m
    assert ops.device_error() == 0
