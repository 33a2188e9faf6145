"""Float32 products of up to 8 tokens that a block takes for all of K: the same bits as the tiles of 64 tokens."""
import pytest
import torch

from test_kernels_gpu import dev

pytestmark = pytest.mark.gpu
NAME = "gemm_f32_stream_kernel"


# rows of a block: 5 (few, and a last block of one row: 593 = 148 x 4 + 1), 14 (two groups of lanes), 21, 33 and 64 (two rows a lane), 65 and
# 113 (three and four); gated twice as many; K with an odd number of stages a run
@pytest.mark.parametrize("N,K,gated", [(593, 2048, False), (2048, 6144, False), (3072, 2304, False), (4800, 2048, False), (9472, 2048, False),
                                       (9500, 2816, False), (16700, 2048, False), (700, 2048, True), (2368, 2304, True), (6144, 2048, True),
                                       (8300, 2560, True)])
@pytest.mark.parametrize("M", [1, 4, 5, 8])
@pytest.mark.parametrize("weights_ready", [False, True])
def test_stream_products_have_the_bits_of_the_tiles(N, K, gated, M, weights_ready):
    from carbon_engine_b200 import ops
    torch.manual_seed(N + M)
    a = torch.randn(64, K + 4, device=dev())[:, :K]                      # rows further apart than they are long
    w = torch.randn((2 if gated else 1) * N, K, device=dev()) / K ** 0.5
    bias = torch.randn(2 * N, device=dev())

    def run(a, mode, glu=None):
        out = torch.full((len(a), N), 0.5, device=dev())
        before = ops.kernel_counts().get(NAME, 0)
        ops.gemm_plain(a, w, out, mode, glu, weights_ready)
        assert ops.kernel_counts().get(NAME, 0) - before == (len(a) <= 8)
        return out

    modes = [(ops.GEMM_SWIGLU, None), (ops.GEMM_RELUGLU, None), (ops.GEMM_CLAMPGLU, ops.GluParams(1.3, 1.702, bias))] if gated else \
        [(ops.GEMM_STORE, None), (ops.GEMM_ACCUM_F32, None), (ops.GEMM_RELU2, None)]
    for mode, glu in modes:
        assert torch.equal(run(a[7:7 + M], mode, glu), run(a, mode, glu)[7:7 + M]), mode


# every depth of a ring that a number of rows can have (a block's rows, then stages for 1 to 4 and 5 to 8 tokens): 8 / 8 and 6 (7, 16 rows),
# 7 / 6 (17), 5 / 4 (26), 4 / 4 (33, 45: three rows a lane, two groups of lanes), 6 / 5 (49), 5 / 4 (60), 4 / 3 (66, 90), 3 / - (100)
@pytest.mark.parametrize("N,K,gated", [(890, 2304, False), (2367, 2048, False), (2500, 2304, False), (3700, 2048, False), (6300, 2304, False),
                                       (6660, 2816, False), (7201, 2048, False), (8879, 2304, False), (9700, 2048, False), (13300, 2048, False),
                                       (14700, 2048, False), (1190, 2048, True), (1340, 2304, True), (3300, 2816, True), (3552, 2048, True)])
@pytest.mark.parametrize("M", [1, 8])
def test_rings_of_every_depth_have_the_bits_of_the_tiles(N, K, gated, M):
    test_stream_products_have_the_bits_of_the_tiles(N, K, gated, M, True)
