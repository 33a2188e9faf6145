"""The float32 path's product at the edges of its tiles and runs, against float64, and bit for bit over the
ways a step can be cut."""
import math

import pytest
import torch

from test_kernels_gpu import dev

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def product(a, w, mode, out=None):
    from carbon_engine_b200 import ops
    n = w.shape[0] // 2 if mode in ops.GEMM_GATED else w.shape[0]
    out = torch.zeros(a.shape[0], n, device=dev()) if out is None else out
    ops.gemm_plain(a, w, out, mode)
    return out


# K: below one run, one run exactly, runs with a short last one, eight runs; K = 301 and 1031 are not whole vectors
@pytest.mark.parametrize("N,K", [(7, 5), (129, 32), (64, 301), (130, 512), (257, 1032), (66, 1031), (200, 2100)])
@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 32, 33, 65])
def test_float32_product_against_float64(M, N, K):
    from carbon_engine_b200 import ops
    torch.manual_seed(M * 1000 + K)
    a, w = torch.randn(M, K + 3, device=dev())[:, :K], torch.randn(2 * N, K, device=dev())
    aligned = a.contiguous()
    # every rounding of a sum of K terms moves it by at most EPS of the sum of the terms' magnitudes; the longest chain of roundings is
    # half a run long, plus the joining of 2 chains and 8 runs
    bound = (math.ceil(K / 2) + 10) * EPS * (a.double().abs() @ w.double().abs().T) + 1e-30
    want = a.double() @ w.double().T
    for x in (a, aligned):
        assert bool(((product(x, w, ops.GEMM_STORE).double() - want).abs() <= bound).all())
        base = torch.randn(M, 2 * N, device=dev())
        got = product(x, w, ops.GEMM_ACCUM_F32, base.clone()).double()
        assert bool(((got - want - base.double()).abs() <= bound + EPS * (want + base.double()).abs() + 1e-7).all())
        gate, up = want[:, :N], want[:, N:]
        for mode, act in ((ops.GEMM_SWIGLU, gate * torch.sigmoid(gate)), (ops.GEMM_RELUGLU, gate.clamp_min(0))):
            # the activation's slope is at most 1.1, so the two sums' bounds come through the product as 1.1 b_gate |up| + |act| b_up (and
            # their own product); the activation and the multiplication add a dozen roundings of the result
            b_gate, b_up = bound[:, :N], bound[:, N:]
            limit = 1.1 * b_gate * (up.abs() + b_up) + act.abs() * b_up + 12 * EPS * (act * up).abs() + 1e-30
            assert bool(((product(x, w, mode).double() - act * up).abs() <= limit).all()), mode
        assert torch.equal(product(x, w, ops.GEMM_RELU2), product(aligned, w, ops.GEMM_STORE).clamp_min(0) ** 2)
    # the vectors' path and the scalars' path take the same sums
    assert torch.equal(product(a, w, ops.GEMM_STORE), product(aligned, w, ops.GEMM_STORE))


# the second size has tiles enough for one block a tile from 1 token on, the first only with many tokens
@pytest.mark.parametrize("N,K", [(1024, 2048), (38000, 520)])
def test_float32_product_has_the_same_bits_in_every_tile_and_cluster(N, K):
    from carbon_engine_b200 import ops
    torch.manual_seed(1)
    a, w = torch.randn(2600 if N < 2000 else 70, K, device=dev()), torch.randn(N, K, device=dev())
    whole = product(a, w, ops.GEMM_STORE)
    for lo, n in ((0, 1), (3, 4), (1, 7), (30, 33), (2, 64), (5, 65)):
        assert torch.equal(product(a[lo:lo + n], w, ops.GEMM_STORE), whole[lo:lo + n]), n
