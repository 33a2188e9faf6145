"""Products of CTA pairs: the tiles' tokens and the parts of K that a cluster's pairs share, at sizes with remainders."""
import math

import pytest
import torch

from test_kernels_gpu import dev, rel_err

pytestmark = pytest.mark.gpu


# one token beyond 128 and beyond a tile, a last tile of one token, K with a last k-block and a last round cut short, N with a last
# tile of rows cut short; few tiles (K shared by two or three pairs) and many (one pair a tile)
@pytest.mark.parametrize("M,N,K,shared", [(129, 4096, 4096, True), (203, 4000, 8200, True), (400, 3850, 8200, True), (161, 3200, 2056, False),
                                          (257, 6000, 1160, False), (225, 12000, 520, False), (673, 4096, 2056, False),
                                          (1733, 3300, 1000, False)])
def test_pair_products_against_float64(M, N, K, shared):
    from carbon_engine_b200 import ops, ops_tensor
    torch.manual_seed(M + N)
    a = torch.randn(M, K, device=dev()).to(torch.bfloat16)
    w = (torch.randn(2 * N, K, device=dev()) / math.sqrt(K)).to(torch.bfloat16)
    ref = a.double() @ w.double().T

    def run(w, mode, dtype, x0=None):
        out = torch.full((M, N), float("nan"), dtype=dtype, device=dev()) if x0 is None else x0.clone()
        assert ops_tensor.gemm_bf16(a, w, out, mode)
        return out

    before = ops.kernel_counts()
    first = run(w[:N], ops.GEMM_STORE_F32, torch.float32)
    # float32 sums of K products of bfloat16 numbers, in the tensor core's and the splits' order
    assert rel_err(first, ref[:, :N]) < 2e-5
    x0 = torch.randn(M, N, device=dev())
    assert rel_err(run(w[:N], ops.GEMM_ACCUM_F32, torch.float32, x0), x0.double() + ref[:, :N]) < 2e-5
    assert torch.equal(run(w[:N], ops.GEMM_STORE, torch.bfloat16), first.to(torch.bfloat16))
    assert torch.equal(run(w[:N], ops.GEMM_RELU2, torch.bfloat16), (first.clamp_min(0) ** 2).to(torch.bfloat16))
    after = ops.kernel_counts()
    name = "gemm_tc_pair_kernel (split-K in a cluster)"
    assert (after.get(name, 0) > before.get(name, 0)) == shared
    for _ in range(3):                                                 # partial sums are added in split order
        assert torch.equal(run(w[:N], ops.GEMM_STORE_F32, torch.float32), first)
    g, u = ref[:, :N], ref[:, N:]
    # one rounding to bfloat16 (2^-9) of the largest results, and the activation's approximate exponential
    assert rel_err(run(w, ops.GEMM_SWIGLU, torch.bfloat16), g * torch.sigmoid(g) * u) < 1e-2
    assert ops_tensor.gemm_status(dev()) == 0


# (tokens, output columns, K, gated, pairs that share K): every number of sharers, gated or not (tests/test_launch_rules.py holds the
# launcher to these numbers), a last tile of rows and a last round of K cut short, a share of the tokens that is not a whole chunk
SHARED = [(203, 4000, 8200, False, 2), (131, 5000, 4104, False, 3), (250, 3300, 8200, False, 4), (500, 3850, 8200, False, 2),
          (203, 2000, 4104, True, 2), (131, 2500, 4104, True, 3), (250, 1600, 8200, True, 4)]


@pytest.mark.parametrize("M,N,K,gated,sharers", SHARED)
def test_every_number_of_pairs_that_share_k(M, N, K, gated, sharers):
    import plain_rapovik
    from carbon_engine_b200 import ops, ops_tensor
    torch.manual_seed(M + N)
    a = torch.randn(M, K, device=dev()).to(torch.bfloat16)
    w = (torch.randn((2 if gated else 1) * N, K, device=dev()) / math.sqrt(K)).to(torch.bfloat16)
    ref = a.double() @ w.double().T
    name = "gemm_tc_pair_kernel (split-K in a cluster)"

    def run(mode, dtype, glu=None, x0=None):
        out = torch.full((M, N), float("nan"), dtype=dtype, device=dev()) if x0 is None else x0.clone()
        before = ops.kernel_counts().get(name, 0)
        assert ops_tensor.gemm_bf16(a, w, out, mode, glu)
        assert ops.kernel_counts().get(name, 0) == before + 1
        return out

    if not gated:
        # float32 sums of K products of bfloat16 numbers, in the tensor core's and the sharers' order
        first = run(ops.GEMM_STORE_F32, torch.float32)
        assert rel_err(first, ref) < 2e-5 and torch.equal(run(ops.GEMM_STORE_F32, torch.float32), first)
        assert torch.equal(run(ops.GEMM_STORE, torch.bfloat16), first.to(torch.bfloat16))
        x0 = torch.randn(M, N, device=dev())
        assert rel_err(run(ops.GEMM_ACCUM_F32, torch.float32, None, x0), x0.double() + ref) < 2e-5
    else:
        g, u = ref[:, :N], ref[:, N:]
        bias = torch.randn(2 * N, device=dev()) * 0.3
        clamped = plain_rapovik.clamped_glu((g + bias[:N].double()).cpu(), (u + bias[N:].double()).cpu(), 1.3)
        # one rounding to bfloat16 (2^-9) of the largest results, and the activation's approximate exponential
        assert rel_err(run(ops.GEMM_SWIGLU, torch.bfloat16), g * torch.sigmoid(g) * u) < 1e-2
        assert rel_err(run(ops.GEMM_RELUGLU, torch.bfloat16), g.clamp_min(0) * u) < 1e-2
        assert rel_err(run(ops.GEMM_CLAMPGLU, torch.bfloat16, ops.GluParams(1.3, 1.702, bias)), clamped) < 1e-2
    assert ops_tensor.gemm_status(dev()) == 0
