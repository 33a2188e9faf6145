"""Decode attention over sequences of unequal lengths: clusters take the longest first and a sequence's blocks share its own tiles."""
import math

import pytest
import torch

from test_kernels_gpu import FakeCache, FakeCtx, dev, paged_layout, rel_err, run_mma_attention

pytestmark = pytest.mark.gpu
NAME = "attention_decode_tma_kernel (merge in the cluster)"

# contexts at the edges of a tile of 64, fewer tiles than blocks, equal ones, one long
LENGTHS = [1, 64, 63, 65, 700, 128, 2900, 129, 700, 1, 191, 193, 1500, 64, 300, 450, 2, 1023, 1025, 640]


# 20 sequences share a sequence's tiles over several blocks; 128 are the most whose order is taken, 130 keep the batch's
@pytest.mark.parametrize("n,nh,nkv,d,ps,window", [(20, 8, 2, 128, 64, 0), (20, 4, 1, 64, 16, 200), (20, 6, 2, 192, 8, 0), (128, 2, 1, 64, 16, 0),
                                                  (130, 2, 1, 64, 16, 0), (2, 32, 8, 128, 64, 0)])
def test_sequences_of_unequal_lengths_in_any_order(n, nh, nkv, d, ps, window):
    from carbon_engine_b200 import ops
    lens = [LENGTHS[(7 * i) % 20] + i // 20 for i in range(n)]
    before = ops.kernel_counts().get(NAME, 0)
    got, want = run_mma_attention([(L - 1, 1) for L in lens], nh, nkv, d, ps, window, 1 / math.sqrt(d), seed=3)
    assert ops.kernel_counts().get(NAME, 0) == before + 1
    for i in range(n):
        assert rel_err(got[i], want[i]) < 2e-2, (i, lens[i])
    # the same sequences in another order: the longest is the same, so every sequence is cut as before and has the same bits
    order = sorted(range(n), key=lambda i: (i * 13) % n)
    again, _ = run_mma_attention([(lens[i] - 1, 1) for i in order], nh, nkv, d, ps, window, 1 / math.sqrt(d), seed=3)
    for at, i in enumerate(order):
        assert torch.equal(again[at], got[i]), (i, lens[i])


def decode(lens, nh, nkv, d, ps, window, scale, sinks, out_scale, slopes, seed):
    """(got, want) [sequences, nh, d] of one token each after lens[i] - 1 cached ones; a sequence's numbers depend on its length."""
    from carbon_engine_b200 import ops_tensor
    table, kp, vp = paged_layout(lens, ps, nkv, d, torch.bfloat16)
    ctx = FakeCtx([(L - 1, 1) for L in lens])
    q_step = torch.zeros(len(lens), (nh + 2 * nkv) * d, dtype=torch.bfloat16, device=dev())
    want = torch.empty(len(lens), nh, d, dtype=torch.float64, device=dev())
    for i, L in enumerate(lens):
        gen = torch.Generator(device=dev()).manual_seed(seed * 10007 + L)
        rows = lambda *shape: torch.randn(*shape, device=dev(), generator=gen).to(torch.bfloat16)
        q, k, v = rows(nh, d), rows(L, nkv, d), rows(L, nkv, d)
        at = torch.arange(L, device=dev())
        kp[table[i].long()[at // ps], :, at % ps] = k
        vp[table[i].long()[at // ps], :, at % ps] = v
        q_step[i, :nh * d] = q.reshape(-1)
        k, v = k.double().repeat_interleave(nh // nkv, 1), v.double().repeat_interleave(nh // nkv, 1)
        s = torch.einsum("hd,lhd->hl", q.double(), k) * scale
        if slopes is not None:
            s = s - slopes.double()[:, None] * (L - 1 - at)
        if window:
            s = s.masked_fill(L - 1 - at >= window, float("-inf"))
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None]], 1)
        p = torch.softmax(s, 1)[:, :L]
        want[i] = torch.einsum("hl,lhd->hd", p, v) * out_scale
    out = torch.full((len(lens), nh * d), float("nan"), dtype=torch.bfloat16, device=dev())
    assert ops_tensor.attention_bf16(ctx, ctx, q_step, out, FakeCache(kp, vp, ps), table, nh, nkv, d, window, scale, sinks, out_scale, slopes)
    assert ctx.status.item() == 0
    return out.view(len(lens), nh, d), want


# 20 and 12 heads a KV head are three and two groups of at most eight, each with an order of its own
@pytest.mark.parametrize("n,nh,nkv,d,ps,window", [(20, 20, 1, 128, 64, 0), (9, 24, 2, 64, 16, 0), (20, 20, 1, 64, 16, 200), (5, 12, 1, 256, 8, 0)])
def test_many_heads_a_group_with_sinks_and_a_penalty_on_distance(n, nh, nkv, d, ps, window):
    from carbon_engine_b200 import ops
    lens = [LENGTHS[(7 * i) % 20] for i in range(n)]
    torch.manual_seed(n)
    sinks, slopes = torch.randn(nh, device=dev()) + 1.0, torch.rand(nh, device=dev()) * 0.01
    before = ops.kernel_counts().get(NAME, 0)
    got, want = decode(lens, nh, nkv, d, ps, window, 1 / math.sqrt(d), sinks, 0.8, slopes, 3)
    assert ops.kernel_counts().get(NAME, 0) == before + 1
    for i in range(n):
        assert rel_err(got[i], want[i]) < 2e-2, (i, lens[i])
    order = sorted(range(n), key=lambda i: (i * 7) % n)
    again, _ = decode([lens[i] for i in order], nh, nkv, d, ps, window, 1 / math.sqrt(d), sinks, 0.8, slopes, 3)
    for at, i in enumerate(order):
        assert torch.equal(again[at], got[i]), (i, lens[i])


# Grids of one to two waves, whose clusters take the longest sequences first (of one, three and two blocks), and one of one wave: unequal
# contexts, and contexts that are about the same, where the batch's order stays
@pytest.mark.parametrize("n,nh,nkv,d,longest", [(64, 8, 8, 128, 700), (21, 8, 8, 128, 9000), (100, 8, 8, 64, 1200), (48, 8, 8, 64, 4000), (30, 8, 8, 256, 300),
                                                (128, 16, 8, 64, 1030), (5, 40, 10, 192, 6000)])
@pytest.mark.parametrize("spread", [0.95, 0.1])
def test_the_longest_first(n, nh, nkv, d, longest, spread):
    lens = [max(1, round(longest * (1 - spread * ((i * 37) % n) / n))) for i in range(n)]
    got, want = decode(lens, nh, nkv, d, 16, 0, 1 / math.sqrt(d), None, 1.0, None, 5)
    for i in range(n):
        assert rel_err(got[i], want[i]) < 2e-2, (i, lens[i])
    order = sorted(range(n), key=lambda i: (i * 11) % n)
    again, _ = decode([lens[i] for i in order], nh, nkv, d, 16, 0, 1 / math.sqrt(d), None, 1.0, None, 5)
    assert torch.equal(again, got[order])
