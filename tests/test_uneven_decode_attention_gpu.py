"""Decode attention over sequences of unequal lengths: clusters take the longest first and a sequence's blocks share its own tiles."""
import math

import pytest
import torch

from test_kernels_gpu import dev, rel_err, run_mma_attention

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
