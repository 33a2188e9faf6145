"""The float32 path's product and attention at the edges of their tiles, runs and chunks, against float64, and bit for bit over the
ways a step can be cut."""
import math

import pytest
import torch

import plain_qwen3 as plain
from test_kernels_gpu import dev, fill_pools, paged_layout, status, step_meta

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def product(a, w, mode, out=None):
    from carbon_engine_b200 import ops
    n = w.shape[0] // 2 if mode in ops.GEMM_GATED else w.shape[0]
    out = torch.zeros(a.shape[0], n, device=dev()) if out is None else out
    ops.gemm_plain(a, w, out, mode)
    return out


# K: below one run, one run exactly, runs with a short last one, every number of runs from one to eight (clusters of that size);
# K = 301, 1031, 1307 and 1801 are not whole vectors
@pytest.mark.parametrize("N,K", [(7, 5), (129, 32), (64, 301), (130, 512), (70, 772), (257, 1032), (66, 1031), (130, 1284), (40, 1307),
                                 (66, 1536), (200, 1801), (200, 2100)])
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


# the second size has tiles enough for one block a tile from 1 token on, the others only with many tokens
@pytest.mark.parametrize("N,K", [(1024, 2048), (38000, 520), (1024, 800), (1024, 1300), (1024, 1536), (1024, 1800)])
def test_float32_product_has_the_same_bits_in_every_tile_and_cluster(N, K):
    from carbon_engine_b200 import ops
    torch.manual_seed(1)
    a, w = torch.randn(2600 if N < 2000 else 70, K, device=dev()), torch.randn(N, K, device=dev())
    whole = product(a, w, ops.GEMM_STORE)
    for lo, n in ((0, 1), (3, 4), (1, 7), (30, 33), (2, 64), (5, 65)):
        assert torch.equal(product(a[lo:lo + n], w, ops.GEMM_STORE), whole[lo:lo + n]), n


@pytest.mark.parametrize("M", [3, 40, 100])
def test_float32_product_reads_a_matrix_that_the_kernel_in_front_makes(M):
    """The second product's W is the first one's result, with dependent launches on: the first takes some 100 us, the second must not
    begin to read before it ends."""
    from carbon_engine_b200 import ops
    torch.manual_seed(5)
    a, b, x = torch.randn(1024, 4096, device=dev()), torch.randn(512, 4096, device=dev()), torch.randn(M, 512, device=dev())
    made = torch.zeros(1024, 512, device=dev())
    ops.set_dependent_launches(True)
    ops.gemm_plain(a, b, made, ops.GEMM_STORE)
    torch.cuda.synchronize()
    want, got = product(x, made, ops.GEMM_STORE), torch.empty(M, 1024, device=dev())
    for _ in range(5):
        made.zero_()
        torch.cuda.synchronize()
        ops.gemm_plain(a, b, made, ops.GEMM_STORE)
        ops.gemm_plain(x, made, got, ops.GEMM_STORE)               # (nothing between the two launches)
        assert torch.equal(got, want)


@pytest.mark.parametrize("M", [3, 8])
def test_float32_stream_product_reads_a_matrix_that_the_kernel_in_front_makes(M):
    """The same at sizes of the kernel that streams weights for up to 8 tokens; the product in front takes some 350 us."""
    from carbon_engine_b200 import ops
    torch.manual_seed(5)
    a, b, x = torch.randn(1024, 2304, device=dev()), torch.randn(2048, 2304, device=dev()), torch.randn(M, 2048, device=dev())
    made = torch.zeros(1024, 2048, device=dev())
    ops.set_dependent_launches(True)
    ops.gemm_plain(a, b, made, ops.GEMM_STORE)
    torch.cuda.synchronize()
    want, got = product(x, made, ops.GEMM_STORE), torch.empty(M, 1024, device=dev())
    for _ in range(5):
        made.zero_()
        torch.cuda.synchronize()
        before = ops.kernel_counts().get("gemm_f32_stream_kernel", 0)
        ops.gemm_plain(a, b, made, ops.GEMM_STORE)
        ops.gemm_plain(x, made, got, ops.GEMM_STORE)               # (nothing between the two launches)
        assert ops.kernel_counts().get("gemm_f32_stream_kernel", 0) == before + 1
        assert torch.equal(got, want)


def attention(seqs, q, kp, vp, table, nh, nkv, d, ps, window, stride):
    from carbon_engine_b200 import ops
    T = sum(n for _, n in seqs)
    positions, _, slots = step_meta(seqs)
    starts = [0]
    for _, n in seqs:
        starts.append(starts[-1] + n)
    n_decode = next((b for b, (_, n) in enumerate(seqs) if n > 1), len(seqs))
    tiles = [(b, t) for b, (_, n) in enumerate(seqs) if b >= n_decode for t in range(0, n, 64)]
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev())
    out, st = torch.full((T, nh * d), 7.0, device=dev()), status()
    assert ops.attention_f32(q, stride, kp, vp, out, positions, slots, ints(starts), table, ints(tiles or [(0, 0)]), st, n_decode, len(tiles),
                             nh, nkv, d, ps, window, max(c + n for c, n in seqs), 1 / math.sqrt(d))
    return out, int(st.item())


# groups of 1, 2, 3, 8, 9 and 20 heads; head sizes below, at and above a column round; pages smaller and larger than a chunk; windows
# that start inside a chunk
@pytest.mark.parametrize("nh,nkv,d,ps,window", [(2, 2, 16, 16, 0), (6, 3, 20, 5, 0), (3, 1, 64, 64, 0), (8, 1, 68, 8, 70), (18, 2, 128, 128, 0),
                                                 (20, 1, 100, 7, 130)])
def test_float32_attention_against_float64(nh, nkv, d, ps, window):
    torch.manual_seed(2)
    seqs = [(0, 1), (63, 1), (64, 1), (700, 1), (0, 2), (61, 7), (0, 64), (0, 65), (600, 130)]
    table, kp, vp = paged_layout([c + n for c, n in seqs], ps, nkv, d, torch.float32, shuffle_seed=3)
    T = sum(n for _, n in seqs)
    stride = (nh + 2 * nkv) * d
    q, want, t = torch.full((T, stride), float("nan"), device=dev()), [], 0
    for b, (ctx, n) in enumerate(seqs):
        q_all, k_all, v_all = torch.randn(ctx + n, nh, d) * 1.5, torch.randn(ctx + n, nkv, d) * 1.5, torch.randn(ctx + n, nkv, d)
        fill_pools(kp, vp, table.cpu().numpy(), b, k_all.to(dev()), v_all.to(dev()), ps)
        q[t:t + n, :nh * d] = q_all[ctx:].reshape(n, nh * d).to(dev())
        want.append(plain.causal_attention(q_all.double(), k_all.double(), v_all.double(), 1 / math.sqrt(d), window)[ctx:])
        t += n
    out, st = attention(seqs, q, kp, vp, table, nh, nkv, d, ps, window, stride)
    want = torch.cat(want)
    # scores of size |q| |k| / sqrt(d) ~ 2 sqrt(d) carry d / 2 roundings each; their error is the probabilities' relative error
    assert st == 0 and float((out.view(T, nh, d).double().cpu() - want).abs().max()) < 2e-5 * float(want.abs().max())


@pytest.mark.parametrize("nh,nkv,d,ps,window", [(16, 4, 128, 64, 0), (5, 1, 24, 16, 100)])
def test_float32_attention_has_the_same_bits_however_the_step_is_cut(nh, nkv, d, ps, window):
    """The last token's neighbours hold values no one before it may meet: a row of infinities at the last position."""
    torch.manual_seed(3)
    L = 777
    table, kp, vp = paged_layout([L], ps, nkv, d, torch.float32, shuffle_seed=1)
    k, v = torch.randn(L, nkv, d, device=dev()), torch.randn(L, nkv, d, device=dev())
    v[L - 1] = float("inf")
    fill_pools(kp, vp, table.cpu().numpy(), 0, k, v, ps)
    q = torch.randn(L, nh * d, device=dev())
    whole, st = attention([(0, L)], q, kp, vp, table, nh, nkv, d, ps, window, nh * d)
    assert st == 0 and torch.isfinite(whole[:L - 1]).all()
    for past, n in ((0, 5), (130, 500), (699, 1), (64, 1), (63, 2), (500, 277), (0, 1), (775, 1)):
        got, st = attention([(past, n)], q[past:past + n].contiguous(), kp, vp, table, nh, nkv, d, ps, window, nh * d)
        end = min(n, L - 1 - past)
        assert st == 0 and torch.equal(got[:end], whole[past:past + end]), (past, n)


def test_float32_attention_flags_a_page_the_request_does_not_hold():
    table, kp, vp = paged_layout([200], 16, 1, 16, torch.float32)
    fill_pools(kp, vp, table.cpu().numpy(), 0, torch.randn(200, 1, 16, device=dev()), torch.randn(200, 1, 16, device=dev()), 16)
    table = table.clone()
    table[0, 5] = -1
    out, st = attention([(199, 1)], torch.randn(1, 16, device=dev()), kp, vp, table, 1, 1, 16, 16, 0, 16)
    assert st == 4 and torch.isfinite(out).all()


@pytest.mark.parametrize("seqs", [[(30, 1), (0, 1)], [(0, 40), (7, 30)]])
def test_float32_attention_of_scores_that_are_all_minus_infinity_is_not_a_number(seqs):
    """Products of finite numbers can overflow.  One row whose scores all do, among rows whose scores do not, alone and in a tile."""
    from carbon_engine_b200 import ops
    torch.manual_seed(4)
    table, kp, vp = paged_layout([c + n for c, n in seqs], 16, 1, 16, torch.float32)
    for b, (c, n) in enumerate(seqs):
        fill_pools(kp, vp, table.cpu().numpy(), b, torch.full((c + n, 1, 16), 1e20, device=dev()), torch.randn(c + n, 1, 16, device=dev()), 16)
    q = torch.randn(sum(n for _, n in seqs), 2 * 16, device=dev()) * 1e-20
    q[0, 16:] = -1e20
    got, st = attention(seqs, q, kp, vp, table, 2, 1, 16, 16, 0, 32)
    positions, seq_of_token, slots = step_meta(seqs)
    want = torch.empty_like(got)
    ops.attention_generic(q, 32, kp, vp, want, positions, seq_of_token, slots, table, status(), 2, 1, 16, 16, 0, 0.25)
    assert st == 0 and torch.equal(got.isnan(), want.isnan())
    assert got[0, 16:].isnan().all() and not got[1:].isnan().any() and not got[0, :16].isnan().any()
