"""The rotation's warp kernel (head sizes 64 to 256, full rotation in half pairs): the order of its sums, and its walk over a token's heads."""
import pytest
import torch

from test_kernels_gpu import DTYPES, dev, paged_layout, status, step_meta

pytestmark = pytest.mark.gpu
NAME = "qk_rope_kvwrite_warp_kernel"
EPS = 1e-5


def add_square(sums, x):
    """fma(x, x, sums) of float32 values."""
    return (x.double() * x.double() + sums.double()).float()


def rms_norm(x, weight):
    """The norm as a warp of 32 lanes takes it that hold d / 64 elements of each half: bit for bit."""
    x = x.float()
    d = x.shape[-1]
    halves = x.reshape(*x.shape[:-1], 2, 32, d // 64)
    sums = torch.zeros(halves.shape[:-3] + (32,), device=x.device)
    for h in range(2):
        for i in range(d // 64):
            sums = add_square(sums, halves[..., h, :, i])
    lane = torch.arange(32, device=x.device)
    for o in (16, 8, 4, 2, 1):
        sums = sums + sums[..., lane ^ o]
    mean = (sums[..., :1].double() * torch.tensor(1.0 / d, dtype=torch.float32).item() + torch.tensor(EPS, dtype=torch.float32).item()).float()
    return x * torch.rsqrt(mean) * weight


def pool_rows(pool, table, positions, page_size):
    """[T, nkv, d]: where the tokens of sequence 0 lie."""
    pos = positions.long()
    return pool[table[0].long()[pos // page_size], :, pos % page_size, :]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,d", [(5, 3, 64), (6, 2, 128), (7, 1, 192), (5, 2, 256)])
@pytest.mark.parametrize("T", [3, 260])
def test_the_norm_keeps_the_order_of_its_sums(dtype, nh, nkv, d, T):
    from carbon_engine_b200 import ops
    torch.manual_seed(d + T)
    table, kp, vp = paged_layout([T], 16, nkv, d, dtype)
    qkv = (torch.randn(T, (nh + 2 * nkv) * d, device=dev()) * 3).to(dtype)
    qw, kw = 1 + 0.2 * torch.randn(d, device=dev()), 1 + 0.2 * torch.randn(d, device=dev())
    positions, sot, slots = step_meta([(0, T)])
    heads = qkv.view(T, nh + 2 * nkv, d).clone()
    before, st = ops.kernel_counts().get(NAME, 0), status()
    ops.qk_rope_kvwrite(qkv, kp, vp, qw, kw, None, None, positions, sot, slots, table, st, nh, nkv, d, 0, 16, EPS)
    assert ops.kernel_counts().get(NAME, 0) == before + 1 and st.item() == 0
    assert torch.equal(qkv.view(T, nh + 2 * nkv, d)[:, :nh], rms_norm(heads[:, :nh], qw).to(dtype))
    assert torch.equal(pool_rows(kp, table, positions, 16), rms_norm(heads[:, nh:nh + nkv], kw).to(dtype))
    assert torch.equal(pool_rows(vp, table, positions, 16), heads[:, nh + nkv:])


@pytest.mark.parametrize("d", [64, 128, 192, 256])
def test_norm_weights_that_the_kernel_in_front_makes(d):
    """With dependent launches on: the product in front takes some 100 us, the rotation must not read its weights before it ends."""
    from carbon_engine_b200 import ops
    torch.manual_seed(d)
    nh, nkv, T = 4, 2, 3
    a, b = torch.randn(1024, 4096, device=dev()), torch.randn(512, 4096, device=dev())
    made = torch.empty(1024, 512, device=dev())
    table, kp, vp = paged_layout([T], 16, nkv, d, torch.float32)
    source = torch.randn(T, (nh + 2 * nkv) * d, device=dev())
    positions, sot, slots = step_meta([(0, T)])
    st = status()

    def rotate(qkv):
        ops.qk_rope_kvwrite(qkv, kp, vp, made[1023, :d], made[1023, d:2 * d], None, None, positions, sot, slots, table, st, nh, nkv, d, 0, 16, EPS)

    ops.set_dependent_launches(True)
    ops.gemm_plain(a, b, made, ops.GEMM_STORE)
    torch.cuda.synchronize()
    want = source.clone()
    rotate(want)
    want_k = pool_rows(kp, table, positions, 16).clone()
    for _ in range(5):
        made.zero_()
        got = source.clone()
        torch.cuda.synchronize()
        ops.gemm_plain(a, b, made, ops.GEMM_STORE)
        rotate(got)                                                # (nothing between the two launches)
        assert torch.equal(got, want) and torch.equal(pool_rows(kp, table, positions, 16), want_k)


def shifted(t, by):
    """The same values from `by` bytes behind a 16-byte boundary on."""
    room = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)
    room = room[by // t.element_size():][:t.numel()].view(t.shape)
    room.copy_(t)
    assert room.data_ptr() % 16 == by % 16
    return room


# the smallest accesses: d / 64 elements, single elements of heads of 192 (bfloat16: 2, 4, 2, 8 bytes; float32: 4, 8, 4, 16)
@pytest.mark.parametrize("dtype,nh,nkv,d,by", [(torch.bfloat16, 4, 2, 64, 2), (torch.bfloat16, 5, 1, 128, 4), (torch.bfloat16, 3, 2, 192, 2),
                                              (torch.bfloat16, 4, 2, 256, 8), (torch.float32, 4, 2, 64, 4), (torch.float32, 5, 1, 128, 8),
                                              (torch.float32, 3, 2, 192, 4)])
@pytest.mark.parametrize("which", ["qkv", "pools", "floats", "all"])
@pytest.mark.parametrize("T", [5, 260])
def test_operands_between_16_byte_boundaries(dtype, nh, nkv, d, by, which, T):
    """The same kernel and the same bits as with operands that start on 16 bytes."""
    from carbon_engine_b200 import ops
    torch.manual_seed(d + T)
    table, kp, vp = paged_layout([T], 16, nkv, d, dtype)
    qkv = torch.randn(T, (nh + 2 * nkv) * d, device=dev()).to(dtype)
    qw, kw = 1 + 0.2 * torch.randn(d, device=dev()), 1 + 0.2 * torch.randn(d, device=dev())
    angles = torch.rand(T, d // 2, device=dev())
    positions, sot, slots = step_meta([(0, T)])
    floats_by = {64: 4, 128: 8, 192: 4, 256: 0}[d]

    def rotate(move):
        row = lambda t, name: shifted(t, by if move in (name, "all") else 0)
        vec = lambda t: shifted(t, floats_by if move in ("floats", "all") else 0)
        x, k, v = row(qkv, "qkv"), row(kp, "pools"), row(vp, "pools")
        before, st = ops.kernel_counts().get(NAME, 0), status()
        ops.qk_rope_kvwrite(x, k, v, vec(qw), vec(kw), vec(angles.cos()), vec(angles.sin()), positions, sot, slots, table, st, nh, nkv, d, d, 16, EPS)
        assert ops.kernel_counts().get(NAME, 0) == before + 1 and st.item() == 0
        return x, pool_rows(k, table, positions, 16), pool_rows(v, table, positions, 16)

    for got, want in zip(rotate(which), rotate(None)):
        assert torch.equal(got, want)


# more heads than a warp takes at once, not a multiple of them: a warp's heads change from query to key to value on the way
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,d", [(70, 3, 64), (19, 3, 128), (19, 3, 192), (19, 3, 256)])
def test_a_heads_bits_do_not_depend_on_the_steps_tokens(dtype, nh, nkv, d):
    """Steps of fewer than 64, of fewer than 256 and of more tokens walk over a token's heads in different portions."""
    from carbon_engine_b200 import ops
    torch.manual_seed(d)
    T, ps = 400, 16
    table, kp, vp = paged_layout([T], ps, nkv, d, dtype)
    qkv = torch.randn(T, (nh + 2 * nkv) * d, device=dev()).to(dtype)
    qw, kw = 1 + 0.2 * torch.randn(d, device=dev()), 1 + 0.2 * torch.randn(d, device=dev())
    angles = torch.rand(T, d // 2, device=dev()) * 6
    cos, sin, st = angles.cos(), angles.sin(), status()

    def steps(cuts):
        k, v, rows, start = kp.clone(), vp.clone(), [], 0
        for n in cuts:
            positions, sot, slots = step_meta([(start, n)])
            x = qkv[start:start + n].clone()
            ops.qk_rope_kvwrite(x, k, v, qw, kw, cos, sin, positions, sot, slots, table, st, nh, nkv, d, d, ps, EPS)
            rows.append(x[:, :nh * d])
            start += n
        assert start == T and st.item() == 0
        return torch.cat(rows), k, v

    whole = steps([400])
    assert int((~torch.isnan(whole[1].float())).sum()) == T * nkv * d
    for cuts in ([255, 63, 64, 1, 17], [256, 144]):
        for got, want in zip(steps(cuts), whole):
            assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(want))
    # a layer that reads another's cache: queries alone
    x = qkv[:300].clone()
    ops.qk_rope_kvwrite(x, None, None, qw, kw, cos, sin, step_meta([(0, 300)])[0], None, None, None, st, nh, nkv, d, d, ps, EPS, write_kv=False)
    assert st.item() == 0 and torch.equal(x[:, :nh * d], whole[0][:300]) and torch.equal(x[:, nh * d:], qkv[:300, nh * d:])
