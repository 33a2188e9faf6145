"""The rules by which the launchers choose grids, clusters and attributes, on the CPU: the kernels' objects linked with a runtime that
records launches (fake_cudart.cpp)."""
import ctypes
import os
import shutil
import subprocess
from types import SimpleNamespace

import pytest

from carbon_engine_b200.csrc import build

STORE, ACCUM, SWIGLU, CLAMPGLU = 0, 2, 3, 6
ADDR = 1 << 20                     # an aligned address that nothing reads


class Launch(ctypes.Structure):
    _fields_ = [("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("cluster", ctypes.c_uint * 3), ("smem", ctypes.c_uint),
                ("dependent", ctypes.c_uint), ("device", ctypes.c_int), ("kernel", ctypes.c_char * 256)]


@pytest.fixture(scope="module")
def linked(tmp_path_factory):
    try:
        nvcc = build._nvcc()
    except build.BuildError:
        pytest.skip("no CUDA toolkit")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    headers = build._sources(build.KERNEL_DIR, (".cuh", ".h"))
    names = ("errors", "tensor_map", "gemm_tc", "gemm_f32", "gemm_f32_stream", "gemm_plain", "attention_f32", "attention_mma")
    objects = build._compile_all(nvcc, build.NVCC_FLAGS, [os.path.join(build.KERNEL_DIR, n + ".cu") for n in names], headers, build.build_dir(), "k")
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    cxx = os.environ.get("CXX") or shutil.which("g++") or shutil.which("c++")
    source = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake_cudart.cpp")
    subprocess.run([cxx, "-shared", "-fPIC", "-std=c++17", "-I", cuda, source] + objects + ["-o", out], check=True)
    return out


class Chip:
    """A process's first look at a chip: every instance loads a copy of the library, with nothing kept from other instances."""

    count = 0

    def __init__(self, linked, room):
        Chip.count += 1
        copy = f"{linked}.{Chip.count}.so"
        shutil.copy(linked, copy)
        self.lib = ctypes.CDLL(copy, mode=os.RTLD_LOCAL | os.RTLD_NOW | getattr(os, "RTLD_DEEPBIND", 0))
        self.lib.ce_last_error.restype = ctypes.c_char_p
        for blocks, clusters in room.items():
            self.lib.fake_room(blocks, clusters)

    def _launched(self, code):
        assert code == 0, self.lib.ce_last_error().decode()
        seen = Launch()
        self.lib.fake_last(ctypes.byref(seen))
        return seen

    def gemm_tc(self, M, N, K, mode=STORE):
        p = ctypes.c_void_p(ADDR)
        return self._launched(self.lib.ce_gemm_tc(p, p, p, M, N, K, K, N, mode, p, ctypes.c_longlong(1 << 40), p, 1 << 20, p, None,
                                                  ctypes.c_float(0), ctypes.c_float(0), None))

    def gemm_f32(self, M, N, K, mode=STORE, weights_ready=1):
        p = ctypes.c_void_p(ADDR)
        return self._launched(self.lib.ce_gemm_plain(p, p, p, 0, M, N, K, K, N, mode, None, ctypes.c_float(0), ctypes.c_float(0), weights_ready, None))

    def stream(self, M, N, K, mode=STORE, lda=None, at=ADDR):
        """The product of a few tokens as a stream of weights; None where the launcher leaves it to the other kernel."""
        p, w = ctypes.c_void_p(at), ctypes.c_void_p(ADDR)
        before = self.lib.fake_launches()
        code = self.lib.ce_gemm_f32_stream(p, w, w, M, N, K, K if lda is None else lda, N, mode, None, ctypes.c_float(0), ctypes.c_float(0), 1, None)
        if code == 1:
            assert self.lib.fake_launches() == before
            return None
        return self._launched(code)

    def attention_f32(self, n_decode, n_tiles, heads=16, kv_heads=4, d=128, longest=4096):
        p = ctypes.c_void_p(ADDR)
        return self._launched(self.lib.ce_attention_f32(*[p] * 10, n_decode, n_tiles, heads, kv_heads, d, heads * d, 64, 100, 100, 0, longest,
                                                        ctypes.c_float(1), None))

    def decode(self, n, longest, heads=32, kv_heads=8, d=128, page=64, slopes=None):
        p = ctypes.c_void_p(ADDR)
        return self._launched(self.lib.ce_attention_decode_bf16_sink(
            *[p] * 6, 1 << 20, *[p] * 6, n, heads, kv_heads, d, (heads + 2 * kv_heads) * d, page, 200, 1000, 0, ctypes.c_float(1),
            (longest + 127) // 128, None, ctypes.c_float(1), slopes, None))


B200 = {2: 74, 3: 60, 4: 33, 5: 30, 6: 22, 7: 20, 8: 15}
OTHER = {2: 74, 4: 30, 6: 17, 8: 12}
# weight rows and K of this engine's products at several widths, gated ones among them
PRODUCTS = [(4096, 4096, STORE), (4096, 12288, ACCUM), (6144, 4096, STORE), (3072, 9728, ACCUM), (5120, 17408, ACCUM), (3840, 8192, STORE),
            (8448, 8192, STORE), (3328, 16384, ACCUM), (2048, 4096, SWIGLU), (1536, 8192, CLAMPGLU), (12288, 4096, SWIGLU)]


def parts(launch):
    assert b"gemm_tc_pair_kernel" in launch.kernel
    return launch.cluster[0] // 2


@pytest.mark.parametrize("N,K,mode", PRODUCTS)
def test_the_pairs_that_share_k_depend_on_the_weights_alone(linked, N, K, mode):
    """A token's sums are taken in the same order in every step of a band of tokens, on every chip, and in one piece beyond 512 tokens."""
    here, there = Chip(linked, B200), Chip(linked, OTHER)
    for band in ((129, 130, 160, 176, 203, 224, 255, 256), (257, 300, 336, 400, 448, 511, 512)):
        assert len({parts(chip.gemm_tc(M, N, K, mode)) for M in band for chip in (here, there)}) == 1
    assert all(parts(chip.gemm_tc(M, N, K, mode)) == 1 for M in (513, 600, 700, 1021, 4096) for chip in (here, there))


def test_products_with_few_tiles_share_k(linked):
    chip = Chip(linked, B200)
    assert [parts(chip.gemm_tc(200, N, K, mode)) for N, K, mode in PRODUCTS[:6]] == [2, 2, 1, 4, 3, 2]
    assert [parts(chip.gemm_tc(400, N, K, mode)) for N, K, mode in PRODUCTS[:6]] == [1, 2, 1, 2, 1, 2]


def test_the_numbers_of_sharers_that_the_kernel_tests_run(linked):
    from test_pair_tiles_gpu import SHARED
    chip = Chip(linked, B200)
    assert [parts(chip.gemm_tc(M, N, K, mode)) for M, N, K, gated, _ in SHARED for mode in ((SWIGLU, CLAMPGLU) if gated else (STORE, ACCUM))] == \
        [n for *_, n in SHARED for _ in range(2)]


@pytest.mark.parametrize("K,runs", [(700, 2), (800, 3), (1032, 4), (1300, 5), (1536, 6), (1800, 7), (2048, 8), (5000, 8)])
def test_float32_products_of_few_tiles_give_each_block_of_a_cluster_a_run_of_k(linked, K, runs):
    seen = Chip(linked, {n: 100 for n in range(2, 9)}).gemm_f32(33, 1024, K)
    assert seen.cluster[2] == seen.grid[2] == runs


@pytest.mark.parametrize("launch", [lambda c: c.gemm_f32(100, 4096, 4096), lambda c: c.attention_f32(0, 40), lambda c: c.gemm_tc(4, 4096, 4096),
                                    lambda c: c.gemm_tc(200, 4096, 4096), lambda c: c.gemm_tc(2048, 4096, 4096), lambda c: c.gemm_tc(2048, 128, 4096),
                                    lambda c: c.decode(64, 700), lambda c: c.decode(64, 300), lambda c: c.decode(64, 300, d=192), lambda c: c.decode(64, 300, d=256)],
                         ids=["float32 product", "float32 attention", "one-block product", "shared pairs", "pairs", "single CTAs", "decode attention, longest first",
                              "decode attention", "decode attention, heads of 192", "decode attention, heads of 256"])
def test_kernels_of_much_shared_memory_run_on_every_device_of_a_process(linked, launch):
    chip = Chip(linked, {1: 296, **B200})
    for device in (0, 1, 0, 70, 71):
        chip.lib.fake_device(device)
        seen = launch(chip)
        assert seen.device == device and seen.smem > 48 * 1024


@pytest.mark.parametrize("answer", [0, -1])                          # no room, and a question that fails
def test_a_chip_without_room_for_shared_k_is_asked_once_and_runs(linked, answer):
    chip = Chip(linked, {2: 4, 4: answer, 6: answer, 8: answer})
    assert parts(chip.gemm_tc(200, 4096, 4096)) == 1
    asked = chip.lib.fake_occupancy_calls()
    assert all(parts(chip.gemm_tc(M, N, 4096)) == 1 for M, N in ((200, 4096), (150, 4096), (250, 3840), (300, 4096)))
    assert chip.lib.fake_occupancy_calls() == asked


@pytest.mark.parametrize("room,overlaps", [(2000, True), (16, True), (15, False), (1, False)])
def test_more_clusters_than_the_chip_holds_stand_alone(linked, room, overlaps):
    """The float32 kernels: 16 tiles of 128 rows, 4 tokens x 4 KV heads."""
    chip = Chip(linked, {8: room})
    for seen in (chip.gemm_f32(4, 2048, 2048), chip.attention_f32(4, 0)):
        assert seen.cluster[2] == seen.grid[2] == 8 and bool(seen.dependent) == overlaps


# sequences, longest context, head size: 2 to 6 blocks a cluster; 8 KV heads
@pytest.mark.parametrize("n,longest,d,blocks", [(21, 9000, 128, 3), (16, 2304, 128, 2), (8, 2304, 64, 4), (1, 2304, 192, 6), (1, 2304, 256, 6)])
@pytest.mark.parametrize("spare", [0, -1])
@pytest.mark.parametrize("slopes", [None, ctypes.c_void_p(ADDR)])
def test_decode_attention_of_more_clusters_than_the_chip_holds_stands_alone(linked, n, longest, d, blocks, spare, slopes):
    seen = Chip(linked, {blocks: 8 * n + spare}).decode(n, longest, d=d, slopes=slopes)
    assert b"attention_decode_tma_kernel" in seen.kernel and seen.cluster[0] == blocks and seen.grid[0] == n * blocks
    assert bool(seen.dependent) == (spare == 0)


# tiles of a sequence, blocks, tiles a block of the longest context (33 tiles in four blocks: 10, 10, 10, 3, not 9, 9, 9, 6)
@pytest.mark.parametrize("tiles,blocks,longest,share", [(33, 4, 10, 10), (36, 4, 10, 10), (37, 4, 10, 10), (40, 4, 10, 10), (32, 4, 10, 8), (1, 4, 10, 1),
                                                        (141, 3, 54, 47), (144, 3, 54, 48), (145, 3, 54, 54), (8, 8, 1, 1), (9, 8, 2, 2), (8, 8, 2, 1), (41, 4, 10, 11), (33, 4, 0, 9), (1, 3, 0, 1)])
def test_a_sequences_tiles_are_dealt_evenly_unless_it_is_about_the_longest(linked, tiles, blocks, longest, share):
    assert Chip(linked, {}).lib.ce_attention_decode_share(tiles, blocks, longest) == share
    assert share * blocks >= tiles                                   # nothing is left out


# clusters at once of the B200 measured, heads of 128: sequences, longest context, room; 8 KV heads
@pytest.mark.parametrize("n,longest,d,room,ordered", [
    (21, 9000, 128, {3: 93}, True), (64, 700, 128, {1: 296}, True), (48, 700, 128, {1: 296}, True),
    (37, 700, 128, {1: 296}, False), (38, 700, 128, {1: 296}, True), (74, 700, 128, {1: 296}, True), (75, 700, 128, {1: 296}, False),      # one and two waves
    (64, 384, 128, {1: 296}, False), (64, 512, 128, {1: 296}, True), (100, 890, 64, {1: 592}, False), (100, 1000, 64, {1: 592}, True),   # work of a block
    (128, 2048, 64, {1: 592}, True), (129, 2048, 64, {1: 592}, False), (8, 2304, 128, {4: 71}, False)])
def test_decode_attention_takes_the_longest_first_in_grids_of_one_to_two_waves(linked, n, longest, d, room, ordered):
    seen = Chip(linked, room).decode(n, longest, d=d)
    assert (f"attention_decode_tma_kernelILi{d}ELi3ELb0ELb{int(ordered)}E".encode()) in seen.kernel


def test_decode_attention_of_one_block_a_sequence_overlaps(linked):
    seen = Chip(linked, {1: 1}).decode(64, 2304)
    assert seen.cluster[0] == 1 and seen.dependent


def test_heads_of_192_and_256_are_asked_for_apart(linked):
    chip = Chip(linked, {6: 100})
    for d in (192, 256, 192, 256):
        chip.decode(1, 2304, d=d)
    assert chip.lib.fake_occupancy_calls() == 2


def ring(rows, tokens, k):
    """Bytes of one stage: eight warps with the rows and tokens of a block."""
    return 8 * 4 * (rows + tokens) * k


# a block's rows, tokens (rounded up to 4 or 8), k and number of a ring's stages
@pytest.mark.parametrize("M,N,K,mode,rows,tokens,k,stages", [
    (1, 2048, 2048, STORE, 14, 4, 32, 8), (4, 2048, 6144, ACCUM, 14, 4, 32, 8), (8, 2048, 2048, STORE, 14, 8, 32, 6), (5, 2368, 2048, STORE, 16, 8, 32, 6),
    (4, 2516, 2560, STORE, 17, 4, 32, 7), (4, 2560, 9728, ACCUM, 18, 4, 32, 6), (8, 2560, 9728, ACCUM, 18, 8, 32, 5), (1, 3072, 2048, STORE, 21, 4, 32, 6),
    (4, 4096, 4096, ACCUM, 28, 4, 32, 4), (3, 5120, 5120, ACCUM, 35, 4, 32, 4), (4, 7104, 2048, STORE, 48, 4, 32, 3), (4, 7168, 5120, STORE, 49, 4, 16, 5),
    (4, 6144, 2048, SWIGLU, 84, 4, 16, 4), (8, 6144, 2048, SWIGLU, 84, 8, 16, 4), (8, 8140, 2048, SWIGLU, 110, 8, 16, 3), (2, 1184, 2304, CLAMPGLU, 16, 4, 32, 7)])
def test_a_streamed_products_ring_takes_all_stages_that_fit(linked, M, N, K, mode, rows, tokens, k, stages):
    seen = Chip(linked, {}).stream(M, N, K, mode)
    blocks = -(-N * (2 if mode >= SWIGLU else 1) // rows)
    assert b"gemm_f32_stream_kernel" in seen.kernel and seen.dependent and seen.grid[0] == blocks
    assert seen.smem == max(stages * ring(rows, tokens, k), 116 * 1024 if blocks < 148 else 0)


def test_streamed_products_fit_every_device(linked):
    """All numbers of rows: the opt-in on each device of a process, and no more shared memory than an SM has."""
    chip = Chip(linked, {})
    taken = set()
    for device, (M, mode) in enumerate([(4, STORE), (8, STORE), (4, SWIGLU), (8, CLAMPGLU), (1, ACCUM)]):
        chip.lib.fake_device(device)
        for rows in range(4, 140):
            seen = chip.stream(M, 148 * rows, 2048, mode)
            if seen:
                taken.add((M, mode, rows))
                assert seen.device == device and seen.grid[0] == 148 and seen.smem <= 200 * 1024
    assert max(r for M, mode, r in taken if (M, mode) == (4, STORE)) == 126 and max(r for M, mode, r in taken if (M, mode) == (8, CLAMPGLU)) == 61


@pytest.mark.parametrize("M,N,K,mode,lda,at", [
    (0, 2048, 2048, STORE, None, ADDR), (9, 2048, 2048, STORE, None, ADDR), (4, 591, 2048, STORE, None, ADDR), (4, 2048, 1792, STORE, None, ADDR),
    (4, 2048, 2080, STORE, None, ADDR), (4, 2048, 2048, STORE, 2050, ADDR), (4, 2048, 2048, STORE, None, ADDR + 4), (4, 2048, 2048, STORE, None, 0),
    (4, 2048, 2048, 7, None, ADDR), (4, 2048, 2048, -1, None, ADDR), (1, 151936, 2048, STORE, None, ADDR), (4, 9728, 2560, SWIGLU, None, ADDR),
    # 33 to 41 rows a block, where the tiles' clusters run side by side: gated ones, and more than 4 tokens beyond K = 2,048
    (4, 2960, 4096, SWIGLU, None, ADDR), (8, 5120, 5120, ACCUM, None, ADDR), (5, 6144, 4096, STORE, None, ADDR)])
def test_products_that_are_not_streamed(linked, M, N, K, mode, lda, at):
    assert Chip(linked, {}).stream(M, N, K, mode, lda, at) is None


def test_without_room_for_a_cluster_the_float32_kernels_run_without(linked):
    chip = Chip(linked, {8: 0})
    for seen in (chip.gemm_f32(4, 2048, 2048), chip.attention_f32(4, 0)):
        assert seen.cluster[2] == seen.grid[2] == 1 and seen.dependent


@pytest.mark.parametrize("launch", [lambda c: c.gemm_f32(100, 65536, 2048), lambda c: c.attention_f32(0, 64)])
def test_grids_without_clusters_overlap(linked, launch):
    seen = launch(Chip(linked, {8: 1}))
    assert seen.cluster[2] == 1 and seen.dependent


@pytest.mark.parametrize("past,clustered", [(0, False), (900, True)])
def test_a_long_decoding_request_leaves_a_short_prompt_its_plan(linked, monkeypatch, past, clustered):
    """150 tokens of a prompt after `past`, beside a request that decodes at 5,000."""
    import torch
    from carbon_engine_b200 import ops, ops_tensor
    from carbon_engine_b200.parts.attention import PagedAttention
    monkeypatch.setattr(ops_tensor, "decode_split", lambda: 128)
    sections, asked = {}, []
    bufs = SimpleNamespace(host_section=lambda name: sections.setdefault(name, [0] * 64), dev_section=lambda name: sections[name])
    ctx = SimpleNamespace(bufs=bufs, B=2, n_decode=1, h_q_start=[0, 1, 151], h_ctx_before=[5000, past], max_ctx=5001, plans={},
                          positions=None, seq_slot=None, q_start=None, status=None)
    mixer = PagedAttention(2048, 16, 4, 128, "m")
    ctx.plans[mixer.plan_key] = mixer.plan_step(ctx)
    monkeypatch.setattr(ops, "attention_f32", lambda *args: asked.append(args) or True)
    mixer.attend(ctx, torch.empty(151, 3072), None, SimpleNamespace(k_pool=None, v_pool=None, page_size=64), None)
    (*_, n_decode, n_tiles, nh, nkv, d, page_size, window, longest, scale), = asked
    assert (n_decode, n_tiles, window) == (1, 3, 0)
    seen = Chip(linked, {8: 1000}).attention_f32(0, n_tiles, longest=longest)
    assert (seen.cluster[2] == 8) == clustered
