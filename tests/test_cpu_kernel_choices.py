"""Host-side choices the kernel library makes, asked without a GPU: into how many parts the keys of a
decode are cut and when those parts merge on chip, which sizes each kernel says it takes, and which
requests are refused with a message.  The library is built by nvcc where it is missing (no device is
needed to build or to load it); without nvcc these tests are skipped."""
import shutil

import pytest

if shutil.which("nvcc") is None:
    pytest.skip("nvcc is not installed here", allow_module_level=True)


@pytest.fixture(scope="module")
def lib():
    from rbitnet_b200.kernels.lib import load
    return load(verbose=False)


@pytest.mark.parametrize("D", [64, 128])
def test_parts_of_a_decode(lib, D):
    parts, on_chip = lib.raw("rb_attention_decode_tma_parts"), lib.raw("rb_attention_decode_tma_on_chip")
    for pairs in (1, 7, 8, 32, 64, 100, 256, 300, 512, 600, 1024, 5000):
        for tiles in (1, 2, 3, 5, 16, 33, 128):
            s = parts(pairs, tiles, D)
            assert 1 <= s <= min(16, tiles), (pairs, tiles, s)          # no part without a tile to start from
            if on_chip(pairs, s, D):
                assert s in (2, 4, 8, 16)                               # cluster sizes
        assert parts(pairs, 1, D) == 1
    # a small batch is cut as far as its context allows, and merges on chip (up to 8 parts on any device)
    assert parts(8, 4, D) == 4 and on_chip(8, 4, D)
    assert parts(64, 32, 128) == 4 and on_chip(64, 4, 128)
    assert parts(0, 5, D) == 1 and parts(5, 0, D) == 1
    # more CTAs fit an SM at head size 64, so more pairs still count as a small grid
    assert parts(256, 32, 64) == 2 and parts(256, 32, 128) == 1
    assert not on_chip(600, 4, D)


def test_sizes_the_kernels_take(lib):
    assert lib.raw("rb_attention_decode_tma_supports")(32, 8, 128, 64)
    assert not lib.raw("rb_attention_decode_tma_supports")(32, 8, 96, 64)      # head size
    assert not lib.raw("rb_attention_decode_tma_supports")(32, 8, 128, 16)     # pages of 16 positions
    assert not lib.raw("rb_attention_decode_tma_supports")(34, 2, 128, 64)     # 17 query heads a group
    assert lib.raw("rb_attention_prefill_tc_supports")(32, 8, 64, 128, 0)
    assert not lib.raw("rb_attention_prefill_tc_supports")(7, 2, 128, 64, 0)      # heads that are no multiple of the groups
    for D in (64, 128, 192, 256):                                              # keys and values that are the same rows
        assert lib.raw("rb_attention_prefill_tc_supports")(32, 1, D, 64, 1)
        assert bool(lib.raw("rb_attention_prefill_tc_supports")(32, 1, D, 64, 0)) == (D <= 128)
    assert not lib.raw("rb_attention_prefill_tc_supports")(129, 1, 128, 64, 1)    # more heads than a tile has rows
    parts = lib.raw("rb_attention_prefill_tc_parts")
    for row_tiles in (1, 8, 100, 1000):
        for context in (1, 128, 129, 2048, 100000):
            n = parts(row_tiles, 1, context)
            assert 1 <= n <= 16 and n <= -(-context // 128)                     # no part without a tile of keys to start from
    assert parts(1, 1, 2048) == 16 and parts(1000, 1, 2048) == 1 and parts(8, 1, 128) == 1
    assert lib.raw("rb_attention_tiled_supports")(6, 2, 96, 64, 1)
    assert not lib.raw("rb_attention_tiled_supports")(6, 2, 100, 64, 1)
    assert lib.raw("rb_gemm_tc_qkv_supports")(8, 128, 4)
    assert not lib.raw("rb_gemm_tc_qkv_supports")(8, 128, 1)                   # K has to be split
    assert not lib.raw("rb_gemm_tc_qkv_supports")(17, 128, 4)                  # few tokens only
    assert not lib.raw("rb_gemm_tc_qkv_supports")(8, 96, 4)                    # a head may not straddle two tiles


def test_requests_are_refused_with_a_message(lib):
    from rbitnet_b200.kernels.lib import KernelError
    with pytest.raises(KernelError, match="multiple of 8"):
        lib.call("rb_gemm_tc", 0, 50, 1, 0, 77, 9, 0, 77, 50, 50, 77, 0, 0, 1, 0, 1.0, 0)
    with pytest.raises(KernelError, match="rows in blocks of 32"):
        lib.call("rb_gemm_tc", 0, 64, 1, 0, 64, 8, 0, 64, 48, 48, 128, 3, 24, 1, 0, 1.0, 0)
    with pytest.raises(KernelError, match="at most 8 splits"):
        lib.call("rb_gemm_tc", 0, 64, 1, 0, 1024, 8, 0, 1024, 64, 64, 1024, 0, 0, 9, 0, 1.0, 0)
    with pytest.raises(KernelError, match="head_dim"):
        lib.call("rb_rotate_append", 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 1, 64, 1, 2, 1, 7, 1, 7, 0, 0)


def test_parts_of_a_product_and_of_the_plain_decode(lib):
    """The choices follow the device's SM count (148 where no device answers, as here without a GPU)."""
    splits, parts = lib.raw("rb_gemm_tc_splits"), lib.raw("rb_attention_decode_parts")
    sms = lib.raw("rb_device_sm_count")()
    assert sms > 0
    assert splits(300, 4096, 4096) == 1                      # beyond 256 tokens K stays whole
    for T, N, K in [(1, 4096, 4096), (8, 6144, 4096), (8, 4096, 14336), (64, 128256, 4096), (16, 64, 64),
                    (200, 4096, 4096), (8, 256, 320)]:
        s = splits(T, N, K)
        blocks = -(-K // 64)
        assert s in range(1, 9) and (s - 1) * -(-blocks // s) < blocks, (T, N, K, s)     # no part is empty
        tiles = -(-N // 128) * -(-T // 64)
        assert s == 1 or tiles * 2 <= 2 * sms                # K is cut only while CTAs are fewer than places
    if sms == 148:
        assert splits(8, 4096, 4096) == 8 and splits(8, 6144, 4096) == 4 and splits(8, 128256, 4096) == 1
    for batch, kvh, ctx in [(1, 8, 2048), (8, 8, 2048), (64, 8, 8192), (3, 1, 10), (500, 8, 4096)]:
        s = parts(batch, kvh, ctx)
        assert 1 <= s <= min(16, max(1, -(-ctx // 64))), (batch, kvh, ctx, s)
    assert parts(1, 1, 64) == 1 and parts(0, 8, 100) == 1


def _plan(lib, T, N, K, sms=148, workspace=1, tile=0):
    import ctypes
    out = (ctypes.c_int * 4)()
    lib.call("rb_gemm_tc_plan", T, N, K, tile, sms, workspace, out, launches=0)
    return dict(tile=out[0], blocks_per_team=out[1], teams=out[2], token_tiles=out[3])


def test_plan_of_a_product_of_many_tokens(lib):
    """Tiles in turn, or (a product added to its output, on a device that has the counters: `workspace`)
    the k blocks of all weight tiles shared out evenly among teams of CTAs."""
    # 2,048 tokens, 4,096 rows: 256 tiles are 1.73 rounds of 148 SMs; 18 teams of 8 CTAs share 32 weight tiles
    p = _plan(lib, 2048, 4096, 14336)
    assert p["tile"] == 256 and p["token_tiles"] == 8 and p["teams"] == 18
    assert p["blocks_per_team"] * 18 >= 32 * 224 > p["blocks_per_team"] * 17 and p["blocks_per_team"] % 4 == 0
    # without the counters, and for few tokens, tiles are taken in turn
    assert _plan(lib, 2048, 4096, 14336, workspace=0)["blocks_per_team"] == 0
    assert _plan(lib, 64, 4096, 4096)["blocks_per_team"] == 0 and _plan(lib, 64, 4096, 4096)["tile"] == 64
    # tiles that fill whole rounds stay as they are: 37 weight tiles x 8 token tiles = 2 x 148
    assert _plan(lib, 2048, 37 * 128, 4096)["blocks_per_team"] == 0
    # few tiles and a long inner dimension: every SM gets a share of some tile's inner dimension
    p = _plan(lib, 300, 4096, 14336)
    assert p["tile"] == 160 and p["token_tiles"] == 2 and p["teams"] > 64 and p["blocks_per_team"] > 0
    # the parts of a tile are added one after the other: not worth it where the products are short
    assert _plan(lib, 2048, 4096, 4096)["blocks_per_team"] == 0
    # every part is at least one block, and the teams cover everything, at any size
    for T in (129, 257, 300, 1000, 2048, 4097, 9000):
        for N in (128, 130, 4096, 6144, 28672, 128256):
            for K in (64, 72, 4096, 14336):
                for sms in (148, 132, 16):
                    p = _plan(lib, T, N, K, sms=sms)
                    w_tiles, blocks = -(-N // 128), -(-K // 64)
                    assert p["tile"] in (128, 160, 192, 224, 256) and p["token_tiles"] == -(-T // p["tile"])
                    if p["blocks_per_team"]:
                        assert p["teams"] * p["token_tiles"] <= sms
                        assert p["teams"] * p["blocks_per_team"] >= w_tiles * blocks > (p["teams"] - 1) * p["blocks_per_team"]


def test_rows_of_the_convolution_fill_the_sms(lib):
    """A thread takes several rows only where enough blocks are left: never fewer than half of four an SM, or two rows."""
    rows, sms = lib.raw("rb_conv_rows"), lib.raw("rb_device_sm_count")()
    for C in (4, 64, 512, 1536, 2048, 4096, 8192):
        for T in (1, 16, 63, 64, 100, 128, 256, 511, 512, 1000, 2048, 100000):
            r = rows(T, C, 4)
            assert r in (0, 2, 4, 8, 16)
            blocks = -(-T // max(r, 1)) * -(-C // 512)
            assert r <= 2 or blocks >= sms, (T, C, r)               # (64 rows of 2,048 channels in 16 blocks took 8.6 us, 3.2 in 128)
            if T >= 512:
                assert r >= 2
            if r == 0:
                assert T * -(-C // 128) < 6 * sms
    assert rows(2048, 2048, 4) == 16 and rows(64, 2048, 4) == 2 and rows(16, 2048, 4) == 0
    assert rows(2048, 2047, 4) == 0 and rows(2048, 2048, 5) == 0 and rows(2048, 2048, 1) == 0


def test_parts_of_the_float32_product(lib):
    """Cluster sizes that the blocks of K (16 values each) suffice for; many tiles of a short K stay whole (2,048 tiles of K 128 took
    78 us in two parts, 66 whole), few tiles of a long K are cut."""
    parts, sms = lib.raw("rb_gemm_simple_parts"), lib.raw("rb_device_sm_count")()
    for M in (17, 33, 64, 130, 300, 512, 1024, 2048, 8192):
        for N in (1, 64, 256, 2048, 5000, 8192):
            for K in (1, 16, 17, 48, 64, 100, 128, 256, 511, 512, 2048, 11008):
                p = parts(M, N, K, 1)
                assert p in ((0,) if M <= 32 and N <= 4096 else (1, 2, 4, 8)) and p <= -(-K // 16), (M, N, K, p)
                tiles = -(-M // 64) * -(-N // 64)
                if K <= 256 and tiles >= 6 * sms:
                    assert p in (0, 1), (M, N, K, p)
    assert parts(64, 2048, 2048, 1) == 8 and parts(2048, 2048, 2048, 1) == 2 and parts(2048, 11264, 2048, 1) == 1
    assert parts(300, 256, 128, 16) == 1 and parts(100, 256, 128, 16) == 4 and parts(1, 1, 1, 1) == 0


def test_float32_products_that_go_to_the_tensor_cores(lib):
    """Enough outputs to fill the chip and a K of 128 and more, little of it padding; clusters of 1, 2 or 4 parts of whole blocks of K."""
    import ctypes
    out = (ctypes.c_int * 2)()

    def plan(M, N, K, Z=1):
        assert lib.raw("rb_f32_tc_plan_of")(M, N, K, Z, 148, out) == 0
        return tuple(out)
    for M in (17, 33, 64, 130, 300, 2048, 8192):
        for N in (1, 64, 96, 256, 2048, 5000, 30000):
            for K in (4, 64, 128, 260, 512, 2048, 11008):
                for Z in (1, 16):
                    bn, parts = plan(M, N, K, Z)
                    assert (bn, parts) == (0, 0) or (bn in (64, 128) and parts in (1, 2, 4) and parts <= -(-K // 64)), (M, N, K, Z)
                    if K < 128 or -(-N // 64) * -(-M // 64) * Z < 16:
                        assert bn == 0, (M, N, K, Z)
    assert plan(64, 2048, 2048) == (64, 4) and plan(600, 11264, 2048) == (128, 1) and plan(2048, 4096, 14336) == (128, 2)
    assert plan(4000, 64, 256, 64) == (0, 0) and plan(2048, 128, 128, 16) == (128, 1) and plan(300, 512, 192) == (0, 0)


def test_when_few_tokens_choices_are_made_by_the_kernel_that_places(lib):
    """Every block makes every token's choice: few blocks times tokens, fewer with more outputs than a warp has lanes or in groups."""
    def pays(T, n, groups, top, tile, shared=0):
        n_tiles = lib.raw("rb_routed_tiles")(T * top, n, tile) + shared
        return bool(lib.raw("rb_route_choose_place_pays")(T, n, groups, n_tiles * tile))
    assert pays(8, 32, 0, 4, 16, 1) and not pays(16, 32, 0, 4, 16) and not pays(4, 32, 0, 4, 64) and pays(2, 32, 0, 4, 64, 1)
    assert pays(4, 32, 8, 4, 16, 1) and not pays(8, 32, 8, 4, 16) and pays(2, 32, 8, 4, 16, 1)
    assert pays(2, 128, 0, 8, 16) and not pays(4, 64, 0, 8, 16) and not pays(2, 64, 0, 8, 64)
    assert pays(1, 256, 8, 8, 16) and not pays(2, 256, 8, 8, 16) and not pays(16, 256, 8, 8, 64)


def test_when_a_matrix_memory_goes_in_chunks():
    """The longest run decides where the runs are few, not their average; small memories and short runs stay token by token."""
    from rbitnet_b200.kernels.ops import memory_chunks_pay

    def pays(lengths, H, D, Dv):
        return memory_chunks_pay(max(lengths), sum(lengths), sum(-(-n // 64) for n in lengths), H, D, Dv)
    assert pays([2048], 8, 128, 256) and pays([2048], 8, 256, 512) and pays([300], 4, 64, 64)
    assert pays([2000] + [1] * 90, 8, 128, 256)                     # one long prompt beside 90 decoding rows
    assert pays([200] + [1] * 7, 8, 256, 512)                       # 256 us token by token, 164 in chunks
    assert not pays([24] * 6, 8, 128, 256)                          # 30 us token by token, 49 in chunks
    assert not pays([48] * 16, 4, 64, 64) and not pays([64] * 16, 2, 16, 24)
    assert pays([64] * 16, 8, 128, 256) and not pays([16] * 64, 8, 128, 256)
    for size in ((8, 128, 256), (2, 512, 512), (1, 1, 1)):
        assert not pays([2], *size) and not pays([1, 1, 2], *size)


@pytest.mark.parametrize("D,Dv,chunks", [(512, 65534, True), (512, 65535, False), (512, 100000, False), (511, 16414, True), (511, 16420, False),
                                         (4, 64 * 65534, True), (4, 64 * 65534 + 1, False)])
def test_a_memory_too_large_for_the_chunks_goes_token_by_token(lib, D, Dv, chunks):
    """Sizes whose sums or whose walk over the chunks would be more than 65,535 blocks a head, which the form that goes token by token
    takes."""
    from types import SimpleNamespace
    from rbitnet_b200.kernels.ops import CudaOps
    ops = SimpleNamespace(lib=lib, memory_chunks_from=(1, 1), memory_scratch_floats=1 << 40)
    meta = SimpleNamespace(extra={}, seqs=[SimpleNamespace(n_new=130)], n_tokens=130)
    assert CudaOps._memory_chunks_chosen(ops, meta, 1, 1, D, Dv) == chunks
    walk = ((Dv + 1) * D // (4 if D % 4 == 0 else 1) + 127) // 128
    sums = 1 + -(-Dv // 64) * -(-D // 64)
    assert (max(walk, sums) <= 65535) == chunks


def test_parts_of_a_gated_product():
    """Two parts of a short K and many parts' sums of many tokens are left out: each was slower than the product whole."""
    from rbitnet_b200.kernels.ops import gated_parts
    assert gated_parts(1, 2816, 2048, 8, 148) == 8 and gated_parts(64, 2816, 2048, 8, 148) == 8
    assert gated_parts(192, 3584, 4096, 2, 148) == 2 and gated_parts(64, 3584, 4096, 2, 148) == 1
    assert gated_parts(65, 192, 512, 2, 148) == 1 and gated_parts(192, 5632, 1024, 2, 148) == 1 and gated_parts(65, 5632, 2048, 2, 148) == 1
    assert gated_parts(48, 8192, 1024, 4, 148) == 1 and gated_parts(17, 8192, 1024, 4, 148) == 4 and gated_parts(48, 5632, 1024, 4, 148) == 4
    assert gated_parts(300, 2816, 2048, 1, 148) == 1


def test_no_pointer_of_a_kernel_is_restrict():
    """The compiler may load what lies behind a restrict pointer before the wait for the kernel that writes it (rb_common.cuh)."""
    from pathlib import Path
    import rbitnet_b200
    sources = sorted((Path(rbitnet_b200.__file__).parent / "csrc").glob("*.cu*"))
    assert sources and not [s.name for s in sources if "__restrict" in s.read_text() or "__ldg(" in s.read_text()]
