"""Products of many tokens at the edges of how their tiles leave and of the order they are taken in, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    from rbitnet_b200.kernels.ops import CudaOps
    return CudaOps(BF16, verbose_build=False)


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def _product(ops, x, w, c, epilogue, tile):
    from rbitnet_b200.kernels.ops import _ptr, _CODE
    T, K = x.shape
    N = w.shape[0]
    ops.lib.call("rb_gemm_tc", _ptr(c), c.stride(0), _CODE[c.dtype], _ptr(x), K, T, _ptr(w), K, N, N, K, epilogue,
                 c.shape[1] if epilogue == 3 else 0, 1, tile, 1.0, ops._stream())
    ops.check_errors()


@pytest.mark.parametrize("tile", [128, 160, 192, 224, 256])
@pytest.mark.parametrize("rest", [1, 16, 17, 47])
def test_a_last_token_tile_of_few_rows(ops, tile, rest):
    """Two groups of warps take every other 16 rows of a tile: with up to 16 rows the second has none, also where the parts of a
    tile whose inner dimension is shared are counted per group."""
    g = torch.Generator(device="cuda").manual_seed(tile + rest)
    T, N, K = 2 * tile + rest, 416, 1032
    x = torch.randn(T, K, device="cuda", generator=g).to(BF16)
    w = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(BF16)
    ref = x.double() @ w.double().T
    guard = 3
    for dtype, bound in ((F32, 2e-5), (BF16, 4e-3)):      # sums in 32 bits; one rounding to 8 bits
        c = torch.full((T + guard, N), 7.0, dtype=dtype, device="cuda")
        _product(ops, x, w, c[:T], 0, tile)
        assert _rel(c[:T], ref) < bound and bool((c[T:] == 7.0).all())
    pairs = w.view(N // 32, 2, 16, K)
    gate, up = (x.double() @ pairs[:, h].reshape(-1, K).double().T for h in (0, 1))
    c = torch.full((T + guard, N // 2), 7.0, dtype=BF16, device="cuda")
    _product(ops, x, w, c[:T], 3, tile)
    assert _rel(c[:T], gate / (1 + torch.exp(-gate)) * up) < 6e-3 and bool((c[T:] == 7.0).all())
    for share in (0, 4):                                   # 17 k blocks in parts of 4: five teams a weight tile
        ops.lib.call("rb_gemm_tc_share_for_test", share, launches=0)
        try:
            c = torch.ones((T + guard, N), dtype=F32, device="cuda")
            for _ in range(2):                             # the counts are back at zero for the second
                _product(ops, x, w, c[:T], 1, tile)
            assert _rel(c[:T], 1.0 + 2.0 * ref) < 2e-5 and bool((c[T:] == 1.0).all())
        finally:
            ops.lib.call("rb_gemm_tc_share_for_test", 0, launches=0)


@pytest.mark.parametrize("T,N,K,tile", [
    (16 * 128, 300, 72, 128), (17 * 128 + 5, 300, 72, 128),   # one band of 16 token tiles; two of 9
    (35 * 128 - 1, 130, 72, 128),                             # three of 12, the last one narrower
    (33 * 256, 520, 64, 256), (641, 300, 65536, 128)])        # bands held to three tiles by the size of X
def test_token_tiles_taken_in_bands(ops, T, N, K, tile):
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, device="cuda", generator=g).to(BF16)
    w = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(BF16)
    ref = x.double() @ w.double().T
    c = torch.full((T, N), float("nan"), dtype=F32, device="cuda")
    _product(ops, x, w, c, 0, tile)
    # sums of K float32 products: their rounding grows with the square root of the k blocks
    assert _rel(c, ref) < (2e-5 if K < 10000 else 1e-4)
    c.zero_()
    _product(ops, x, w, c, 1, tile)
    assert _rel(c, ref) < (2e-5 if K < 10000 else 1e-4)


# ---------------------------------------------------------------- float32 products of values in three bfloat16 parts
@pytest.fixture(scope="module")
def ops32():
    from rbitnet_b200.kernels.ops import CudaOps
    return CudaOps(F32, verbose_build=False)


def _f32(ops32, x, w, out, accumulate=0, alpha=1.0, batch=1, strides=(0, 0, 0), bias=None, gate=None, want=True):
    import ctypes
    from ctypes import c_void_p
    from rbitnet_b200.kernels.ops import _ptr
    (M, K), N = (x.shape[0], w.shape[-1]), w.shape[-2]
    plan = (ctypes.c_int * 2)()
    ops32.lib.call("rb_f32_tc_plan_of", M, N, K, batch, ops32.lib.raw("rb_device_sm_count")(), plan, launches=0)
    assert (plan[0] > 0) == want, "these sizes were chosen for the one or the other"
    if bias is not None or gate is not None:
        ops32.lib.call("rb_gemm_simple_next", _ptr(bias), _ptr(gate), gate.stride(0) if gate is not None else 0, 0, 1, launches=0)
    ops32.lib.call("rb_gemm_simple_batched", _ptr(out), out.stride(0), 0, _ptr(x), x.stride(0), _ptr(w), w.stride(-2), 0, M, N, K,
                   accumulate, float(alpha), batch, *strides, ops32._stream())
    ops32.check_errors()
    return plan[0], plan[1]


@pytest.mark.parametrize("M,N,K", [(1000, 130, 516), (65, 1000, 2052), (129, 2048, 128), (333, 2500, 132), (600, 2048, 2048),
                                   (2049, 384, 260), (64, 2048, 5632), (700, 3001, 1028), (300, 300, 1000)])
def test_float32_products_from_three_parts(ops32, M, N, K):
    """Rows, weight rows and values of K that fill no tile; K whole and in parts; stored, added, scaled, with bias and gate; rows
    wider than K.  Per block of 64 values of K the tensor cores cut off at most 68 times 2^-24 of the magnitudes' sum (four sums
    of 17 values each), adding the blocks rounds once each, and the dropped products of parts are below 2^-25 of theirs."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K + 4, device="cuda", generator=g)[:, :K]
    w = torch.randn(N, K + 8, device="cuda", generator=g)[:, :K]
    ref, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = (72 + -(-K // 64)) * 2.0 ** -24 * mag
    out = torch.full((M + 2, N), 5.0, device="cuda")
    _f32(ops32, x, w, out[:M])
    assert ((out[:M].double() - ref).abs() <= bound).all() and bool((out[M:] == 5.0).all())
    plain = torch.empty((M, N), device="cuda")                 # rows without 16-byte loads: the FFMA tiles
    x1 = torch.empty(M * (K + 1), device="cuda").view(M, K + 1)[:, 1:].copy_(x)
    _f32(ops32, x1, w, plain)
    assert (out[:M].double() - ref).norm() <= (plain.double() - ref).norm()
    bias, gate = torch.randn(N, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g)
    acc = torch.ones((M, N), device="cuda")
    _f32(ops32, x, w, acc, accumulate=1, alpha=0.5, bias=bias, gate=gate)
    s = torch.sigmoid(gate.double())
    want = 1.0 + (0.5 * ref + bias.double()) * s
    assert ((acc.double() - want).abs() <= bound + 2.0 ** -21 * (want.abs() + 1.0 + bias.double().abs())).all()


def test_float32_products_of_blocks_from_three_parts(ops32):
    """Sixteen products at once, a fixed distance apart."""
    g = torch.Generator(device="cuda").manual_seed(5)
    Z, M, N, K = 16, 333, 128, 128
    x = torch.randn(M, Z * K, device="cuda", generator=g)
    w = torch.randn(Z, N, K, device="cuda", generator=g)
    out = torch.empty(M, Z * N, device="cuda")
    _f32(ops32, x[:, :K], w[0], out, batch=Z, strides=(N, K, N * K))
    a = x.double().view(M, Z, K)
    ref = torch.einsum("mzk,znk->mzn", a, w.double()).reshape(M, Z * N)
    mag = torch.einsum("mzk,znk->mzn", a.abs(), w.double().abs()).reshape(M, Z * N)
    assert ((out.double() - ref).abs() <= 74 * 2.0 ** -24 * mag).all()


@pytest.mark.parametrize("K", [512, 2048])
def test_float32_products_that_are_not_finite(ops32, K):
    """Infinities, NaN, values above the largest bfloat16 and very small ones leave what float32 sums leave."""
    g = torch.Generator(device="cuda").manual_seed(6)
    M, N = 128, 1024
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g)
    x[3, 7], x[5, 9], x[70, 1], w[100, 2] = float("inf"), float("nan"), float("-inf"), float("inf")
    w[101, 2] = 0.0
    x[3, 2] = 1.0
    x[9] = 0.0
    x[9, 0], w[:, 0] = 3.4e38, w[:, 0].clamp(-0.9, 0.9)         # rounds to infinity as a bfloat16
    x[10] *= 1e-30
    out = torch.empty(M, N, device="cuda")
    _f32(ops32, x, w, out)
    ref = x.double() @ w.double().T
    assert torch.equal(torch.isnan(out), torch.isnan(ref))
    assert torch.equal(torch.isposinf(out), torch.isposinf(ref)) and torch.equal(torch.isneginf(out), torch.isneginf(ref))
    fin = torch.isfinite(ref)
    mag = torch.where(torch.isfinite(x), x, 0).double().abs() @ torch.where(torch.isfinite(w), w, 0).double().abs().T
    assert ((out.double() - ref).abs()[fin] <= ((K + 8) * 2.0 ** -24 * mag)[fin]).all()      # (K: the sums made by FFMA)


@pytest.mark.parametrize("M,N,K", [(600, 2048, 2048), (128, 1024, 2048), (700, 1000, 516)])
def test_float32_rows_that_are_not_numbers_stay_by_themselves(ops32, M, N, K):
    """One NaN anywhere in a token's values makes all of its sums NaN and nobody else's anything; and that is seen by one look at the
    row: made again value by value, a fifth of the tokens took 15 to 70 times the whole product."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    want, out = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    _f32(ops32, x, w, want)
    y = x.clone()
    rows = torch.arange(3, M, 5, device="cuda")
    y[rows, (rows * 37) % K] = math.nan
    y[rows[1]], y[M - 1, K - 1] = math.nan, math.nan
    _f32(ops32, y, w, out)
    lost = torch.isnan(y).any(1)
    assert bool(torch.isnan(out[lost]).all()) and torch.equal(out[~lost], want[~lost])

    def ms(v):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        times = []
        for _ in range(5):
            a.record()
            _f32(ops32, v, w, out)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    assert ms(y) < 5.0 * ms(x) + 0.2


@pytest.mark.parametrize("T,tile", [(1, 16), (5, 16), (16, 16), (30, 32), (33, 32), (64, 32), (50, 64), (64, 64)])
@pytest.mark.parametrize("parts", [2, 3, 4, 5, 8])
def test_parts_of_a_few_tokens_product(ops, T, tile, parts):
    """Parts summed with all of a CTA's loads in flight (2, 4, 8) and in rounds (others), tokens that fill no tile, two tiles of 32."""
    from rbitnet_b200.kernels.ops import _ptr, _CODE
    g = torch.Generator(device="cuda").manual_seed(T * parts)
    N, K = 416, 2552                                             # 40 blocks of K: whole parts but with 3
    x = torch.randn(T, K, device="cuda", generator=g).to(BF16)
    w = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(BF16)
    ref = x.double() @ w.double().T
    pairs = w.view(N // 32, 2, 16, K)
    gate, up = (x.double() @ pairs[:, h].reshape(-1, K).double().T for h in (0, 1))
    for epilogue, c, want, bound in ((0, torch.full((T + 2, N), 7.0, device="cuda"), ref, 2e-5), (1, torch.ones((T + 2, N), device="cuda"), 1.0 + ref, 2e-5),
                                     (3, torch.full((T + 2, N // 2), 7.0, dtype=BF16, device="cuda"), gate / (1 + torch.exp(-gate)) * up, 6e-3)):
        keep = c[T:].clone()
        ops.lib.call("rb_gemm_tc", _ptr(c), c.stride(0), _CODE[c.dtype], _ptr(x), K, T, _ptr(w), K, N, N, K, epilogue,
                     c.shape[1] if epilogue == 3 else 0, parts, tile, 1.0, ops._stream())
        assert _rel(c[:T], want) < bound and torch.equal(c[T:], keep)
    ops.check_errors()


@pytest.mark.parametrize("T", [33, 48, 64])
@pytest.mark.parametrize("N,K", [(2048, 2048), (96, 2048), (10304, 520), (2048, 768)])
def test_two_tiles_of_32_tokens(ops, T, N, K):
    """What the operations choose for 33 to 64 tokens, stored, added and gated."""
    assert ops._token_tile(T, N, K) == 32 and ops._token_tile(32, N, K) == 0
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, device="cuda", generator=g).to(BF16)
    w = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(BF16)
    ref, lw = x.double() @ w.double().T, ops.prepare_linear([w])
    acc = torch.ones(T, N, device="cuda")
    ops.linear(x, lw, accumulate_into=acc)
    assert _rel(ops.linear(x, lw, out_dtype=F32), ref) < 2e-5 and _rel(acc, 1.0 + ref) < 2e-5
    gate, up = ref[:, :N // 2], ref[:, N // 2:]
    assert _rel(ops.gated_linear(x, ops.prepare_gate_up(w[:N // 2], w[N // 2:])), gate / (1 + torch.exp(-gate)) * up) < 6e-3
    ops.check_errors()
