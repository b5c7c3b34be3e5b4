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
