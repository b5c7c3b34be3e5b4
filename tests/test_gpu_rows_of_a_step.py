"""The small kernels between a decode step's products at the edges of their forms, against float64 or against the kernels apart."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16


@pytest.fixture(scope="module")
def ops_of():
    from rbitnet_b200.kernels.ops import CudaOps
    made = {}
    return lambda dtype: made.setdefault(dtype, CudaOps(dtype, verbose_build=False))


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("E,groups,K", [(1024, 1, 4), (1028, 1, 4), (2048, 2, 1), (2048, 2, 2), (60, 5, 3), (4, 1, 4), (2048, 2, 5)])
def test_rows_between_two_sublayers_by_part(ops_of, dtype, E, groups, K):
    """Parts of up to 1,024 values and four taps in registers, larger ones not: against the kernels apart, from the first position."""
    from rbitnet_b200.engine.step import SeqChunk, build_meta
    ops = ops_of(dtype)
    g = torch.Generator(device="cuda").manual_seed(E + K)
    T = 3
    w, bias = torch.randn(E, device="cuda", generator=g), torch.randn(E, device="cuda", generator=g)
    taps = torch.randn(E, K, device="cuda", generator=g)
    ring_a = torch.randn(6, K, E, device="cuda", generator=g)
    ring_b = ring_a.clone()
    x_a = torch.randn(T, E, device="cuda", generator=g)
    x_b = x_a.clone()
    wide = torch.randn(T, E + 8, device="cuda", generator=g)
    for pos in range(7):
        meta = build_meta([SeqChunk(slot, pos, 1, i) for i, slot in enumerate((4, 0, 2))], np.zeros(T, dtype=np.int32),
                          np.zeros(0, dtype=np.int32), ops.device)
        y, z = torch.randn(T, E, device="cuda", generator=g), wide[:, 4:E + 4]
        add = None if pos == 3 else (y, z, bias if pos % 2 else None)
        h, hf = ops.norm_filter_rows(x_a, w, groups, 1e-5, taps, ring_a, meta, add=add)
        if add is not None:
            ops.gated_add(x_b, y, z, add[2])
        want = ops.rmsnorm_grouped(x_b, w, groups, 1e-5)
        want_f = ops.input_filter(want, taps, ring_b, meta)
        assert torch.equal(x_a, x_b)
        tol = 1e-5 if dtype == F32 else 1e-2                       # sums of squares in another order; a rounding to 8 bits
        for a, b in ((h, want), (hf, want_f), (ring_a[[4, 0, 2]], ring_b[[4, 0, 2]])):
            if K > 1 or b.dim() == 2:
                assert float((a.double() - b.double()).abs().max()) <= tol * float(b.double().abs().max())


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("T,H,Dv,pad", [(1, 1, 4, 0), (8, 8, 256, 0), (5, 3, 512, 4), (3, 2, 516, 0), (7, 5, 30, 0), (2, 3, 128, 1)])
@pytest.mark.parametrize("shared,silu", [(0, 0), (1, 1)])
def test_norm_and_gate_per_head(ops_of, dtype, T, H, Dv, pad, shared, silu):
    """Heads in registers (up to 512 values, 16-byte loads) and longer or misaligned ones, in float64."""
    from rbitnet_b200.kernels.ops import _ptr
    ops = ops_of(dtype)
    g = torch.Generator(device="cuda").manual_seed(Dv + T)
    o = torch.randn(T, H, Dv, device="cuda", generator=g)
    w = torch.randn(Dv if shared else H * Dv, device="cuda", generator=g)
    proj = torch.randn(T, 8 + H * Dv + pad, device="cuda", generator=g)
    out = torch.empty(T, H * Dv, dtype=dtype, device="cuda")
    off = 4 + pad
    ops.lib.call("rb_head_norm_gate", _ptr(out), ops.code, _ptr(o), _ptr(w), _ptr(proj), proj.stride(0), 0, off, T, H, Dv, 1e-5, shared, silu,
                 ops._stream())
    x, gate = o.double(), proj[:, off:off + H * Dv].double().view(T, H, Dv)
    n = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * (w.double() if shared else w.double().view(H, Dv))
    want = (n * torch.sigmoid(gate) * (gate if silu else 1.0)).view(T, H * Dv)
    assert float((out.double() - want).abs().max()) <= (1e-5 if dtype == F32 else 5e-3) * float(want.abs().max())
