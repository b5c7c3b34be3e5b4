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
