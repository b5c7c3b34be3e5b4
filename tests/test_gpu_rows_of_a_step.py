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


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("H,Kh,D,Dv,rot,interleaved,norm,taps,keys,mix,gates", [
    (16, 4, 128, 128, 64, True, "head_weight", 4, False, False, False), (20, 4, 64, 72, 24, False, "projection", 4, False, True, True),
    (5, 1, 12, 4, 6, True, None, 4, False, False, True), (3, 1, 260, 260, 12, False, "head_weight", 0, True, False, True),
    (300, 1, 4, 4, 4, False, None, 0, False, False, True), (2, 60, 4, 132, 2, False, "projection", 0, False, True, False),
    (97, 3, 128, 128, 32, False, "projection", 4, False, False, True)])
def test_q_and_k_preparation_in_quads(ops_of, dtype, H, Kh, D, Dv, rot, interleaved, norm, taps, keys, mix, gates):
    """Quads of values against the form that takes any size and address (rows that begin one value late), over runs of several rows
    and single rows, from the first position: the ring, the cache's pages, q and the gates."""
    from rbitnet_b200.cache import SequenceCache
    from rbitnet_b200.parts.base import CacheNeed
    from rbitnet_b200.engine.step import SeqChunk, build_meta
    ops = ops_of(dtype)
    g = torch.Generator(device="cuda").manual_seed(H + D)
    dev = {"device": "cuda", "generator": g}
    C, Dc = (H + Kh) * D, max(D, Dv)
    width = C + (0 if keys else Kh * Dv) + (H if gates else 0)
    table = (10000.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64, device="cuda") / rot), 1.25, interleaved, rot)
    qw, kw = {"projection": (torch.randn(H * D, **dev), torch.randn(Kh * D, **dev)), "head_weight": (torch.randn(D, **dev), torch.randn(D, **dev)),
              None: (None, None)}[norm]
    conv = torch.randn(C, taps, **dev) if taps else None
    made = []
    for late in (0, 1):
        cache = SequenceCache({0: CacheNeed(Kh, Dc)}, reads={}, state_needs={}, max_tokens=16 * 64, max_seq=256, dtype=dtype,
                              device="cuda", page_size=16, n_slots=4)
        for pages in (cache.view(0).k, cache.view(0).v):
            pages.zero_()
        slots = [cache.alloc() for _ in range(3)]
        made.append((cache, slots, torch.zeros(4, max(taps, 1), C, device="cuda")))
    at = [0, 0, 0]
    for lengths in ((1, 1, 1), (5, 1, 40), (1, 1, 1), (1, 1, 1), (2, 33, 1), (1, 1, 1)):
        T = sum(lengths)
        rows, other = torch.randn(T, (width + 7) // 4 * 4, **dev), torch.randn(T, Kh * Dv + 8, **dev)
        got = []
        for late, (cache, slots, ring) in enumerate(made):
            chunks, first = [], 0
            for s, p, n in zip(slots, at, lengths):
                cache.reserve(s, n)
                cache.advance(s, n)
                chunks.append(SeqChunk(s, p, n, first))
                first += n
            cache.upload_tables()
            meta = build_meta(chunks, np.zeros(T, dtype=np.int32), np.zeros(0, dtype=np.int32), ops.device)
            x = torch.empty(rows.numel() + late, device="cuda")[late:].view(rows.shape)
            x.copy_(rows)
            got.append(ops.qk_prepare(x, meta, cache.view(0), H, D, Dv, table, norm, qw, kw, 1e-5, conv=conv, tail=ring if taps else None,
                                      values_are_keys=keys, v_mix=(0.3, other, 4) if mix else None, gate_heads=gates))
        at = [a + n for a, n in zip(at, lengths)]
        (q, gate), (q1, gate1) = got
        a, b = made[0][0].view(0), made[1][0].view(0)
        tol = 2e-6 if dtype == F32 else 8e-3               # sums of squares in another order; a rounding to 8 bits
        for one, two in ((q, q1), (a.k, b.k), (a.v, b.v)):
            assert float((one.double() - two.double()).abs().max()) <= tol * float(two.double().abs().max())
        assert torch.equal(made[0][2], made[1][2]) and (gate is None or torch.equal(gate, gate1))
    ops.check_errors()


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("E,shift", [(4096, 0), (4100, 0), (16384, 0), (16388, 0), (20000, 0), (32772, 0), (16390, 0), (2048, 2), (5120, 2)])
def test_normed_result_added_to_wide_rows(ops_of, dtype, E, shift):
    """Rows in registers, wider ones four values at a time, no multiple of four; ``shift``: rounded rows that begin between two places
    of a wide store.  A sum of E squares and a division are within a few units of float32."""
    from rbitnet_b200.kernels.ops import _ptr
    ops = ops_of(dtype)
    g = torch.Generator(device="cuda").manual_seed(E)
    T = 3
    x, y = torch.randn(T, E, device="cuda", generator=g), 30.0 * torch.randn(T, E, device="cuda", generator=g)
    w = torch.randn(E, device="cuda", generator=g)
    want = x.double() + y.double() / (y.double().square().mean(1, keepdim=True) + 1e-5).sqrt() * w.double()
    to = torch.full((T * E + 8,), 9.0, dtype=dtype, device="cuda")
    ops.lib.call("rb_norm_add", _ptr(x), _ptr(y), _ptr(w), 1e-5, T, E, _ptr(to[shift:]), ops.code, ops._stream())
    assert float((x.double() - want).norm() / want.norm()) <= 1e-6
    assert torch.equal(to[shift:shift + T * E].view(T, E), x.to(dtype))
    assert bool((to[:shift] == 9.0).all()) and bool((to[shift + T * E:] == 9.0).all())


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("E", [4100, 5120, 16384])
@pytest.mark.parametrize("fresh", [False, True])
def test_a_results_norm_and_the_norm_after_it_of_few_and_many_wide_rows(ops_of, dtype, E, fresh):
    """Sixteen values a thread, the second weights asked for before the rows (as many rows as SMs) and after their first sum (more):
    the same bits, and those of float64 within a few units of float32."""
    ops = ops_of(dtype)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(E)
    x, y = torch.randn(sms + 1, E, device="cuda", generator=g), 30.0 * torch.randn(sms + 1, E, device="cuda", generator=g)
    w, w2 = torch.randn(E, device="cuda", generator=g), torch.randn(E, device="cuda", generator=g)
    many, h_many = ops.norm_add_norm(None if fresh else x.clone(), y, w, 1e-5, w2, 1e-5)
    few, h_few = ops.norm_add_norm(None if fresh else x[:sms].clone(), y[:sms], w, 1e-5, w2, 1e-5)
    assert torch.equal(many[:sms], few) and torch.equal(h_many[:sms], h_few)

    def rms(v):
        return v / (v.square().mean(1, keepdim=True) + 1e-5).sqrt()
    want = (0.0 if fresh else x.double()) + rms(y.double()) * w.double()
    assert float((many.double() - want).norm() / want.norm()) <= 1e-6
    rows = rms(want) * w2.double()
    assert float((h_many.double() - rows).norm() / rows.norm()) <= (2e-6 if dtype == F32 else 4e-3)
