"""Kernels start while the kernel before them still runs; none may read what that one writes before it has waited for it."""
import numpy as np
import pytest
import torch
from ctypes import c_void_p

pytestmark = pytest.mark.gpu
DELAY_NS = 400_000


def _meta(ops, runs):
    """runs: (slot, start, n) per sequence."""
    from rbitnet_b200.engine.step import SeqChunk, build_meta
    chunks, at = [], 0
    for slot, start, n in runs:
        chunks.append(SeqChunk(slot, start, n, at))
        at += n
    return build_meta(chunks, np.zeros(at, dtype=np.int32), np.zeros(0, dtype=np.int32), ops.device)


def _random_part(part, ops, g):
    part.bind({k: 0.3 * torch.randn(shape, device="cuda", generator=g) for k, (shape, _) in part.weight_shapes().items()}, ops)
    return part


def _linear(ops, g, M, N, K, odt):
    w = ops.prepare_linear([torch.randn(N, K, device="cuda", generator=g)])
    return (M, K), ops.dtype, lambda x: ops.linear(x, w, out_dtype=odt)


def _gated(ops, g, M, N, K):
    w = ops.prepare_gate_up(*(torch.randn(N, K, device="cuda", generator=g) for _ in range(2)))
    return (M, K), ops.dtype, lambda x: ops.gated_linear(x, w)


def _mixer(ops, g, which, lengths):
    from rbitnet_b200.parts.recurrent import MatrixMemory, GatedLinearRecurrence
    from rbitnet_b200.parts.delta import GatedDeltaRule
    from rbitnet_b200.parts.gla import GatedLinearAttention
    from rbitnet_b200.parts.retention import Retention
    H, D, Dv = 4, 32, 48
    part, call, width = {
        "memory": lambda: (MatrixMemory(16, H, D, Dv, 6.0, 1e-5), ops.matrix_memory, 2 * H * D + 2 * H * Dv + 2 * H),
        "delta": lambda: (GatedDeltaRule(16, H, 2, D, Dv, 3, 1e-5), ops.gated_delta, 4 * D + 2 * H * Dv + 2 * H),
        "gla": lambda: (GatedLinearAttention(16, H, D, Dv, 8, 16.0, 1e-5), ops.gated_linear_attention, 2 * H * D + 2 * H * Dv + 8),
        "retention": lambda: (Retention(16, H, D, Dv, [0.9] * H, 1e-5), ops.retention, 2 * H * D + 2 * H * Dv),
        "gated": lambda: (GatedLinearRecurrence(16, 128, 4, 3), ops.gated_recurrence, 256)}[which]()
    _random_part(part, ops, g)
    meta = _meta(ops, [(i, 5, n) for i, n in enumerate(lengths)])
    start = {k: torch.randn((len(lengths), *s.shape), device="cuda", generator=g) for k, s in part.state_need().items()}

    def prepared():                                  # with a state of its own, made before the late copy
        states = {k: v.clone() for k, v in start.items()}
        return lambda rows: call(rows, part, states, meta)
    return (sum(lengths), width), torch.float32, prepared


def _route(ops, g, T):
    router = torch.randn(24, 96, device="cuda", generator=g)
    return (T, 96), ops.dtype, lambda x: torch.cat([t.float() for t in ops.route(x, router, None, 3, 1, 1)], dim=1)


def _experts(ops, g, T):
    from rbitnet_b200.kernels.ops import LinearWeight
    up, down = (torch.randn(6 * a, b, device="cuda", generator=g).to(ops.dtype) for a, b in ((40, 96), (96, 40)))
    ids = torch.stack([torch.randperm(6, device="cuda", generator=g)[:2] for _ in range(T)]).to(torch.int32)
    weights = torch.rand(T, 2, device="cuda", generator=g)
    return (T, 96), ops.dtype, lambda x: ops.routed_experts(x, ids, weights, LinearWeight(up, 240, 96), LinearWeight(down, 576, 40), 6, 40)


def _norm(ops, g, T):
    w = torch.rand(200, device="cuda", generator=g)
    return (T, 200), torch.float32, lambda x: ops.rmsnorm(x, w, 1e-5)


def _attention(ops, g, T, D):
    H, page = 4, 64
    k, v = (torch.randn(2, 2, page, D, device="cuda", generator=g).to(ops.dtype) for _ in range(2))
    table = torch.tensor([[0, 1]], dtype=torch.int32, device="cuda")
    pos = torch.arange(100 - T, 100, dtype=torch.int32, device="cuda")
    slot = torch.zeros(T, dtype=torch.int32, device="cuda")
    ptr = lambda t: c_void_p(t.data_ptr())

    def run(q):
        out = torch.empty_like(q)
        ops.lib.call("rb_attention_simple", ptr(out), ptr(q), 0 if q.dtype == torch.float32 else 1, ptr(k), ptr(v), ptr(table), 2, page,
                     ptr(pos), ptr(slot), T, H, 2, D, D ** -0.5, 0, ops._stream())
        return out
    return (T, H * D), ops.dtype, run


CASES = [("linear", _linear, (1, 200, 256, None)), ("linear", _linear, (8, 40, 130, None)), ("linear", _linear, (70, 200, 256, None)),
         ("linear", _linear, (64, 50, 50, None)), ("linear", _linear, (150, 36, 36, torch.float32)), ("linear", _linear, (100, 13, 19, None)),
         ("gated", _gated, (1, 96, 256)), ("gated", _gated, (70, 50, 50)), ("gated", _gated, (70, 96, 1024)),
         ("memory", _mixer, ("memory", [1, 1, 1])), ("memory", _mixer, ("memory", [9, 2])), ("memory", _mixer, ("memory", [300])),
         ("delta", _mixer, ("delta", [1, 1, 1])), ("delta", _mixer, ("delta", [70, 3])), ("delta", _mixer, ("delta", [1] * 70)),
         ("gla", _mixer, ("gla", [1, 1, 1])), ("gla", _mixer, ("gla", [70, 3])), ("retention", _mixer, ("retention", [1, 1])),
         ("retention", _mixer, ("retention", [70])), ("recurrence", _mixer, ("gated", [1, 1])), ("recurrence", _mixer, ("gated", [70, 600])),
         ("route", _route, (1,)), ("route", _route, (70,)), ("experts", _experts, (3,)), ("experts", _experts, (200,)),
         ("norm", _norm, (3,)), ("norm", _norm, (300,)), ("attention", _attention, (1, 64)), ("attention", _attention, (40, 30)),
         ("attention", _attention, (90, 128))]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name,make,args", CASES, ids=[f"{n}-{'-'.join(str(a) for a in args)}" for n, _, args in CASES])
def test_rows_that_are_written_late(name, make, args, dtype):
    """The rows that an operation reads are written by the kernel before it, 0.4 ms after it has let the operation's kernel begin; until
    then they are NaN.  The result is the one of rows that were there all along, bit for bit."""
    from rbitnet_b200.kernels.ops import CudaOps
    ops = CudaOps(dtype)
    g = torch.Generator(device="cuda").manual_seed(61)
    shape, rows_dtype, run = make(ops, g, *args)
    prepared = make is _mixer
    count = shape[0] * shape[1]
    padded = -(-count * (2 if rows_dtype == torch.bfloat16 else 4) // 16) * 16 // (2 if rows_dtype == torch.bfloat16 else 4)
    there = torch.randn(padded, device="cuda", generator=g).to(rows_dtype)
    ready = run() if prepared else run
    want = ready(there[:count].view(shape))
    for _ in range(3):
        late = torch.full((padded,), float("nan"), dtype=rows_dtype, device="cuda")
        ready = run() if prepared else run
        torch.cuda.synchronize()
        ops.lib.call("rb_late_copy_for_test", c_void_p(late.data_ptr()), c_void_p(there.data_ptr()), late.numel() * late.element_size(),
                     DELAY_NS, ops._stream())
        got = ready(late[:count].view(shape))
        assert torch.equal(got, want), (got - want).abs().max()
    ops.check_errors()
