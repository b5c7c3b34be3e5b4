"""The Safuvik decoder on the GPU: the package's kernels against the plain implementation (whole models
in both dtypes, the same cases as on the CPU), and each new kernel alone against the plain functions."""
import math

import numpy as np
import pytest
import torch

import plain_safuvik as plain
import safuvik_cases as cases
from safuvik_tiny import CONFIGS, make_tensors, tokens_for, run_cut, rel_err
from rbitnet_b200.config import config_from_dict

pytestmark = pytest.mark.gpu

# Fractions of the largest reference value.  float32: the weights are scaled up so that faults show, which
# amplifies rounding (the plain model in float32 differs from itself in float64 by 2e-5 on them).
# bfloat16: operands of the products, q/k/v, the cache and the attention's P are rounded to 8 bits;
# measured 0.6 to 1.9 % on these configurations.
TOL = {"float32": 2e-4, "bfloat16": 5e-2}
DTYPES = ["float32", "bfloat16"]


def tol(dtype, name=""):
    """Configuration D is matrix memories only, with gates capped at 20: a memory's output is divided by |n . q|, which
    is a difference of a few products at the first tokens, and the bfloat16 rounding of the layer's input rows moves
    such an output by up to 9 % of the largest logit (measured, the same request alone or in a batch; in float32 the same
    positions are right to 6e-6).  The band for it in bfloat16 is 12 %; a lost state or a wrong slot moves the
    logits by more than that, and the float32 run of the same case keeps the tight band."""
    if name == "D" and dtype == "bfloat16":
        return 0.12
    # F (three layers, sharp scores over keys of 64 and 128): one position of 90 differs by 2.4 % whole and 5.2 % decoded
    # (the other 89 by 0.4 to 1.6 %, both ways; float32 2e-5 everywhere), so its band is 8 %
    if name == "F" and dtype == "bfloat16":
        return 0.08
    return TOL[dtype]


def engine_maker(dtype):
    from rbitnet_b200.engine import Engine

    def make(cfg, tensors, max_tokens=64 * 16, graphs=False, **kw):
        return Engine(config_from_dict(cfg), dict(tensors), dtype=dtype, max_tokens=max_tokens, max_seq=1024,
                      use_graphs=graphs, **kw)
    return make


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E", "F"])
def test_whole(name, dtype):
    cases.whole_and_layers(engine_maker(dtype), name, tol(dtype, name))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E", "F"])
def test_prefill_against_decoding(name, dtype):
    cases.prefill_against_decoding(engine_maker(dtype), name, tol(dtype, name))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "F"])
def test_portions(name, dtype):
    cases.portions(engine_maker(dtype), name, tol(dtype, name))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E", "F"])
def test_batches(name, dtype):
    cases.batches_against_alone(engine_maker(dtype), name, tol(dtype, name))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B"])
def test_slots_and_pages_used_again(name, dtype):
    cases.slots_and_pages_used_again(engine_maker(dtype), name, TOL[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "C"])
def test_long_decoding(name, dtype):
    cases.long_decoding(engine_maker(dtype), name, TOL[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_first_tokens(name, dtype):
    cases.first_tokens(engine_maker(dtype), name, TOL[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window,n,cuts", [(5, 30, [11, 25, 26, 27, 28, 29]), (64, 150, [100] + list(range(140, 150))),
                                           (65, 140, []), (9, 80, list(range(60, 80)))])
def test_window_edges(window, n, cuts, dtype):
    cases.window_edges(engine_maker(dtype), TOL[dtype] * (3 if dtype == "bfloat16" else 1), window, n, cuts)


@pytest.mark.parametrize("name", ["A", "B"])
def test_far_token(name):
    # float32 only: the first token of 180 moves the last logits by about 1 %, which is bfloat16's rounding
    cases.far_token_moves_the_logits(engine_maker("float32"), name, TOL["float32"])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,Kh,D,Dv,window", [(4, 1, 128, 80, 75), (2, 2, 16, 40, 70), (4, 2, 64, 64, 64), (3, 1, 24, 24, 5),
                                              (2, 1, 96, 32, 129)])
def test_one_key_stands_out_at_the_window_edge(H, Kh, D, Dv, window, dtype):
    """Keys and queries are made by hand: every score is 0 but one key's, which is far above.  Its value
    row alone carries a 1 in the first column.  Just inside the window the output's first column is near
    1, just outside it is 0: for a prompt in one step, in two portions, and token by token; with pages of
    64 the edges fall inside pages and on their borders.  No norm, no rotation: the mask and the cache alone."""
    from rbitnet_b200.cache import SequenceCache
    from rbitnet_b200.kernels.ops import CudaOps
    from rbitnet_b200.parts.base import CacheNeed
    dt = {"float32": torch.float32, "bfloat16": torch.bfloat16}[dtype]
    ops = CudaOps(dt)
    Dc = ops.cache_head_width(D, Dv)
    n = 2 * window + 70
    for special in (n - window, n - window - 1, 63, 64):
        for cuts in ([0, n], [0, n - window + 3, n], [0, n - 20] + list(range(n - 19, n + 1))):
            cache = SequenceCache({0: CacheNeed(Kh, Dc, window)}, {}, {}, 64 * 8, 1024, dt, ops.device)
            cache.alloc()
            slot = cache.alloc()
            proj = torch.zeros(n, (H + Kh) * D + Kh * Dv)
            proj[:, 0:H * D:D] = 6.0                        # every query: 6 in its first value
            proj[special, H * D:(H + Kh) * D:D] = 6.0       # one key: 6 there too, the others 0
            proj[special, (H + Kh) * D::Dv] = 1.0           # and its value row is marked
            outs = []
            for a, b in zip(cuts[:-1], cuts[1:]):
                cache.reserve(slot, b - a)
                cache.upload_tables()
                meta = _meta(ops, [(slot, a, b - a)])
                view = cache.view(0)
                q = ops.norm_rotate_append(proj[a:b].to(dt).cuda().contiguous(), None, meta, view, H, D, Dv, None, None, 1e-6)
                att = ops.attention(q, meta, view, H, 1.0, window)
                outs.append(ops.head_gate(att, None, None, H, Dv, Dc).float().cpu())
                cache.advance(slot, b - a)
            got = torch.cat(outs).view(n, H, Dv)[:, :, 0]
            for i in range(special, n):
                seen = i - special < window
                share = math.exp(36.0) / (math.exp(36.0) + min(i + 1, window) - 1)
                want = share if seen else 0.0
                assert float((got[i] - want).abs().max()) <= 1e-2, (special, cuts[:3], i, got[i], want)
            ops.check_errors()


@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E"])
def test_greedy_generation_through_captured_steps(name):
    cases.greedy_generation(engine_maker("float32"), name)


def test_captured_step_in_bfloat16():
    """The captured decode step (padding rows, state saved around the trial run) against the plain model."""
    from rbitnet_b200.engine.step import StepEntry
    cfg = CONFIGS["A"]
    tensors = make_tensors(cfg, 23)
    eng = engine_maker("bfloat16")(cfg, tensors, graphs=True)
    reqs = [tokens_for(cfg, n, 70 + n) for n in (20, 9, 33)]
    slots = [eng.new_sequence() for _ in reqs]
    eng.step([StepEntry(s, r[:-6], []) for s, r in zip(slots, reqs)])
    got = [[] for _ in reqs]
    for k in range(6, 0, -1):
        out = eng.step([StepEntry(s, [r[-k]], [0]) for s, r in zip(slots, reqs)], captured=True)
        for i in range(len(reqs)):
            got[i].append(out[i:i + 1])
    for i, r in enumerate(reqs):
        assert rel_err(torch.cat(got[i]).float().cpu(), plain.forward(cfg, tensors, r)[-6:]) <= TOL["bfloat16"]


# ---------------------------------------------------------------- kernels alone
@pytest.fixture(scope="module")
def ops32():
    from rbitnet_b200.kernels.ops import CudaOps
    return CudaOps(torch.float32)


def _meta(ops, runs):
    """runs: (slot, start, n) per sequence."""
    from rbitnet_b200.engine.step import SeqChunk, build_meta
    chunks, at = [], 0
    for slot, start, n in runs:
        chunks.append(SeqChunk(slot, start, n, at))
        at += n
    return build_meta(chunks, np.zeros(at, dtype=np.int32), np.zeros(0, dtype=np.int32), ops.device)


@pytest.mark.parametrize("s,E,n_y", [(4, 96, 2), (1, 64, 1), (3, 1000, 2), (8, 40, 1), (5, 50, 2), (6, 64, 1), (16, 33, 3), (2, 4100, 1)])
def test_stream_step_fused_against_pieces_and_plain(ops32, s, E, n_y):
    g = torch.Generator().manual_seed(s * 100 + E)
    T = 7
    X = torch.randn(s, T, E, generator=g, dtype=torch.float64)
    ys = [torch.randn(T, E, generator=g, dtype=torch.float64) * 3 for _ in range(n_y)]
    ws = [torch.randn(E, generator=g, dtype=torch.float64) for _ in range(n_y)]
    mix, w_out, w_in = (torch.randn(s, s, generator=g, dtype=torch.float64), torch.randn(s, generator=g, dtype=torch.float64),
                        torch.randn(s, generator=g, dtype=torch.float64))
    nw, eps = torch.randn(E, generator=g, dtype=torch.float64), 1e-5
    y = sum(plain.rms(a, eps) * w for a, w in zip(ys, ws)) / n_y if n_y > 1 else ys[0]
    X2 = plain.hyper_write(X, mix, w_out, y)
    h_ref = plain.rms(plain.hyper_read(X2, w_in), eps) * nw
    dev = lambda t: t.float().cuda().contiguous()
    packed = lambda Z: dev(Z.permute(1, 0, 2).reshape(T, s * E))
    xa = packed(X)
    h = ops32.stream_step(xa, s, results=[dev(a) for a in ys], result_norms=[dev(w) for w in ws] if n_y > 1 else None,
                          norm_eps=eps, write=(dev(mix), dev(w_out)), read=(dev(w_in), dev(nw), eps))
    assert rel_err(xa.cpu(), packed(X2).cpu()) <= 1e-5 and rel_err(h.cpu(), h_ref) <= 1e-5
    xb = packed(X)
    yb = ops32.normed_mean([dev(a) for a in ys], [dev(w) for w in ws], eps) if n_y > 1 else dev(ys[0])
    ops32.stream_step(xb, s, results=[yb], write=(dev(mix), dev(w_out)))
    hb = ops32.stream_step(xb, s, read=(dev(w_in), dev(nw), eps))
    assert torch.equal(xa, xb) or rel_err(xb.cpu(), xa.cpu()) <= 1e-6
    assert rel_err(hb.cpu(), h.cpu()) <= 1e-6
    assert rel_err(ops32.streams_sum(xa, s).cpu(), X2.sum(0)) <= 1e-5
    assert torch.equal(ops32.streams_expand(dev(ys[0]), s), dev(ys[0]).repeat(1, s))


@pytest.mark.parametrize("H,D,Dv", [(2, 16, 24), (1, 40, 8), (3, 100, 33), (2, 128, 64), (1, 8, 130), (1, 200, 40), (2, 256, 24), (1, 300, 20)])
def test_matrix_memory_kernel(ops32, H, D, Dv):
    """Whole runs, portions and single tokens through the state, sizes that one to four lanes hold."""
    from rbitnet_b200.parts.recurrent import MatrixMemory
    g = torch.Generator().manual_seed(H * 1000 + D)
    E, T = 32, 45
    part = MatrixMemory(E, H, D, Dv, gate_cap=6.0, norm_eps=1e-5)
    w = {k: torch.randn(*shape, generator=g, dtype=torch.float64) * (0.3 if len(shape) > 1 else 1.0)
         for k, (shape, _) in part.weight_shapes().items()}
    w["f.b"] = w["f.b"] + 3.0
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops32)
    h = torch.randn(T, E, generator=g, dtype=torch.float64)
    p = {"heads": H, "dim": D, "vdim": Dv, "gate_cap": 6.0}
    want = plain.matrix_memory(w, p, h, 1e-5)

    class Ctx:
        ops = ops32
        def state_view(self, entry):
            return state
    for cuts in ([0, T], [0, 1, 2, 20, 36, 37, T], list(range(T + 1))):
        state = {k: torch.zeros((3, *n.shape), device="cuda") for k, n in part.state_need().items()}
        outs = []
        for a, b in zip(cuts[:-1], cuts[1:]):
            ctx = Ctx()
            ctx.meta = _meta(ops32, [(1, a, b - a)])
            outs.append(part.forward(ctx, h[a:b].float().cuda(), 0))
        assert rel_err(torch.cat(outs).cpu(), want) <= 2e-4, cuts
        assert float(state["C"][0].abs().max()) == 0.0 and float(state["C"][2].abs().max()) == 0.0


@pytest.mark.parametrize("C,K,lengths,start", [(64, 4, [40, 1, 2, 60], 0), (4, 2, [64], 5), (516, 3, [15, 17, 33, 3], 2), (1024, 4, [700], 1),
                                               (64, 4, [1] * 70, 3), (2048, 4, None, 9), (8192, 3, [70, 1, 130], 2), (2048, 2, [2100], 0),
                                               (64, 4, [513], 6), (4096, 4, [300, 1, 1, 1, 40], 3), (1024, 4, [1] * 600, 8)])
def test_convolution_of_many_rows(ops32, C, K, lengths, start):
    """Two to sixteen rows a thread against a thread per row and channel (which rows that 16-byte loads cannot take get), bit for bit:
    runs that begin inside a block's rows, in the middle of a sequence (inputs from the ring) and at its start, rows that are their
    own runs without a table of runs (lengths None: 130 of them), with biases and SiLU."""
    from ctypes import c_void_p
    g = torch.Generator(device="cuda").manual_seed(C + K)
    alone = lengths is None
    lengths = lengths or [1] * 130
    S, T = len(lengths), sum(lengths)
    x = torch.randn(T, C + 8, device="cuda", generator=g)
    taps, b, xb = torch.randn(C, K, device="cuda", generator=g), torch.randn(C, device="cuda", generator=g), torch.randn(C, device="cuda", generator=g)
    tail = torch.randn(S, K, C, device="cuda", generator=g)
    rows = [(i, sum(lengths[:i]), j) for i, n in enumerate(lengths) for j in range(n)]
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    first, slot, pos = None if alone else dev([r[1] for r in rows]), dev([r[0] for r in rows]), dev([start + r[2] for r in rows])
    ptr = lambda t: c_void_p(t.data_ptr() if t is not None else 0)
    outs = []
    for misaligned in (False, True):                     # the second call's rows start one value behind a 16-byte boundary
        buf = torch.zeros(T * (C + 8) + 1, device="cuda")
        src = buf[1:] if misaligned else buf[:-1]
        src.copy_(x.flatten())
        u = torch.empty(T, C, device="cuda")
        for silu, bias in ((1, b), (0, None)):
            ops32.lib.call("rb_conv_causal", ptr(u), ptr(src), C + 8, 4, 0, ptr(xb) if bias is not None else c_void_p(0), ptr(taps),
                           ptr(b) if bias is not None else c_void_p(0), ptr(tail), ptr(first), ptr(slot), ptr(pos), T, C, K, silu,
                           ops32._stream())
            outs.append(u.clone())
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[3])


@pytest.mark.parametrize("H,D,Dv,lengths", [(2, 16, 24, [64, 1, 65]), (1, 7, 5, [130]), (3, 64, 64, [63, 200, 17]),
                                            (2, 100, 68, [129, 128]), (8, 128, 256, [90] * 16), (1, 260, 40, [70, 3])])
@pytest.mark.parametrize("chunks", [True, False])
def test_matrix_memory_of_several_runs(ops32, H, D, Dv, lengths, chunks):
    """Runs of unequal lengths side by side (as many as fill the GPU several times over among them), in chunks of 64 at their
    edges and token by token, in two portions and a decode step for all, against the plain function run by run.  The bound is
    that of the test above: float32 sums over D and over the tokens, through a quotient and a norm."""
    from rbitnet_b200.parts.recurrent import MatrixMemory
    g = torch.Generator().manual_seed(H * 1000 + D + len(lengths))
    E = 32
    part = MatrixMemory(E, H, D, Dv, gate_cap=6.0, norm_eps=1e-5)
    w = {k: torch.randn(*shape, generator=g, dtype=torch.float64) * (0.3 if len(shape) > 1 else 1.0)
         for k, (shape, _) in part.weight_shapes().items()}
    w["f.b"] = w["f.b"] + 3.0
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops32)
    hs = [torch.randn(n + 1, E, generator=g, dtype=torch.float64) for n in lengths]
    want = [plain.matrix_memory(w, {"heads": H, "dim": D, "vdim": Dv, "gate_cap": 6.0}, h, 1e-5) for h in hs]
    state = {k: torch.zeros((len(lengths) + 2, *n.shape), device="cuda") for k, n in part.state_need().items()}

    class Ctx:
        ops = ops32

        def state_view(self, entry):
            return state
    got = [[] for _ in lengths]
    before = ops32.memory_in_chunks, ops32.memory_chunks_from
    ops32.memory_in_chunks, ops32.memory_chunks_from = chunks, (1, 1)
    try:
        for ends in ([n // 2 for n in lengths], lengths, [n + 1 for n in lengths]):
            bring = [(i, sum(len(x) for x in got[i]), e) for i, e in enumerate(ends)]
            bring = [(i, a, e) for i, a, e in bring if e > a]
            ctx = Ctx()
            ctx.meta = _meta(ops32, [(i + 1, a, e - a) for i, a, e in bring])
            out = part.forward(ctx, torch.cat([hs[i][a:e] for i, a, e in bring]).float().cuda(), 0)
            for (i, _, _), rows in zip(bring, out.cpu().split([e - a for _, a, e in bring])):
                got[i].append(rows)
    finally:
        ops32.memory_in_chunks, ops32.memory_chunks_from = before
    for rows, one in zip(got, want):
        assert rel_err(torch.cat(rows), one) <= 2e-4
    assert float(state["C"][0].abs().max()) == 0.0 and float(state["C"][-1].abs().max()) == 0.0


@pytest.mark.parametrize("D,Dv,T", [(128, 64, 128), (256, 64, 300), (256, 40, 130)])
def test_matrix_memory_in_chunks_is_as_exact_as_token_by_token(ops32, D, Dv, T):
    """Both forms against float64 on the same rows, the mean over six draws of the error's 2-norm.  Token by token a value is the
    sum of D products, D / 32 to a lane; in chunks it is the sum of 64 + D, which must not cost more."""
    from rbitnet_b200.parts.recurrent import MatrixMemory
    H, E = 4, 8
    part = MatrixMemory(E, H, D, Dv, gate_cap=15.0, norm_eps=1e-5)
    part.bind({k: torch.full(shape, 4.0 if k == "f.b" else 1.0, device="cuda") for k, (shape, _) in part.weight_shapes().items()}, ops32)
    at, meta = part.offsets(), _meta(ops32, [(0, 0, T)])
    errors = {True: [], False: []}
    before = ops32.memory_in_chunks
    for seed in range(6):
        g = torch.Generator(device="cuda").manual_seed(seed)
        proj = torch.randn(T, 2 * H * D + 2 * H * Dv + 2 * H, device="cuda", generator=g)
        q, k = (proj[:, at[n]:at[n] + H * D].double().view(T, H, D) for n in "qk")
        v, gate = (proj[:, at[n]:at[n] + H * Dv].double().view(T, H, Dv) for n in "vg")
        i, f = (15.0 * torch.tanh((proj[:, at[n]:at[n] + H].double() + b) / 15.0) for n, b in (("i", 1.0), ("f", 4.0)))
        F = torch.nn.functional.logsigmoid(f).cumsum(0)                                  # [T, H]
        m = F + torch.cummax(i - F, 0).values.clamp(min=0.0)
        later = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)[:, :, None]
        weight = torch.exp(((F - m)[:, None] + (i - F)[None]).masked_fill(later, -math.inf))
        scores = torch.einsum("thd,shd->tsh", q, k) * D ** -0.5 * weight
        o = torch.einsum("tsh,shv->thv", scores, v)
        o = o / (torch.maximum(scores.sum(1).abs(), torch.exp(-m)) + part.floor)[:, :, None]
        want = o / (o.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * torch.sigmoid(gate)
        for chunks in (True, False):
            ops32.memory_in_chunks = chunks
            state = {n: torch.zeros((1, *s.shape), device="cuda") for n, s in part.state_need().items()}
            try:
                got = ops32.matrix_memory(proj, part, state, meta).double().view(T, H, Dv)
            finally:
                ops32.memory_in_chunks = before
            errors[chunks].append(float((got - want).norm() / want.norm()))
    assert sum(errors[True]) <= 1.05 * sum(errors[False]), errors


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_token_that_is_not_finite_leaves_the_ones_before_it(ops32, bad):
    """The matrix memory in chunks, one value of one token infinite or NaN: that token and later ones of its sequence may become
    anything, the tokens before it and the other sequence stay as they are."""
    from rbitnet_b200.parts.recurrent import MatrixMemory
    H, D, Dv, T, at = 2, 40, 72, 150, 101
    g = torch.Generator(device="cuda").manual_seed(43)
    part = MatrixMemory(16, H, D, Dv, gate_cap=15.0, norm_eps=1e-5)
    part.bind({k: 0.3 * torch.randn(shape, device="cuda", generator=g) for k, (shape, _) in part.weight_shapes().items()}, ops32)
    proj = torch.randn(2 * T, 2 * H * D + 2 * H * Dv + 2 * H, device="cuda", generator=g)
    outs = []
    for value in (None, bad):
        rows = proj.clone()
        if value is not None:
            rows[at, part.offsets()["v"] + 5] = value               # a value of head 0
        state = {n: torch.zeros((2, *s.shape), device="cuda") for n, s in part.state_need().items()}
        outs.append(ops32.matrix_memory(rows, part, state, _meta(ops32, [(0, 0, T), (1, 0, T)])))
    assert torch.isfinite(outs[0]).all() and not torch.isfinite(outs[1][at]).all()
    assert torch.equal(outs[0][:at], outs[1][:at]) and torch.equal(outs[0][T:], outs[1][T:])


@pytest.mark.parametrize("W,B,K", [(48, 3, 3), (32, 1, 2), (200, 5, 4), (24, 2, 1)])
def test_gated_recurrence_kernels(ops32, W, B, K):
    from rbitnet_b200.parts.recurrent import GatedLinearRecurrence
    g = torch.Generator().manual_seed(W + K)
    E, T = 40, 50
    part = GatedLinearRecurrence(E, W, B, K)
    w = {k: torch.randn(*shape, generator=g, dtype=torch.float64) * (0.3 if k in ("x", "y", "o", "ra", "ri") else 1.0)
         for k, (shape, _) in part.weight_shapes().items()}
    w["lam"] = w["lam"] - 3.0
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops32)
    h = torch.randn(T, E, generator=g, dtype=torch.float64)
    want = plain.gated_recurrence(w, {"width": W, "blocks": B}, h)

    class Ctx:
        ops = ops32
        def state_view(self, entry):
            return state
    # single rows take one fused kernel (convolution, gates, recurrence); with it switched off, the kernels of a prompt
    for cuts, fused in (([0, T], True), ([0, 1, 2, 3, 4, 30, T - 1, T], True), (list(range(T + 1)), True),
                        (list(range(T + 1)), False), ([0, 2, 3, 40, 41, T], False)):
        ops32.fuse_recurrent_step = fused
        state = {k: torch.zeros((2, *n.shape), device="cuda") for k, n in part.state_need().items()}
        outs = []
        for a, b in zip(cuts[:-1], cuts[1:]):
            ctx = Ctx()
            ctx.meta = _meta(ops32, [(1, a, b - a)])
            outs.append(part.forward(ctx, h[a:b].float().cuda(), 0))
        ops32.fuse_recurrent_step = True
        assert rel_err(torch.cat(outs).cpu(), want) <= 2e-4, (cuts, fused)


@pytest.mark.parametrize("T,fused", [(19, True), (19, False), (300, True), (700, True)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_limited_gated_activation(dtype, T, fused):
    """In the tensor-core product's epilogue (bfloat16: tiles of 16 to 256 tokens) and as a kernel of its own."""
    from rbitnet_b200.kernels.ops import CudaOps
    from rbitnet_b200.parts.feed_forward import GatedDense
    ops = CudaOps(dtype)
    ops.fuse_gated_act = fused
    g = torch.Generator().manual_seed(5)
    E, F = 64, 88
    part = GatedDense(E, F, "swish_limited", limit=0.8)
    w = {k: (torch.randn(*shape, generator=g) * 0.4).to(torch.bfloat16).double() for k, (shape, _) in part.weight_shapes().items()}
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops)
    h = torch.randn(T, E, generator=g).to(torch.bfloat16).double()
    want = plain.clamped_feed_forward(w, {"limit": 0.8}, h)

    class Ctx:
        pass
    ctx = Ctx()
    ctx.ops = ops
    got = part.forward(ctx, h.to(dtype).cuda())
    assert rel_err(got.cpu(), want) <= (1e-5 if dtype == torch.float32 else 2e-2)
    # the limit is in use: without it the result differs
    assert rel_err(plain.clamped_feed_forward(w, {"limit": 100.0}, h), want) > 0.05


@pytest.mark.parametrize("lengths", [[1, 1, 1], [20, 3]])
def test_a_failed_allocation_leaves_no_store_behind(ops32, lengths, monkeypatch):
    """An allocation that fails inside the matrix memory (token by token), whichever it is: the memory is as it was before the call,
    and what another mixer does next on the same thread does not change it.  The call after that is whole."""
    from rbitnet_b200.parts.recurrent import MatrixMemory
    from rbitnet_b200.parts.retention import Retention
    H, D, Dv, E = 2, 24, 40, 16
    g = torch.Generator(device="cuda").manual_seed(47)
    part = MatrixMemory(E, H, D, Dv, gate_cap=6.0, norm_eps=1e-5)
    part.bind({k: 0.3 * torch.randn(shape, device="cuda", generator=g) for k, (shape, _) in part.weight_shapes().items()}, ops32)
    other = Retention(E, 2, 8, 8, [0.9, 0.5], 1e-5)
    other.bind({k: 0.3 * torch.randn(shape, device="cuda", generator=g) for k, (shape, _) in other.weight_shapes().items()}, ops32)
    T, n = sum(lengths), len(lengths)
    proj = torch.randn(T, 2 * H * D + 2 * H * Dv + 2 * H, device="cuda", generator=g)
    meta = _meta(ops32, [(i, 4, c) for i, c in enumerate(lengths)])
    start = {k: torch.randn((n, *s.shape), device="cuda", generator=g) for k, s in part.state_need().items()}
    good = {k: v.clone() for k, v in start.items()}
    want = ops32.matrix_memory(proj, part, good, meta)
    real = torch.empty
    for which in range(10):
        state = {k: v.clone() for k, v in start.items()}
        calls = []

        def failing(*a, **k):
            calls.append(1)
            if len(calls) == which + 1:
                raise torch.OutOfMemoryError("planted")
            return real(*a, **k)
        monkeypatch.setattr(torch, "empty", failing)
        try:
            ops32.matrix_memory(proj, part, state, meta)
            failed = False
        except torch.OutOfMemoryError:
            failed = True
        finally:
            monkeypatch.setattr(torch, "empty", real)
        if not failed:
            break
        rows = torch.randn(2, 4 * 16, device="cuda", generator=g)
        ops32.retention(rows, other, {"S": torch.zeros(2, 2, 8, 8, device="cuda")}, _meta(ops32, [(0, 0, 1), (1, 0, 1)]))
        assert all(torch.equal(state[k], start[k]) for k in start), which
        assert torch.equal(ops32.matrix_memory(proj, part, state, meta), want)
        assert all(torch.equal(state[k], good[k]) for k in start)
    assert not failed and which >= 2


def test_a_prompt_without_room_for_the_chunks_scratch(ops32, monkeypatch):
    """Where the chunked form's scratch cannot be had the prompt goes token by token, with that form's bits."""
    from rbitnet_b200.parts.recurrent import MatrixMemory
    H, D, Dv, T = 2, 64, 48, 300
    g = torch.Generator(device="cuda").manual_seed(53)
    part = MatrixMemory(16, H, D, Dv, gate_cap=6.0, norm_eps=1e-5)
    part.bind({k: 0.3 * torch.randn(shape, device="cuda", generator=g) for k, (shape, _) in part.weight_shapes().items()}, ops32)
    proj = torch.randn(T, 2 * H * D + 2 * H * Dv + 2 * H, device="cuda", generator=g)
    floats = ops32.lib.raw("rb_matrix_memory_chunk_floats")(-(-T // 64), H, D, Dv)
    real, refused, results = torch.empty, [], []

    def no_room(*a, **k):
        if a and a[0] == (floats,):
            refused.append(1)
            raise torch.OutOfMemoryError("planted")
        return real(*a, **k)
    for chunks, empty in ((False, real), (True, no_room)):
        state = {k: torch.zeros((1, *s.shape), device="cuda") for k, s in part.state_need().items()}
        monkeypatch.setattr(ops32, "memory_in_chunks", chunks)
        monkeypatch.setattr(torch, "empty", empty)
        out = ops32.matrix_memory(proj, part, state, _meta(ops32, [(0, 0, T)]))
        monkeypatch.setattr(torch, "empty", real)
        results.append((out, state))
    assert refused == [1] and torch.equal(results[0][0], results[1][0])
    assert all(torch.equal(results[0][1][k], results[1][1][k]) for k in results[0][1])


@pytest.mark.parametrize("dtype", DTYPES)
def test_many_sequences_give_the_same_bits_again(dtype):
    """Sixteen unequal prompts in one step, then captured decode steps for all: matrix memories whose blocks are several times what the
    GPU holds at once, so that blocks of one (sequence, head) run at different times.  A second engine gives the same bits, and
    float32 logits are the plain model's."""
    from rbitnet_b200.engine.step import StepEntry
    from safuvik_tiny import memory_layer, dense
    cfg = {"architecture": "Safuvik", "vocab": 80, "width": 128, "norm": {"eps": 1e-5}, "streams": 2, "logit_scale": 0.5,
           "layers": [memory_layer(16, 64, 128, 10.0, dense(96, 2.0)), memory_layer(8, 128, 256, 10.0, None)]}
    tensors = make_tensors(cfg, seed=21)
    lengths = [3, 17, 40, 1, 26, 9, 33, 2, 12, 65, 5, 21, 30, 8, 14, 48]
    steps = 4
    toks = [tokens_for(cfg, n + steps, 60 + i) for i, n in enumerate(lengths)]
    runs = []
    for _ in range(2):
        eng = engine_maker(dtype)(cfg, tensors, max_tokens=64 * 64, graphs=True)
        slots = [eng.new_sequence() for _ in lengths]
        out = [eng.step([StepEntry(s, t[:n], [n - 1]) for s, t, n in zip(slots, toks, lengths)]).float().cpu()]
        for k in range(steps):
            out.append(eng.step([StepEntry(s, [t[n + k]], [0]) for s, t, n in zip(slots, toks, lengths)], captured=True).float().cpu())
        runs.append(torch.stack(out))                                # [1 + steps, sequences, vocab]
    assert torch.equal(runs[0], runs[1])
    if dtype == "float32":
        for i, (t, n) in enumerate(zip(toks, lengths)):
            assert rel_err(runs[0][:, i], plain.forward(cfg, tensors, t, torch.float64)[n - 1:n + steps]) <= TOL[dtype], i
