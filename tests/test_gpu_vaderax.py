"""The Vaderax decoder on the GPU: the package's kernels against the plain implementation (whole models in both
dtypes, the same cases as on the CPU), and each new kernel alone against the plain functions."""
import ctypes
import math

import numpy as np
import pytest
import torch

import plain_vaderax as plain
import vaderax_cases as cases
from safuvik_tiny import tokens_for, rel_err
from vaderax_tiny import CONFIGS, make_tensors
from rbitnet_b200.config import config_from_dict

pytestmark = pytest.mark.gpu

# Fractions of the largest reference value.  float32: the weights are scaled up so that faults show, which amplifies
# rounding.  bfloat16: operands of the products, q/k/v, the cache, the attention's P and the experts' inner rows are
# rounded to 8 bits.
TOL = {"float32": 2e-4, "bfloat16": 6e-2}
# whole models: measured in bfloat16 on these configurations with matrices spread by 4, the median position differs by
# 0.3 to 0.9 %, nine of ten by less than 2.3 %, and single positions where a router's choice fell the other way by up to 15 %
BAND = {"float32": cases.Band(2e-4), "bfloat16": cases.Band(6e-2, spikes=0.1, spread=4.0)}
DTYPES = ["float32", "bfloat16"]


def engine_maker(dtype):
    from rbitnet_b200.engine import Engine

    def make(cfg, tensors, max_tokens=64 * 16, graphs=False, **kw):
        return Engine(config_from_dict(cfg), dict(tensors), dtype=dtype, max_tokens=max_tokens, max_seq=1024,
                      use_graphs=graphs, **kw)
    return make


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E"])
def test_whole(name, dtype):
    cases.whole(engine_maker(dtype), name, BAND[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E"])
def test_prefill_against_decoding(name, dtype):
    cases.prefill_against_decoding(engine_maker(dtype), name, BAND[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "D"])
def test_portions(name, dtype):
    cases.portions(engine_maker(dtype), name, BAND[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E"])
def test_batches(name, dtype):
    cases.batches_against_alone(engine_maker(dtype), name, BAND[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "C"])
def test_slots_and_pages_used_again(name, dtype):
    cases.slots_and_pages_used_again(engine_maker(dtype), name, BAND[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "E"])
def test_long_decoding(name, dtype):
    cases.long_decoding(engine_maker(dtype), name, BAND[dtype])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", ["A", "B", "C"])
def test_first_tokens(name, dtype):
    cases.first_tokens(engine_maker(dtype), name, BAND[dtype])


@pytest.mark.parametrize("conv", [1, 3])
def test_far_token_through_the_state(conv):
    # float32 only: what the first token of 180 leaves in the last logits is of the size of bfloat16's rounding
    cases.far_token_moves_the_logits(engine_maker("float32"), cases.delta_only(conv), TOL["float32"], least=10.0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,far,cuts", [(300, 2, []), (300, 63, [250] + list(range(290, 300))), (200, 64, list(range(1, 200))),
                                        (700, 0, [64, 128, 699]), (130, 127, [129])])
def test_one_far_key(n, far, cuts, dtype):
    cases.one_far_key_stands_out(engine_maker(dtype), TOL[dtype], n, far, cuts, last_only=dtype == "bfloat16")


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
def _ops(dtype):
    from rbitnet_b200.kernels.ops import CudaOps
    return CudaOps(dtype)


def _meta(ops, runs):
    """runs: (slot, start, n) per sequence."""
    from rbitnet_b200.engine.step import SeqChunk, build_meta
    chunks, at = [], 0
    for slot, start, n in runs:
        chunks.append(SeqChunk(slot, start, n, at))
        at += n
    return build_meta(chunks, np.zeros(at, dtype=np.int32), np.zeros(0, dtype=np.int32), ops.device)


@pytest.mark.parametrize("T,E", [(1, 64), (7, 100), (300, 1000), (3, 4100), (5, 7)])
def test_layer_norm_kernel(T, E):
    ops = _ops(torch.float32)
    g = torch.Generator().manual_seed(E)
    x = torch.randn(T, E, generator=g, dtype=torch.float64) * 3 + 5          # a mean far from zero
    w, b = torch.randn(E, generator=g, dtype=torch.float64), torch.randn(E, generator=g, dtype=torch.float64)
    got = ops.layernorm(x.float().cuda(), w.float().cuda(), b.float().cuda(), 1e-5)
    assert rel_err(got.cpu(), plain.layer_norm(x, w, b, 1e-5)) <= 1e-5
    got = ops.layernorm(x.float().cuda(), w.float().cuda(), None, 1e-5)
    assert rel_err(got.cpu(), plain.layer_norm(x, w, 0.0, 1e-5)) <= 1e-5


@pytest.mark.parametrize("n_experts,identity,top,groups", [(16, 4, 4, (4, 3)), (5, 0, 1, None), (3, 3, 3, (3, 3)), (60, 4, 6, (8, 3)),
                                                           (7, 2, 2, (3, 1)), (2, 0, 2, None), (130, 30, 8, (40, 5))])
@pytest.mark.parametrize("T,K", [(50, 48), (333, 100), (7, 70)])
def test_router_kernel(n_experts, identity, top, groups, T, K):
    """Scores, the choice among the kept groups by score plus correction, weights without it; corrections large
    enough to change the choice, and negative choice scores in whole groups.  Few tokens (a block per token) and many
    (the router's sums as a tiled product), inner sizes that are and are not multiples of 4."""
    ops = _ops(torch.float32)
    g = torch.Generator().manual_seed(n_experts * 10 + top)
    n = n_experts + identity
    h = torch.randn(T, K, generator=g).double()
    w = {"router": torch.randn(n, K, generator=g).double() * 0.3, "correction": torch.randn(n, generator=g).double() * 0.2 - 0.3}
    r = {"experts": n_experts, "identity": identity, "top": top}
    if groups:
        r["groups"] = {"count": groups[0], "keep": groups[1]}
    want_ids, want_w = plain.route(h, r, w)
    ids, weights = ops.route(h.float().cuda(), w["router"].float().cuda(), w["correction"].float().cuda(), top,
                             groups[0] if groups else 0, groups[1] if groups else 0)
    ids, weights = ids.cpu().long(), weights.cpu().double()
    for t in range(T):
        assert sorted(ids[t].tolist()) == sorted(want_ids[t].tolist()), t
        order = torch.argsort(ids[t]), torch.argsort(want_ids[t])
        assert float((weights[t][order[0]] - want_w[t][order[1]]).abs().max()) <= 3e-6
    # the correction decides: without it other experts are chosen somewhere
    other, _ = plain.route(h, r, {"router": w["router"], "correction": torch.zeros(n, dtype=torch.float64)})
    assert any(sorted(other[t].tolist()) != sorted(want_ids[t].tolist()) for t in range(T)) or top == n or T < 50


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,E,F,n_experts,identity,top", [(1, 64, 40, 6, 2, 2), (3, 64, 40, 6, 2, 4), (70, 64, 24, 3, 0, 1),
                                                          (300, 128, 72, 16, 4, 4), (45, 100, 36, 4, 1, 2), (9, 64, 44, 2, 6, 3),
                                                          (2500, 64, 32, 5, 0, 2), (33, 64, 40, 0, 3, 2)])
def test_routed_experts(dtype, T, E, F, n_experts, identity, top):
    """Few pairs and many, tiles of every size, experts without any token, identity experts, a width and an inner
    size that the tensor-core products refuse."""
    from rbitnet_b200.parts.feed_forward import RoutedExperts
    ops = _ops(dtype)
    g = torch.Generator().manual_seed(T + E)
    part = RoutedExperts(E, F, n_experts, top, n_identity=identity)
    w = {k: (torch.randn(*shape, generator=g) * (0.5 if len(shape) > 1 else 0.1)).to(torch.bfloat16).double()
         for k, (shape, _) in part.weight_shapes().items()}
    if n_experts > 2:
        w["correction"][1] = -10.0            # an expert that nobody chooses
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops)
    h = torch.randn(T, E, generator=g).to(torch.bfloat16).double()
    mlp = {"router": {"experts": n_experts, "identity": identity, "top": top}}
    want = plain.routed_ff(h, mlp, w)

    class Ctx:
        pass
    ctx = Ctx()
    ctx.ops = ops
    got = part.forward(ctx, h.to(dtype).cuda())
    assert rel_err(got.cpu(), want) <= (1e-5 if dtype == torch.float32 else 2e-2)
    x = torch.randn(T, E, generator=g).float().cuda()
    before = x.clone()
    part.forward(ctx, h.to(dtype).cuda(), accumulate_into=x)
    assert rel_err((x - before).cpu(), want) <= (1e-5 if dtype == torch.float32 else 2e-2)
    ops.check_errors()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("weighed", [False, True])
@pytest.mark.parametrize("T,E,n_experts,top,tile", [(1, 64, 1, 1, 16), (1, 2048, 40, 4, 16), (8, 100, 33, 3, 16), (64, 36, 5, 4, 64),
                                                    (64, 64, 70, 4, 32), (51, 1032, 3, 5, 16)])
def test_few_pairs_are_placed_as_many_are(dtype, weighed, T, E, n_experts, top, tile):
    """rb_routed_place against the plan and the gather: the same tiles for the same experts, every pair's row in one of its
    expert's rows (in the pairs' order), the same values, zeros elsewhere; identity experts among the ids."""
    ops = _ops(dtype)
    g = torch.Generator().manual_seed(T * 100 + E + top)
    ids = torch.stack([torch.randperm(max(n_experts + 2, top), generator=g)[:top] for _ in range(T)]).to(torch.int32).cuda()
    weights = torch.rand(T, top, generator=g).cuda()
    h = torch.randn(T, E, generator=g).to(dtype).cuda()
    pairs = T * top
    n_tiles = ops.lib.raw("rb_routed_tiles")(pairs, n_experts, tile)
    rows = n_tiles * tile
    ptr = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)
    new = lambda *shape, dt=torch.int32: torch.full(shape, -7, dtype=dt, device="cuda")
    code = 0 if dtype == torch.float32 else 1
    pos, row_token, groups, xp = new(pairs), new(rows), new(n_tiles), new(rows, E, dt=dtype)
    ops.lib.call("rb_routed_plan", ptr(pos), ptr(row_token), ptr(groups), ptr(ids), pairs, top, n_experts, tile, n_tiles, ops._stream())
    if weighed:
        ops.lib.call("rb_routed_gather_scaled", ptr(xp), ptr(h), h.stride(0), code, ptr(row_token), ptr(pos), ptr(weights), top,
                     rows, E, ops._stream())
    else:
        ops.lib.call("rb_routed_gather", ptr(xp), ptr(h), h.stride(0), code, ptr(row_token), rows, E, ops._stream())
    pos2, groups2, xp2 = new(pairs), new(n_tiles), new(rows, E, dt=dtype)
    ops.lib.call("rb_routed_place", ptr(xp2), ptr(pos2), ptr(groups2), ptr(h), h.stride(0), code, ptr(ids),
                 ptr(weights if weighed else None), pairs, top, n_experts, tile, n_tiles, E, ops._stream())
    assert torch.equal(groups, groups2)
    flat = ids.flatten().tolist()
    at, at2 = pos.tolist(), pos2.tolist()
    assert [p < 0 for p in at] == [p < 0 for p in at2] == [e >= n_experts for e in flat]
    taken = [p for p in at2 if p >= 0]
    assert len(set(taken)) == len(taken)
    for e in range(n_experts):
        mine = [p for p, i in zip(at2, flat) if i == e]
        assert mine == sorted(mine) and sorted(mine) == sorted(p for p, i in zip(at, flat) if i == e)
    kept = torch.tensor([p >= 0 for p in at])
    assert torch.equal(xp.cpu()[pos.cpu()[kept].long()], xp2.cpu()[pos2.cpu()[kept].long()])
    empty = torch.ones(rows, dtype=torch.bool)
    empty[pos2.cpu()[kept].long()] = False
    assert float(xp2.cpu()[empty].abs().max()) == 0.0


@pytest.mark.parametrize("T,inner,E", [(1, 96, 1024), (16, 1408, 2048), (17, 200, 1032), (64, 48, 1024), (65, 1408, 2048), (200, 96, 4096)])
@pytest.mark.parametrize("act", [None, (1.702, 7.0, 1.0), "gelu_tanh", "relu", "biases", "norm"])
def test_gated_products_with_parts_of_k(T, inner, E, act):
    """Parts of K in a cluster against K whole: both round the same float32 value once, so a value differs by one step of bfloat16
    (2^-8 of it) where the sums' last bits decide; with room for the sums' own error, K 2^-24 of their magnitudes.  Also with biases, and on rows whose norm is pending (as a product
    of up to 16 tokens takes them)."""
    from rbitnet_b200.kernels.ops import NormedRows
    kind, act = act, None if act in ("biases", "norm") else act
    ops = _ops(torch.bfloat16)
    g = torch.Generator().manual_seed(T + inner)
    x = torch.randn(T, E, generator=g).to(torch.bfloat16).cuda()
    biases = [torch.randn(inner, generator=g).cuda() for _ in range(2)] if kind == "biases" else []
    w = ops.prepare_gate_up(*(torch.randn(inner, E, generator=g).to(torch.bfloat16).cuda() / E ** 0.5 for _ in range(2)), *biases)
    if kind == "norm":
        rows, gw = torch.randn(T, E, generator=g).cuda(), torch.rand(E, generator=g).cuda() + 0.5
        x = NormedRows(rows, gw, 1e-5, (rows * gw).to(torch.bfloat16), rows.square().sum(-1)[None].contiguous())
    before = ops.split_gated
    try:
        ops.split_gated = True
        assert ops._gated_splits(T, w.w.shape[0], E)[0] > 1
        parts = ops.gated_linear(x, w, act).float()
        ops.split_gated = False
        whole = ops.gated_linear(x, w, act).float()
    finally:
        ops.split_gated = before
    assert ((parts - whole).abs() <= 2.0 ** -7 * whole.abs() + 64 * E * 2.0 ** -24).all()
    ops.check_errors()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [5, 100, 400])
def test_dense_feed_forward(dtype, T):
    from rbitnet_b200.parts.feed_forward import Dense
    ops = _ops(dtype)
    g = torch.Generator().manual_seed(T)
    E, F = 64, 88
    part = Dense(E, F)
    w = {k: (torch.randn(*shape, generator=g) * 0.4).to(torch.bfloat16).double() for k, (shape, _) in part.weight_shapes().items()}
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops)
    h = torch.randn(T, E, generator=g).to(torch.bfloat16).double()

    class Ctx:
        pass
    ctx = Ctx()
    ctx.ops = ops
    assert rel_err(part.forward(ctx, h.to(dtype).cuda()).cpu(), plain.dense_ff(h, w)) <= (1e-5 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("chunks,one_launch", [(True, True), (False, False), (True, False)])
@pytest.mark.parametrize("H,G,D,Dv,K", [(4, 2, 16, 24, 3), (1, 1, 40, 8, 1), (6, 3, 32, 64, 4), (2, 2, 128, 64, 2), (3, 1, 100, 33, 5),
                                        (2, 1, 8, 130, 2), (1, 1, 300, 20, 3), (2, 2, 600, 8, 2), (2, 1, 30, 16, 2)])
def test_gated_delta_kernels(H, G, D, Dv, K, chunks, one_launch):
    """Whole runs, portions and single tokens through the state and the convolution's ring; key sizes that one to
    thirty-two lanes hold; decays near one, so that the memory of the first tokens is still there at the end.  Runs of
    several tokens in chunks of 32 (a run of 100 tokens ends inside its fourth chunk) and token by token; single tokens
    in the one kernel of a decode step and in the kernels of a prompt."""
    from rbitnet_b200.parts.delta import GatedDeltaRule
    ops = _ops(torch.float32)
    ops.delta_in_chunks = chunks
    ops.fuse_delta_step = one_launch
    g = torch.Generator().manual_seed(H * 1000 + D)
    E, T = 32, 100
    part = GatedDeltaRule(E, H, G, D, Dv, K, norm_eps=1e-5)
    w = {k: torch.randn(*shape, generator=g, dtype=torch.float64) * (0.3 if len(shape) > 1 and not k.endswith("conv") else 1.0)
         for k, (shape, _) in part.weight_shapes().items()}
    w["A_log"] = w["A_log"] - 3.0
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops)
    h = torch.randn(T, E, generator=g, dtype=torch.float64)
    m = {"heads": H, "kv_heads": G, "dim": D, "vdim": Dv}
    want = plain.delta_mixer(h, m, w, 1e-5)

    class Ctx:
        def state_view(self, entry):
            return state
    for cuts in ([0, T], [0, 1, 2, 20, 36, 37, T], list(range(T + 1)), [0, 32, 33, 97, T], [0, 64, T]):
        state = {k: torch.zeros((3, *n.shape), device="cuda") for k, n in part.state_need().items()}
        outs = []
        for a, b in zip(cuts[:-1], cuts[1:]):
            ctx = Ctx()
            ctx.ops = ops
            ctx.meta = _meta(ops, [(1, a, b - a)])
            outs.append(part.forward(ctx, h[a:b].float().cuda(), 0))
        assert rel_err(torch.cat(outs).cpu(), want) <= 2e-4, cuts
        assert float(state["S"][0].abs().max()) == 0.0 and float(state["S"][2].abs().max()) == 0.0


@pytest.mark.parametrize("T", [32, 75])
@pytest.mark.parametrize("H,G,D,Dv", [(2, 1, 16, 24), (1, 1, 128, 64), (2, 2, 100, 33)])
def test_a_chunk_of_the_delta_rule_rounds_once_at_the_memorys_size(H, G, D, Dv, T):
    """A large memory that forgets nothing, unit keys and a beta of 2^-12, so that the updates are small: a chunk of 32 tokens may
    round the memory once, 2^-24 of it at most.  The updates' own error: u = beta (v - S^T k) is off by at most (D + 40) 2^-24 of
    beta sum |S k| and of itself, and is summed with |k| <= 1 over the run; a factor of 2 for the exponentials and the products
    of the system's small matrix."""
    import ctypes
    ops = _ops(torch.float32)
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + D + T)
    S0 = 1000.0 * torch.randn(3, H, Dv, D, device="cuda", generator=g)
    state = S0.clone()
    qk = torch.nn.functional.normalize(torch.randn(T, 2 * G, D, device="cuda", generator=g).double(), dim=-1).float()
    v = torch.randn(T, H, Dv, device="cuda", generator=g)
    u = torch.cat([qk.view(T, -1), v.view(T, -1)], dim=1).contiguous()
    beta = torch.full((T, H), 2.0 ** -12, device="cuda")
    log_decay = torch.zeros(T, H, device="cuda")
    meta = _meta(ops, [(1, 0, T)])
    first, count, _, runs = ops._runs(meta)
    run0, row, length, n_chunks = ops._delta_chunks(meta)
    o = torch.empty(T, H * Dv, device="cuda")
    scratch = torch.empty(n_chunks * H * ops.lib.raw("rb_gated_delta_chunk_floats")(D, Dv), device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    u = torch.nn.functional.pad(u, (0, -u.shape[1] % 4)).contiguous()         # rows that start on 16 bytes
    ops.lib.call("rb_gated_delta_chunked", ptr(o), ptr(u), u.stride(0), ptr(beta), ptr(log_decay), ptr(state), ptr(scratch), ptr(first),
                 ptr(count), ptr(run0), ptr(row), ptr(length), ptr(meta.tok_slot), runs, n_chunks, H, G, D, Dv, ops._stream())
    S = S0[1].double()                                                       # [H, Dv, D]
    slack = torch.zeros_like(S)
    for t in range(T):
        k = qk[t, G:].double().repeat_interleave(H // G, 0)                  # [H, D]
        new = 2.0 ** -12 * (v[t].double() - torch.einsum("hvd,hd->hv", S, k))
        size = 2.0 ** -12 * (v[t].double().abs() + torch.einsum("hvd,hd->hv", S.abs(), k.abs()))
        S = S + new[:, :, None] * k[:, None, :]
        slack += 2 * (D + 40) * size.unsqueeze(2) * k.abs().unsqueeze(1)
    bound = 2.0 ** -24 * (-(-T // 32) * (torch.maximum(S0[1].double().abs(), S.abs()) + slack / (D + 40)) + slack)
    assert ((state[1].double() - S).abs() <= bound).all()
    assert torch.equal(state[0], S0[0]) and torch.equal(state[2], S0[2])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_token_that_is_not_finite_leaves_the_ones_before_it(bad):
    """The delta rule in chunks, one value of one token infinite or NaN: that token and later ones of its sequence may become
    anything, the tokens before it and the other sequence stay as they are."""
    from rbitnet_b200.parts.delta import GatedDeltaRule
    ops = _ops(torch.float32)
    g = torch.Generator(device="cuda").manual_seed(41)
    H, G, D, Dv, K, T, at = 4, 2, 32, 40, 2, 70, 45
    part = GatedDeltaRule(16, H, G, D, Dv, K, norm_eps=1e-5)
    part.bind({k: 0.3 * torch.randn(shape, device="cuda", generator=g) for k, (shape, _) in part.weight_shapes().items()}, ops)
    proj = torch.randn(2 * T, 2 * G * D + 2 * H * Dv + 2 * H, device="cuda", generator=g)
    outs = []
    for value in (None, bad):
        rows = proj.clone()
        if value is not None:
            rows[at, 2 * G * D + 3] = value                        # a value channel of head 0
        state = {k: torch.zeros((2, *n.shape), device="cuda") for k, n in part.state_need().items()}
        outs.append(ops.gated_delta(rows, part, state, _meta(ops, [(0, 0, T), (1, 0, T)])))
    assert torch.isfinite(outs[0]).all() and not torch.isfinite(outs[1][at]).all()
    assert torch.equal(outs[0][:at], outs[1][:at]) and torch.equal(outs[0][T:], outs[1][T:])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Kh,D,Dv,rot", [(4, 2, 32, 16, 8), (2, 2, 16, 40, 16), (3, 1, 24, 24, 0), (4, 2, 64, 64, 32), (2, 1, 128, 96, 64),
                                           (1, 1, 200, 8, 2)])
def test_attention_part(dtype, H, Kh, D, Dv, rot):
    """The attention with its rotation in pairs (i, i + dims/2), the norm per head after it and the gate per value,
    through the paged cache: whole, in portions across a page border, and token by token."""
    from rbitnet_b200.cache import SequenceCache
    from rbitnet_b200.parts.attention import Attention
    ops = _ops(dtype)
    g = torch.Generator().manual_seed(H * 100 + D)
    E, T = 64, 90
    position = {"kind": "rotary", "params": {"head_dim": D, "theta": 30.0, "pairing": "half", "rot_dim": rot}} if rot else None
    part = Attention(E, H, Kh, D, position=position, scale=0.4, value_dim=Dv, qk_norm="head", norm_eps=1e-5, value_gate=True)
    w = {k: (torch.randn(*shape, generator=g) * 0.3).to(torch.bfloat16).double() for k, (shape, _) in part.weight_shapes().items()}
    part.bind({k: v.float().cuda() for k, v in w.items()}, ops)
    h = torch.randn(T, E, generator=g).to(torch.bfloat16).double()
    m = {"heads": H, "kv_heads": Kh, "dim": D, "vdim": Dv, "scale": 0.4}
    if rot:
        m["rot"] = {"base": 30.0, "dims": rot}
    want = plain.attention(h, m, w, 1e-5)
    for cuts in ([0, T], [0, 60, 64, 65, T], [0, 50] + list(range(51, T + 1))):
        cache = SequenceCache({0: part.cache_need()}, {}, {}, 64 * 4, 1024, dtype, ops.device)
        cache.alloc()
        slot = cache.alloc()

        class Ctx:
            def cache_view(self, entry):
                return cache.view(0)
        outs = []
        for a, b in zip(cuts[:-1], cuts[1:]):
            cache.reserve(slot, b - a)
            cache.upload_tables()
            ctx = Ctx()
            ctx.ops = ops
            ctx.meta = _meta(ops, [(slot, a, b - a)])
            outs.append(part.forward(ctx, h[a:b].to(dtype).cuda(), 0))
            cache.advance(slot, b - a)
        assert rel_err(torch.cat(outs).cpu(), want) <= (2e-5 if dtype == torch.float32 else 3e-2), cuts
    ops.check_errors()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,K,n,top,groups,keep", [(1, 2048, 32, 4, 1, 1), (8, 4096, 30, 4, 1, 1), (63, 1024, 33, 5, 3, 2), (9, 1030, 17, 2, 1, 1),
                                                   (5, 516, 64, 8, 8, 3), (2, 64, 1600, 3, 1, 1)])
def test_the_routers_sums_of_few_tokens(dtype, T, K, n, top, groups, keep):
    """The softmax router for fewer than 64 tokens: the bits of the kernel that makes the sums (lanes over k, FFMA) and chooses, also
    where a tensor-core product could make them, whose sums are 2 to 5 times further from float64.
    Against float64: a lane adds K / 32 products one after the other and the lanes' sums meet in five more, errors that walk to
    (sqrt(K / 64) + sqrt(5)) 2^-24 of the products' 2-norm; four times that for the largest of T x top values, and 16
    roundings for the softmax.  A router that is too large for the kernel that chooses from sums in memory is still taken."""
    ops = _ops(dtype)
    g = torch.Generator(device="cuda").manual_seed(T + K + n)
    h = torch.randn(T, K, device="cuda", generator=g).to(dtype)
    router = (torch.randn(n, K, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16).float()
    ids, weights = torch.empty(T, top, dtype=torch.int32, device="cuda"), torch.empty(T, top, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)
    ops.lib.call("rb_route", ptr(ids), ptr(weights), ptr(h), h.stride(0), 0 if dtype == torch.float32 else 1, ptr(router), ptr(None), T, K,
                 n, top, groups, keep, ptr(None), ops._stream())
    got_ids, got = ops.route(h, router, None, top, groups, keep, ops.prepare_router(router))
    assert torch.equal(got_ids, ids) and torch.equal(got, weights)
    want = torch.softmax(h.double() @ router.double().T, -1).gather(1, ids.long())
    size = (h.double().square() @ router.double().square().T).max(1, keepdim=True).values.sqrt()
    bound = 4 * 2.0 ** -24 * (((K / 64) ** 0.5 + 5 ** 0.5) * size + 16)
    assert ((weights.double() - want).abs() <= bound * want).all()
