"""The router of a few tokens: sums spread over the chip, the choice with a lane per output, the placing that makes the choice itself,
and a shared expert that is one more group, each against the same thing in float64 or against the kernels apart."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16


@pytest.fixture(scope="module")
def ops_of():
    from rbitnet_b200.kernels.ops import CudaOps
    made = {}
    return lambda dtype: made.setdefault(dtype, CudaOps(dtype, verbose_build=False))


def _choice(z, corr, top, groups, keep, scoring, normalize, scale):
    """Ids and weights of one token's sums z (float64)."""
    n = len(z)
    s = torch.softmax(z, 0) if scoring == "softmax" else torch.sigmoid(z) if scoring == "sigmoid" else z
    c = s + (corr.double() if corr is not None else 0.0)
    c = torch.where(torch.isnan(c), torch.tensor(-math.inf, dtype=c.dtype), c)      # not a number: never chosen
    if groups > 1 and keep < groups:
        best = c.view(groups, -1).max(1).values
        order = sorted((g for g in range(groups) if best[g] > -math.inf), key=lambda g: (-float(best[g]), g))[:keep]
        c = torch.where(torch.tensor([i // (n // groups) in order for i in range(n)]), c, torch.tensor(-math.inf, dtype=c.dtype))
    ids = sorted((i for i in range(n) if c[i] > -math.inf), key=lambda i: (-float(c[i]), i))[:top]
    w = [float(s[i]) for i in ids] + [0.0] * (top - len(ids))
    ids += [0] * (top - len(ids))
    w = torch.tensor(w, dtype=torch.float64)
    if scoring == "softmax_chosen":
        w = torch.softmax(w, 0)
    if normalize is not None:
        w = w / (w.sum() + normalize)
    return ids, w * scale


@pytest.mark.parametrize("n,groups,keep", [(1, 1, 1), (5, 0, 0), (32, 8, 4), (30, 3, 2), (31, 31, 5), (32, 1, 1), (32, 2, 1), (33, 0, 0), (48, 4, 2)])
@pytest.mark.parametrize("scoring,normalize,scale", [("softmax", None, 1.0), ("sigmoid", 1e-20, 2.5), ("softmax_chosen", None, 1.0)])
@pytest.mark.parametrize("T", [1, 9, 16, 17])
def test_choices(ops_of, n, groups, keep, scoring, normalize, scale, T):
    """Up to 32 outputs and more, in groups or not, ties, outputs that cannot be chosen, fewer choosable ones than choices; the
    same ids and weights from the kernel that also places (up to 16 tokens)."""
    ops = ops_of(F32)
    g = torch.Generator(device="cuda").manual_seed(n * 31 + T)
    K, top = 260, min(4, n)
    h = torch.randn(T, K, device="cuda", generator=g)
    router = torch.randn(n, K, device="cuda", generator=g) / math.sqrt(K)
    h[0] = 0.0                                                   # all sums equal: the lowest outputs
    corr = 0.3 * torch.randn(n, device="cuda", generator=g)
    corr[::3] = -math.inf
    corr[1::5] = float("nan") if n > 10 else 0.0
    for c in ((None, corr) if groups == 0 or n > 1 else (None,)):
        ids, w, _ = ops.route_scored(h, router, c, top, groups, keep, scoring=scoring, normalize=normalize, weight_scale=scale)
        for t in range(T):
            z = (h[t].double() @ router.double().T).cpu()
            want_ids, want = _choice(z, None if c is None else c.cpu(), top, groups, keep, scoring, normalize, scale)
            assert ids[t].tolist() == want_ids
            # float32 sums of 260 products of about 1/16, an exponential or two, a division
            assert torch.allclose(w[t].double().cpu(), want, rtol=2e-5, atol=1e-7)
        placed = ops.route_and_place(h, router, c, top, groups, keep, n, 64, scoring=scoring, normalize=normalize, weight_scale=scale)
        assert (placed is None) == (T > 16)
        if placed is not None:
            assert torch.equal(placed.weights, w)
            rows = placed.pos.view(T, top)
            assert torch.equal(placed.rows[rows.flatten().long()], h.repeat_interleave(top, 0))
            assert torch.equal(placed.tile_group[(rows // placed.tile).long()], ids)


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("n,groups,keep,top", [(3, 0, 0, 2), (30, 3, 2, 4), (32, 0, 0, 4), (33, 0, 0, 1), (64, 8, 3, 8)])
@pytest.mark.parametrize("T", [2, 8, 9, 16])
def test_choices_made_by_the_kernel_that_places_and_apart(ops_of, dtype, n, groups, keep, top, T):
    """The same weights, extra sums, places and rows both ways, whatever the rule between them says: a turn of eight tokens and two."""
    ops = ops_of(dtype)
    lib = ops.lib

    class Ruled:
        def __init__(self, pays):
            self.pays = pays

        def raw(self, name):
            return (lambda *sizes: self.pays) if name == "rb_route_choose_place_pays" else lib.raw(name)

        def call(self, name, *args, launches=1):
            assert name != "rb_route_choose_place" or self.pays
            lib.call(name, *args, launches=launches)
    g = torch.Generator(device="cuda").manual_seed(T * n)
    K = 128
    h = torch.randn(T, K, device="cuda", generator=g).to(dtype)
    router, corr = torch.randn(n + 1, K, device="cuda", generator=g), 0.3 * torch.randn(n, device="cuda", generator=g)
    made = []
    for pays in (0, 1):
        ops.lib = Ruled(pays)
        try:
            made.append(ops.route_and_place(h, router, corr, top, groups, keep, n, 64, scoring="sigmoid", extra_rows=1, normalize=1e-20,
                                            weight_scale=1.5, weight_on_input=True, with_shared=True))
        finally:
            ops.lib = lib
    a, b = made
    for one, two in ((a.weights, b.weights), (a.extra, b.extra), (a.rows, b.rows), (a.pos, b.pos), (a.tile_group, b.tile_group)):
        assert torch.equal(one, two)
    assert a.n_shared == b.n_shared == 1 and torch.equal(a.rows[:T], h) and int(a.tile_group[0]) == n
    ops.check_errors()


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("K", [4, 96, 2048, 2052, 4100])
def test_sums_of_few_tokens(ops_of, dtype, K):
    """Rows of up to 2,048 values and longer ones.  A float32 sum of K products is within K 2^-24 of the sum of their magnitudes."""
    from rbitnet_b200.kernels.ops import _ptr
    ops = ops_of(dtype)
    g = torch.Generator(device="cuda").manual_seed(K)
    for T, n in ((1, 1), (7, 33), (63, 130)):
        h = torch.randn(T, K, device="cuda", generator=g).to(dtype)
        w = torch.randn(n, K, device="cuda", generator=g)
        z = torch.empty(T, n, device="cuda")
        ops.lib.call("rb_route_sums", _ptr(z), _ptr(h), K, ops.code, _ptr(w), T, K, n, ops._stream())
        bound = (K + 2) * 2.0 ** -24 * (h.double().abs() @ w.double().abs().T)
        assert ((z.double() - h.double() @ w.double().T).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("T,experts,inner,E,identity", [(1, 32, 88, 128, 0), (5, 6, 40, 96, 0), (16, 3, 64, 200, 0), (3, 40, 24, 64, 8),
                                                        (9, 32, 88, 128, 0), (16, 70, 24, 64, 8)])
@pytest.mark.parametrize("weight_on_input", [False, True])
def test_a_shared_expert_behind_the_others(ops_of, dtype, T, experts, inner, E, identity, weight_on_input):
    """The shared expert's rows ahead of the pairs' in one buffer, its matrices behind the others', beside the same made apart."""
    if identity and weight_on_input:
        pytest.skip("identity experts go with weights on the results")
    ops = ops_of(dtype)
    g = torch.Generator(device="cuda").manual_seed(T + experts)

    def m(*shape):
        return torch.randn(*shape, device="cuda", generator=g).to(dtype) / math.sqrt(shape[-1])
    gates, ups, downs = ([m(*s) for _ in range(experts + 1)] for s in ((inner, E), (inner, E), (E, inner)))
    w_up, w_down = ops.prepare_expert_gate_up(gates, ups), ops.prepare_linear(downs)
    gate_up, down = ops.expert_of(w_up, w_down, experts)
    h = torch.randn(T, E, device="cuda", generator=g).to(dtype)
    router = torch.randn(experts + identity + 1, E, device="cuda", generator=g) / math.sqrt(E)
    act, top = (1.0, 0.0, 0.0), 2
    ids, w, gate = ops.route_scored(h, router, None, top, 0, 0, scoring="sigmoid", extra_rows=1)
    shared = ops.linear(ops.gated_linear(h, gate_up, act=act), down, out_dtype=F32)
    x0 = torch.randn(T, E, device="cuda", generator=g)
    apart, one = x0.clone(), x0.clone()
    kw = {"act": act, "weight_on_input": weight_on_input}
    ops.routed_experts(h, ids, w, w_up, w_down, experts, inner, accumulate_into=apart, shared=(shared, gate), **kw)
    placed = ops.route_and_place(h, router, None, top, 0, 0, experts, inner, scoring="sigmoid", extra_rows=1,
                                 weight_on_input=weight_on_input, with_shared=True)
    assert placed.n_shared == -(-T // placed.tile) and torch.equal(placed.weights, w) and torch.equal(placed.extra, gate)
    ops.routed_experts(h, None, None, w_up, w_down, experts, inner, accumulate_into=one, shared=(None, placed.extra), placed=placed, **kw)
    # sums of up to 200 products in another order, one rounding of the inner rows to the compute dtype
    bound = 1e-5 if dtype == F32 else 1e-2
    assert float((one - apart).norm() / (apart - x0).norm()) < bound
    ops.check_errors()


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("T,E,top,accumulate,shared,gated,norm", [
    (1, 4, 1, 1, False, False, False), (3, 1028, 4, 1, True, True, True), (300, 2052, 5, 0, True, False, True), (2, 2048, 9, 1, False, False, True),
    (148, 256, 4, 1, True, True, False), (5, 30, 3, 1, True, True, True), (7, 2048, 4, 0, False, False, False)])
def test_weighted_sum_of_the_experts_rows(ops_of, dtype, T, E, top, accumulate, shared, gated, norm):
    """Few tokens and many, four columns a thread and one (widths that are no multiple of four), choices around groups of four, some of
    them the token's own row; the row of infinities is nobody's.  In float64."""
    from rbitnet_b200.kernels.ops import _ptr
    ops = ops_of(dtype)
    g = torch.Generator(device="cuda").manual_seed(T * 10 + top)
    dev = {"device": "cuda", "generator": g}
    y, h = torch.randn(T * top + 1, E, **dev), torch.randn(T, E, **dev).to(dtype)
    y[0] = math.inf
    pos = torch.randint(1, T * top + 1, (T, top), dtype=torch.int32, **dev)
    pos[torch.rand(T, top, **dev) < 0.3] = -1
    w, x = torch.rand(T, top, **dev), torch.randn(T, E, **dev)
    z = torch.randn(T, E, **dev) if shared else None
    gate = torch.randn(T, 3, **dev)[:, 1:2] if gated else None
    nw, nb = torch.randn(E, **dev), torch.randn(E, **dev)
    out = torch.empty(T, E, dtype=dtype, device="cuda")
    rows = torch.where((pos >= 0)[..., None], y[pos.clamp(min=1).long()].double(), h.double()[:, None])
    want = (w.double()[..., None] * rows).sum(1) + (x.double() if accumulate else 0.0)
    if shared:
        want = want + z.double() * (torch.sigmoid(gate.double()) if gated else 1.0)
    if shared or norm:
        ops.lib.call("rb_routed_combine_next", _ptr(z), _ptr(gate), gate.stride(0) if gated else 0, _ptr(nw if norm else None),
                     _ptr(nb if norm else None), 0.4, _ptr(out if norm else None), launches=0)
    ops.lib.call("rb_routed_combine", _ptr(x), x.stride(0), _ptr(y), _ptr(h), h.stride(0), ops.code, _ptr(pos), _ptr(w), T, top, E, accumulate,
                 ops._stream())
    assert float((x.double() - want).abs().max()) <= 1e-6 * float(want.abs().max()) * (top + 3)
    if norm:
        after = nw.double() * torch.tanh(0.4 * want) + nb.double()
        assert float((out.double() - after).abs().max()) <= (2e-5 if dtype == F32 else 8e-3) * float(after.abs().max())


def test_a_refused_choice_leaves_nothing_for_the_next_placing(ops_of):
    """A choice with the tokens' own rows that is refused (more choices than outputs, unequal groups, an unknown scoring) and then a
    plain placing: its rows, places and tiles, and nothing behind them."""
    from rbitnet_b200.kernels.lib import KernelError
    from rbitnet_b200.kernels.ops import _ptr
    ops = ops_of(F32)
    g = torch.Generator(device="cuda").manual_seed(3)
    T, K, experts, top = 5, 64, 6, 2
    h, router = (torch.randn(n, K, device="cuda", generator=g) for n in (T, experts))
    pairs, tile, guard = T * top, 64, 256
    n_tiles = ops.lib.raw("rb_routed_tiles")(pairs, experts, tile)
    ids = torch.randint(0, experts, (T, top), dtype=torch.int32, device="cuda", generator=g)

    def placed():
        xp = torch.full((n_tiles * tile + guard, K), 7.0, device="cuda")
        pos, groups = (torch.full((n + guard,), 77, dtype=torch.int32, device="cuda") for n in (pairs, n_tiles))
        ops.lib.call("rb_routed_place", _ptr(xp), _ptr(pos), _ptr(groups), _ptr(h), K, ops.code, _ptr(ids), None, pairs, top, experts, tile,
                     n_tiles, K, ops._stream())
        return xp, pos, groups
    want = placed()
    for refused, error in (({"top": experts + 1, "groups": 0, "keep": 0}, KernelError), ({"top": top, "groups": 4, "keep": 1}, KernelError),
                           ({"top": top, "groups": 0, "keep": 0, "scoring": "?"}, KeyError)):
        with pytest.raises(error):
            ops.route_and_place(h, router, None, n_experts=experts, inner=64, with_shared=True, **refused)
        for got, expected in zip(placed(), want):
            assert torch.equal(got, expected)
    xp, pos, groups = want
    assert bool((xp[n_tiles * tile:] == 7.0).all()) and bool((pos[pairs:] == 77).all()) and bool((groups[n_tiles:] == 77).all())
    assert torch.equal(xp[pos[:pairs].long()], h.repeat_interleave(top, 0))
    ops.check_errors()


@pytest.mark.parametrize("T", [3, 20, 70])
def test_a_refused_scoring_leaves_no_weighing_for_the_next_choice(ops_of, T):
    """Weights as they are after a call that asked for others and was refused."""
    ops = ops_of(F32)
    g = torch.Generator(device="cuda").manual_seed(T)
    h, router = (torch.randn(n, 64, device="cuda", generator=g) for n in (T, 8))
    ids, want, _ = ops.route_scored(h, router, None, 2, 0, 0)
    for refused in (lambda: ops.route_scored(h, router, None, 2, 0, 0, scoring="?", normalize=1e-20, weight_scale=3.0),
                    lambda: ops.route_and_place(h, router, None, 2, 0, 0, 8, 64, scoring="?", normalize=1e-20, weight_scale=3.0)):
        with pytest.raises(KeyError):
            refused()
        again, weights, _ = ops.route_scored(h, router, None, 2, 0, 0)
        assert torch.equal(again, ids) and torch.equal(weights, want)


@pytest.mark.parametrize("weighed", [False, True])
def test_few_pairs_of_as_many_experts_as_are_counted(ops_of, weighed):
    """9,984 experts are placed (more than the plan for many pairs takes), one more is refused."""
    from rbitnet_b200.kernels.lib import KernelError
    from rbitnet_b200.kernels.ops import _ptr
    ops = ops_of(F32)
    T, K, top, tile, experts = 3, 64, 2, 16, 9984
    g = torch.Generator(device="cuda").manual_seed(1)
    h, w = torch.randn(T, K, device="cuda", generator=g), torch.rand(T, top, device="cuda", generator=g)
    ids = torch.tensor([[9983, 0], [5, 9983], [9728, 9984]], dtype=torch.int32, device="cuda")        # the last is an identity expert
    n_tiles = ops.lib.raw("rb_routed_tiles")(T * top, experts, tile)
    xp, pos, groups = torch.full((n_tiles * tile, K), 7.0, device="cuda"), *(torch.full((n,), -7, dtype=torch.int32, device="cuda") for n in (T * top, n_tiles))

    def place(n):
        ops.lib.call("rb_routed_place", _ptr(xp), _ptr(pos), _ptr(groups), _ptr(h), K, ops.code, _ptr(ids), _ptr(w if weighed else None),
                     T * top, top, n, tile, n_tiles, K, ops._stream())
    place(experts)
    assert groups.tolist() == [0, 5, 9728, 9983, -1, -1] and pos.tolist() == [48, 0, 16, 49, 32, -1]
    rows = torch.zeros_like(xp)
    at = pos[pos >= 0].long()
    rows[at] = (h.repeat_interleave(top, 0) * (w.view(-1, 1) if weighed else 1.0))[pos >= 0]
    assert torch.equal(xp, rows)
    with pytest.raises(KernelError, match="9985 experts"):
        place(experts + 1)


@pytest.mark.parametrize("T,K,n,kernels", [(3, 64, 8, 2), (3, 66, 8, 1), (70, 66, 8, 2), (3, 64, 1600, 1), (63, 64, 1500, 2)])
def test_as_many_launches_are_counted_as_there_are(ops_of, T, K, n, kernels):
    """Few tokens with rows of wide loads, without, and with more outputs than the choice by itself has room for."""
    from torch.profiler import profile, ProfilerActivity
    ops = ops_of(F32)
    g = torch.Generator(device="cuda").manual_seed(n)
    h, router = torch.randn(T, K, device="cuda", generator=g), torch.randn(n, K, device="cuda", generator=g) / math.sqrt(K)
    for choose in (lambda: ops.route_scored(h, router, None, 2, 0, 0)[:2], lambda: ops.route(h, router, None, 2, 0, 0)):
        choose()
        torch.cuda.synchronize()
        before = ops.lib.launches
        with profile(activities=[ProfilerActivity.CUDA]) as seen:
            ids, w = choose()
            torch.cuda.synchronize()
        assert sum("route" in e.name and "kernel" in e.name for e in seen.events()) == kernels == ops.lib.launches - before
        z = torch.softmax(h.double() @ router.double().T, 1)
        best = z.topk(2, dim=1)
        assert torch.equal(ids.long(), best.indices) and torch.allclose(w.double(), best.values, rtol=2e-5, atol=1e-7)
