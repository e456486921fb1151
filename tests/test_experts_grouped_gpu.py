"""Experts' products over the tokens that chose them, against the same in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _gate(T, E, top, how, g):
    """[T, E + 3] with at most ``top`` weights a row in the first E columns; what stands behind them is not theirs."""
    gate = torch.full((T, E + 3), 7.0, device="cuda")
    gate[:, :E] = 0.0
    if how == "spread":
        chosen = torch.rand((T, E), generator=g, device="cuda").topk(top, dim=1).indices
    elif how == "same":                 # every token the same experts: some of 16 tiles and more, the others without a token
        chosen = torch.arange(E - top, E, device="cuda").expand(T, top)
    else:                               # the first 129 tokens one expert, the next 128 another, one token a third, the last none
        chosen = torch.full((T, top), E - 1, device="cuda")
        chosen[:129], chosen[129:257], chosen[257:258] = 0, 1, 3
    gate.scatter_(1, chosen, torch.rand((T, top), generator=g, device="cuda") + 0.2)
    if how == "uneven":
        gate[-1, :E] = 0.0
    return gate


@pytest.mark.parametrize("T,H,E,F,S,top,how,weigh_output,shared", [
    (128, 512, 8, 128, 128, 2, "spread", False, True), (129, 264, 8, 128, 256, 1, "spread", True, False), (300, 1024, 32, 128, 128, 4, "spread", False, True),
    (640, 256, 40, 256, 384, 5, "same", False, True), (400, 328, 4, 128, 128, 1, "uneven", True, True), (2048, 512, 256, 128, 128, 8, "spread", False, False), (257, 256, 64, 128, 128, 16, "spread", True, True)])
def test_grouped_experts(T, H, E, F, S, top, how, weigh_output, shared, monkeypatch):
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "GROUPED_MIN_WORK", 0)
    g = torch.Generator(device="cuda").manual_seed(T + H)

    def draw(*s, std=1.0):
        return (torch.randn(s, generator=g, device="cuda") * std).bfloat16()

    x, first, down = draw(T, H), draw(2 * (E * F + S), H, std=H ** -0.5), draw(H, E * F + S, std=F ** -0.5)
    gate = _gate(T, E, top, how, g)
    logit = torch.randn((T, 2), generator=g, device="cuda")[:, 1] if shared else None
    limit, shared_limit, alpha, offset = 1.5, 0.8, 1.702, 1.0
    assert ops.experts_grouped_ok(x, first, down, E, F, S, top)
    out = ops.experts_grouped(x, first, down, gate, logit, E, F, S, top, limit, shared_limit, alpha, weigh_output, offset)
    assert int(ops.kernel_status(x.device).item()) == 0
    p = x.double() @ first.double().T
    act = torch.zeros((T, E * F + S), dtype=torch.float64, device="cuda")

    def one(gv, uv, w, lim):
        gv, uv = (w * gv).clamp(max=lim), (w * uv).clamp(-lim, lim)
        return gv * torch.sigmoid(alpha * gv) * (uv + offset)

    for e in range(E):
        w = gate[:, e:e + 1].double()
        gv, uv = p[:, 2 * e * F:(2 * e + 1) * F], p[:, (2 * e + 1) * F:(2 * e + 2) * F]
        act[:, e * F:(e + 1) * F] = torch.where(w != 0, w * one(gv, uv, 1.0, limit) if weigh_output else one(gv, uv, w, limit), 0.0)
    act[:, E * F:] = one(p[:, 2 * E * F:2 * E * F + S], p[:, 2 * E * F + S:], 1.0, shared_limit)
    if shared:
        act[:, E * F:] *= torch.sigmoid(logit.double())[:, None]
    ref, scale = act @ down.double().T, act.abs() @ down.double().abs().T
    # one rounding to bfloat16 of every activation (2^-8 of it bounds it and the float32 sums in front of it) and one of the result
    assert bool(((out.double() - ref).abs() <= 2.0 ** -8 * (scale + ref.abs()) + 1e-6).all())
    again = ops.experts_grouped(x, first, down, gate, logit, E, F, S, top, limit, shared_limit, alpha, weigh_output, offset)
    assert torch.equal(out, again)


def test_little_work_and_sizes_that_tiles_do_not_divide_stay_with_the_products_over_all(monkeypatch):
    from kv_cache_optimization_for_llm_b200 import ops
    x = torch.zeros((128, 64), dtype=torch.bfloat16, device="cuda")
    w1, w2 = (torch.zeros(s, dtype=torch.bfloat16, device="cuda") for s in ((2 * (8 * 128 + 128), 64), (64, 8 * 128 + 128)))
    assert not ops.experts_grouped_ok(x, w1, w2, 8, 128, 128, 2)
    monkeypatch.setattr(ops, "GROUPED_MIN_WORK", 128 * 64 * 8 * 128)
    assert ops.experts_grouped_ok(x, w1, w2, 8, 128, 128, 2)
    for bad in (dict(x=x[:127]), dict(ff=64), dict(shared_ff=0), dict(shared_ff=64), dict(top=3), dict(experts=68, top=17), dict(x=x.float())):
        kw = dict(dict(x=x, first=w1, down=w2, experts=8, ff=128, shared_ff=128, top=2), **bad)
        assert not ops.experts_grouped_ok(**kw)
