"""The forms of the row-by-row kernels that long bfloat16 steps take (16-byte accesses, blocks of tokens): against the general forms
and float64, at sizes on either side of their lines."""

import numpy as np
import pytest
import torch

from test_walk_gpu import _batch

pytestmark = pytest.mark.gpu


def _rn(gen, *s):
    return torch.randn(s, generator=gen, device="cuda")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("taps,act,biases", [(4, "silu", True), (3, "none", False), (2, "silu", False)])
def test_convolution_over_blocks_of_tokens(dtype, taps, act, biases):
    """A step long enough for blocks of tokens, its runs shorter and longer than the taps and the blocks, some of which continue:
    the bits of the same requests alone, a step each (a token a thread)."""
    from kv_cache_optimization_for_llm_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(taps)
    C, G, D = 7168, 2, 64
    k_off, v_off = C - 2 * G * D, C - G * D
    runs = [(0, 0, 1), (1, 9, 2), (2, 0, 3), (3, 1, 7), (4, 0, 8), (5, 30, 9), (6, 0, 61), (7, 2, 300), (8, 0, 90)]
    T = sum(n for *_, n in runs)
    assert T * C // (4 if dtype == torch.float32 else 8) // 8 >= 256 * ops.sm_count("cuda:0")
    order = [e for e in runs if e[2] == 1] + [e for e in runs if e[2] != 1]
    x, w = _rn(gen, T, C + 16).to(dtype), _rn(gen, C, taps)
    ib, ob = (_rn(gen, C), _rn(gen, C)) if biases else (None, None)
    tails = _rn(gen, 12, (taps - 1) * C)
    slots = {r: (5 * r + 2) % 11 for r, *_ in runs}
    pages = [torch.zeros((64 * 9, G, 16, 2 * D), dtype=dtype, device="cuda") for _ in range(2)]
    tables = {r: list(range(64 * r, 64 * r + 64)) for r, *_ in runs}
    whole, alone, got = tails.clone(), tails.clone(), []
    for tl, pg, steps in ((whole, pages[0], [order]), (alone, pages[1], [[e] for e in order])):
        t, outs = 0, []
        for step in steps:
            from kv_cache_optimization_for_llm_b200.engine.batch import BatchBuilder, StepEntry
            from part_harness import _Manager
            dev = torch.device("cuda:0")
            batch = BatchBuilder(4096, 64, [64], dev, ops.kernel_status(dev)).build(
                [StepEntry(r, [0] * n, s, ()) for r, s, n in step], _Manager(tables, slots))
            n = sum(m for *_, m in step)
            outs.append(ops.conv_silu(x[t:t + n, 8:C + 8], 0, C, w, tl, batch, act=act, in_bias=ib, out_bias=ob,
                                      append=(pg, batch.block_tables[0], k_off, v_off, G, D, D)).clone())
            t += n
        got.append(torch.cat(outs))
    assert torch.equal(got[0], got[1]) and torch.equal(whole, alone) and torch.equal(pages[0], pages[1])
    assert bool(pages[0].any()) and int(ops.kernel_status("cuda:0").item()) == 0


@pytest.mark.parametrize("T,H,Dv", [(1, 1, 8), (3, 5, 64), (65, 3, 128), (7, 2, 256), (130, 32, 64), (5, 3, 32)])
def test_head_norm_and_gate(T, H, Dv):
    from kv_cache_optimization_for_llm_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(T + Dv)
    y, g, w = _rn(gen, T, H * Dv) * 3, _rn(gen, T, H * Dv + 8).bfloat16(), _rn(gen, H * Dv)
    out = ops.head_norm_gate(y, (g, 8), w, H, 1e-5, torch.bfloat16)
    odd = ops.head_norm_gate(y, (torch.cat([g[:, :1], g], 1), 9), w, H, 1e-5, torch.bfloat16)      # rows that start off a boundary
    yd = y.double().view(T, H, Dv)
    ref = (yd / torch.sqrt(yd.square().mean(-1, keepdim=True) + 1e-5)).view(T, -1) * w.double() * torch.sigmoid(g[:, 8:].double())
    # one rounding to bfloat16 (2^-9), the rest float32
    for o in (out, odd):
        assert bool(((o.double() - ref).abs() <= ref.abs() * 2.0 ** -7.99 + 1e-30).all())


@pytest.mark.parametrize("T,groups,gs", [(1, 1, 256), (9, 3, 512), (64, 2, 768), (5, 8, 1024), (4, 2, 1280), (3, 2, 40)])
def test_gated_group_norm(T, groups, gs):
    from kv_cache_optimization_for_llm_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(T + gs)
    W = groups * gs
    y, z, w = _rn(gen, T, W) * 2, _rn(gen, T, W + 8).bfloat16(), _rn(gen, W)
    out = ops.gated_group_norm(y, (z, 8), w, groups, 1e-5, torch.bfloat16)
    v = (y.double() * torch.nn.functional.silu(z[:, 8:].double())).view(T, groups, gs)
    ref = (v / torch.sqrt(v.square().mean(-1, keepdim=True) + 1e-5)).view(T, W) * w.double()
    assert bool(((out.double() - ref).abs() <= ref.abs() * 2.0 ** -7.99 + 1e-30).all())


# (head size, requests): grids of one block a (request, kv head) that beyond 2048 positions are cut in 4, 2 and 4 (8 kv heads on 148 SMs)
@pytest.mark.parametrize("d,R", [(128, 24), (128, 40), (64, 48)])
@pytest.mark.parametrize("window", [None, 700])
def test_decode_attention_of_full_grids_beyond_2048(d, R, window):
    from kv_cache_optimization_for_llm_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(R + d)
    nkv, G, ps = 8, 4, 16
    ctxs = [2049 + (r * 977) % 1400 if r % 3 else 1 + (r * 131) % 2048 for r in range(R)]
    pages = [-(-c // ps) for c in ctxs]
    perm = torch.randperm(sum(pages) + 1, generator=gen, device="cuda").int()
    table, at = torch.full((R, max(pages)), -1, dtype=torch.int32, device="cuda"), 0
    for r, n in enumerate(pages):
        table[r, :n] = perm[at:at + n]
        at += n
    pools = [torch.randn(sum(pages) + 1, nkv, ps, d, generator=gen, device="cuda").bfloat16() for _ in range(2)]
    qkv = torch.randn(R, (G + 2) * nkv * d, generator=gen, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(rows):
        k, v = (p.clone() for p in pools)
        n = len(rows)
        out = ops.decode_attention_mma(qkv[rows].contiguous(), k, v, True, table[rows].contiguous(),
                                       torch.arange(n + 1, dtype=torch.int32, device="cuda"),
                                       torch.tensor([ctxs[r] for r in rows], dtype=torch.int32, device="cuda"), None, None, 0, G * nkv, nkv, d,
                                       d ** -0.5, window, status, max_ctx=max(ctxs))
        return out, k, v

    out, k, v = run(list(range(R)))
    for r in (0, 1, R // 2, R - 1):
        assert torch.equal(run([r])[0][0], out[r])           # a token's sums are cut by its positions, whatever blocks make them
        c, lo = ctxs[r], max(0, ctxs[r] - window) if window else 0
        kr, vr = (p[table[r, :pages[r]].long()].transpose(1, 2).reshape(-1, nkv, d)[lo:c].float() for p in (k, v))
        q = qkv[r, :G * nkv * d].float().view(nkv, G, d)
        want = torch.einsum("hgk,khd->hgd", torch.softmax(torch.einsum("hgd,khd->hgk", q, kr) * d ** -0.5, -1), vr).reshape(-1)
        # probabilities and results rounded to bfloat16, 2^-8 each at most
        assert float((out[r].float() - want).norm() / want.norm()) < 2**-7
    assert int(status.item()) == 0
