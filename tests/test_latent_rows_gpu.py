"""Latent attention over keys and values that were made for a step, with a rotated part behind every head's key and an output
gate: against float64 and beside the form that attends over the cached latents, in steps with one run, several, runs that
continue, single tokens beside them."""

import math

import numpy as np
import pytest
import torch

from part_harness import _ctx, _make, _run_in_steps, _w

pytestmark = pytest.mark.gpu


def _plain(x, w, heads, dim, rot, vdim, rank, scale, eps, sink, gate, window, dims=None):
    """One whole sequence in float64: x [T, W]; the first ``dims`` (all) of the rotated part's channels turn."""
    dims = rot if dims is None else dims
    rms = lambda v, g: v / np.sqrt((v * v).mean(-1, keepdims=True) + eps) * g
    T = x.shape[0]
    q = (rms(x @ w["dq"].T, w["dq_norm"]) @ w["uq"].T).reshape(T, heads, dim + rot)
    kv = x @ w["dkv"].T
    c, kr = rms(kv[:, :rank], w["dkv_norm"]), kv[:, rank:]
    if dims:
        ang = np.arange(T)[:, None] * 10000.0 ** (-np.arange(0, dims, 2) / dims)
        cos, sin = np.cos(ang), np.sin(ang)

        def turn(v, cs, sn):
            out = v.copy()
            out[..., 0::2], out[..., 1::2] = v[..., 0::2] * cs - v[..., 1::2] * sn, v[..., 1::2] * cs + v[..., 0::2] * sn
            return out
        q[..., dim:dim + dims] = turn(q[..., dim:dim + dims], cos[:, None], sin[:, None])
        kr = np.concatenate([turn(kr[:, :dims], cos, sin), kr[:, dims:]], 1)
    k = np.concatenate([(c @ w["uk"].T).reshape(T, heads, dim), np.repeat(kr[:, None], heads, 1)], -1)
    v = (c @ w["uv"].T).reshape(T, heads, vdim)
    i, j = np.arange(T)[:, None], np.arange(T)[None]
    seen = (j <= i) & ((i - j < window) if window else True)
    out = np.zeros((T, heads, vdim))
    for h in range(heads):
        s = np.where(seen, q[:, h] @ k[:, h].T * scale, -np.inf)
        m = s.max(1, keepdims=True)
        e = np.exp(s - m)
        out[:, h] = e @ v[:, h] / (e.sum(1, keepdims=True) + (np.exp(w["sink"][h] - m) if sink else 0.0))
    out = out.reshape(T, heads * vdim)
    if gate:
        out = out / (1.0 + np.exp(-(x @ w["g"].T)))
    return out @ w["o"].T


@pytest.mark.parametrize("heads,dim,rot,vdim,rank,sink,gate,window", [
    (4, 128, 64, 128, 128, True, False, None), (2, 64, 32, 64, 64, False, True, None), (3, 24, 8, 40, 72, True, True, 100),
    (2, 96, 96, 16, 64, False, False, 64), (2, 120, 8, 128, 64, True, True, None)])
def test_made_rows_with_a_rotated_part(heads, dim, rot, vdim, rank, sink, gate, window, scale=None):
    from kv_cache_optimization_for_llm_b200 import ops
    from kv_cache_optimization_for_llm_b200.models.spec import PartSpec
    rng = np.random.default_rng(dim + rot)
    W, qr = 64, 48
    ctx = _ctx("bfloat16")
    shapes = {"dq": (qr, W), "uq": (heads * (dim + rot), qr), "dkv": (rank + rot, W), "uk": (heads * dim, rank),
              "uv": (heads * vdim, rank), "o": (W, heads * vdim), "dq_norm": (qr,), "dkv_norm": (rank,)}
    if sink:
        shapes["sink"] = (heads,)
    if gate:
        shapes["g"] = (heads * vdim, W)
    wt, w64 = {}, {}
    for n, s in shapes.items():
        wt[n], w64[n] = _w(rng, s, 0.1, 1.0) if n.endswith("norm") else _w(rng, s, 1.0 / math.sqrt(s[-1]) if len(s) > 1 else 0.5)
    params = {"hidden_size": W, "heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "q_rank": qr, "kv_rank": rank,
              "scale": (dim + rot) ** -0.5 if scale is None else scale, "eps": 1e-6, "sink": sink, "gate": gate, "window": window,
              "position": PartSpec("rope_interleaved", {"dims": rot, "base": 10000.0})}
    mixer = _make("mixer", "latent_attention", params, wt, ctx)
    assert mixer.ukv is not None
    xs, refs = {}, {}
    for r, T in enumerate((400, 330, 5)):
        x, x64 = _w(rng, (T, W), 1.0)
        xs[r] = x.cuda()
        refs[r] = _plain(x64, w64, heads, dim, rot, vdim, rank, params["scale"], 1e-6, sink, gate, window)
    steps = [[(0, 300), (2, 1)], [(2, 1), (0, 100), (1, 290)], [(2, 3)], [(1, 40)]]
    before, line = ops.choices["latent_up_library"], ops.LATENT_UP_MIN_CONTEXT
    ops.LATENT_UP_MIN_CONTEXT = 64      # here short contexts go this way as well
    got = _run_in_steps(mixer, ctx, xs, steps, page=16)
    ops.LATENT_UP_MIN_CONTEXT = line
    assert ops.choices["latent_up_library"] == before + 3       # the steps with runs of 16 tokens and more
    old, ops.LATENT_UP_MIN_ROWS = ops.LATENT_UP_MIN_ROWS, 0
    absorbed = _run_in_steps(mixer, ctx, xs, steps, page=16)
    ops.LATENT_UP_MIN_ROWS = old
    rms = lambda a: float(np.sqrt((a ** 2).mean()))
    for r in xs:
        off, off_absorbed = (rms(g[r].double().numpy() - refs[r]) / rms(refs[r]) for g in (got, absorbed))
        # bfloat16 steps between the products: about 2^-8 a piece, and no further off than over the cached latents
        assert off < 1.5e-2 and off < 1.5 * off_absorbed + 2e-3, (r, off, off_absorbed)


@pytest.mark.parametrize("heads,dim,rot,vdim,rank,sink,window", [
    (2, 64, 32, 64, 64, False, None), (3, 64, 32, 64, 72, True, None), (2, 64, 32, 64, 64, True, 100), (2, 128, 64, 128, 64, False, 70),
    (1, 160, 32, 128, 64, True, None)])
def test_made_rows_with_keys_wider_than_values_on_tcgen05(heads, dim, rot, vdim, rank, sink, window):
    from kv_cache_optimization_for_llm_b200 import ops
    before = ops.choices["flash_attention_rows_masked"]
    test_made_rows_with_a_rotated_part(heads, dim, rot, vdim, rank, sink, False, window)
    assert ops.choices["flash_attention_rows_masked"] > before


@pytest.mark.parametrize("heads,dim,rot,vdim,rank,sink,window", [
    (2, 96, 32, 128, 64, True, None), (3, 32, 32, 64, 72, False, 100), (2, 64, 64, 128, 64, True, 70)])
def test_made_rows_of_equal_sizes_with_a_rotated_part_on_tcgen05(heads, dim, rot, vdim, rank, sink, window, monkeypatch):
    """Steps with tiles enough to fill the GPU take this kernel; here every step does."""
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "FLASH_ROWS_WIDE", 3)
    before = ops.choices["flash_attention_rows_masked"]
    test_made_rows_with_a_rotated_part(heads, dim, rot, vdim, rank, sink, False, window)
    assert ops.choices["flash_attention_rows_masked"] > before


@pytest.mark.parametrize("scale", [0.0, -0.07])
def test_scales_that_the_tcgen05_kernel_refuses_stay_on_the_other(scale):
    from kv_cache_optimization_for_llm_b200 import ops
    before = ops.choices["flash_attention_rows_masked"]
    test_made_rows_with_a_rotated_part(2, 64, 32, 64, 64, True, False, None, scale)
    assert ops.choices["flash_attention_rows_masked"] == before


@pytest.mark.parametrize("dims", [0, 8, 24])       # of 24 channels behind the key: none (the layer has no position), some, all
@pytest.mark.parametrize("gate", [False, True])
def test_made_rows_whose_shared_part_turns_in_part_or_not_at_all(dims, gate):
    from kv_cache_optimization_for_llm_b200 import ops
    from kv_cache_optimization_for_llm_b200.models.spec import PartSpec
    rng = np.random.default_rng(dims)
    W, qr, heads, dim, rot, vdim, rank = 64, 48, 3, 40, 24, 32, 64
    ctx = _ctx("bfloat16")
    shapes = {"dq": (qr, W), "uq": (heads * (dim + rot), qr), "dkv": (rank + rot, W), "uk": (heads * dim, rank),
              "uv": (heads * vdim, rank), "o": (W, heads * vdim), "dq_norm": (qr,), "dkv_norm": (rank,)}
    if gate:
        shapes["g"] = (heads * vdim, W)
    wt, w64 = {}, {}
    for n, s in shapes.items():
        wt[n], w64[n] = _w(rng, s, 0.1, 1.0) if n.endswith("norm") else _w(rng, s, 1.0 / math.sqrt(s[-1]))
    params = {"hidden_size": W, "heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "q_rank": qr, "kv_rank": rank,
              "scale": (dim + rot) ** -0.5, "eps": 1e-6, "sink": False, "gate": gate, "window": None,
              "position": PartSpec("rope_interleaved", {"dims": dims, "base": 10000.0}) if dims else None}
    mixer = _make("mixer", "latent_attention", params, wt, ctx)
    x, x64 = _w(rng, (900, W), 1.0)
    y, y64 = _w(rng, (4, W), 1.0)
    refs = [_plain(v, w64, heads, dim, rot, vdim, rank, params["scale"], 1e-6, False, gate, None, dims) for v in (x64, y64)]
    xs, before = {0: x.cuda(), 1: y.cuda()}, ops.choices["latent_up_library"]
    steps = [[(0, 760), (1, 1)], [(1, 1), (0, 16)], [(0, 90), (1, 1)], [(0, 34), (1, 1)]]     # from position 768 on the rows are made
    got = _run_in_steps(mixer, ctx, xs, steps, page=16)
    assert ops.choices["latent_up_library"] == before + 3
    for r, ref in enumerate(refs):
        # bfloat16 steps between the products: about 2^-8 a piece
        assert float(np.sqrt(((got[r].double().numpy() - ref) ** 2).mean())) < 1.5e-2 * float(np.sqrt((ref ** 2).mean())), r


def test_rotation_outside_the_table_is_reported():
    from kv_cache_optimization_for_llm_b200 import ops
    st = ops.kernel_status("cuda:0")
    st.zero_()

    class B:
        positions, status = torch.tensor([0, 7], dtype=torch.int32, device="cuda"), st
    q = torch.randn(2, 16, device="cuda").bfloat16()
    want = q.clone()
    cos, sin = torch.ones(4, 4, device="cuda"), torch.zeros(4, 4, device="cuda")
    ops.latent_rotate(q, 0, 1, 16, 8, cos, sin, B)
    assert int(st.item()) == 2 and torch.equal(q, want)
    st.zero_()


@pytest.mark.parametrize("budget,made", [(64, False), (512, True)])
def test_steps_of_an_engine_allocate_nothing_for_made_rows(budget, made):
    """Short runs far behind the start, one beside a single token: rows are made only where the largest step's memory holds them."""
    import tempfile

    import plain_rezusun as R
    import tiny_rezusun as tiny
    from kv_cache_optimization_for_llm_b200 import ops
    from kv_cache_optimization_for_llm_b200.engine.batch import StepEntry
    from test_rezusun_gpu import TOL_MODEL, _logit_err, _runner
    cfg = tiny.config([tiny.latent(heads=4, dim=32, rot_dim=16, vdim=32, q_rank=24, kv_rank=64, ff=64)] * 2, width=64)
    folder = tempfile.mkdtemp(prefix="kvb200_rows_")
    w = tiny.write_model(folder, cfg, seed=4)
    r = _runner(folder, "bfloat16", num_pages=400, max_num_batched_tokens=budget, max_model_len=2000)
    seq = np.random.default_rng(3).integers(0, cfg["vocab"], 1444).tolist()
    before, pos, got = ops.choices["latent_up_library"], 0, []
    for n in [64] * 22 + [20]:
        beside = [StepEntry(1, [7], 0, ())] if n == 20 else []
        got.append(r.step(beside + [StepEntry(0, seq[pos:pos + n], pos, [n - 1])]).cpu().numpy())
        pos += n
    assert (ops.choices["latent_up_library"] > before) == made
    assert r.arena.bypassed == 0 and r.arena.blocks_grown() == 0
    ref = R.forward(cfg, w, seq[:pos])
    ends = list(range(63, 64 * 22, 64)) + [pos - 1]
    assert _logit_err(np.concatenate(got), ref[ends], "bfloat16") < TOL_MODEL["bfloat16"]
    r.check_status()
