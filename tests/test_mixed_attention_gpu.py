"""Single tokens beside runs: their attention runs beside the runs' attention, with the bits of the two one after the other."""

import pytest
import torch

from part_harness import _Manager

pytestmark = pytest.mark.gpu


# forms of the runs' kernel: blocks of 64 rows, of 128 rows (pages too short for the tensor maps: without roles), with roles; a grid of
# many rounds in front, and one of a single block behind which hundreds wait
@pytest.mark.parametrize("d,group,page,singles,runs", [
    (64, 4, 16, 3, [(0, 40)]), (64, 4, 16, 60, [(900, 2)]), (64, 4, 4, 20, [(0, 900), (3, 700)]), (64, 4, 16, 40, [(512, 1500)]),
    (128, 4, 16, 60, [(77, 33)]), (128, 3, 16, 40, [(512, 701)]), (128, 4, 16, 1, [(0, 1900), (1, 64)]), (128, 4, 4, 20, [(0, 700)]),
])
@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("write", [True, False])
def test_single_tokens_beside_runs(d, group, page, singles, runs, write, captured, monkeypatch):
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "BESIDE_MIN_WORK", 0.0)
    from kv_cache_optimization_for_llm_b200.engine.batch import BatchBuilder, StepEntry
    gen = torch.Generator(device="cuda").manual_seed(d + singles)
    dev, nkv, nq = torch.device("cuda:0"), 8, 8 * group
    reqs = [((r * 331) % 2500, 1) for r in range(singles)] + runs
    tables, at = {}, 0
    for r, (s, n) in enumerate(reqs):
        tables[r] = list(range(at, at + -(-(s + n) // page)))
        at += len(tables[r])
    heights = [ops.flash_tokens_per_tile(group, w) for w in (False, True)]
    T = sum(n for _, n in reqs)
    builder = BatchBuilder(T, len(reqs), [2600 // page], dev, ops.kernel_status(dev), page_size=page, tile_heights=heights)
    batch = builder.build([StepEntry(r, [0] * n, s, ()) for r, (s, n) in enumerate(reqs)], _Manager(tables, {r: 0 for r in tables}))
    assert batch.num_single == singles
    pools = [torch.randn(at, nkv, page, d, generator=gen, device="cuda").bfloat16() for _ in range(2)]
    angles = torch.rand(2600, d // 2, generator=gen, device="cuda") * 6
    cos, sin, scale, table = angles.cos(), angles.sin(), d ** -0.5, batch.block_tables[0]

    def after_one_another(x, k, v):
        ns, out = singles, torch.zeros(T, nq * d, dtype=x.dtype, device="cuda")
        ops.decode_attention_mma(x, k, v, write, table[:ns], batch.q_start[:ns + 1], batch.ctx_len[:ns], cos, sin, d, nq, nkv, d, scale,
                                 None, batch.status, max_ctx=ops.decode_launch_context(batch), out=out)
        torch.cuda.synchronize()
        ops.rope_kv_write(x[ns:], batch.positions[ns:], batch.token_req[ns:], cos, sin, k if write else None, v if write else None, table,
                          page, nq, nkv, d, d, batch.status)
        return ops.flash_attention(x, k, v, table, batch, nq, nkv, d, scale, None, skip_single=True, out=out)

    def step(x, k, v):
        return ops.attention_step(x, k, v, write, table, batch, nq, nkv, d, scale, None, 2600, cos, sin, d)

    if not captured:
        replay = step
    qkv, (kb, vb) = torch.empty(T, (nq + 2 * nkv) * d, dtype=torch.bfloat16, device="cuda"), [p.clone() for p in pools]
    if captured:
        step(qkv.zero_(), kb, vb)
        graph, held = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graph):
            held.append(step(qkv, kb, vb))

        def replay(x, k, v):
            graph.replay()
            return held[0]
    for _ in range(6):      # the rows and pages that a pass reads have just been written by launches in front of it
        rows = torch.randn(qkv.shape, generator=gen, device="cuda").bfloat16()
        ka, va = (p.clone() for p in pools)
        want = after_one_another(rows.clone(), ka, va)
        torch.cuda.synchronize()
        kb.copy_(pools[0]), vb.copy_(pools[1]), qkv.copy_(rows)
        got = replay(qkv, kb, vb)
        assert torch.equal(got, want) and torch.equal(ka, kb) and torch.equal(va, vb)
    assert int(batch.status.item()) == 0


def test_callers_streams_have_side_streams_of_their_own():
    """More callers' streams, of two threads, than side streams are kept; a fork that is open keeps its own."""
    import ctypes
    import threading
    from kv_cache_optimization_for_llm_b200 import ops
    library = ops.lib("decode_attention")
    streams = [torch.cuda.Stream(priority=-(i % 2)) for i in range(60)]
    raw = [ctypes.c_void_p(s.cuda_stream) for s in streams]
    errors = []

    def work(mine):
        for turn in range(20):
            for s in mine:
                beside = ctypes.c_void_p()
                if library.kvb_side_fork(s, ctypes.byref(beside)) or beside.value in (None, s.value) or library.kvb_side_join(s):
                    errors.append((turn, s.value))

    open_one = ctypes.c_void_p()
    assert library.kvb_side_fork(raw[0], ctypes.byref(open_one)) == 0
    threads = [threading.Thread(target=work, args=(raw[1 + i::2],)) for i in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    again = ctypes.c_void_p()
    assert library.kvb_side_fork(raw[0], ctypes.byref(again)) == 0 and again.value == open_one.value
    assert library.kvb_side_join(raw[0]) == 0 and library.kvb_side_join(raw[0]) == 0
    torch.cuda.synchronize()
