"""Room for the scratch of the state memories' launches: declared where a step can be long enough for them, and nowhere else."""

import pytest
import torch


def _part(kind, params):
    from kv_cache_optimization_for_llm_b200.parts import BuildContext, lookup
    cls = lookup("mixer", kind)
    ctx = BuildContext(dtype=torch.bfloat16, device=torch.device("cpu"), max_positions=64, status=torch.zeros(1, dtype=torch.int32))
    weights = {r: torch.zeros(ws.shape, dtype=torch.float32 if ws.kind in ("vector", "bias") else torch.bfloat16)
               for r, ws in cls.weight_specs(params).items()}
    return cls(params, weights, ctx)


MLSTM = {"hidden_size": 64, "dim": 64, "vdim": 64, "gate_cap": 15.0, "eps": 1e-6}
SSD = {"hidden_size": 64, "vdim": 64, "state": 128, "groups": 8, "norm_groups": 8, "conv": 4, "eps": 1e-6}
DELTA = {"hidden_size": 64, "kv_heads": 4, "dim": 64, "vdim": 64, "conv": 4, "eps": 1e-6}


@pytest.mark.parametrize("kind,params,heads,tokens,wanted", [
    ("mlstm", MLSTM, 16, 2048, False), ("mlstm", MLSTM, 16, 4096, True), ("mlstm", MLSTM, 32, 1024, False), ("mlstm", MLSTM, 32, 2048, True),
    ("state_space_duality", SSD, 64, 512, False), ("state_space_duality", SSD, 64, 2048, True),
    ("gated_delta", DELTA, 16, 511, False), ("gated_delta", DELTA, 16, 512, True)])
def test_scratch_is_declared_where_a_step_can_take_it(kind, params, heads, tokens, wanted):
    part = _part(kind, dict(params, heads=heads))
    without, any_step, here = sum(part.activation_widths(1)), sum(part.activation_widths()), sum(part.activation_widths(tokens))
    assert any_step > without and here == (any_step if wanted else without)


@pytest.mark.parametrize("rule", ["ssd", "delta"])
@pytest.mark.parametrize("runs", [1, 40])
@pytest.mark.parametrize("taken", [0.0, 0.9])
def test_a_step_without_the_room_left_walks_in_one_launch(rule, runs, taken, monkeypatch):
    """A layer's region of which other tensors hold a part, and a step of many short runs beside a long one, whose pieces are more than
    its tokens'."""
    from types import SimpleNamespace
    from kv_cache_optimization_for_llm_b200 import ops
    from kv_cache_optimization_for_llm_b200.engine.arena import StepArena
    device, tokens = torch.device("cpu"), 2048
    monkeypatch.setattr(ops, "DELTA_PIECES_MIN_RUN", 512)
    batch = SimpleNamespace(max_q_len=1024, num_reqs=runs, num_single=0)
    width = ops.pieces_width("ssd", 64, 128, 64) if rule == "ssd" else ops.delta_pieces_width(32, 64, 64)
    arena = StepArena(device, 1 << 16, int(1.2 * 2 * tokens * width))
    arena.begin_layer()
    with ops.use_arena(arena):
        arena.new((int(taken * arena.current.capacity),), torch.uint8)
        nbytes = (ops._pieces_bytes("ssd", batch, tokens, 64, 128, 64, device) if rule == "ssd"
                  else ops._delta_pieces_bytes(batch, tokens, 32, 64, 64, device))
        assert (nbytes > 0) == (runs == 1 and not taken)
        if nbytes:
            with ops.lent((nbytes,), torch.uint8, device):
                pass
    assert arena.blocks_grown() == 0 and arena.bypassed == 0


@pytest.mark.parametrize("tokens,runs,heads,wanted", [(4096, 4, 64, True), (64 * 65000, 600, 64, False), (4096, 65500, 64, False)])
def test_grids_beyond_the_hardwares_limit_walk_in_one_launch(tokens, runs, heads, wanted, monkeypatch):
    """More pieces than a grid's second dimension holds, which the walk in one launch, a block a run, takes."""
    from types import SimpleNamespace
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "DELTA_PIECES_MIN_RUN", 512)
    batch = SimpleNamespace(max_q_len=1024, num_reqs=runs, num_single=0)
    assert (ops._delta_pieces_bytes(batch, tokens, heads, 64, 64, torch.device("cpu")) > 0) == wanted
    assert (ops._pieces_bytes("ssd", batch, tokens, heads, 128, 64, torch.device("cpu")) > 0) == wanted
    assert ops._pieces_bytes("ssd", batch, 4096, 65536, 128, 64, torch.device("cpu")) == 0
