"""The walks of the matrix memories in three launches and in one, whatever the length of the runs: against the recurrences in float64,
beside the token-by-token scans, over long runs, and with values that are not finite."""

import pytest
import torch

import test_walk_gpu as W

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 1 << 30])
def form(request, monkeypatch):
    """From which run on the three launches take a step: always, never."""
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "PIECES_MIN_RUN", request.param)
    monkeypatch.setattr(ops, "PIECES_MIN_WORK", 0)
    count = lambda: ops.choices["ssd_pieces"] + ops.choices["mlstm_pieces"]
    before = count()
    yield request.param
    assert (count() > before) == (request.param == 1)


@pytest.mark.parametrize("steps", W.STEPS)
@pytest.mark.parametrize("H,G,N,Dv", [(2, 1, 64, 64), (4, 2, 128, 64), (40, 8, 128, 128), (6, 2, 64, 192)])
def test_ssd_in_both_forms(form, steps, H, G, N, Dv):
    W.test_ssd_walk(steps, H, G, N, Dv)


@pytest.mark.parametrize("steps", W.STEPS)
@pytest.mark.parametrize("H,N,Dv", [(2, 64, 64), (3, 128, 128), (64, 64, 128)])
def test_mlstm_in_both_forms(form, steps, H, N, Dv):
    W.test_mlstm_walk(steps, H, N, Dv)


@pytest.mark.parametrize("slow", [False, True])
@pytest.mark.parametrize("kind,N", [("ssd", 64), ("ssd", 128), ("mlstm", 64), ("mlstm", 128)])
def test_long_runs_in_both_forms(form, kind, N, slow):
    W.test_long_runs_lose_no_precision(kind, N, slow)


@pytest.mark.parametrize("at", [0, 15, 63, 64, 150])
@pytest.mark.parametrize("what", ["value", "key", "query", "gate"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("kind", ["ssd", "mlstm"])
def test_what_is_not_finite_in_both_forms(form, kind, what, bad, at):
    W.test_what_is_not_finite_stays_behind_its_token(kind, what, bad, at)


def test_an_arena_without_the_room(monkeypatch):
    """Steps whose scratch an arena cannot hold walk in one launch."""
    from kv_cache_optimization_for_llm_b200 import ops
    from kv_cache_optimization_for_llm_b200.engine.arena import StepArena
    monkeypatch.setattr(ops, "PIECES_MIN_WORK", 0)
    batch = W._batch([(0, 0, 256)], {0: 0})
    dev, unit = torch.device("cuda:0"), ops._pieces_unit("ssd", 8, 128, 64)
    for room, taken in ((4 * unit, False), (8 * unit, True)):
        arena = StepArena(dev, 1 << 16, room)
        with ops.use_arena(arena):
            arena.begin_step()
            arena.begin_layer()
            assert bool(ops._pieces_bytes("ssd", batch, 256, 8, 128, 64, dev)) == taken
