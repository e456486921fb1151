"""The delta rule's walk in three launches and in one, whatever the length of the runs: against the recurrence in float64, beside the
token-by-token scan, over long runs, and with values that are not finite."""

import pytest

import test_walk_gpu as W

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 1 << 30])
def form(request, monkeypatch):
    """From which run on the three launches take a step: always, never."""
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "DELTA_PIECES_MIN_RUN", request.param)
    before = ops.choices["delta_pieces"]
    yield request.param
    assert (ops.choices["delta_pieces"] > before) == (request.param == 1)


@pytest.mark.parametrize("alike", [False, True])
@pytest.mark.parametrize("steps", W.STEPS)
@pytest.mark.parametrize("H,G,N,Dv", [(2, 1, 64, 32), (4, 4, 64, 64), (3, 3, 64, 32), (64, 16, 64, 64)])
def test_delta_walk_in_both_forms(form, steps, H, G, N, Dv, alike):
    W.test_delta_walk(steps, H, G, N, Dv, alike)


@pytest.mark.parametrize("slow", [False, True])
def test_long_runs_in_both_forms(form, slow):
    W.test_long_runs_lose_no_precision("delta", 64, slow)


@pytest.mark.parametrize("what", ["key", "value", "gate", "query"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 63, 64, 130])
def test_what_is_not_finite_in_both_forms(form, what, bad, at):
    W.test_what_is_not_finite_stays_behind_its_token("delta", what, bad, at)


@pytest.mark.parametrize("N,Dv", [(64, 96), (64, 256), (128, 32)])
def test_other_sizes_stay_with_the_walk_in_one_launch(N, Dv, monkeypatch):
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "DELTA_PIECES_MIN_RUN", 1)
    before = ops.choices["delta_pieces"]
    W.test_delta_walk(W.STEPS[2], 2, 1, N, Dv, False)
    assert ops.choices["delta_pieces"] == before
