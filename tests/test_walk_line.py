"""From how many tokens on a step's runs are walked on tensor cores."""

import pytest


@pytest.mark.parametrize("rule,runs,singles,line", [
    ("ssd", 1, 0, 16), ("delta", 1, 0, 16), ("mlstm", 1, 8, 24), ("delta", 1, 8, 40), ("ssd", 4, 8, 36), ("ssd", 32, 0, 36),
    ("mlstm", 16, 0, 36), ("mlstm", 17, 8, 44), ("delta", 16, 0, 39), ("delta", 17, 0, 44), ("delta", 4, 8, 60), ("delta", 32, 8, 60)])
def test_single_tokens_beside_the_runs_and_many_runs_raise_the_line(rule, runs, singles, line):
    from kv_cache_optimization_for_llm_b200 import ops
    assert ops.walk_line(rule, runs, singles) == line


# us in three launches and in one, launched by hand: layers of width 1024
@pytest.mark.parametrize("heads,dv,runs,three,one", [
    (8, 64, [512], 97, 87), (32, 32, [512], 98, 87), (4, 64, [600] + [60] * 10, 99, 88), (8, 32, [600] + [60] * 10, 99, 87),
    (8, 64, [640, 640], 98, 87), (8, 64, [2048], 116, 189), (16, 64, [768], 96, 109), (32, 64, [2048], 192, 286),
    (64, 64, [512] * 4, 312, 358), (32, 64, [1548, 500], 217, 306), (64, 32, [3000], 323, 421), (32, 32, [1024, 1024], 154, 178)])
def test_delta_rule_in_three_launches_where_that_is_faster(heads, dv, runs, three, one):
    from kv_cache_optimization_for_llm_b200 import ops
    assert ops.delta_pieces_faster(runs, heads, dv, False) == (three < one)


def test_captured_steps_do_not_pay_for_launches():
    from kv_cache_optimization_for_llm_b200 import ops
    assert ops.delta_pieces_faster([640, 640], 8, 64, True) and not ops.delta_pieces_faster([640, 640], 8, 64, False)
