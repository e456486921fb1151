"""Attention of single tokens beside runs: on which stream each launch goes, in which order, and that no kernel begins without waiting for
the launch in front of it.  Without a GPU: the libraries are stand-ins that write down what they are asked."""

import re
from ctypes import c_void_p
from pathlib import Path
from types import SimpleNamespace

import pytest
import torch

MAIN, BESIDE = 0x1000, 0x2000


class _Library:
    def __init__(self, calls, fails=()):
        self.calls, self.fails = calls, fails

    def __getattr__(self, name):
        def call(*args):
            if name.endswith(("_supported", "_tokens_per_tile")):
                return 32
            at = next(a.value for a in reversed(args) if isinstance(a, c_void_p)) if name != "kvb_side_fork" else args[0].value
            if name == "kvb_side_fork":
                args[1]._obj.value = BESIDE
            self.calls.append((name, at))
            return 3 if name in self.fails else 0
        return call


def _step(monkeypatch, fails=(), line=0.0, capturing=False):
    from kv_cache_optimization_for_llm_b200 import ops
    calls = []
    monkeypatch.setattr(ops, "BESIDE_MIN_WORK", line)
    monkeypatch.setattr(ops, "_step_capturing", capturing)
    library = _Library(calls, fails)
    monkeypatch.setattr(ops, "lib", lambda name: library)
    monkeypatch.setattr(ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "sm_count", lambda d: 148)
    monkeypatch.setattr(ops, "_step_stream", c_void_p(MAIN))
    monkeypatch.setattr(ops, "_tokens_per_tile", {})
    ns, n, nq, nkv, d, page = 3, 40, 8, 2, 64, 16
    T = ns + n
    ints = lambda k: torch.zeros(k, dtype=torch.int32)
    batch = SimpleNamespace(decode_only=False, num_single=ns, num_reqs=ns + 1, num_tokens=T, positions=ints(T), token_req=ints(T),
                            q_start=ints(ns + 2), ctx_len=ints(ns + 1), status=ints(1), max_ctx_len=50, token_ids=ints(T),
                            tiles={32: torch.zeros(ns + 2, 4, dtype=torch.int32)}, host={"ctx_len": [9, 9, 9, 50], "q_start": [0, 1, 2, 3, T]})
    pages = torch.zeros(8, nkv, page, d, dtype=torch.bfloat16)
    cos = torch.zeros(64, d // 2)
    ops.attention_step(torch.zeros(T, (nq + 2 * nkv) * d, dtype=torch.bfloat16), pages, pages.clone(), True,
                       torch.zeros(ns + 1, 4, dtype=torch.int32), batch, nq, nkv, d, 0.125, None, 64, cos, cos, d)
    return calls


@pytest.mark.parametrize("line,capturing", [(0.0, False), (1e30, True)])
def test_the_single_tokens_launch_waits_for_all_in_front_and_is_waited_for(monkeypatch, line, capturing):
    assert _step(monkeypatch, line=line, capturing=capturing) == [
        ("kvb_rope_kv_write", MAIN), ("kvb_side_fork", MAIN), ("kvb_paged_flash_attention", MAIN),
        ("kvb_decode_attention_mma", BESIDE), ("kvb_side_join", MAIN)]


def test_below_the_line_one_launch_comes_after_the_other(monkeypatch):
    assert _step(monkeypatch, line=1e30) == [("kvb_decode_attention_mma", MAIN), ("kvb_rope_kv_write", MAIN), ("kvb_paged_flash_attention", MAIN)]


@pytest.mark.parametrize("width,singles,runs,wanted", [     # (start, tokens) of the runs
    (2048, 52, [(108, 64)], False), (2048, 6, [(1154, 446)], False), (3072, 12, [(0, 233), (0, 98)], False), (3072, 58, [(0, 343)], True),
    (2048, 4, [(661, 121), (1166, 511)], True), (3072, 40, [(512, 701)], True)])
def test_side_by_side_where_the_host_is_not_the_bound(monkeypatch, width, singles, runs, wanted):
    from kv_cache_optimization_for_llm_b200 import ops
    monkeypatch.setattr(ops, "_step_capturing", False)
    batch = SimpleNamespace(num_single=singles, num_tokens=singles + sum(n for _, n in runs),
                            host={"ctx_len": [9000] * singles + [s + n for s, n in runs]})
    assert ops.attention_beside_wanted(batch, width) == wanted
    assert ops.attention_beside_wanted(batch, width) == wanted


@pytest.mark.parametrize("fails", ["kvb_paged_flash_attention", "kvb_decode_attention_mma"])
def test_a_launch_that_fails_leaves_no_fork_open(monkeypatch, fails):
    from kv_cache_optimization_for_llm_b200 import ops
    calls = []
    with pytest.raises(ops.KernelError):
        calls = _step(monkeypatch, (fails,))
    library = ops.lib("decode_attention")
    assert [c[0] for c in library.calls if "side" in c[0]] == ["kvb_side_fork", "kvb_side_join"] and not calls


def test_every_kernel_that_may_begin_early_waits_for_the_launch_in_front():
    """A grid that was let in by ``griddepcontrol.launch_dependents`` finds memory in order only behind ``griddepcontrol.wait``: no kernel makes
    that wait depend on a condition of the launch."""
    kernels = Path(__file__).resolve().parent.parent / "kv_cache_optimization_for_llm_b200" / "csrc" / "kernels"
    for path in sorted(kernels.glob("*.cu*")):
        text = path.read_text()
        assert not re.search(r"\b(if|else)\b[^;{\n]*pdl_wait\(\)", text), path.name
        assert text.count("griddepcontrol") == (2 if path.name == "common.cuh" else 0), path.name
