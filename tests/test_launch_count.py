"""The count of this package's launches and of the dispatch's choices, for calls of several kernels.  Without a GPU: the libraries are
stand-ins."""

import pytest
import torch


@pytest.fixture
def ops(monkeypatch):
    from kv_cache_optimization_for_llm_b200 import ops

    class Library:
        def __getattr__(self, name):
            return lambda *args: 0

    monkeypatch.setattr(ops, "lib", lambda name: Library())
    monkeypatch.setattr(ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "kernel_status", lambda device: torch.zeros(1, dtype=torch.int32))
    return ops


@pytest.mark.parametrize("k,kernels,chosen", [(1024, 2, ["sgemm_nt", "sgemm_nt_split"]), (512, 1, ["sgemm_nt"])])
def test_float32_products(ops, k, kernels, chosen):
    before, choices = ops.launch_count, ops.choices.copy()
    ops.linear(torch.zeros(3, k), torch.zeros(64, k))
    assert ops.launch_count - before == kernels
    assert dict(ops.choices - choices) == dict.fromkeys(chosen, 1)


def test_grouped_experts(ops, monkeypatch):
    monkeypatch.setattr(ops, "_library_product", lambda x, w, dtype: torch.zeros(x.shape[0], w.shape[0], dtype=dtype))
    E, F, S, H, T = 8, 128, 128, 64, 40
    x = torch.zeros(T, H, dtype=torch.bfloat16)
    before = ops.launch_count
    ops.experts_grouped(x, torch.zeros(2 * (E * F + S), H, dtype=torch.bfloat16), torch.zeros(H, E * F + S, dtype=torch.bfloat16),
                        torch.zeros(T, E), None, E, F, S, 2, 7.0, 7.0, 1.0)
    assert ops.launch_count - before == 5       # lists, gather, both products; join
