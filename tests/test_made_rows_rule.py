"""Which scales the prompt attention over made rows takes on tcgen05: those above zero."""

import math
from types import SimpleNamespace

import pytest
import torch


@pytest.mark.parametrize("scale,wanted", [(0.07, True), (0.0, False), (-0.07, False), (math.nan, False)])
@pytest.mark.parametrize("dk,dv", [(192, 128), (96, 64)])
def test_scales_of_made_rows(scale, wanted, dk, dv):
    from kv_cache_optimization_for_llm_b200 import ops
    batch = SimpleNamespace(num_tokens=300, token_ids=torch.zeros(300))
    assert ops.flash_attention_rows_masked_wanted(batch, 4, 4, dk, dv, 16, torch.bfloat16, made=True, scale=scale) == wanted
