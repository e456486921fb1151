"""The largest step of every design finds room in the arena that was made for it, at widths whose float32 products borrow room for three
bfloat16 parts of their rows, and in steps long enough for the scratch of the state memories' launches and of the grouped experts."""

import numpy as np
import pytest
import torch

import tiny_lobuzen
import tiny_nonetar
import tiny_rezusun
import tiny_solulix
import tiny_tevanex
import tiny_zatusun

pytestmark = pytest.mark.gpu

W = 1024
LLAMA = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": 128, "hidden_size": W, "intermediate_size": 8 * W,
         "num_hidden_layers": 2, "num_attention_heads": 16, "num_key_value_heads": 4, "head_dim": 64, "rms_norm_eps": 1e-5,
         "rope_theta": 10000.0, "max_position_embeddings": 4096, "tie_word_embeddings": True, "hidden_act": "silu"}


def _designs():
    lo, no, re, so, te, za = tiny_lobuzen, tiny_nonetar, tiny_rezusun, tiny_solulix, tiny_tevanex, tiny_zatusun
    return {
        "llama": LLAMA,
        "lobuzen_dense": lo.config([lo.layer("attention", lo.attention(16, 4, 64, 64, size=512), lo.dense(8 * W)),
                                    lo.layer("latent_attention", lo.latent(16, 64, 64, 256, size=512), lo.dense(4 * W))], W),
        "lobuzen_experts": lo.config([lo.layer("attention", lo.attention(16, 4, 64, 64, size=512), lo.moe(16, 2, 512, None))], W),
        "nonetar": no.config([no.mamba(32, 64, 128, 8, 8, mlp=no.dense(8 * W)),
                              no.parallel(no.left(16, 4, 64, 64, size=512), no.right(W, 16, 4), mlp=no.dense(4 * W))], W),
        "nonetar_mixers": no.config([no.mamba(64, 64, 128, 8, 8), no.parallel(no.left(16, 4, 64, 64, size=512), no.right(2 * W, 16, 4))], W),
        "rezusun_dense": re.config([re.general(16, 64, 64, ff=8 * W), re.latent(16, 64, 32, 64, 256, 128, ff=4 * W),
                                    re.channel(16, 4, 64, 64, rank=32, gate_rank=64, ff=8 * W)], W),
        "rezusun_loop": re.config([re.channel(16, 4, 64, 64, rank=32, gate_rank=64), re.latent(16, 64, 32, 64, 1024, 512)], W,
                                  loop={"start": 0, "stop": 2, "times": 2}),
        "solulix_dense": so.config([so.delta(16, 4, 64, 64, mlp=so.dense(8 * W)), so.attention(16, 4, 64, 64, mlp=so.dense(4 * W))], W),
        "solulix_experts": so.config([so.delta(32, 4, 64, 64, mlp=so.moe(16, 1, 2, ff=256, shared=W))], W),
        "tevanex": te.config([te.layer("mlstm", te.mlstm(16, 64, 64), te.moe(32, 4, 256, shared_ff=W)),
                              te.layer("attention", te.attention(16, 4, 64, 64, size=512, rot_dims=64), te.moe(8, 2, 512, shared_ff=4 * W))], W),
        "tevanex_mixers": te.config([te.layer("mlstm", te.mlstm(32, 64, 64), None),
                                     te.layer("attention", te.attention(16, 4, 64, 64, size=512, rot_dims=64), None)], W),
        "zatusun": za.config([za.layer("hgrn2", za.hgrn2(16, 64, 64), za.moe(16, 2, 512)),
                              za.layer("latent_attention", za.latent(16, 64, 32, 64, 1024, 512), za.moe(8, 2, 256))], W,
                             loop=(0, 2, 2), max_positions=4096),
    }


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", sorted(_designs()))
def test_the_largest_step_finds_room(name, dtype):
    from kv_cache_optimization_for_llm_b200 import EngineConfig
    from kv_cache_optimization_for_llm_b200.engine.batch import StepEntry
    from kv_cache_optimization_for_llm_b200.engine.runner import ModelRunner
    cfg = _designs()[name]
    T = 1024
    r = ModelRunner(None, EngineConfig(dtype=dtype, page_size=16, num_pages=400, max_num_seqs=4, max_num_batched_tokens=T, max_model_len=1100,
                                       use_cuda_graphs=False), random_init={"config": cfg, "seed": 5, "std": 0.02})
    rng = np.random.default_rng(3)
    ids = rng.integers(0, cfg.get("vocab") or cfg["vocab_size"], T + 8).tolist()
    out = r.step([StepEntry(0, ids[:T], 0, [T - 1])])
    assert bool(torch.isfinite(out).all())
    r.step([StepEntry(0, ids[T:T + 1], T, [0]), StepEntry(1, ids[:T - 3], 0, [T - 4]), StepEntry(2, ids[:2], 0, [1])])
    r.check_status()
    # (an embedding that norms its rows makes them twice: the region of the whole step takes one block more for it)
    assert [h.grown for h in r.arena.halves] == [0, 0] and r.arena.step.grown <= int(name.startswith("solulix")) and r.arena.bypassed == 0
