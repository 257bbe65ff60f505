"""What prompts in the expanded latent form hold is part of the memory profile that sizes the cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
def test_workspace_is_in_the_profile(wide, monkeypatch):
    from vllm_gcu_b200.engine.llm import LLM
    from vllm_gcu_b200.models import deepseek
    from vllm_gcu_b200.ops import cuda as C
    monkeypatch.setattr(deepseek, "USE_EXPANDED_PROMPTS", wide)
    llm = LLM("tiny-deepseek", device="cuda", cuda_graph_sizes=[4], seed=0, hidden_size=512, intermediate_size=1024,
              num_hidden_layers=2, num_attention_heads=16, num_key_value_heads=16, q_lora_rank=128, kv_lora_rank=512,
              qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128, head_dim=192, moe_intermediate_size=128,
              num_nextn_predict_layers=0, dtype="bfloat16", max_num_seqs=8, max_num_batched_tokens=128,
              max_model_len=512, num_gpu_blocks=64)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    llm.engine.runner._dummy_forward(128)
    torch.cuda.synchronize()
    peak = torch.cuda.max_memory_allocated() - before
    assert (peak > C.LATENT_PREFILL_BYTES) == wide, peak
