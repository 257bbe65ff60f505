"""Latent attention whose projected rows do not end at 16-byte boundaries."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("latent", [36, 512])
def test_generates(latent):
    from vllm_gcu_b200.engine.llm import LLM
    from vllm_gcu_b200.engine.request import SamplingParams
    from vllm_gcu_b200.ops import _native
    llm = LLM("tiny-deepseek", device="cuda", cuda_graph_sizes=[4], seed=0, hidden_size=512, intermediate_size=1024,
              num_hidden_layers=2, num_attention_heads=16, num_key_value_heads=16, q_lora_rank=128,
              kv_lora_rank=latent, qk_nope_head_dim=64, qk_rope_head_dim=64, v_head_dim=64, head_dim=128,
              moe_intermediate_size=128, num_nextn_predict_layers=0, dtype="bfloat16", max_num_seqs=4,
              max_num_batched_tokens=64, max_model_len=128, num_gpu_blocks=64)
    outs = llm.generate([[5, 6, 7, 8, 9], [3]], SamplingParams(max_tokens=4, temperature=0.0, ignore_eos=True))
    torch.cuda.synchronize()
    _native.check_status()
    assert all(len(o.outputs[0].token_ids) == 4 for o in outs)
