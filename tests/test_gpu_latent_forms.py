"""Latent attention of prompts in a model: steps run in the absorbed form, and with USE_EXPANDED_PROMPTS long ones in
the expanded form beside decoding requests and short ones, to the same logits but for rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_prompts_in_both_forms(monkeypatch):
    from vllm_gcu_b200.engine.llm import LLM
    from vllm_gcu_b200.engine.request import SamplingParams
    from vllm_gcu_b200.models import deepseek
    from vllm_gcu_b200.ops import _native
    from vllm_gcu_b200.ops import cuda as C
    # (no experts: a choice between nearly equal ones would turn a rounding into another layer)
    kw = dict(hidden_size=512, intermediate_size=1024, num_hidden_layers=2, first_k_dense_replace=2,
              num_attention_heads=16, num_key_value_heads=16, q_lora_rank=128, kv_lora_rank=512,
              qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128, head_dim=192,
              moe_intermediate_size=128, num_nextn_predict_layers=0, dtype="bfloat16",
              max_num_seqs=8, max_num_batched_tokens=640, max_model_len=1024, num_gpu_blocks=512)
    g = torch.Generator().manual_seed(0)
    prompts = [torch.randint(0, 1024, (n,), generator=g).tolist() for n in (400, 70, 300, 7)]
    calls, real = [], C.latent_prefill
    monkeypatch.setattr(C, "latent_prefill", lambda *a, **k: (calls.append(1), real(*a, **k))[1])
    got = {}
    for wide in (False, True):
        if wide:
            monkeypatch.setattr(deepseek, "USE_EXPANDED_PROMPTS", True)
        calls.clear()
        llm = LLM("tiny-deepseek", device="cuda", cuda_graph_sizes=[4, 8], seed=0, **kw)
        llm.generate(prompts, SamplingParams(max_tokens=6, temperature=0.0, ignore_eos=True))
        llm.engine.runner.keep_logits = True
        llm.engine.runner.graphs = {}
        llm.generate(prompts[1:], SamplingParams(max_tokens=1, temperature=0.0, ignore_eos=True))
        torch.cuda.synchronize()
        _native.check_status()
        assert bool(calls) == wide
        got[wide] = llm.engine.runner.last_logits.float().cpu()
        del llm
    err, size = (got[True] - got[False]).abs().max().item(), got[False].std().item()
    assert err < 0.05 * size + 0.03, (err, size)
