"""Work that users of the serving engine have it do, as cases that can be timed and checked.

A case is one engine step of a model: the decode step of a batch, the prefill of prompts (or of a
chunk behind cached tokens), or both in one step.  Models keep the layer sizes of the benchmark
configurations with fewer layers and a smaller vocabulary:

* ``llama``    Llama-3-8B layers (grouped-query attention, dense feed-forward), bf16
* ``gptq``     the same layers from a 4-bit GPTQ checkpoint, groups of 128
* ``fp8``      the same layers from an fp8 checkpoint, per-channel weights, per-token activations
* ``moe``      Qwen3-30B-A3B layers (QK norm, 128 experts, 8 per token), bf16
* ``mla``      DeepSeek-V3 layers (latent attention of 128 heads, grouped sigmoid routing, shared
               expert), one dense layer and one with a rank's share of the experts, bf16

A decode step goes through ``ModelRunner.execute``, as the engine issues it: input copies, CUDA graph,
sampling.  Steps with prompts call the model and its LM head with the step's metadata, as the runner
does for every step that is not a pure decode.  Outputs are the logits of every row that would be
sampled.
"""
from __future__ import annotations

import math

import torch

BLOCK = 16
VOCAB = 32768
GROUP = 128                       # columns per scale of a 4-bit weight
EPS = 1e-5

#: width, heads, key heads, head dimension, feed-forward, layers
SIZES = {
    "llama": dict(H=4096, heads=32, kv=8, D=128, ff=14336, layers=8, theta=5e5),
    "gptq": dict(H=4096, heads=32, kv=8, D=128, ff=14336, layers=8, theta=5e5),
    "fp8": dict(H=4096, heads=32, kv=8, D=128, ff=14336, layers=4, theta=5e5),
    "moe": dict(H=2048, heads=32, kv=4, D=128, ff=768, layers=4, theta=1e6, experts=128, top=8),
    "mla": dict(H=7168, heads=128, q_rank=1536, rank=512, nope=128, rope=64, D=128, dense_ff=18432,
                ff=2048, layers=2, theta=1e4, experts=32, top=8, groups=8, keep=4, factor=2.5),
}


def listed() -> list[dict]:
    def case(name, family, decodes=0, context=0, prompts=0, new=0, cached=0):
        return dict(name=name, family=family, decodes=decodes, context=context, prompts=prompts,
                    new=new, cached=cached)
    return [
        # one user waits for each token of an answer
        case("llama-decode-1", "llama", 1, 640),
        # the benchmark's decode step: 256 requests behind 1024 tokens of prompt
        case("llama-decode-256", "llama", 256, 1152),
        # one short chat prompt: time to first token
        case("llama-prefill-301", "llama", prompts=1, new=301),
        # the benchmark's mixed step: a full token budget of prompts beside running requests
        case("llama-mixed-7x1024-200", "llama", 200, 1100, 7, 1024),
        # one long document
        case("llama-prefill-8192", "llama", prompts=1, new=8192),
        # a 4-bit checkpoint on a small server, a few users and many
        case("gptq-decode-12", "gptq", 12, 900),
        case("gptq-decode-96", "gptq", 96, 1000),
        # an fp8 checkpoint at the concurrency of a serving run
        case("fp8-decode-64", "fp8", 64, 1500),
        # experts: decode at medium concurrency, prompts of the serving configuration (2048 tokens)
        case("moe-decode-64", "moe", 64, 2304),
        case("moe-prefill-2x2048", "moe", prompts=2, new=2048),
        # latent attention: 128 concurrent requests of 1024 + 1024 tokens, and prompts of 1024
        case("mla-decode-128", "mla", 128, 1536),
        case("mla-prefill-2x1024", "mla", prompts=2, new=1024),
    ]


def draw(rng) -> dict:
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    family = rng.choice(["llama", "llama", "gptq", "fp8", "moe", "mla"])
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "mixed"])
    c = dict(family=family, decodes=0, context=0, prompts=0, new=0, cached=0)
    # prompt tokens of a step
    budget = {"mla": 2048, "moe": 4096}.get(family, 8192 if kind == "prefill" else 7168)
    if kind != "prefill":
        c["decodes"] = log(1, 128 if family == "mla" else 256)
        c["context"] = log(33, 1536 if family == "mla" else 2304)
        while c["decodes"] * c["context"] > 256 * 1152:
            c["context"] = c["context"] * 2 // 3
    if kind != "decode":
        new = log(17, budget)
        c["prompts"] = max(1, min(rng.choice([1, 1, 2, 3, 5, 8]), budget // new))
        c["new"] = new
        if rng.random() < 0.3:       # a later chunk of a long prompt, or behind a cached prefix
            c["cached"] = min(log(1, 128) * BLOCK, 8192 - min(new * c["prompts"], 8176))
    return c


def _contexts(case) -> list[int]:
    """Keys of every decoding request after this step: uneven, as requests finish and start."""
    c = case["context"]
    return [max(2, c - i * 61 % (c // 8 + 1)) for i in range(case["decodes"])]


def _portions(case) -> list[int]:
    n = case["new"]
    return [max(2, n - i * 17 % (n // 16 + 1)) for i in range(case["prompts"])]


# -- weights ---------------------------------------------------------------------------------
def _gen(seed: int, *what: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    h = seed
    for w in what:
        h = (h * 1000003 + w + 1) & 0x7FFFFFFF
    g.manual_seed(h)
    return g


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)


def _norm_weight(g, n):
    return (1.0 + 0.1 * torch.randn(n, device="cuda", generator=g)).to(torch.bfloat16)


def _matrix(family, g, n, k, gain):
    """One projection ``[n, k]`` as a checkpoint stores it: {suffix: tensor}."""
    std = gain / math.sqrt(k)
    if family == "gptq":
        q = torch.randint(-2**31, 2**31, (k // 8, n), device="cuda", generator=g).to(torch.int32)
        s = (std / 4.61 * (0.5 + torch.rand(k // GROUP, n, device="cuda", generator=g)))
        # zero points 7 and 8 (stored less one), so that the weights of a group have no common part
        z = torch.randint(0, 256, (k // GROUP, n // 8), device="cuda", generator=g)
        z = sum((6 + (z >> i & 1)) << 4 * i for i in range(8))
        return {"qweight": q, "scales": s.to(torch.bfloat16), "qzeros": z.to(torch.int32)}
    if family == "fp8":
        s = std * (0.5 + torch.rand(n, 1, device="cuda", generator=g))
        return {"weight": _normal(g, n, k).to(torch.float8_e4m3fn), "weight_scale": s}
    return {"weight": _normal(g, n, k, std=std)}


def _wide(m: dict) -> torch.Tensor:
    """The matrix that ``_matrix`` stores, in 64 bits."""
    if "qweight" in m:
        shifts = torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)
        q = (m["qweight"][:, None, :] >> shifts[None, :, None]) & 15
        q = q.reshape(-1, m["qweight"].shape[1]).double()
        z = (m["qzeros"][:, :, None] >> shifts & 15).reshape(q.shape[0] // GROUP, -1).double() + 1
        s = m["scales"].double()
        return ((q.view(-1, GROUP, q.shape[1]) - z[:, None]) * s[:, None]).view_as(q).t()
    w = m["weight"].double()
    return w * m["weight_scale"].double() if "weight_scale" in m else w


# input projections have rows of unit gain, output projections give a sublayer a part of the stream;
# a routed expert gives a small one, as behind a trained router, and so do sublayers behind rows of
# fp8, of which a step of a bf16 number moves many
_IN = 1.25
_ATT = {"llama": 3.0, "gptq": 3.0, "fp8": 1.0, "moe": 3.0, "mla": 3.0}
_FF = {"llama": 0.6, "gptq": 0.6, "fp8": 0.2, "moe": 0.2, "mla": 0.6}
_EXPERT = {"moe": 0.2, "mla": 0.1}


def _projections(case, layer):
    """Name -> (rows, columns, gain) of the layer's matrices outside of the routed experts."""
    s, f = SIZES[case["family"]], case["family"]
    H = s["H"]
    if f == "mla":
        qk = s["nope"] + s["rope"]
        p = {"self_attn.q_a_proj": (s["q_rank"], H, _IN),
             "self_attn.q_b_proj": (s["heads"] * qk, s["q_rank"], _IN),
             "self_attn.kv_a_proj_with_mqa": (s["rank"] + s["rope"], H, _IN),
             "self_attn.kv_b_proj": (s["heads"] * (s["nope"] + s["D"]), s["rank"], _IN),
             "self_attn.o_proj": (H, s["heads"] * s["D"], _ATT[f])}
    else:
        p = {"self_attn.q_proj": (s["heads"] * s["D"], H, _IN),
             "self_attn.k_proj": (s["kv"] * s["D"], H, _IN),
             "self_attn.v_proj": (s["kv"] * s["D"], H, _IN),
             "self_attn.o_proj": (H, s["heads"] * s["D"], _ATT[f])}
    if f == "moe" or f == "mla" and layer > 0:
        p["mlp.gate"] = (s["experts"], H, _IN)
        if f == "mla":
            p.update({"mlp.shared_experts.gate_proj": (s["ff"], H, _IN),
                      "mlp.shared_experts.up_proj": (s["ff"], H, _IN),
                      "mlp.shared_experts.down_proj": (H, s["ff"], _FF[f])})
    else:
        ff = s["dense_ff"] if f == "mla" else s["ff"]
        p.update({"mlp.gate_proj": (ff, H, _IN), "mlp.up_proj": (ff, H, _IN),
                  "mlp.down_proj": (H, ff, _FF[f])})
    return p


def _norms(case):
    s, f = SIZES[case["family"]], case["family"]
    n = {"input_layernorm": s["H"], "post_attention_layernorm": s["H"]}
    if f == "moe":
        n.update({"self_attn.q_norm": s["D"], "self_attn.k_norm": s["D"]})
    if f == "mla":
        n.update({"self_attn.q_a_layernorm": s["q_rank"], "self_attn.kv_a_layernorm": s["rank"]})
    return n


def _layer(case, seed, i):
    """Layer i as a checkpoint has it: ({name: norm}, {name: matrix}, experts or None)."""
    s = SIZES[case["family"]]
    norms = {n: _norm_weight(_gen(seed, i, 100 + j), k)
             for j, (n, k) in enumerate(_norms(case).items())}
    mats = {n: _matrix(case["family"] if n != "mlp.gate" else "", _gen(seed, i, j), *shape)
            for j, (n, shape) in enumerate(_projections(case, i).items())}
    experts = None
    if "mlp.gate" in mats:
        E, H, F = s["experts"], s["H"], s["ff"]
        experts = (_normal(_gen(seed, i, 200), E, 2 * F, H, std=_IN / math.sqrt(H)),
                   _normal(_gen(seed, i, 201), E, H, F,
                           std=_EXPERT[case["family"]] / math.sqrt(F)))
    return norms, mats, experts


def _ends(case, seed):
    """Embedding, final norm, LM head."""
    H = SIZES[case["family"]]["H"]
    return (_normal(_gen(seed, 300), VOCAB, H), _norm_weight(_gen(seed, 301), H),
            _normal(_gen(seed, 302), VOCAB, H, std=_IN / math.sqrt(H)))


def _bias(case, seed, i):
    return 0.05 * torch.randn(SIZES[case["family"]]["experts"], device="cuda",
                              generator=_gen(seed, i, 202))


def _checkpoint(case, seed):
    emb, norm, head = _ends(case, seed)
    yield "model.embed_tokens.weight", emb
    yield "model.norm.weight", norm
    yield "lm_head.weight", head
    for i in range(SIZES[case["family"]]["layers"]):
        norms, mats, experts = _layer(case, seed, i)
        p = f"model.layers.{i}."
        for n, t in norms.items():
            yield p + n + ".weight", t
        for n, m in mats.items():
            for suffix, t in m.items():
                yield p + n + "." + suffix, t
        if experts is not None:
            yield p + "mlp.experts.gate_up_proj", experts[0]
            yield p + "mlp.experts.down_proj", experts[1]
            if case["family"] == "mla":
                yield p + "mlp.gate.e_score_correction_bias", _bias(case, seed, i)


# -- inputs ----------------------------------------------------------------------------------
def _tokens(case, seed) -> torch.Tensor:
    n = case["decodes"] + sum(_portions(case))
    return torch.randint(0, VOCAB, (n,), generator=torch.Generator().manual_seed(seed + 17))


def _past(case) -> list[int]:
    """Tokens of every request that lie in the cache before the step."""
    return [c - 1 for c in _contexts(case)] + [case["cached"]] * case["prompts"]


def _cached(case, seed, i) -> torch.Tensor:
    """Layer i's cache rows of the past tokens, request after request: ``[2, n, kv, D]`` (keys with
    their positions, values) or ``[n, rank + rope]``."""
    s, n = SIZES[case["family"]], sum(_past(case))
    if case["family"] == "mla":
        return _normal(_gen(seed, i, 400), n, s["rank"] + s["rope"])
    return _normal(_gen(seed, i, 400), 2, n, s["kv"], s["D"])


def _model_config(case):
    from vllm_gcu_b200.config import ModelConfig, preset
    f, s = case["family"], SIZES[case["family"]]
    if f == "moe":
        return preset("qwen3-30b-a3b", num_hidden_layers=s["layers"], vocab_size=VOCAB,
                      rms_norm_eps=EPS, max_position_embeddings=16384)
    if f == "mla":
        return preset("deepseek-v3", num_hidden_layers=s["layers"], vocab_size=VOCAB,
                      num_experts=s["experts"], first_k_dense_replace=1, rms_norm_eps=EPS,
                      num_nextn_predict_layers=0, max_position_embeddings=16384)
    kw = {} if f == "llama" else dict(
        quantization=f, quant_config={"bits": 4, "group_size": GROUP} if f == "gptq" else {})
    mc = preset("llama-3-8b", num_hidden_layers=s["layers"], vocab_size=VOCAB,
                max_position_embeddings=16384, **kw)
    assert isinstance(mc, ModelConfig)
    return mc


class _Step:
    """A model with its caches, and one step of it."""

    def __init__(self, case, seed):
        from vllm_gcu_b200.config import CacheConfig, EngineConfig, SchedulerConfig
        from vllm_gcu_b200.engine.model_runner import ModelRunner
        from vllm_gcu_b200.engine.request import Request, SamplingParams
        from vllm_gcu_b200.engine.scheduler import ScheduledRequest, SchedulerOutput
        from vllm_gcu_b200.layers.attention import AttentionMetadata
        from vllm_gcu_b200.models import build_model
        dev = torch.device("cuda", torch.cuda.current_device())
        mc = _model_config(case)
        model = build_model(mc, dev)
        model.load_weights(_checkpoint(case, seed))
        model.eval()
        past, ids = _past(case), _tokens(case, seed)
        nd, new = case["decodes"], _portions(case)
        steps = [1] * nd + new
        total = [a + b for a, b in zip(past, steps)]
        blocks = [-(-t // BLOCK) for t in total]
        first = [1 + sum(blocks[:i]) for i in range(len(blocks))]       # block 0 stays unused
        cfg = EngineConfig(
            model=mc, cache=CacheConfig(block_size=BLOCK, num_gpu_blocks=1 + sum(blocks)),
            scheduler=SchedulerConfig(max_num_seqs=max(nd, 1),
                                      max_num_batched_tokens=max(sum(steps), 16),
                                      max_model_len=max(total) + 16),
            additional_config={"keep_graph_logits": True})
        self.runner = runner = ModelRunner(cfg, model, dev)
        runner.init_kv_cache(1 + sum(blocks))
        slots = torch.cat([torch.arange(n) + f * BLOCK for n, f in zip(past, first)]).to(dev)
        for i, cache in enumerate(runner.kv_caches):
            rows = _cached(case, seed, i)
            if cache.dim() == 3:
                cache.view(-1, cache.shape[-1])[slots] = rows
            else:
                cache.view(2, -1, *cache.shape[3:])[:, slots] = rows
        self.pure = case["prompts"] == 0
        if self.pure:
            runner.capture_graphs([nd])
            sched = []
            for i in range(nd):
                r = Request(f"r{i}", [0] * past[i] + [int(ids[i])],
                            SamplingParams(temperature=0.0, max_tokens=1 << 20, ignore_eos=True))
                r.block_ids = list(range(first[i], first[i] + blocks[i]))
                sched.append(ScheduledRequest(r, past[i], 1, [], True, will_sample=True))
            self.step = SchedulerOutput(scheduled=sched, total_tokens=nd)
            return
        pos = torch.cat([torch.arange(n) + p for n, p in zip(steps, past)])
        slot = torch.cat([torch.arange(n) + p + f * BLOCK for n, p, f in zip(steps, past, first)])
        table = torch.zeros(len(steps), max(blocks), dtype=torch.int32)
        for i, (f, b) in enumerate(zip(first, blocks)):
            table[i, :b] = torch.arange(f, f + b)
        cu = torch.tensor([0] + new).cumsum(0)
        self.model, self.ids = model, ids.to(dev)
        self.last = torch.cat([torch.arange(nd), nd + cu[1:] - 1]).to(dev)
        self.md = AttentionMetadata(
            num_tokens=sum(steps), num_decodes=nd, num_prefills=len(new), num_decode_tokens=nd,
            positions=pos.to(dev), slot_mapping=slot.to(dev), block_tables=table.to(dev),
            seq_lens=torch.tensor(total, dtype=torch.int32, device=dev),
            cu_q_prefill=cu.to(torch.int32).to(dev), num_q_tiles=sum(-(-n // 64) for n in new),
            num_q_tiles_128=sum(-(-n // 128) for n in new), max_seq_len=max(total),
            decode_splits=0, q_lens_cpu=steps, seq_lens_cpu=total)

    def run(self):
        if self.pure:
            key = (self.step.total_tokens, self.runner.step_counter & 1, True)
            self.runner.execute(self.step)
            return {"logits": self.runner.graph_logits[key]}
        with torch.inference_mode():
            h = self.model(self.ids, self.md, self.runner.kv_caches)
            return {"logits": self.model.compute_logits(h.index_select(0, self.last))}


def prepare(case, seed):
    return _Step(case, seed)


def run(state):
    return state.run()


# -- what a pass cannot do without -------------------------------------------------------------
def work(case) -> dict:
    f, s = case["family"], SIZES[case["family"]]
    T = case["decodes"] + sum(_portions(case))
    rows = case["decodes"] + case["prompts"]
    size = {"gptq": 0.5 + 2 * 2 / GROUP, "fp8": 1.0}.get(f, 2.0)
    nbytes, flops = 0.0, 0.0
    for i in range(s["layers"]):
        for name, (n, k, _) in _projections(case, i).items():
            nbytes += n * k * (2.0 if name == "mlp.gate" else size)
            flops += 2.0 * n * k * T
        if "mlp.gate" in _projections(case, i):
            one = 3 * s["ff"] * s["H"]
            touched = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** T)
            nbytes += 2.0 * one * touched
            flops += 2.0 * one * s["top"] * T
    pairs = sum(_contexts(case)) + sum(n * case["cached"] + n * (n + 1) // 2
                                       for n in _portions(case))
    keys = sum(_past(case)) + T
    if f == "mla":
        # scores and values: over latent rows in a decode, per head where prompts are long
        flops += s["layers"] * 2.0 * s["heads"] * pairs * (s["nope"] + s["rope"] + s["D"])
        nbytes += s["layers"] * 2.0 * keys * (s["rank"] + s["rope"])
    else:
        flops += s["layers"] * 4.0 * s["heads"] * s["D"] * pairs
        nbytes += s["layers"] * 4.0 * keys * s["kv"] * s["D"]
    flops += 2.0 * rows * VOCAB * s["H"]
    nbytes += 2.0 * VOCAB * s["H"] + 2.0 * T * s["H"] + 2.0 * rows * VOCAB
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # bf16 activations through the layers (measured against 64 bits: 0.5 to 1.5 per cent); fp8 rounds
    # every activation to 4 bits, and a routing tie gives a token another expert
    return {"rel": 0.03, "max": 0.9}


# -- the same step in 64 bits --------------------------------------------------------------------
def _rms(x, w, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _rotate(x, pos, theta, neighbours):
    """x ``[T, heads, R]``: pairs (i, i + R/2), or neighbours."""
    R = x.shape[-1]
    inv = theta ** (-torch.arange(0, R, 2, device="cuda", dtype=torch.float64) / R)
    a = pos.double()[:, None] * inv
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = (x[..., 0::2], x[..., 1::2]) if neighbours else (x[..., :R // 2], x[..., R // 2:])
    y = (u * c - v * s, u * s + v * c)
    return torch.stack(y, -1).flatten(-2) if neighbours else torch.cat(y, -1)


def _attend(q, k, v, scale):
    """q ``[n, heads, Dk]``, k ``[m, kv, Dk]``, v ``[m, kv, Dv]``: the last n of m positions."""
    n, m, kv = q.shape[0], k.shape[0], k.shape[1]
    g = q.shape[1] // kv
    out = torch.empty(n, q.shape[1], v.shape[-1], dtype=torch.float64, device="cuda")
    hide = None
    if n > 1:
        hide = torch.ones(n, m, dtype=torch.bool, device="cuda").triu(m - n + 1)
    per = kv if n * m * g * kv < 1 << 27 else 1
    for h in range(0, kv, per):
        qh = q[:, h * g:(h + per) * g].reshape(n, per, g, -1).permute(1, 2, 0, 3)
        for j in range(0, g, g if per > 1 or n * m * g < 1 << 27 else 1):
            w = g if per > 1 or n * m * g < 1 << 27 else 1
            sc = qh[:, j:j + w].reshape(per, w * n, -1) @ k[:, h:h + per].permute(1, 2, 0) * scale
            if hide is not None:
                sc.view(per, w, n, m).masked_fill_(hide, float("-inf"))
            o = torch.softmax(sc, -1) @ v[:, h:h + per].transpose(0, 1)
            out[:, h * g:(h + per) * g].view(n, per, g, -1)[:, :, j:j + w] = \
                o.view(per, w, n, -1).permute(2, 0, 1, 3)
    return out


def _route(case, z, bias):
    s = SIZES[case["family"]]
    if case["family"] == "moe":
        w, e = torch.softmax(z, -1).topk(s["top"], -1)
        return w / w.sum(-1, keepdim=True), e
    p = torch.sigmoid(z)
    sel = p + bias.double()
    best = sel.view(-1, s["groups"], s["experts"] // s["groups"]).topk(2, -1).values.sum(-1)
    keep = torch.zeros_like(best).scatter_(1, best.topk(s["keep"], -1).indices, 1.0)
    sel = sel.masked_fill(keep.repeat_interleave(s["experts"] // s["groups"], 1) == 0, -math.inf)
    e = sel.topk(s["top"], -1).indices
    w = p.gather(1, e)
    return w / w.sum(-1, keepdim=True) * s["factor"], e


def _gated(x, gate, up, down):
    return (torch.nn.functional.silu(x @ gate.t()) * (x @ up.t())) @ down.t()


@torch.inference_mode()
def exact(case, seed):
    f, s = case["family"], SIZES[case["family"]]
    past, new = _past(case), [1] * case["decodes"] + _portions(case)
    pos = torch.cat([torch.arange(n) + p for n, p in zip(new, past)]).cuda()
    emb, norm, head = _ends(case, seed)
    x = emb[_tokens(case, seed).cuda()].double()
    T, D = x.shape[0], s["D"]
    for i in range(s["layers"]):
        norms, mats, experts = _layer(case, seed, i)
        w = {n: _wide(m) for n, m in mats.items() if n != "self_attn.kv_b_proj"}
        rows = _cached(case, seed, i)
        h = _rms(x, norms["input_layernorm"])
        if f == "mla":
            L, R, N = s["rank"], s["rope"], s["heads"]
            q = _rms(h @ w["self_attn.q_a_proj"].t(), norms["self_attn.q_a_layernorm"], EPS)
            q = (q @ w["self_attn.q_b_proj"].t()).view(T, N, -1)
            kv = h @ w["self_attn.kv_a_proj_with_mqa"].t()
            c = _rms(kv[:, :L], norms["self_attn.kv_a_layernorm"])
            pe = _rotate(kv[:, None, L:], pos, s["theta"], True)[:, 0]
            b = _wide(mats["self_attn.kv_b_proj"]).view(N, -1, L)
            q = torch.cat([torch.einsum("tnd,ndl->tnl", q[..., :s["nope"]], b[:, :s["nope"]]),
                           _rotate(q[..., s["nope"]:], pos, s["theta"], True)], -1)
            k = torch.cat([c, pe], -1)
            scale = (s["nope"] + R) ** -0.5
        else:
            q = (h @ w["self_attn.q_proj"].t()).view(T, -1, D)
            k = (h @ w["self_attn.k_proj"].t()).view(T, -1, D)
            v = (h @ w["self_attn.v_proj"].t()).view(T, -1, D)
            if f == "moe":
                q, k = (_rms(a, norms[f"self_attn.{n}_norm"]) for a, n in ((q, "q"), (k, "k")))
            q, k = (_rotate(a, pos, s["theta"], False) for a in (q, k))
            scale = D ** -0.5
        out, at, seen = [], 0, 0
        for n, p in zip(new, past):
            qi, t = q[at:at + n], slice(at, at + n)
            if f == "mla":
                ki = torch.cat([rows[seen:seen + p].double(), k[t]])[:, None]
                out.append(_attend(qi, ki, ki[..., :s["rank"]], scale))
            else:
                out.append(_attend(qi, torch.cat([rows[0, seen:seen + p].double(), k[t]]),
                                   torch.cat([rows[1, seen:seen + p].double(), v[t]]), scale))
            at, seen = at + n, seen + p
        o = torch.cat(out)
        if f == "mla":
            o = torch.einsum("tnl,nvl->tnv", o, b[:, s["nope"]:])
        x = x + o.reshape(T, -1) @ w["self_attn.o_proj"].t()
        h = _rms(x, norms["post_attention_layernorm"])
        if experts is None:
            x = x + _gated(h, *(w[f"mlp.{n}_proj"] for n in ("gate", "up", "down")))
            continue
        rw, re = _route(case, h @ w["mlp.gate"].t(), _bias(case, seed, i))
        y = torch.zeros_like(x)
        for e in range(s["experts"]):
            t, j = (re == e).nonzero(as_tuple=True)
            g, d = experts[0][e].double(), experts[1][e].double()
            y.index_add_(0, t, _gated(h[t], g[:s["ff"]], g[s["ff"]:], d) * rw[t, j, None])
        if f == "mla":
            y += _gated(h, *(w[f"mlp.shared_experts.{n}_proj"] for n in ("gate", "up", "down")))
        x = x + y
    last = torch.tensor(new).cumsum(0).cuda() - 1
    return {"logits": _rms(x[last], norm) @ head.double().t()}
