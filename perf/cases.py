"""What the framework is timed on: the blocks that an engine step consists of, over the sizes that serving gives them, and a small model
served from end to end.

A case of kind ``mlp``, ``attention``, ``experts``, ``gdn`` or ``mla`` is one call of that layer (``onecat_vllm.layers``) on the tokens of
one engine step, with the weights loaded in their checkpoint format and the caches and the step's metadata as the runner lays them out: pages
in no particular order, every request with its own context length. ``serve`` loads a checkpoint folder into an engine and replays given
tokens through it: prompts in one step, then a token per request and step. Widths are those of the benchmark configurations."""
import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

from onecat_vllm.config import ModelConfig
from onecat_vllm.engine.replay import TraceReplay
from onecat_vllm.layers.attention import Attention
from onecat_vllm.layers.gdn import GatedDeltaNet
from onecat_vllm.layers.mla import MLAAttention
from onecat_vllm.layers.mlp import MLP
from onecat_vllm.layers.moe import FusedMoE
from onecat_vllm.loader.weights import process_weights_after_loading
from onecat_vllm.worker.attn_metadata import AttentionMetadata

DEV = "cuda"
BLOCK = 16          # tokens of a cache page
EPS = 1e-6
THETA = 1e6
MAX_POS = 40960
MAX_COST = 2.0 * 8192 * 3 * 5120 * 17408   # operations of the largest listed case


def listed():
    mlp = dict(kind="mlp", hidden=5120, inter=17408)
    attn = dict(kind="attention", hidden=5120, heads=40, kv_heads=8, dim=128, gated=False, quant="awq", kv="bf16")
    return [
        # one user, one token at a time: the feed-forward of a 4-bit 27B model reads its weights for a single row
        dict(mlp, name="mlp-awq-1", quant="awq", tokens=1),
        # the same block for 64 concurrent requests, the headline workload's decode step
        dict(mlp, name="mlp-awq-64", quant="awq", tokens=64),
        # a mixed step of that workload: a fresh 1024-token prompt beside 63 decoding requests
        dict(mlp, name="mlp-awq-1087", quant="awq", tokens=1087),
        # a full prefill step (the 8192-token budget) of a model with unquantised weights; the largest case
        dict(mlp, name="mlp-bf16-8192", quant="bf16", tokens=8192),
        # decoding: 64 requests half-way through 1024 in / 256 out
        dict(attn, name="attn-decode-64", requests=64, context=1152, prompts=0, prompt=0),
        # the mixed step: one of the 64 requests brings its prompt
        dict(attn, name="attn-mixed-64", requests=64, context=1152, prompts=1, prompt=1024),
        # a long prompt in one step
        dict(attn, name="attn-prompt-8192", requests=1, context=8192, prompts=1, prompt=8192),
        # a few users with long documents, cache in 8 bits
        dict(attn, name="attn-long-fp8kv-8", requests=8, context=32768, prompts=0, prompt=0, kv="fp8"),
        # decode step of a mixture of 256 experts with 256 concurrent requests, block-scaled fp8 weights
        dict(kind="experts", name="experts-fp8-256", quant="fp8", tokens=256, hidden=2048, inter=512, experts=256, top_k=8),
        # a step of a hybrid model's recurrent layer: three prompts of odd lengths beside 13 decoding requests
        dict(kind="gdn", name="gdn-mixed-16", requests=16, prompts=3, prompt=1500, hidden=5120, key_heads=16, value_heads=48),
        # latent attention with 128 heads, decoding
        dict(kind="mla", name="mla-decode-32", requests=32, context=4096, prompts=0, prompt=0, heads=128, hidden=7168),
        # a small 4-bit model served: five prompts, eight tokens each
        dict(kind="serve", name="serve-small-5", requests=5, prompt=120, steps=8, layers=2, hidden=1024, inter=2048, vocab=4096),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["mlp", "mlp", "attention", "attention", "attention", "experts", "gdn", "mla", "serve"])
    if kind == "mlp":
        hidden, inter = rng.choice([(5120, 17408), (2048, 5632), (4096, 12288), (7168, 18432), (1024, 2048)])
        most = min(8192, int(MAX_COST / (6 * hidden * inter)))
        return dict(kind=kind, hidden=hidden, inter=inter, quant=rng.choice(["awq", "awq", "bf16", "fp8"]), tokens=log(1, most))
    if kind == "attention":
        hidden, heads, kv_heads, dim, gated = rng.choice([(5120, 40, 8, 128, False), (5120, 40, 8, 128, False), (5120, 24, 4, 256, True), (2048, 16, 2, 256, True),
                                                          (2048, 16, 8, 128, False)])
        c = dict(kind=kind, hidden=hidden, heads=heads, kv_heads=kv_heads, dim=dim, gated=gated, quant=rng.choice(["awq", "bf16"]), kv=rng.choice(["bf16", "bf16", "fp8"]))
    elif kind == "experts":
        hidden, inter, experts, top_k = rng.choice([(2048, 512, 256, 8), (2048, 768, 128, 8), (4096, 1536, 64, 6)])
        return dict(kind=kind, quant=rng.choice(["fp8", "mxfp4", "bf16"]), tokens=log(1, 8192), hidden=hidden, inter=inter, experts=experts, top_k=top_k)
    elif kind == "gdn":
        requests = log(1, 64)
        prompts = rng.randint(0, min(requests, 4))
        hidden, value_heads = rng.choice([(5120, 48), (2048, 32)])
        return dict(kind=kind, requests=requests, prompts=prompts, prompt=log(2, 8000 // prompts) if prompts else 0, hidden=hidden, key_heads=16, value_heads=value_heads)
    elif kind == "mla":
        heads = rng.choice([16, 64, 128])
        c = dict(kind=kind, heads=heads, hidden=7168 if heads == 128 else 2048)
    else:
        return dict(kind=kind, requests=log(1, 24), prompt=log(2, 500), steps=rng.randint(1, 16), layers=rng.randint(1, 4), hidden=1024, inter=rng.choice([2048, 4096]), vocab=4096)
    # a step of either attention: decoding requests, and in half of the cases one to four prompts (the last chunk of a context)
    context = log(16, 32768)
    requests = log(1, max(1, min(256, 262144 // context)))
    prompts = rng.randint(1, min(requests, 4)) if rng.random() < 0.5 else 0
    c.update(requests=requests, context=context, prompts=prompts, prompt=log(2, max(2, min(context, 8192 // prompts))) if prompts else 0)
    return c


# ----------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEV, generator=g) * std).to(dtype)


def _fp8(g, *shape):
    out = torch.empty(shape, dtype=torch.float8_e4m3fn, device=DEV)
    flat = out.view(-1)
    for a in range(0, flat.numel(), 1 << 27):   # a piece at a time: the draws are 32-bit
        n = min(1 << 27, flat.numel() - a)
        flat[a:a + n] = torch.randn(n, device=DEV, generator=g).to(torch.float8_e4m3fn)
    return out


def _bytes(g, *shape):
    return torch.randint(0, 256, shape, dtype=torch.uint8, device=DEV, generator=g)


def _linear(g, quant, n_out, n_in):
    """Checkpoint tensors of a linear layer whose weights have a spread of about 0.02."""
    if quant == "bf16":
        return dict(weight=_randn(g, n_out, n_in, std=0.02))
    if quant == "fp8":
        return dict(weight=_fp8(g, n_out, n_in), weight_scale_inv=0.01 + 0.02 * torch.rand(-(-n_out // 128), -(-n_in // 128), device=DEV, generator=g))
    words = lambda rows: torch.randint(-2 ** 31, 2 ** 31, (rows, n_out // 8), device=DEV, generator=g).to(torch.int32)
    return dict(qweight=words(n_in), qzeros=words(n_in // 128), scales=(0.0015 + 0.003 * torch.rand(n_in // 128, n_out, device=DEV, generator=g)).half())


def _quant_config(quant):
    return {"bf16": None, "awq": dict(quant_method="awq", bits=4, group_size=128, zero_point=True),
            "fp8": dict(quant_method="fp8", weight_block_size=[128, 128]), "mxfp4": dict(quant_method="fp8", weight_block_size=[128, 128], expert_method="mxfp4")}[quant]


def _hf(case, arch, **more):
    return dict(architectures=[arch], hidden_size=case["hidden"], rms_norm_eps=EPS, rope_theta=THETA, max_position_embeddings=MAX_POS,
                **{k: v for k, v in dict(quantization_config=_quant_config(case.get("quant", "bf16"))).items() if v}, **more)


def _load(layer, tensors):
    for name, t in tensors.items():
        layer.load_weight(name, t)


def _spread(i):
    """Numbers of 0 to 1 in no order, the same ones for every seed (a case's shapes are its own)."""
    return (0.5 + 0.6180339887498949 * i) % 1.0


def _finish(module):
    process_weights_after_loading(torch.nn.ModuleList([module]))
    return module.eval()


def _step(case, g, pages=True):
    """New tokens and context length of every request, and the step's metadata. The context lengths are spread over the eighth below the
    case's, a prompt's chunk over the quarter below; prompts come last."""
    R, P = case["requests"], case["prompts"]
    u = [[_spread(r + 100 * j) for r in range(R)] for j in (0, 1)]
    new = [1] * (R - P) + [max(1, round(case["prompt"] * (0.75 + 0.25 * x))) if R > 1 else case["prompt"] for x in u[0][R - P:]]
    ctx = [max(n, round(case.get("context", 0) * (0.875 + 0.125 * x))) if R > 1 else max(n, case.get("context", 0)) for n, x in zip(new, u[1])]
    T = sum(new)
    start = np.concatenate([[0], np.cumsum(new)]).astype(np.int32)
    pos = np.concatenate([np.arange(c - n, c) for n, c in zip(new, ctx)]).astype(np.int32)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.int32, device=DEV)
    table, slots, total = None, None, 1
    if pages:
        per = [-(-c // BLOCK) for c in ctx]
        total = 1 + sum(per)
        order = (torch.randperm(total - 1, device=DEV, generator=g) + 1).cpu().numpy()   # page 0 is the runner's placeholder
        table = np.zeros((R, max(per)), np.int32)
        at, sl = 0, []
        for r in range(R):
            table[r, :per[r]] = order[at:at + per[r]]
            at += per[r]
            p = np.arange(ctx[r] - new[r], ctx[r])
            sl.append(table[r][p // BLOCK] * BLOCK + p % BLOCK)
        slots = np.concatenate(sl)
    md = AttentionMetadata(R, T, dev(start), dev(ctx), dev(table) if pages else None, dev(slots) if pages else None, dev(pos), max(new), max(ctx),
                           query_lens_cpu=list(new), seq_lens_cpu=list(ctx), is_uniform_decode=max(new) == 1)
    return new, ctx, md, total


def _mlp_inputs(case, seed):
    g = _gen(seed)
    return dict(gate_up=_linear(g, case["quant"], 2 * case["inter"], case["hidden"]), down=_linear(g, case["quant"], case["hidden"], case["inter"]),
                x=_randn(g, case["tokens"], case["hidden"]))


def _attention_inputs(case, seed):
    g = _gen(seed)
    H, Hq, Hkv, D = case["hidden"], case["heads"], case["kv_heads"], case["dim"]
    new, ctx, md, total = _step(case, g)
    gemma = 0.0 if case["gated"] else 1.0   # the gated family stores norm weights minus one
    norm = lambda: (gemma + 0.1 * torch.randn(D, device=DEV, generator=g)).bfloat16()
    cache = torch.empty(total, 2, Hkv, BLOCK, D, dtype=torch.float8_e4m3fn if case["kv"] == "fp8" else torch.bfloat16, device=DEV)
    for a in range(0, total, 4096):
        b = min(a + 4096, total)
        cache[a:b] = torch.randn(b - a, 2, Hkv, BLOCK, D, device=DEV, generator=g).to(cache.dtype)
    return dict(qkv=_linear(g, case["quant"], (Hq * (2 if case["gated"] else 1) + 2 * Hkv) * D, H), o=_linear(g, case["quant"], H, Hq * D), q_norm=norm(),
                k_norm=norm(), x=_randn(g, sum(new), H), cache=cache, new=new, ctx=ctx, md=md)


def _experts_inputs(case, seed):
    g = _gen(seed)
    E, H, I, T, k, quant = case["experts"], case["hidden"], case["inter"], case["tokens"], case["top_k"], case["quant"]
    if quant == "fp8":
        scale = lambda *s: 0.01 + 0.02 * torch.rand(*s, device=DEV, generator=g)
        w = dict(w13=_fp8(g, E, 2 * I, H), w2=_fp8(g, E, H, I), w13_scale=scale(E, 2 * I // 128, H // 128), w2_scale=scale(E, H // 128, I // 128))
    elif quant == "mxfp4":   # powers of two that bring the codes (spread 2.6) to about 0.02
        scale = lambda *s: torch.randint(119, 122, s, dtype=torch.uint8, device=DEV, generator=g)
        w = dict(w13=_bytes(g, E, 2 * I, H // 2), w2=_bytes(g, E, H, I // 2), w13_scale=scale(E, 2 * I, H // 32), w2_scale=scale(E, H, I // 32))
    else:
        w = dict(w13=_randn(g, E, 2 * I, H, std=0.02), w2=_randn(g, E, H, I, std=0.02))
    top, ids = torch.randn(T, E, device=DEV, generator=g).topk(k, dim=-1)
    return dict(w, x=_randn(g, T, H), topk_w=torch.softmax(top, -1), topk_ids=ids.to(torch.int32))


def _gdn_inputs(case, seed):
    g = _gen(seed)
    H, Hk, Hv, K, taps = case["hidden"], case["key_heads"], case["value_heads"], 128, 4
    new, _, md, _ = _step(case, g, pages=False)
    R, C = case["requests"], (2 * Hk + Hv) * K
    md.state_slots = (torch.randperm(R, device=DEV, generator=g) + 1).to(torch.int32)
    md.has_initial_state = torch.tensor([1] * (R - case["prompts"]) + [0] * case["prompts"], dtype=torch.int32, device=DEV)
    return dict(qkvz=_randn(g, C + Hv * K, H, std=0.02), ba=_randn(g, 2 * Hv, H, std=0.02), out=_randn(g, H, Hv * K, std=0.02), conv=_randn(g, C, taps, std=0.3),
                A_log=torch.rand(Hv, device=DEV, generator=g), dt_bias=torch.rand(Hv, device=DEV, generator=g),
                norm=(1 + 0.1 * torch.randn(K, device=DEV, generator=g)).bfloat16(), x=_randn(g, sum(new), H), conv_state=_randn(g, R + 1, C, taps - 1),
                state=0.1 * torch.randn(R + 1, Hv, K, K, device=DEV, generator=g), new=new, md=md)


MLA = dict(q_lora=1536, lora=512, nope=128, rope=64, v=128)   # latent sizes of the MLA cases


def _mla_inputs(case, seed):
    g = _gen(seed)
    H, n, z = case["hidden"], case["heads"], MLA
    new, ctx, md, total = _step(case, g)
    norm = lambda w: (1 + 0.1 * torch.randn(w, device=DEV, generator=g)).bfloat16()
    lin = lambda o, i: _linear(g, "fp8", o, i)
    return dict(q_a=lin(z["q_lora"], H), q_b=lin(n * (z["nope"] + z["rope"]), z["q_lora"]), kv_a=lin(z["lora"] + z["rope"], H),
                kv_b=lin(n * (z["nope"] + z["v"]), z["lora"]), o=lin(H, n * z["v"]), q_norm=norm(z["q_lora"]), kv_norm=norm(z["lora"]), x=_randn(g, sum(new), H),
                cache=_randn(g, total, BLOCK, z["lora"] + z["rope"]), new=new, ctx=ctx, md=md)


def _serve_inputs(case, seed):
    g = _gen(seed)
    H, I, D, heads, kv = case["hidden"], case["inter"], 128, 8, 2
    w = {"model.embed_tokens.weight": _randn(g, case["vocab"], H, std=0.02)}
    ones = lambda n: (1 + 0.1 * torch.randn(n, device=DEV, generator=g)).bfloat16()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for name, o, k in (("self_attn.q_proj", heads * D, H), ("self_attn.k_proj", kv * D, H), ("self_attn.v_proj", kv * D, H), ("self_attn.o_proj", H, heads * D),
                           ("mlp.gate_proj", I, H), ("mlp.up_proj", I, H), ("mlp.down_proj", H, I)):
            w.update({f"{p}{name}.{n}": t for n, t in _linear(g, "awq", o, k).items()})
        w.update({p + "self_attn.q_norm.weight": ones(D), p + "self_attn.k_norm.weight": ones(D), p + "input_layernorm.weight": ones(H),
                  p + "post_attention_layernorm.weight": ones(H)})
    w.update({"model.norm.weight": ones(H), "lm_head.weight": _randn(g, case["vocab"], H, std=0.02)})
    lens = [max(1, round(case["prompt"] * (0.25 + 0.75 * _spread(r)))) for r in range(case["requests"])]
    tokens = [torch.randint(0, case["vocab"], (n + case["steps"],), device=DEV, generator=g).tolist() for n in lens]
    return w, lens, tokens


def _write_checkpoint(folder, config, weights):
    """config.json and one safetensors file (8 bytes with the header's length, the header in JSON, the tensors' bytes)."""
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(config, f)
    names = {torch.bfloat16: "BF16", torch.float16: "F16", torch.int32: "I32"}
    header, at = {}, 0
    for name, t in weights.items():
        n = t.numel() * t.element_size()
        header[name] = dict(dtype=names[t.dtype], shape=list(t.shape), data_offsets=[at, at + n])
        at += n
    head = json.dumps(header).encode()
    head += b" " * (-len(head) % 8)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(head)) + head)
        for t in weights.values():
            f.write(t.contiguous().view(torch.uint8).cpu().numpy().tobytes())


# ----------------------------------------------------------------------------- the calls
@torch.inference_mode()
def prepare(case, seed):
    kind, dt = case["kind"], torch.bfloat16
    if kind == "serve":
        w, lens, tokens = _serve_inputs(case, seed)
        config = _hf(dict(case, quant="awq"), "Qwen3ForCausalLM", intermediate_size=case["inter"], num_hidden_layers=case["layers"], num_attention_heads=8,
                     num_key_value_heads=2, head_dim=128, vocab_size=case["vocab"])
        room = sum(-(-len(t) // BLOCK) * BLOCK for t in tokens)
        with tempfile.TemporaryDirectory() as d:
            _write_checkpoint(d, config, w)
            engine = TraceReplay(d, "bfloat16", room, max_live=case["requests"])
        return dict(kind=kind, engine=engine, lens=lens, tokens=tokens, steps=case["steps"])
    with torch.device(DEV):
        if kind == "mlp":
            i = _mlp_inputs(case, seed)
            m = MLP(case["hidden"], case["inter"], ModelConfig.from_hf_dict(_hf(case, "Qwen3ForCausalLM")).quant, "mlp", dt)
            _load(m.gate_up_proj, i["gate_up"])
            _load(m.down_proj, i["down"])
            return dict(kind=kind, layer=_finish(m), x=i["x"])
        if kind == "attention":
            i = _attention_inputs(case, seed)
            hf = _hf(case, "Qwen3_5ForCausalLM" if case["gated"] else "Qwen3ForCausalLM", num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"],
                     head_dim=case["dim"], **(dict(partial_rotary_factor=0.25) if case["gated"] else {}))
            m = Attention(ModelConfig.from_hf_dict(hf, dtype=dt, max_model_len=MAX_POS), 3, "self_attn", DEV)
            _load(m.qkv_proj, i["qkv"])
            _load(m.o_proj, i["o"])
            m.q_norm.data.copy_(i["q_norm"])
            m.k_norm.data.copy_(i["k_norm"])
            return dict(kind=kind, layer=_finish(m), x=i["x"], md=i["md"], cache=i["cache"])
        if kind == "experts":
            i = _experts_inputs(case, seed)
            hf = _hf(case, "Qwen3MoeForCausalLM", num_experts=case["experts"], num_experts_per_tok=case["top_k"], moe_intermediate_size=case["inter"])
            m = FusedMoE(ModelConfig.from_hf_dict(hf, dtype=dt), "experts")
            for name in ("w13", "w2", "w13_scale", "w2_scale"):
                if name in i:
                    getattr(m, name).data.copy_(i[name])
            return dict(kind=kind, layer=_finish(m), x=i["x"], topk_w=i["topk_w"], topk_ids=i["topk_ids"])
        if kind == "gdn":
            i = _gdn_inputs(case, seed)
            hf = _hf(case, "Qwen3_5ForCausalLM", num_attention_heads=24, num_key_value_heads=4, head_dim=256, linear_num_key_heads=case["key_heads"],
                     linear_num_value_heads=case["value_heads"])
            m = GatedDeltaNet(ModelConfig.from_hf_dict(hf, dtype=dt), 0, "linear_attn")
            m.in_proj_qkvz.load_weight("weight", i["qkvz"])
            m.in_proj_ba.load_weight("weight", i["ba"])
            m.out_proj.load_weight("weight", i["out"])
            for name, t in (("conv_weight", i["conv"]), ("A_log", i["A_log"]), ("dt_bias", i["dt_bias"])):
                m.load_weight(name, t)
            m.norm_weight.data.copy_(i["norm"])
            return dict(kind=kind, layer=_finish(m), x=i["x"], md=i["md"], cache=(i["conv_state"], i["state"]))
        i = _mla_inputs(case, seed)
        hf = _hf(dict(case, quant="fp8"), "DeepseekV3ForCausalLM", num_attention_heads=case["heads"], num_key_value_heads=case["heads"], q_lora_rank=MLA["q_lora"],
                 kv_lora_rank=MLA["lora"], qk_nope_head_dim=MLA["nope"], qk_rope_head_dim=MLA["rope"], v_head_dim=MLA["v"])
        m = MLAAttention(ModelConfig.from_hf_dict(hf, dtype=dt, max_model_len=MAX_POS), 0, "self_attn", DEV)
        for lin, name in ((m.q_a_proj, "q_a"), (m.q_b_proj, "q_b"), (m.kv_a_proj_with_mqa, "kv_a"), (m.kv_b_proj, "kv_b"), (m.o_proj, "o")):
            _load(lin, i[name])
        m.q_a_layernorm.load_weight("weight", i["q_norm"])
        m.kv_a_layernorm.load_weight("weight", i["kv_norm"])
        return dict(kind=kind, layer=_finish(m), x=i["x"], md=i["md"], cache=i["cache"])


@torch.inference_mode()
def run(state):
    kind = state["kind"]
    if kind == "serve":
        e, names = state["engine"], [f"r{i}" for i in range(len(state["lens"]))]
        logits = [e.step([dict(id=n, tokens=t[:k], want=[k - 1]) for n, t, k in zip(names, state["tokens"], state["lens"])])]
        for j in range(state["steps"]):
            logits.append(e.step([dict(id=n, tokens=[t[k + j]], want=[0]) for n, t, k in zip(names, state["tokens"], state["lens"])],
                                 end=names if j == state["steps"] - 1 else ()))
        return logits
    layer, x = state["layer"], state["x"]
    if kind == "mlp":
        return layer(x)
    if kind == "experts":
        return layer(x, state["topk_w"], state["topk_ids"])
    y = layer(x, state["md"], state["cache"])
    return [y, *state["cache"]] if kind == "gdn" else [y, state["cache"]]


# ----------------------------------------------------------------------------- what a pass needs, and what it may differ by
def _weight_bytes(quant, n):
    return n * {"bf16": 2.0, "fp8": 1.0 + 4.0 / 16384, "awq": 0.5 + 2.5 / 128, "mxfp4": 0.5 + 1.0 / 32}[quant]


def _lengths(case):
    """Mean new tokens and context lengths of a step, as ``_step`` spreads them."""
    R, P = case["requests"], case["prompts"]
    chunk, ctx = (0.875 * case["prompt"], 0.9375 * case.get("context", 0)) if R > 1 else (case["prompt"], case.get("context", 0))
    return R - P, P, chunk, max(ctx, chunk, 1.0)


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        T, n = case["tokens"], 3 * case["hidden"] * case["inter"]
        return dict(bytes=_weight_bytes(case["quant"], n) + 4 * T * case["hidden"], flops=2 * T * n)
    if kind == "experts":
        T, k, n = case["tokens"], case["top_k"], 3 * case["hidden"] * case["inter"]
        used = case["experts"] * (1 - (1 - k / case["experts"]) ** T)   # experts that some token chooses
        return dict(bytes=_weight_bytes(case["quant"], n) * used + 4 * T * case["hidden"] + 8 * T * k, flops=2 * T * k * n)
    if kind == "serve":
        T, R = 0.625 * case["prompt"] * case["requests"], case["requests"]
        per = case["layers"] * (case["hidden"] * (12 + 8) * 128 + 3 * case["hidden"] * case["inter"])
        head = case["vocab"] * case["hidden"]
        return dict(bytes=(1 + case["steps"]) * (_weight_bytes("awq", per) + 2 * head + 4 * R * case["vocab"]),
                    flops=2 * (T + R * case["steps"]) * per + 2 * (1 + case["steps"]) * R * head)
    dec, P, chunk, ctx = _lengths(case)
    T = dec + P * chunk
    if kind == "gdn":
        C, V = (2 * case["key_heads"] + case["value_heads"]) * 128, case["value_heads"] * 128
        n = case["hidden"] * (C + 2 * V + 2 * case["value_heads"])
        state = case["requests"] * (V * 128 * 4 + C * 3 * 2)
        return dict(bytes=2 * n + 4 * T * case["hidden"] + 2 * state - P * (V * 128 * 4 + C * 3 * 2), flops=2 * T * n + 6 * T * V * 128)
    pairs = dec * ctx + P * (chunk * (ctx - chunk) + chunk * (chunk + 1) / 2)   # (query, key) pairs of a head
    keys = dec * ctx + P * ctx
    if kind == "attention":
        D, G = case["dim"], 2 if case["gated"] else 1
        n = case["hidden"] * D * ((G + 1) * case["heads"] + 2 * case["kv_heads"])
        row = 2 * case["kv_heads"] * D * (1 if case["kv"] == "fp8" else 2)
        return dict(bytes=_weight_bytes(case["quant"], n) + 4 * T * case["hidden"] + row * keys, flops=2 * T * n + 4 * pairs * case["heads"] * D)
    z, H = MLA, case["heads"]
    n = case["hidden"] * (z["q_lora"] + z["lora"] + z["rope"] + H * z["v"]) + z["q_lora"] * H * (z["nope"] + z["rope"]) + z["lora"] * H * (z["nope"] + z["v"])
    wide = 2 * z["lora"] + z["rope"]   # decoding scores and sums latents; a prompt may expand them to heads of 128 + 64 and 128
    per = dec * ctx * wide + P * (chunk * (ctx - chunk) + chunk * (chunk + 1) / 2) * (z["nope"] + z["rope"] + z["v"])
    return dict(bytes=_weight_bytes("fp8", n) + 4 * T * case["hidden"] + 2 * (z["lora"] + z["rope"]) * keys, flops=2 * T * n + 2 * per * H)


def tolerance(case):
    """Two correct bf16 implementations round the same intermediate results (activations between the products, dequantised weights, softmax
    weights) at other places or after other sums. Measured against 64 bits: 0.5e-2 for the blocks, 1.5e-2 after the layers of a served model."""
    return {"mlp": dict(rel=1e-2), "experts": dict(rel=1e-2), "attention": dict(rel=1.5e-2), "gdn": dict(rel=2e-2), "mla": dict(rel=2e-2), "serve": dict(rel=3e-2)}[case["kind"]]


# ----------------------------------------------------------------------------- the same in 64 bits
def _dense(quant, t):
    """[out, in] weight of a linear layer's checkpoint tensors."""
    if quant == "bf16":
        return t["weight"].double()
    if quant == "fp8":
        w = t["weight"].to(torch.float32).double()
        s = t["weight_scale_inv"].double().repeat_interleave(128, 0).repeat_interleave(128, 1)
        return w * s[: w.shape[0], : w.shape[1]]

    def codes(words):   # nibble i of a word is this column of its eight
        out = torch.empty(*words.shape, 8, dtype=torch.float64, device=DEV)
        for i, c in enumerate((0, 4, 1, 5, 2, 6, 3, 7)):
            out[..., c] = ((words >> (4 * i)) & 15).double()
        return out.view(words.shape[0], -1)
    q, z, s = codes(t["qweight"]), codes(t["qzeros"]), t["scales"].double()
    return ((q - z.repeat_interleave(128, 0)) * s.repeat_interleave(128, 0)).t()


def _rms(x, w, plus=0.0):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * (w.double() + plus)


def _rope(x, pos, n, adjacent=False):
    """x ``[T, heads, D]`` with its first n dimensions rotated; pairs (i, i + n/2), or neighbours."""
    f = pos.double().view(-1, 1, 1) * THETA ** (-torch.arange(0, n, 2, device=DEV, dtype=torch.float64) / n)
    a, b = (x[..., :n:2], x[..., 1:n:2]) if adjacent else (x[..., : n // 2], x[..., n // 2: n])
    return torch.cat([a * f.cos() - b * f.sin(), b * f.cos() + a * f.sin(), x[..., n:]], -1)


def _softmax_sum(q, k, v, scale):
    """Causal attention of the last rows of a sequence: q ``[n, D]`` per row of ``[rows, n, D]``, k and v ``[S, D]``."""
    n, S, out = q.shape[1], k.shape[0], []
    for a in range(0, n, 512):   # a piece at a time: all scores of a long prompt do not fit
        s = torch.einsum("rnd,sd->rns", q[:, a:a + 512], k) * scale
        seen = torch.arange(S, device=DEV) <= torch.arange(S - n + a, S - n + min(a + 512, n), device=DEV).view(-1, 1)
        out.append(torch.softmax(s.masked_fill_(~seen, -math.inf), -1) @ v)
    return torch.cat(out, 1)


def _attend(q, k, v, case, i):
    """New queries, keys and values ``[T, heads, D]`` over the cached ones of every request."""
    out, at, G, D = torch.empty_like(q), 0, case["heads"] // case["kv_heads"], case["dim"]
    for r, (n, c) in enumerate(zip(i["new"], i["ctx"])):
        pages = i["cache"][i["md"].block_table[r, : -(-c // BLOCK)].long()].float().double()   # [pages, 2, Hkv, 16, D]
        old = pages.permute(1, 2, 0, 3, 4).reshape(2, case["kv_heads"], -1, D)[:, :, : c - n]
        for h in range(case["kv_heads"]):
            keys, vals = (torch.cat([old[j, h], t[at:at + n, h]]) for j, t in ((0, k), (1, v)))
            out[at:at + n, h * G:(h + 1) * G] = _softmax_sum(q[at:at + n, h * G:(h + 1) * G].transpose(0, 1), keys, vals, D ** -0.5).transpose(0, 1)
        at += n
    return out


def _attention_exact(case, seed):
    i = _attention_inputs(case, seed)
    Hq, Hkv, D, gated = case["heads"], case["kv_heads"], case["dim"], case["gated"]
    y, pos = i["x"].double() @ _dense(case["quant"], i["qkv"]).t(), i["md"].positions
    T, w = y.shape[0], Hq * D * (2 if gated else 1)
    q, gate = (y[:, :w].view(T, Hq, 2 * D)[..., :D], y[:, :w].view(T, Hq, 2 * D)[..., D:]) if gated else (y[:, :w].view(T, Hq, D), None)
    k, v = (y[:, w + j * Hkv * D: w + (j + 1) * Hkv * D].view(T, Hkv, D) for j in (0, 1))
    plus, n = (1.0, D // 4) if gated else (0.0, D)
    o = _attend(_rope(_rms(q, i["q_norm"], plus), pos, n), _rope(_rms(k, i["k_norm"], plus), pos, n), v, case, i)
    if gated:
        o = o * torch.sigmoid(gate)
    return [o.reshape(T, -1) @ _dense(case["quant"], i["o"]).t(), None]


def _silu(x):
    return x * torch.sigmoid(x)


def _experts_exact(case, seed):
    i = _experts_inputs(case, seed)
    x, inter, quant = i["x"].double(), case["inter"], case["quant"]
    fp4 = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device=DEV)

    def weight(name, e):
        w = i[name][e]
        if quant == "bf16":
            return w.double()
        s = i[name + "_scale"][e]
        if quant == "fp8":
            return w.float().double() * s.double().repeat_interleave(128, 0).repeat_interleave(128, 1)
        return fp4[torch.stack([w & 15, w >> 4], -1).long().flatten(1)] * torch.exp2(s.double() - 127).repeat_interleave(32, 1)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        t, j = (i["topk_ids"] == e).nonzero(as_tuple=True)
        if t.numel():
            h = x[t] @ weight("w13", e).t()
            out.index_add_(0, t, (_silu(h[:, :inter]) * h[:, inter:]) @ weight("w2", e).t() * i["topk_w"][t, j].double().unsqueeze(1))
    return out


def _gdn_exact(case, seed):
    i = _gdn_inputs(case, seed)
    Hk, Hv, K, md = case["key_heads"], case["value_heads"], 128, i["md"]
    C, slots, first = (2 * Hk + Hv) * K, md.state_slots.long(), md.has_initial_state.double()
    x = i["x"].double()
    y, ba = x @ i["qkvz"].double().t(), x @ i["ba"].double().t()
    decay = torch.exp(-torch.exp(i["A_log"].double()) * torch.nn.functional.softplus(ba[:, Hv:] + i["dt_bias"].double()))
    beta = torch.sigmoid(ba[:, :Hv])
    window = i["conv_state"].double()[slots] * first.view(-1, 1, 1)   # [R, C, 3]
    S = i["state"].double()[slots] * first.view(-1, 1, 1, 1)
    conv, o = i["conv"].double(), torch.empty(x.shape[0], Hv, K, dtype=torch.float64, device=DEV)
    start = torch.tensor(np.concatenate([[0], np.cumsum(i["new"])[:-1]]), device=DEV)
    unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
    new = torch.tensor(i["new"], device=DEV)
    for t in range(max(i["new"])):   # token t of every request that has one
        live = (new > t).nonzero().flatten() if t < 2 or len(i["new"]) > 1 else slice(None)
        at = start[live] + t
        w = torch.cat([window[live], y[at, :C].unsqueeze(-1)], -1)
        window[live] = w[..., 1:]
        c = _silu((w * conv).sum(-1))
        q, k = (unit(c[:, j * Hk * K:(j + 1) * Hk * K].view(-1, Hk, K)).repeat_interleave(Hv // Hk, 1) for j in (0, 1))
        s = S[live] * decay[at].view(-1, Hv, 1, 1)
        delta = (c[:, 2 * Hk * K:].view(-1, Hv, K) - torch.einsum("rhk,rhkv->rhv", k, s)) * beta[at].unsqueeze(-1)
        s = s + k.unsqueeze(-1) * delta.unsqueeze(-2)
        S[live] = s
        o[at] = torch.einsum("rhk,rhkv->rhv", q, s) * K ** -0.5
    o = _rms(o, i["norm"]) * _silu(y[:, C:].view(-1, Hv, K))
    conv_state, state = i["conv_state"].double(), i["state"].double()
    conv_state[slots], state[slots] = window, S
    return [o.reshape(x.shape[0], -1) @ i["out"].double().t(), conv_state, state]


def _mla_exact(case, seed):
    i, z, H = _mla_inputs(case, seed), MLA, case["heads"]
    x, pos, w = i["x"].double(), i["md"].positions, {n: _dense("fp8", i[n]) for n in ("q_a", "q_b", "kv_a", "kv_b", "o")}
    T = x.shape[0]
    q = (_rms(x @ w["q_a"].t(), i["q_norm"]) @ w["q_b"].t()).view(T, H, -1)
    kv = x @ w["kv_a"].t()
    lat = _rms(kv[:, : z["lora"]], i["kv_norm"])

    def pairs(t):   # rotated neighbours stay neighbours, as in the cached rows
        h = t.shape[-1] // 2
        return torch.stack([t[..., :h], t[..., h:]], -1).flatten(-2)
    pe = lambda t: pairs(_rope(t, pos, z["rope"], adjacent=True))
    key_pe, q_pe = pe(kv[:, z["lora"]:].unsqueeze(1)).squeeze(1), pe(q[..., z["nope"]:])
    up = w["kv_b"].view(H, z["nope"] + z["v"], z["lora"])
    q_lat = torch.einsum("thn,hnl->thl", q[..., : z["nope"]], up[:, : z["nope"]])
    o, at, scale = torch.empty(T, H, z["lora"], dtype=torch.float64, device=DEV), 0, (z["nope"] + z["rope"]) ** -0.5
    for r, (n, c) in enumerate(zip(i["new"], i["ctx"])):
        old = i["cache"][i["md"].block_table[r, : -(-c // BLOCK)].long()].double().flatten(0, 1)[: c - n]
        rows = torch.cat([old, torch.cat([lat[at:at + n], key_pe[at:at + n]], -1)])
        for h in range(0, H, 16):
            qq = torch.cat([q_lat[at:at + n, h:h + 16], q_pe[at:at + n, h:h + 16]], -1).transpose(0, 1)
            o[at:at + n, h:h + 16] = _softmax_sum(qq, rows, rows[:, : z["lora"]], scale).transpose(0, 1)
        at += n
    o = torch.einsum("thl,hvl->thv", o, up[:, z["nope"]:])
    return [o.reshape(T, -1) @ w["o"].t(), None]


def _serve_exact(case, seed):
    w, lens, tokens = _serve_inputs(case, seed)
    lin = lambda p, *names: [_dense("awq", {n: w[f"{p}{name}.{n}"] for n in ("qweight", "qzeros", "scales")}).t() for name in names]
    rows = []
    for n, ids in zip(lens, tokens):
        pos = torch.arange(len(ids), device=DEV)
        h = w["model.embed_tokens.weight"].double()[torch.tensor(ids, device=DEV)]
        for j in range(case["layers"]):
            p = f"model.layers.{j}."
            x = _rms(h, w[p + "input_layernorm.weight"])
            q, k, v, o = lin(p + "self_attn.", "q_proj", "k_proj", "v_proj", "o_proj")
            q, k, v = ((x @ t).view(len(ids), -1, 128) for t in (q, k, v))
            q, k = _rope(_rms(q, w[p + "self_attn.q_norm.weight"]), pos, 128), _rope(_rms(k, w[p + "self_attn.k_norm.weight"]), pos, 128)
            a = [_softmax_sum(q[:, 4 * g:4 * g + 4].transpose(0, 1), k[:, g], v[:, g], 128 ** -0.5).transpose(0, 1) for g in range(2)]
            h = h + torch.cat(a, 1).reshape(len(ids), -1) @ o
            x = _rms(h, w[p + "post_attention_layernorm.weight"])
            gate, up, down = lin(p + "mlp.", "gate_proj", "up_proj", "down_proj")
            h = h + (_silu(x @ gate) * (x @ up)) @ down
        rows.append(_rms(h[n - 1:], w["model.norm.weight"]) @ w["lm_head.weight"].double().t())
    return [torch.stack([r[j] for r in rows]).cpu() for j in range(case["steps"] + 1)]


@torch.inference_mode()
def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        i = _mlp_inputs(case, seed)
        h = i["x"].double() @ _dense(case["quant"], i["gate_up"]).t()
        return (_silu(h[:, : case["inter"]]) * h[:, case["inter"]:]) @ _dense(case["quant"], i["down"]).t()
    return dict(attention=_attention_exact, experts=_experts_exact, gdn=_gdn_exact, mla=_mla_exact, serve=_serve_exact)[kind](case, seed)
