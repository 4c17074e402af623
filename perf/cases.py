"""Steps of served models, as a program around this framework runs them: prefill of a batch of prompts, and decode of one token for every
live request, through `DynamicInferenceContext` and the inference wrapper.

Dense GPT models at the layer shapes of `configs.py` (bf16, MXFP8 and blockwise FP8 linears, bf16 and E4M3 key/value pools) and the four hybrid
designs at the layer shapes of the design benchmarks, a few layers of each (of Maginex those in front of its first layer of latent attention).
Decode steps replay a CUDA graph of the model, as the engine does; every step includes what the host prepares for it.  A decode step of a dense
model finds seeded keys and values in the pool, one of a hybrid design what its prompts left there.  Weights are seeded noise at the scale of
their inputs.

Which experts a token takes is settled by features of its embedding that no sublayer writes to, different for every token: so tokens spread over the
experts as they do in a trained model, and rounding never changes a choice."""
from __future__ import annotations

import math
import random
import zlib

import torch

BF16, F64 = torch.bfloat16, torch.float64
CHUNK = 256
KV8_SCALE = 2.0 ** -6

GPT = {
    "8b": dict(width=4096, heads=32, groups=8, dim=128, ff=14336, vocab=128256, base=500000.0),
    "70b": dict(width=8192, heads=64, groups=8, dim=128, ff=28672, vocab=128256, base=500000.0),
}
HYBRID_VOCAB = 32768


def _case(model, size, layers, precision, step, requests, shortest, longest, log_lengths=False, lengths=1):
    """Contexts (decode) or prompts (prefill) of ``shortest`` to ``longest`` tokens, drawn with the number ``lengths``."""
    return {"model": model, "size": size, "layers": layers, "precision": precision, "step": step, "requests": requests,
            "shortest": shortest, "longest": longest, "log_lengths": log_lengths, "lengths": lengths}


def listed():
    return [
        # one user of a small model: a step is a few dozen launches, each of a few microseconds
        {"name": "zinurax_decode_1"} | _case("zinurax", "2k", 4, "bf16", "decode", 1, 700, 700),
        # the three serving batches of configs.py: bf16, MXFP8, blockwise FP8 at 70B layer shapes
        {"name": "gpt_bf16_decode_64"} | _case("gpt", "8b", 4, "bf16", "decode", 64, 128, 2048),
        {"name": "gpt_mxfp8_decode_128"} | _case("gpt", "8b", 4, "mxfp8", "decode", 128, 256, 4096),
        {"name": "gpt_block_decode_256"} | _case("gpt", "70b", 2, "blockwise", "decode", 256, 512, 8192),
        # long contexts in an E4M3 pool
        {"name": "gpt_kv8_decode_32"} | _case("gpt", "8b", 2, "mxfp8_kv8", "decode", 32, 32768, 131072, log_lengths=True),
        # prompts entering those batches
        {"name": "gpt_bf16_prefill"} | _case("gpt", "8b", 4, "bf16", "prefill", 7, 128, 2048),
        {"name": "gpt_mxfp8_prefill"} | _case("gpt", "8b", 4, "mxfp8", "prefill", 6, 256, 4096),
        {"name": "gpt_block_prefill"} | _case("gpt", "70b", 2, "blockwise", "prefill", 2, 512, 8192),
        # the hybrid designs: prompts, and a batch of live requests
        {"name": "zinurax_prefill"} | _case("zinurax", "2k", 4, "bf16", "prefill", 5, 512, 2048),
        {"name": "fabivik_prefill"} | _case("fabivik", "2k", 4, "bf16", "prefill", 4, 1000, 2048),
        {"name": "maginex_prefill"} | _case("maginex", "4k", 3, "bf16", "prefill", 4, 777, 2048),
        {"name": "lukarax_decode_64"} | _case("lukarax", "2k", 4, "bf16", "decode", 64, 128, 1024),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    decode = rng.random() < 0.5
    if rng.random() < 0.6:
        size, layers, precision, most, longest = rng.choice([
            ("8b", 4, "bf16", 64, 2048), ("8b", 4, "mxfp8", 128, 4096), ("70b", 2, "blockwise", 256, 8192), ("8b", 2, "mxfp8_kv8", 32, 131072)])
        if precision == "mxfp8_kv8":
            decode = True  # (contexts of this length are a matter of decoding)
        shortest = {"bf16": 128, "mxfp8": 256, "blockwise": 512, "mxfp8_kv8": 32768}[precision]
        n = log(1, most) if decode else log(1, 8)
        longest = log(shortest, longest)
        if not decode and n * longest > 2 * 8192:
            longest = max(shortest, 2 * 8192 // n)
        return _case("gpt", size, layers, precision, "decode" if decode else "prefill", n, shortest, longest,
                     log_lengths=precision == "mxfp8_kv8", lengths=rng.randrange(1 << 20))
    model = rng.choice(["zinurax", "fabivik", "lukarax", "maginex"])
    size = rng.choice(["2k", "2k", "4k"])
    n, longest = (log(1, 64), log(64, 1024)) if decode else (log(1, 8), log(128, 2048))
    return _case(model, size, 3 if model == "maginex" else 4, "bf16", "decode" if decode else "prefill", n, max(1, longest // 8), longest,
                 lengths=rng.randrange(1 << 20))


def lengths_of(case):
    """Tokens per request, the newest one included; the longest is there."""
    r = random.Random(case["lengths"])
    a, b = case["shortest"], case["longest"]
    out = [b] + [int(math.exp(r.uniform(math.log(a), math.log(b)))) if case["log_lengths"] else r.randint(a, b) for _ in range(case["requests"] - 1)]
    r.shuffle(out)
    return out


def tokens_of(case, seed):
    """Token ids per request: whole sequences, or for decode steps of a dense model (whose cache holds noise) only the newest token."""
    r = torch.Generator().manual_seed(seed * 7919 + 5)
    vocab = GPT[case["size"]]["vocab"] if case["model"] == "gpt" else HYBRID_VOCAB
    newest = case["model"] == "gpt" and case["step"] == "decode"
    return [torch.randint(0, vocab, (1 if newest else n,), generator=r) for n in lengths_of(case)]


class Noise:
    """Seeded tensors by name, on the GPU."""

    def __init__(self, seed):
        self.seed = seed

    def __call__(self, name, *shape, std=1.0, mean=0.0):
        g = torch.Generator(device="cuda").manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
        t = torch.randn(*shape, generator=g, device="cuda", dtype=BF16)
        return t if std == 1.0 and mean == 0.0 else t.mul_(std).add_(mean) if mean else t.mul_(std)

    def mat(self, name, n, k, gain=1.0):
        return self(name, n, k, std=gain / math.sqrt(k))

    def vec(self, name, n, mean=1.0, std=0.2):
        return self(name, n, std=std, mean=mean)


# ---------------------------------------------------------------------------------------------------------------------
# Dense models
# ---------------------------------------------------------------------------------------------------------------------
def gpt_weights(case, seed):
    """Linears keep the scale of their input; the feed-forward adds a third of it to a stream that starts at scale 1, as behind the first layers of a
    trained model.  (With a smaller stream the 8-bit roundings of the layers' inputs would be nearly all of the logits' error, and one rounding in another
    place would move them by most of it.)"""
    s, noise, out = GPT[case["size"]], Noise(seed), {}
    W, qkv = s["width"], (s["heads"] + 2 * s["groups"]) * s["dim"]

    def put(name, *shape):
        norm = name.endswith("layernorm.weight")
        std = 0.02 if norm else 1.0 if name.startswith("embedding") else (0.35 if "fc2" in name else 1.0) / math.sqrt(shape[-1])
        out[name] = noise(name, *shape, std=std, mean=1.0 if norm else 0.0)

    put("embedding.word_embeddings.weight", s["vocab"], W)
    for i in range(case["layers"]):
        p = f"decoder.layers.{i}."
        put(p + "input_layernorm.weight", W)
        put(p + "self_attention.linear_qkv.weight", qkv, W)
        put(p + "self_attention.linear_proj.weight", W, s["heads"] * s["dim"])
        put(p + "pre_mlp_layernorm.weight", W)
        put(p + "mlp.linear_fc1.weight", 2 * s["ff"], W)
        put(p + "mlp.linear_fc2.weight", W, s["ff"])
    put("decoder.final_layernorm.weight", W)
    put("output_layer.weight", s["vocab"], W)
    return out


def cached(case, seed, layer, request, tokens):
    """(keys, values) [tokens, groups, dim] in front of a request's newest token: bf16, or E4M3 in units of the pool's scale."""
    s = GPT[case["size"]]
    both = Noise(seed)(f"kv.{layer}.{request}", 2, tokens, s["groups"], s["dim"], std=0.5)
    return (both / KV8_SCALE).to(torch.float8_e4m3fn) if case["precision"] == "mxfp8_kv8" else both


def prepare_gpt(case, seed):
    from megatron_mixtera_b200 import model_registry as R
    from megatron_mixtera_b200 import ops
    from megatron_mixtera_b200.gpt.gpt_model import GPTModel
    from megatron_mixtera_b200.inference.contexts.dynamic_context import DynamicInferenceContext
    from megatron_mixtera_b200.transformer.transformer_config import TransformerConfig

    s, lengths, ids, kv8 = GPT[case["size"]], lengths_of(case), tokens_of(case, seed), case["precision"] == "mxfp8_kv8"
    most = max(lengths) + 64
    model = GPTModel(
        TransformerConfig(num_layers=case["layers"], hidden_size=s["width"], num_attention_heads=s["heads"], num_query_groups=s["groups"],
                          kv_channels=s["dim"], ffn_hidden_size=s["ff"], normalization="RMSNorm", gated_linear_unit=True, activation="silu",
                          add_bias_linear=False, enable_cuda_graph=True, fp8={"bf16": None, "mxfp8_kv8": "mxfp8"}.get(case["precision"], case["precision"])),
        vocab_size=s["vocab"], max_sequence_length=most, position_embedding_type="rope", rotary_base=s["base"])
    model.load_full_state_dict(gpt_weights(case, seed))
    if case["precision"] != "bf16":
        model.release_checkpoint_weights()
    torch.cuda.empty_cache()
    chunks = sum(-(-n // CHUNK) for n in lengths) + len(lengths) + 2
    portion = 65536 if case["step"] == "decode" else sum(lengths)
    ctx = DynamicInferenceContext(
        params_dtype=BF16, num_layers=case["layers"], kv_channels=s["dim"], num_attention_heads=s["groups"], max_sequence_length=most,
        buffer_size_gb=(chunks + 0.5) * (2 - kv8) * 2 * case["layers"] * CHUNK * s["groups"] * s["dim"] / 1024**3, buffer_guaranteed_fraction=0.0,
        chunk_size_tokens=CHUNK, max_requests_override=len(lengths), max_tokens_override=max(portion, len(lengths)),
        kv_cache_dtype=torch.float8_e4m3fn if kv8 else None)
    if kv8:
        ctx.kv_scales.fill_(KV8_SCALE)
    wrapper = R.make_controller(model, ctx).inference_wrapped_model
    if case["step"] == "prefill":
        ctx.schedule_tokens(list(enumerate(ids)))
        return ctx, wrapper
    for r, n in enumerate(lengths):  # what came before the newest token: the bookkeeping of a prefill, and noise as its keys and values
        for a in range(0, n - 1, portion):
            ctx.schedule_tokens([(r, [0] * min(portion, n - 1 - a))])
            ctx.complete_step()
    ctx.schedule_tokens(list(enumerate(ids)))
    for row, r in enumerate(ctx.request_ids[: len(lengths)].tolist()):
        n = lengths[r] - 1
        if n == 0:
            continue
        blocks = -(-n // CHUNK)
        at = ctx.request_to_kv_chunk_ids[row, :blocks].long().to(ctx.memory_buffer.device)
        for layer in range(case["layers"]):
            both = torch.zeros(2, blocks * CHUNK, s["groups"], s["dim"], dtype=ctx.memory_buffer.dtype, device=ctx.memory_buffer.device)
            both[:, :n] = cached(case, seed, layer, r, n).view(both.dtype)
            both = both.view(2, blocks, CHUNK, s["groups"], s["dim"])
            ctx.memory_buffer[0, layer][at] = both[0]
            ctx.memory_buffer[1, layer][at] = ops.fp8_values_to_pool_layout(both[1]) if kv8 else both[1]
    return ctx, wrapper


# ---------------------------------------------------------------------------------------------------------------------
# Hybrid designs
# ---------------------------------------------------------------------------------------------------------------------
SIZES = {
    ("zinurax", "2k"): dict(width=2048, heads=16, kv_rank=512, rot=64, dim=128, d_heads=32, d_dim=64, rank=64, ff=8192),
    ("zinurax", "4k"): dict(width=4096, heads=32, kv_rank=512, rot=64, dim=128, d_heads=64, d_dim=64, rank=128, ff=21504),
    ("fabivik", "2k"): dict(width=2048, heads=16, groups=8, dim=128, w_heads=32, w_dim=64, rank=64, d_heads=16, d_kv=8, d_dim=128, experts=32,
                            top=4, ff=512, shared=1024),
    ("fabivik", "4k"): dict(width=4096, heads=32, groups=8, dim=128, w_heads=64, w_dim=64, rank=128, d_heads=32, d_kv=16, d_dim=128, experts=64,
                            top=8, ff=1024, shared=2048),
    ("lukarax", "2k"): dict(width=2048, heads=16, groups=8, m_dim=64, dim=128, m_heads=16, experts=32, identity=2, sets=2, top=4, ff=512, dense=2048),
    ("lukarax", "4k"): dict(width=4096, heads=32, groups=8, m_dim=64, dim=128, m_heads=32, experts=64, identity=8, sets=4, top=8, ff=1024, dense=8192),
    ("maginex", "2k"): dict(width=2048, heads=16, groups=8, dim=128, kv_rank=512, q_rank=768, rot=64, scan=3072, experts=32, top=4, ff=768, shared=1536),
    ("maginex", "4k"): dict(width=4096, heads=32, groups=8, dim=128, kv_rank=512, q_rank=1536, rot=64, scan=6144, experts=64, top=8, ff=1024, shared=2048),
}
WINDOW, TAPS, STREAMS, KEEP, BIAS_ROWS = 1024, 4, 4, 4, 32


def hybrid_config(case):
    """The model's ``config.json``; the fourth layer of Zinurax and Lukarax reads earlier rows where there is one to read."""
    s, model = SIZES[case["model"], case["size"]], case["model"]
    out = {"architecture": model.capitalize(), "vocab": HYBRID_VOCAB, "width": s["width"], "norm": {"eps": 1e-5}}
    mask, dense = {"size": WINDOW}, {"kind": "dense", "ff": s.get("dense", s["ff"])}
    moe = {"kind": "moe", "expert": {"ff": s["ff"]}, "router": {"experts": s.get("experts"), "top": s.get("top")}}
    if model == "zinurax":
        yarn = {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}
        latent = {"heads": s["heads"], "dim": s["dim"], "rot_dim": s["rot"], "vdim": s["dim"], "kv_rank": s["kv_rank"], "mask": {"size": 4 * WINDOW},
                  "rot": {"base": 10000.0, "dims": s["rot"], "scaling": yarn}, "scale": (s["dim"] + s["rot"]) ** -0.5}
        cycle = [("general_delta", {"heads": s["d_heads"], "dim": s["d_dim"]}), ("latent_attention", latent),
                 ("general_delta", {"heads": s["d_heads"], "dim": s["d_dim"]}), ("latent_attention", {**latent, "kv_from": 1})]
        ff = [dense] * 4
    elif model == "fabivik":
        for part, width in (("expert", s["ff"]), ("shared", s["shared"])):
            moe[part] = {"ff": width, "limit": 7.0}
        attention = {"heads": s["heads"], "kv_heads": s["groups"], "dim": s["dim"], "vdim": s["dim"], "scale": s["dim"] ** -0.5, "conv": TAPS,
                     "mask": mask, "v_mix": True}
        delta = {"heads": s["d_heads"], "kv_heads": s["d_kv"], "dim": s["d_dim"], "vdim": s["d_dim"], "conv": TAPS}
        cycle = [("attention", attention), ("wkv", {"heads": s["w_heads"], "dim": s["w_dim"]}), ("attention", attention), ("delta", delta)]
        ff = [moe] * 4
        out.update(embedding={"scale": math.sqrt(s["width"])}, logit_scale=1.0)
    elif model == "lukarax":
        moe["router"].update(identity=s["identity"], groups={"count": s["sets"], "keep": s["sets"] // 2}, scale=2.0)
        common = {"heads": s["heads"], "kv_heads": s["groups"], "vdim": s["dim"]}
        diff = {**common, "dim": s["m_dim"], "scale": s["m_dim"] ** -0.5, "diff": 0.3, "rot": {"base": 500000.0, "dims": s["m_dim"]}}
        yarn = {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}
        sink = {**common, "dim": s["dim"], "scale": s["dim"] ** -0.5, "softcap": 20.0, "mask": mask,
                "rot": {"base": 500000.0, "dims": s["dim"] // 2, "scaling": yarn}}
        side = {"left": {**common, "dim": s["dim"], "scale": s["dim"] ** -0.5, "mask": {"size": WINDOW, "keep_first": KEEP}, "bias_max": 128},
                "right": {"heads": s["m_heads"], "dim": s["dim"], "vdim": s["dim"], "gate_cap": 15.0}, "left_scale": 0.8, "right_scale": 0.9}
        cycle = [("attention", diff), ("parallel", side), ("attention_2", sink), ("attention", {**diff, "kv_from": 0})]
        ff = [dense, moe, moe, moe]
        out.update(embedding={"scale": math.sqrt(s["width"])}, streams=STREAMS)
    else:
        moe["shared"] = {"ff": s["shared"]}
        windowed = {"heads": s["heads"], "kv_heads": s["groups"], "dim": s["dim"], "vdim": s["dim"], "scale": s["dim"] ** -0.5, "mask": mask, "v_mix": True,
                    "rot": {"base": 500000.0, "dims": s["rot"]}}
        latent = {"heads": s["heads"], "dim": s["dim"], "vdim": s["dim"], "kv_rank": s["kv_rank"], "q_rank": s["q_rank"], "scale": s["dim"] ** -0.5}
        cycle = [("mingru", {"width": s["scan"]}), ("attention", windowed), ("mingru", {"width": s["scan"]}), ("latent_attention", latent)]
        ff = [moe] * 4
        out.update(embedding={"scale": math.sqrt(s["width"])}, canon={"taps": TAPS})
    out["layers"] = [{"type": cycle[i % 4][0], "mixer": cycle[i % 4][1], "mlp": ff[i % 4]} for i in range(case["layers"])]
    return out


def columns_of(cfg):
    """(router outputs, groups of them, experts per token) of a design with experts."""
    r = next((x["mlp"]["router"] for x in cfg["layers"] if x["mlp"]["kind"] == "moe"), None)
    return None if r is None else (r["experts"] + r.get("identity", 0), (r.get("groups") or {"count": 1})["count"], r["top"])


def feature_of(layer, column, columns, groups):
    """The embedding feature that router output ``column`` of a layer looks at: another one in every layer, groups kept together."""
    size = columns // groups
    return ((column // size + layer) % groups) * size + (column % size + 3 * layer) % size


def embedding(noise, cfg, seed):
    """Unit-scale rows; the first ones of their features say which experts a token takes."""
    W, V = cfg["width"], cfg["vocab"]
    e = noise("embed", V, W)
    if columns_of(cfg) is not None:
        columns, groups, top = columns_of(cfg)
        g = torch.Generator(device="cuda").manual_seed(seed * 31 + 7)
        score = torch.rand(V, columns, generator=g, device="cuda")
        if groups > 1:  # experts of the groups a token keeps
            order = torch.rand(V, groups, generator=g, device="cuda").argsort(dim=1) < groups // 2
            score = score + order.repeat_interleave(columns // groups, dim=1).float()
        chosen = torch.zeros(V, columns, device="cuda").scatter_(1, score.topk(top, dim=1).indices, 1.0)
        e[:, :columns] = (chosen * (5.0 + 2.0 * torch.rand(V, columns, generator=g, device="cuda"))).to(BF16)
    return e


def hybrid_weights(case, seed):
    cfg, s, noise = hybrid_config(case), SIZES[case["model"], case["size"]], Noise(seed)
    W, model, out = s["width"], case["model"], {}
    routed = columns_of(cfg)
    kept = 0 if routed is None else routed[0]  # features of the stream that no sublayer writes to
    scale = cfg.get("embedding", {"scale": 1.0})["scale"]
    off = 0.0 if model == "fabivik" else 1.0

    def put(name, *shape, std=None, mean=0.0, gain=1.0):
        out[name] = noise(name, *shape, std=gain / math.sqrt(shape[-1]) if std is None else std, mean=mean)

    def out_proj(name, k):
        put(name, W, k)
        out[name][:kept] = 0

    out["embed"] = embedding(noise, cfg, seed).mul_(1.0 / scale)
    put("final.norm", W, std=0.2, mean=off)
    if model == "zinurax":
        put("embed.norm", W, std=0.2, mean=1.0)
    elif model == "lukarax":
        put("final.norm.b", W, std=0.1)
    else:
        put("head", HYBRID_VOCAB, W)
    mixing = 0
    for i, layer in enumerate(cfg["layers"]):
        p, m, kind, mlp = f"l{i}.mix.", layer["mixer"], layer["type"], layer["mlp"]
        put(f"l{i}.norm1", W, std=0.2, mean=off)
        if model == "fabivik":
            put(f"l{i}.norm2", W, std=0.2, mean=off)
        elif model == "zinurax":
            put(f"l{i}.norm2", W, std=0.2, mean=off)
        elif model == "maginex":
            for n in (1, 2):
                put(f"l{i}.canon{n}", W, TAPS, std=0.3)
            out[f"l{i}.canon2"][:kept] = 0
        else:
            put(f"l{i}.norm2", W, std=0.2, mean=off)
            for n in (1, 2):
                put(f"l{i}.norm{n}.b", W, std=0.1)
                put(f"l{i}.hc{n}.in", STREAMS, std=0.05, mean=1.0 / STREAMS)
                put(f"l{i}.hc{n}.out", STREAMS, std=0.2, mean=0.8)
                out[f"l{i}.hc{n}.mix"] = (0.9 * torch.eye(STREAMS, device="cuda") + 0.1 / STREAMS + noise(f"l{i}.hc{n}.mix", STREAMS, STREAMS, std=0.02)).to(BF16)
        if kind == "general_delta":
            n = m["heads"] * m["dim"]
            for k in ("r", "k", "v", "g", "a"):
                put(p + k, n, W)
            put(p + "a.b", n, std=1.0), put(p + "w0", n, std=2.0, mean=-2.0), put(p + "w1", s["rank"], W), put(p + "w2", n, s["rank"])
            put(p + "norm", n, std=0.2, mean=1.0), put(p + "o", W, n)
        elif kind == "latent_attention":
            H, rank = m["heads"], m["kv_rank"]
            if model == "zinurax":
                put(p + "q", H * (m["dim"] + m["rot_dim"]), W, gain=2.0), put(p + "g", H, W)
            else:
                put(p + "dq", m["q_rank"], W), put(p + "dq.norm", m["q_rank"], std=0.2, mean=1.0), put(p + "uq", H * m["dim"], m["q_rank"], gain=2.0)
                put(p + "sink", H, std=1.0, mean=1.0), put(p + "g", H * m["vdim"], W)
            if "kv_from" not in m:
                put(p + "dkv", rank + m.get("rot_dim", 0), W), put(p + "dkv.norm", rank, std=0.2, mean=1.0)
            put(p + "uk", H * m["dim"], rank), put(p + "uv", H * m["vdim"], rank)
            out_proj(p + "o", H * m["vdim"])
        elif kind == "wkv":
            n = m["heads"] * m["dim"]
            for k in "rkvg":
                put(p + k, n, W)
            for k in "rkvgw":
                out[p + "mu." + k] = torch.sigmoid(noise(p + "mu." + k, W))
            put(p + "w1", s["rank"], W), put(p + "w2", n, s["rank"]), put(p + "w0", n, std=2.0, mean=-3.0), put(p + "u", m["heads"], m["dim"], std=0.5, mean=0.5)
            put(p + "norm", n, std=0.2, mean=1.0), out_proj(p + "o", n)
        elif model == "fabivik":
            H, G = m["heads"], m["kv_heads"]
            for k, heads, size in zip("qkv", (H, G, G) if kind == "attention" else (G, G, H), (m["dim"], m["dim"], m["vdim"])):
                put(p + k, heads * size, W), put(p + k + ".conv", heads * size, TAPS, std=0.4)
                out[p + k + ".conv"][:, -1] += 1.0
            out_proj(p + "o", H * m["vdim"])
            if kind == "attention":
                put(p + "q.norm", m["dim"], std=0.2, mean=1.5), put(p + "k.norm", m["dim"], std=0.2, mean=1.5)
                if mixing:
                    out[p + "vmix"] = torch.tensor(0.3, device="cuda").to(BF16)
                mixing += 1
            else:
                put(p + "g", H * m["vdim"], W), put(p + "b", H, W, gain=2.0), put(p + "a", H, W)
                put(p + "A_log", H, std=0.7), put(p + "dt_bias", H, std=1.5, mean=-2.5), put(p + "norm", m["vdim"], std=0.2, mean=1.0)
        elif kind == "parallel":
            a, r = m["left"], m["right"]
            for k, n in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                put(p + "left." + k, n, W)
            put(p + "left.rel", BIAS_ROWS, a["heads"], std=1.0), out_proj(p + "left.o", a["heads"] * a["vdim"])
            h, n = r["heads"], r["heads"] * r["vdim"]
            for k, rows in (("q", h * r["dim"]), ("k", h * r["dim"]), ("v", n), ("g", n), ("i", h), ("f", h)):
                put(p + "right." + k, rows, W)
            put(p + "right.i.b", h, std=0.5, mean=-0.5), put(p + "right.f.b", h, std=1.5, mean=2.5), put(p + "right.norm", n, std=0.2, mean=1.0)
            out_proj(p + "right.o", n)
        elif kind == "attention_2":
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            put(p + "q", H * d, W), put(p + "q.b", H * d, std=0.3), put(p + "k", G * d, W), put(p + "k.b", G * d, std=0.3)
            put(p + "sink", H, std=1.0, mean=1.0), out_proj(p + "o", H * d), put(p + "o.b", W, std=0.2)
            out[p + "o.b"][:kept] = 0
        elif kind == "mingru":
            n = m["width"]
            for k in "zxg":
                put(p + k, n, W, gain=1.5)
            put(p + "z.b", n, std=1.5, mean=-1.5), put(p + "x.b", n, std=0.5), out_proj(p + "o", n)
        elif model == "lukarax":
            H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            put(p + "q", H * 2 * d, W)
            if "kv_from" not in m:
                put(p + "k", G * 2 * d, W), put(p + "v", G * dv, W)
            for k in ("lq1", "lk1", "lq2", "lk2"):
                put(p + k, d, std=0.7 / d ** 0.25)
            put(p + "g", H * dv, W), out_proj(p + "o", H * dv)
        else:
            H, G = m["heads"], m["kv_heads"]
            put(p + "q", H * m["dim"], W), put(p + "k", G * m["dim"], W), put(p + "v", G * m["vdim"], W)
            put(p + "sink", H, std=1.0, mean=1.0), put(p + "g", H, W), out_proj(p + "o", H * m["vdim"])
            out[p + "vmix"] = torch.tensor(0.35, device="cuda").to(BF16)
        p = f"l{i}.mlp."
        if mlp["kind"] == "dense":
            parts = [("", mlp["ff"])]
        else:
            columns, groups, _ = routed
            put(p + "router", columns, W, std=0.1 / math.sqrt(W))
            out[p + "router"][:, :kept] = 0
            for e in range(columns):
                out[p + "router"][e, feature_of(i, e, columns, groups)] = 1.2
            out[f"l{i}.norm{1 if model == 'maginex' else 2}"][:kept] = off  # (what the router reads is scaled alike for every token)
            if model == "lukarax":
                put(p + "correction", columns, std=0.002)
            elif model == "maginex":
                put(p + "router.b", columns, std=0.1)
            parts = [(f"e{e}.", mlp["expert"]["ff"]) for e in range(mlp["router"]["experts"])]
            if "shared" in mlp:
                parts.append(("shared.", mlp["shared"]["ff"]))
                if model == "fabivik":
                    put(p + "shared.sg", 1, W)
        for name, ff in parts:
            if model in ("fabivik", "lukarax"):
                put(p + name + "gate", ff, W, gain=2.0)
            put(p + name + "up", ff, W), out_proj(p + name + "down", ff)
    return out


def prepare_hybrid(case, seed):
    from megatron_mixtera_b200 import model_registry as R

    lengths, ids, w, cfg = lengths_of(case), tokens_of(case, seed), hybrid_weights(case, seed), hybrid_config(case)
    model = R.ARCHITECTURES[cfg["architecture"]](cfg, {k: tuple(v.shape) for k, v in w.items()}, BF16, max(lengths) + 64)
    model.load_checkpoint(w)
    del w
    model.config.enable_cuda_graph = True
    portion = max(16384, max(lengths)) if case["step"] == "decode" else sum(lengths)
    ctx = R.make_context(model, max_cached_tokens=sum(-(-n // CHUNK) for n in lengths) * CHUNK, max_requests=len(lengths),
                         max_step_tokens=max(portion, len(lengths)), chunk_size_tokens=CHUNK)
    controller = R.make_controller(model, ctx)
    if case["step"] == "prefill":
        ctx.schedule_tokens(list(enumerate(ids)))
    else:
        step = []
        for r, t in enumerate(ids):  # everything in front of the newest tokens, in a few steps
            if step and sum(len(x) for _, x in step) + len(t) > portion:
                controller.run_given_tokens(step, [[] for _ in step])
                step = []
            if len(t) > 1:
                step.append((r, t[:-1]))
        if step:
            controller.run_given_tokens(step, [[] for _ in step])
        ctx.schedule_tokens([(r, t[-1:]) for r, t in enumerate(ids)])
    return ctx, controller.inference_wrapped_model


# ---------------------------------------------------------------------------------------------------------------------
class Served:
    """A model, its context and the step they are about to run.  The cache's memory is given back with it."""

    def __init__(self, context, wrapper):
        self.context, self.wrapper = context, wrapper

    def __del__(self):
        for pool in [self.context.memory_buffer] + (self.context.latent_buffers or []):
            if pool is not None:
                pool.untyped_storage().resize_(0)


def prepare(case, seed):
    with torch.no_grad():
        return Served(*(prepare_gpt if case["model"] == "gpt" else prepare_hybrid)(case, seed))


def run(state):
    """Logits of the step's last token per request.  (A step writes the same rows and states whenever it is repeated: the context counts a step
    only when it is told that it is over.)"""
    ctx = state.context
    ctx.initialize_attention_state()
    ids, positions = ctx.current_input_and_position_ids()
    return state.wrapper.run_one_forward_step({"tokens": ids, "position_ids": positions, "attention_mask": None})


def work(case):
    """Weights that the step's tokens reach, cached rows and states, logits; products of linears, attention and recurrences."""
    lengths, decode = lengths_of(case), case["step"] == "decode"
    T, B = (len(lengths) if decode else sum(lengths)), len(lengths)

    def pairs(window=None):
        if decode:
            return sum(min(n, window or n) for n in lengths)
        return sum(n * (n + 1) // 2 if not window or n <= window else window * (window + 1) // 2 + (n - window) * window for n in lengths)

    if case["model"] == "gpt":
        s, L = GPT[case["size"]], case["layers"]
        linear = s["width"] * (s["heads"] + 2 * s["groups"]) * s["dim"] + s["width"] * s["heads"] * s["dim"] + 3 * s["width"] * s["ff"]
        per_weight = {"bf16": 2.0, "mxfp8": 33 / 32, "mxfp8_kv8": 33 / 32, "blockwise": 1.0 + 4 / 16384}[case["precision"]]
        per_value = 1 if case["precision"] == "mxfp8_kv8" else 2
        head = s["vocab"] * s["width"]
        return {"bytes": L * (linear * per_weight + 2 * s["groups"] * s["dim"] * per_value * sum(lengths)) + 2.0 * head + 2.0 * B * s["vocab"] + 2.0 * T * s["width"],
                "flops": L * (2.0 * linear * T + 4.0 * s["heads"] * s["dim"] * pairs()) + 2.0 * head * B}
    cfg, s, W = hybrid_config(case), SIZES[case["model"], case["size"]], SIZES[case["model"], case["size"]]["width"]
    nbytes, flops = 2.0 * HYBRID_VOCAB * (W + B), 2.0 * HYBRID_VOCAB * W * B
    for layer in cfg["layers"]:
        kind, m, mlp = layer["type"], layer["mixer"], layer["mlp"]
        if kind == "latent_attention":
            H, d, r = m["heads"], m["dim"], m.get("rot_dim", 0)
            up = H * (d + m["vdim"]) * m["kv_rank"]
            size = (W * H * (d + r) if "q_rank" not in m else m["q_rank"] * (W + H * d) + W * H * m["vdim"]) + W * (m["kv_rank"] + r) + up + W * H * m["vdim"]
            window = (m.get("mask") or {}).get("size")
            nbytes += 2.0 * (m["kv_rank"] + r) * (pairs(window) if decode else T)
            flops += 2.0 * pairs(window) * H * (2 * m["kv_rank"] + r if decode else d + r + m["vdim"])
        elif kind in ("general_delta", "wkv", "delta"):
            H, d = m["heads"], m["dim"]
            size = W * H * d * (4 if kind == "delta" else 6)
            nbytes, flops = nbytes + (8.0 if decode else 4.0) * B * H * d * d, flops + 8.0 * T * H * d * d
        elif kind == "mingru":
            size = 4 * W * m["width"]
        else:
            a = m.get("left", m)
            maps = 2 if "diff" in a else 1
            size = W * (a["heads"] * (a["dim"] * maps + a["vdim"] * (2 if maps == 2 else 1)) + a["kv_heads"] * (a["dim"] * maps + a["vdim"]))
            window = (a.get("mask") or {}).get("size")
            nbytes += 2.0 * a["kv_heads"] * (maps * a["dim"] + a["vdim"]) * (pairs(window) if decode else T)
            flops += 2.0 * pairs(window) * a["heads"] * maps * (a["dim"] + a["vdim"])
            if "right" in m:
                r = m["right"]
                size += 5 * W * r["heads"] * r["dim"]
                nbytes, flops = nbytes + (8.0 if decode else 4.0) * B * r["heads"] * r["dim"] ** 2, flops + 6.0 * T * r["heads"] * r["dim"] ** 2
        nbytes, flops = nbytes + 2.0 * size, flops + 2.0 * size * T
        products = 2 if case["model"] in ("zinurax", "maginex") else 3
        if mlp["kind"] == "dense":
            nbytes, flops = nbytes + 2.0 * products * W * mlp["ff"], flops + 2.0 * T * products * W * mlp["ff"]
        else:
            E, top, shared = mlp["router"]["experts"], mlp["router"]["top"], (mlp.get("shared") or {"ff": 0})["ff"]
            reached = E * (1.0 - (1.0 - top / E) ** T)
            nbytes += 2.0 * products * W * (reached * s["ff"] + shared)
            flops += 2.0 * T * products * W * (top * s["ff"] + shared)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Outputs are bf16 logits behind a few layers of 16-bit or 8-bit activations: against 64 bits they are 0.5 to 0.8 % off (Zinurax, whose recurrences
    carry what they read for long: 2 %), with 8-bit activations 3 to 7 %.  A sum in another order moves some of those roundings."""
    return {"rel": 0.02 if case["precision"] == "bf16" and case["model"] != "zinurax" else 0.03, "max": 0.3}


# ---------------------------------------------------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def e4m3(x):
    return x.clamp(-448.0, 448.0).to(torch.float8_e4m3fn).to(F64)


def linear64(w, precision):
    """A weight as the model holds it: bf16, or E4M3 with a power of two per 32 inputs, or with a scale per 128 x 128 block."""
    n, k = w.shape
    if precision.startswith("mxfp8"):
        x = w.double().view(n, k // 32, 32)
        top = x.abs().amax(dim=-1, keepdim=True).clamp_min(2.0 ** -120)
        scale = torch.exp2(torch.ceil(torch.log2(top / 448.0)))
        return (e4m3(x / scale) * scale).view(n, k)
    if precision == "blockwise":
        x = w.double().view(n // 128, 128, k // 128, 128)
        scale = x.abs().amax(dim=(1, 3), keepdim=True).clamp_min(1e-30) / 448.0
        return (e4m3(x / scale) * scale).view(n, k)
    return w.double()


def rms64(x, weight=None, eps=1e-5):
    y = x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def layer_norm64(x, weight, bias=0.0, eps=1e-5):
    d = x - x.mean(dim=-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(dim=-1, keepdim=True) + eps) * weight + bias


def silu64(x):
    return x * torch.sigmoid(x)


def rotate64(x, positions, base, dims, halves, scaling=None):
    """x [T, heads, dim]: the first ``dims`` turn, in pairs (i, i + dims / 2) or (2i, 2i + 1), with YaRN's frequencies where scaled."""
    freq, mag = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    if scaling:
        def where(turns):
            return dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

        lo, hi = max(math.floor(where(scaling["fast"])), 0), min(math.ceil(where(scaling["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        freq = [f / scaling["factor"] * a + f * (1.0 - a) for f, a in zip(freq, ramp)]
        mag = 0.1 * math.log(scaling["factor"]) + 1.0
    angle = positions.double()[:, None] * torch.tensor(freq, dtype=F64, device=x.device)
    c, s = (torch.cos(angle) * mag)[:, None, :], (torch.sin(angle) * mag)[:, None, :]
    out = x.clone()
    i = torch.arange(dims // 2, device=x.device)
    iu, iv = (i, i + dims // 2) if halves else (2 * i, 2 * i + 1)
    u, v = x[..., iu], x[..., iv]
    out[..., iu], out[..., iv] = u * c - v * s, v * c + u * s
    return out


def attend64(q, k, v, scale, size=None, keep=0, bias=None, cap=None, sink=None):
    """One request: queries [Tq, H, d] are its newest tokens, keys [Tk, G, d], values [Tk, G, dv]; ``bias`` [distance, H], ``sink`` [H]."""
    tq, tk, group = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    age = torch.arange(tk - tq, tk, device=q.device)[:, None] - torch.arange(tk, device=q.device)[None, :]
    seen = age >= 0
    if size is not None:
        seen = seen & ((age < size) | (torch.arange(tk, device=q.device) < keep))
    out = torch.empty(tq, q.shape[1], v.shape[2], dtype=F64, device=q.device)
    for h in range(q.shape[1]):
        score = q[:, h].double() @ k[:, h // group].double().T * scale
        if cap:
            score = cap * torch.tanh(score / cap)
        if bias is not None:
            score = score + bias[:, h][age.clamp(min=0)]
        score = score.masked_fill(~seen, -math.inf)
        if sink is not None:
            score = torch.cat([score, sink[h].expand(tq, 1)], dim=1)
        out[:, h] = torch.softmax(score, dim=-1)[:, :tk] @ v[:, h // group].double()
    return out


def exact_gpt(case, seed):
    s, w, lengths, ids = GPT[case["size"]], gpt_weights(case, seed), lengths_of(case), tokens_of(case, seed)
    H, G, d = s["heads"], s["groups"], s["dim"]
    decode, scale = case["step"] == "decode", KV8_SCALE if case["precision"] == "mxfp8_kv8" else 1.0
    flat = torch.cat(ids).cuda()
    counts = [len(t) for t in ids]
    pos = torch.cat([torch.arange(n - c, n) for n, c in zip(lengths, counts)]).cuda()
    x = w["embedding.word_embeddings.weight"][flat].double()
    for i in range(case["layers"]):
        p = f"decoder.layers.{i}."
        h = rms64(x, w[p + "input_layernorm.weight"].double())
        qkv = (h @ linear64(w[p + "self_attention.linear_qkv.weight"], case["precision"]).T).view(-1, G, H // G + 2, d)
        q = rotate64(qkv[:, :, :-2].reshape(-1, H, d), pos, s["base"], d, True)
        k, v = rotate64(qkv[:, :, -2], pos, s["base"], d, True), qkv[:, :, -1]
        y, a = torch.empty_like(q), 0
        for r, (n, c) in enumerate(zip(lengths, counts)):
            b = a + c
            if decode and n > 1:
                old = cached(case, seed, i, r, n - 1)
                for g in range(G):
                    both = old[:, :, g].double() * scale
                    y[a:b, g * H // G:(g + 1) * H // G] = attend64(q[a:b, g * H // G:(g + 1) * H // G], torch.cat([both[0], k[a:b, g]])[:, None],
                                                                   torch.cat([both[1], v[a:b, g]])[:, None], d ** -0.5)
            else:
                y[a:b] = attend64(q[a:b], k[a:b], v[a:b], d ** -0.5)
            a = b
        x = x + y.reshape(-1, H * d) @ linear64(w[p + "self_attention.linear_proj.weight"], case["precision"]).T
        h = rms64(x, w[p + "pre_mlp_layernorm.weight"].double())
        gate, up = (h @ linear64(w[p + "mlp.linear_fc1.weight"], case["precision"]).T).chunk(2, dim=-1)
        x = x + (silu64(gate) * up) @ linear64(w[p + "mlp.linear_fc2.weight"], case["precision"]).T
    last = torch.tensor(counts).cumsum(0).cuda() - 1
    return (rms64(x[last], w["decoder.final_layernorm.weight"].double()) @ w["output_layer.weight"].double().T)[None]


class Sequences:
    """Rows of several requests back to back, and what needs to know where one ends."""

    def __init__(self, lengths):
        self.lengths = lengths
        self.pos = torch.cat([torch.arange(n) for n in lengths]).cuda()
        self.starts = [sum(lengths[:i]) for i in range(len(lengths))]
        t = torch.arange(max(lengths)).expand(len(lengths), -1)
        self.grid = (torch.tensor(self.starts)[:, None] + torch.minimum(t, torch.tensor(lengths)[:, None] - 1)).cuda()
        self.valid = (t < torch.tensor(lengths)[:, None]).cuda()

    def parts(self):
        return [slice(a, a + n) for a, n in zip(self.starts, self.lengths)]

    def past(self, x, age):
        return x if age == 0 else torch.where((self.pos >= age)[:, None], x.roll(age, 0), 0.0)

    def conv(self, x, taps):
        n = taps.shape[1]
        return sum(taps[:, n - 1 - age] * self.past(x, age) for age in range(n))

    def steps(self, *xs):
        """Per token number, the rows of all requests (repeated past a request's end, where nothing is read)."""
        for t in range(self.grid.shape[1]):
            yield t, [x[self.grid[:, t]] for x in xs]

    def attend(self, q, k, v, scale, **kw):
        return torch.cat([attend64(q[p], k[p], v[p], scale, **kw) for p in self.parts()])


def outer64(k, v):
    return k[..., :, None] * v[..., None, :]


def read64(S, q):
    return (q[..., None, :] @ S)[..., 0, :]


def moe64(model, x, w, p, mlp):
    r, z = mlp["router"], x @ w(p + "router").T
    if model == "fabivik":
        weight, chosen = torch.sigmoid(z).topk(r["top"], dim=-1)
    elif model == "maginex":
        weight, chosen = (z + w(p + "router.b")).topk(r["top"], dim=-1)
        weight = torch.softmax(weight, dim=-1)
    else:
        score, count = torch.softmax(z, dim=-1), r["groups"]["count"]
        sets = (score + w(p + "correction")).view(len(x), count, -1)
        opened = torch.zeros(len(x), count, dtype=torch.bool, device=x.device).scatter_(1, sets.amax(-1).topk(r["groups"]["keep"]).indices, True)
        chosen = sets.masked_fill(~opened[:, :, None], -math.inf).view(len(x), -1).topk(r["top"], dim=-1).indices
        weight = score.gather(1, chosen)
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20) * r["scale"]

    def ff(h, name):
        if model == "maginex":
            return torch.relu(h @ w(p + name + ".up").T).square() @ w(p + name + ".down").T
        g, u = h @ w(p + name + ".gate").T, h @ w(p + name + ".up").T
        if model == "fabivik":
            limit = mlp["expert"]["limit"]
            g, u = g.clamp(max=limit), u.clamp(-limit, limit) + 1.0
            return (g * torch.sigmoid(1.702 * g) * u) @ w(p + name + ".down").T
        return (silu64(g) * u) @ w(p + name + ".down").T

    out = torch.zeros_like(x)
    for e in range(r["experts"] + r.get("identity", 0)):
        t, k = (chosen == e).nonzero(as_tuple=True)
        if len(t):
            a = weight[t, k][:, None]
            out[t] += ff(a * x[t], f"e{e}") if model == "fabivik" else a * (ff(x[t], f"e{e}") if e < r["experts"] else x[t])
    if "shared" in mlp:
        out = out + (torch.sigmoid(x @ w(p + "shared.sg").T) if model == "fabivik" else 1.0) * ff(x, "shared")
    return out


def mixer64(model, layer, h, w, p, seq, carried, index):
    kind, m, T = layer["type"], layer["mixer"], len(h)
    mask = m.get("mask") or {}
    if kind == "general_delta":
        shape = (T, m["heads"], m["dim"])
        r, k, v = ((h @ w(p + n).T).view(shape) for n in "rkv")
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0"))).view(shape)
        a = torch.sigmoid(h @ w(p + "a").T + w(p + "a.b")).view(shape)
        u, o = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6), torch.empty_like(v)
        S = torch.zeros(len(seq.lengths), m["heads"], m["dim"], m["dim"], dtype=F64, device=h.device)
        for t, (rt, kt, vt, dt, at, ut) in seq.steps(r, k, v, decay, a, u):
            S = dt[..., None] * S - outer64(at * ut, read64(S, ut)) + outer64(kt, vt)
            o[seq.grid[seq.valid[:, t], t]] = read64(S, rt)[seq.valid[:, t]]
        return (rms64(o).reshape(T, -1) * w(p + "norm") * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T
    if kind == "latent_attention":
        H, d, rank = m["heads"], m["dim"], m["kv_rank"]
        if model == "zinurax":
            rot = m["rot"]
            turn = lambda x: rotate64(x, seq.pos, rot["base"], rot["dims"], False, rot["scaling"])  # noqa: E731
            if "kv_from" not in m:
                c = h @ w(p + "dkv").T
                carried[index] = rms64(c[:, :rank], w(p + "dkv.norm")), turn(c[:, None, rank:])
            c, k_rot = carried[m.get("kv_from", index)]
            q = (h @ w(p + "q").T).view(T, H, -1)
            q = torch.cat([q[..., :d], turn(q[..., d:].contiguous())], dim=-1)
            k = torch.cat([(c @ w(p + "uk").T).view(T, H, d), k_rot.expand(-1, H, -1)], dim=-1)
            o = seq.attend(q, k, (c @ w(p + "uv").T).view(T, H, -1), m["scale"], size=mask.get("size"))
            return (o * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).reshape(T, -1) @ w(p + "o").T
        q = (rms64(h @ w(p + "dq").T, w(p + "dq.norm")) @ w(p + "uq").T).view(T, H, d)
        c = rms64(h @ w(p + "dkv").T, w(p + "dkv.norm"))
        o = seq.attend(q, (c @ w(p + "uk").T).view(T, H, d), (c @ w(p + "uv").T).view(T, H, -1), m["scale"], sink=w(p + "sink"))
        return (o.reshape(T, -1) * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T
    if kind == "wkv":
        prev, shape = seq.past(h, 1), (T, m["heads"], m["dim"])
        mix = {n: h + (prev - h) * w(p + "mu." + n) for n in "rkvgw"}
        r, k, v = ((mix[n] @ w(p + n).T).view(shape) for n in "rkv")
        decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0"))).view(shape)
        bonus, o = w(p + "u"), torch.empty_like(v)
        S = torch.zeros(len(seq.lengths), m["heads"], m["dim"], m["dim"], dtype=F64, device=h.device)
        for t, (rt, kt, vt, dt) in seq.steps(r, k, v, decay):
            kv = outer64(kt, vt)
            o[seq.grid[seq.valid[:, t], t]] = read64(S + bonus[..., None] * kv, rt)[seq.valid[:, t]]
            S = dt[..., None] * S + kv
        return (rms64(o).reshape(T, -1) * w(p + "norm") * silu64(mix["g"] @ w(p + "g").T)) @ w(p + "o").T
    if kind == "delta":
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (silu64(seq.conv(h @ w(p + n).T, w(p + n + ".conv"))) for n in "qkv")
        q, k = ((y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1) for y in (q.view(T, G, d), k.view(T, G, d)))
        q, v, beta = q * d ** -0.5, v.view(T, H, -1), torch.sigmoid(h @ w(p + "b").T)
        decay = torch.exp(-torch.exp(w(p + "A_log")) * torch.nn.functional.softplus(h @ w(p + "a").T + w(p + "dt_bias")))
        o = torch.empty_like(v)
        S = torch.zeros(len(seq.lengths), H, d, v.shape[2], dtype=F64, device=h.device)
        for t, (qt, kt, vt, bt, dt) in seq.steps(q, k, v, beta, decay):
            S = dt[..., None, None] * S
            S = S + outer64(kt, bt[..., None] * (vt - read64(S, kt)))
            o[seq.grid[seq.valid[:, t], t]] = read64(S, qt)[seq.valid[:, t]]
        return ((rms64(o) * w(p + "norm")).reshape(T, -1) * silu64(h @ w(p + "g").T)) @ w(p + "o").T
    if kind == "mingru":
        z = torch.sigmoid(h @ w(p + "z").T + w(p + "z.b"))
        u = h @ w(p + "x").T + w(p + "x.b")
        c, o = torch.where(u >= 0, u + 0.5, torch.sigmoid(u)), torch.empty_like(z)
        S = torch.zeros(len(seq.lengths), z.shape[1], dtype=F64, device=h.device)
        for t, (zt, ct) in seq.steps(z, c):
            S = (1 - zt) * S + zt * ct
            o[seq.grid[seq.valid[:, t], t]] = S[seq.valid[:, t]]
        return (o * silu64(h @ w(p + "g").T)) @ w(p + "o").T
    if kind == "parallel":
        a, r = m["left"], m["right"]
        q, k, v = ((h @ w(p + "left." + n).T).view(T, heads, -1) for n, heads in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])))
        half, longest = BIAS_ROWS // 2, a["bias_max"]
        rows = [n if n < half else min(BIAS_ROWS - 1, half + math.floor(math.log(n / half) / math.log(longest / half) * (BIAS_ROWS - half)))
                for n in range(max(seq.lengths))]
        left = seq.attend(q, k, v, a["scale"], size=a["mask"]["size"], keep=a["mask"]["keep_first"], bias=w(p + "left.rel")[rows])
        H, d, cap = r["heads"], r["dim"], r["gate_cap"]
        q, k, v = ((h @ w(p + "right." + n).T).view(T, H, -1) for n in "qkv")
        gi, gf = (cap * torch.tanh((h @ w(p + "right." + n).T + w(p + "right." + n + ".b")) / cap) for n in "if")
        q, gf, o = q * d ** -0.5, torch.nn.functional.logsigmoid(gf), torch.empty_like(v)
        B = len(seq.lengths)
        S, total = torch.zeros(B, H, d, v.shape[2], dtype=F64, device=h.device), torch.zeros(B, H, d, dtype=F64, device=h.device)
        top = torch.zeros(B, H, dtype=F64, device=h.device)
        for t, (qt, kt, vt, it, ft) in seq.steps(q, k, v, gi, gf):
            new = torch.maximum(ft + top, it)
            keep, write, top = torch.exp(ft + top - new), torch.exp(it - new), new
            S, total = keep[..., None, None] * S + outer64(write[..., None] * kt, vt), keep[..., None] * total + write[..., None] * kt
            below = torch.maximum((total * qt).sum(-1).abs(), torch.exp(-top)) + 1e-6
            o[seq.grid[seq.valid[:, t], t]] = (read64(S, qt) / below[..., None])[seq.valid[:, t]]
        right = rms64(o).reshape(T, -1) * w(p + "right.norm") * torch.sigmoid(h @ w(p + "right.g").T)
        return m["left_scale"] * (left.reshape(T, -1) @ w(p + "left.o").T) + m["right_scale"] * (right @ w(p + "right.o").T)
    H, G, rot = m["heads"], m["kv_heads"], m.get("rot")
    if kind == "attention_2":
        q = (h @ w(p + "q").T + w(p + "q.b")).view(T, H, -1)
        v = (h @ w(p + "k").T + w(p + "k.b")).view(T, G, -1)
        q, k = (rms64(rotate64(y, seq.pos, rot["base"], rot["dims"], True, rot["scaling"])) for y in (q, v))
        o = seq.attend(q, k, v, m["scale"], size=mask.get("size"), cap=m["softcap"], sink=w(p + "sink"))
        return o.reshape(T, -1) @ w(p + "o").T + w(p + "o.b")
    if model == "lukarax":
        d = m["dim"]
        if "kv_from" not in m:
            carried[index] = (rotate64((h @ w(p + "k").T).view(T, G * 2, d), seq.pos, rot["base"], rot["dims"], False).view(T, G, 2, d),
                              (h @ w(p + "v").T).view(T, G, -1))
        k, v = carried[m.get("kv_from", index)]
        q = rotate64((h @ w(p + "q").T).view(T, H * 2, d), seq.pos, rot["base"], rot["dims"], False).view(T, H, 2, d)
        a1, a2 = (seq.attend(q[:, :, i], k[:, :, i], v, m["scale"], size=mask.get("size")) for i in range(2))
        share = torch.exp((w(p + "lq1") * w(p + "lk1")).sum()) - torch.exp((w(p + "lq2") * w(p + "lk2")).sum()) + m["diff"]
        o = rms64(a1 - share * a2) * (1.0 - m["diff"])
        return (o.reshape(T, -1) * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T
    q, k, v = ((h @ w(p + n).T) for n in "qkv")
    if model == "fabivik":
        q, k, v = (seq.conv(y, w(p + n + ".conv")) for n, y in (("q", q), ("k", k), ("v", v)))
    q, k, v = q.view(T, H, -1), k.view(T, G, -1), v.view(T, G, -1)
    if "first" in carried:
        v = (1.0 - w(p + "vmix")) * v + w(p + "vmix") * carried["first"]
    else:
        carried["first"] = v
    if model == "fabivik":
        q, k = rms64(q) * w(p + "q.norm"), rms64(k) * w(p + "k.norm")
        return seq.attend(q, k, v, m["scale"], size=mask.get("size")).reshape(T, -1) @ w(p + "o").T
    q, k = (rotate64(y, seq.pos, rot["base"], rot["dims"], True) for y in (q, k))
    o = seq.attend(q, k, v, m["scale"], size=mask.get("size"), sink=w(p + "sink"))
    return (o * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).reshape(T, -1) @ w(p + "o").T


def exact_hybrid(case, seed):
    cfg, held, model = hybrid_config(case), hybrid_weights(case, seed), case["model"]
    seq, flat, carried = Sequences(lengths_of(case)), torch.cat(tokens_of(case, seed)).cuda(), {}

    def w(name):
        return held[name].double()

    last = torch.tensor(seq.lengths).cumsum(0).cuda() - 1
    x = held["embed"][flat].double() * cfg.get("embedding", {"scale": 1.0})["scale"]
    if model == "zinurax":
        x = layer_norm64(x, w("embed.norm"))
    if model == "lukarax":
        x = x[None].repeat(STREAMS, 1, 1)
    for i, layer in enumerate(cfg["layers"]):
        p, mlp = f"l{i}.", layer["mlp"]
        if model == "zinurax":
            x = x + layer_norm64(mixer64(model, layer, x, w, p + "mix.", seq, carried, i), w(p + "norm1"))
            x = x + layer_norm64(torch.relu(x @ w(p + "mlp.up").T).square() @ w(p + "mlp.down").T, w(p + "norm2"))
        elif model == "fabivik":
            y = mixer64(model, layer, rms64(x, 1.0 + w(p + "norm1")), w, p + "mix.", seq, carried, i)
            x = x + y + moe64(model, rms64(x, 1.0 + w(p + "norm2")), w, p + "mlp.", mlp)
        elif model == "maginex":
            h = rms64(x, w(p + "norm1"))
            y = mixer64(model, layer, h + seq.conv(h, w(p + "canon1")), w, p + "mix.", seq, carried, i)
            x = x + y + moe64(model, h + seq.conv(h, w(p + "canon2")), w, p + "mlp.", mlp)
        else:
            for n in (1, 2):
                hc = f"{p}hc{n}."
                h = layer_norm64(torch.einsum("s,stw->tw", w(hc + "in"), x), w(f"{p}norm{n}"), w(f"{p}norm{n}.b"))
                if n == 1:
                    y = mixer64(model, layer, h, w, p + "mix.", seq, carried, i)
                elif mlp["kind"] == "dense":
                    y = (silu64(h @ w(p + "mlp.gate").T) * (h @ w(p + "mlp.up").T)) @ w(p + "mlp.down").T
                else:
                    y = moe64(model, h, w, p + "mlp.", mlp)
                x = torch.einsum("st,snw->tnw", w(hc + "mix"), x) + w(hc + "out")[:, None, None] * y
    if model == "zinurax":
        return (layer_norm64(x[last], w("final.norm")) @ w("embed").T)[None]
    if model == "lukarax":
        return (layer_norm64(x.sum(0)[last], w("final.norm"), w("final.norm.b")) @ w("embed").T)[None]
    return (rms64(x[last], w("final.norm") + (1.0 if model == "fabivik" else 0.0)) @ w("head").T)[None]


def exact(case, seed):
    with torch.inference_mode():
        return (exact_gpt if case["model"] == "gpt" else exact_hybrid)(case, seed)
