"""Work that programs on this framework have it do, as cases for measuring: decode steps, prompts, drafted tokens and embeddings of
random models through the engines' public calls (``decode``, ``prefill``, ``verify``, ``hidden``).

The models are the benchmark's and the tests' own architectures.  Deep ones are cut to a part of their layers, so that a model is made
in about a second; every layer of a model has the same sizes, so a layer costs what it costs in the whole model.  Weights are random
blocks of the encodings that a checkpoint of that kind holds, drawn here and decoded here once more in 64 bits for :func:`exact`.
"""
from __future__ import annotations

import math
import zlib

import torch

# n_layers is the full depth; cases name the depth they run
MODELS = {
    "tiny-qwen3": dict(arch="qwen3", n_layers=2, d_model=256, n_heads=4, n_kv_heads=2, head_dim=64, d_ff=768, vocab_size=4096, rope_base=1e6, norm_eps=1e-6),
    "dense-1b": dict(arch="llama", n_layers=20, d_model=2048, n_heads=16, n_kv_heads=4, head_dim=128, d_ff=5504, vocab_size=32768, rope_base=500000.0, norm_eps=1e-5),
    "llama-3.1-8b": dict(arch="llama", n_layers=32, d_model=4096, n_heads=32, n_kv_heads=8, head_dim=128, d_ff=14336, vocab_size=128256, rope_base=500000.0,
                         norm_eps=1e-5),
    "gpt-oss-120b": dict(arch="gpt-oss", n_layers=36, d_model=2880, n_heads=64, n_kv_heads=8, head_dim=64, d_ff=2880, vocab_size=201088, rope_base=150000.0,
                         norm_eps=1e-5, n_experts=128, n_experts_used=4, d_ff_expert=2880, sliding_window=128),
    "kavenex-1b": dict(arch="kavenex", n_layers=16, d_model=2048, n_heads=16, d_nope=128, d_rot=64, d_value=128, rank=512, d_ff=5504, vocab_size=32768, side=256,
                       rope_base=500000.0, norm_eps=1e-5, loop=(0, 4, 2), mult=0.5),
}
BITS = {"f32": 32.0, "bf16": 16.0, "q8_0": 8.5, "q6_k": 6.5625, "q4_k": 4.5, "mxfp4": 4.25}
CHUNK = 2048                     # rows of a prompt that a server hands to one prefill call


def listed() -> list[dict]:
    return [
        # a small test model answering one user: what launches and host calls cost
        dict(name="tiny step", kind="step", model="tiny-qwen3", quant="q4_k_m", layers=2, nb=1, ctx=201, kv="f16", n_ctx=512),
        # the headline: one user's chat, the model reads its weights for every token
        dict(name="chat step", kind="step", model="llama-3.1-8b", quant="q4_k_m", layers=12, nb=1, ctx=640, kv="f16", n_ctx=8192),
        # a server with eight slots of uneven long conversations and the 8-bit cache that long contexts are run with
        dict(name="8 slots, long, q8 cache", kind="step", model="llama-3.1-8b", quant="q4_k_m", layers=12, nb=8, ctx=3001, kv="q8_0", n_ctx=8192),
        # a full server: 32 slots
        dict(name="32 slots", kind="step", model="llama-3.1-8b", quant="q4_k_m", layers=12, nb=32, ctx=467, kv="f16", n_ctx=2048),
        # the headline's prompt: 512 tokens, time to first token
        dict(name="prompt 512", kind="prompt", model="llama-3.1-8b", quant="q4_k_m", layers=12, nb=512, ctx=0, kv="f16", n_ctx=8192),
        # a document: one full chunk in the middle of a long prompt
        dict(name="chunk 2048 at 6144", kind="prompt", model="llama-3.1-8b", quant="q4_k_m", layers=12, nb=2048, ctx=6144, kv="f16", n_ctx=8192),
        # speculative decoding: the target scores seven tokens, six of them drafted
        dict(name="7 drafted tokens", kind="drafted", model="llama-3.1-8b", quant="q4_k_m", layers=12, nb=7, ctx=901, kv="f16", n_ctx=4096),
        # embedding of a paragraph by a small 16-bit model
        dict(name="embed 331", kind="embed", model="dense-1b", quant="bf16", layers=20, nb=331, ctx=0, kv="f16", n_ctx=2048),
        # 4-bit experts: sixteen sequences, the benchmark's step of that model
        dict(name="experts, 16 slots", kind="step", model="gpt-oss-120b", quant="mxfp4", layers=10, nb=16, ctx=1024, kv="f16", n_ctx=8192),
        # the same model's prompt
        dict(name="experts, prompt 1024", kind="prompt", model="gpt-oss-120b", quant="mxfp4", layers=10, nb=1024, ctx=0, kv="f16", n_ctx=8192),
        # a stack model in 16 bits: latent attention, looped layers, paged cache
        dict(name="stack, 4 slots", kind="step", model="kavenex-1b", quant="bf16", layers=16, nb=4, ctx=1024, kv="f16", n_ctx=2112),
        dict(name="stack, prompt 1777", kind="prompt", model="kavenex-1b", quant="bf16", layers=16, nb=1777, ctx=0, kv="f16", n_ctx=2112),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    model, quant, layers = rng.choices([("tiny-qwen3", "q4_k_m", 2), ("tiny-qwen3", "q8_0", 2), ("dense-1b", "bf16", 20), ("dense-1b", "q8_0", 20),
                                        ("llama-3.1-8b", "q4_k_m", 12), ("gpt-oss-120b", "mxfp4", 10), ("kavenex-1b", "bf16", 16)],
                                       weights=[1, 1, 1, 1, 6, 3, 2])[0]
    small = model in ("tiny-qwen3", "kavenex-1b")
    kind = rng.choices(["step", "prompt", "drafted", "embed"], weights=[5, 4, 1, 1])[0]
    kv = "q8_0" if model in ("llama-3.1-8b", "dense-1b") and rng.random() < 0.3 else "f16"
    n_ctx = 2112 if small else 8192
    if kind == "step":
        nb = _log(rng, 1, 32)
        ctx = _log(rng, 17, (1100 if small else 4000) if nb <= 8 else 700)
    elif kind == "drafted":
        nb, ctx = rng.randint(2, 17), _log(rng, 17, n_ctx - 64)
    elif kind == "embed":
        nb, ctx = _log(rng, 5, 1024), 0
    else:
        nb = _log(rng, 9, 1024 if model == "gpt-oss-120b" else 2048)
        ctx = 0 if rng.random() < 0.5 else rng.randint(0, min(n_ctx - nb, 6144))
    return dict(kind=kind, model=model, quant=quant, layers=layers, nb=nb, ctx=ctx, kv=kv, n_ctx=n_ctx)


# ---- what a checkpoint holds ------------------------------------------------------------------------------------------------------
def _more_bits(i: int, n: int) -> bool:
    return i < n // 8 or i >= 7 * n // 8 or (i - n // 8) % 3 == 2


def _table(case: dict) -> dict[str, tuple[tuple[int, ...], str]]:
    """name -> (shape, encoding)."""
    m, q, n = MODELS[case["model"]], case["quant"], case["layers"]
    d, v = m["d_model"], m["vocab_size"]
    if m["arch"] == "kavenex":
        H, side = m["n_heads"], m["side"]
        t = {"embed": ((v, d), "bf16"), "head": ((v, d), "bf16"), "final.norm": ((d,), "f32"), "final.norm.b": ((d,), "f32"), "loop.step": ((m["loop"][2], d), "bf16"),
             "side.embed": ((v, n * side), "bf16")}
        for i in range(n):
            p = f"l{i}."
            t.update({p + x: ((d,), "f32") for x in ("norm1", "norm1.b", "norm2", "norm2.b", "side.norm")})
            t.update({p + "mix.dkv.norm": ((m["rank"],), "f32"), p + "mix.q": ((H * (m["d_nope"] + m["d_rot"]), d), "bf16"),
                      p + "mix.dkv": ((m["rank"] + m["d_rot"], d), "bf16"), p + "mix.uk": ((H * m["d_nope"], m["rank"]), "bf16"),
                      p + "mix.uv": ((H * m["d_value"], m["rank"]), "bf16"), p + "mix.o": ((d, H * m["d_value"]), "bf16"),
                      p + "mlp.gate": ((m["d_ff"], d), "bf16"), p + "mlp.up": ((m["d_ff"], d), "bf16"), p + "mlp.down": ((d, m["d_ff"]), "bf16"),
                      p + "side.gate": ((side, d), "bf16"), p + "side.proj": ((d, side), "bf16")})
        return t
    dense = {"q4_k_m": "q4_k", "mxfp4": "bf16"}.get(q, q)
    qd, kd = m["n_heads"] * m["head_dim"], m["n_kv_heads"] * m["head_dim"]
    t = {"token_embd.weight": ((v, d), dense), "output_norm.weight": ((d,), "f32"), "output.weight": ((v, d), "q6_k" if q == "q4_k_m" else dense)}
    for i in range(n):
        p, wide = f"blk.{i}.", "q6_k" if q == "q4_k_m" and _more_bits(i, n) else dense
        t.update({p + "attn_norm.weight": ((d,), "f32"), p + "attn_q.weight": ((qd, d), dense), p + "attn_k.weight": ((kd, d), dense),
                  p + "attn_v.weight": ((kd, d), wide), p + "attn_output.weight": ((d, qd), dense)})
        if m["arch"] == "qwen3":
            t.update({p + "attn_q_norm.weight": ((m["head_dim"],), "f32"), p + "attn_k_norm.weight": ((m["head_dim"],), "f32")})
        if m["arch"] == "gpt-oss":
            E, f = m["n_experts"], m["d_ff_expert"]
            t.update({p + "attn_q.bias": ((qd,), "f32"), p + "attn_k.bias": ((kd,), "f32"), p + "attn_v.bias": ((kd,), "f32"), p + "attn_output.bias": ((d,), "f32"),
                      p + "attn_sinks.weight": ((m["n_heads"],), "f32"), p + "post_attention_norm.weight": ((d,), "f32"), p + "ffn_gate_inp.weight": ((E, d), "f32"),
                      p + "ffn_gate_inp.bias": ((E,), "f32"), p + "ffn_gate_exps.weight": ((E, f, d), "mxfp4"), p + "ffn_up_exps.weight": ((E, f, d), "mxfp4"),
                      p + "ffn_down_exps.weight": ((E, d, f), "mxfp4"), p + "ffn_gate_exps.bias": ((E, f), "f32"), p + "ffn_up_exps.bias": ((E, f), "f32"),
                      p + "ffn_down_exps.bias": ((E, d), "f32")})
        else:
            t.update({p + "ffn_norm.weight": ((d,), "f32"), p + "ffn_gate.weight": ((m["d_ff"], d), dense), p + "ffn_up.weight": ((m["d_ff"], d), dense),
                      p + "ffn_down.weight": ((d, m["d_ff"]), wide)})
    return t


def _half(x: torch.Tensor) -> torch.Tensor:
    return x.to(torch.float16).view(-1, 1).view(torch.uint8)


def _encoded(name: str, shape: tuple[int, ...], enc: str, seed: int, dev) -> torch.Tensor:
    """Random blocks of an encoding as a checkpoint's bytes.  The values have a standard deviation of about 0.02, token embeddings of 1 and the
    matrices whose results are added to the stream of 0.02 / sqrt(2 x 32 layers): a layer then changes the stream by a part, as in trained models
    (otherwise rounding grows from layer to layer until two correct programs differ by a tenth)."""
    log2 = -3 if name.endswith(("attn_output.weight", "ffn_down.weight", "ffn_down_exps.weight")) else 0
    gain = 50.0 if name == "token_embd.weight" else 2.0 ** log2
    g = torch.Generator(device=dev).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)
    n = math.prod(shape)

    def byte(*s):
        return torch.randint(0, 256, s, device=dev, dtype=torch.uint8, generator=g)

    def code(*s):                # 0..15 about 7.5, as quantised normal values are spread
        r = byte(*s)
        return (r & 7) + ((r >> 3) & 7) + (r >> 7)

    if enc in ("f32", "bf16"):
        x = torch.randn(n, device=dev, generator=g) * (0.02 * gain)
        if enc == "bf16":
            return x.to(torch.bfloat16).view(torch.uint8)
        if "norm" in name and not name.endswith(".b"):
            x = x + 1.0
        return x.view(torch.uint8)
    if enc == "q8_0":
        q = (torch.randn(n // 32, 32, device=dev, generator=g) * 50).round().clamp(-127, 127).to(torch.int8)
        return torch.cat([_half(4e-4 * gain * (0.9 + 0.2 * torch.rand(n // 32, device=dev, generator=g))), q.view(torch.uint8)], 1).view(-1)
    if enc == "q4_k":
        b = n // 256
        d = (1.1e-4 * gain * (0.9 + 0.2 * torch.rand(b, device=dev, generator=g))).to(torch.float16)
        sc = 44 + byte(b, 8) % 20
        lo, hi = sc[:, :4], sc[:, 4:]
        packed = torch.cat([lo | (hi >> 4 << 6), lo | (hi >> 4 << 6), (hi & 15) | (hi << 4)], 1)       # minima: the scales' numbers times 7.5 d
        return torch.cat([_half(d), _half(7.5 * d.float()), packed, code(b, 128) | (code(b, 128) << 4)], 1).view(-1)
    if enc == "q6_k":
        b = n // 256
        sc = (70 + byte(b, 16) % 58).to(torch.int8) * (1 - 2 * (byte(b, 16) & 1).to(torch.int8))
        return torch.cat([byte(b, 192), sc.view(torch.uint8), _half(1.08e-5 * gain * (0.9 + 0.2 * torch.rand(b, device=dev, generator=g)))], 1).view(-1)
    b = n // 32                   # mxfp4
    return torch.cat([119 + log2 + (byte(b, 1) & 1), byte(b, 16)], 1).view(-1)


def _decoded(raw: torch.Tensor, shape: tuple[int, ...], enc: str) -> torch.Tensor:
    """The values of :func:`_encoded`'s bytes, in 64 bits."""
    f8 = torch.float64
    if enc in ("f32", "bf16"):
        return raw.view(torch.float32 if enc == "f32" else torch.bfloat16).to(f8).view(shape)
    if enc == "q8_0":
        r = raw.view(-1, 34)
        x = r[:, :2].contiguous().view(torch.float16).to(f8) * r[:, 2:].contiguous().view(torch.int8).to(f8)
    elif enc == "q4_k":
        r = raw.view(-1, 144)
        d = r[:, :4].contiguous().view(torch.float16).to(f8)
        s = r[:, 4:16]
        sc = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6 << 4)], 1).to(f8)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | (s[:, 4:8] >> 6 << 4)], 1).to(f8)
        q = r[:, 16:].view(-1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32).to(f8)
        x = (d[:, :1] * sc)[..., None] * q - (d[:, 1:] * mn)[..., None]
    elif enc == "q6_k":
        r = raw.view(-1, 210)
        lo, hi = r[:, :128].view(-1, 2, 2, 32), r[:, 128:192].view(-1, 2, 1, 32)
        q = torch.cat([lo & 15, lo >> 4], 2) | ((torch.cat([hi, hi >> 2, hi >> 4, hi >> 6], 2) & 3) << 4)
        sc = r[:, 192:208].contiguous().view(torch.int8).to(f8) * r[:, 208:].contiguous().view(torch.float16).to(f8)
        x = (q.to(f8) - 32).view(-1, 16, 16) * sc[..., None]
    else:
        r = raw.view(-1, 17)
        val = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], dtype=f8, device=raw.device)
        q = torch.cat([r[:, 1:] & 15, r[:, 1:] >> 4], 1).int()
        x = torch.where(q > 7, -1.0, 1.0).to(f8) * val[q & 7] * torch.exp2(r[:, :1].to(f8) - 127)
    return x.reshape(shape)


class _Tensors:
    """A checkpoint's tensors by name, each drawn when it is asked for."""

    def __init__(self, case: dict, seed: int, dev, rename=None):
        self.table, self.seed, self.dev = _table(case), seed, dev
        self.names = {(rename(n) if rename else n): n for n in self.table}

    def __contains__(self, name: str) -> bool:
        return name in self.names

    def keys(self):
        return self.names.keys()

    def __getitem__(self, name: str):
        from ollama_b200.gguf.types import GGMLType
        from ollama_b200.models.weights import QWeight
        own = self.names[name]
        shape, enc = self.table[own]
        return QWeight(name, GGMLType[enc.upper()], shape, _encoded(own, shape, enc, self.seed, self.dev))


def _contexts(case: dict) -> list[int]:
    """Tokens that each sequence holds before the step: spread about ``ctx``."""
    nb, ctx = case["nb"], case["ctx"]
    if case["kind"] != "step":
        return [ctx]
    return [ctx] if nb == 1 else [max(1, ctx // 4 + (ctx * 3 // 2) * j // (nb - 1)) for j in range(nb)]


def _tokens(case: dict, seed: int) -> tuple[list[list[int]], list[list[int]]]:
    """(what each sequence holds, the tokens of the pass for each sequence)."""
    g = torch.Generator().manual_seed(seed)
    v, per = MODELS[case["model"]]["vocab_size"], 1 if case["kind"] == "step" else case["nb"]

    def some(n):
        return torch.randint(3, v, (n,), generator=g).tolist()

    held = _contexts(case)
    return [some(n) for n in held], [some(per) for _ in held]


def _stack_config(case: dict) -> dict:
    m, n = MODELS[case["model"]], case["layers"]
    mix = {"heads": m["n_heads"], "dim": m["d_nope"], "rot_dim": m["d_rot"], "vdim": m["d_value"], "kv_rank": m["rank"], "scale": (m["d_nope"] + m["d_rot"]) ** -0.5,
           "rot": {"base": m["rope_base"], "dims": m["d_rot"]}}
    lo, hi, times = m["loop"]
    return {"architecture": "Kavenex", "embedding": {"scale": math.sqrt(m["d_model"])}, "width": m["d_model"], "vocab": m["vocab_size"], "norm": {"eps": m["norm_eps"]},
            "residual_mult": m["mult"], "token_side": {"dim": m["side"]}, "loop": {"start": lo, "stop": hi, "times": times},
            "layers": [{"type": "latent_attention", "mixer": mix, "mlp": {"kind": "dense", "ff": m["d_ff"]}} for _ in range(n)]}


def _engine(case: dict, seed: int, dev: str):
    m = MODELS[case["model"]]
    if m["arch"] == "kavenex":
        from ollama_b200.convert.stack import map_stack_name
        from ollama_b200.engine.stack import StackBackend
        from ollama_b200.models.synth import stack_model_config
        cfg = _stack_config(case)
        return StackBackend(None, device=dev, cfg=stack_model_config(cfg), tensors=_Tensors(case, seed, dev, lambda n: map_stack_name(n, cfg)))
    from ollama_b200.engine.b200 import B200Backend
    from ollama_b200.models.config import ModelConfig
    kw = {**m, "n_layers": case["layers"], "v_head_dim": m["head_dim"], "rope_dim": m["head_dim"], "ctx_train": 131072, "name": case["model"]}
    if m["arch"] == "qwen3":
        kw.update(rope_style="neox", qk_norm=True)
    if m["arch"] == "gpt-oss":
        kw.update(rope_style="neox", act="swiglu_oai", attn_bias=True, attn_out_bias=True, attn_sinks=True, moe_router="topk_softmax", moe_bias=True,
                  rope_scaling_type="yarn", rope_scaling_factor=32.0, rope_orig_ctx=4096, swa_layers=[i % 2 == 0 for i in range(case["layers"])])
    return B200Backend(None, device=dev, cfg=ModelConfig(**kw), tensors=_Tensors(case, seed, dev), kv_type=case["kv"])


def prepare(case: dict, seed: int) -> dict:
    """A loaded model whose slots hold their conversations, and the tokens of the pass."""
    held, new = _tokens(case, seed)
    be = _engine(case, seed, "cuda:0")
    be.alloc(len(held), case["n_ctx"])
    for slot, toks in enumerate(held):
        for c in range(0, len(toks), CHUNK):
            be.prefill(slot, toks[c:c + CHUNK], c, need_logits=False)
    return {"engine": be, "kind": case["kind"], "slots": list(range(len(held))), "at": [len(h) for h in held], "new": new}


def run(state: dict):
    be, kind, new = state["engine"], state["kind"], state["new"]
    if kind == "step":
        return be.decode(state["slots"], [t[0] for t in new], state["at"])
    if kind == "drafted":
        return be.verify(0, new[0], state["at"][0])
    if kind == "embed":
        return be.hidden(0, new[0])
    return be.prefill(0, new[0], state["at"][0])


def work(case: dict) -> dict:
    m, n = MODELS[case["model"]], case["layers"]
    rows = case["nb"]
    used = 1.0
    if "n_experts" in m:         # share of the experts that so many rows choose
        used = 1.0 - (1.0 - m["n_experts_used"] / m["n_experts"]) ** rows
    logits = {"step": rows, "drafted": rows, "prompt": 1, "embed": 0}[case["kind"]]
    byts = flops = 0.0
    for name, (shape, enc) in _table(case).items():
        size, one = math.prod(shape), math.prod(shape) * BITS[enc] / 8
        if name in ("token_embd.weight", "embed", "side.embed"):
            byts += rows * one / m["vocab_size"]
        elif name in ("output.weight", "head"):
            byts += one if logits else 0
            flops += 2.0 * size * logits
        else:
            runs = 2 if "loop" in m and name.startswith("l") and m["loop"][0] <= int(name[1:].split(".")[0] if name[1].isdigit() else 99) < m["loop"][1] else 1
            expert = "_exps" in name
            byts += one * (used if expert else 1.0)
            if len(shape) > 1:
                flops += 2.0 * size * rows * runs * (m["n_experts_used"] / m["n_experts"] if expert else 1.0)
    runs = n + (m["loop"][1] - m["loop"][0] if "loop" in m else 0)
    per = 2.0 * (m["rank"] + m["d_rot"]) if "rank" in m else 2.0 * m["n_kv_heads"] * m["head_dim"] * (2.0 if case["kv"] == "f16" else 1.0625)
    dots = m["n_heads"] * (m["d_nope"] + m["d_rot"] + m["d_value"] if "rank" in m else 2 * m["head_dim"])
    for ctx in _contexts(case):
        new = 1 if case["kind"] == "step" else rows
        for i in range(runs):
            seen = min(ctx, m["sliding_window"]) if "sliding_window" in m and i % 2 == 0 else ctx
            byts += per * (seen + new)
            pairs = sum(min(ctx + j + 1, m["sliding_window"]) for j in range(new)) if "sliding_window" in m and i % 2 == 0 else new * ctx + new * (new + 1) / 2
            flops += 2.0 * dots * pairs
    byts += 4.0 * (logits * m["vocab_size"] if logits else rows * m["d_model"])
    return {"bytes": byts, "flops": flops}


def tolerance(case: dict) -> dict:
    """About four times the error against 64 bits that was measured, at most 0.03: steps on K-quants multiply 8-bit activations (0.018), other products 16-bit ones (0.005 on
    rounded K-quants, 0.003 on 16-bit and 4-bit weights); few rows of a stack model stay in 32 bits (7e-5)."""
    if case["model"] == "kavenex-1b":
        rel = 3e-4 if case["kind"] == "step" and case["nb"] <= 4 else 0.012
    elif case["kind"] == "step" and case["quant"] in ("q4_k_m", "q8_0"):
        rel = 0.03
    else:
        rel = 0.02
    return {"rel": rel, "max": 10 * rel}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rows(x, fn, step: int = 4096):
    return torch.cat([fn(x[i:i + step]) for i in range(0, len(x), step)])


def _causal(q, k, v, scale, window=0, sinks=None, step: int = 512):
    """q [T, H, D], k [S, Hkv, D], v [S, Hkv, Dv]: the queries are the last T of the S positions."""
    T, H, _ = q.shape
    S, Hkv, dv = v.shape
    out = torch.empty(T, H, dv, dtype=q.dtype, device=q.device)
    for a in range(0, T, step):
        b = min(T, a + step)
        lo = max(0, S - T + a - window + 1) if window else 0
        hi = S - T + b
        at, kp = torch.arange(S - T + a, hi, device=q.device)[:, None], torch.arange(lo, hi, device=q.device)[None]
        hide = kp > at
        if window:
            hide = hide | (at - kp >= window)
        for h in range(Hkv):
            hs = slice(h * (H // Hkv), (h + 1) * (H // Hkv))
            s = torch.einsum("thd,sd->hts", q[a:b, hs], k[lo:hi, h]) * scale
            s = s.masked_fill(hide, -math.inf)
            if sinks is not None:
                s = torch.cat([s, sinks[hs].view(-1, 1, 1).expand(-1, b - a, 1)], -1)
            out[a:b, hs] = torch.einsum("hts,sd->thd", torch.softmax(s, -1)[..., :hi - lo], v[lo:hi, h])
    return out.reshape(T, -1)


def _turn(x, pos, inv, pairs: bool, mag: float = 1.0):
    a = pos.to(torch.float64)[:, None] * inv[None]
    c, s = (torch.cos(a) * mag)[:, None], (torch.sin(a) * mag)[:, None]
    if pairs:
        u, w = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - w * s, u * s + w * c], -1).flatten(-2)
    u, w = x.chunk(2, -1)
    return torch.cat([u * c - w * s, u * s + w * c], -1)


def _decoder(case, W, m, seqs):
    """Hidden rows (normalised) of all sequences one after the other."""
    dev, D, eps = "cuda:0", m["head_dim"], m["norm_eps"]
    i = torch.arange(D // 2, device=dev, dtype=torch.float64)
    inv, mag = m["rope_base"] ** (-2.0 * i / D), 1.0
    if m["arch"] == "gpt-oss":   # YaRN, 32 times 4096 positions
        def dim(turns):
            return D * math.log(4096 / (turns * 2 * math.pi)) / (2 * math.log(m["rope_base"]))
        lo, hi = max(0.0, math.floor(dim(32.0))), min(D - 1.0, math.ceil(dim(1.0)))
        keep = 1.0 - ((i - lo) / max(0.001, hi - lo)).clamp(0, 1)
        inv, mag = inv / 32.0 * (1 - keep) + inv * keep, 1.0 + 0.1 * math.log(32.0)
    pos = torch.cat([torch.arange(len(s), device=dev) for s in seqs])
    x = W("token_embd.weight")[torch.tensor([t for s in seqs for t in s], device=dev)]
    for n in range(case["layers"]):
        p = f"blk.{n}."
        h = _rms(x, W(p + "attn_norm.weight"), eps)
        q, k, v = (h @ W(p + f"attn_{c}.weight").t() + (W(p + f"attn_{c}.bias") if m["arch"] == "gpt-oss" else 0) for c in "qkv")
        q, k, v = q.view(-1, m["n_heads"], D), k.view(-1, m["n_kv_heads"], D), v.view(-1, m["n_kv_heads"], D)
        if m["arch"] == "qwen3":
            q, k = _rms(q, W(p + "attn_q_norm.weight"), eps), _rms(k, W(p + "attn_k_norm.weight"), eps)
        q, k = (_turn(z, pos, inv, m["arch"] == "llama", mag) for z in (q, k))
        o, at = [], 0
        for s in seqs:
            r = slice(at, at + len(s))
            o.append(_causal(q[r], k[r], v[r], D ** -0.5, m["sliding_window"] if m["arch"] == "gpt-oss" and n % 2 == 0 else 0,
                             W(p + "attn_sinks.weight") if m["arch"] == "gpt-oss" else None))
            at += len(s)
        x = x + torch.cat(o) @ W(p + "attn_output.weight").t()
        if m["arch"] != "gpt-oss":
            h, g, u, dn = _rms(x, W(p + "ffn_norm.weight"), eps), W(p + "ffn_gate.weight"), W(p + "ffn_up.weight"), W(p + "ffn_down.weight")
            x = x + _rows(h, lambda r: (torch.nn.functional.silu(r @ g.t()) * (r @ u.t())) @ dn.t())
            continue
        x = x + W(p + "attn_output.bias")
        h = _rms(x, W(p + "post_attention_norm.weight"), eps)
        val, ids = torch.topk(h @ W(p + "ffn_gate_inp.weight").t() + W(p + "ffn_gate_inp.bias"), m["n_experts_used"], -1)
        wt = torch.softmax(val, -1)
        gw, uw, dw = (W.some(p + f"ffn_{c}_exps.weight") for c in ("gate", "up", "down"))
        gb, ub, db = (W(p + f"ffn_{c}_exps.bias") for c in ("gate", "up", "down"))
        y = torch.zeros_like(x)
        for e in ids.unique().tolist():
            rows, place = (ids == e).nonzero(as_tuple=True)
            g = (h[rows] @ gw(e).t() + gb[e]).clamp(max=7.0)
            u = (h[rows] @ uw(e).t() + ub[e]).clamp(-7.0, 7.0)
            y[rows] += wt[rows, place][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ dw(e).t() + db[e])
        x = x + y
    return _rms(x, W("output_norm.weight"), eps)


def _latent(case, W, m, seqs):
    dev, eps, mult, H, dn, dr = "cuda:0", m["norm_eps"], m["mult"], m["n_heads"], m["d_nope"], m["d_rot"]

    def norm(name, x):
        c = x - x.mean(-1, keepdim=True)
        return c * torch.rsqrt((c * c).mean(-1, keepdim=True) + eps) * W(name) + W(name + ".b")

    def gelu(x):
        return torch.nn.functional.gelu(x, approximate="tanh")

    inv = m["rope_base"] ** (-2.0 * torch.arange(dr // 2, device=dev, dtype=torch.float64) / dr)
    pos = torch.cat([torch.arange(len(s), device=dev) for s in seqs])
    toks = torch.tensor([t for s in seqs for t in s], device=dev)
    first = x = W("embed")[toks] * math.sqrt(m["d_model"])
    side = W("side.embed")[toks].view(len(toks), case["layers"], -1)
    lo, hi, times = m["loop"]
    for turn, n in [(0, i) for i in range(lo)] + [(t, i) for t in range(times) for i in range(lo, hi)] + [(0, i) for i in range(hi, case["layers"])]:
        p = f"l{n}."
        if n == lo:
            x = (x if turn == 0 else x + first) + W("loop.step")[turn]
        h = norm(p + "norm1", x)
        q = (h @ W(p + "mix.q").t()).view(-1, H, dn + dr)
        q = torch.cat([q[..., :dn], _turn(q[..., dn:], pos, inv, True)], -1)
        down = h @ W(p + "mix.dkv").t()
        c = _rms(down[:, :m["rank"]], W(p + "mix.dkv.norm"), eps)
        kr = _turn(down[:, None, m["rank"]:], pos, inv, True)
        k = torch.cat([(c @ W(p + "mix.uk").t()).view(-1, H, dn), kr.expand(-1, H, dr)], -1)
        v = (c @ W(p + "mix.uv").t()).view(-1, H, m["d_value"])
        o, at = [], 0
        for s in seqs:
            r = slice(at, at + len(s))
            o.append(_causal(q[r], k[r], v[r], (dn + dr) ** -0.5))
            at += len(s)
        x = x + mult * (torch.cat(o) @ W(p + "mix.o").t())
        h = norm(p + "norm2", x)
        x = x + mult * ((gelu(h @ W(p + "mlp.gate").t()) * (h @ W(p + "mlp.up").t())) @ W(p + "mlp.down").t())
        x = x + mult * _rms((gelu(x @ W(p + "side.gate").t()) * side[:, n]) @ W(p + "side.proj").t(), W(p + "side.norm"), eps)
    return norm("final.norm", x)


class _Weights64:
    def __init__(self, case: dict, seed: int):
        self.table, self.seed = _table(case), seed

    def __call__(self, name: str) -> torch.Tensor:
        shape, enc = self.table[name]
        return _decoded(_encoded(name, shape, enc, self.seed, "cuda:0"), shape, enc)

    def some(self, name: str):
        """Of stacked matrices: one matrix by its number."""
        shape, enc = self.table[name]
        raw = _encoded(name, shape, enc, self.seed, "cuda:0").view(shape[0], -1)
        return lambda e: _decoded(raw[e], shape[1:], enc)


@torch.no_grad()
def exact(case: dict, seed: int):
    m, W = MODELS[case["model"]], _Weights64(case, seed)
    held, new = _tokens(case, seed)
    seqs = [h + t for h, t in zip(held, new)]
    x = (_latent if m["arch"] == "kavenex" else _decoder)(case, W, m, seqs)
    if case["kind"] == "embed":
        return x
    head = W("head" if m["arch"] == "kavenex" else "output.weight")
    if case["kind"] == "step":
        ends = torch.tensor([len(s) for s in seqs], device=x.device).cumsum(0) - 1
        return x[ends] @ head.t()
    return x[-case["nb"]:] @ head.t() if case["kind"] == "drafted" else x[-1] @ head.t()
