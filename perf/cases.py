"""The work that is measured: what programs built on this package have it do, through its public entry points.

Kinds of case
  gemv      `gemv` on raw device pointers: y = W x, weights [N,K] (the layout of Linear) or [K,N], f32 or bf16
  sample    `sample_top_p` on logits that are on the device, once per sequence of a batch
  generate  a model's answer to prompts: caches are reset, the prompts go in at once (logits of the last position), then
            `steps` given tokens follow one by one (teacher-forced, so that outputs can be compared).  One sequence: host
            ids in, host logits out, as the chat loop and the trace replay do; several: decode steps with ids and logits on
            the device, as a serving loop does.  steps == 0 is prefill alone.

Models are named as in the benchmark: the LlamaModel shapes of `lumen_b200.synth` (with all or some of their layers) and
the layer lists of Fegetar (routed experts or dense) and Fekorax.  Weights are random, N(0, 0.02), seeded by their names; a program keeps
its model between requests, so the last one is kept loaded here and every state has caches, tokens and logits of its own.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

import lumen_b200 as L
from lumen_b200 import synth

DEV = "cuda:0"
MAX_SEQ = 2048
STD = 0.02

LLAMAS = {"tinyllama": synth.TINYLLAMA, "llama2_7b": synth.LLAMA2_7B, "qwen3_8b": synth.QWEN3_8B}


def listed() -> list:
    return [
        # the key projection of a TinyLlama layer on its own: the smallest product there is, all launch and latency
        dict(name="gemv_small", kind="gemv", k=2048, n=256, dtype="f32", layout="nk"),
        # weights kept as [K,N] (the layout a framework that multiplies x W holds them in), the largest of the benchmark's sweep
        dict(name="gemv_kn_bf16", kind="gemv", k=4096, n=11008, dtype="bf16", layout="kn"),
        # a chat server draws the next token of each of its sequences
        dict(name="sample_32k", kind="sample", vocab=32000, rows=8, temperature=0.8, top_p=0.9),
        # the configuration that the headline is quoted on: f32 weights, short prompt, one user
        dict(name="chat_tiny_f32", kind="generate", model="tinyllama", layers=22, dtype="f32", batch=1, prompt=32, steps=48),
        # one user, a conversation that already has a thousand tokens, bf16 checkpoint
        dict(name="chat_tiny_bf16_long", kind="generate", model="tinyllama", layers=22, dtype="bf16", batch=1, prompt=1023, steps=48),
        # one user of a 7B model, prompt of 512
        dict(name="chat_7b_bf16", kind="generate", model="llama2_7b", layers=32, dtype="bf16", batch=1, prompt=512, steps=32),
        # sixteen users of the f32 model
        dict(name="batch16_tiny_f32", kind="generate", model="tinyllama", layers=22, dtype="f32", batch=16, prompt=64, steps=40),
        # a full serving batch: grouped queries of 128, q/k norm, the large vocabulary; a quarter of the model's depth
        dict(name="batch64_qwen_bf16", kind="generate", model="qwen3_8b", layers=9, dtype="bf16", batch=64, prompt=60, steps=32),
        # reading one document of odd length, f32
        dict(name="prefill_tiny_f32", kind="generate", model="tinyllama", layers=22, dtype="f32", batch=1, prompt=1777, steps=0),
        # reading four long documents at once, bf16: the largest single call
        dict(name="prefill_qwen_bf16", kind="generate", model="qwen3_8b", layers=9, dtype="bf16", batch=4, prompt=2048, steps=0),
        # the models given as a list of layers: latent attention; matrix memory and chunked attention
        dict(name="chat_fegetar", kind="generate", model="fegetar_dense", layers=8, dtype="bf16", batch=1, prompt=96, steps=40),
        dict(name="chat_fekorax", kind="generate", model="fekorax", layers=6, dtype="bf16", batch=1, prompt=700, steps=40),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choices(["gemv", "sample", "chat", "batch", "prefill", "list"], [4, 1, 5, 5, 4, 3])[0]
    if kind == "gemv":
        k, n = _log(rng, 256, 12288), _log(rng, 128, 33000)
        if rng.random() < 0.7:  # most layers have round sizes
            k, n = -(-k // 64) * 64, -(-n // 64) * 64
        return dict(kind="gemv", k=k, n=n, dtype=rng.choice(["f32", "bf16"]), layout=rng.choice(["nk", "kn"]))
    if kind == "sample":
        return dict(kind="sample", vocab=rng.choice([4096, 32000, 32000, 50257, 151936]), rows=_log(rng, 1, 16),
                    temperature=rng.choice([0.6, 0.8, 1.0]), top_p=rng.choice([0.9, 0.95]))
    if kind == "list":
        model = rng.choice(["fegetar_moe", "fegetar_dense", "fekorax"])
        layers = {"fegetar_moe": rng.randint(1, 2), "fegetar_dense": rng.randint(1, 8), "fekorax": 6}[model]
        # (routed experts in 32 bits: in 16 bits rounding decides between near-equal experts, and no two orders of summation agree)
        return dict(kind="generate", model=model, layers=layers, dtype="f32" if model == "fegetar_moe" else "bf16", batch=1, prompt=_log(rng, 16, 1900),
                    steps=rng.randint(0, 40))
    model = rng.choice(list(LLAMAS))
    layers = rng.randint(2, {"tinyllama": 22, "llama2_7b": 8, "qwen3_8b": 9}[model])
    dtype = "bf16" if model != "tinyllama" else rng.choice(["f32", "bf16"])
    if kind == "chat":
        batch, prompt, steps = 1, _log(rng, 8, 1900), rng.randint(8, 48)
    elif kind == "batch":
        batch, steps = _log(rng, 2, 64), rng.randint(8, 32)
        prompt = _log(rng, 8, min(1900, 4096 // batch))
    else:
        batch, steps = rng.choice([1, 1, 2, 4]), 0
        prompt = _log(rng, 100, 2048)
    return dict(kind="generate", model=model, layers=layers, dtype=dtype, batch=batch, prompt=prompt, steps=steps)


# ---- models -------------------------------------------------------------------------------------------------
def _list_config(case: dict) -> dict:
    """config.json of the models given as a list of layers: the geometries of the layer benchmark at width 2048."""
    n, name = case["layers"], case["model"]
    if name == "fekorax":
        def attention(**more):
            return dict(type="attention", mlp=dict(kind="dense", ff=5632),
                        mixer=dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=3072), **more,
                                   rot=dict(base=500000.0, dims=64, scaling=dict(factor=8.0, low=1.0, high=4.0, original=8192))))
        matrix = dict(type="mlstm", mixer=dict(heads=8, dim=128, vdim=256, gate_cap=15.0), mlp=None)
        layers = [matrix, matrix, attention(), matrix, matrix, attention(kv_from=2)][:n]
        return dict(architecture="Fekorax", vocab=4096, width=2048, norm=dict(eps=1e-5), embedding=dict(scale=2048 ** 0.5), layers=layers)
    mixer = dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5, rot=dict(base=10000.0, dims=64))
    mlp = dict(kind="dense", ff=8448)
    if name == "fegetar_moe":
        mlp = dict(kind="moe", router=dict(experts=64, top=6), expert=dict(ff=1408, limit=7.0), shared=dict(ff=2816, limit=7.0))
    return dict(architecture="Fegetar", vocab=4096, width=2048, norm=dict(eps=1e-5), token_side=dict(dim=256),
                embedding=dict(bigram=dict(buckets=65521, mul_prev=1000003, mul_cur=101)),
                layers=[dict(type="latent_attention", mixer=mixer, mlp=mlp)] * n)


def _config(case: dict):
    """The model's configuration object."""
    name = case["model"]
    if name in LLAMAS:
        return L.LlamaConfig(**{**LLAMAS[name], "num_hidden_layers": case["layers"], "max_seq_len": MAX_SEQ}, weight_dtype=case["dtype"])
    cls = L.FekoraxConfig if name == "fekorax" else L.FegetarConfig
    return cls.from_dict(_list_config(case), MAX_SEQ, case["dtype"])


def _weight(model: str, name: str, shape: tuple, dtype: str) -> torch.Tensor:
    """One parameter on the GPU, by its name alone: matrices N(0, 0.02) in the storage type, vectors f32."""
    g = torch.Generator(device=DEV).manual_seed(zlib.crc32(f"{model}/{name}".encode()))
    w = torch.randn(shape, generator=g, device=DEV)
    if len(shape) == 2:
        return (w.mul_(STD)).to(torch.bfloat16 if dtype == "bf16" else torch.float32)
    if name.endswith(".f.b"):     # forget gates start open
        return w + 3.0
    if name.endswith((".i.b", ".sink")):
        return w
    centre = 0.0 if model.startswith("fegetar") and not name.endswith(("dkv.norm", "side.norm")) else 1.0  # (that model's other gains are 1 + w)
    return w * 0.1 + centre


_kept: dict = {}  # the one model that is loaded, by its configuration


def _model(case: dict):
    key = (case["model"], case["layers"], case["dtype"])
    if key not in _kept:
        _kept.clear()
        cfg = _config(case)
        cls = L.LlamaModel if case["model"] in LLAMAS else L.FekoraxModel if case["model"] == "fekorax" else L.FegetarModel
        model = cls(cfg)
        shapes = cfg.param_shapes()
        staging = torch.empty(max(math.prod(s) for s in shapes.values()) * 4, dtype=torch.uint8, pin_memory=True)
        for name, shape in shapes.items():
            w = _weight(case["model"], name, shape, case["dtype"])
            half = w.dtype == torch.bfloat16
            host = staging[: w.numel() * w.element_size()].view(w.dtype).view(w.shape)
            host.copy_(w)
            model.set_param(name, (host.view(torch.int16).numpy().view(np.uint16) if half else host.numpy()), as_bf16_bits=half)
        del w, host, staging
        torch.cuda.empty_cache()
        _kept[key] = model
    return _kept[key]


# ---- inputs ---------------------------------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed * 7919 + 17)


def _vocab(case: dict) -> int:
    return LLAMAS[case["model"]]["vocab_size"] if case["model"] in LLAMAS else 4096


def _tokens(case: dict, seed: int) -> np.ndarray:
    """Token ids [batch, prompt + steps]."""
    return np.random.default_rng(seed).integers(0, _vocab(case), (case["batch"], case["prompt"] + case["steps"]))


def _product(case: dict, seed: int):
    g = _gen(seed)
    k, n = case["k"], case["n"]
    x = torch.randn(k, generator=g, device=DEV)
    w = (torch.randn((n, k) if case["layout"] == "nk" else (k, n), generator=g, device=DEV) * STD).to(torch.bfloat16 if case["dtype"] == "bf16" else torch.float32)
    return x, w


def _logits(case: dict, seed: int):
    """Logits of a trained model's shape: a few candidates above a long tail; recent tokens and the uniform draws."""
    g = _gen(seed)
    z = torch.randn((case["rows"], case["vocab"]), generator=g, device=DEV) * 2.5
    z[:, : case["vocab"] // 64] += 4.0
    order = torch.argsort(torch.rand((case["rows"], case["vocab"]), generator=g, device=DEV), dim=1)
    z = torch.gather(z, 1, order).contiguous()
    rng = np.random.default_rng(seed)
    return z, rng.integers(0, case["vocab"], (case["rows"], 96)).astype(np.int32), rng.random(case["rows"])


def prepare(case: dict, seed: int) -> dict:
    ctx = L.default_context()
    s = dict(case=case, ctx=ctx)
    if case["kind"] == "gemv":
        s["x"], s["w"] = _product(case, seed)
        s["y"] = torch.empty(case["n"], device=DEV)
    elif case["kind"] == "sample":
        s["logits"], s["recent"], s["uniform"] = _logits(case, seed)
    else:
        s["model"] = _model(case)
        s["caches"] = s["model"].init_kv_caches(case["batch"])
        ids = _tokens(case, seed).astype(np.float32)
        s["prompt"], s["steps"] = np.ascontiguousarray(ids[:, : case["prompt"]]), np.ascontiguousarray(ids[:, case["prompt"]:].T[:, :, None])
        if case["batch"] > 1:
            s["ids"] = torch.from_numpy(s["steps"]).to(DEV)
            s["out"] = torch.empty((case["steps"], case["batch"], _vocab(case)), device=DEV)
    torch.cuda.synchronize()
    return s


def run(s: dict):
    case = s["case"]
    if case["kind"] == "gemv":
        L.gemv(s["ctx"], s["x"].data_ptr(), s["w"].data_ptr(), L.BF16 if case["dtype"] == "bf16" else L.F32, case["layout"] == "kn", case["k"], case["n"],
               s["y"].data_ptr())
        return s["y"]
    if case["kind"] == "sample":
        return [L.sample_top_p(s["ctx"], z.data_ptr(), case["vocab"], case["temperature"], case["top_p"], 1.05, rec, u)
                for z, rec, u in zip(s["logits"], s["recent"], s["uniform"])]
    model, caches = s["model"], s["caches"]
    with L.no_grad():
        model.reset_kv_caches(caches)
        first = model.forward(s["prompt"], caches, last_only=True)
        if case["batch"] == 1:
            return [first] + [model.forward(ids, caches) for ids in s["steps"]]
        for ids, out in zip(s["ids"], s["out"]):
            model.forward_device(ids.data_ptr(), case["batch"], 1, caches, out.data_ptr())
        return [first, s["out"]] if case["steps"] else [first]


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def _matrices(case: dict) -> tuple:
    """(numbers in the matrices that every token is multiplied with, numbers in the output matrix, numbers that only some tokens use)."""
    shapes = _config(case).param_shapes()
    head = {"lm_head.weight", "head"} if case["model"] != "fekorax" else {"embed"}
    tables = {"model.embed_tokens.weight", "embed", "bigram", "side.embed"} - head
    body = sum(math.prod(s) for n, s in shapes.items() if len(s) == 2 and n not in tables and n not in head and ".mlp.e" not in n)
    routed = sum(math.prod(s) for n, s in shapes.items() if ".mlp.e" in n)
    return body, sum(math.prod(shapes[n]) for n in head if n in shapes), routed


def work(case: dict) -> dict:
    size = 2 if case.get("dtype") == "bf16" else 4
    if case["kind"] == "gemv":
        return dict(bytes=size * case["k"] * case["n"] + 4 * (case["k"] + case["n"]), flops=2 * case["k"] * case["n"])
    if case["kind"] == "sample":
        return dict(bytes=4 * case["rows"] * case["vocab"], flops=10 * case["rows"] * case["vocab"])
    b, p, t = case["batch"], case["prompt"], case["steps"]
    body, head, routed = _matrices(case)
    used = routed * 6 // 64  # of the experts, by one token
    total = p + t
    cache = flops = 0
    if case["model"] in LLAMAS:
        c = LLAMAS[case["model"]]
        d = c.get("head_dim") or c["hidden_size"] // c["num_attention_heads"]
        row = case["layers"] * 2 * c["num_key_value_heads"] * d * 4
        cache = b * row * (p + sum(range(p + 1, total + 1)))
        flops = case["layers"] * b * c["num_attention_heads"] * 4 * d * (total * (total + 1) / 2)
    elif case["model"] == "fekorax":
        state = 4 * 8 * 128 * (256 + 1) * 4  # four matrix layers, f32
        row = 2 * 4 * 128 * 2
        cache = state * (1 + 2 * t) + row * p + 2 * row * sum(range(p + 1, total + 1))
        flops = 4 * total * 4 * 8 * 128 * 256 + 2 * 16 * 4 * 128 * (total * (total + 1) / 2)
    else:
        row = case["layers"] * 576 * 2
        cache = row * (p + sum(range(p + 1, total + 1)))
        flops = case["layers"] * 16 * 2 * (192 + 128) * (total * (total + 1) / 2)
    experts = min(1.0, b * p * 6 / 64)
    weights = size * ((1 + t) * (body + head) + experts * routed + t * used)
    return dict(bytes=weights + cache + 4 * b * (1 + t) * _vocab(case), flops=flops + 2 * b * (total * (body + used) + (1 + t) * head))


def tolerance(case: dict):
    """About four times what the present code was seen to be off the 64-bit result."""
    if case["kind"] == "sample":
        return "exact"  # token ids
    if case["kind"] == "gemv":
        return {"rel": 2e-6, "max": 4e-5}
    if case["model"] in LLAMAS:
        return {"rel": 5e-4, "max": 1e-2}  # (f32 activations in two bf16 halves through up to 32 layers: 2e-4 seen)
    return {"rel": 5e-4, "max": 1e-2} if case["dtype"] == "f32" else {"rel": 0.03, "max": 0.5}  # (16-bit activations: up to 1e-2)


# ---- the same in 64 bits ------------------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    if case["kind"] == "gemv":
        x, w = _product(case, seed)
        return torch.mv(w.double() if case["layout"] == "nk" else w.double().T, x.double())
    if case["kind"] == "sample":
        return None
    ids = torch.from_numpy(_tokens(case, seed)).to(DEV)
    cfg = _config(case)
    shapes = cfg.param_shapes()

    def weight(name):
        return _weight(case["model"], name, shapes[name], case["dtype"]).double()

    keep = slice(case["prompt"] - 1, None)
    if case["model"] in LLAMAS:
        logits = _llama(cfg, weight, ids, keep)
    else:
        plain = _fekorax if case["model"] == "fekorax" else _fegetar
        logits = plain(_list_config(case), weight, ids[0], keep)[None]
    if case["batch"] == 1:
        return [logits[:, 0]] + [logits[:, t:t + 1] for t in range(1, case["steps"] + 1)]
    return [logits[:, 0], logits[:, 1:].transpose(0, 1).contiguous()] if case["steps"] else [logits[:, 0]]


def _norm(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, freq, interleaved=False):
    """x [..., S, n]: pairs (i, i + half), or (2i, 2i + 1), turn by position times frequency."""
    half, s = len(freq), x.shape[-2]
    angle = torch.arange(s, device=DEV, dtype=freq.dtype)[:, None] * freq
    c, n = angle.double().cos(), angle.double().sin()
    part, rest = x[..., : 2 * half], x[..., 2 * half:]
    a, b = (part[..., 0::2], part[..., 1::2]) if interleaved else (part[..., :half], part[..., half:])
    u, v = a * c - b * n, b * c + a * n
    return torch.cat([torch.stack([u, v], -1).flatten(-2) if interleaved else torch.cat([u, v], -1), rest], -1)


def _attend(q, k, v, scale, sink=None):
    """q [H,S,D], k [G,S,D], v [G,S,E] -> [H,S,E], causal."""
    group, s = q.shape[0] // k.shape[0], q.shape[1]
    hidden = torch.ones((s, s), dtype=torch.bool, device=DEV).triu(1)
    out = []
    for h in range(q.shape[0]):
        z = (q[h] @ k[h // group].T * scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink[h].expand(s, 1)], 1)
        out.append(torch.softmax(z, -1)[:, :s] @ v[h // group])
    return torch.stack(out)


def _llama(cfg, weight, ids, keep):
    b, s = ids.shape
    hq, hkv, d, eps = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.resolved_head_dim, cfg.rms_norm_eps
    # (the model's tables of angles are f32 by definition)
    freq = (1.0 / torch.tensor(cfg.rope_theta, dtype=torch.float32) ** (torch.arange(0, d, 2, dtype=torch.float32) / d)).to(DEV)
    x = weight("model.embed_tokens.weight")[ids]
    for i in range(cfg.num_hidden_layers):
        p = f"model.layers.{i}."
        h = _norm(x, weight(p + "input_layernorm.weight"), eps)
        q, k, v = ((h @ weight(f"{p}self_attn.{n}_proj.weight").T).view(b, s, -1, d).transpose(1, 2) for n in "qkv")
        if cfg.qk_norm:
            q, k = _norm(q, weight(p + "self_attn.q_norm.weight"), eps), _norm(k, weight(p + "self_attn.k_norm.weight"), eps)
        q, k = _turn(q, freq), _turn(k, freq)
        a = torch.stack([_attend(q[j], k[j], v[j], d ** -0.5) for j in range(b)])
        x = x + a.transpose(1, 2).reshape(b, s, hq * d) @ weight(p + "self_attn.o_proj.weight").T
        h = _norm(x, weight(p + "post_attention_layernorm.weight"), eps)
        u = torch.nn.functional.silu(h @ weight(p + "mlp.gate_proj.weight").T) * (h @ weight(p + "mlp.up_proj.weight").T)
        x = x + u @ weight(p + "mlp.down_proj.weight").T
    return _norm(x[:, keep], weight("model.norm.weight"), eps) @ weight("lm_head.weight").T


def _gelu(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


def _fegetar(cfg, weight, ids, keep):
    s, eps = len(ids), cfg["norm"]["eps"]
    big, side = cfg["embedding"]["bigram"], cfg["token_side"]["dim"]
    pair = (ids[:-1] * big["mul_prev"] + ids[1:] * big["mul_cur"]) % big["buckets"]
    x = weight("embed")[ids] + weight("bigram")[torch.cat([pair.new_tensor([big["buckets"]]), pair])]
    token = weight("side.embed")[ids]

    def expert(h, p, limit):
        g = (h @ weight(p + ".gate").T).clamp(max=limit)
        u = (h @ weight(p + ".up").T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ weight(p + ".down").T

    for i, layer in enumerate(cfg["layers"]):
        m, mlp, p = layer["mixer"], layer["mlp"], f"l{i}."
        heads, d, rank = m["heads"], m["dim"], m["kv_rank"]
        freq = m["rot"]["base"] ** (-torch.arange(0, m["rot"]["dims"], 2, device=DEV, dtype=torch.float64) / m["rot"]["dims"])
        q = (x @ weight(p + "mix.q").T).view(s, heads, -1).transpose(0, 1)
        down = x @ weight(p + "mix.dkv").T
        c = _norm(down[:, :rank], weight(p + "mix.dkv.norm"), eps)
        k_rot = _turn(down[:, rank:], freq, True)
        q = torch.cat([q[..., :d], _turn(q[..., d:], freq, True)], -1)
        k = torch.cat([(c @ weight(p + "mix.uk").T).view(s, heads, d).transpose(0, 1), k_rot.expand(heads, s, -1)], -1)
        v = (c @ weight(p + "mix.uv").T).view(s, heads, -1).transpose(0, 1)
        a = _attend(q, k, v, m["scale"]) * torch.sigmoid(x @ weight(p + "mix.g").T).T[:, :, None]
        x = x + _norm(a.transpose(0, 1).reshape(s, -1) @ weight(p + "mix.o").T, 1 + weight(p + "norm1"), eps)
        if mlp["kind"] == "dense":
            y = _gelu(x @ weight(p + "mlp.up").T) @ weight(p + "mlp.down").T
        else:
            y = expert(x, p + "mlp.shared", mlp["shared"]["limit"])
            score, which = torch.sigmoid(x @ weight(p + "mlp.router").T).topk(mlp["router"]["top"], dim=1)
            for e in range(mlp["router"]["experts"]):
                t, j = torch.where(which == e)
                if len(t):
                    y[t] += expert(x[t] * score[t, j][:, None], f"{p}mlp.e{e}", mlp["expert"]["limit"])
        x = x + _norm(y, 1 + weight(p + "norm2"), eps)
        y = (_gelu(x @ weight(p + "side.gate").T) * token[:, i * side:(i + 1) * side]) @ weight(p + "side.proj").T
        x = x + _norm(y, weight(p + "side.norm"), eps)
    return _norm(x[keep], 1 + weight("final.norm"), eps) @ weight("head").T


def _fekorax(cfg, weight, ids, keep):
    s, eps = len(ids), cfg["norm"]["eps"]
    x = weight("embed")[ids] * cfg["embedding"]["scale"]
    kept = {}

    def matrix(h, m, p):
        heads, d = m["heads"], m["dim"]
        q, k, v = ((h @ weight(p + n).T).view(s, heads, -1) for n in "qkv")
        cap = m["gate_cap"]
        i, f = (cap * torch.tanh((h @ weight(p + n).T + weight(p + n + ".b")) / cap) for n in "if")
        # log weight of token j in the state after token t: sum of the log forget gates in between plus j's input gate
        run = torch.nn.functional.logsigmoid(f).cumsum(0)
        out = []
        for a in range(heads):
            z = run[:, a, None] - run[None, :, a] + i[None, :, a]
            z = z.masked_fill(torch.ones((s, s), dtype=torch.bool, device=DEV).triu(1), -math.inf)
            top = torch.maximum(z.amax(1), run[:, a])  # (the empty memory's running maximum is 0)
            w = torch.exp(z - top[:, None]) * (q[:, a] @ k[:, a].T) * d ** -0.5
            out.append(w @ v[:, a] / (torch.maximum(w.sum(1).abs(), torch.exp(-top)) + 1e-6)[:, None])
        y = _norm(torch.stack(out, 1), 1.0, eps).reshape(s, -1) * weight(p + "norm")
        return (y * torch.sigmoid(h @ weight(p + "g").T)) @ weight(p + "o").T

    def attention(h, m, p, i):
        rot = m["rot"]
        sc = rot["scaling"]
        freq = rot["base"] ** (-torch.arange(0, rot["dims"], 2, device=DEV, dtype=torch.float64) / rot["dims"])
        length = 2 * math.pi / freq
        mix = ((sc["original"] / length - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
        freq = (1 - mix) * freq / sc["factor"] + mix * freq
        if "kv_from" not in m:
            k = _norm((h @ weight(p + "k").T).view(s, m["kv_heads"], -1).transpose(0, 1), weight(p + "k.norm"), eps)
            kept[i] = _turn(k, freq), (h @ weight(p + "v").T).view(s, m["kv_heads"], -1).transpose(0, 1)
        k, v = kept[m.get("kv_from", i)]
        q = _turn(_norm((h @ weight(p + "q").T).view(s, m["heads"], -1).transpose(0, 1), weight(p + "q.norm"), eps), freq)
        a = _attend(q, k, v, m["scale"], weight(p + "sink")) * torch.sigmoid(h @ weight(p + "g").T).T[:, :, None]  # (shorter than a chunk)
        return a.transpose(0, 1).reshape(s, -1) @ weight(p + "o").T

    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        h = _norm(x, weight(p + "norm1"), eps)
        y = matrix(h, layer["mixer"], p + "mix.") if layer["type"] == "mlstm" else attention(h, layer["mixer"], p + "mix.", i)
        x = x + _norm(y, weight(p + "norm1b"), eps)
        if layer["mlp"]:
            h = _norm(x, weight(p + "norm2"), eps)
            y = (_gelu(h @ weight(p + "mlp.gate").T) * (h @ weight(p + "mlp.up").T)) @ weight(p + "mlp.down").T
            x = x + _norm(y, weight(p + "norm2b"), eps)
    return _norm(x[keep], weight("final.norm"), eps) @ weight("embed").T
