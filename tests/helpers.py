"""Shared helpers for the parity tests."""
from __future__ import annotations

import numpy as np

# Tolerances from the north star: per-step logits within rel 1e-4 for f32 weights, 1e-2 for bf16
# weights, where rel = max|a-b| / max|b| over one logits vector (error against the logit scale).
TOL_F32 = 1e-4
TOL_BF16 = 1e-2

# Sizes at which products run on pairs of SMs (test_plans.py checks that they do).
# m, k, n of plain products; all take the 256-wide tile but the last, whose f32 form takes the 128-wide one (and bf16 single SMs)
PAIRED_PRODUCTS = [(129, 1096, 9601), (513, 1160, 4865), (1281, 1160, 1921), (2300, 1544, 1031), (9473, 1096, 129), (5000, 1032, 1030)]
# hidden size, intermediate size, positions of a prompt, slices of K of its down product, tile widths of that and of its gate-and-up product,
# with bf16 and with f32 weights
PAIRED_PROMPTS = [
    (128, 136, 129, (1, 1), (128, 128), (128, 128)), (128, 200, 300, (1, 1), (128, 128), (128, 128)), (128, 264, 513, (1, 1), (128, 128), (128, 128)),
    (128, 128, 256, (1, 1), (128, 128), (128, 128)), (128, 1096, 129, (2, 2), (128, 128), (128, 128)), (128, 1544, 300, (3, 3), (128, 128), (128, 128)),
    (128, 2008, 513, (4, 4), (128, 128), (256, 256)), (768, 2248, 1500, (2, 4), (128, 256), (128, 128)),
]


def rel_err(a, b) -> float:
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    denom = max(float(np.max(np.abs(b))), 1e-30)
    return float(np.max(np.abs(a - b))) / denom


def small_cfg(**over) -> dict:
    cfg = dict(vocab_size=97, hidden_size=64, intermediate_size=160, num_hidden_layers=2, num_attention_heads=4,
               num_key_value_heads=2, rms_norm_eps=1e-5, max_seq_len=48, rope_theta=10000.0)
    cfg.update(over)
    return cfg


def cfg_obj(L, cfg: dict, weight_dtype="f32"):
    return L.LlamaConfig(**cfg, weight_dtype=weight_dtype)


def make_params(L, cfg: dict, seed: int, std: float = 0.02, round_bf16: bool = False, random_norms: bool = False) -> dict:
    from lumen_b200 import synth
    params = dict(synth.iter_params(L.LlamaConfig(**cfg), seed, std=std, round_bf16=round_bf16))
    if random_norms:
        rng = np.random.default_rng(seed + 1000)
        for k in params:
            if params[k].ndim == 1:
                params[k] = (1.0 + 0.1 * rng.standard_normal(params[k].shape)).astype(np.float32)
    return params
