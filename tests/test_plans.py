"""Which kernel multiplies many rows, and which attends in a batched decode step: the rules of dispatch on the CPU, against what was measured on a B200 (148 SMs)."""
import subprocess
from pathlib import Path

import pytest

from helpers import PAIRED_PRODUCTS, PAIRED_PROMPTS

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    out = tmp_path_factory.mktemp("plan") / "plan_check"
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", str(ROOT / "lumen_b200" / "csrc"), str(ROOT / "tests" / "cpp" / "plan_check.cpp"),
                        "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]

    def run(*line):
        r = subprocess.run([str(out)], input=" ".join(str(int(x) if isinstance(x, bool) else x) for x in line), capture_output=True, text=True, timeout=60)
        return tuple(int(x) for x in r.stdout.split())

    return run


# m, k, n, bf16 weights, microseconds of the whole product with 128 x 128 tiles of single SMs, 256 x 128 and 256 x 256 tiles of pairs
MEASURED = [
    (129, 5632, 2048, True, 48.9, 56.1, 67.0), (192, 2048, 256, True, 25.5, 29.0, 35.4), (257, 2048, 5632, True, 29.2, 49.4, 39.8),
    (384, 2048, 11264, True, 49.1, 68.3, 62.5), (512, 4096, 6144, True, 75.4, 82.7, 61.2), (768, 4096, 4096, True, 73.7, 80.5, 58.3),
    (1025, 1024, 1024, True, 21.6, 24.2, 28.5), (1025, 2048, 2048, True, 29.6, 49.6, 39.3), (1777, 4096, 4096, True, 136.6, 148.9, 106.4),
    (2048, 2048, 256, True, 29.0, 33.2, 39.7), (2048, 5632, 2048, True, 100.2, 110.7, 83.1), (4096, 4096, 12288, True, 814.8, 736.8, 579.3),
    (257, 4096, 12288, False, 179.3, 206.1, 207.3), (640, 576, 1536, False, 25.9, 29.1, 35.7), (768, 12288, 4096, False, 324.2, 331.6, 266.1),
    (1777, 4096, 4096, False, 206.0, 207.8, 167.5), (8192, 11008, 4096, False, 1860.5, 2141.6, 1570.0),
]


@pytest.mark.parametrize("m,k,n,bf16,single,pair128,pair256", MEASURED)
def test_plain_products_take_the_kernel_that_was_faster(plan, m, k, n, bf16, single, pair128, pair256):
    times = {0: single, 128: pair128, 256: pair256}
    bn, splits, per = plan("plain", m, k, n, bf16)
    assert times[bn] <= 1.1 * min(times.values()) and splits == 1 and per * 64 >= k


# m, k, n, bf16 weights, microseconds with tiles of 256, 224 and 192 columns
WIDTHS = [
    (3000, 1024, 1024, False, 38.6, 36.5, 34.8), (1536, 2048, 2560, False, 64.7, 60.7, 78.6), (4096, 2048, 2560, False, 139.3, 128.0, 134.4),
    (1777, 2048, 5632, False, 134.6, 123.6, 113.6), (900, 4096, 24576, False, 577.7, 535.0, 540.5), (257, 1024, 32000, False, 133.8, 126.1, 131.6),
    (4096, 4096, 6144, True, 331.5, 328.9, 331.7), (1280, 12288, 4096, True, 276.7, 249.9, 241.7), (1777, 11008, 4096, True, 266.5, 251.0, 322.4),
    (1777, 5632, 2048, True, 83.6, 78.1, 116.7), (513, 4096, 4096, True, 57.8, 53.2, 52.4),
]


@pytest.mark.parametrize("m,k,n,bf16,w256,w224,w192", WIDTHS)
def test_widths_of_tiles_that_were_faster(plan, m, k, n, bf16, w256, w224, w192):
    (bn,) = plan("width", m, n, 0, 1)
    assert plan("plain", m, k, n, bf16)[0] == 256 and {256: w256, 224: w224, 192: w192}[bn] <= 1.02 * min(w256, w224, w192)


def test_sizes_of_the_gpu_tests_reach_what_they_claim(plan):
    for m, k, n in PAIRED_PRODUCTS[:-1]:
        assert plan("plain", m, k, n, True)[0] == plan("plain", m, k, n, False)[0] == 256
    assert plan("plain", *PAIRED_PRODUCTS[-1], False)[0] == 128 and plan("plain", *PAIRED_PRODUCTS[-1], True)[0] == 0
    for h, inter, prompt, slices, down, gate_up in PAIRED_PROMPTS:
        for bf16 in (True, False):
            products = 2 if bf16 else 3
            assert plan("pair", prompt, inter, h, products, False, True)[:2] == (down[not bf16], slices[not bf16])
            assert plan("pair", prompt, h, 2 * inter, products, True, False)[0] == gate_up[not bf16]


def test_plans_cover_the_whole_of_k(plan):
    for m in (129, 300, 1025, 8192):
        for k in (8, 64, 520, 1096, 2008, 4096, 11008):
            for n in (128, 136, 1032, 4096):
                for products in (2, 3):
                    for kind in ((False, False), (False, True), (True, False)):
                        bn, splits, per = plan("pair", m, k, n, products, *kind)
                        assert bn in (128, 256) and 1 <= splits <= 4 and (splits - 1) * per * 64 < k <= splits * per * 64
                bn, splits, per = plan("plain", m, k, n, True)
                assert bn in (0, 128, 256) and splits == 1 and per * 64 >= k


# sequences, query heads, KV heads, head size, positions, microseconds of a step of four layers with the batched kernel and with the general one
ATTENDED = [
    (64, 32, 4, 64, 500, 318.1, 343.5), (64, 32, 4, 64, 1500, 501.2, 457.9), (64, 32, 4, 64, 4096, 927.2, 770.2), (32, 32, 4, 64, 1000, 276.8, 286.6),
    (32, 32, 4, 64, 2000, 372.8, 340.2), (16, 32, 4, 64, 2000, 257.7, 295.9), (16, 32, 4, 64, 4096, 364.1, 335.6), (8, 32, 4, 64, 3000, 278.7, 250.2),
    (4, 32, 4, 64, 3000, 232.4, 262.9), (2, 32, 4, 64, 2000, 188.9, 263.4), (64, 32, 8, 64, 1000, 490.2, 498.0), (64, 32, 8, 64, 2000, 710.2, 661.3),
    (16, 32, 8, 64, 1500, 266.4, 273.2), (16, 32, 8, 64, 4096, 460.9, 395.0), (4, 32, 8, 64, 4096, 272.6, 252.1), (64, 16, 8, 64, 4096, 938.4, 973.1),
    (64, 32, 8, 128, 4096, 1741.9, 2046.6), (64, 32, 4, 128, 4096, 1284.9, 1497.7), (32, 16, 16, 128, 4096, 1552.8, 1987.0), (64, 16, 16, 64, 4096, 1724.6, 1886.1),
]


@pytest.mark.parametrize("b,hq,hkv,d,at,rows,general", ATTENDED)
def test_batched_steps_take_the_attention_that_was_faster(plan, b, hq, hkv, d, at, rows, general):
    (parts,) = plan("attn", b, hq, hkv, d, at)
    assert (rows if parts else general) <= 1.02 * min(rows, general) and parts in (0, 1, 2, 4, 8)
