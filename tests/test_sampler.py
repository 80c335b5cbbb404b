"""Nucleus sampling: the oracle's restatement of `sample_top_p` (src/main.rs:74-137) on CPU, and the device
sampler against it on a GPU (same token for the same uniform draw)."""
import subprocess
import sys
import textwrap
from pathlib import Path

import numpy as np
import pytest

from helpers import small_cfg, make_params


def test_oracle_sampler_properties(oracle):
    rng = np.random.default_rng(0)
    lg = (rng.standard_normal(500) * 3).astype(np.float32)
    top = int(lg.argmax())
    # a vanishing nucleus or temperature is greedy
    assert oracle.sample_top_p(lg, 1.0, 0.0, 1.0, [], 0.7) == top
    assert oracle.sample_top_p(lg, 1e-9, 0.9, 1.0, [], 0.3) == top
    # r = 0 always returns the most probable token, r -> 1 the last token of the nucleus
    assert oracle.sample_top_p(lg, 0.8, 0.9, 1.0, [], 0.0) == top
    p = np.exp((lg / np.float32(0.8)).astype(np.float64))
    p /= p.sum()
    order = np.argsort(-p, kind="stable")
    cut = int(np.searchsorted(np.cumsum(p[order]), 0.9) + 1)
    assert oracle.sample_top_p(lg, 0.8, 0.9, 1.0, [], 0.999999) in set(order[max(0, cut - 2):cut + 1].tolist())
    # a penalty > 1 divides once per occurrence: enough of them dethrone the top token
    assert oracle.sample_top_p(lg, 1.0, 0.0, 4.0, [top] * 6, 0.5) != top
    assert oracle.sample_top_p(lg, 1.0, 0.0, 1.0, [top] * 6, 0.5) == top   # penalty 1.0 is off
    # empirical frequencies follow the renormalised nucleus
    draws = [oracle.sample_top_p(lg, 0.8, 0.5, 1.0, [], float(u)) for u in rng.random(4000)]
    cut5 = int(np.searchsorted(np.cumsum(p[order]), 0.5) + 1)
    assert set(draws) <= set(order[:cut5].tolist())
    freq = np.bincount(draws, minlength=lg.size) / len(draws)
    want = np.zeros_like(p)
    want[order[:cut5]] = p[order[:cut5]] / p[order[:cut5]].sum()
    assert np.abs(freq - want).max() < 0.03


@pytest.mark.gpu
@pytest.mark.parametrize("vocab,scale", [(97, 3.0), (32000, 4.0), (32000, 0.05), (151936, 6.0)])
def test_device_sampler_matches_oracle(L, ctx, oracle, vocab, scale):
    rng = np.random.default_rng(vocab)
    lg = (rng.standard_normal(vocab) * scale).astype(np.float32)
    lg[5] = lg[6]  # a tie: the stable sort keeps index order
    t = L.Tensor.from_array_no_grad(lg)
    recent = rng.integers(0, vocab, size=40).tolist() + [int(lg.argmax())] * 3
    mismatches = 0
    cases = [(0.8, 0.9, 1.1, recent), (1.0, 0.5, 1.0, []), (0.3, 0.95, 1.3, recent[:7]), (1.0, 0.0, 1.0, []), (1.5, 1.0, 1.0, [])]
    for temp, top_p, pen, rec in cases:
        for u in rng.random(12).astype(np.float32):
            got = L.sample_top_p(ctx, t.data_ptr, vocab, temp, top_p, pen, rec, float(u))
            want = oracle.sample_top_p(lg, temp, top_p, pen, rec, float(u))
            mismatches += int(got != want)
    # the softmax denominator is a tree sum on the device and a sequential sum in the reference: a draw that sits
    # within an ulp of a boundary may fall on the other side
    assert mismatches <= 1, mismatches


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [1, 2, 33, 256, 257, 1023, 1025, 4099, 32000, 151936, 262144, 262145])
@pytest.mark.parametrize("shape", ["peaked", "broad", "close", "masked", "equal"])
def test_sampler_paths_draw_from_the_nucleus(L, ctx, vocab, shape):
    """Edges of the sampler's cluster kernel (vocabulary, nuclei of one to 10^5 tokens, crowded bins) and of the general path behind it.

    Bound: the drawn token's interval of the cumulative distribution, in 64 bits over the stable order, holds the draw.  A sum
    of n probabilities in f32 is off by at most n * 2^-24 of itself, and so is the nucleus' mass; tokens of nearly equal probability may change
    places, which moves an interval by less than their spread (expf is good to 2 ulp: 2^-22 of a probability per place)."""
    rng = np.random.default_rng(vocab * 7 + len(shape))
    lg = rng.standard_normal(vocab) * {"peaked": 3.0, "broad": 0.9, "close": 0.02, "masked": 1.0, "equal": 0.0}[shape]
    if shape == "peaked":
        lg[rng.permutation(vocab)[: max(1, vocab // 64)]] += 5.0
    if shape == "masked":
        lg[rng.random(vocab) < 0.4] = -np.inf
        lg[vocab // 2] = 1.0
    lg = lg.astype(np.float32)
    t = L.Tensor.from_array_no_grad(lg)
    for temp, top_p, pen, recent in [(0.8, 0.9, 1.05, rng.integers(0, vocab, 96).tolist()), (1.0, 0.95, 1.0, []), (0.6, 0.99, 1.3, [vocab - 1] * 2), (1.0, 0.9995, 1.0, [])]:
        z = lg.copy()
        for tok in recent if pen > 1 else []:
            z[tok] = np.float32(z[tok] / np.float32(pen))
        z = (z / np.float32(temp)).astype(np.float32)
        p = np.exp(z.astype(np.float64) - z.max())
        p /= p.sum()
        order = np.argsort(-z, kind="stable")
        cum = np.cumsum(p[order])
        m = min(int(np.searchsorted(cum, np.float64(np.float32(top_p)))) + 1, vocab)
        place = np.empty(vocab, np.int64)
        place[order] = np.arange(vocab)
        slack = 3 * vocab * 2.0 ** -24 + 2.0 ** -22 + 2 * p[order[m - 1]]
        for u in list(rng.random(6).astype(np.float32)) + [np.float32(0), np.float32(1)]:
            got = L.sample_top_p(ctx, t.data_ptr, vocab, temp, top_p, pen, recent, float(u))
            i = place[got]
            assert cum[i] - p[got] <= top_p * (1 + slack), (temp, top_p, u)
            top = cum[m - 1]
            # (the last of the nucleus also answers draws beyond the sum, but only those)
            assert (cum[i] - p[got] - slack) / top <= u and (u <= (cum[i] + slack) / top or i >= m - 1), (temp, top_p, u, i, m)


@pytest.mark.gpu
def test_lists_on_both_sides_of_the_shared_memory(L, ctx, oracle):
    """Lists of up to 2048 candidates stay in one SM's shared memory, longer ones cross the L2: nearly all of m likely tokens make the list."""
    rng = np.random.default_rng(12)
    mismatches = 0
    for m in range(2040, 2200, 10):
        lg = np.full(9000, -30.0, np.float32)
        lg[rng.permutation(9000)[:m]] = (rng.standard_normal(m) * 0.7).astype(np.float32)
        t = L.Tensor.from_array_no_grad(lg)
        for u in list(rng.random(5).astype(np.float32)) + [np.float32(0), np.float32(1)]:
            mismatches += L.sample_top_p(ctx, t.data_ptr, 9000, 1.0, 0.99, 1.0, [], float(u)) != oracle.sample_top_p(lg, 1.0, 0.99, 1.0, [], float(u))
    assert mismatches <= 2, mismatches  # (as above: draws within an ulp of a boundary)


@pytest.mark.gpu
def test_a_report_of_earlier_work_comes_back_from_the_draw(L, ctx, oracle):
    """An id beyond the vocabulary in a step whose errors nothing has asked for yet: the draw behind it raises, the next one draws."""
    cfg = small_cfg()
    model = L.LlamaModel(L.LlamaConfig(**cfg))
    model.load_state(make_params(L, cfg, 17))
    caches = model.init_kv_caches(2)
    rng = np.random.default_rng(4)
    lg = (rng.standard_normal(500) * 2).astype(np.float32)
    t, ids, out = (L.Tensor.from_array_no_grad(a) for a in (lg, np.array([3.0, cfg["vocab_size"]], np.float32), np.zeros((2, cfg["vocab_size"]), np.float32)))
    with L.no_grad():
        model.forward_device(ids.data_ptr, 2, 1, caches, out.data_ptr)
        with pytest.raises(L.LumenError) as e:
            L.sample_top_p(ctx, t.data_ptr, 500, 0.8, 0.9, 1.0, [], 0.4)
    assert e.value.code == L._lib.ERR_EMBED_RANGE
    for u in (0.1, 0.4, 0.8):
        assert L.sample_top_p(ctx, t.data_ptr, 500, 0.8, 0.9, 1.0, [], u) == oracle.sample_top_p(lg, 0.8, 0.9, 1.0, [], u)


WAITER = textwrap.dedent("""
    import ctypes, sys, time
    sys.path.insert(0, %r)
    cuda, dev = ctypes.CDLL("libcuda.so.1"), ctypes.c_int()
    assert cuda.cuInit(0) == 0 and cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cuda.cuDevicePrimaryCtxSetFlags_v2(dev, 4) == 0  # of this process: threads that wait for the device sleep
    import numpy as np
    import lumen_b200 as L
    ctx = L.default_context()
    logits = L.Tensor.from_array_no_grad((np.random.default_rng(0).standard_normal(32000) * 3).astype(np.float32))
    n = 6144
    a = L.Tensor.from_array_no_grad(np.ones((n, n), np.float32))
    draw = lambda: L.sample_top_p(ctx, logits.data_ptr, 32000, 0.8, 0.9, 1.0, [], 0.5)
    first = draw()
    with L.no_grad():
        L.matmul(a, a)
        ctx.synchronize()
        for _ in range(300):
            L.matmul(a, a)
    wall, cpu = time.perf_counter(), time.thread_time()
    same = draw() == first
    print("WAITED", round(time.perf_counter() - wall, 3), round(time.thread_time() - cpu, 3), same)
""")


@pytest.mark.gpu
def test_a_draw_behind_a_long_backlog_waits_as_the_device_is_told():
    """A tenth of a second and more of work ahead of the draw, in a process whose waits for the device sleep: the call does not keep a core busy all that time."""
    r = subprocess.run([sys.executable, "-c", WAITER % str(Path(__file__).resolve().parents[1])], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    wall, cpu, same = r.stdout.split("WAITED")[1].split()
    assert same == "True" and float(wall) > 0.1 and float(cpu) < 0.02 + 0.4 * float(wall), r.stdout


@pytest.mark.gpu
def test_forward_sample_equals_forward_then_oracle_sampler(L, oracle):
    cfg = small_cfg()
    params = make_params(L, cfg, 17, std=0.3)
    m1, m2 = (L.LlamaModel(L.LlamaConfig(**cfg)) for _ in range(2))
    m1.load_state(params)
    m2.load_state(params)
    c1, c2 = m1.init_kv_caches(1), m2.init_kv_caches(1)
    rng = np.random.default_rng(3)
    toks = [3, 9, 27, 11]
    with L.no_grad():
        ids = np.asarray(toks, np.float32)[None]
        for step in range(10):
            u = float(rng.random())
            logits = m1.forward(ids, c1)[0, -1]
            want = oracle.sample_top_p(logits, 0.8, 0.9, 1.1, toks[-96:], u)
            got = m2.forward_sample(ids, c2, 0.8, 0.9, 1.1, toks[-96:], u)
            assert got == want, step
            toks.append(got)
            ids = np.asarray([[got]], np.float32)   # generated token fed back, as main.rs:367-372
    assert c1[0].len == c2[0].len == 4 + 9
