"""Wide prompt passes (tens to hundreds of positions per pass): products, attention and the passes as a whole against
float64 and against the position-by-position loop, at the edges of the tiles of positions, rows and passes."""
import numpy as np
import pytest
import torch

import oracle
from conftest import ATOL, RTOL, assert_close
from helpers import SMALL_GPT2, SMALL_LLAMA, gpt2_pair, llama_pair
from wgml_b200 import synth

pytestmark = pytest.mark.gpu


def value_rows(fmt, dim, kv_heads, heads, n, seed):
    """Values of layer 0 for n prompt positions (cache rows) and the same in float64: one product of the normed embedding."""
    cfg = dict(SMALL_LLAMA, dim=dim, hidden_dim=256, n_layers=1, n_q_heads=heads, n_kv_heads=kv_heads, vocab_size=700, seq_len=n + 8)
    t = synth.llama_tensors(cfg, seed, scale=0.002)
    kv = dim * kv_heads // heads
    t["blk.0.attn_v.weight"] = synth.matrix(fmt, kv, dim, seed, "v", 0.002)
    t["token_embd.weight"] = (synth.F32, np.random.default_rng(seed).standard_normal(700 * dim).astype(np.float32) *
                              np.repeat(10.0 ** np.random.default_rng(1).uniform(-3, 3, 700), dim).astype(np.float32))
    gpu, _, _ = llama_pair(cfg, tensors=t)
    prompt = synth.prompt(n + 1, 700, seed)
    emb = t["token_embd.weight"][1].reshape(700, dim)[prompt[:n]].astype(np.float64)
    xn = emb / np.sqrt((emb ** 2).mean(1, keepdims=True) + cfg["rms_norm_eps"]) * t["blk.0.attn_norm.weight"][1].astype(np.float64)
    w = oracle.dequantize(fmt, t["blk.0.attn_v.weight"][1]).reshape(kv, dim).astype(np.float64)
    return gpu, prompt, xn @ w.T


@pytest.mark.parametrize("fmt", [synth.Q4_K, synth.Q6_K, synth.Q8_0])
@pytest.mark.parametrize("shape", [(256, 2, 4, 16), (768, 12, 12, 132), (4096, 32, 32, 260), (1024, 16, 16, 520), (2048, 16, 16, 128)])
def test_wide_product_vs_f64(fmt, shape):
    """As exact as the position-by-position product: the sums of both are good to a few units of 2^-22 of the row's
    terms, so the error of each row of outputs stays below 2e-6 of its norm and no element is off by more than 1e-5 of
    the row's RMS (f32 sums of up to 4096 products)."""
    dim, kvh, heads, n = shape
    gpu, prompt, ref = value_rows(fmt, dim, kvh, heads, n, 5)
    gpu.set_prefill(True)
    gpu.decode(prompt, 1)
    assert gpu.prefill_positions() == n - (n % 8 if n % 8 < 4 else 0)
    n = gpu.prefill_positions()
    got = gpu.value_cache(0)[:n].cpu().numpy().astype(np.float64)
    err = np.linalg.norm(got - ref[:n], axis=1) / np.linalg.norm(ref[:n], axis=1)
    worst = np.abs(got - ref[:n]).max(1) / np.sqrt((ref[:n] ** 2).mean(1))
    assert err.max() < 2e-6 and worst.max() < 1e-5, (err.max(), worst.max())


UNEVEN = ["loud", "louder", "heavy", "mean", "near constant", "scales"]


@pytest.mark.parametrize("fmt", [synth.Q4_K, synth.Q6_K, synth.Q8_0])
@pytest.mark.parametrize("kind", UNEVEN)
@pytest.mark.parametrize("dim,heads,kv_heads", [(1024, 16, 8), (4096, 32, 4)])
def test_wide_product_of_uneven_data(fmt, kind, dim, heads, kv_heads):
    """Loud columns, heavy tails, inputs of one sign, group scales that lie far apart: the product's error stays within three units
    of 2^-23 of the row of outputs (2-norm), one each for the two digits of an activation (2^-24 of the loudest of its 256
    columns), the sums of a unit and those over the units.  (The eight-position product, whose exponents belong to 32
    columns: 1.2e-7 to 1.6e-6 on the same data.)"""
    rng = np.random.default_rng(11)
    n, kv = 132, dim // heads * kv_heads
    cfg = dict(SMALL_LLAMA, dim=dim, hidden_dim=256, n_layers=1, n_q_heads=heads, n_kv_heads=kv_heads, vocab_size=300, seq_len=n + 8)
    t = synth.llama_tensors(cfg, 3, scale=0.002)
    w = np.ascontiguousarray(synth.matrix(fmt, kv, dim, 5, "v", 0.002)[1]).view(np.uint8).reshape(-1, {synth.Q4_K: 144, synth.Q6_K: 210, synth.Q8_0: 34}[fmt]).copy()
    at = 208 if fmt == synth.Q6_K else 0
    d = w[:, at:at + 2].copy().view(np.float16)[:, 0].astype(np.float32)
    if kind == "scales":
        d *= np.exp(rng.standard_normal(len(d)).astype(np.float32))
        w[:, at:at + 2] = d.astype(np.float16).view(np.uint8).reshape(-1, 2)
    if fmt == synth.Q4_K:   # mins that centre the codes, as quantised weights have them
        w[:, 2:4] = (w[:, :2].copy().view(np.float16)[:, 0].astype(np.float32) * 7.5).astype(np.float16).view(np.uint8).reshape(-1, 2)
    t["blk.0.attn_v.weight"] = (fmt, w.reshape(-1))
    t["blk.0.attn_norm.weight"] = (synth.F32, np.ones(dim, np.float32))
    e = rng.standard_t(2, (300, dim)) if kind == "heavy" else rng.standard_normal((300, dim))
    if kind == "loud": e[:, ::256] *= 100
    if kind == "louder": e[:, 5] *= 1000
    if kind == "mean": e += 1
    if kind == "near constant": e = 1 + 0.05 * e
    e = e.astype(np.float32)
    t["token_embd.weight"] = (synth.F32, e.reshape(-1))
    gpu, _, _ = llama_pair(cfg, tensors=t)
    gpu.set_prefill(True)
    prompt = rng.integers(0, 300, n + 1, dtype=np.uint32)
    gpu.decode(prompt, 1)
    assert gpu.prefill_positions() == n
    x = e[prompt[:n]].astype(np.float64)
    x /= np.sqrt((x ** 2).mean(1, keepdims=True) + cfg["rms_norm_eps"])
    ref = x @ oracle.dequantize(fmt, w.reshape(-1)).reshape(kv, dim).astype(np.float64).T
    got = gpu.value_cache(0)[:n].cpu().numpy().astype(np.float64)
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.mean() < 3 * 2.0 ** -23, (err.mean(), err.max())


def _caches(gpu, n):
    return [(gpu.key_cache(l)[:n].cpu().numpy(), gpu.value_cache(l)[:n].cpu().numpy()) for l in range(gpu.config.n_layers)]


@pytest.mark.parametrize("case", [
    dict(n_prompt=17, heads=8, kv=8, qwen=False, mixed=False),              # the smallest wide pass
    dict(n_prompt=72, heads=8, kv=2, qwen=True, mixed=False),               # 71: 64-position attention tile + 7; biases, Neox RoPE, grouped heads
    dict(n_prompt=90, heads=4, kv=4, qwen=False, mixed=True),               # head size 128; three formats in one layer's products
    dict(n_prompt=700, heads=4, kv=2, qwen=False, mixed=False, seq_len=720),   # two passes: the second attends to the first's rows
    dict(n_prompt=530, heads=8, kv=4, qwen=False, mixed=True, seq_len=700, start=150, n_layers=1),   # a pass that starts at a later position
    # few positions at a later one: blocks of the attention share the cache rows of a head
    dict(n_prompt=17, heads=8, kv=2, qwen=True, mixed=False, seq_len=1700, start=1630, n_layers=2),  # 26 tiles of rows, the last one short
    dict(n_prompt=73, heads=4, kv=4, qwen=False, mixed=False, seq_len=900, start=762, n_layers=2),   # head size 128; two tiles of positions, of 12 and 13
    dict(n_prompt=41, heads=8, kv=8, qwen=False, mixed=False, seq_len=256, start=200, n_layers=2),   # two blocks of two tiles each
])
def test_wide_passes_match_sequential_loop(case):
    cfg = dict(SMALL_LLAMA, n_layers=case.get("n_layers", 3), n_q_heads=case["heads"], n_kv_heads=case["kv"], seq_len=case.get("seq_len", 128))
    t = synth.llama_tensors(cfg, 21, biases=case["qwen"], scale=0.002)
    if case["mixed"]:
        kv = 512 * case["kv"] // case["heads"]
        t["blk.0.attn_v.weight"] = synth.matrix(synth.Q6_K, kv, 512, 3, "v6", 0.002)
        t["blk.0.ffn_down.weight"] = synth.matrix(synth.Q6_K, 512, 1024, 3, "d6", 0.002)
        t["blk.0.ffn_up.weight"] = synth.matrix(synth.Q8_0, 1024, 512, 3, "up8", 0.002)
        t["blk.0.attn_k.weight"] = synth.matrix(synth.Q8_0, kv, 512, 3, "k8", 0.002)
    seq, _, _ = llama_pair(cfg, qwen=case["qwen"], tensors=t)
    bat, _, _ = llama_pair(cfg, qwen=case["qwen"], tensors=t)
    bat.set_prefill(True)
    start = case.get("start", 0)
    before = synth.prompt(start + 1, cfg["vocab_size"], seed=4)
    prompt = synth.prompt(case["n_prompt"], cfg["vocab_size"], seed=5)
    toks = []
    for m in (seq, bat):
        if start:
            m.decode(before, 0)
        toks.append(m.decode(prompt, 6, start_pos=start))
    assert np.array_equal(*toks), "greedy tokens differ between wide and sequential prompt"
    n = start + case["n_prompt"] - 1 + 6
    for l, ((kb, vb), (ks, vs)) in enumerate(zip(_caches(bat, n), _caches(seq, n))):
        assert_close(kb, ks, RTOL, ATOL * max(1.0, float(np.abs(ks).max())), f"key cache {l}")
        assert_close(vb, vs, RTOL, ATOL * max(1.0, float(np.abs(vs).max())), f"value cache {l}")
    lb, ls = bat.logits().cpu().numpy(), seq.logits().cpu().numpy()
    assert_close(lb, ls, RTOL, ATOL * max(1.0, float(np.abs(ls).max())), "final logits")


@pytest.mark.parametrize("qtype,n_prompt", [(synth.Q8_0, 65), (synth.Q4_K, 121)])
def test_wide_gpt2_passes_match_sequential_loop(qtype, n_prompt):
    cfg = dict(SMALL_GPT2, default_qtype=qtype)
    seq, _, _ = gpt2_pair(cfg, seed=31, scale=0.002)
    bat, _, _ = gpt2_pair(cfg, seed=31, scale=0.002)
    bat.set_prefill(True)
    prompt = synth.prompt(n_prompt, cfg["n_vocab"], seed=7)
    assert np.array_equal(bat.decode(prompt, 6), seq.decode(prompt, 6))
    for l in range(cfg["n_layer"]):
        for a, b in ((bat.key_cache(l), seq.key_cache(l)), (bat.value_cache(l), seq.value_cache(l))):
            a, b = a[:n_prompt].cpu().numpy(), b[:n_prompt].cpu().numpy()
            assert_close(a, b, RTOL, ATOL * max(1.0, float(np.abs(b).max())), f"cache {l}")


@pytest.mark.parametrize("heads,n_prompt,bad", [(8, 90, (40, 70)), (4, 140, (63, 64, 100)), (8, 40, (38,))])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_later_positions_reach_no_earlier_one(heads, n_prompt, bad, value):
    """Positions whose embedding (hence every cache row from them on) is not finite leave the rows of the positions before them
    as the token loop has them, in every layer: attention is causal also where a weight of zero meets an infinity."""
    cfg = dict(SMALL_LLAMA, n_layers=3, n_q_heads=heads, n_kv_heads=heads, seq_len=160)
    t = synth.llama_tensors(cfg, 23, scale=0.002)
    emb = t["token_embd.weight"]
    t["token_embd.weight"] = (synth.F32, oracle.dequantize(emb[0], emb[1]).reshape(cfg["vocab_size"], cfg["dim"]).astype(np.float32).copy())
    t["token_embd.weight"][1][7, ::5] = value
    t["token_embd.weight"] = (synth.F32, t["token_embd.weight"][1].ravel())
    prompt = synth.prompt(n_prompt, cfg["vocab_size"], seed=5)
    prompt[prompt == 7] = 8
    prompt[list(bad)] = 7
    seq, _, _ = llama_pair(cfg, tensors=t)
    wide, _, _ = llama_pair(cfg, tensors=t)
    wide.set_prefill(True)
    for m in (seq, wide):
        m.decode(prompt, 1)
    assert wide.prefill_positions() > bad[-1]
    n = bad[0]
    for l, ((kb, vb), (ks, vs)) in enumerate(zip(_caches(wide, n), _caches(seq, n))):
        assert np.isfinite(ks).all() and np.isfinite(vs).all()
        assert_close(kb, ks, RTOL, ATOL * max(1.0, float(np.abs(ks).max())), f"key cache {l}")
        assert_close(vb, vs, RTOL, ATOL * max(1.0, float(np.abs(vs).max())), f"value cache {l}")


@pytest.mark.parametrize("arch", ["llama", "gpt2"])
def test_prompt_passes_without_room_for_the_wide_ones(arch):
    """With device memory for the eight-position passes but not for the buffers of the wide ones, enabling prompt passes
    succeeds, what was half allocated is given back and prompts go through passes of eight positions."""
    if arch == "llama":   # the wide buffers are about 0.3 GB here, the others 0.1 GB
        cfg = dict(SMALL_LLAMA, hidden_dim=28672, n_layers=1, seq_len=700)
        seq, _, t = llama_pair(cfg, seed=3, scale=0.002)
        m, _, _ = llama_pair(cfg, tensors=t)
        vocab = cfg["vocab_size"]
    else:
        cfg = dict(SMALL_GPT2, ff_len=28672, n_layer=1, n_seq=700)
        seq, _, _ = gpt2_pair(cfg, seed=3, scale=0.002)
        m, _, _ = gpt2_pair(cfg, seed=3, scale=0.002)
        vocab = cfg["n_vocab"]

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    prompt = synth.prompt(41, vocab, 8)
    exp = seq.decode(prompt, 4)
    m.decode(prompt, 4)   # what decode itself allocates is there
    torch.cuda.empty_cache()
    before = free()
    m.set_prefill(True)
    need = before - free()
    m.set_prefill(False)
    short = 120 << 20
    filler = torch.empty(free() - (need - short), dtype=torch.uint8, device="cuda")
    try:
        m.set_prefill(True)
        assert free() > short // 2, "buffers of the wide passes are kept although they are not complete"
        got = m.decode(prompt, 4)
        assert m.prefill_positions() == 40
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(got, exp)
