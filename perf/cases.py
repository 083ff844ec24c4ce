"""Workloads whose speed is watched: what a user of this package has it do, through its public entry points.

Kinds of a case:
  gemv       one `GemvQuant.dispatch`: a matrix of GGUF blocks times one vector
  gemm       one `Q4KTiles` / `Q6KTiles` / `Q80Tiles` product with 1 to 8 vectors
  attention  one `BatchedMultiqueryAttention.dispatch` over a filled KV cache (no weights asked for)
  layer      one decoder layer at one position, op by op, as a host program that keeps its own schedule calls it
  model      one `decode` call of `Llama2` or `Gpt2`: `prompt` forced ids from position `start`, then `gen` ids,
             greedy (temperature 0) or sampled; `prefill` says whether batched prompt passes are switched on

No weights or vocabularies exist offline: blocks are random, with block scales such that a matrix row has the norm of
a trained one (entries of standard deviation ~ 1/sqrt(ncols), centred), so that activations keep the magnitudes and
the tokens the variety of real use.  All of it is drawn from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from wgml_b200 import ops
from wgml_b200.models import Gpt2, Gpt2Params, Llama2, Llama2Config, LlamaModelType

F32, F16, Q4_0, Q8_0, Q4_K, Q5_K, Q6_K = ops.F32, ops.F16, ops.Q4_0, ops.Q8_0, ops.Q4_K, ops.Q5_K, ops.Q6_K
QTYPE = {"f32": F32, "f16": F16, "q4_0": Q4_0, "q8_0": Q8_0, "q4_k": Q4_K, "q5_k": Q5_K, "q6_k": Q6_K}
# standard deviation of a dequantised value over the block scale, uniform codes and sub-scales, mins centring the codes
SPREAD = {Q4_0: 4.6, Q8_0: 73.9, Q4_K: 258.0, Q5_K: 530.0, Q6_K: 1367.0}
DMIN = {Q4_K: 7.5, Q5_K: 15.5}          # dmin = DMIN * d: mean of the codes
SCALE_AT = {Q4_0: 0, Q8_0: 0, Q4_K: 0, Q5_K: 0, Q6_K: 208}


def listed():
    return [
        # The smallest call: one projection of a 7B-sized layer, dispatched by a host that keeps its own schedule.
        dict(name="gemv q4_k 4096x4096", kind="gemv", qtype="q4_k", nrows=4096, ncols=4096),
        # The largest single product of a 7B model: the output head, in its usual format.
        dict(name="gemv q6_k 32000x4096", kind="gemv", qtype="q6_k", nrows=32000, ncols=4096),
        # Several vectors at once (parallel requests, a short prompt chunk) against one FFN matrix.
        dict(name="gemm q4_k 11008x4096 x8", kind="gemm", qtype="q4_k", nrows=11008, ncols=4096, nvec=8),
        # Grouped-query attention at a long context, heads of the 70B configuration.
        dict(name="attention gqa 4000", kind="attention", heads=64, kv_mul=8, head_size=128, seq_len=4224, pos=3999),
        # A host that records op after op, like the reference's own transformer: 7B layer at an odd position.
        dict(name="layer ops 7b", kind="layer", qtype="q4_k", dim=4096, hidden=11008, heads=32, kv_mul=1, seq_len=768, pos=611),
        # Tiny f32 decoder, short prompt, 128 greedy steps: launches and latency, hardly any bytes.
        dict(name="decode tiny f32", kind="model", arch="llama", qtype="f32", dim=288, hidden=768, layers=6, heads=6, kv_mul=1,
             vocab=32000, seq_len=256, start=0, prompt=8, gen=128, prefill=False, temperature=0.0, topp=0.0),
        # GPT-2 124M in Q8_0: 64-token prompt, then greedy generation.
        dict(name="decode gpt2 q8_0", kind="model", arch="gpt2", qtype="q8_0", dim=768, hidden=3072, layers=12, heads=12, kv_mul=1,
             vocab=50257, seq_len=1024, start=0, prompt=64, gen=128, prefill=True, temperature=0.0, topp=0.0),
        # The headline: a 7B Q4_K_M-style model continuing a conversation after 512 positions.
        dict(name="decode 7b q4_k_m", kind="model", arch="llama", qtype="q4_k_m", dim=4096, hidden=11008, layers=32, heads=32, kv_mul=1,
             vocab=32000, seq_len=768, start=512, prompt=1, gen=48, prefill=True, temperature=0.0, topp=0.0),
        # Chat in full: ragged prompt, then a sampled answer; Qwen2 variant (Neox RoPE, biases, grouped queries).
        dict(name="chat qwen2 q8_0 sampled", kind="model", arch="qwen2", qtype="q8_0", dim=2048, hidden=5632, layers=12, heads=16, kv_mul=4,
             vocab=32000, seq_len=512, start=0, prompt=45, gen=32, prefill=True, temperature=0.8, topp=0.9),
        # Time to the first token of the 7B model on its 512-token prompt.
        dict(name="prompt 7b 512", kind="model", arch="llama", qtype="q4_k_m", dim=4096, hidden=11008, layers=32, heads=32, kv_mul=1,
             vocab=32000, seq_len=768, start=0, prompt=512, gen=1, prefill=True, temperature=0.0, topp=0.0),
        # Long prompt through layers of the 70B widths (grouped queries), two of its layers.
        dict(name="prompt 70b-wide 2047", kind="model", arch="llama", qtype="q4_k", dim=8192, hidden=28672, layers=2, heads=64, kv_mul=8,
             vocab=32000, seq_len=4224, start=0, prompt=2047, gen=1, prefill=True, temperature=0.0, topp=0.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["gemv", "gemm", "attention", "layer", "model"], [3, 2, 2, 1, 6])[0]
    if kind == "gemv":
        qtype = rng.choices(["q4_k", "q6_k", "q8_0", "f32", "f16", "q5_k", "q4_0"], [4, 3, 3, 2, 1, 1, 1])[0]
        return dict(kind=kind, qtype=qtype, nrows=_log(rng, 512, 50257), ncols=256 * _log(rng, 2, 44))
    if kind == "gemm":
        return dict(kind=kind, qtype=rng.choice(["q4_k", "q6_k", "q8_0"]), nrows=128 * _log(rng, 4, 250), ncols=256 * _log(rng, 2, 44),
                    nvec=rng.randint(1, 8))
    if kind == "attention":
        head_size, kv_mul = rng.choice([64, 80, 128]), rng.choice([1, 1, 2, 4, 8])
        seq_len = _log(rng, 256, 8192)
        return dict(kind=kind, heads=kv_mul * rng.choice([4, 8, 12, 32 // kv_mul]), kv_mul=kv_mul, head_size=head_size, seq_len=seq_len,
                    pos=_log(rng, 16, seq_len) - 1)
    if kind == "layer":
        dim, kv_mul = rng.choice([1024, 2048, 3072, 4096]), rng.choice([1, 4])
        return dict(kind=kind, qtype=rng.choice(["q4_k", "q6_k", "q8_0"]), dim=dim, hidden=256 * round(dim * rng.uniform(2.5, 3.5) / 256),
                    heads=dim // 128, kv_mul=kv_mul, seq_len=1024, pos=_log(rng, 8, 1024) - 1)
    arch = rng.choice(["llama", "llama", "qwen2", "gpt2"])
    if arch == "gpt2":
        heads = rng.choice([8, 12, 16, 20])
        dim = 64 * heads
        hidden, kv_mul, qtype = 4 * dim, 1, "q8_0"
    else:
        dim = rng.choice([512, 768, 1024, 2048, 3072, 4096, 5120])
        kv_mul = rng.choice([1, 2, 4])
        heads = dim // (64 if dim < 2048 else 128)
        kv_mul = kv_mul if heads % kv_mul == 0 else 1
        hidden = 256 * max(2, round(dim * rng.uniform(2.5, 3.6) / 256))
        qtype = rng.choice(["q4_k_m", "q4_k", "q6_k", "q8_0"] + (["f32"] if dim < 1024 else []))
    layers = max(1, min(_log(rng, 2, 24), int(6e8 / (4 * dim * dim + 3 * dim * hidden))))
    prompt = _log(rng, 1, 1500 if qtype != "f32" else 64)
    gen = _log(rng, 1, 96)
    while layers * (prompt / 8 + gen) > 2500:      # bounds a pass to a fraction of a second
        prompt, gen = max(1, prompt * 3 // 4), max(1, gen * 3 // 4)
    sampled = rng.random() < 0.25
    return dict(kind=kind, arch=arch, qtype=qtype, dim=dim, hidden=hidden, layers=layers, heads=heads, kv_mul=kv_mul,
                vocab=_log(rng, 4000, 50257), seq_len=prompt + gen + rng.choice([0, 7, 512]), start=0, prompt=prompt, gen=gen,
                prefill=dim % 256 == 0 and hidden % 256 == 0 and qtype != "f32", temperature=0.8 if sampled else 0.0, topp=0.9 if sampled else 0.0)


# ---- inputs ------------------------------------------------------------------------------------------------------

def _blocks(qtype, nblocks, sd, rng):
    """`nblocks` random GGUF blocks as rows of bytes, their values of standard deviation ~sd (F32 / F16: raw values)."""
    if qtype in (F32, F16):
        v = rng.standard_normal((nblocks, 1), dtype=np.float32) * np.float32(sd)
        return v.astype(np.float16 if qtype == F16 else np.float32).view(np.uint8)
    size = ops.BLOCK_BYTES[qtype]
    raw = np.frombuffer(bytearray(rng.bytes(nblocks * size)), dtype=np.uint8).reshape(nblocks, size)
    d = ((rng.random(nblocks, dtype=np.float32) + np.float32(0.5)) * np.float32(sd / SPREAD[qtype] / 1.04)).astype(np.float16)
    at = SCALE_AT[qtype]
    raw[:, at:at + 2] = d.view(np.uint8).reshape(nblocks, 2)
    if qtype in DMIN:
        raw[:, 2:4] = (d.astype(np.float32) * np.float32(DMIN[qtype])).astype(np.float16).view(np.uint8).reshape(nblocks, 2)
    return raw


def _matrix(qtype, nrows, ncols, rng, gain=1.0):
    return _blocks(qtype, nrows * (ncols // ops.BLOCK_LEN[qtype]), gain / math.sqrt(ncols), rng).reshape(-1)


class _Weights:
    """Matrices of one model: windows into one run of random blocks per format and width (drawing every byte of a 7B
    model afresh would take longer than everything that is timed)."""

    def __init__(self, rng, largest):
        self.rng, self.largest, self.pools, self.n = rng, largest, {}, 0

    def matrix(self, qtype, nrows, ncols, gain=1.0, spread=0.0):
        bpr = ncols // ops.BLOCK_LEN[qtype]
        key = (qtype, ncols, gain)
        if key not in self.pools:
            self.pools[key] = _blocks(qtype, (self.largest[ncols] * 5 // 4 + 1) * bpr, gain / math.sqrt(ncols), self.rng)
        pool = self.pools[key]
        self.n += 1
        at = (self.n * 7919 * bpr) % (pool.shape[0] - nrows * bpr + 1)
        w = pool[at:at + nrows * bpr]
        if spread:   # rows of differing norms, as a trained head has them
            f = np.exp(self.rng.standard_normal(nrows, dtype=np.float32) * np.float32(spread))
            w = w.copy()
            if qtype == F32:
                w.view(np.float32).reshape(nrows, bpr)[:] *= f[:, None]
            else:
                for off in (SCALE_AT[qtype],) + ((2,) if qtype in DMIN else ()):
                    d = np.ascontiguousarray(w[:, off:off + 2]).view(np.float16).reshape(nrows, bpr)
                    w[:, off:off + 2] = (d.astype(np.float32) * f[:, None]).astype(np.float16).view(np.uint8).reshape(nrows * bpr, 2)
        return qtype, w.reshape(-1)

    def vector(self, n, mean=0.0):
        return F32, np.float32(mean) + self.rng.standard_normal(n, dtype=np.float32) * np.float32(0.05)


def _formats(case, layer):
    """Formats of (a layer's matrices, its ffn_down, token embedding, output head)."""
    if case["qtype"] == "q4_k_m":
        return Q4_K, Q6_K if layer % 2 == 0 else Q4_K, Q4_K, Q6_K
    q = QTYPE[case["qtype"]]
    return q, q, q, q


def _model(case, rng):
    dim, hid, vocab, nl = case["dim"], case["hidden"], case["vocab"], case["layers"]
    t = {}
    if case["arch"] == "gpt2":
        w = _Weights(rng, {dim: max(vocab, hid, 3 * dim), hid: dim})
        q = QTYPE[case["qtype"]]
        for l in range(nl):
            p = f"blk.{l}."
            for nm, r, c, g in (("attn_qkv", 3 * dim, dim, 1.0), ("attn_output", dim, dim, 0.5), ("ffn_up", hid, dim, 1.0), ("ffn_down", dim, hid, 0.5)):
                t[p + nm + ".weight"] = w.matrix(q, r, c, g)
                t[p + nm + ".bias"] = w.vector(r)
            for nm in ("attn_norm", "ffn_norm"):
                t[p + nm + ".weight"], t[p + nm + ".bias"] = w.vector(dim, 1.0), w.vector(dim)
        t["token_embd.weight"] = w.matrix(q, vocab, dim, 1.0, spread=0.5)
        t["position_embd.weight"] = F32, w.rng.standard_normal(case["seq_len"] * dim, dtype=np.float32) * np.float32(0.02)
        t["output_norm.weight"], t["output_norm.bias"] = w.vector(dim, 1.0), w.vector(dim)
        m = Gpt2(Gpt2Params(n_vocab=vocab, n_seq=case["seq_len"], n_embd=dim, n_head=case["heads"], n_layer=nl, ff_len=hid, attn_b=3 * dim))
    else:
        kv = dim // case["kv_mul"]
        w = _Weights(rng, {dim: max(vocab, hid, dim), hid: dim})
        for l in range(nl):
            p = f"blk.{l}."
            q, qd, qe, qo = _formats(case, l)
            for nm, r, g in (("attn_q", dim, 1.0), ("attn_k", kv, 1.0), ("attn_v", kv, 1.0), ("attn_output", dim, 0.5),
                             ("ffn_gate", hid, 1.0), ("ffn_up", hid, 1.0)):
                t[p + nm + ".weight"] = w.matrix(q, r, dim, g)
            t[p + "ffn_down.weight"] = w.matrix(qd, dim, hid, 0.5)
            t[p + "attn_norm.weight"], t[p + "ffn_norm.weight"] = w.vector(dim, 1.0), w.vector(dim, 1.0)
            if case["arch"] == "qwen2":
                for nm, r in (("attn_q", dim), ("attn_k", kv), ("attn_v", kv)):
                    t[p + nm + ".bias"] = w.vector(r)
        t["token_embd.weight"] = w.matrix(qe, vocab, dim, 0.3 * math.sqrt(dim))
        t["output.weight"] = w.matrix(qo, vocab, dim, 1.0, spread=0.5)
        t["output_norm.weight"] = w.vector(dim, 1.0)
        m = Llama2(Llama2Config(dim, hid, nl, case["heads"], case["heads"] // case["kv_mul"], vocab, case["seq_len"], 10000.0, 1e-5),
                   LlamaModelType.Qwen2 if case["arch"] == "qwen2" else LlamaModelType.Llama)
    m.load_tensors(t)
    return m


def _gpu(rng, *shape, sd=1.0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(rng.integers(1 << 62)))
    return torch.randn(*shape, device="cuda", generator=g) * sd


def prepare(case, seed):
    rng = np.random.Generator(np.random.SFC64(seed))
    kind = case["kind"]
    if kind == "gemv":
        q, n, k = QTYPE[case["qtype"]], case["nrows"], case["ncols"]
        return dict(case=case, op=ops.GemvQuant.from_device(), m=ops.GpuQuantMatrix(q, _matrix(q, n, k, rng), n, k), v=_gpu(rng, k),
                    out=torch.zeros(n, device="cuda"))
    if kind == "gemm":
        q, n, k = QTYPE[case["qtype"]], case["nrows"], case["ncols"]
        cls = {Q4_K: ops.Q4KTiles, Q6_K: ops.Q6KTiles, Q8_0: ops.Q80Tiles}[q]
        return dict(case=case, m=cls(_matrix(q, n, k, rng), n, k), v=_gpu(rng, case["nvec"], k), out=torch.zeros(case["nvec"], n, device="cuda"))
    if kind == "attention":
        h, hs, kv_dim = case["heads"], case["head_size"], case["heads"] // case["kv_mul"] * case["head_size"]
        return dict(case=case, op=ops.BatchedMultiqueryAttention.from_device(),
                    params=ops.BatchedMultiqueryAttentionParams(case["seq_len"], kv_dim, case["kv_mul"], h, hs, case["pos"]),
                    q=_gpu(rng, h * hs), k=_gpu(rng, case["seq_len"], kv_dim), v=_gpu(rng, case["seq_len"], kv_dim),
                    out=torch.zeros(h * hs, device="cuda"))
    if kind == "layer":
        return _prepare_layer(case, rng)
    m = _model(case, rng)
    if case["prefill"]:
        m.set_prefill(True)
    if case["start"]:   # the conversation so far
        m.decode(rng.integers(0, case["vocab"], size=case["start"] + 1, dtype=np.uint32), 0)
    if case["temperature"]:
        m.set_sampler(case["temperature"], case["topp"], seed)
    return dict(case=case, m=m, prompt=rng.integers(0, case["vocab"], size=case["prompt"], dtype=np.uint32))


def _prepare_layer(case, rng):
    dim, hid, kv = case["dim"], case["hidden"], case["dim"] // case["kv_mul"]
    q = QTYPE[case["qtype"]]

    def mat(n, k, gain=1.0):
        return ops.GpuQuantMatrix(q, _matrix(q, n, k, rng, gain), n, k)

    def buf(n):
        return torch.zeros(n, device="cuda")

    dev = None
    return dict(
        case=case, rms=ops.RmsNorm.from_device(dev), gemv=ops.GemvQuant.from_device(dev), rope=ops.RoPE.from_device(dev),
        attn=ops.BatchedMultiqueryAttention.from_device(dev), silu=ops.Silu.from_device(dev), add=ops.OpAssign.new(dev, ops.OpAssignVariant.Add),
        norm=ops.RmsNormConfig(1e-5), rope_cfg=ops.RoPEConfig(dim // case["heads"], kv, case["pos"], 10000.0),
        params=ops.BatchedMultiqueryAttentionParams(case["seq_len"], kv, case["kv_mul"], case["heads"], dim // case["heads"], case["pos"]),
        wq=mat(dim, dim), wk=mat(kv, dim), wv=mat(kv, dim), wo=mat(dim, dim, 0.5), w1=mat(hid, dim), w3=mat(hid, dim), w2=mat(dim, hid, 0.5),
        n1=1.0 + _gpu(rng, dim, sd=0.05), n2=1.0 + _gpu(rng, dim, sd=0.05), k=_gpu(rng, case["seq_len"], kv), v=_gpu(rng, case["seq_len"], kv),
        x0=_gpu(rng, dim), x=buf(dim), xb=buf(dim), xb2=buf(dim), q=buf(dim), h1=buf(hid), h2=buf(hid))


# ---- one pass ----------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "gemv":
        s["op"].dispatch(s["out"], s["m"], s["v"])
        return s["out"]
    if kind == "gemm":
        s["m"].gemm(s["out"], s["v"])
        return s["out"]
    if kind == "attention":
        s["op"].dispatch(s["params"], s["q"], s["k"], s["v"], None, s["out"])
        return s["out"]
    if kind == "layer":
        return _run_layer(s)
    m = s["m"]
    tokens = m.decode(s["prompt"], case["gen"], case["start"])
    # copies, as the views live no longer than the model
    out = {"tokens": tokens, "logits": m.logits().clone()}
    if case["prompt"] > 8:   # the rows that the prompt left in the last layer's cache
        n = case["prompt"] - 1
        out["keys"], out["values"] = (cache(case["layers"] - 1)[:n].clone() for cache in (m.key_cache, m.value_cache))
    return out


def _run_layer(s):
    pos, gemv, x, xb, xb2 = s["case"]["pos"], s["gemv"], s["x"], s["xb"], s["xb2"]
    kc, vc = s["k"][pos], s["v"][pos]
    x.copy_(s["x0"])
    s["rms"].dispatch(s["norm"], xb, x, s["n1"])
    gemv.dispatch(s["q"], s["wq"], xb)
    gemv.dispatch(kc, s["wk"], xb)
    gemv.dispatch(vc, s["wv"], xb)
    s["rope"].dispatch(ops.RoPEVariant.Original, s["rope_cfg"], s["q"], kc)
    s["attn"].dispatch(s["params"], s["q"], s["k"], s["v"], None, xb)
    gemv.dispatch(xb2, s["wo"], xb)
    s["add"].dispatch(x, xb2)
    s["rms"].dispatch(s["norm"], xb, x, s["n2"])
    gemv.dispatch(s["h1"], s["w1"], xb)
    gemv.dispatch(s["h2"], s["w3"], xb)
    s["silu"].dispatch(s["h1"], s["h2"])
    gemv.dispatch(xb2, s["w2"], s["h1"])
    s["add"].dispatch(x, xb2)
    return {"x": x, "k": kc, "v": vc}


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def _bytes(qtype, n, k):
    return n * k * ops.BLOCK_BYTES[qtype] / ops.BLOCK_LEN[qtype]


def work(case):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        n, k, m = case["nrows"], case["ncols"], case.get("nvec", 1)
        return {"bytes": _bytes(QTYPE[case["qtype"]], n, k) + 4 * m * (n + k), "flops": 2.0 * m * n * k}
    if kind == "attention":
        rows, h, hs = case["pos"] + 1, case["heads"], case["head_size"]
        return {"bytes": 8.0 * rows * h // case["kv_mul"] * hs + 8 * h * hs, "flops": 4.0 * rows * h * hs}
    dim, hid, kv = case["dim"], case["hidden"], case["dim"] // case["kv_mul"]
    if kind == "layer":
        q, rows = QTYPE[case["qtype"]], case["pos"] + 1
        par = 2 * dim * dim + 2 * kv * dim + 3 * hid * dim
        return {"bytes": _bytes(q, par, 1) + 8.0 * rows * kv + 4.0 * (4 * dim + 2 * kv), "flops": 2.0 * par + 4.0 * rows * dim}
    layer_bytes, layer_params = 0.0, 0
    gpt2 = case["arch"] == "gpt2"
    for l in range(case["layers"]):
        q, qd, _, qo = _formats(case, l)
        up = hid if gpt2 else 2 * hid
        layer_bytes += _bytes(q, 2 * dim + 2 * kv + up, dim) + _bytes(qd, dim, hid)
        layer_params += (2 * dim + 2 * kv + up + hid) * dim
    head = _bytes(qo, case["vocab"], dim)
    n0, n, g, nl = case["start"], case["prompt"] - 1, case["gen"], case["layers"]
    # the prompt's rows can share one read of the weights and of the cache; every generated id needs its own
    rows_read = sum(n0 + n + i for i in range(g)) + (n0 if n else 0)
    seen = n * n0 + n * (n + 1) / 2 + sum(n0 + n + i + 1 for i in range(g))
    return {"bytes": layer_bytes * (g + (1 if n else 0)) + head * g + 8.0 * nl * kv * (rows_read + n + g) + 4.0 * case["vocab"],
            "flops": 2.0 * layer_params * (n + g) + 2.0 * g * case["vocab"] * dim + 4.0 * nl * dim * seen}


def tolerance(case):
    # All arithmetic is f32 or its equivalent.  Measured: a product or an attention against the same sums in 64 bits 5e-7
    # (largest element 2.3e-6), a 32-layer model against its own op-by-op schedule 2.5e-6 (1.9e-5); depth adds up.
    if case["kind"] != "model":
        return {"rel": 3e-6, "max": 3e-5}
    return {"rel": 1.5e-5, "max": 2e-4, "differ": 0.01}
