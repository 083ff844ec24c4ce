"""Decode attention against BatchedMultiqueryAttention::run_cpu (oracle), incl. grouped-query heads,
which the reference never tests."""
import numpy as np
import pytest
import torch

import oracle
from conftest import ATOL, RTOL, assert_close
from helpers import attention_kernel
from wgml_b200 import ops

pytestmark = pytest.mark.gpu


def run(seq_len, n_heads, hs, kv_mul, pos, want_attn, seed=0):
    rng = np.random.default_rng(seed)
    kv_dim = n_heads // kv_mul * hs
    q = rng.standard_normal(n_heads * hs).astype(np.float32)
    kc = rng.standard_normal((seq_len, kv_dim)).astype(np.float32)
    vc = rng.standard_normal((seq_len, kv_dim)).astype(np.float32)
    p = ops.BatchedMultiqueryAttentionParams(seq_len, kv_dim, kv_mul, n_heads, hs, pos)
    xb = torch.full((n_heads * hs,), float("nan"), device="cuda")
    attn = torch.zeros(n_heads * seq_len, device="cuda") if want_attn else None
    a = ops.BatchedMultiqueryAttention.from_device()
    a.dispatch(p, torch.from_numpy(q).cuda(), torch.from_numpy(kc).cuda(), torch.from_numpy(vc).cuda(), attn, xb)
    exb, eattn = oracle.attention(seq_len, kv_dim, kv_mul, n_heads, hs, pos, q, kc, vc)
    assert_close(xb.cpu().numpy(), exb, RTOL, ATOL, f"xb pos={pos} kv_mul={kv_mul}")
    if want_attn:
        got = attn.cpu().numpy().reshape(n_heads, seq_len)
        assert_close(got[:, : pos + 1], eattn[:, : pos + 1], RTOL, 1e-6, "attention weights")
    return xb


# Every kernel of the stand-alone call, each width (query heads per KV head) of those that have them.  Short contexts are the
# cluster kernel's as long as its blocks are resident, so the others' cases have more heads than that, longer contexts or wider heads.
KERNELS = [
    ("rows", (2112, 32, 128, 1, 2100)), ("rows", (2112, 32, 64, 2, 1700)), ("rows", (512, 264, 64, 4, 300)), ("rows", (512, 264, 64, 8, 300)),
    ("rows", (512, 264, 64, 2, 300)), ("rows", (4224, 64, 128, 8, 4100)),
    ("split", (512, 132, 128, 1, 190)), ("split", (512, 132, 128, 12, 250)), ("split", (512, 12, 256, 1, 300)), ("split", (512, 10, 256, 5, 301)),
    ("split, several chunks a block", (2112, 60, 64, 5, 2100)), ("split, several chunks a block", (512, 132, 256, 1, 400)),
    ("cluster", (512, 32, 128, 1, 300)), ("cluster", (512, 12, 64, 3, 300)), ("cluster", (512, 32, 128, 4, 300)),
]


@pytest.mark.parametrize("kernel,case", KERNELS)
def test_each_kernel(kernel, case):
    """Against the oracle, and again: tickets and scratch are left as the next call needs them."""
    assert attention_kernel(*case) == kernel
    a = run(*case, want_attn=False, seed=7)
    b = run(*case, want_attn=False, seed=7)
    assert torch.equal(a, b)


@pytest.mark.parametrize("want_attn", [True, False])
def test_reference_test_sizes(want_attn):  # ops/batched_multiquery_attention.rs:210-413
    for pos in list(range(9)):
        run(1024, 12, 64, 1, pos, want_attn, seed=pos)


@pytest.mark.parametrize("case", [
    (256, 6, 48, 1, 255), (768, 32, 128, 1, 600), (4224, 64, 128, 8, 4100), (1024, 12, 64, 1, 1023),
    (512, 12, 64, 3, 130), (512, 16, 32, 2, 63), (512, 16, 32, 2, 64), (512, 10, 256, 5, 77), (128, 4, 4, 4, 100)])
def test_split_kernel_shapes(case):   # (most of them short contexts of few heads: now the cluster kernel's)
    run(*case, want_attn=False, seed=1)


@pytest.mark.parametrize("case", [
    (4224, 32, 128, 1, 4100),    # 7B heads, long context: four blocks per KV head
    (4224, 32, 128, 1, 4095),    # last group of eight rows exactly full
    (4224, 32, 128, 4, 4100),    # four query heads per KV head
    (4224, 32, 128, 2, 2049),    # two, last group of two rows
    (4224, 40, 128, 5, 3000),    # five query heads per KV head: split kernel, two groups of four (tail masked)
    (4224, 96, 128, 12, 1500),   # twelve: split kernel, three groups of four
    (512, 264, 64, 8, 64), (512, 264, 64, 8, 71),    # row-streaming kernel: nine groups over four blocks a KV head, one row in the last and full
    (512, 144, 128, 8, 130),     # seventeen groups over eight blocks a KV head
    (8256, 64, 64, 8, 8200),     # head size 64: half of the lanes idle
    (8256, 24, 96, 1, 5000),     # head size 96
    (4224, 64, 128, 8, 2047), (4224, 64, 128, 8, 2048),   # last group full, one row in it
    (4224, 64, 128, 8, 1300),    # cluster kernel, as the four below
    (8256, 32, 96, 4, 7001),     # four heads per KV head, a quarter of the lanes idle
    (4224, 64, 128, 8, 0),
    (4224, 64, 128, 8, 63), (4224, 64, 128, 8, 64), (4224, 64, 128, 8, 130),
])
def test_streaming_kernel_shapes(case):
    """Stand-alone calls on long contexts or with many query heads per KV head: the row-streaming kernel (one, two, four or
    eight query heads per KV head) or the split kernel with several chunks per block, up to 1536 positions also the cluster kernel.  (The streaming kernel proper wants the rows
    of a head side by side, as the models' caches have them: test_gpu_decode_attention.py.)"""
    run(*case, want_attn=False, seed=3)


def test_repeated_calls_reuse_the_ticket_counters():   # (cluster kernel, which has none; the others: test_each_kernel)
    a = run(512, 8, 64, 2, 300, False, seed=2)
    b = run(512, 8, 64, 2, 300, False, seed=2)
    assert torch.equal(a, b)


def test_repeated_streaming_calls_reuse_the_ticket_counters():   # row-streaming kernel
    a = run(4224, 64, 128, 8, 4100, False, seed=4)
    b = run(4224, 64, 128, 8, 4100, False, seed=4)
    assert torch.equal(a, b)


@pytest.mark.parametrize("case", [
    (512, 32, 64, 2, 300), (512, 12, 64, 3, 130),   # cluster kernel
] + [case for _, case in KERNELS])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_output_at_any_word(case, offset):
    """`xb` may start at any float: only q and the caches are read sixteen bytes at a time.  Same bits, nothing beside it."""
    seq_len, n_heads, hs, kv_mul, pos = case
    g = torch.Generator(device="cuda").manual_seed(5)
    kv_dim, n = n_heads // kv_mul * hs, n_heads * hs
    q, k, v = (torch.randn(*s, device="cuda", generator=g) for s in ((n,), (seq_len, kv_dim), (seq_len, kv_dim)))
    p, a = ops.BatchedMultiqueryAttentionParams(seq_len, kv_dim, kv_mul, n_heads, hs, pos), ops.BatchedMultiqueryAttention.from_device()
    exp, buf = torch.empty(n, device="cuda"), torch.full((n + 8,), 7.0, device="cuda")
    a.dispatch(p, q, k, v, None, exp)
    a.dispatch(p, q, k, v, None, buf[offset:offset + n])
    assert torch.equal(buf[offset:offset + n], exp)
    assert (buf[:offset] == 7.0).all() and (buf[offset + n:] == 7.0).all()


@pytest.mark.parametrize("case", [
    (512, 32, 64, 2, 300), (4224, 64, 128, 8, 1300),   # cluster kernel
] + [case for _, case in KERNELS])
@pytest.mark.parametrize("masked", [(0, 8), (0, 23), (0, 130), (8, 16), (40, 290), (1, 297)])
def test_rows_scored_minus_infinity_weigh_nothing(case, masked):
    """Cache rows a host has masked with keys of -inf (left padding): whole groups, warps and blocks of the row-streaming
    kernel and chunks of the split kernel see nothing but -inf, and the answer is that of the other rows (RTOL / ATOL as everywhere)."""
    seq_len, n_heads, hs, kv_mul, pos = case
    rng = np.random.default_rng(9)
    n_kv = n_heads // kv_mul
    q, k, v = (rng.standard_normal(s).astype(np.float32) for s in ((n_heads, hs), (seq_len, n_kv, hs), (seq_len, n_kv, hs)))
    q[:, 0] = np.abs(q[:, 0]) + 0.5
    k[masked[0]:masked[1], :, 0] = -np.inf
    p = ops.BatchedMultiqueryAttentionParams(seq_len, n_kv * hs, kv_mul, n_heads, hs, pos)
    xb = torch.full((n_heads * hs,), float("nan"), device="cuda")
    ops.BatchedMultiqueryAttention.from_device().dispatch(p, *(torch.from_numpy(t.reshape(len(t), -1) if t.ndim == 3 else t.ravel()).cuda() for t in (q, k, v)), None, xb)
    keep = np.r_[0:masked[0], masked[1]:pos + 1]
    s = np.einsum("ghd,tgd->ght", q.reshape(n_kv, kv_mul, hs).astype(np.float64), k[keep].astype(np.float64)) / np.sqrt(hs)
    w = np.exp(s - s.max(-1, keepdims=True))
    exp = np.einsum("ght,tgd->ghd", w / w.sum(-1, keepdims=True), v[keep].astype(np.float64))
    assert_close(xb.cpu().numpy(), exp.ravel(), RTOL, ATOL, f"rows {masked} masked")


def test_parameter_checks():
    a = ops.BatchedMultiqueryAttention.from_device()
    z = torch.zeros(64 * 128, device="cuda")
    with pytest.raises(ops.WgbError):
        a.dispatch(ops.BatchedMultiqueryAttentionParams(64, 128, 1, 2, 64, 64), z[:128], z, z, None, z[:128])  # pos == seq_len
    with pytest.raises(ops.WgbError):
        a.dispatch(ops.BatchedMultiqueryAttentionParams(64, 128, 3, 2, 64, 1), z[:128], z, z, None, z[:128])


@pytest.mark.parametrize("hs", [4, 20, 32, 36, 64, 80, 96, 100, 128])
@pytest.mark.parametrize("heads,kv_mul", [(1, 1), (6, 3), (16, 4), (24, 1), (40, 5), (72, 8), (130, 1)])
def test_cluster_kernel_edges(hs, heads, kv_mul):
    """Blocks per head 8, 4, 2 and 1 (and none resident: heads of more than 64 elements, 130 of them), head sizes around a lane's
    four float4, contexts around a group of eight rows, the warps of one block and of eight, what a warp requests ahead, and the
    lines of the dispatch rule."""
    for pos in (0, 6, 7, 8, 63, 64, 127, 128, 191, 192, 193, 511, 767, 768, 1023, 1024, 1535, 1536):
        run(1600, heads, hs, kv_mul, pos, want_attn=False, seed=pos)


@pytest.mark.parametrize("case", [(512, 132, 128, 1, 300), (512, 132, 96, 2, 300), (512, 132, 128, 3, 200), (512, 264, 64, 4, 130), (512, 260, 32, 1, 200),
                                  (512, 132, 80, 12, 77), (2048, 264, 64, 8, 1700)])
def test_more_heads_than_resident_blocks(case):
    """One, two, three, four, eight and twelve query heads per KV head where the cluster kernel leaves more than a chunk to the others."""
    run(*case, want_attn=False, seed=2)


def test_more_heads_than_a_grid_has_rows():
    """Short contexts with more query heads than the second axis of a grid holds (65535), on a quarter as many KV heads."""
    run(8, 65540, 4, 4, 5, want_attn=False, seed=6)


def test_rows_of_a_group_meet_before_the_running_sum():
    """Equal weights, a value of 2^24 in the first row and 1 in the others, one block per head: a lane adds sixteen groups of two rows to
    its running sum, then quarters of a warp (2 additions), warps (8) and the division round; each within half an ulp of 2^24, 1."""
    heads, hs, kv_mul, pos = 96, 128, 4, 1000
    assert attention_kernel(1024, heads, hs, kv_mul, pos) == "cluster"
    kv_dim = heads // kv_mul * hs
    v = torch.ones(1024, kv_dim, device="cuda")
    v[0] = 2.0 ** 24
    xb = torch.zeros(heads * hs, device="cuda")
    ops.BatchedMultiqueryAttention.from_device().dispatch(ops.BatchedMultiqueryAttentionParams(1024, kv_dim, kv_mul, heads, hs, pos),
                                                          torch.ones(heads * hs, device="cuda"), torch.zeros(1024, kv_dim, device="cuda"), v, None, xb)
    n = pos + 1
    err = (xb.double() - (2.0 ** 24 + pos) / n).abs().max().item() * n
    assert err <= 16 + 2 + 8 + 1 + 1, err
