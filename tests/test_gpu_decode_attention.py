"""Attention of the decode step (position on the device, head-major caches, programmatic launches) at contexts and groupings
that the model tests do not reach: the cluster kernel (short contexts), the streaming kernel (one or two query heads per KV head, more chunks of 64 rows than
the split kernel's blocks fit in one wave) and the row-streaming kernel (four or eight) with and without its requests
ahead of the wait for the launch before.  The caches are filled on both sides with the same rows, then a few greedy
steps run against the oracle."""
import numpy as np
import pytest
import torch

from conftest import ATOL, RTOL, assert_close
from helpers import SMALL_LLAMA, attention_kernel, llama_pair
from wgml_b200 import _lib, synth
from wgml_b200.models import _device_view

pytestmark = pytest.mark.gpu


def steps(heads, kv_heads, head_size, start, gen, seq_len, seed=3, kernel=None):
    if kernel:
        assert attention_kernel(seq_len, heads, head_size, heads // kv_heads, start + gen - 1, decode=True) == kernel
    cfg = dict(SMALL_LLAMA, dim=heads * head_size, hidden_dim=512, n_layers=1, n_q_heads=heads, n_kv_heads=kv_heads, vocab_size=300, seq_len=seq_len)
    t = synth.llama_tensors(cfg, seed, scale=0.002)
    rng = np.random.default_rng(seed)
    # a faint embedding: the residual stream, hence the logits, come from the attention
    t["token_embd.weight"] = (synth.F32, rng.standard_normal(300 * cfg["dim"]).astype(np.float32) * np.float32(1e-3))
    gpu, cpu, _ = llama_pair(cfg, tensors=t)
    kv_dim = kv_heads * head_size
    caches = [rng.standard_normal((seq_len, kv_dim)).astype(np.float32) for _ in range(2)]
    lib = _lib.load()
    for rows, host, ptr in zip(caches, cpu.caches(), (lib.wgb_llama2_key_cache(gpu._h, 0), lib.wgb_llama2_value_cache(gpu._h, 0))):
        host[0] = rows
        dev = _device_view(ptr, seq_len * kv_dim).view(kv_heads, seq_len, head_size)
        dev.copy_(torch.from_numpy(rows).cuda().view(seq_len, kv_heads, head_size).permute(1, 0, 2))
    tok = np.array([17], np.uint32)
    exp = cpu.decode(tok, gen, start)[0]
    got = gpu.decode(tok, gen, start)
    assert np.array_equal(got, exp)
    ref = cpu.logits()
    assert_close(gpu.logits().cpu().numpy(), ref, RTOL, ATOL * max(1.0, float(np.abs(ref).max())), f"logits after position {start + gen - 1}")


@pytest.mark.parametrize("shape", [(32, 32, 64), (64, 32, 64), (32, 32, 96)])
@pytest.mark.parametrize("start", [955, 1022, 2100])
def test_streaming_kernel_in_decode_steps(shape, start):
    """Three blocks of the split kernel per SM hold 444 chunks: with 32 KV heads a context of more than 13 chunks is over one wave.
    (Up to 1536 positions of these few heads: the cluster kernel.)"""
    steps(*shape, start, 4, 2176, kernel="stream" if start == 2100 else "cluster")


@pytest.mark.parametrize("shape,start,gen", [
    ((320, 320, 8), 0, 140), ((320, 160, 8), 0, 300),                               # from the first position on
    ((320, 320, 8), 955, 4), ((320, 160, 8), 955, 4), ((288, 144, 16), 955, 4),
    ((320, 320, 8), 1022, 4), ((320, 160, 8), 1022, 4), ((288, 144, 16), 1022, 4),  # a chunk fills up and the next one begins
])
def test_streaming_kernel_of_many_heads_in_decode_steps(shape, start, gen):
    """More heads than resident blocks of the cluster kernel; from position 0 on, in launches sized for the call's last position: most
    blocks have no rows at first."""
    steps(*shape, start, gen, 1100, kernel="stream")


def test_streaming_kernel_with_several_chunks_per_block():
    steps(32, 32, 128, 4090, 8, 4160)


@pytest.mark.parametrize("shape", [(32, 8, 64), (32, 4, 64), (16, 4, 128), (32, 4, 128), (40, 5, 64)])
@pytest.mark.parametrize("start", [0, 126, 200, 1001, 3003])
def test_row_streaming_kernel_in_decode_steps(shape, start):
    """Ten steps leave every number of rows in the last group of eight.  Up to about 140 positions there are fewer groups
    than blocks, and no warp requests anything ahead of the wait; from 1001 on most do.  (Up to 1536 positions of these few heads: the
    cluster kernel.)"""
    steps(*shape, start, 10, 3072, kernel="rows" if start == 3003 else "cluster")


@pytest.mark.parametrize("shape,start,gen", [
    ((288, 72, 16), 0, 70), ((320, 40, 8), 0, 530),                                 # from the first position on
    ((288, 72, 16), 126, 10), ((288, 72, 16), 1001, 10), ((320, 40, 8), 1001, 10), ((288, 36, 16), 1001, 10),
])
def test_row_streaming_kernel_of_many_heads_in_decode_steps(shape, start, gen):
    """More heads than resident blocks of the cluster kernel: the row-streaming kernel from the first position on, with fewer groups of
    rows than blocks (nothing is requested ahead of the wait) and with more."""
    steps(*shape, start, gen, 1100, kernel="rows")


@pytest.mark.parametrize("shape", [(12, 12, 64), (16, 4, 128), (40, 40, 64), (36, 12, 128), (66, 33, 128)])
@pytest.mark.parametrize("start", [0, 60, 186, 250, 1018, 1530])
def test_cluster_kernel_in_decode_steps(shape, start):
    """Eight, four and two blocks per head and one; ten steps that leave every number of rows in the last group of eight and cross the
    lines of the dispatch rule (192, 1024 and 1536 positions; a call's launches are those of its last position)."""
    steps(*shape, start, 10, 1600)
