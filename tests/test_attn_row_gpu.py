"""One query row through b200_attn_bf16 (csrc/attn.cu attn_row_kernel) against fp64 attention, at the edges of its splits: key counts around a pass, a
cluster's share and several passes, one and two heads per CTA, both head sizes, and the causal form (row 0 sees key 0 only).  Probabilities
are fp32, the result bf16: 2-norm error below 2⁻⁸.  And the fused decode kernel's merge of many splits."""
import ctypes as C

import pytest
import torch

from tinygpt_b200 import engine, models, ops
from tinygpt_b200._lib import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def randn(*shape, seed, std=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * std).to(torch.bfloat16)


def shifted(t):
    """The same values two bytes off a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


def attend(q, k, v):
    group = q.shape[2] // k.shape[2]
    k, v = k.double().repeat_interleave(group, 2), v.double().repeat_interleave(group, 2)
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k) * q.shape[-1] ** -0.5
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 127, 128, 129, 255, 257, 1000, 2049, 5000])
@pytest.mark.parametrize("B,Hq,Hkv,D", [(1, 14, 2, 64), (1, 3, 1, 128), (1, 16, 8, 128), (3, 64, 8, 64), (5, 32, 8, 128)])
def test_one_row(built_lib, n, B, Hq, Hkv, D):
    q, k, v = randn(B, 1, Hq, D, seed=n, std=2.0), randn(B, n, Hkv, D, seed=1), randn(B, n, Hkv, D, seed=2)
    got = ops.flash_attention(q, k, v, False)
    want = attend(q, k, v)
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
    assert torch.equal(got, ops.flash_attention(q, k, v, False))
    first = ops.flash_attention(q, k, v, True)
    assert torch.equal(first, v[:, :1].repeat_interleave(Hq // Hkv, 2))


@pytest.mark.parametrize("which", ["q", "k", "v", "kv", "qkv"])
@pytest.mark.parametrize("n,rows,causal", [(1, 1, False), (300, 1, False), (300, 1, True), (90, 90, True), (90, 90, False), (90, 5, False)])
@pytest.mark.parametrize("D", [64, 128])
def test_views_off_a_16_byte_boundary(built_lib, which, n, rows, causal, D):
    """Contiguous views that start two bytes off give what aligned tensors give."""
    q, k, v = randn(2, rows, 6, D, seed=n, std=2.0), randn(2, n, 2, D, seed=1), randn(2, n, 2, D, seed=2)
    want = ops.flash_attention(q, k, v, causal).double()
    got = ops.flash_attention(shifted(q) if "q" in which else q, shifted(k) if "k" in which else k, shifted(v) if "v" in which else v, causal).double()
    assert float((got - want).norm() / want.norm()) < 2.0 ** -8      # the kernels' order of sums, and P in bf16 in the prompt's


@pytest.mark.parametrize("ctx", [256, 2304])
def test_decode_caches_off_a_16_byte_boundary_are_refused(built_lib, ctx):
    from tinygpt_b200._lib import B200Error
    qkv, cache = randn(10 * 64, seed=1), randn(ctx, 2, 64, seed=2)
    for k, v in ((shifted(cache), cache), (cache, shifted(cache))):
        with pytest.raises(B200Error, match="aligned"):
            ops.attn_decode(qkv, k, v, q_heads=6, kv_heads=2, head_dim=64, fixed_len=9)


def test_huge_scores_and_zeros(built_lib):
    """Scores thousands apart (one key takes all), equal scores, and a row of zeros."""
    q = torch.full((1, 1, 2, 64), 8.0, device=DEV, dtype=torch.bfloat16)
    k, v = randn(1, 700, 1, 64, seed=3, std=20.0), randn(1, 700, 1, 64, seed=4)
    want = attend(q, k, v)
    got = ops.flash_attention(q, k, v, False)
    assert float((got.double() - want).abs().max()) <= 2.0 ** -7 * float(v.float().abs().max())
    flat = ops.flash_attention(q * 0, k, v, False).double()
    assert float((flat - attend(q * 0, k, v)).abs().max()) < 2.0 ** -9


@pytest.mark.parametrize("Hq,Hkv,D,ctxs", [(6, 2, 128, (1024, 1025)), (14, 2, 64, (2048, 2049, 4096))])
@pytest.mark.parametrize("table", [False, True])
def test_fixed_length_does_not_depend_on_the_cache(built_lib, Hq, Hkv, D, ctxs, table):
    """Attention over the first rows of a cache that appends nothing: the same on either side of the context where the cluster kernel
    takes over, q rotated as the last of those rows' tokens if there is a table."""
    n = 700
    qkv = randn((Hq + 2 * Hkv) * D, seed=9, std=1.5)
    kc, vc = randn(max(ctxs), Hkv, D, seed=10), randn(max(ctxs), Hkv, D, seed=11)
    ang = torch.arange(max(ctxs), device=DEV, dtype=torch.float64)[:, None] * (1e4 ** (-torch.arange(0, D, 2, device=DEV, dtype=torch.float64) / D))
    rope = torch.stack([ang.cos().repeat(1, 2), ang.sin().repeat(1, 2)], -1).float().contiguous() if table else None
    q = qkv[:Hq * D].view(Hq, D).float()
    if table:
        c, s = rope[n - 1, :D // 2, 0], rope[n - 1, :D // 2, 1]
        lo, hi = q[:, :D // 2], q[:, D // 2:]
        q = torch.cat([lo * c - hi * s, hi * c + lo * s], 1)
    want = attend(q.to(torch.bfloat16)[None, None], kc[None, :n], vc[None, :n]).reshape(-1)
    for ctx in ctxs:
        got = ops.attn_decode(qkv, kc[:ctx].clone(), vc[:ctx].clone(), q_heads=Hq, kv_heads=Hkv, head_dim=D, fixed_len=n, rope_table=rope)
        assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8, ctx


@pytest.mark.parametrize("Hq,Hkv,D,at", [(6, 2, 128, 1023), (6, 2, 128, 1025), (14, 2, 64, 2400), (24, 8, 128, 4000), (8, 8, 128, 3999)])
def test_fused_decode_merges_many_splits(built_lib, Hq, Hkv, D, at):
    ctx = 4096
    qkv = randn((Hq + 2 * Hkv) * D, seed=5, std=1.5)
    kc, vc = randn(ctx, Hkv, D, seed=6), randn(ctx, Hkv, D, seed=7)
    pos = torch.tensor([at], dtype=torch.int32, device=DEV)
    got = ops.attn_decode(qkv, kc, vc, q_heads=Hq, kv_heads=Hkv, head_dim=D, pos=pos)
    q, k, v = (t.view(1, 1, -1, D) for t in qkv.split([Hq * D, Hkv * D, Hkv * D]))
    want = attend(q, torch.cat([kc[None, :at], k], 1), torch.cat([vc[None, :at], v], 1)).reshape(-1)
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
    assert torch.equal(kc[at], k[0, 0]) and torch.equal(vc[at], v[0, 0])
    assert torch.equal(got, ops.attn_decode(qkv, kc, vc, q_heads=Hq, kv_heads=Hkv, head_dim=D, pos=pos))


@pytest.mark.parametrize("ctx", [256, 4096])
def test_every_launch_of_a_traced_token_has_its_stamps(built_lib, monkeypatch, ctx):
    """b200_engine_debug_trace: entry, end of the dependency wait, operands staged and exit of the GEMV and attention launches, short and long
    contexts alike."""
    monkeypatch.setenv("B200_TRACE", "1")
    spec = models.TINY_QWEN2.with_ctx(ctx)
    eng = engine.DecodeEngine(spec, {k: v.to(DEV) for k, v in models.synth_weights(spec, seed=3).items()})
    eng.forward(torch.arange(20, device=DEV).view(1, -1))
    eng.decode(3)
    torch.cuda.synchronize()
    n = 5 * spec.layers + 1
    buf = (C.c_uint64 * (8 * n))()
    assert lib().b200_engine_debug_trace(eng._h, buf, n) == n
    for launch in range(n):
        entry, waited, done, staged = buf[8 * launch:8 * launch + 4]
        assert 0 < entry <= waited <= staged <= done, launch
    eng.close()
