"""Prompt attention on tcgen05 (csrc/prefill_attn_tc.cu) against fp64 softmax attention at the edges of its tiles: row counts around 64 and 128,
both head sizes, grouped heads, batches, cached prefixes, windows with kept first keys, and infinities in keys and values that a row does
not see.  P and the result are bf16: 2-norm error below 2⁻⁸ of the result's, each element within 2⁻⁷ of the largest |V|."""
import pytest
import torch

from tinygpt_b200 import engine, models, ops, stack_bench

pytestmark = pytest.mark.gpu
DEV = "cuda"


def randn(*shape, seed, std=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * std).to(torch.bfloat16)


def attend(q, k, v):
    """fp64, key by key visible only: masked keys never meet V."""
    n, group = q.shape[1], q.shape[2] // k.shape[2]
    k, v = k.double().repeat_interleave(group, 2), v.double().repeat_interleave(group, 2)
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k) * q.shape[-1] ** -0.5
    s = s.masked_fill(~torch.ones(n, n, dtype=torch.bool, device=DEV).tril(), float("-inf"))
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v)


def close(got, want, vmax):
    e = got.double() - want
    assert float(e.norm() / want.norm()) < 2.0 ** -8
    assert float(e.abs().max()) <= 2.0 ** -7 * vmax


@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(1, 1, 2, 1, 64), (2, 2, 2, 2, 128), (1, 63, 4, 2, 128), (1, 64, 3, 1, 64), (2, 65, 4, 4, 128), (1, 127, 7, 1, 64),
                                          (1, 128, 2, 2, 128), (3, 129, 4, 2, 64), (1, 191, 2, 1, 128), (2, 321, 6, 2, 64), (1, 700, 4, 1, 128)])
def test_causal(built_lib, monkeypatch, B, S, Hq, Hkv, D):
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    q, k, v = randn(B, S, Hq, D, seed=1, std=2.0), randn(B, S, Hkv, D, seed=2), randn(B, S, Hkv, D, seed=3)
    got = ops.flash_attention(q, k, v, True)
    close(got, attend(q, k, v), float(v.float().abs().max()))
    assert torch.equal(got, ops.flash_attention(q, k, v, True))


@pytest.mark.parametrize("S", [65, 129, 150, 192, 256, 321, 449])
@pytest.mark.parametrize("D", [64, 128])
def test_last_tile_sees_part_of_the_block(built_lib, monkeypatch, S, D):
    """The result is read after the products of a block's last tiles, also where no warp has waited for them to rescale: maxima in the first tile; last tiles of one key, of
    half of them and of all; up to eleven blocks to a CTA, the next of which is under way while one is stored."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    q, k, v = randn(4, S, 96, D, seed=11), randn(4, S, 96, D, seed=12), randn(4, S, 96, D, seed=13)
    q, k[:, 0] = q.abs(), 6.0 * D ** -0.5   # key 0: a score of about five, the others' stay below four
    want = attend(q, k, v)
    first = ops.flash_attention(q, k, v, True)
    close(first, want, float(v.float().abs().max()))
    for _ in range(20):
        assert torch.equal(ops.flash_attention(q, k, v, True), first)


@pytest.mark.parametrize("D", [64, 128])
def test_what_a_row_does_not_see(built_lib, monkeypatch, D):
    """Rows in front of an infinity, a NaN, or a huge key keep finite, correct results; a batch's next sequence keeps its own."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    S, at = 200, 100
    q, k, v = randn(2, S, 4, D, seed=4), randn(2, S, 2, D, seed=5), randn(2, S, 2, D, seed=6)
    want = attend(q, k, v)
    v2, k2 = v.clone(), k.clone()
    v2[0, at], v2[0, at + 50] = float("inf"), float("nan")
    k2[0, at] = float("nan")
    got = ops.flash_attention(q, k2, v2, True)
    close(got[0, :at], want[0, :at], float(v.float().abs().max()))
    close(got[1], want[1], float(v.float().abs().max()))
    assert not bool(torch.isfinite(got[0, at + 50:].float()).any())


def test_growing_maxima(built_lib, monkeypatch):
    """Scores that grow by hundreds from tile to tile (every tile rescales) and ones that only fall."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    S, D = 400, 64
    q = torch.ones(1, S, 2, D, device=DEV, dtype=torch.bfloat16)
    ramp = torch.arange(S, device=DEV, dtype=torch.float32).view(1, S, 1, 1)
    v = randn(1, S, 2, D, seed=7)
    for sign in (0.5, -0.5):
        k = (sign * ramp).expand(1, S, 2, D).to(torch.bfloat16).contiguous()
        close(ops.flash_attention(q, k, v, True), attend(q, k, v), float(v.float().abs().max()))


@pytest.mark.parametrize("window,keep", [(0, 0), (70, 0), (130, 5), (64, 64), (1, 0)])
@pytest.mark.parametrize("dim", [64, 128])
def test_window_prefix_and_gate(built_lib, monkeypatch, window, keep, dim):
    """Through a layer-stack engine: a prompt in two portions (cached prefix), windows with kept first keys, the per-head gate — against
    the mma.sync kernel, to the bf16 roundings of the two kernels' P and sums."""
    attn = models.AttnSpec(4, 2, dim, dim, dim ** -0.5, window, keep)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=500, layers=(models.StackLayerSpec(attn, 128),) * 2,
                            embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=512, max_slots=1)
    eng = engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device(DEV), 8))
    toks = torch.randint(0, 500, (1, 400), generator=torch.Generator().manual_seed(9)).to(DEV)
    out = {}
    for side in ("tc", "mma"):
        monkeypatch.setenv("B200_ATTN_TC", side)
        eng.reset_cache()
        out[side] = torch.cat([eng.forward(toks[:, :150].contiguous(), True), eng.forward(toks[:, 150:].contiguous(), True)], 1).double()
    assert float((out["tc"] - out["mma"]).norm() / out["mma"].norm()) < 1e-2
    eng.close()
