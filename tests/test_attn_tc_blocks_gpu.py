"""Prompt attention on tcgen05 (csrc/prefill_attn_tc.cu) where its work is shared out: the kernel for up to 128 keys and the one that runs through blocks of
rows, each against fp64 at the edges of its tiles; CTAs with several blocks whose groups of warps have no tile for a while; maxima that grow a
little and a lot with every tile; windows whose kept and recent tiles fall to the same group; and portions of a prompt that change from
one kernel to the other.  P and the result are bf16 (2-norm error below 2⁻⁸ of the result's, each element within 2⁻⁷ of the
largest |V|)."""
import pytest
import torch

from test_attn_tc_gpu import DEV, attend, close, randn
from tinygpt_b200 import engine, models, ops, stack_bench

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [2, 15, 16, 17, 31, 32, 33, 48, 63, 96, 97, 127, 128, 129, 255, 256, 257, 384, 385])
@pytest.mark.parametrize("D", [64, 128])
def test_edges(built_lib, monkeypatch, S, D):
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    q, k, v = randn(2, S, 6, D, seed=1, std=2.0), randn(2, S, 2, D, seed=2), randn(2, S, 2, D, seed=3)
    close(ops.flash_attention(q, k, v, True), attend(q, k, v), float(v.float().abs().max()))


@pytest.mark.parametrize("B,S,H", [(5, 128, 120), (4, 129, 150), (3, 300, 110), (2, 513, 60), (1, 1100, 40)])
@pytest.mark.parametrize("D", [64, 128])
def test_many_blocks_per_cta(built_lib, monkeypatch, B, S, H, D):
    """Up to nine blocks to a CTA, with one, two, three … tiles: groups without a tile run ahead of their barriers' phases if nothing holds them."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    q, k, v = randn(B, S, H, D, seed=4, std=2.0), randn(B, S, H // 2, D, seed=5), randn(B, S, H // 2, D, seed=6)
    first = ops.flash_attention(q, k, v, True)
    close(first, attend(q, k, v), float(v.float().abs().max()))
    for _ in range(10):
        assert torch.equal(ops.flash_attention(q, k, v, True), first)


@pytest.mark.parametrize("step", [0.5, 3.0, 7.5, 8.5, 40.0])
@pytest.mark.parametrize("D", [64, 128])
def test_maxima_that_grow_by_a_step_per_tile(built_lib, monkeypatch, D, step):
    """Scores in powers of two: tile t lies t · step above the first, so that every tile rescales O."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    S = 900
    q, k, v = randn(1, S, 2, D, seed=7, std=0.3), randn(1, S, 2, D, seed=8, std=0.3), randn(1, S, 2, D, seed=9)
    q[..., 0] = 8.0
    lift = (torch.arange(S, device=DEV) // 128) * (step * 0.6931 * D ** 0.5 / 8.0)   # bf16: within 2⁻⁸ of it, alike for a whole tile
    k[..., 0] = lift.to(torch.bfloat16)[None, :, None]
    close(ops.flash_attention(q, k, v, True), attend(q, k, v), float(v.float().abs().max()))


@pytest.mark.parametrize("S", [40, 100])
@pytest.mark.parametrize("D", [64, 128])
def test_one_tile_and_what_a_row_does_not_see(built_lib, monkeypatch, S, D):
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    q, k, v = randn(2, S, 4, D, seed=10), randn(2, S, 2, D, seed=11), randn(2, S, 2, D, seed=12)
    want, at = attend(q, k, v), S // 2
    v2, k2 = v.clone(), k.clone()
    v2[0, at], v2[0, at + 5], k2[0, at + 7] = float("inf"), float("nan"), float("nan")
    got = ops.flash_attention(q, k2, v2, True)
    close(got[0, :at], want[0, :at], float(v.float().abs().max()))
    close(got[1], want[1], float(v.float().abs().max()))
    assert not bool(torch.isfinite(got[0, at + 5:].float()).any())


@pytest.mark.parametrize("window,keep", [(0, 0), (100, 130), (300, 3), (257, 260)])
@pytest.mark.parametrize("dim", [64, 128])
def test_portions(built_lib, monkeypatch, window, keep, dim):
    """A prompt in one portion and in portions that begin within 128 keys and end blocks elsewhere: the same bits; and the mma.sync kernel's
    results to the bf16 roundings of P and the sums."""
    attn = models.AttnSpec(4, 2, dim, dim, dim ** -0.5, window, keep)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=500, layers=(models.StackLayerSpec(attn, 128),) * 2,
                            embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=1024, max_slots=1)
    eng = engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device(DEV), 8))
    ids = torch.randint(0, 500, (1, 900), generator=torch.Generator().manual_seed(9)).to(DEV)
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    whole = eng.forward(ids, True)
    eng.reset_cache()
    parts = torch.cat([eng.forward(ids[:, a:b].contiguous(), True) for a, b in ((0, 40), (40, 120), (120, 377), (377, 900))], 1)
    assert torch.equal(whole, parts)
    monkeypatch.setenv("B200_ATTN_TC", "mma")
    eng.reset_cache()
    other = eng.forward(ids, True).double()
    assert float((whole.double() - other).norm() / other.norm()) < 1e-2
    eng.close()
