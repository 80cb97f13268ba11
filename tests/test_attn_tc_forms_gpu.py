"""The two kernels of the tcgen05 prompt attention — one for up to 128 keys, a CTA per block of 128 rows, and one whose CTAs, one per SM, run through blocks with
tiles of 128 keys that two groups of warps take in turn — against fp64 at the edges of their tiles, with as many blocks as CTAs and a few more; P and
the result are bf16 (2-norm error below 2⁻⁸ of the result's, each element within 2⁻⁷ of the largest |V|)."""
import pytest
import torch

from test_attn_tc_gpu import DEV, attend, close, randn
from tinygpt_b200 import engine, models, ops, stack_bench

pytestmark = pytest.mark.gpu


# sequences · heads · ceil(rows / 128) blocks: some 148, one for each CTA, and a second for two of them; one to five tiles of 128 keys, the last one full or not
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 1, 150, 10), (1, 64, 160, 8), (3, 65, 64, 8), (1, 129, 74, 37), (1, 129, 75, 25), (2, 192, 40, 8), (1, 200, 80, 16),
                                        (1, 385, 37, 1), (1, 385, 38, 19), (1, 577, 32, 4)])
@pytest.mark.parametrize("D", [64, 128])
def test_causal(built_lib, monkeypatch, B, S, Hq, Hkv, D):
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    q, k, v = randn(B, S, Hq, D, seed=1, std=2.0), randn(B, S, Hkv, D, seed=2), randn(B, S, Hkv, D, seed=3)
    got = ops.flash_attention(q, k, v, True)
    close(got, attend(q, k, v), float(v.float().abs().max()))
    assert torch.equal(got, ops.flash_attention(q, k, v, True))


@pytest.mark.parametrize("heads", [4, 152])
@pytest.mark.parametrize("D", [64, 128])
def test_what_a_row_does_not_see(built_lib, monkeypatch, D, heads):
    """Infinities and NaNs in keys and values behind a row, in tiles of either parity: rows in front of them stay right, the others are not finite."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    S = 300
    for at in (40, 100, 190):
        q, k, v = randn(1, S, heads, D, seed=4), randn(1, S, heads // 2, D, seed=5), randn(1, S, heads // 2, D, seed=6)
        want = attend(q, k, v)
        v[0, at], v[0, at + 50], k[0, at + 60] = float("inf"), float("nan"), float("nan")
        got = ops.flash_attention(q, k, v, True)
        close(got[0, :at], want[0, :at], float(randn(1, S, heads // 2, D, seed=6).float().abs().max()))
        assert not bool(torch.isfinite(got[0, at + 50:].float()).any())


@pytest.mark.parametrize("D", [64, 128])
def test_keys_without_a_number(built_lib, monkeypatch, D):
    """Scores that are NaN in part of a tile, and in the whole of a tile, which is all that one of the two groups has for the rows of one block (it has no maximum, and a
    sum that is NaN): a row that sees one is NaN, not what the other group holds, and no other row is."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    for S, a, b in ((200, 64, 128), (400, 0, 128), (400, 128, 256), (500, 256, 384), (700, 128, 256)):
        q, k, v = randn(1, S, 2, D, seed=7), randn(1, S, 2, D, seed=8), randn(1, S, 2, D, seed=9)
        want = attend(q, k, v)
        k[0, a:b] = float("nan")
        got = ops.flash_attention(q, k, v, True)
        if a > 0:
            close(got[:, :a], want[:, :a], float(v.float().abs().max()))
        assert bool(got[0, a:].isnan().all())


@pytest.mark.parametrize("heads,window,keep", [(16, 0, 0), (16, 130, 5), (16, 65, 64), (6, 300, 70), (6, 1, 0)])
def test_window_prefix_and_gate(built_lib, monkeypatch, heads, window, keep):
    """Through a layer-stack engine with caches for 2 048 positions: a prompt in two portions, windows with kept first keys, the per-head gate,
    against the mma.sync kernel, to the bf16 roundings of the two kernels' P and sums."""
    attn = models.AttnSpec(heads, 2, 64, 64, 64 ** -0.5, window, keep)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=500, layers=(models.StackLayerSpec(attn, 128),) * 2,
                            embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=2048, max_slots=1)
    eng = engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device(DEV), 8))
    toks = torch.randint(0, 500, (1, 500), generator=torch.Generator().manual_seed(9)).to(DEV)
    out = {}
    for side in ("tc", "mma"):
        monkeypatch.setenv("B200_ATTN_TC", side)
        eng.reset_cache()
        out[side] = torch.cat([eng.forward(toks[:, :150].contiguous(), True), eng.forward(toks[:, 150:].contiguous(), True)], 1).double()
        if side == "tc":   # and in one portion: the same bits
            eng.reset_cache()
            assert torch.equal(eng.forward(toks, True).double(), out[side])
    assert float((out["tc"] - out["mma"]).norm() / out["mma"].norm()) < 1e-2
    eng.close()
