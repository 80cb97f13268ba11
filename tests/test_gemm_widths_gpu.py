"""Tiles of 256, 224 and 192 columns on the persistent CTA pairs: every epilogue against one tile per CTA, bit for bit (a row's sum has one order
whatever the tile), at column counts that end inside a tile, a store's chunk and a pair's half, and row counts around one and several tiles per pair."""
import pytest
import torch

from tinygpt_b200 import engine, models, ops, stack_bench

pytestmark = pytest.mark.gpu
DEV = "cuda"
WIDTHS = ["persistent256", "persistent224", "persistent192"]


def rand(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("N", [8, 184, 192, 200, 232, 448, 456, 1000, 5000])
@pytest.mark.parametrize("M,K", [(17, 64), (256, 136), (300, 72), (2003, 520)])
def test_store_and_bias(built_lib, monkeypatch, N, M, K):
    x, w, b = rand(M, K, seed=1), rand(N, K, seed=2, scale=K ** -0.5), rand(N, seed=3)
    monkeypatch.setenv("B200_GEMM", "tile")
    want = ops.gemm(x, w), ops.linear(x, w, b)
    err = (want[0].double() - x.double() @ w.double().t()).norm() / want[0].double().norm()
    assert float(err) < 2.0 ** -8
    for side in WIDTHS:
        monkeypatch.setenv("B200_GEMM", side)
        assert torch.equal(ops.gemm(x, w), want[0]) and torch.equal(ops.linear(x, w, b), want[1]), side


@pytest.mark.parametrize("ff", [3080, 5464])
def test_prompt_tails(built_lib, monkeypatch, ff):
    """Bias, residual and SiLU products of a one-layer model: the logits of the last row."""
    spec = models.ModelSpec("wide", "qwen2", 7176, 1, 40, 8, 128, ff, 512, 1e6, 1e-6, tie=True, qkv_bias=True, max_ctx=2048)
    eng = engine.DecodeEngine(spec, models.synth_weights(spec, seed=5, device=DEV))
    for S in (300, 2003):
        ids = torch.randint(0, spec.vocab, (1, S), generator=torch.Generator().manual_seed(S)).to(DEV)
        got = {}
        for side in ["tile", *WIDTHS]:
            monkeypatch.setenv("B200_GEMM", side)
            eng.reset_cache()
            got[side] = eng.forward(ids)
        assert all(torch.equal(got["tile"], got[side]) for side in WIDTHS), S
    eng.close()


def test_fp32_tails(built_lib, monkeypatch):
    """fp32 bias, the fp32 residual sum and fp32 logits of a layer-stack model, every row."""
    attn = models.AttnSpec(8, 2, 64, 64, 64 ** -0.5, 0, 0)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=1160, vocab=5000, layers=(models.StackLayerSpec(attn, 1528),) * 2,
                            embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=2048, max_slots=1)
    eng = engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device(DEV), 8))
    toks = torch.randint(0, 5000, (1, 1500), generator=torch.Generator().manual_seed(9)).to(DEV)
    got = {}
    for side in ["tile", *WIDTHS]:
        monkeypatch.setenv("B200_GEMM", side)
        eng.reset_cache()
        got[side] = eng.forward(toks, True)
    assert all(torch.equal(got["tile"], got[side]) for side in WIDTHS)
    eng.close()


@pytest.mark.parametrize("side", ["persistent128", "persistent0", "persistent257"])
def test_a_width_that_is_not_built(built_lib, monkeypatch, side):
    """Any of those that are: the persistent pairs all the same."""
    x, w = rand(300, 136, seed=1), rand(456, 136, seed=2, scale=136 ** -0.5)
    monkeypatch.setenv("B200_GEMM", "persistent")
    want = ops.gemm(x, w)
    monkeypatch.setenv("B200_GEMM", side)
    assert torch.equal(ops.gemm(x, w), want)
