"""Products on tiles of 64 and 32 columns (csrc/gemm.cu): the same bits as on 128 columns at the edges of their tiles and rings — few rows and one more than a
tile's, columns that end inside a tile, k ranges of one block, of a full ring and of one more — with and without a bias, with a residual (a prompt),
with fp32 results, sums into fp32 and logits in fp32 and bf16 (a layer-stack prompt); and against the product in 64 bits (one bf16 rounding: 2⁻⁸
of a value, and fp32 sums)."""
import pytest
import torch

from tinygpt_b200 import engine, models, ops, stack_bench

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("form", ["half", "narrow"])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (9, 40, 64), (17, 96, 72), (64, 72, 832), (65, 256, 896), (128, 104, 960), (129, 64, 1024), (200, 520, 136)])
def test_same_bits_as_wider_tiles(built_lib, monkeypatch, form, M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) * 0.1).bfloat16()
    b = torch.randn(N, generator=g, device=DEV).bfloat16()
    out = {}
    for side in ("tile", form):
        monkeypatch.setenv("B200_GEMM", side)
        out[side] = [ops.gemm(x, w), ops.linear(x, w, b) if M > 16 else ops.gemm(x, w)]
    assert all(torch.equal(a, c) for a, c in zip(out["tile"], out[form]))
    want = x.double() @ w.double().t()
    got = out[form][0].double()
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + K ** 0.5 * 2.0 ** -20).all())


@pytest.mark.parametrize("form", ["half", "narrow"])
@pytest.mark.parametrize("spec", [models.TINY_QWEN2, models.TINY_QWEN3], ids=lambda s: s.name)
def test_prompt_has_the_same_bits(built_lib, monkeypatch, form, spec):
    """Bias and residual tails through an engine's prompt of 150 rows."""
    eng = engine.DecodeEngine(spec.with_ctx(256), {k: v.to(DEV) for k, v in models.synth_weights(spec.with_ctx(256), seed=6).items()})
    ids = torch.randint(0, spec.vocab, (1, 150), generator=torch.Generator().manual_seed(7)).to(DEV)
    out = []
    for side in ("persistent", form):
        monkeypatch.setenv("B200_GEMM", side)
        eng.reset_cache()
        out.append(eng.forward(ids))
    assert torch.equal(*out)
    eng.close()


@pytest.mark.parametrize("softcap", [0.0, 5.0])
@pytest.mark.parametrize("rows", [20, 70, 150])
def test_layer_stack_prompt_has_the_same_bits(built_lib, monkeypatch, rows, softcap):
    """Products summed into the fp32 stream (out), handed out in fp32 (the loop's mix; the side input's up to 31 rows) and with a bias (in), and logits in
    bf16 alone and beside fp32; 72, 256 and 504 columns."""
    attn = models.AttnSpec(4, 2, 64, 64, 0.125, 0, 0)
    spec = models.StackSpec(name="s", architecture="Kozusun", width=256, vocab=504, layers=(models.StackLayerSpec(attn, 328),) * 2, loop_start=0, loop_stop=1,
                            loop_times=2, embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, side_dim=72, max_ctx=256, max_slots=1,
                            logit_softcap=softcap)
    eng = engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device(DEV), 4))
    ids = torch.randint(0, spec.vocab, (1, rows), generator=torch.Generator().manual_seed(7)).to(DEV)
    out = {}
    for form in ("tile", "half", "narrow"):
        monkeypatch.setenv("B200_GEMM", form)
        eng.reset_cache()
        logits = eng.forward(ids, True)
        eng.reset_cache()
        out[form] = logits, eng.step([(0, ids[0].tolist(), list(range(rows)))]).clone()
    eng.close()
    assert bool(torch.isfinite(out["tile"][1]).all()) and out["tile"][1].dtype == torch.float32
    for form in ("half", "narrow"):
        assert all(torch.equal(a, b) for a, b in zip(out["tile"], out[form])), form
