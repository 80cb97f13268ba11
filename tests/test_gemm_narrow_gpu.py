"""Products on tiles of 64 and 32 columns (csrc/gemm.cu): the same bits as on 128 columns at the edges of their tiles and rings — few rows and one more than a
tile's, columns that end inside a tile, k ranges of one block, of a full ring and of one more — with and without a bias, a residual and fp32
results, and against the product in 64 bits (one bf16 rounding: 2⁻⁸ of a value, and fp32 sums)."""
import pytest
import torch

from tinygpt_b200 import engine, models, ops

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
