"""The prompt pass's row-wise kernels (csrc/ops.cu, prefill.cu) and Linears with their tails (csrc/gemm.cu) at vector edges: row lengths that
take the 16-byte kernels and ones that do not, unaligned views, every tail through small engines, and prompts in portions.  The vector kernels
keep the scalar ones' order of operations, so where both exist the results are the same bits."""
import pytest
import torch

from tinygpt_b200 import engine, models, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rand(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


def shifted(t):
    """The same values two bytes off a 16-byte boundary: the scalar kernels."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


@pytest.mark.parametrize("rows,dim", [(1, 8), (3, 64), (5, 896), (2, 2048), (7, 2056), (3, 8192), (2, 8200), (3, 100)])
def test_vector_kernels_match_scalar_bits(built_lib, rows, dim):
    x, y, w = rand(rows, dim, seed=1), rand(rows, dim, seed=2), rand(dim, seed=3)
    assert torch.equal(ops.rms_norm(x, w, 1e-6), ops.rms_norm(shifted(x), w, 1e-6))
    assert torch.equal(ops.rms_norm(x, None, 1e-6), ops.rms_norm(shifted(x), None, 1e-6))
    assert torch.equal(ops.add(x, y), ops.add(shifted(x), y))
    gu = rand(rows, 2 * dim, seed=4, scale=3.0)
    gu[0, 0], gu[0, 1] = float("-inf"), float("inf")
    a, b = ops.silu_mul(gu), ops.silu_mul(shifted(gu))
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(9.0), b.nan_to_num(9.0))


@pytest.mark.parametrize("spec", [models.TINY_QWEN2, models.TINY_QWEN3, models.TINY_LLAMA, models.TINY_MISTRAL], ids=lambda s: s.name)
def test_prompt_rows_do_not_depend_on_the_pass(built_lib, spec, monkeypatch):
    """A Linear's K order does not depend on the row count: a prompt in portions gives the same logits as in one pass, bit for bit
    (attention on the CUDA cores here, whose rows are independent of the pass as well)."""
    spec = spec.with_ctx(1024)
    w = {k: v.to(DEV) for k, v in models.synth_weights(spec, seed=6).items()}
    monkeypatch.setenv("B200_PREFILL_ATTN", "cuda")
    eng = engine.DecodeEngine(spec, w)
    ids = torch.randint(0, spec.vocab, (1, 700), generator=torch.Generator().manual_seed(7)).to(DEV)
    eng.reset_cache()
    whole = eng.forward(ids)
    eng.reset_cache()
    for a, b in ((0, 9), (9, 137), (137, 400), (400, 700)):
        parts = eng.forward(ids[:, a:b].contiguous())
    assert torch.equal(whole, parts)
    eng.close()


@pytest.mark.parametrize("spec", [models.TINY_QWEN2, models.TINY_QWEN3, models.TINY_MISTRAL], ids=lambda s: s.name)
@pytest.mark.parametrize("kernels", [("", ""), ("persistent", "tile"), ("tile", "persistent"), ("wide", "tile")], ids=lambda k: "-".join(k) or "default")
def test_prompt_rows_do_not_depend_on_the_kernel(built_lib, spec, kernels, monkeypatch):
    """The same with the default attention, and with the whole prompt on the CTA pairs and its portions on one-CTA tiles, as a long prompt
    and its short portions are."""
    spec = spec.with_ctx(1024)
    eng = engine.DecodeEngine(spec, {k: v.to(DEV) for k, v in models.synth_weights(spec, seed=6).items()})
    ids = torch.randint(0, spec.vocab, (1, 700), generator=torch.Generator().manual_seed(7)).to(DEV)
    if kernels[0]:
        monkeypatch.setenv("B200_GEMM", kernels[0])
    whole = eng.forward(ids)
    if kernels[1]:
        monkeypatch.setenv("B200_GEMM", kernels[1])
    eng.reset_cache()
    for a, b in ((0, 9), (9, 137), (137, 400), (400, 700)):
        parts = eng.forward(ids[:, a:b].contiguous())
    assert torch.equal(whole, parts)
    eng.close()


@pytest.mark.parametrize("S", [1795, 2003, 2048])
def test_tails_on_pairs_that_run_three_tiles(built_lib, S, monkeypatch):
    """Bias, residual and SiLU on the persistent pairs with more tiles than twice the pairs (a TMEM accumulator is used again) and ragged
    rows and columns, against one tile per CTA: a one-layer model, whose last row of logits holds that row's whole products."""
    spec = models.ModelSpec("wide", "qwen2", 7176, 1, 40, 8, 128, 3080, 512, 1e6, 1e-6, tie=True, qkv_bias=True, max_ctx=2048)
    eng = engine.DecodeEngine(spec, models.synth_weights(spec, seed=5, device=DEV))
    ids = torch.randint(0, spec.vocab, (1, S), generator=torch.Generator().manual_seed(S)).to(DEV)
    got = {}
    for side in ("tile", "wide", "persistent"):
        monkeypatch.setenv("B200_GEMM", side)
        eng.reset_cache()
        got[side] = eng.forward(ids)
    assert torch.equal(got["tile"], got["persistent"]) and torch.equal(got["tile"], got["wide"])
    eng.close()


@pytest.mark.parametrize("side", ["tile", "wide", "persistent"])
def test_bias_tail_of_many_tiles(built_lib, side, monkeypatch):
    """Every row and column of a product with its bias as the second rounding: three tiles for a pair, ragged edges."""
    monkeypatch.setenv("B200_GEMM", side)
    M, N, K = 2003, 5400, 520
    x, w, b = rand(M, K, seed=1), rand(N, K, seed=2, scale=K ** -0.5), rand(N, seed=3)
    prod = (x.float() @ w.float().t()).to(torch.bfloat16)
    want, got = prod + b, ops.linear(x, w, b)
    # another order of the fp32 sum: the product may round to its other neighbour, and the sum with the bias to the neighbour of that
    ulp = lambda t: torch.exp2(torch.floor(torch.log2(t.float().abs().clamp_min(2.0 ** -126))) - 7)
    off = (got.float() - want.float()).abs()
    assert bool((off <= ulp(prod) + ulp(torch.maximum(got.abs(), want.abs()))).all())
    assert float((off == 0).float().mean()) >= 0.97


def test_unaligned_bias(built_lib):
    """A qkv bias off a 16-byte boundary takes the launch of its own: same bits as riding on the store."""
    spec = models.TINY_QWEN2
    w = {k: v.to(DEV) for k, v in models.synth_weights(spec, seed=8).items()}
    ids = torch.randint(0, spec.vocab, (1, 50), generator=torch.Generator().manual_seed(9)).to(DEV)
    a = engine.DecodeEngine(spec, w)
    want = a.forward(ids)
    b = engine.DecodeEngine(spec, {k: shifted(v) if k.endswith("qkv_proj.bias") else v for k, v in w.items()})
    assert torch.equal(b.forward(ids), want)
    a.close()
    b.close()
