"""The layer-stack engine's 16-byte row kernels (csrc/stack_ops.cu) and the products' fp32 tails (csrc/gemm.cu) where they can go wrong: row lengths
with and without a vector kernel, unaligned rows, and heads of more rows than a decode batch."""
import pytest
import torch

from tinygpt_b200 import engine, models, ops, stack_bench

pytestmark = pytest.mark.gpu
DEV = "cuda"
ACTS = {"gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh"), "silu": torch.nn.functional.silu,
        "gelu_erf": torch.nn.functional.gelu, "relu2": lambda z: torch.relu(z) ** 2, "tanh": torch.tanh}


def randn(*shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV).to(dtype)


@pytest.mark.parametrize("dim", [4, 36, 2048, 4096, 4100, 6, 101])
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
def test_norm_rows(built_lib, dim, out):
    x, w = randn(5, dim, seed=1, dtype=torch.float32), randn(dim, seed=2, dtype=torch.float32)
    got = ops.stack_rmsnorm(x, w, 1e-5, 1.0, out)
    xd = x.double()
    want = xd / (xd.square().mean(-1, keepdim=True) + 1e-5).sqrt() * (1 + w.double())
    # fp32 sums of up to 4100 squares, then at most three roundings; bf16: half an ulp of the result
    tol = 2.0 ** -8 if out == torch.bfloat16 else 2e-6
    assert float(((got.double() - want).abs() / (want.abs() + 1e-6)).max()) <= tol


@pytest.mark.parametrize("act", sorted(ACTS))
@pytest.mark.parametrize("n", [8, 24, 1001, 2048, 4104])
def test_activation_rows(built_lib, act, n):
    g, u = randn(3, n, seed=3), randn(3, n, seed=4)
    got = ops.stack_act_mul(g, u, act).double()
    want = ACTS[act](g.double()).to(torch.bfloat16).double() * u.double()
    # the activation may round to the other neighbour (one bf16 ulp), then the product rounds once
    assert bool(((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-6).all())
    alone = ops.stack_act(g, act).double()
    assert bool(((alone - ACTS[act](g.double())).abs() <= 2.0 ** -7 * alone.abs() + 1e-6).all())


@pytest.mark.parametrize("rows", [8, 9, 31, 32, 130, 300])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_head_of_many_rows(built_lib, rows, softcap):
    """step() with every position wanted: the same logits as fed in portions of at most eight rows (decode kernels), up to the order of fp32
    sums and the bf16 roundings of one layer that a portion's other kernels make."""
    attn = models.AttnSpec(4, 2, 64, 64, 64 ** -0.5, 0, 0)
    spec = models.StackSpec(name="head", architecture="Kozusun", width=256, vocab=1000, layers=(models.StackLayerSpec(attn, 128),),
                            embed_scale=4.0, residual_mult=0.3, norm_eps=1e-5, norm_offset=1.0, logit_softcap=softcap, max_ctx=512,
                            max_slots=2)
    eng = engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device(DEV), 5))
    toks = torch.randint(0, 1000, (rows,), generator=torch.Generator().manual_seed(6)).tolist()
    got = eng.step([(0, toks, list(range(rows)))])
    want = torch.cat([eng.step([(1, toks[a:a + 8], list(range(len(toks[a:a + 8]))))]) for a in range(0, rows, 8)])
    assert float((got - want).norm() / want.norm()) < 1.5e-2
    eng.reset_cache()
    bf = eng.forward(torch.tensor([toks], device=DEV), all_positions=True)[0]
    assert float((bf.float() - got).abs().max()) <= 2.0 ** -8 * float(got.abs().max()) + 1e-6
    eng.close()
