"""Rows of a layer-stack engine's prompt keep their bits whatever else runs with them: a prompt in one step, in portions and beside another
request gives the same logits, as long as every step is one of the tensor-core products (32 rows or more; 16 or more per sequence).  The
products sum over the whole K in one order, and the attention kernel is chosen by the model and the context alone.  Sizes reach both
attention kernels' ranges, short and long K, routed experts whose groups grow with the other request, and the soft cap."""
import pytest
import torch

from tinygpt_b200 import engine, models, stack_bench

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def parallel(dim, window, keep, ctx, ff=1024):
    attn = models.AttnSpec(8, 2, dim, dim, dim ** -0.5, window, keep)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=512, vocab=520, layers=(models.StackLayerSpec(attn, ff),) * 2,
                            embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=ctx, max_slots=2)
    return spec, stack_bench.device_stack_weights(spec, DEV, 8)


def latent_experts(ctx):
    rot = models.RotarySpec(dims=64, base=5e5, factor=4.0, original=2048, fast=32.0, slow=1.0)
    lat = models.LatentSpec(4, 64, 64, 128, 128, 128 ** -0.5, rot)
    moe = models.MoeSpec(8, 2, 1024, 7.0, 512, 7.0)
    L = models.StackLayerSpec
    spec = models.StackSpec(name="s", architecture="Silatar", width=768, vocab=520, norm_eps=1e-5, block="sandwich", norm_kind="layer",
                            layers=(L(mixer="latent_attention", latent=lat, ff_kind="moe", moe=moe),
                                    L(mixer="latent_attention", latent=lat, ff_kind="dense", ff=2048, ff_act="gelu_erf")),
                            loop_mix=False, logit_softcap=30.0, max_ctx=ctx, max_slots=2)
    return spec, stack_bench.device_silatar_weights(spec, DEV, 9)


CASES = {"long": lambda: parallel(128, 0, 0, 2304), "short": lambda: parallel(64, 0, 0, 640), "window": lambda: parallel(128, 300, 5, 2304),
         "long k": lambda: parallel(64, 0, 0, 2304, 4608), "experts": lambda: latent_experts(2304)}


@pytest.mark.parametrize("name", sorted(CASES))
def test_logits_do_not_depend_on_what_else_a_step_holds(built_lib, name):
    spec, w = CASES[name]()
    n = min(1500, spec.max_ctx - 40)
    toks = torch.randint(0, spec.vocab, (n,), generator=torch.Generator().manual_seed(1)).tolist()
    other = torch.randint(0, spec.vocab, (n,), generator=torch.Generator().manual_seed(2)).tolist()
    eng = engine.DecodeEngine(spec, w)
    whole = eng.step([(0, toks, range(n))])
    for cuts in ((40, 168, 400), (32, 65, 333, n - 60)):
        eng.reset_cache()
        at = [0, *cuts, n]
        parts = [eng.step([(1, toks[a:b], range(b - a))]) for a, b in zip(at, at[1:])]
        assert torch.equal(torch.cat(parts), whole), cuts
    eng.reset_cache()
    beside = [eng.step([(0, other[:b], []), (1, toks[a:b], range(b - a))] if a == 0 else [(1, toks[a:b], range(b - a)), (0, other[a:b], [])])
              for a, b in ((0, 200), (200, n))]
    assert torch.equal(torch.cat(beside), whole)
    eng.verify()
    eng.close()
