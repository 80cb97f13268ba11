"""Layer-stack prompts of 9 to 31 rows, whose products run on the tcgen05 GEMM like those of longer ones: portions of such lengths give the bits of the whole
prompt (attention takes one kernel from 16 rows on), and results agree with the general kernels' to the bf16 roundings of a few layers; a
matrix off the 16-byte boundary stays with the general kernel."""
import pytest
import torch

from tinygpt_b200 import engine, models, stack_bench

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _spec():
    attn = models.AttnSpec(4, 2, 64, 64, 64 ** -0.5, 0, 0)
    return models.StackSpec(name="s", architecture="Kozusun", width=256, vocab=500, layers=(models.StackLayerSpec(attn, 320),) * 2, embed_scale=4.0,
                            residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=512, max_slots=1)


def _ids(n):
    return torch.randint(0, 500, (1, n), generator=torch.Generator().manual_seed(n)).to(DEV)


def test_portions(built_lib):
    eng = engine.DecodeEngine(_spec(), stack_bench.device_stack_weights(_spec(), torch.device(DEV), 3))
    ids = _ids(100)
    whole = eng.forward(ids, True)
    for cuts in ((0, 16, 47, 100), (0, 31, 48, 69, 100)):
        eng.reset_cache()
        parts = [eng.forward(ids[:, a:b].contiguous(), True) for a, b in zip(cuts, cuts[1:])]
        assert torch.equal(torch.cat(parts, 1), whole)
    eng.close()


@pytest.mark.parametrize("rows", [9, 15, 16, 17, 31, 32])
def test_against_the_general_kernels(built_lib, monkeypatch, rows):
    w = stack_bench.device_stack_weights(_spec(), torch.device(DEV), 4)
    out = []
    for plain in ("", "1"):
        monkeypatch.setenv("B200_STACK_PLAIN", plain)
        eng = engine.DecodeEngine(_spec(), w)
        out.append(eng.forward(_ids(rows), True).double())
        eng.close()
    assert float((out[0] - out[1]).norm() / out[1].norm()) < 1e-2
