"""Layer-stack prompts of 9 to 31 rows, whose products run on the tcgen05 GEMM like those of longer ones: portions of such lengths give the bits of the whole
prompt (attention takes one kernel from 16 rows on), and results agree with the general kernels' to the bf16 roundings of a few layers; matrices
off the 16-byte boundary stay with the general kernel, those of the side input in a narrow model at any length."""
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


def _off_boundary(w, name):
    t = w[name]
    room = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    return {**w, name: room[1:1 + t.numel()].copy_(t.view(-1)).view(t.shape)}


@pytest.mark.parametrize("name", ["l0.w_in", "l1.w_out"])
@pytest.mark.parametrize("rows", [9, 16, 31])
def test_matrix_off_the_boundary(built_lib, name, rows):
    w = stack_bench.device_stack_weights(_spec(), torch.device(DEV), 5)
    out = []
    for weights in (w, _off_boundary(w, name)):
        eng = engine.DecodeEngine(_spec(), weights)
        out.append(eng.forward(_ids(rows), True).double())
        eng.close()
    assert float((out[0] - out[1]).norm() / out[0].norm()) < 1e-2


@pytest.mark.parametrize("rows", [4, 9, 31, 32, 40])
def test_side_input_of_a_narrow_model_off_the_boundary(built_lib, rows):
    """Width 32: the side input's first product has too few columns for the GEMM, its second one has enough."""
    attn = models.AttnSpec(2, 2, 16, 16, 0.25, 0, 0)
    spec = models.StackSpec(name="s", architecture="Kozusun", width=32, vocab=500, layers=(models.StackLayerSpec(attn, 64),) * 2, embed_scale=4.0,
                            residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=64, max_slots=1, side_dim=64)
    w = stack_bench.device_stack_weights(spec, torch.device(DEV), 6)
    out = []
    for weights in (w, _off_boundary(w, "l0.side_proj")):
        eng = engine.DecodeEngine(spec, weights)
        out.append(eng.forward(_ids(rows), True).double())
        eng.close()
    assert float((out[0] - out[1]).norm() / out[0].norm()) < 1e-2
