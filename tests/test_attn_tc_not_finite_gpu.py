"""Values that are not finite, in the tcgen05 prompt attention (csrc/prefill_attn_tc.cu): the rows of a block that go over their keys one after another, which over a
long cache takes longer than the kernel's waits last, fail nobody who has work behind them; and rows that do not see such a value — in front of
it, or a window behind it — keep results as if it were not there, also in CTAs with several blocks and behind a cached prefix.  Bounds as in
test_attn_tc_gpu; a step's logits against those of a step without the value: 1e-2 of a row's norm, the bf16 roundings of P and sums."""
import pytest
import torch

from test_attn_tc_gpu import DEV, close, randn
from tinygpt_b200 import engine, models, ops, stack_bench
from tinygpt_b200._lib import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
def test_long_rows_one_after_another(built_lib, D):
    """300 000 keys: the last block, its CTA's first of many, walks them for one or two seconds; a row to a lane, whose keys were read again for each eight
    columns, took a multiple of the 2 s that the kernel's waits last, in front of the CTA's other blocks."""
    S, at = 300_000, 299_950
    q, k, v = randn(1, S, 1, D, seed=1, std=2.0), randn(1, S, 1, D, seed=2), randn(1, S, 1, D, seed=3)
    rows = torch.cat([torch.arange(0, S - 96, 1499), torch.arange(S - 96, at)]).to(DEV)
    s = (q[0, rows, 0].double() @ k[0, :, 0].double().t()) * D ** -0.5
    s.masked_fill_(torch.arange(S, device=DEV)[None] > rows[:, None], float("-inf"))
    want, vmax = torch.softmax(s, -1) @ v[0, :, 0].double(), float(v.float().abs().max())
    del s
    v[0, at] = float("inf")
    v[0, at + 9] = float("nan")
    got = ops.flash_attention(q, k, v, True)[0, :, 0]
    torch.cuda.synchronize()
    assert lib().b200_wait_status() == 0
    close(got[rows], want, vmax)
    assert bool(torch.isfinite(got[:at].float()).all()) and not bool(torch.isfinite(got[at:].float()).any())


@pytest.mark.parametrize("window,keep", [(0, 0), (1, 0), (130, 5), (300, 200), (700, 0)])
@pytest.mark.parametrize("dim", [64, 128])
def test_rows_that_do_not_see_it(built_lib, monkeypatch, window, keep, dim):
    """A layer-stack prompt of 192 blocks in two portions, one token of which is not finite."""
    monkeypatch.setenv("B200_ATTN_TC", "tc")
    attn = models.AttnSpec(16, 2, dim, dim, dim ** -0.5, window, keep)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=500, layers=(models.StackLayerSpec(attn, 128),), embed_scale=4.0,
                            residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=2048, max_slots=1)
    w = stack_bench.device_stack_weights(spec, torch.device(DEV), 8)
    w["embed"][499] = float("inf")
    eng = engine.DecodeEngine(spec, w)
    ids = torch.randint(0, 499, (1, 1700), generator=torch.Generator().manual_seed(9)).to(DEV)

    def run(x):
        eng.reset_cache()
        return torch.cat([eng.forward(x[:, :200].contiguous(), True), eng.forward(x[:, 200:].contiguous(), True)], 1)[0].double()

    plain = run(ids)
    for at in (3, 150, 700, 1690):
        ids2 = ids.clone()
        ids2[0, at] = 499
        got, r = run(ids2), torch.arange(1700, device=DEV)
        sees = r >= at
        if window > 0 and at >= keep:
            sees &= r - at < window
        assert not bool(torch.isfinite(got[sees]).any())
        assert float(((got - plain).norm(dim=1) / plain.norm(dim=1))[~sees].max()) < 1e-2
    eng.close()
