"""A sequence's logits do not depend on how many others are decoded beside it, to the bit, over caches long enough for attn_row_kernel (csrc/attn.cu): batches of
two and more cut the keys into the same ranges.  (A single sequence has products of its own, which sum in another order.)"""
import dataclasses

import pytest
import torch

from tinygpt_b200 import engine, models

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("q,kv,dim", [(16, 8, 128), (14, 2, 64), (32, 32, 64), (14, 14, 128), (6, 2, 128)])
@pytest.mark.parametrize("at", [9, 130, 700, 2290])
def test_batches_of_two_five_and_eight(built_lib, q, kv, dim, at):
    spec = dataclasses.replace(models.TINY_QWEN3, q_heads=q, kv_heads=kv, head_dim=dim, layers=2).with_ctx(2304)
    eng = engine.DecodeEngine(spec, {k: t.to(DEV) for k, t in models.synth_weights(spec, seed=4).items()})
    ids = torch.randint(0, spec.vocab, (8, at + 6), generator=torch.Generator().manual_seed(at)).to(DEV)
    got = {}
    for B in (2, 5, 8):
        eng.reset_cache()
        eng.forward(ids[:B, :at].contiguous())
        got[B] = torch.stack([eng.forward(ids[:B, at + t:at + t + 1].contiguous())[:2].clone() for t in range(6)])
    assert bool(torch.isfinite(got[2].float()).all())
    for B in (5, 8):
        assert torch.equal(got[B], got[2]), B
    eng.close()
