"""The kernel that norms and rotates a prompt's q and k heads (csrc/prefill.cu): long prompts give a lane two heads of 64, short ones read the
rotation ahead of the kernel in front.  Each form does the same operations on a head, so a prompt on either side of a line, with an odd number of
heads too, gives the bits of its portions, which lie on the short side."""
import dataclasses

import pytest
import torch

from tinygpt_b200 import engine, models

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("base", [models.TINY_QWEN3, models.TINY_QWEN2], ids=lambda s: s.name)   # with and without the heads' norms
@pytest.mark.parametrize("q,kv,dim", [(7, 1, 64), (14, 2, 128)])   # lines at 1 052 rows: 148 and 4·148 CTAs of 256 lanes
@pytest.mark.parametrize("rows", [1052, 1053, 1100])
def test_long_prompts_have_the_bits_of_their_portions(built_lib, base, q, kv, dim, rows):
    spec = dataclasses.replace(base, q_heads=q, kv_heads=kv, head_dim=dim, layers=2).with_ctx(1280)
    w = {k: v.to(DEV) for k, v in models.synth_weights(spec, seed=6).items()}
    eng = engine.DecodeEngine(spec, w)
    ids = torch.randint(0, spec.vocab, (1, rows), generator=torch.Generator().manual_seed(7)).to(DEV)
    whole = eng.forward(ids)
    eng.reset_cache()
    for a, b in ((0, 512), (512, 1024), (1024, rows)):
        parts = eng.forward(ids[:, a:b].contiguous())
    assert torch.equal(whole, parts)
    eng.close()
