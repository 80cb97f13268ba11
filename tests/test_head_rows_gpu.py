"""Logits of every position of a layer-stack prompt.  Where the head is a GEMM they are stored as bf16 straight into the caller's rows, and the
last positions are read from there; what does not fit that form (a handful of rows, several sequences in several passes, rows that are not
16-byte aligned) goes through the engine's own buffer.  Both are the fp32 logits of a ragged step over the same tokens, rounded to bf16 (7
rows: the head of both calls is a GEMV; with 8 only the step's would be)."""
import pytest
import torch

from tinygpt_b200 import engine, models, stack_bench
from tinygpt_b200._lib import check, lib

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def build(vocab, cap):
    attn = models.AttnSpec(4, 2, 64, 64, 0.125, 0, 0)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=vocab, layers=(models.StackLayerSpec(attn, 512),) * 2,
                            embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, logit_softcap=cap, max_ctx=4224, max_slots=3)
    return engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, DEV, 8))


@pytest.mark.parametrize("vocab,cap", [(520, 0.0), (520, 2.0), (516, 0.0)])   # 516: no rows of the GEMM's
@pytest.mark.parametrize("batch,rows", [(1, 7), (1, 9), (1, 257), (3, 3), (3, 40), (1, 4096 + 5), (1, 4096 + 9), (3, 1500)])
def test_every_position(built_lib, vocab, cap, batch, rows):
    eng = build(vocab, cap)
    ids = torch.randint(0, vocab, (batch, rows), generator=torch.Generator().manual_seed(rows), dtype=torch.int64)
    want = eng.step([(b, ids[b].tolist(), range(rows)) for b in range(batch)]).view(batch, rows, vocab).to(torch.bfloat16)
    dev = ids.to(DEV)
    for shift in (0, 1):   # the caller's rows on and off a 16-byte boundary
        eng.reset_cache()
        out = torch.zeros(batch * rows * vocab + 8, dtype=torch.bfloat16, device=DEV)
        check(lib().b200_engine_forward(eng._h, dev.data_ptr(), batch, rows, out.data_ptr() + 2 * shift, 1, eng._stream()), "forward")
        got = out[shift:shift + batch * rows * vocab].view(batch, rows, vocab)
        assert torch.equal(got, want)
        assert not out[:shift].any() and not out[shift + batch * rows * vocab:].any()
        last = got[:, -1].float()
        best = [int((row == row.max()).nonzero()[-1]) for row in last]   # of equals the highest
        token = torch.empty(batch, 1, dtype=torch.int64, device=DEV)
        check(lib().b200_engine_last_token(eng._h, token.data_ptr(), eng._stream()), "last_token")
        assert token.flatten().tolist() == best
    eng.verify()
    eng.close()
