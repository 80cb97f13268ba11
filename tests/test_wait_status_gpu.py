"""A kernel that gives up a bounded wait leaves a code in a host word (csrc/common.cu): set here from the host, as the kernel would.  The
engine that owns the word fails from then on, after its synchronisations too, until it is reset; other engines and the operators do
not, and the operators report their own word once."""
import ctypes as C

import pytest
import torch

from tinygpt_b200 import engine, models, ops, stack_bench
from tinygpt_b200._lib import B200Error, lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def word(eng=None):
    return C.c_uint32.from_address(lib().b200_debug_wait_word(eng._h if eng else None))


def llama():
    spec = models.TINY_QWEN2
    return engine.DecodeEngine(spec, {k: v.to(DEV) for k, v in models.synth_weights(spec, seed=3).items()})


def stack():
    attn = models.AttnSpec(4, 2, 64, 64, 0.125, 0, 0)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=500, layers=(models.StackLayerSpec(attn, 128),),
                            embed_scale=4.0, residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=512, max_slots=2)
    return engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device(DEV), 8))


@pytest.mark.parametrize("make", [llama, stack])
def test_an_engine_that_lost_rows_says_so_until_it_is_reset(built_lib, make):
    a, b = make(), make()
    ids = torch.arange(40, device=DEV).view(1, -1)
    want = a.forward(ids)
    b.forward(ids)
    word(a).value = 0x6E000003                 # as if a product of that prompt had given up
    torch.cuda.synchronize()
    for call in (a.verify, lambda: a.decode(1), lambda: a.forward(ids[:, :1]), lambda: a.gen_next_token(ids[:, :1]), a.verify):
        with pytest.raises(B200Error, match="gave up"):
            call()
    if a.is_stack:
        with pytest.raises(B200Error, match="gave up"):
            a.step([(0, [1], [0])])
    b.decode(1)                                # nobody else's
    ops.gemm(torch.zeros(8, 8, dtype=torch.bfloat16, device=DEV), torch.zeros(8, 8, dtype=torch.bfloat16, device=DEV))
    torch.cuda.synchronize()
    b.verify()
    assert word(b).value == 0 and word(a).value != 0
    a.reset_cache()
    assert torch.equal(a.forward(ids), want)
    torch.cuda.synchronize()
    a.verify()
    a.close()
    b.close()


def test_generated_tokens_are_checked_when_they_reach_the_host(built_lib, monkeypatch):
    eng = llama()
    prompt, decode = list(range(12)), eng.decode

    def lose(n):
        word(eng).value = 0xA7000001           # while the steps are on their way
        monkeypatch.undo()
        return torch.zeros(n, dtype=torch.int64, device=DEV)

    monkeypatch.setattr(eng, "decode", lose)
    with pytest.raises(B200Error, match="gave up"):
        eng.generate_sync(prompt, 4)
    assert eng.decode == decode
    first = eng.generate_sync(prompt, 4)       # starts over
    assert torch.equal(first, eng.generate_sync(prompt, 4))
    eng.close()


def test_operators_report_their_own_once(built_lib):
    eng = llama()
    a = torch.ones(8, 8, dtype=torch.bfloat16, device=DEV)
    want = ops.gemm(a, a)
    word().value = 0x6E000007
    eng.forward(torch.arange(12, device=DEV).view(1, -1))
    torch.cuda.synchronize()
    eng.verify()
    with pytest.raises(B200Error, match="0x6e000007"):
        ops.gemm(a, a)
    assert torch.equal(ops.gemm(a, a), want)
    word().value = 0x6E000007
    assert lib().b200_wait_status() != 0 and lib().b200_wait_status() == 0
    word().value = 0xA7000001
    other = llama()                            # an engine neither minds nor takes the report
    assert lib().b200_device_check() == 0
    q = torch.ones(1, 8, 2, 64, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(B200Error, match="0xa7000001"):
        ops.flash_attention(q, q, q, True)
    ops.flash_attention(q, q, q, True)
    other.close()
    eng.close()
