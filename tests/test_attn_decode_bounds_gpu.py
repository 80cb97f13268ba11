"""attn_decode with a position outside its caches (csrc/attn.cu): the kernel's own check leaves the caches and what lies around them as they are, with and without
a rotation table, and the result is zero; the next call with a position inside is right."""
import pytest
import torch

from tinygpt_b200._lib import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,hd", [(14, 2, 64), (24, 8, 128)])
@pytest.mark.parametrize("ctx", [1, 100, 256, 1024, 4096])
def test_position_outside(built_lib, Hq, Hkv, hd, ctx):
    pad = 64
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    qkv, big_k, big_v = r((Hq + 2 * Hkv) * hd), r(ctx + 2 * pad, Hkv, hd), r(ctx + 2 * pad, Hkv, hd)
    rope = torch.ones(ctx + 2 * pad, hd, 2, device="cuda")
    k, v = big_k[pad:pad + ctx], big_v[pad:pad + ctx]
    was = big_k.clone(), big_v.clone()
    ws = torch.zeros(lib().b200_attn_decode_workspace_bytes(Hq, Hkv, hd, ctx), dtype=torch.uint8, device="cuda")
    out, pos = torch.full((Hq * hd,), 7.0, device="cuda").bfloat16(), torch.zeros(1, dtype=torch.int32, device="cuda")

    def call(table):
        rc = lib().b200_attn_decode_bf16(out.data_ptr(), qkv.data_ptr(), None, None, 0.0, table, pos.data_ptr(), 0, k.data_ptr(), v.data_ptr(), Hq, Hkv, hd, ctx,
                                         ws.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0

    for at in (-1, -2 ** 31, ctx, ctx + 1, ctx + 40, 2 ** 31 - 1):
        pos.fill_(at)
        for table in (None, rope[pad:].data_ptr()):
            out.fill_(7.0)
            call(table)
            torch.cuda.synchronize()
            assert torch.equal(big_k, was[0]) and torch.equal(big_v, was[1]) and not bool(out.any())
    pos.fill_(ctx - 1)
    call(None)
    torch.cuda.synchronize()
    assert torch.equal(k[-1].reshape(-1), qkv[Hq * hd:(Hq + Hkv) * hd]) and torch.equal(v[-1].reshape(-1), qkv[(Hq + Hkv) * hd:])
    assert torch.equal(big_k[:pad + ctx - 1], was[0][:pad + ctx - 1]) and torch.equal(big_k[pad + ctx:], was[0][pad + ctx:])
    s = torch.einsum("hd,khd->hk", qkv[:Hq * hd].double().view(Hq, hd), k.double().repeat_interleave(Hq // Hkv, 1)) * hd ** -0.5
    want = torch.einsum("hk,khd->hd", torch.softmax(s, -1), v.double().repeat_interleave(Hq // Hkv, 1)).reshape(-1)
    assert float((out.double() - want).abs().max()) <= 2.0 ** -7 * float(v.double().abs().max())
