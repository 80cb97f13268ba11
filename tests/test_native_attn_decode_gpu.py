"""attn_decode over caches of any length on the cluster kernel (csrc/attn.cu), as a native call (csrc/torch_ops.cpp) and from Python (a strided view of the
rows goes that way): the same bits, call after call, on the edges of the key ranges, on another stream and captured; against 64 bits within
two bf16 roundings of the largest value; and into a result at any address of a bf16, with the same bits and whatever lies in the workspace."""
import pytest
import torch

from tinygpt_b200 import ops

pytestmark = pytest.mark.gpu


def _inputs(Hq, Hkv, hd, ctx, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    return r((Hq + 2 * Hkv) * hd), r(ctx, Hkv, hd), r(ctx, Hkv, hd)


def _call(qkv, k, v, hq, hkv, hd, at):
    k, v = k.clone(), v.clone()
    pos = torch.tensor([at], dtype=torch.int32, device="cuda")
    return ops.attn_decode(qkv, k, v, q_heads=hq, kv_heads=hkv, head_dim=hd, pos=pos), k, v


@pytest.mark.parametrize("Hq,Hkv,hd", [(14, 2, 64), (16, 8, 128), (3, 1, 64)])
@pytest.mark.parametrize("ctx,at", [(1, 0), (64, 63), (128, 127), (129, 128), (256, 3), (1000, 999), (1024, 500), (1030, 1029)])
def test_same_bits_as_from_python(built_lib, Hq, Hkv, hd, ctx, at):
    qkv, k, v = _inputs(Hq, Hkv, hd, ctx)
    strided = torch.stack([qkv, qkv], 1)[:, 0]
    want = _call(strided, k, v, Hq, Hkv, hd, at)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(_call(qkv, k, v, Hq, Hkv, hd, at), want))
    with torch.cuda.stream(torch.cuda.Stream()):
        other = _call(qkv, k, v, Hq, Hkv, hd, at)
        torch.cuda.current_stream().synchronize()
    assert all(torch.equal(a, b) for a, b in zip(other, want))
    keys, vals = want[1][:at + 1].double().repeat_interleave(Hq // Hkv, 1), want[2][:at + 1].double().repeat_interleave(Hq // Hkv, 1)
    q = qkv[:Hq * hd].double().view(Hq, hd)
    p = torch.softmax(torch.einsum("hd,khd->hk", q, keys) * hd ** -0.5, -1)
    exact = torch.einsum("hk,khd->hd", p, vals).reshape(-1)
    assert float((want[0].double() - exact).abs().max()) <= 2.0 ** -7 * float(vals.abs().max())
    assert torch.equal(want[1][at], qkv[Hq * hd:(Hq + Hkv) * hd].view(Hkv, hd)) and torch.equal(want[2][at], qkv[(Hq + Hkv) * hd:].view(Hkv, hd))


def test_result_off_the_boundary(built_lib):
    from tinygpt_b200._lib import lib
    qkv, k, v = _inputs(4, 2, 64, 600)
    want = _call(qkv, k, v, 4, 2, 64, 555)[0]
    ws = torch.full((lib().b200_attn_decode_workspace_bytes(4, 2, 64, 600),), 0xa5, dtype=torch.uint8, device="cuda")
    buf, pos = torch.zeros(4 * 64 + 4, dtype=torch.bfloat16, device="cuda"), torch.tensor([555], dtype=torch.int32, device="cuda")
    for off in (1, 2, 4):
        out = buf[off:off + 256]
        rc = lib().b200_attn_decode_bf16(out.data_ptr(), qkv.data_ptr(), None, None, 0.0, None, pos.data_ptr(), 0, k.data_ptr(), v.data_ptr(), 4, 2, 64, 600,
                                         ws.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        assert torch.equal(out, want) and bool((ws == 0xa5).all())


def test_captured(built_lib):
    qkv, k, v = _inputs(16, 8, 128, 256)
    pos = torch.tensor([200], dtype=torch.int32, device="cuda")
    f = lambda: ops.attn_decode(qkv, k, v, q_heads=16, kv_heads=8, head_dim=128, pos=pos)
    want = f()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        f()
    torch.cuda.current_stream().wait_stream(s)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = f()
    for _ in range(3):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)
