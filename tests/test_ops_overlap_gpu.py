"""Operators launched beside the end of the one in front (programmatic dependent launch): what each reads was written by the operator, or the torch
kernel, right before it — activations, weights, caches and positions alike.  Against the same calls with a synchronisation between, bit for bit."""
import pytest
import torch

from tinygpt_b200 import engine, models, ops, stack_bench

pytestmark = pytest.mark.gpu


def maker(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s, k=1.0: (torch.randn(*s, generator=g, device="cuda") * k).to(torch.bfloat16)


@pytest.mark.parametrize("rows", [1, 2, 7, 16, 40, 130, 300, 1000])
def test_chain_of_operators(built_lib, rows):
    r = maker(3)
    x0 = r(rows, 512)
    layers = [(r(2048, 512, k=.04), r(512, 1024, k=.03), r(512, k=.1) + 1, r(512, 512, k=.04)) for _ in range(4)]
    kc, vc = r(1, 700, 2, 64), r(1, 700, 2, 64)

    def chain(sync):
        def s(t):
            if sync:
                torch.cuda.synchronize()
            return t
        x = x0
        for w1, w2, n, wq in layers:
            h = s(ops.rms_norm(x, n, 1e-6))
            h = s(ops.gemm(h, w1)) if rows > 8 else s(ops.linear(h, w1))
            x = s(ops.add(x, s(ops.linear(s(ops.silu_mul(h)), w2))))
            q = s(ops.linear(x, wq)).view(1, rows, 8, 64)
            x = s(ops.add(x, s(ops.flash_attention(q, q[:, :, :4], q[:, :, 4:], True)).view(rows, -1)))
            if rows == 1:
                y = s(ops.gemv_fused(x.view(-1), w1, norm_weight=n, eps=1e-6, silu_mul=True))
                x = s(ops.gemv_fused(y, w2, residual=x.view(-1))).view(1, -1)
                x = s(ops.add(x, s(ops.flash_attention(x.view(1, 1, 8, 64), kc, vc)).view(1, -1)))
        return x

    want = chain(True)
    assert bool(torch.isfinite(want.float()).all())
    for _ in range(20):
        assert torch.equal(chain(False), want)


def test_weights_that_were_just_written(built_lib):
    r = maker(4)
    for rows in (1, 8, 300):
        w, x = r(1152, 896), r(rows, 896)
        want = ops.linear(x, w + w), ops.linear(x, w)
        torch.cuda.synchronize()
        for _ in range(30):
            w2 = ops.add(w, w)               # an operator in front
            a = ops.linear(x, w2)
            w2.mul_(0.5)                     # a torch kernel in front
            assert torch.equal(a, want[0]) and torch.equal(ops.linear(x, w2), want[1])


@pytest.mark.parametrize("ctx", [512, 2304])
def test_decode_steps_behind_each_other(built_lib, ctx):
    """Each step appends the row that the next one reads, at a position written right before it."""
    r = maker(5)
    kc, vc, qkv = r(ctx, 2, 64), r(ctx, 2, 64), r(10 * 64)

    def steps(sync):
        k, v, out, x = kc.clone(), vc.clone(), [], qkv
        for t in range(30):
            pos = torch.tensor([200 + t], dtype=torch.int32, device="cuda")
            x = ops.add(x, qkv) if t % 2 else qkv
            if sync:
                torch.cuda.synchronize()
            out.append(ops.attn_decode(x, k, v, q_heads=6, kv_heads=2, head_dim=64, pos=pos))
        return torch.stack(out), k, v

    want = steps(True)
    for _ in range(10):
        assert all(torch.equal(a, b) for a, b in zip(steps(False), want))


def test_captured_operators_have_plain_edges(built_lib):
    """A captured graph ends with the operators' own kernels: what is enqueued behind its launch sees their results."""
    r = maker(6)
    x, w = r(8, 2048), r(4096, 2048, k=.02)
    want = ops.linear(x, w)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            y = ops.linear(ops.add(x, x), w)
        for i in range(50):
            y.zero_()
            graph.replay()
            assert torch.equal(y.clone(), ops.linear(x + x, w)), i
    torch.cuda.synchronize()
    assert torch.equal(ops.linear(x, w), want)


def test_operators_right_behind_a_graph(built_lib):
    """An operator, and no torch kernel, is the first thing behind a graph's launch: it sees what the graph's last kernel has written, be that an operator's, a
    torch kernel's or the engine's."""
    r = maker(7)
    x, w, n = r(8, 2048), r(4096, 2048, k=.02), r(2048, k=.1) + 1
    xs = [r(8, 2048) for _ in range(20)]
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        want = [(ops.linear(t + t, w), ops.rms_norm(t + t, n, 1e-6), ops.add(t + t, t + t)) for t in xs]
        ends = []
        for end in (ops.add, torch.add):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st):
                y = end(x, x)
            ends.append((graph, y))
        torch.cuda.synchronize()
        for graph, y in ends:
            for t, (lin, norm, both) in zip(xs, want):
                for call, expect in ((lambda: ops.linear(y, w), lin), (lambda: ops.rms_norm(y, n, 1e-6), norm), (lambda: ops.add(y, y), both)):
                    x.copy_(t)
                    y.zero_()
                    graph.replay()
                    assert torch.equal(call(), expect)


def test_engine_and_operators_without_a_kernel_between(built_lib):
    """Operators right behind a decode step's graph read its logits; a prompt right behind the operator that wrote its ids."""
    spec = models.TINY_QWEN2
    eng = engine.DecodeEngine(spec, {k: v.to("cuda") for k, v in models.synth_weights(spec, seed=3, std=0.05).items()})
    attn = models.AttnSpec(4, 2, 64, 64, 0.125, 0, 0)
    stack = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=spec.vocab, layers=(models.StackLayerSpec(attn, 512),) * 2, embed_scale=4.0,
                             residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=256, max_slots=1)
    other = engine.DecodeEngine(stack, stack_bench.device_stack_weights(stack, torch.device("cuda"), 8))
    r = maker(8)
    for i in range(10):
        rows = r(40, spec.vocab)
        ids = ops.argmax(rows, keepdim=False).view(1, -1)
        torch.cuda.synchronize()
        for e in (eng, other):
            e.reset_cache()
            want = e.forward(ids).clone()
            step = e.forward(ids[:, -1:]).clone()
            torch.cuda.synchronize()
            e.reset_cache()
            got = e.forward(ops.argmax(rows, keepdim=False).view(1, -1))
            assert torch.equal(got, want), i
            logits = e.forward(ids[:, -1:])
            twice = ops.add(logits, logits)
            assert torch.equal(logits, step) and torch.equal(twice, step + step), i
    eng.close()
    other.close()


def test_the_switch_turns_operators_overlap_off(built_lib):
    """B200_NO_PDL=1 in a process of its own: device time of calls queued behind each other, the best of many runs.  With overlap a call's launch, barriers and tensor
    memory lie beside the end of the call in front (4.1 µs a call, 6.2 without)."""
    import os
    import subprocess
    import sys
    code = """
import torch
from tinygpt_b200 import ops
q, k = torch.randn(1, 1, 16, 128, device="cuda").bfloat16(), torch.randn(1, 300, 8, 128, device="cuda").bfloat16()
best = 1e9
for _ in range(30):
    a, b = torch.cuda.Event(True), torch.cuda.Event(True)
    torch.cuda.synchronize()
    torch.cuda._sleep(3000000)   # the calls are queued meanwhile
    a.record()
    for _ in range(200):
        ops.flash_attention(q, k, k)
    b.record()
    b.synchronize()
    best = min(best, a.elapsed_time(b))
print(best)
"""
    took = [float(subprocess.run([sys.executable, "-c", code], env=dict(os.environ, B200_NO_PDL=off), capture_output=True, text=True, check=True).stdout)
            for off in ("0", "1")]
    assert took[1] > 1.2 * took[0], took
