"""Which calls the native operators (csrc/torch_ops.cpp) take themselves, and that all others go ops.py's own way: same results, same errors."""
import pytest
import torch

from tinygpt_b200 import ops
from tinygpt_b200._lib import B200Error

BF16 = torch.bfloat16


def test_cpu_tensors_are_refused(built_lib):
    x, w = torch.zeros(2, 8, dtype=BF16), torch.zeros(8, 8, dtype=BF16)
    assert ops._fast.linear(x, w, None) is None and ops._fast.add(x, x) is None and ops._fast.linear(x, 3, None) is None
    for call in (lambda: ops.linear(x, w), lambda: ops.gemm(x, w), lambda: ops.rms_norm(x, None, 1e-6), lambda: ops.silu_mul(x),
                 lambda: ops.add(x, x), lambda: ops.flash_attention(*[x.view(1, 1, 2, 8)] * 3), lambda: ops.gemv_fused(x, w)):
        with pytest.raises(B200Error, match="CUDA device"):
            call()


def test_a_library_under_another_name_and_place(built_lib, tmp_path):
    """B200_LIB names the library that the native operators call too; no other is loaded, and nothing need lie beside it."""
    import os
    import shutil
    import subprocess
    import sys
    other = tmp_path / "other_name.so"
    shutil.copy(built_lib, other)
    code = """
import torch
from tinygpt_b200 import ops
from tinygpt_b200._lib import B200Error
x = torch.zeros(2, 8, dtype=torch.bfloat16)
assert ops._fast.linear(x, x, None) is None and ops._fast.attn_decode(x, x, x, 1, 1, 64, None, 1, None, None, None, 0.0) is None
maps = open("/proc/self/maps").read()
assert "other_name.so" in maps and "libb200decode.so" not in maps
"""
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, B200_LIB=str(other)), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.gpu
class TestOnDevice:
    def setup_method(self):
        g = torch.Generator(device="cuda").manual_seed(1)
        self.r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF16)

    def test_plain_calls_are_taken(self, built_lib):
        x, w, b = self.r(3, 2, 64), self.r(40, 64), self.r(40)
        y = ops._fast.linear(x, w, b)
        assert y.shape == (3, 2, 40) and torch.equal(y, ops.linear(x, w, b))
        assert ops._fast.linear(x[0, 0], w, None).shape == (40,)
        assert torch.equal(ops._fast.linear(x, torch.nn.Parameter(w), b), y) and not ops.linear(x, torch.nn.Parameter(w), b).requires_grad
        want = x.double() @ w.double().t() + b.double()
        assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -7

    def test_other_calls_go_the_python_way(self, built_lib):
        x, w = self.r(64, 6), self.r(40, 64)
        assert ops._fast.linear(x.t(), w, None) is None and torch.equal(ops.linear(x.t(), w), ops.linear(x.t().contiguous(), w))
        assert ops._fast.linear(x.t(), w, None) is None and ops._fast.rms_norm(x, None, 1) is None
        assert torch.equal(ops.rms_norm(x, None, 1), ops.rms_norm(x, None, 1.0))
        a = self.r(4, 8)
        assert torch.equal(ops.add(a[:, :4], a[:, 4:]), a[:, :4] + a[:, 4:])

        class Sub(torch.Tensor):
            pass

        assert ops._fast.add(a.as_subclass(Sub), a) is None
        with torch.overrides.TorchFunctionMode():
            assert ops._fast.add(a, a) is None
        assert ops._fast.add(a, a) is not None

    def test_what_was_refused_stays_refused(self, built_lib):
        x, w = self.r(2, 64), self.r(40, 64)
        for call in (lambda: ops.linear(x.float(), w), lambda: ops.linear(x, w.half()), lambda: ops.linear(x[:, :56], w), lambda: ops.silu_mul(x[:, :63]),
                     lambda: ops.add(x, w), lambda: ops.linear(x.view(-1)[1:65].view(1, 64), w), lambda: ops.gemm(self.r(2, 60), self.r(40, 60))):
            with pytest.raises(B200Error):
                call()
        with pytest.raises(RuntimeError):   # a batched tensor has no address
            torch.vmap(lambda t: ops.add(t, t))(x)
        from torch._subclasses.fake_tensor import FakeTensorMode
        with FakeTensorMode(allow_non_fake_inputs=True) as mode:
            fake = mode.from_tensor(x)
            assert ops._fast.add(fake, fake) is None

    def test_capture_streams_and_the_allocator(self, built_lib):
        x, w = self.r(5, 64), self.r(40, 64)
        want = ops.linear(x, w)
        st = torch.cuda.Stream()
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            assert torch.equal(ops.linear(x, w), want)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st):
                y = ops.linear(x, w)
            x.copy_(x.flip(0))
            graph.replay()
            assert torch.equal(y, want.flip(0))
        torch.cuda.synchronize()
        seen = []
        from torch.utils._python_dispatch import TorchDispatchMode

        class Watch(TorchDispatchMode):
            def __torch_dispatch__(self, func, types, args=(), kwargs=None):
                seen.append(func)
                return func(*args, **(kwargs or {}))

        with Watch():
            ops.linear(x, w)
        assert any("empty" in str(f) for f in seen)
