"""ops.linear over 1 … 40 rows: one row (weight stream), up to eight rows per pass over the weights, two passes, the GEMM — at the edges between
them, with n that is no multiple of 8, k that leaves the last 256-column piece ragged, rows too long to share a pass, and a bias as the second
rounding.  Reference: fp32 matmul, rounded, bias added, rounded.  Another order of the fp32 sum: one bf16 ulp (1e-4 near zero) without a bias, two
ulps (1e-2 near zero, an ulp of the larger term) with one, 95 % identical."""
import pytest
import torch

from helpers import assert_close_bf16
from tinygpt_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rand(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 15, 16, 17, 40])
@pytest.mark.parametrize("n,k", [(1152, 896), (13, 72), (4096, 2048), (897, 4864), (64, 14344), (24, 40960)])
@pytest.mark.parametrize("bias", [False, True])
def test_rows(built_lib, m, n, k, bias):
    x, w = rand(m, k, seed=m), rand(n, k, seed=n, scale=k ** -0.5)
    b = rand(n, seed=3) if bias else None
    got = ops.linear(x, w, b)
    want = (x.float() @ w.float().t()).to(torch.bfloat16)
    if bias:
        want = want + b
    # a sum that rounds to the other neighbour moves the rounded sum with the bias by at most one ulp of the larger of the two
    assert_close_bf16(got.float().cpu(), want.float().cpu(), 1 if not bias else 2, f"linear {m}x{n}x{k}", atol=1e-2 if bias else 1e-4, frac_exact=0.95)
    guard = torch.full((m + 1, n), 3.0, dtype=torch.bfloat16, device=DEV)
    from tinygpt_b200._lib import check, lib
    check(lib().b200_gemv_bf16(guard.data_ptr(), x.data_ptr(), w.data_ptr(), b.data_ptr() if bias else None, m, n, k,
                               torch.cuda.current_stream().cuda_stream), "gemv")
    assert torch.equal(guard[:m], got) and bool((guard[m:] == 3.0).all())


@pytest.mark.parametrize("m", [1, 5, 40])
def test_rows_off_a_16_byte_boundary_are_refused(built_lib, m):
    """x is read 16 bytes at a time: a view that starts elsewhere is an error on the host."""
    from tinygpt_b200._lib import B200Error
    x, w = rand(m * 72 + 1, seed=1)[1:].view(m, 72), rand(13, 72, seed=2)
    with pytest.raises(B200Error, match="aligned"):
        ops.linear(x, w)
    assert torch.equal(ops.linear(x.clone(), w), ops.linear(x.clone(), w))
