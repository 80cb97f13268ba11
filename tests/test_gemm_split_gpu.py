"""The GEMM kernels that pick_gemm chooses between (csrc/gemm.cu), at the edges of their tiles: row counts around 8, 64, 128 and 256, short
and long K (whole, split over 2 … 8 CTAs, ragged last k-block), N short of a tile.  Reference: fp32 matmul of the same bf16
operands.  One bf16 rounding of an fp32 sum, whose own error against another order of K products is far below half a bf16 ulp: at
most one ulp apart, 97 % identical (the gate of test_gemm_gpu.py)."""
import pytest
import torch

from helpers import assert_close_bf16
from tinygpt_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rand(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("M", [1, 7, 9, 64, 65, 127, 129, 255, 257, 300, 700])
@pytest.mark.parametrize("N,K", [(136, 4104), (1152, 896), (2048, 6144), (3072, 1032), (8200, 512)])
def test_gemm_edges(built_lib, M, N, K):
    a, w = rand(M, K, seed=M + K), rand(N, K, seed=N, scale=0.02)
    got = ops.gemm(a, w)
    want = (a.float() @ w.float().t()).to(torch.bfloat16)
    assert torch.equal(got, ops.gemm(a, w))            # the sum's order is fixed
    assert_close_bf16(got.float().cpu(), want.float().cpu(), 1, f"gemm {M}x{N}x{K}", atol=1e-4, frac_exact=0.97)


@pytest.mark.parametrize("side", ["tile", "wide"])
@pytest.mark.parametrize("M", [1, 9, 40, 127, 129, 300])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 520), (264, 2048), (1032, 896)])
def test_one_tile_per_cta(built_lib, monkeypatch, side, M, N, K):
    """Whole K on one CTA, tiles of 128 and of 256 columns: ragged rows, columns and last k-block, rows and columns outside left alone."""
    from tinygpt_b200._lib import check, lib
    monkeypatch.setenv("B200_GEMM", side)
    a, w = rand(M, K, seed=M + K), rand(N, K, seed=N, scale=0.02)
    buf = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)
    check(lib().b200_gemm_bf16(buf.data_ptr(), a.data_ptr(), w.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream), "gemm")
    want = (a.float() @ w.float().t()).to(torch.bfloat16)
    assert_close_bf16(buf[:M].float().cpu(), want.float().cpu(), 1, f"gemm {M}x{N}x{K}", atol=1e-4, frac_exact=0.95)
    assert bool((buf[M:] == 7.0).all())


def test_more_rows_than_a_grid_has_rows_of_tiles(built_lib, monkeypatch):
    """8.4 M rows and a few: the one-tile kernel's grid ends there, whatever was asked for."""
    monkeypatch.setenv("B200_GEMM", "tile")
    M = 65535 * 128 + 9
    a, w = rand(M, 8, seed=1), rand(8, 8, seed=2)
    got = ops.gemm(a, w)
    tail = slice(M - 300, M)
    assert_close_bf16(got[tail].float().cpu(), (a[tail].float() @ w.float().t()).to(torch.bfloat16).float().cpu(), 1, "gemm", atol=1e-4, frac_exact=0.97)
    assert torch.equal(got[:128], ops.gemm(a[:128], w))


def test_rows_outside_are_left_alone(built_lib):
    """Only rows below M and columns below N are written."""
    from tinygpt_b200._lib import check, lib
    M, N, K = 70, 264, 2048
    buf = torch.full((M + 2, N), 7.0, dtype=torch.bfloat16, device=DEV)
    a, w = rand(M, K, seed=1), rand(N, K, seed=2, scale=0.02)
    check(lib().b200_gemm_bf16(buf.data_ptr(), a.data_ptr(), w.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream), "gemm")
    assert bool((buf[M:] == 7.0).all())
    assert torch.equal(buf[:M], ops.gemm(a, w))
