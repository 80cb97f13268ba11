"""Outputs of the linear scan with a removal leave beside the next four tokens' steps: sequences that end with none, some or all of four on their way,
inside a chunk of sixteen and at its end, in one go and cut in two, give the same bits; and against the recurrence in 64 bits (the bound of
test_scan_removal_gpu: 2e-5 of the largest value)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,dk,dv,scalar", [(2, 32, 17, False), (3, 64, 16, True), (1, 65, 33, False), (2, 128, 30, True), (2, 128, 16, False)])
@pytest.mark.parametrize("n", [1, 3, 4, 7, 16, 20, 23, 32, 37])
def test_in_one_go_and_cut(built_lib, H, dk, dv, scalar, n):
    from tinygpt_b200 import ops
    g = torch.Generator().manual_seed(n * 100 + dk)
    key = torch.nn.functional.normalize(torch.randn(n, H, dk, generator=g), dim=-1)
    cols = dict(d=torch.exp(-0.5 * torch.rand(n, H, 1 if scalar else dk, generator=g)), p=torch.rand(n, H, 1, generator=g) * key, q=key,
                b=torch.randn(n, H, dk, generator=g) * 0.3, r=torch.randn(n, H, dk, generator=g) * 0.3, v=torch.randn(n, H, dv, generator=g))
    big = torch.cat([t.reshape(n, -1) for t in cols.values()], 1).cuda()

    def run(state, a, b):
        views, at = {}, 0
        for k, t in cols.items():
            views[k], at = big[a:b, at:at + t[0].numel()], at + t[0].numel()
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        return ops.stack_lin_scan(views["d"], views["b"], views["r"], views["v"], state, i32([0]), i32([b - a]), i32([0] * (b - a)), i32(list(range(a, b))),
                                  heads=H, dk=dk, dv=dv, p=views["p"], q=views["q"])

    whole_s = torch.zeros(1, H * dk * dv, device="cuda")
    whole = run(whole_s, 0, n)
    for cut in {1, n // 2, n - 1} - {0, n}:
        s = torch.zeros_like(whole_s)
        assert torch.equal(torch.cat([run(s, 0, cut), run(s, cut, n)]), whole) and torch.equal(s, whole_s)
    x, S = {k: t.double() for k, t in cols.items()}, torch.zeros(H, dk, dv, dtype=torch.float64)
    want = torch.empty(n, H, dv, dtype=torch.float64)
    for t in range(n):
        S = x["d"][t][..., None] * S - x["p"][t][..., None] * torch.einsum("hk,hkv->hv", x["q"][t], S)[:, None] + x["b"][t][..., None] * x["v"][t][:, None]
        want[t] = torch.einsum("hk,hkv->hv", x["r"][t], S)
    assert float((whole.cpu().double().reshape(want.shape) - want).abs().max() / want.abs().max()) < 2e-5
