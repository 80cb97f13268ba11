"""Linear scan with a removal against the recurrence in 64 bits, at the edges of its split: key sizes either side of each lane
layout, value sizes that end inside a column pair, a warp or a CTA, sequences that end inside a chunk or a group of four
tokens, rows that rule out 16-byte copies, both kinds of decay, and values scaled per head."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(H, dk, dv, lens, scalar, scaled, pad, carried):
    from tinygpt_b200 import ops

    g = torch.Generator().manual_seed(dk * 1000 + dv)
    n, dev = sum(lens), "cuda"
    key = torch.nn.functional.normalize(torch.randn(n, H, dk, generator=g), dim=-1)
    cols = dict(d=torch.exp(-0.5 * torch.rand(n, H, 1 if scalar else dk, generator=g)), p=torch.rand(n, H, 1, generator=g) * key, q=key,
                b=torch.randn(n, H, dk, generator=g) * 0.3, r=torch.randn(n, H, dk, generator=g) * 0.3, v=torch.randn(n, H, dv, generator=g))
    if scaled:
        cols["vscale"] = torch.rand(n, H, generator=g) + 0.1
    big = torch.cat([t.reshape(n, -1) for t in cols.values()] + [torch.zeros(n, pad)], 1).to(dev)
    views, at = {}, 0
    for k, t in cols.items():
        w = t[0].numel()
        views[k], at = big[:, at:at + w], at + w
    state0 = torch.randn(len(lens), H, dk, dv, generator=g) * 0.3
    state = state0.reshape(len(lens), -1).to(dev)
    first = 5 if carried else 0   # position 0 starts from nothing
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=dev)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    o = ops.stack_lin_scan(views["d"], views["b"], views["r"], views["v"], state, i32(starts), i32(lens),
                           i32([s for s, c in enumerate(lens) for _ in range(c)]), i32([first + t for c in lens for t in range(c)]),
                           heads=H, dk=dk, dv=dv, p=views["p"], q=views["q"], vscale=views.get("vscale"), share=1)
    x = {k: t.double() for k, t in cols.items()}
    want_o, want_s = torch.empty(n, H, dv, dtype=torch.float64), torch.empty(state0.shape, dtype=torch.float64)
    for s, c in enumerate(lens):
        S = state0[s].double() if carried else torch.zeros(H, dk, dv, dtype=torch.float64)
        for t in range(starts[s], starts[s] + c):
            v = x["v"][t] * (x["vscale"][t][:, None] if scaled else 1.0)
            rem = torch.einsum("hk,hkv->hv", x["q"][t], S)
            S = x["d"][t][..., None] * S - x["p"][t][..., None] * rem[:, None] + x["b"][t][..., None] * v[:, None]
            want_o[t] = torch.einsum("hk,hkv->hv", x["r"][t], S)
        want_s[s] = S
    return (o.cpu().double(), want_o.reshape(n, -1)), (state.cpu().double(), want_s.reshape(len(lens), -1))


CASES = [(2, 32, 16, [17], True), (2, 33, 17, [16, 1], False), (1, 64, 1, [5], False), (2, 65, 31, [33, 2, 4], True), (3, 128, 16, [48], False),
         (2, 127, 18, [49, 3], False), (1, 129, 33, [9, 8], True), (1, 256, 16, [26], False), (1, 260, 9, [13, 4], True), (1, 512, 8, [14], False),
         (2, 4, 3, [35], True)]


@pytest.mark.parametrize("H,dk,dv,lens,scalar", CASES)
@pytest.mark.parametrize("pad", [0, 3])
def test_removal_scan_at_the_edges(H, dk, dv, lens, scalar, pad):
    # A sum of dk products in fp32 rounds by about eps·sqrt(dk) of its size, and the decay (mean about 0.78) lets fewer than
    # ten tokens' errors add up: 10 · 6e-8 · sqrt(512) < 2e-5.
    for got, want in _run(H, dk, dv, lens, scalar, scaled=pad == 3, pad=pad, carried=pad == 3):
        assert torch.isfinite(got).all()
        assert float((got - want).abs().max() / want.abs().max()) < 2e-5
