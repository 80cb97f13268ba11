"""One query row over many keys (csrc/attn.cu attn_row_kernel) against fp64: every size of a head group, one to sixteen CTAs per cluster, key counts
around a warp's sixteen, a unit of 128 and a ring's worth of units, and the fused decode form, whose new key may be the first of a warp, of a
unit and of a CTA.  Probabilities are fp32, the result bf16: 2-norm error below 2⁻⁸."""
import pytest
import torch

from test_attn_row_gpu import DEV, attend, randn
from tinygpt_b200 import ops

pytestmark = pytest.mark.gpu


# heads of a group 1, 2, 3, 5, 6, 8 (and 12: two groups of six); sequences · groups of 2 … 160: clusters of 16, 8, 4, 2 and 1
@pytest.mark.parametrize("B,Hq,Hkv", [(1, 2, 2), (1, 6, 3), (6, 9, 3), (20, 10, 2), (10, 12, 2), (5, 24, 2), (20, 16, 2), (160, 2, 1)])
@pytest.mark.parametrize("n", [1, 16, 17, 127, 129, 400, 1600])
@pytest.mark.parametrize("D", [64, 128])
def test_groups_and_clusters(built_lib, B, Hq, Hkv, n, D):
    q, k, v = randn(B, 1, Hq, D, seed=n, std=2.0), randn(B, n, Hkv, D, seed=1), randn(B, n, Hkv, D, seed=2)
    got = ops.flash_attention(q, k, v, False)
    want = attend(q, k, v)
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
    assert torch.equal(got, ops.flash_attention(q, k, v, False))


@pytest.mark.parametrize("at", [0, 1, 15, 16, 17, 127, 128, 255, 256, 2047, 2048, 2300])
@pytest.mark.parametrize("Hq,Hkv,D", [(14, 2, 64), (6, 6, 128), (24, 8, 128), (64, 64, 64)])
def test_appended_key(built_lib, at, Hq, Hkv, D):
    """The cache holds NaNs behind the position: what lies there is never read."""
    ctx = 2304
    qkv = randn((Hq + 2 * Hkv) * D, seed=at, std=1.5)
    kc, vc = randn(ctx, Hkv, D, seed=6), randn(ctx, Hkv, D, seed=7)
    kc[at:], vc[at:] = float("nan"), float("nan")
    pos = torch.tensor([at], dtype=torch.int32, device=DEV)
    q, k, v = (t.view(1, 1, -1, D) for t in qkv.split([Hq * D, Hkv * D, Hkv * D]))
    want = attend(q, torch.cat([kc[None, :at], k], 1), torch.cat([vc[None, :at], v], 1)).reshape(-1)
    got = ops.attn_decode(qkv, kc, vc, q_heads=Hq, kv_heads=Hkv, head_dim=D, pos=pos)
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
    assert torch.equal(kc[at], k[0, 0]) and torch.equal(vc[at], v[0, 0])


def test_a_score_that_is_no_number(built_lib):
    """A NaN in one key, an infinity in another value: the heads that see them are not finite, the others keep their results."""
    q, k, v = randn(1, 1, 6, 64, seed=1), randn(1, 300, 3, 64, seed=2), randn(1, 300, 3, 64, seed=3)
    want = attend(q, k, v)
    k[0, 200, 0], v[0, 10, 1] = float("nan"), float("inf")
    got = ops.flash_attention(q, k, v, False)[0, 0].float()
    assert bool(got[:2].isnan().all()) and bool((got[2:4] == float("inf")).all())
    assert float((got[4:].double() - want[0, 0, 4:]).norm() / want[0, 0, 4:].norm()) < 2.0 ** -8
