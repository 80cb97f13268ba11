"""The new token's row in the shared-memory ring of attn_row_kernel (csrc/attn.cu).  The copies of a partly filled unit write zeros where it belongs, from a
lane that is not the one which stores it at most places: every place among a warp's sixteen keys, of the first and of later units, with a key that outweighs all others,
so that the result is its value to the bit.  A lost key leaves the cached ones' mean, a lost value zeros."""
import pytest
import torch

from test_attn_row_gpu import DEV, randn
from tinygpt_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [1, 640, 4000])
@pytest.mark.parametrize("Hq,Hkv,D", [(14, 2, 64), (16, 8, 128), (3, 3, 128)])
def test_every_place(built_lib, first, Hq, Hkv, D):
    kc, vc = randn(4160, Hkv, D, seed=1, std=0.1), randn(4160, Hkv, D, seed=2)
    v = randn(Hkv, D, seed=3)
    qkv = torch.cat([torch.full(((Hq + Hkv) * D,), 2.0, dtype=v.dtype, device=DEV), v.view(-1)])   # scores of 32 and more, the others' below 2
    want = v.repeat_interleave(Hq // Hkv, 0).view(-1)
    for at in range(first, first + 64):
        pos = torch.tensor([at], dtype=torch.int32, device=DEV)
        for _ in range(3):
            got = ops.attn_decode(qkv, kc.clone(), vc.clone(), q_heads=Hq, kv_heads=Hkv, head_dim=D, pos=pos)
            assert torch.equal(got, want), at
