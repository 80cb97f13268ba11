"""Which of the two prompt attentions a windowed layer takes by itself (prefill_attn_tc_wins in csrc/prefill_attn_tc.cu), told by the bits of its logits: heads of 64 with a
narrow window, or with blocks that just fill the SMs, stay with mma.sync; wider windows, more blocks and heads of 128 take tcgen05."""
import pytest
import torch

from tinygpt_b200 import engine, models, stack_bench

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,rows,window,keep,tc", [
    (24, 64, 1024, 16, 0, False), (24, 64, 1024, 64, 0, False), (14, 64, 2048, 64, 4, False), (14, 64, 2048, 100, 4, False), (14, 64, 2048, 130, 64, False),
    (14, 64, 2048, 256, 4, True), (24, 64, 1024, 130, 64, True), (16, 64, 2048, 100, 4, True), (24, 64, 512, 256, 4, True), (24, 64, 512, 0, 0, True), (16, 128, 2048, 16, 0, True)])
def test_windowed_layer(built_lib, monkeypatch, heads, dim, rows, window, keep, tc):
    attn = models.AttnSpec(heads, 2, dim, dim, dim ** -0.5, window, keep)
    spec = models.StackSpec(name="w", architecture="Kozusun", width=256, vocab=500, layers=(models.StackLayerSpec(attn, 128),), embed_scale=4.0,
                            residual_mult=0.5, norm_eps=1e-5, norm_offset=1.0, max_ctx=rows, max_slots=1)
    eng = engine.DecodeEngine(spec, stack_bench.device_stack_weights(spec, torch.device("cuda"), 8))
    ids = torch.randint(0, 500, (1, rows), generator=torch.Generator().manual_seed(9)).cuda()
    out = {}
    for side in ("", "tc", "mma"):
        monkeypatch.setenv("B200_ATTN_TC", side) if side else monkeypatch.delenv("B200_ATTN_TC", raising=False)
        eng.reset_cache()
        out[side] = eng.forward(ids, True)
    eng.close()
    assert not torch.equal(out["tc"], out["mma"])
    assert torch.equal(out[""], out["tc" if tc else "mma"])
