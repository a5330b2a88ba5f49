"""Large results of host-buffer calls: in four blocks of columns into page-locked memory, in one piece into any other (needs a B200)."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth

pytestmark = pytest.mark.gpu


def launches(ctx, call):
    before = ctx.stats().kernel_launches
    call()
    ctx.synchronize()
    return ctx.stats().kernel_launches - before


@pytest.mark.parametrize("T,pinned,blocks", [(2048, True, 4), (2048, False, 1), (2047, True, 1)])      # 16 MB are the line
def test_launches_and_bits(T, pinned, blocks):
    cfg = synth.MoeConfig(f"pageable{T}", H=2048, I=256, E=4, k=2, fmt=synth.FMT_INT4, T=T, seed=9)
    ctx = MoeContext(0)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    x, out = layer.x.cpu(), torch.empty(T, cfg.H)
    if pinned:
        x, out = x.pin_memory(), out.pin_memory()
    want = ml.forward(layer.x)
    ctx.synchronize()
    on_device = launches(ctx, lambda: ml.forward(layer.x))
    on_host = launches(ctx, lambda: ml.forward_host(x, out))
    assert on_host == on_device + 2 * (blocks - 1)      # the down projection and the combine of every block
    assert torch.equal(out.cuda(), want)
