"""Host-buffer calls whose large result goes out in blocks of columns: the bits of the device call (needs a B200)."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth

pytestmark = pytest.mark.gpu


# 16 MB of result are the line (T * H * 4): 2048 tokens of 2048 columns reach it, 2047 do not; 1280 columns are no four blocks
@pytest.mark.parametrize("fmt,H,T,shared", [(synth.FMT_INT4, 2048, 2048, 0), (synth.FMT_INT4, 2048, 2047, 0), (synth.FMT_MXFP4, 2048, 2100, 256),
                                            (synth.FMT_NVFP4, 1280, 3300, 128)])
def test_same_bits_as_on_the_device(fmt, H, T, shared):
    cfg = synth.MoeConfig(f"columns{fmt}_{T}", H=H, I=256, E=4, k=2, fmt=fmt, T=T, I_shared=shared, seed=9, output_scale=2.5)
    ctx = MoeContext(0)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    x = layer.x.cpu().pin_memory()
    out = torch.empty(T, H, dtype=torch.float32, pin_memory=True).fill_(float("nan"))
    for _ in range(2):
        ml.forward_host(x, out)
    want = ml.forward(layer.x)
    ctx.synchronize()
    assert torch.equal(out.cuda(), want)
    ctx.check_canaries()
