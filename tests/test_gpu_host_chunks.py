"""Host-buffer calls in token chunks whose size another expert path would take: the bits of the device call (needs a B200)."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth

pytestmark = pytest.mark.gpu


# 32 experts, top-4; the digit planes take up to 24 rows per expert.  600 tokens: 75 rows in one piece, 18.75 in four chunks, 25 in
# three; 385: 48 and 16; 384: 48 and 24; 192: 24 and 12, planes either way
@pytest.mark.parametrize("fmt", [synth.FMT_MXFP4, synth.FMT_NVFP4])
@pytest.mark.parametrize("T,chunks", [(600, 4), (600, 3), (385, 3), (384, 2), (192, 2)])
def test_same_bits_as_on_the_device(fmt, T, chunks, monkeypatch):
    monkeypatch.setenv("STRATA_MOE_HOST_CHUNKS", str(chunks))
    cfg = synth.MoeConfig(f"chunks{fmt}_{T}", H=512, I=512, E=32, k=4, fmt=fmt, T=T, seed=12)
    ctx = MoeContext(0)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    x = layer.x.cpu().pin_memory()
    out = torch.empty(T, cfg.H, dtype=torch.float32, pin_memory=True).fill_(float("nan"))
    want = ml.forward(layer.x)
    ctx.synchronize()
    for _ in range(2):
        ml.forward_host(x, out)
    assert torch.equal(out.cuda(), want)
    ctx.check_canaries()
