"""Borrowed scale tensors on boundaries smaller than the tensor-core tiles load (needs a B200)."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, StrataMoeError, synth

pytestmark = pytest.mark.gpu


def shifted(t, offset):
    """A copy of t whose rows start `offset` bytes behind a 256-byte boundary."""
    pitch = (t.shape[1] + offset + 255) // 256 * 256
    buf = torch.zeros(t.shape[0] * pitch, dtype=torch.uint8, device=t.device)
    rows = buf.view(t.shape[0], pitch)[:, offset:offset + t.shape[1]]
    rows.copy_(t)
    return rows


def forward(ctx, cfg, layer):
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    out = ml.forward(layer.x)
    ctx.synchronize()
    ml.close()
    return out


# A 256-column block of a row has 8 (MXFP4), 16 (NVFP4) or 4 (INT4) scale bytes, which the tile decoders take in one load
# when rows are whole blocks and in two when they are not (384 columns).
@pytest.mark.parametrize("fmt,offset,cols,tiles", [
    (synth.FMT_MXFP4, 1, 512, False), (synth.FMT_MXFP4, 4, 512, False), (synth.FMT_MXFP4, 8, 512, True),
    (synth.FMT_MXFP4, 4, 384, True), (synth.FMT_NVFP4, 2, 512, False), (synth.FMT_NVFP4, 8, 512, False),
    (synth.FMT_NVFP4, 8, 384, True), (synth.FMT_INT4, 2, 512, False), (synth.FMT_INT4, 2, 384, True),
    (synth.FMT_INT4, 4, 512, True)])
@pytest.mark.parametrize("T", [9, 400])      # 2 rows per expert: paired tiles, 100: single-f16 tiles
def test_scales_off_the_tile_boundary(fmt, offset, cols, tiles, T, monkeypatch):
    """The layer gives the bits of the path its scales allow: the tiles', or the weight-streaming kernels'."""
    ctx = MoeContext(0)
    monkeypatch.setenv("STRATA_MOE_NO_STREAM_RING", "1")
    monkeypatch.setenv("STRATA_MOE_PAIR_NTILE", "16")
    cfg = synth.MoeConfig(f"shift{fmt}_{cols}", H=cols, I=cols, E=8, k=2, fmt=fmt, T=T, seed=3)
    layer = synth.build_layer(cfg, "cuda")
    on_tiles = forward(ctx, cfg, layer)
    with monkeypatch.context() as m:
        m.setenv("STRATA_MOE_NO_PREFILL_PATH", "1")
        streamed = forward(ctx, cfg, layer)
    assert not torch.equal(on_tiles, streamed)
    layer.scales = {role: shifted(s, offset) for role, s in layer.scales.items()}
    assert torch.equal(forward(ctx, cfg, layer), on_tiles if tiles else streamed)


@pytest.mark.parametrize("fmt", [synth.FMT_NVFP4, synth.FMT_INT4])
def test_odd_scale_addresses_are_refused(fmt):
    cfg = synth.MoeConfig("odd", H=256, I=128, E=2, k=1, fmt=fmt, T=2, seed=1)
    layer = synth.build_layer(cfg, "cuda")
    layer.scales["up"] = shifted(layer.scales["up"], 1)
    with pytest.raises(StrataMoeError, match="2-byte aligned"):
        MoeLayer(MoeContext(0), cfg).load_synth(layer)
