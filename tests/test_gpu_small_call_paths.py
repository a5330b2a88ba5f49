"""Which kernels small calls take: weight streaming where tiles would leave most SMs idle, tiles beyond (needs a B200).

The two paths sum in different orders, so the bits of a call tell which one served it."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth
from tests import helpers as Hh

pytestmark = pytest.mark.gpu

MX, NV, I4 = synth.FMT_MXFP4, synth.FMT_NVFP4, synth.FMT_INT4


@pytest.fixture(scope="module")
def ctx():
    return MoeContext(0)


def run(ctx, cfg, layer, grouped):
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    if grouped:
        ids, _ = ml.route(layer.x)
        _, offsets, perm = ml.group(ids)
        out = ml.experts_grouped(ml.gather_rows(layer.x, perm, cfg.k), offsets)
    else:
        out = ml.forward(layer.x)
    ctx.synchronize()
    ml.close()
    return out


# (format, H, I, E, k, T, stage call, streams): each line of the rule from both sides
@pytest.mark.parametrize("fmt,H,I,E,k,T,grouped,streams", [
    (MX, 1536, 128, 16, 2, 16, False, True), (MX, 1536, 128, 16, 2, 17, False, False),
    (MX, 1536, 768, 128, 8, 8, False, True), (MX, 1536, 768, 128, 8, 16, False, False),     # 303 and 486 tiles of 3 x 148
    (NV, 1408, 128, 32, 2, 64, False, True), (NV, 1408, 128, 32, 2, 65, False, False),
    (I4, 1536, 128, 16, 2, 16, False, True), (I4, 1536, 128, 16, 2, 17, False, False),
    (I4, 1408, 128, 32, 2, 64, False, True), (I4, 1408, 128, 32, 2, 65, False, False),
    (I4, 2048, 1408, 64, 6, 3, False, True), (I4, 2048, 1408, 64, 6, 6, False, False),      # 178 and 305 tiles
    (MX, 1024, 384, 32, 4, 33, True, True), (MX, 1024, 384, 64, 4, 33, True, False),
    (I4, 1024, 384, 32, 4, 33, True, True), (I4, 1536, 384, 32, 4, 33, True, False)])
def test_small_call_path(ctx, fmt, H, I, E, k, T, grouped, streams, monkeypatch):
    monkeypatch.setenv("STRATA_MOE_NO_STREAM_RING", "1")
    cfg = synth.MoeConfig(f"path{fmt}_{H}_{E}_{T}", H=H, I=I, E=E, k=k, fmt=fmt, T=T, norm_init=1e-20, seed=13)
    layer = synth.build_layer(cfg, "cuda")
    got = run(ctx, cfg, layer, grouped)
    with monkeypatch.context() as m:
        m.setenv("STRATA_MOE_NO_PAIR_TILES", "1")
        streamed = run(ctx, cfg, layer, grouped)
    with monkeypatch.context() as m:
        m.setenv("STRATA_MOE_PAIR_NTILE", "64")
        on_tiles = run(ctx, cfg, layer, grouped)
    assert not torch.equal(streamed, on_tiles)
    assert torch.equal(got, streamed if streams else on_tiles)
    # 22-bit (FP4) or 16-bit (INT4, general decoders) activation pairs and FP32 sums on either path
    rel, _ = Hh.error_metrics(streamed.cpu().numpy(), on_tiles.cpu().numpy())
    assert rel <= 1e-4, rel
