"""Tile geometries of the tensor-core expert kernel at their edges, against the CPU oracle (needs a B200)."""
import numpy as np
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth
from tests import helpers as Hh

pytestmark = pytest.mark.gpu

# One f16 rounding per SwiGLU output and, for the formats with a block scale, one per decoded weight (2^-12 each, a sum
# of independent errors): 1e-3 holds all of it.  BF16 experts carry the SwiGLU output as a BF16 pair (2^-17): what is
# left is FP32 summation order.
TOL_F16, TOL_PAIR = 1e-3, 1e-4


@pytest.fixture(scope="module")
def ctx():
    return MoeContext(0)


def check(ctx, cfg, tol):
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    out, aux = ml.forward(layer.x, want_aux=True)
    ctx.synchronize()
    ref = Hh.run_oracle(cfg, layer.x.cpu())
    assert np.array_equal(aux["perm"].cpu().numpy().astype(np.uint32), ref["perm"])
    rel, mx = Hh.error_metrics(out.cpu().numpy(), ref["out"])
    assert rel <= tol and mx <= 2.0 ** -6, (rel, mx)
    return aux["counts"].cpu().numpy()


def config(fmt, T, E, k, H=512, I=256):
    return synth.MoeConfig(f"tiles{fmt}_{T}", H=H, I=I, E=E, k=k, fmt=fmt, T=T, seed=11)


@pytest.mark.parametrize("T,E,k", [(8, 8, 8), (16, 16, 8), (5, 4, 3)])
def test_int4_decode_batch_on_tensor_tiles(ctx, T, E, k, monkeypatch):
    # at most 16 tokens: the fused front end converts the rows, and the tiles read INT4 columns in their own order
    monkeypatch.setenv("STRATA_MOE_PREFILL_MIN_ROWS", "1")
    check(ctx, config(synth.FMT_INT4, T, E, k), TOL_F16)


@pytest.mark.parametrize("H", [512, 384])       # 384: single weight tiles in the down projection, half a block at the end
@pytest.mark.parametrize("fmt", [synth.FMT_MXFP4, synth.FMT_NVFP4, synth.FMT_INT4])
@pytest.mark.parametrize("ntile,T", [(32, 33), (64, 65), (128, 129), (160, 161), (192, 193)])
def test_one_row_beyond_a_tile(ctx, fmt, ntile, T, H, monkeypatch):
    # every token visits both experts: a full tile and a tile of one row each
    monkeypatch.setenv("STRATA_MOE_PREFILL_MIN_ROWS", "1")
    monkeypatch.setenv("STRATA_MOE_PREFILL_NTILE", str(ntile))
    counts = check(ctx, config(fmt, T, 2, 2, H=H), TOL_F16)
    assert counts.tolist() == [T, T]


@pytest.mark.parametrize("H", [512, 384])
@pytest.mark.parametrize("T,E,k", [(3, 16, 2), (17, 2, 2), (33, 8, 4), (65, 2, 2), (130, 2, 2)])
def test_bf16_expert_tiles(ctx, T, E, k, H, monkeypatch):
    # tiles of 16, 32 and 64 token rows (hi + lo pairs), one row beyond them, empty groups
    monkeypatch.setenv("STRATA_MOE_PREFILL_MIN_ROWS", "0")
    check(ctx, config(synth.FMT_BF16, T, E, k, H=H), TOL_PAIR)


@pytest.mark.parametrize("H", [512, 384])
@pytest.mark.parametrize("fmt", [synth.FMT_MXFP4, synth.FMT_NVFP4, synth.FMT_INT4])
@pytest.mark.parametrize("rows,T,E,k", [(16, 3, 16, 2), (16, 17, 4, 2), (32, 33, 8, 2), (64, 65, 16, 2), (64, 130, 32, 2)])
def test_paired_activation_tiles(ctx, fmt, rows, T, E, k, H, monkeypatch):
    # fewer than eight rows per expert on average (raised by the switch for the small shapes), a row beyond a tile
    monkeypatch.setenv("STRATA_MOE_PREFILL_MIN_ROWS", "1000")
    monkeypatch.setenv("STRATA_MOE_NO_STREAM_RING", "1")
    monkeypatch.setenv("STRATA_MOE_PAIR_NTILE", str(rows))
    check(ctx, config(fmt, T, E, k, H=H), TOL_PAIR)


@pytest.mark.parametrize("asked,used", [(1, 16), (15, 16), (17, 32), (1000, 64)])
def test_paired_tile_switch_takes_existing_sizes_only(ctx, asked, used, monkeypatch):
    # the tile list is sized for 16-row tiles: other numbers select the next size there is
    cfg = config(synth.FMT_INT4, 40, 8, 8)
    monkeypatch.setenv("STRATA_MOE_PREFILL_MIN_ROWS", "1000")
    layer, outs = synth.build_layer(cfg, "cuda"), []
    for rows in (asked, used):
        monkeypatch.setenv("STRATA_MOE_PAIR_NTILE", str(rows))
        ml = MoeLayer(ctx, cfg)
        ml.load_synth(layer)
        outs.append(ml.forward(layer.x))
        ctx.synchronize()
    ctx.check_canaries()
    assert torch.equal(*outs) and bool((outs[0] != 0).any())


def test_int4_scales_outside_f16_keep_the_general_decoders(ctx, monkeypatch):
    # q * scale would not be exact in f16: the call must take the same path as with the tiles switched off
    monkeypatch.setenv("STRATA_MOE_PAIR_NTILE", "16")      # the tiles whatever the size of the call
    cfg = config(synth.FMT_INT4, 9, 16, 2)
    layer = synth.build_layer(cfg, "cuda")
    layer.scales["down"] = (layer.scales["down"].view(torch.bfloat16) * 2.0 ** -12).view(torch.uint8)
    outs = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("STRATA_MOE_NO_PAIR_TILES", "1")
        ml = MoeLayer(ctx, cfg)
        ml.load_synth(layer)
        outs.append(ml.forward(layer.x))
        ctx.synchronize()
    assert torch.equal(*outs) and bool((outs[0] != 0).any())


def test_registering_an_int4_expert_again_decides_anew(ctx, monkeypatch):
    # scales off f16 registered over one expert of a layer in use, rewritten in place and registered, and taken back
    monkeypatch.setenv("STRATA_MOE_PAIR_NTILE", "16")
    cfg = config(synth.FMT_INT4, 9, 16, 2)
    layer = synth.build_layer(cfg, "cuda")

    def fresh():
        ml = MoeLayer(ctx, cfg)
        ml.load_synth(layer)
        out = ml.forward(layer.x)
        ctx.synchronize()
        return out

    def streamed():
        with monkeypatch.context() as m:
            m.setenv("STRATA_MOE_NO_PAIR_TILES", "1")
            return fresh()

    ml, on_tiles = MoeLayer(ctx, cfg), fresh()
    ml.load_synth(layer)
    assert torch.equal(ml.forward(layer.x), on_tiles) and not torch.equal(on_tiles, streamed())
    good, rows = layer.scales["down"].clone(), layer.scales["down"]
    rows[3] = (good[3].view(torch.bfloat16) * 2.0 ** -12).view(torch.uint8)
    ml.set_expert(3, 2, layer.packed["down"][3], rows[3])
    assert torch.equal(ml.forward(layer.x), streamed())
    rows.copy_(good)
    ml.set_expert(3, 2, layer.packed["down"][3], rows[3])
    assert torch.equal(ml.forward(layer.x), on_tiles)
    ctx.synchronize()


@pytest.mark.parametrize("fmt", [synth.FMT_BF16, synth.FMT_NVFP4])
def test_weights_registered_at_another_address_are_used(ctx, fmt, monkeypatch):
    monkeypatch.setenv("STRATA_MOE_PREFILL_MIN_ROWS", "0")
    cfg = config(fmt, 33, 8, 4)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    before = ml.forward(layer.x).clone()
    other = {role: layer.packed[role].flip(0).contiguous() for role in synth.ROLES}      # the experts in reverse order
    layer.packed = {role: torch.cat([other[role][:4], layer.packed[role][4:]]) for role in synth.ROLES}
    for r, role in enumerate(synth.ROLES):
        for e in range(4):
            ml.set_expert(e, r, layer.packed[role][e], layer.scales[role][e], layer.global_scale(role))
    after = ml.forward(layer.x).clone()
    ml2 = MoeLayer(ctx, cfg)
    ml2.load_synth(layer)
    want = ml2.forward(layer.x)
    ctx.synchronize()
    assert torch.equal(after, want) and not torch.equal(after, before)
