"""FP4 experts on the block-scaled tensor-core instructions, activations as digit planes (needs a B200)."""
import ctypes

import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth
from strata_b200.api import StrataMoeError
from tests import helpers as Hh

pytestmark = pytest.mark.gpu

MX, NV = synth.FMT_MXFP4, synth.FMT_NVFP4
# Exact weights and products, activations to 2^-23 of their block's maximum: what is left is the order of FP32 sums of up to
# 512 terms, in the oracle and here (512 * 2^-24 = 3e-5 at the very worst).
TOL = 1e-5


@pytest.fixture(scope="module")
def ctx():
    return MoeContext(0)


@pytest.fixture(autouse=True)
def planes(monkeypatch):
    monkeypatch.setenv("STRATA_MOE_PLANES_MAX_ROWS", "1000")


def config(fmt, T, E, k, H=512, I=512, **kw):
    return synth.MoeConfig(f"planes{fmt}_{T}_{E}", H=H, I=I, E=E, k=k, fmt=fmt, T=T, seed=17, **kw)


def outputs(ctx, cfg, layer, x=None):
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    out = ml.forward(layer.x if x is None else x)
    ctx.synchronize()
    return ml, out


# every token visits both experts: groups of T rows at and beyond the edges of the tiles (8, 16, 24 rows; a list of groups up to
# 24 tokens, a tile list beyond); 768 and 1280 columns: an odd number of stages; many empty groups
@pytest.mark.parametrize("fmt,H,I,E,k,T", [
    *[(f, 512, 512, 2, 2, T) for f in (MX, NV) for T in (1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25, 40, 49)],
    (MX, 1536, 1024, 3, 2, 19), (NV, 768, 1280, 3, 2, 19), (NV, 256, 256, 2, 2, 5), (MX, 512, 512, 64, 2, 3), (NV, 512, 512, 64, 4, 30)])
def test_against_the_oracle(ctx, fmt, H, I, E, k, T):
    cfg = config(fmt, T, E, k, H=H, I=I)
    layer = synth.build_layer(cfg, "cuda")
    ml, out = outputs(ctx, cfg, layer)
    ref = Hh.run_oracle(cfg, layer.x.cpu(), accumulate_double=True)
    rel, mx = Hh.error_metrics(out.cpu().numpy(), ref["out"])
    assert rel <= TOL and mx <= 10 * TOL, (rel, mx)
    # the stage call on grouped rows takes the tile list and has the same sums
    ids, w = ml.route(layer.x)
    _, offsets, perm, inv = ml.group(ids, want_inv=True)
    y = ml.experts_grouped(ml.gather_rows(layer.x, perm, cfg.k), offsets)
    assert torch.equal(ml.combine(y, inv, w), out)
    ctx.check_canaries()


@pytest.mark.parametrize("asked", ["-3", "1", "8", "17", "32", "1000000"])
def test_tile_switch_takes_existing_sizes_only(ctx, asked, monkeypatch):
    # a tile list of fewer than 16 rows per tile would outgrow its scratch, one of more than 24 the kernel's stages
    monkeypatch.setenv("STRATA_MOE_PLANES_TILE", asked)
    cfg = config(MX, 40, 8, 8)
    layer = synth.build_layer(cfg, "cuda")
    ml, out = outputs(ctx, cfg, layer)
    monkeypatch.delenv("STRATA_MOE_PLANES_TILE")
    ctx.check_canaries()
    assert torch.equal(out, outputs(ctx, cfg, layer)[1])


@pytest.mark.parametrize("fmt", [MX, NV])
def test_rows_of_uneven_magnitude(ctx, fmt):
    # a row of zeros, blocks of zeros, one column 2^20 above the rest of its row, a row of the smallest normal numbers, a row
    # whose blocks differ by 2^30 (beyond the E4M3 range of block scales: an error of 2^-40 of the row's maximum)
    cfg = config(fmt, 8, 2, 2)
    layer = synth.build_layer(cfg, "cuda")
    x = layer.x.clone()
    x[0] = 0
    x[1, 64:256] = 0
    x[2, 77] = 2.0 ** 20
    x[3] = (x[3].float() * 2.0 ** -60).bfloat16()
    x[4, 256:] = (x[4, 256:].float() * 2.0 ** -30).bfloat16()
    _, out = outputs(ctx, cfg, layer, x)
    ref = Hh.run_oracle(cfg, x.cpu(), accumulate_double=True)["out"]
    got = out.cpu().numpy()
    assert not got[0].any()
    for t in range(1, 8):
        rel, _ = Hh.error_metrics(got[t:t + 1], ref[t:t + 1])
        assert rel <= TOL, (t, rel)


# An outlier whose weight is zero must not be seen in any output: the digits of its block, fixed point against its maximum, hold
# the rest of the block to 2^-23 of the outlier only, the remainder holds what they leave.  Groups of T rows at the edges of the
# tiles (8, 16, 24 rows, remainders counted), every row, every third one or one with an outlier; a tile list beyond 24 tokens.
# Without remainders 4e-6 (2^12) to 4e-3 (2^20) of the output differ; with them the order of FP32 sums is left, about 2e-7.
EDGES = [(T, step) for T in (1, 4, 5, 8, 12, 13, 18, 24, 25, 49) for step in (1, 3, 100)]


def without_column(layer, role, cfg, col):
    """Zero weights in the byte of column `col` (two columns) of every row of a projection."""
    rows, cols = cfg.role_shape(role)
    layer.packed[role].view(cfg.E, rows, cols // 2)[:, :, col // 2] = 0


@pytest.mark.parametrize("fmt", [MX, NV])
@pytest.mark.parametrize("T,step", EDGES)
def test_token_outlier_of_zero_weight(ctx, fmt, T, step):
    cfg = config(fmt, T, 2, 2)
    layer = synth.build_layer(cfg, "cuda")
    for role in ("gate", "up"):
        without_column(layer, role, cfg, 76)
    layer.router_w[:, 76:78] = 0
    x = layer.x.clone()
    x[:, 76:78] = 0
    _, want = outputs(ctx, cfg, layer, x)
    for t in range(0, T, step):
        x[t, 77] = 2.0 ** (12, 16, 20)[t // step % 3]
    _, got = outputs(ctx, cfg, layer, x)
    for t in range(T):
        assert float((got[t] - want[t]).norm() / want[t].norm()) <= 1e-6, t
    ctx.check_canaries()


@pytest.mark.parametrize("fmt", [MX, NV])
@pytest.mark.parametrize("T", [1, 5, 13, 24, 49])
def test_activation_outlier_of_zero_weight(ctx, fmt, T):
    # one feature of every expert whose gate and up rows are 2^5 times the others', under a zero column of the down projection
    cfg = config(fmt, T, 2, 2)
    layer = synth.build_layer(cfg, "cuda")
    without_column(layer, "down", cfg, 76)
    _, want = outputs(ctx, cfg, layer)
    for role in ("gate", "up"):
        rows, cols = cfg.role_shape(role)
        s = layer.scales[role].view(cfg.E, rows, -1)
        s[:, 77] += 5 if fmt == MX else 5 << 3      # exponent fields
        assert fmt == MX or int(s[:, 77].max()) < 0x7F
    _, got = outputs(ctx, cfg, layer)
    for t in range(T):
        assert float((got[t] - want[t]).norm() / want[t].norm()) <= 1e-6, t
    ctx.check_canaries()


@pytest.mark.parametrize("fmt", [MX, NV])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_rows_that_are_not_finite_are_reported(ctx, fmt, value):
    cfg = config(fmt, 4, 2, 2)
    layer = synth.build_layer(cfg, "cuda")
    x = layer.x.clone()
    x[1, 5] = value
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    out = ml.forward(x)
    with pytest.raises(StrataMoeError):
        ctx.synchronize()
    assert not torch.isfinite(out[1]).any() and bool(torch.isfinite(out[[0, 2, 3]]).all())


def test_negative_nvfp4_scales_keep_the_other_kernels(ctx, monkeypatch):
    # the block-scaled instructions read E4M3 scales unsigned; found at registration, also of one expert of a layer in use
    cfg = config(NV, 6, 4, 2)
    layer = synth.build_layer(cfg, "cuda")
    ml, on_planes = outputs(ctx, cfg, layer)
    good = layer.scales["up"].clone()
    layer.scales["up"][2, 33] |= 0x80
    ml.set_expert(2, 1, layer.packed["up"][2], layer.scales["up"][2], global_scale=layer.global_scale("up"))
    mixed = ml.forward(layer.x).clone()
    monkeypatch.setenv("STRATA_MOE_PLANES_MAX_ROWS", "0")
    assert torch.equal(mixed, outputs(ctx, cfg, layer)[1])
    layer.scales["up"].copy_(good)
    ml.set_expert(2, 1, layer.packed["up"][2], layer.scales["up"][2], global_scale=layer.global_scale("up"))
    assert torch.equal(ml.forward(layer.x), on_planes)
    ctx.synchronize()


@pytest.mark.parametrize("fmt,T", [(MX, 3), (NV, 21)])
def test_ids_of_the_caller_may_name_an_expert_twice(ctx, fmt, T):
    # forward_routed takes any ids: a group can have more rows than there are tokens
    cfg = config(fmt, T, 4, 3)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    ids = torch.full((T, 3), 1, dtype=torch.int32, device="cuda")
    ids[:, 2] = 2
    w = torch.rand(T, 3, device="cuda")
    once = ids.clone()      # the same sum with distinct ids: the second one's weight goes to the first
    once[:, 1] = 3
    def routed(ids, w):
        out = torch.empty(T, cfg.H, device="cuda")
        ctx.check(ctx.lib.strata_moe_forward_routed(ml.h, *(ctypes.c_void_p(t) if i != 1 else ctypes.c_uint32(t) for i, t in enumerate(
            (layer.x.data_ptr(), T, ids.data_ptr(), w.data_ptr(), out.data_ptr())))))
        return out

    got = routed(ids, w)
    w2 = w.clone()
    w2[:, 0] += w2[:, 1]
    w2[:, 1] = 0
    want = routed(once, w2)
    ctx.synchronize()
    assert float((got - want).norm() / want.norm()) <= TOL
