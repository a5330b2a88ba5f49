"""Which FP4 calls take the digit planes: up to 24 rows per expert on average and 384 tokens (needs a B200).

The planes round otherwise than the f16 kernels, so the bits of a call tell which served it."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth

pytestmark = pytest.mark.gpu

MX, NV = synth.FMT_MXFP4, synth.FMT_NVFP4


@pytest.fixture(scope="module")
def ctx():
    return MoeContext(0)


@pytest.fixture(autouse=True)
def no_switch(monkeypatch):
    for name in ("STRATA_MOE_PLANES_MAX_ROWS", "STRATA_MOE_NO_F16_PATH", "STRATA_MOE_NO_PREFILL_PATH", "STRATA_MOE_NO_STREAM_RING",
                 "STRATA_MOE_STREAM_RING_MAX_ROWS", "STRATA_MOE_PREFILL_MIN_ROWS", "STRATA_MOE_PREFILL_NTILE", "STRATA_MOE_PAIR_NTILE",
                 "STRATA_MOE_NO_PAIR_TILES"):
        monkeypatch.delenv(name, raising=False)


def run(ctx, cfg, layer, x):
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    out = ml.forward(x)
    ctx.synchronize()
    return out


# tokens: 32 experts, one each; rows: 16 experts, top-4, 96 tokens bring 24 rows each, 97 a little more; H, I: what the kernels cut
@pytest.mark.parametrize("fmt,H,I,E,k,T,planes", [
    (MX, 512, 512, 32, 1, 1, True), (NV, 512, 512, 32, 1, 384, True), (MX, 512, 512, 32, 1, 384, True),
    (NV, 512, 512, 32, 1, 385, False), (MX, 512, 512, 32, 1, 385, False),
    (MX, 512, 512, 16, 4, 96, True), (MX, 512, 512, 16, 4, 97, False), (NV, 512, 512, 16, 4, 96, True), (NV, 512, 512, 16, 4, 97, False),
    (MX, 768, 512, 32, 1, 20, False), (NV, 768, 512, 32, 1, 20, True), (NV, 640, 512, 32, 1, 20, False)])
def test_both_sides_of_the_rule(ctx, fmt, H, I, E, k, T, planes, monkeypatch):
    cfg = synth.MoeConfig(f"rule{fmt}_{T}_{H}", H=H, I=I, E=E, k=k, fmt=fmt, T=T, norm_init=1e-20, seed=19)
    layer = synth.build_layer(cfg, "cuda")
    got = run(ctx, cfg, layer, layer.x)
    monkeypatch.setenv("STRATA_MOE_PLANES_MAX_ROWS", "0")
    without = run(ctx, cfg, layer, layer.x)
    monkeypatch.setenv("STRATA_MOE_PLANES_MAX_ROWS", "64")
    with_planes = run(ctx, cfg, layer, layer.x)
    assert torch.equal(got, with_planes if planes else without)
    if H % (512 if fmt == MX else 256) == 0:
        assert not torch.equal(with_planes, without)


@pytest.mark.parametrize("fmt,shared,T", [(MX, 0, 1), (MX, 256, 8), (NV, 256, 16), (NV, 0, 30)])
def test_calls_queued_on_changing_inputs(ctx, fmt, shared, T):
    # the kernels of a call come up while their predecessors run: nothing waits on the host between the calls, the token rows
    # change in place between them, and rows of the first call have outliers, those of the next none
    cfg = synth.MoeConfig(f"queue{fmt}_{T}", H=512, I=512, E=16, k=4, fmt=fmt, T=T, I_shared=shared, seed=23)
    layer = synth.build_layer(cfg, "cuda")
    inputs = [layer.x * (1 + i) for i in range(12)]
    for x in inputs[::3]:
        x[:, 5] = 2.0 ** 12
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    want = []
    for x in inputs:
        want.append(ml.forward(x).clone())
        ctx.synchronize()
    x, outs = torch.empty_like(layer.x), [torch.empty(T, cfg.H, device="cuda") for _ in inputs]
    torch.cuda.synchronize()
    for i, (v, out) in enumerate(zip(inputs, outs)):
        x.copy_(v)
        ml.forward(x, out)
    torch.cuda.synchronize()
    for i, (out, ref) in enumerate(zip(outs, want)):
        assert torch.equal(out, ref), i
    ctx.check_canaries()
