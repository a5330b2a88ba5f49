"""Every route to the expert ids gives the same bits: staged, whole-row and tensor-core projection (needs a B200)."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return MoeContext(0)


# tokens around the edges: one warp per token and CTA (16), a CTA per token (444 on the fast path, 592 for the scores)
@pytest.mark.parametrize("T", [1, 16, 17, 33, 444, 445, 593])
@pytest.mark.parametrize("E,k,H,kind", [(128, 8, 384, synth.SCORE_SIGMOID), (896, 16, 512, synth.SCORE_SIGMOID_PLAIN),
                                        (256, 6, 1024, synth.SCORE_SQRTSOFTPLUS)])
def test_router_paths_agree(ctx, T, E, k, H, kind, monkeypatch):
    cfg = synth.MoeConfig(f"router{T}_{E}", H=H, I=128, E=E, k=k, fmt=synth.FMT_MXFP4, T=T, score_kind=kind, zipf_s=0.7, seed=5)
    layer = synth.build_layer(cfg, "cuda")
    results = []
    for env in ({"STRATA_MOE_FAST_ROUTER_MIN_TOKENS": "-1", "STRATA_MOE_NO_SMALL_FRONT": "1"},
                {"STRATA_MOE_FAST_ROUTER_MIN_TOKENS": "-1"}, {"STRATA_MOE_FAST_ROUTER_MIN_TOKENS": "1"}):
        with monkeypatch.context() as m:
            for name, value in env.items():
                m.setenv(name, value)
            ml = MoeLayer(ctx, cfg)
        ml.load_synth(layer)
        results.append(ml.route(layer.x))
        ctx.synchronize()
    for ids, weights in results[1:]:
        assert torch.equal(ids, results[0][0])
        assert torch.equal(weights, results[0][1])


@pytest.mark.parametrize("magnitude", [2.0 ** 13, 2.0 ** 16, 2.0 ** 19])
@pytest.mark.parametrize("T", [200, 511])
def test_cancelling_products_below_512_tokens(ctx, T, magnitude, monkeypatch):
    """Two large products of opposite sign in one expert's logit: its tensor-core sum is off by far more than its final size
    suggests, while the logits of the experts that are selected instead are as good as ever."""
    cfg = synth.MoeConfig(f"cancel{T}", H=512, I=128, E=128, k=8, fmt=synth.FMT_MXFP4, T=T, seed=6)
    layer = synth.build_layer(cfg, "cuda")
    layer.x[:, 0] = layer.x[:, 256] = magnitude
    layer.router_w[:, 0] = layer.router_w[:, 256] = 0.0
    layer.router_w[77, 0], layer.router_w[77, 256] = 1.0, -1.0
    results = []
    for threshold in ("-1", "1"):
        with monkeypatch.context() as m:
            m.setenv("STRATA_MOE_FAST_ROUTER_MIN_TOKENS", threshold)
            ml = MoeLayer(ctx, cfg)
        ml.load_synth(layer)
        results.append(ml.route(layer.x))
        ctx.synchronize()
    differ = int((results[0][0] != results[1][0]).any(dim=1).sum())
    assert differ == 0, differ
    assert torch.equal(results[0][1], results[1][1])
