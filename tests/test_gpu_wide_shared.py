"""Wide shared experts of decode batches on the tensor-core tiles, the activation as a BF16 pair (needs a B200)."""
import pytest

from strata_b200 import MoeContext, MoeLayer, synth
from tests import helpers as Hh

pytestmark = pytest.mark.gpu

# BF16 weights, the SwiGLU output as a BF16 pair (2^-17), FP32 sums
TOL = 1e-4


@pytest.mark.parametrize("I_shared", [4992, 5120])      # 39 tiles: the streaming kernel; 40: tiles
@pytest.mark.parametrize("T", [1, 16, 17, 23])
def test_against_the_oracle(T, I_shared):
    cfg = synth.MoeConfig(f"wide{T}_{I_shared}", H=512, I=128, E=8, k=2, fmt=synth.FMT_INT4, T=T, I_shared=I_shared, seed=21)
    ctx = MoeContext(0)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    out = ml.forward(layer.x)
    ctx.synchronize()
    rel, mx = Hh.error_metrics(out.cpu().numpy(), Hh.run_oracle(cfg, layer.x.cpu())["out"])
    assert rel <= TOL and mx <= 10 * TOL, (rel, mx)
