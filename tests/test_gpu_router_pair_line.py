"""Router projection on both sides of the line between two and eight expert rows per CTA: the oracle's canonical sums (needs a B200)."""
import numpy as np
import pytest

from oracle import oracle as O
from strata_b200 import MoeContext, MoeLayer, synth
from tests import helpers as Hh

pytestmark = pytest.mark.gpu


# experts times tokens against six times the columns; tokens against 8 + columns / 128
@pytest.mark.parametrize("H,E,T", [(512, 1024, 3), (512, 1024, 4), (512, 256, 12), (512, 256, 13), (1024, 511, 12), (1024, 513, 12), (128, 5, 9),
                                   (128, 5, 10), (512, 16, 12), (512, 16, 13), (2048, 768, 16), (2048, 769, 16)])
def test_logits_bit_for_bit(H, E, T):
    cfg = synth.MoeConfig(f"line{H}_{E}", H=H, I=128, E=E, k=1, fmt=synth.FMT_INT4, T=T, seed=31)
    ctx = MoeContext(0)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    logits = ml.route(layer.x, want_logits=True)[2]
    ctx.synchronize()
    want = O.router_logits(Hh.np_u16(layer.x), Hh.np_u16(layer.router_w))
    assert np.array_equal(logits.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
