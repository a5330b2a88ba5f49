"""Router projection with two expert rows per CTA: bit for bit the oracle's canonical sums at its edges (needs a B200)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from strata_b200 import MoeContext, MoeLayer, synth
from tests import helpers as Hh

pytestmark = pytest.mark.gpu


# odd numbers of experts, one column quarter of a single step, the last token count that fits 100 KB and the next one
@pytest.mark.parametrize("H,E,T", [(128, 3, 1), (128, 256, 16), (1152, 1, 2), (4096, 255, 10), (4096, 255, 11), (7168, 65, 5), (7168, 65, 6),
                                   (3072, 32, 14), (3072, 32, 15), (3072, 32, 16)])
def test_logits_bit_for_bit(H, E, T):
    cfg = synth.MoeConfig(f"pairs{H}_{E}", H=H, I=128, E=E, k=1, fmt=synth.FMT_INT4, T=T, seed=31)
    ctx = MoeContext(0)
    layer = synth.build_layer(cfg, "cuda")
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    logits = ml.route(layer.x, want_logits=True)[2]
    ctx.synchronize()
    want = O.router_logits(Hh.np_u16(layer.x), Hh.np_u16(layer.router_w))
    assert np.array_equal(logits.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
