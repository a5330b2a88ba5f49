"""INT4 tiles that decode with one multiply-add: scales at the ends of its six octaves against the general f16 decode (needs a B200)."""
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return MoeContext(0)


def forward(ctx, cfg, layer):
    ml = MoeLayer(ctx, cfg)
    ml.load_synth(layer)
    out = ml.forward(layer.x)
    ctx.synchronize()
    return out


# pairs (22-bit activation) and single f16 rows; H = 384: half a block of scales at the end of a row
@pytest.mark.parametrize("T,H", [(9, 512), (40, 512), (70, 384), (200, 512)])
@pytest.mark.parametrize("top", [8.0, 16.0])
def test_same_bits_as_the_general_decode(ctx, T, H, top, monkeypatch):
    # group scales over six octaves below `top` x 0.0043, both signs, some zero.  A fifth expert that no token selects spans seven
    # octaves in one of the two layers, which takes that layer off the narrow decode: power-of-two factors are all that differs.
    monkeypatch.setenv("STRATA_MOE_PAIR_NTILE", "64")
    cfg = synth.MoeConfig(f"octaves{T}_{H}", H=H, I=256, E=5, k=2, fmt=synth.FMT_INT4, T=T, seed=5)
    layer = synth.build_layer(cfg, "cuda")
    layer.bias = torch.tensor([0.0, 0.0, 0.0, 0.0, -100.0], device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(T)
    for role in synth.ROLES:
        s = layer.scales[role].view(torch.bfloat16)
        octave = torch.randint(0, 6, s.shape, device="cuda", generator=gen)
        octave[:, 0], octave[:, 1] = 0, 5
        sign = torch.randint(0, 2, s.shape, device="cuda", generator=gen) * 2 - 1
        mantissa = 0.00434 * top * (1.0 + 0.5 * torch.rand(s.shape, device="cuda", generator=gen))
        s.copy_(mantissa * torch.pow(2.0, -octave.float()) * sign)       # 0.00434 x 8 .. x 12 lies in one octave
        s[:, 5] = 0
    narrow = forward(ctx, cfg, layer)
    layer.scales["up"].view(torch.bfloat16)[4, 1] *= 0.5
    general = forward(ctx, cfg, layer)
    assert bool((narrow != 0).any()) and torch.equal(narrow, general)
