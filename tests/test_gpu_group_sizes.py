"""Grouping at the edges of its one-CTA kernel: rounds of 32 pairs per warp, its largest size and one pair more (needs a B200)."""
import numpy as np
import pytest
import torch

from strata_b200 import MoeContext, MoeLayer, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [1, 31, 33, 1023, 1024, 1025, 4097, 8191, 8192, 8193])
@pytest.mark.parametrize("E,begin,count", [(1, 0, 1), (100, 0, 100), (1024, 0, 1024), (896, 100, 33)])
def test_against_a_stable_sort(pairs, E, begin, count):
    cfg = synth.MoeConfig("group", H=128, I=128, E=E, k=1, fmt=synth.FMT_INT4, T=pairs, seed=3)
    ctx = MoeContext(0)
    ml = MoeLayer(ctx, cfg)
    rng = np.random.RandomState(pairs + E)
    # skewed: half of the pairs go to one expert, so that a warp's run holds long repeats
    ids = np.where(rng.rand(pairs) < 0.5, min(E - 1, begin + count // 2), rng.randint(0, E, pairs)).astype(np.int32)
    counts, offsets, perm, inv = ml.group(torch.from_numpy(ids).cuda().view(pairs, 1), begin, count, want_inv=True)
    ctx.synchronize()
    local = ids - begin
    mine = np.flatnonzero((local >= 0) & (local < count))
    want = mine[np.argsort(local[mine], kind="stable")]
    assert np.array_equal(counts.cpu().numpy(), np.bincount(local[mine], minlength=count))
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(local[mine], minlength=count))]))
    assert np.array_equal(perm.cpu().numpy()[:len(want)], want)
    pos = np.full(pairs, -1, np.int64)
    pos[want] = np.arange(len(want))
    assert np.array_equal(inv.cpu().numpy().view(np.int32).reshape(-1), pos)
    ctx.check_canaries()
