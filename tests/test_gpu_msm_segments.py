"""The bucket sums of the multi-scalar multiplication are taken over equal runs of the sorted index list, one run per
thread, so a bucket may lie inside a run, meet its neighbour's, span several threads, or span several blocks
(dpb_msm_g1).  The bases are the consecutive multiples of the generator: sum_i s_i (i + 1) G is one scalar
multiplication of the oracle.  Group arithmetic is exact, so results are compared as integers."""
import importlib

import numpy as np
import pytest

from oracle import g1

pytestmark = pytest.mark.gpu


def column(kind, n, rng):
    i = np.arange(n, dtype=np.int64)
    if kind == "one":  # one bucket for the whole grid
        return np.full(n, 7, dtype=np.int64)
    if kind == "three":  # buckets of many blocks each, ends inside a block
        return np.where(i < n // 3, 5, np.where(i < 2 * n // 3 + 17, -6, 900))
    if kind == "ramp":  # buckets of 1, 2, 3, ... points: inside a run, over two, over several
        return (np.sqrt(2.0 * i + 0.25) + 0.5).astype(np.int64) * np.where(i % 2, 1, -1)
    if kind == "sparse":  # far fewer points than threads, and empty stretches of buckets between them
        return np.where(rng.random(n) < 40.0 / n, rng.integers(1, 1 << 15, n), 0)
    if kind == "crowd":  # a huge bucket among single ones
        return np.where(rng.random(n) < 0.7, 12, rng.integers(0, 1 << 13, n))
    assert kind == "wide"
    return rng.integers(-(1 << 31), 1 << 31, n)


@pytest.mark.parametrize("kind", ["one", "three", "ramp", "sparse", "crowd", "wide"])
@pytest.mark.parametrize("log2_n", [0, 5, 10, 14, 18])  # windows of 8, 10, 13 and 16 bits
def test_msm_bucket_spans(dpb, ctx, kind, log2_n):
    pcs = importlib.import_module("deep_prove_b200.pcs")
    n = 1 << log2_n
    x = column(kind, n, np.random.default_rng(7000 + log2_n))
    bases = pcs.G1Bases.synthetic(ctx, n)
    k = int(sum(int(v) * (i + 1) for i, v in enumerate(x)) % g1.R_ORDER)
    want = g1.boundary(g1.mul(k, g1.GENERATOR)) if k else (0, 0)
    assert pcs.msm(ctx, bases, ctx.upload_ints(x, dpb.FR_I32)) == want
    assert pcs.batch_commit(ctx, bases, [ctx.upload_ints(x, dpb.FR_I64)] * 2) == [want, want]
    bases.free()


def test_msm_same_and_opposite_points_in_every_step(dpb, ctx):
    """All points equal, and points next to their negatives: every addition of a run, of the pieces and of the trees
    meets its special case."""
    pcs = importlib.import_module("deep_prove_b200.pcs")
    n = 1 << 14
    p = g1.synthetic_bases(1, seed=9)[0]
    bases = pcs.G1Bases(ctx, np.tile(pcs.points_to_array([p]), (n, 1)))
    i = np.arange(n, dtype=np.int64)
    for x in (np.full(n, 3, dtype=np.int64), np.where(i % 2, 3, -3), np.where(i % 256 < 128, 3, -3), i % 4096, i % 512 - 256):
        k = int(x.sum()) % g1.R_ORDER
        want = g1.boundary(g1.mul(k, p)) if k else (0, 0)
        assert pcs.msm(ctx, bases, ctx.upload_ints(x, dpb.FR_I32)) == want
    bases.free()
