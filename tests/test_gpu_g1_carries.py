"""Additions of G1 points whose one double product  R (Q - X) - Y1 PPP  (g1_add_xy, reduced once) has a word of ones where
the reduction's carries end.  A word of random operands is all ones once in 2^32, so the pairs were searched for:
(a, b) below is the sum a G + b G, taken in this order; the word that is all ones is the fourth to last, and so on down
(words 8, 10, 12 and 14 of sixteen)."""
import importlib

import numpy as np
import pytest

from oracle import g1

PAIRS = [(80306, 89408, 8), (78260, 25538, 8), (55929, 42354, 10), (83748, 85083, 10), (79997, 122947, 12), (26089, 53551, 14),
         (56134, 52849, 14), (70388, 3592, 14)]


@pytest.fixture(scope="module")
def points():
    return [[g1.mul(k, g1.GENERATOR) for k in pair[:2]] for pair in PAIRS]


def double_product(p, q):
    """The two products' sum for p + q, p affine, every operand in Montgomery form."""
    m = lambda v: v % g1.Q * 2**256 % g1.Q
    dx, r = q[0] - p[0], q[1] - p[1]
    ppp, t = dx**3, p[0] * dx**2
    x = r * r - ppp - 2 * t
    return m(r) * m(t - x) + m(-p[1]) * m(ppp)


def test_the_pairs_have_the_word(points):
    for (p, q), (_, _, word) in zip(points, PAIRS):
        assert double_product(p, q) >> (32 * word) & 0xffffffff == 0xffffffff


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(PAIRS)))
def test_one_addition(dpb, ctx, points, case):
    """One bucket of two points; the order in which they are added is the bucket list's, so both orders of the bases."""
    pcs = importlib.import_module("deep_prove_b200.pcs")
    p, q = points[case]
    want = g1.mul(sum(PAIRS[case][:2]), g1.GENERATOR)
    for two in ([p, q], [q, p]):
        bases = pcs.G1Bases(ctx, two)
        assert pcs.msm(ctx, bases, ctx.upload_ints(np.ones(2, dtype=np.int64), dpb.FR_I32)) == want
        bases.free()


@pytest.mark.gpu
def test_all_pairs_in_their_own_buckets(dpb, ctx, points):
    pcs = importlib.import_module("deep_prove_b200.pcs")
    flat = [v for pair in points for v in pair]
    for bases_list in (flat, flat[::-1]):
        bases = pcs.G1Bases(ctx, bases_list)
        x = np.repeat(np.arange(1, len(PAIRS) + 1, dtype=np.int64), 2)
        order = PAIRS if bases_list is flat else PAIRS[::-1]
        k = sum((i + 1) * (a + b) for i, (a, b, _) in enumerate(order))
        got = pcs.batch_commit(ctx, bases, [ctx.upload_ints(x, dpb.FR_I32), ctx.upload_ints(x, dpb.FR_I64)])
        assert got == [g1.mul(k, g1.GENERATOR)] * 2
        bases.free()
