"""Sums of products that are reduced once at their end: partial evaluation, the linear combination and the evaluation
of many tables at one point, over integer and field tables, at the values and counts where the unreduced sums are
largest.  All arithmetic is exact: results equal the oracle's over the converted tables."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import upload

pytestmark = pytest.mark.gpu

FIELDS = [orc.FrField, orc.GlField]
EXTREMES = {4: [-2**31, 2**31 - 1, 0, -1], 8: [-2**63, 2**63 - 1, -2**31 - 1, 2**31, -2**31, 2**31 - 1, -1, 0]}


def layouts(dpb, F):
    return (dpb.FR_I32, dpb.FR_I64) if F is orc.FrField else (dpb.GL_I32, dpb.GL_I64)


def int_table(dpb, ctx, F, rng, dtype, n, fill=None):
    size = np.dtype(dpb.INT_DTYPES[dtype]).itemsize
    x = np.full(n, fill, dtype=np.int64) if fill is not None else rng.choice(np.array(EXTREMES[size], dtype=np.int64), size=n)
    if fill is None:
        x[::3] = rng.integers(-2**12, 2**12, size=x[::3].size)
    return ctx.upload_ints(x, dtype), F.table_from_i64(x)


def field_table(dpb, ctx, F, rng, n, top):
    t = F.random_table_fast(rng, n)
    if top:  # every entry p - 1
        t = F.table_from_i64(np.full(n, -1, dtype=np.int64))
    return upload(dpb, ctx, F, t), t


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("n,k", [(1, 1), (2, 1), (2, 2), (5, 5), (6, 6), (11, 2), (11, 5), (11, 6), (12, 10)])
def test_partial_evaluation(dpb, ctx, F, n, k):
    rng = np.random.default_rng(9100 + 16 * n + k)
    i32, i64 = layouts(dpb, F)
    tabs = [int_table(dpb, ctx, F, rng, i32, 1 << n), int_table(dpb, ctx, F, rng, i64, 1 << n),
            int_table(dpb, ctx, F, rng, i32, 1 << n, -2**31), int_table(dpb, ctx, F, rng, i64, 1 << n, 2**63 - 1),
            field_table(dpb, ctx, F, rng, 1 << n, False), field_table(dpb, ctx, F, rng, 1 << n, True)]
    for pt in ([F.random_scalar(rng) for _ in range(k)], [F.neg(F.one)] * k, [F.from_int(0)] * k):
        pa = orc.scalars_to_array(F, pt)
        for m, t in tabs:
            low, high = ctx.fix_low(m, pa), ctx.fix_high(m, pa)
            assert (low.to_host() == orc.fix_low_variables(F, t, pt)).all()
            assert (high.to_host() == orc.fix_high_variables(F, t, pt)).all()
            low.free()
            high.free()
    for m, _ in tabs:
        m.free()


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("count", [1, 3, 130, 1030])
def test_linear_combination_of_many(dpb, ctx, F, count):
    """More row products than one unreduced sum holds (1024), in all layouts and lengths."""
    rng = np.random.default_rng(9200 + count)
    i32, i64 = layouts(dpb, F)
    tabs = []
    for j in range(count):
        n = 1 << int(rng.integers(1, 7))
        kind = j % 3 if count < 1000 else min(j % 10, 2)
        tabs.append(field_table(dpb, ctx, F, rng, n, j % 2 == 0) if kind == 0 else
                    int_table(dpb, ctx, F, rng, i32 if kind == 1 else i64, n))
    coeffs = [F.neg(F.one) if j % 4 == 0 else F.random_scalar(rng) for j in range(count)]
    got = dpb.linear_combination(ctx, [m for m, _ in tabs], orc.scalars_to_array(F, coeffs))
    assert (got.to_host() == orc.linear_combination(F, [t for _, t in tabs], coeffs)).all()
    got.free()
    for m, _ in tabs:
        m.free()


@pytest.mark.parametrize("F", FIELDS)
def test_evaluate_many_pieces(dpb, ctx, F):
    """Tables shorter than a piece, of exactly one piece (1024 entries) and of many, next to each other."""
    rng = np.random.default_rng(9300)
    i32, i64 = layouts(dpb, F)
    nv = 15
    tabs = []
    for j, m in enumerate([0, 15, 1, 10, 11, 3, 15, 10, 0, 12, 15, 7]):
        tabs.append(field_table(dpb, ctx, F, rng, 1 << m, j % 2 == 0) if j % 3 == 1 else
                    int_table(dpb, ctx, F, rng, (i32, i64)[j % 2], 1 << m))
    pt = [F.random_scalar(rng) for _ in range(nv)]
    got = orc.array_to_scalars(F, dpb.evaluate_many(ctx, [m for m, _ in tabs], orc.scalars_to_array(F, pt)))
    for (m, t), g in zip(tabs, got):
        v = int(m.len).bit_length() - 1
        want = orc.evaluate(F, t, pt[:v]) if v else F.table_to_ints(t)[0]
        if v == 0 and not isinstance(want, tuple) and F is orc.GlField:
            want = (want, 0)
        for j in range(v, nv):
            want = F.mul(want, F.sub(F.one, pt[j]))
        assert g == want
        m.free()
