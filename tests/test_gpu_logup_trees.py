"""Fraction trees of a batch, two levels per launch and the last ones in one block: every level of every instance equals
the oracle's, for integer, field and mixed columns at their largest values and sizes around every switch."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import family_dtype, upload

pytestmark = pytest.mark.gpu

FIELDS = [orc.FrField, orc.GlField]


def column(dpb, ctx, F, rng, m, kind):
    fam = family_dtype(dpb, F)
    i32, i64 = (dpb.FR_I32, dpb.FR_I64) if fam == dpb.FR else (dpb.GL_I32, dpb.GL_I64)
    if kind == "field":
        t = F.random_table_fast(rng, 1 << m)
        return upload(dpb, ctx, F, t), t
    if kind == "i32":
        x = rng.integers(-2**31, 2**31, size=1 << m, dtype=np.int64)
        x[:2] = [-2**31, 2**31 - 1]
        return ctx.upload_ints(x, i32), F.table_from_i64(x)
    x = rng.integers(-2**63, 2**63 - 1, size=1 << m, dtype=np.int64)
    x[1::2] = rng.integers(-2**12, 2**12, size=x[1::2].size)
    x[:2] = [-2**63, 2**63 - 1]
    return ctx.upload_ints(x, i64), F.table_from_i64(x)


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("m", [2, 3, 4, 9, 10, 11, 12, 13, 15])
@pytest.mark.parametrize("kinds,table", [(("i64",), False), (("i64", "i32"), False), (("field", "field"), False),
                                         (("i32", "field"), False), (("i64",) * 8, False), (("i32", "i64"), True), (("field",), True)])
def test_every_level(dpb, ctx, F, m, kinds, table):
    rng = np.random.default_rng(9600 + m + len(kinds))
    cols = [column(dpb, ctx, F, rng, m, k) for k in kinds]
    mult = column(dpb, ctx, F, rng, m, "i64" if len(kinds) > 1 else "field") if table else None
    # the largest constant and separation challenge: the denominator's sum of rows at its bound
    for c, s in ((F.random_scalar(rng), F.random_scalar(rng)), (F.neg(F.one), F.neg(F.one))):
        lu = ctx.logup(dpb.LOGUP_TABLE if table else dpb.LOGUP_LOOKUP, [x for x, _ in cols], orc.scalars_to_array(F, [c])[0],
                       orc.scalars_to_array(F, [s])[0], mult=mult[0] if table else None)
        assert lu.num_levels == m - 1
        num, den = orc.logup_next(F, 1 if table else 0, [t for _, t in cols], mult[1] if table else None, c, s)
        for level in range(1, m):
            if level > 1:
                num, den = orc.logup_next(F, 2, [num, den], None, c, s)
            half = 1 << (m - level - 1)
            views = lu.level(level)
            for v, w in zip(views, (num[:half], num[half:], den[:half], den[half:])):
                assert (v.to_host() == w).all(), level
                v.free()
        out = lu.outputs()
        assert (out[:2] == num).all() and (out[2:] == den).all()
        lu.free()
    for x, _ in cols + ([mult] if table else []):
        x.free()
