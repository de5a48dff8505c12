"""Fraction trees large enough for launches of one level each: every level equals the oracle's, and a batch that mixes
field columns, integer columns and sizes gives the proof that integer columns alone give."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import family_dtype
from tests.test_gpu_logup_trees import FIELDS, column

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("m,kinds,table", [(19, ("field", "i64"), False), (20, ("field",), False), (20, ("i64", "field", "field"), True),
                                           (22, ("field", "field"), False), (22, ("i32", "i64"), True)])
def test_every_level(dpb, ctx, F, m, kinds, table):
    rng = np.random.default_rng(9650 + m + len(kinds))
    cols = [column(dpb, ctx, F, rng, m, k) for k in kinds]
    mult = column(dpb, ctx, F, rng, m, "field") if table else None
    c, s = F.random_scalar(rng), F.neg(F.one)
    lu = ctx.logup(dpb.LOGUP_TABLE if table else dpb.LOGUP_LOOKUP, [x for x, _ in cols], orc.scalars_to_array(F, [c])[0],
                   orc.scalars_to_array(F, [s])[0], mult=mult[0] if table else None)
    num, den = orc.logup_next(F, 1 if table else 0, [t for _, t in cols], mult[1] if table else None, c, s)
    for level in range(1, m):
        if level > 1:
            num, den = orc.logup_next(F, 2, [num, den], None, c, s)
        half = 1 << (m - level - 1)
        for v, w in zip(lu.level(level), (num[:half], num[half:], den[:half], den[half:])):
            assert (v.to_host() == w).all(), level
            v.free()
    lu.free()
    for x, _ in cols + ([mult] if table else []):
        x.free()


@pytest.mark.parametrize("F", FIELDS)
def test_mixed_batch(dpb, ctx, F):
    from deep_prove_b200 import prover as P
    rng = np.random.default_rng(9660)
    fam = family_dtype(dpb, F)
    base, i64 = (dpb.FR, dpb.FR_I64) if fam == dpb.FR else (dpb.GL_BASE, dpb.GL_I64)
    data = [(m, rng.integers(-2**31, 2**31, size=(2, 1 << m), dtype=np.int64)) for m in (19, 19, 18, 4, 2)]
    chal = [[orc.scalars_to_array(F, [F.random_scalar(rng)])[0] for _ in range(2)] for _ in data]

    def proof(as_field):
        inputs, handles = [], []
        for i, ((m, x), (c, s)) in enumerate(zip(data, chal)):
            cols = [ctx.upload_i64(v, base) if as_field and i in (0, 2, 4) else ctx.upload_ints(v, i64) for v in x]
            handles += cols
            inputs.append(P.LogUpInput.new_lookup(cols, c, s, 2))
        tr = P.Blake3Transcript(fam)
        out = P.new_batch_multiple_sizes_prove(ctx, inputs, tr)
        tr.free()
        for h in handles:
            h.free()
        return out

    assert proof(True) == proof(False)
