"""Zero-padded sumchecks over  sum_t c_t * table_t * eq_t  (the claim batching's form), whose rounds sum against the eq
table of the variables still to come: messages, point and final evaluations equal the oracle's on the materialised
tables, and those of the same sumcheck with the eq tables' tags lost (the general zero-padded kernels)."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import family_dtype, gpu_sumcheck_prove, upload

pytestmark = pytest.mark.gpu

FIELDS = [orc.FrField, orc.GlField]


def ints(rng, n, wide):
    x = rng.integers(-2**63, 2**63 - 1, size=n, dtype=np.int64) if wide else rng.integers(-2**31, 2**31, size=n, dtype=np.int64)
    if n > 2:
        x[::2] = rng.integers(-2**12, 2**12, size=x[::2].size)
        x[:2] = [-2**63, 2**63 - 1] if wide else [-2**31, 2**31 - 1]
    return x


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("sizes", [[2, 1], [9, 1, 2], [13, 13, 3, 9, 8, 1, 12], [16, 4, 16, 10, 15]])
@pytest.mark.parametrize("special", [False, True])
def test_eq_pair_rounds(dpb, ctx, F, sizes, special):
    rng = np.random.default_rng(9500 + len(sizes) + special)
    n, fam = max(sizes), family_dtype(dpb, F)
    i32, i64 = (dpb.FR_I32, dpb.FR_I64) if fam == dpb.FR else (dpb.GL_I32, dpb.GL_I64)
    owned, views, plain, tables, terms = [], [], [], [], {}
    for t, m in enumerate(sizes):
        kind = (t + special) % 4
        if kind == 0:
            x = ints(rng, 1 << m, False)
            f, tab = ctx.upload_ints(x, i32), F.table_from_i64(x)
        elif kind == 1:
            x = ints(rng, 1 << m, True)
            f, tab = ctx.upload_ints(x, i64), F.table_from_i64(x)
        else:
            tab = F.random_table_fast(rng, 1 << m)
            f = upload(dpb, ctx, F, tab)
        # coordinates 0 and 1 have no inverse of q or 1 - q: nothing here needs one
        pt = [F.from_int(int(rng.integers(0, 2))) if special and j % 2 else F.random_scalar(rng) for j in range(m)]
        eq = ctx.eq_table(fam, orc.scalars_to_array(F, pt))
        eq_tab = orc.eq_evals(F, pt)
        copy = upload(dpb, ctx, F, eq_tab)
        owned += [f, eq, copy]
        pair = [(f.zero_padded(), f.zero_padded(), tab), (eq.zero_padded(), copy.zero_padded(), eq_tab)]
        if t % 2:
            pair.reverse()  # the eq table may come first
        for v, p, tb in pair:
            views.append(v)
            plain.append(p)
            tables.append(orc.zero_pad_table(F, tb, n))
        terms[(2 * t, 2 * t + 1)] = F.one if t == 0 else F.random_scalar(rng)
    want = orc.sumcheck_prove(F, n, tables, terms, orc.Transcript(F))
    assert gpu_sumcheck_prove(dpb, ctx, F, n, views, terms, orc.Transcript(F)) == want
    assert gpu_sumcheck_prove(dpb, ctx, F, n, plain, terms, orc.Transcript(F)) == want
    # a table shared by two terms, or a term of another shape, is not of this form and takes the general kernels
    if len(sizes) > 2:
        other = dict(terms)
        other[(0,)] = F.random_scalar(rng)
        want = orc.sumcheck_prove(F, n, tables, other, orc.Transcript(F))
        assert gpu_sumcheck_prove(dpb, ctx, F, n, views, other, orc.Transcript(F)) == want
    for h in views + plain + owned:
        h.free()
