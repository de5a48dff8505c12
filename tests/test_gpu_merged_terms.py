"""Terms that share a cofactor and differ in one private table run as one term over the tables' linear combination:
messages, point and every table's final evaluation equal the oracle's, next to terms that must not be merged."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import family_dtype, gpu_sumcheck_prove, upload

pytestmark = pytest.mark.gpu

FIELDS = [orc.FrField, orc.GlField]


def int_mle(dpb, ctx, F, rng, n, wide):
    fam = family_dtype(dpb, F)
    dt = {(True, False): dpb.FR_I32, (True, True): dpb.FR_I64, (False, False): dpb.GL_I32, (False, True): dpb.GL_I64}[(fam == dpb.FR, wide)]
    x = rng.integers(-2**63, 2**63 - 1, size=1 << n, dtype=np.int64) if wide else rng.integers(-2**31, 2**31, size=1 << n, dtype=np.int64)
    return ctx.upload_ints(x, dt), F.table_from_i64(x)


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("n", [9, 10, 11, 14])  # below, at and above the size from which terms are merged
def test_groups_next_to_other_terms(dpb, ctx, F, n):
    rng = np.random.default_rng(9900 + n)
    fam = family_dtype(dpb, F)
    mles, tabs = [], []
    pts = [[F.random_scalar(rng) for _ in range(n)] for _ in range(3)]
    for p in pts:                                   # 0..2: eq tables
        mles.append(ctx.eq_table(fam, orc.scalars_to_array(F, p)))
        tabs.append(orc.eq_evals(F, p))
    for j in range(6):                              # 3..8: integer and field tables
        if j % 3 < 2:
            m, t = int_mle(dpb, ctx, F, rng, n, j % 3 == 1)
        else:
            t = F.random_table_fast(rng, 1 << n)
            m = upload(dpb, ctx, F, t)
        mles.append(m)
        tabs.append(t)
    small = F.random_table_fast(rng, 1 << (n - 2))  # 9: constant in the first two rounds
    mles.append(upload(dpb, ctx, F, small))
    tabs.append(small)
    c = lambda: F.random_scalar(rng)
    cases = [
        # heads under one eq, mask and selector; two terms of the cofactor alone
        {(0, 3, 4): c(), (0, 3, 5): c(), (0, 3, 6): F.one, (0, 3, 7): F.neg(F.one), (0, 3): c(), (0,): c()},
        # claims on one tensor: the private tables are eq tables
        {(0, 3): F.one, (1, 3): c(), (2, 3): c()},
        # two groups, and a linear term list without a cofactor
        {(0, 3, 4): c(), (0, 3, 5): c(), (1, 3, 6): c(), (1, 3, 7): c()},
        {(4,): c(), (5,): c(), (6,): c()},
        # not merged: private tables multiplied with each other, a square, a smaller private table, a shared one
        {(0, 3, 4): c(), (0, 5, 6): c(), (7, 7): c(), (0, 8): c(), (0, 9): c(), (8, 8): c()},
        {(0, 9): c(), (0, 3): c(), (0, 4): c(), (9, 5): c()},
    ]
    for terms in cases:
        want = orc.sumcheck_prove(F, n, tabs, terms, orc.Transcript(F))
        assert gpu_sumcheck_prove(dpb, ctx, F, n, mles, terms, orc.Transcript(F)) == want
    for m in mles:
        m.free()


def test_states_and_refusals(dpb, ctx):
    """A merged sumcheck answers calls in the wrong state and bad arguments as any other."""
    F = orc.FrField
    rng = np.random.default_rng(9950)
    n = 10
    tabs = [F.random_table_fast(rng, 1 << n) for _ in range(3)]
    mles = [upload(dpb, ctx, F, t) for t in tabs]
    arr = dpb.make_terms([(F.one, [0, 1]), (F.one, [0, 2])], F.to_native)
    sc = ctx.sumcheck(n, mles, arr)
    r = orc.scalars_to_array(F, [F.random_scalar(rng)])
    with pytest.raises(dpb.DpbError) as e:
        sc.round(r)
    assert e.value.code == dpb.ESTATE
    with pytest.raises(dpb.DpbError) as e:
        sc.finish(r)
    assert e.value.code == dpb.ESTATE
    sc.round()
    sc.free()  # dropped in the middle
    bad = dpb.make_terms([(F.one, [0, 1]), (F.one, [0, 7])], F.to_native)
    with pytest.raises(dpb.DpbError) as e:
        ctx.sumcheck(n, mles, bad)
    assert e.value.code == dpb.EINVAL
    for m in mles:
        m.free()
