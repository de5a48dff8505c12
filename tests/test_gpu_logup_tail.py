"""The last rounds of a logup layer in their own resident kernel (one block, or a cluster of blocks that hands over to
one): proof bytes equal the oracle's at sizes around every switch, for all kinds of input layer, and stay the same
when the host is held up past the kernel's wait at any of its challenges, so that the kernel is started again and its
rounds played once more."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import family_dtype, upload

pytestmark = pytest.mark.gpu

FIELDS = [orc.FrField, orc.GlField]


def build(dpb, ctx, F, rng, spec, m, ints):
    """spec: a list of (kind, columns) of one size; ints: integer columns.  -> (library inputs, oracle inputs, handles)"""
    from deep_prove_b200 import prover as P
    fam = family_dtype(dpb, F)
    i32, i64 = (dpb.FR_I32, dpb.FR_I64) if fam == dpb.FR else (dpb.GL_I32, dpb.GL_I64)
    lib_in, orc_in, handles = [], [], []
    for j, (kind, ncol) in enumerate(spec):
        c, s = F.random_scalar(rng), F.random_scalar(rng)
        ca, sa = orc.scalars_to_array(F, [c])[0], orc.scalars_to_array(F, [s])[0]
        cols, tabs = [], []
        for q in range(ncol):
            x = rng.integers(-2**15, 2**15, size=1 << m, dtype=np.int64)
            tab = F.table_from_i64(x)
            cols.append(ctx.upload_ints(x, (i32, i64)[(j + q) % 2]) if ints else upload(dpb, ctx, F, tab))
            tabs.append(tab)
        handles += cols
        if kind == "table":
            x = rng.integers(0, 2**20, size=1 << m, dtype=np.int64)
            mult, mt = ctx.upload_i64(x, dpb.FR if fam == dpb.FR else dpb.GL_BASE), F.table_from_i64(x)
            handles.append(mult)
            lib_in.append(P.LogUpInput.new_table(cols, mult, ca, sa))
            orc_in.append(orc.LogUpInput(F, 1, tabs, c, s, mult=mt))
        else:
            lib_in.append(P.LogUpInput.new_lookup(cols, ca, sa, ncol))
            orc_in.append(orc.LogUpInput(F, 0, tabs, c, s, columns_per_instance=ncol))
    return lib_in, orc_in, handles


def prove(ctx, F, fam, lib_in):
    from deep_prove_b200 import prover as P
    tr = P.Blake3Transcript(fam)
    out = P.new_batch_multiple_sizes_prove(ctx, lib_in, tr)
    tr.free()
    return out


LOOKUPS = {"one": [("lookup", 1)], "three": [("lookup", 1), ("lookup", 2), ("lookup", 2)], "nine": [("lookup", 2)] * 9,
           "forty": [("lookup", 1 + j % 2) for j in range(40)]}
TABLES = {"tables": [("table", 1), ("table", 2), ("table", 2)], "one table": [("table", 2)]}


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("name", list(LOOKUPS) + list(TABLES))
@pytest.mark.parametrize("m", [2, 3, 6, 7, 8, 9, 11, 13])
def test_proofs_around_the_switches(dpb, ctx, F, name, m):
    if name == "forty" and m > 9:
        m -= 2
    spec = {**LOOKUPS, **TABLES}[name]
    rng = np.random.default_rng(9700 + 16 * m + len(spec))
    lib_in, orc_in, handles = build(dpb, ctx, F, rng, spec, m, ints=m % 2 == 1)
    want = orc.serialize_logup_proof(F, orc.logup_batch_prove(F, orc_in, orc.Transcript(F)))
    assert prove(ctx, F, family_dtype(dpb, F), lib_in) == want
    for h in handles:
        h.free()


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("name,m,ints", [("three", 12, True), ("nine", 9, False), ("tables", 10, True)])
def test_host_held_up(dpb, F, name, m, ints):
    """The kernel waits 5 ms for a challenge; the host holds one back for 20 ms: every challenge of the proof in turn, so
    that kernels are started again at each of their rounds (one block, a cluster, the hand-over) and at their end."""
    hold = dpb.lib.dpb_resident_hold  # not part of the interface
    hold.restype, hold.argtypes = ctypes.c_uint64, [ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint32]
    none = 2**64 - 1
    ctx = dpb.Context(0)
    rng = np.random.default_rng(9790 + m)
    lib_in, orc_in, handles = build(dpb, ctx, F, rng, {**LOOKUPS, **TABLES}[name], m, ints=ints)
    fam = family_dtype(dpb, F)
    want = orc.serialize_logup_proof(F, orc.logup_batch_prove(F, orc_in, orc.Transcript(F)))
    hold(ctx.h, none, 0)
    before = ctx.sumcheck_launches()
    assert prove(ctx, F, fam, lib_in) == want
    undisturbed = ctx.sumcheck_launches() - before
    ctx.resident_rounds(True, 5)
    posts = hold(ctx.h, none, 0)
    assert posts > m
    for post in range(posts):
        hold(ctx.h, post, 20)
        before = ctx.sumcheck_launches()
        assert prove(ctx, F, fam, lib_in) == want, f"challenge {post} of {posts}"
        # the last one ends the input layer, whose kernel may have nothing left to report
        assert ctx.sumcheck_launches() - before > undisturbed or post == posts - 1, f"challenge {post} of {posts}"
    for h in handles:
        h.free()
    ctx.close()
