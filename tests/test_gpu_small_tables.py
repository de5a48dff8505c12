"""Eq tables made from the tables of a point's parts, and einsum contractions whose outer index is cut over a block's
warps, over blocks, or over a whole block per output: sizes around every switch, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.helpers import family_dtype

pytestmark = pytest.mark.gpu

FIELDS = [orc.FrField, orc.GlField]


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("m", list(range(0, 15)) + [22, 23])
def test_eq_table_sizes(dpb, ctx, F, m):
    rng = np.random.default_rng(9800 + m)
    pt = [F.random_scalar(rng) for _ in range(m)]
    pa = orc.scalars_to_array(F, pt) if m else np.zeros((0, F.elem_words), np.uint64)
    t = ctx.eq_table(family_dtype(dpb, F), pa)
    assert (t.to_host() == orc.eq_evals(F, pt)).all()
    t.free()


O, C, S = 1, 0, 2  # DPB_AXIS_OUTER, CONTRACTED, STACKED


@pytest.mark.parametrize("F", FIELDS)
@pytest.mark.parametrize("shape,kinds", [
    ((1, 5), (O, C)), ((7, 33), (O, C)), ((8, 32), (O, C)), ((127, 31), (O, C)), ((512, 40), (O, C)), ((4099, 3), (O, C)),
    ((700, 1), (O, C)), ((3, 65, 66), (S, O, C)), ((40, 200, 130), (S, O, C)), ((5, 511), (C, O)), ((5, 512), (C, O)),
    ((3, 513), (C, O)), ((200, 1030), (C, O)), ((4, 9, 31), (S, C, O)), ((6, 7, 90), (O, C, O)), ((600, 2, 3), (O, O, C))])
def test_contraction_splits(dpb, ctx, F, shape, kinds):
    rng = np.random.default_rng(9850 + sum(shape))
    t = rng.integers(-2**63, 2**63 - 1, size=shape, dtype=np.int64)
    t[..., ::2] = rng.integers(-2**13, 2**13, size=t[..., ::2].shape)
    pts = [[F.random_scalar(rng) for _ in range(max(d - 1, 0).bit_length())] if k == O else None for d, k in zip(shape, kinds)]
    arrs = [None if p is None else orc.scalars_to_array(F, p) if p else np.zeros((0, F.elem_words), np.uint64) for p in pts]
    want = orc.mles_from_tensor(F, t, kinds, pts)
    owner, views = ctx.einsum_fix_axes(family_dtype(dpb, F), None, kinds, arrs, device_tensor=ctx.upload_tensor_i64(t))
    assert len(views) == len(want)
    for v, w in zip(views, want):
        assert (v.to_host() == w).all()
        v.free()
    owner.free()
