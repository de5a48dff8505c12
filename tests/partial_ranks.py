"""Child process of test_gpu_partial_forms.py: two ranks of a partial sumcheck as threads on one GPU (their exchange is
one_gpu_comm.c's).  argv: field, variables, case, exchange ("shared" or "nccl")."""
import os
import sys
import threading

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from oracle import oracle as orc  # noqa: E402
from tests.conftest import load_package  # noqa: E402
from tests.helpers import family_dtype, terms_array, upload  # noqa: E402


def parts(F, n, case):
    """Per rank: its tables as (entries, point of the eq table they are or None, zero-padded) and its terms."""
    rng = np.random.default_rng(8800 + n)
    full = lambda m=n: (F.random_table_fast(rng, 1 << m), None, False)
    point = lambda m: [F.random_scalar(rng) for _ in range(m)]
    c = [F.random_scalar(rng) for _ in range(4)]
    if case == "padded":  # table * eq table; the second rank's eq tables do not say that they are ones
        out = []
        for tagged in (True, False):
            tabs = []
            for m in (n, n - 2):
                p = point(m)
                tabs += [(F.random_table_fast(rng, 1 << m), None, True), (orc.eq_evals(F, p), p if tagged else None, True)]
            out.append((tabs, {(0, 1): c[0], (2, 3): c[1]}))
        return out
    if case == "product":  # one product of all tables; a list of terms
        return [([full(), full(), full()], {(0, 1, 2): F.one}), ([full(), full(), full()], {(0, 1, 2): c[0], (0, 1): c[1]})]
    assert case == "eq"  # two points; a list without an eq table
    out = []
    for tagged in (True, True, False):
        p = point(n)
        out.append(([full(), full(), (orc.eq_evals(F, p), p if tagged else None, False)], {(2, 0, 1): c[0], (2, 0): c[1]}))
    return [out[0], (out[1][0] + out[2][0], {**out[1][1], **{tuple(i + 3 for i in m): v for m, v in out[2][1].items()}})]


def drive(dpb, ctx, F, n, mles, terms, result, rank):
    tr = orc.Transcript(F)
    sc = dpb.Sumcheck(ctx, n, mles, terms_array(dpb, F, terms), sharded="partial")
    tr.append_scalars([F.from_int(n), F.from_int(sc.degree)])
    proof, point, r = [], [], None
    for _ in range(n):
        proof.append(orc.array_to_scalars(F, sc.round(r)))
        tr.append_scalars(proof[-1])
        point.append(tr.append_and_sample(orc.ROUND_LABEL))
        r = orc.scalars_to_array(F, [point[-1]])
    result[rank] = (proof, point, orc.array_to_scalars(F, sc.finish(r)))
    sc.free()


def main(field, n, case, exchange):
    dpb, F, ranks = load_package(), orc.FIELDS[field], 2
    both = parts(F, n, case)
    tables, terms = [], {}
    for tabs, tm in both:
        terms.update({tuple(i + len(tables) for i in m): v for m, v in tm.items()})
        tables += [orc.zero_pad_table(F, t, n) if padded else t for t, _, padded in tabs]
    proof, point, finals = orc.sumcheck_prove(F, n, tables, terms, orc.Transcript(F))
    uid = dpb.comm_unique_id()
    result, shared = [None] * ranks, [None] * ranks

    def rank_main(g):
        ctx = dpb.Context(0)
        ctx.comm_init(uid, g, ranks)
        shared[g] = ctx.comm_shared_exchange()
        fam, mles = family_dtype(dpb, F), []
        for entries, p, padded in both[g][0]:
            m = upload(dpb, ctx, F, entries) if p is None else ctx.eq_table(fam, orc.scalars_to_array(F, p))
            mles.append(m.zero_padded() if padded else m)
        drive(dpb, ctx, F, n, mles, both[g][1], result, g)
        ctx.comm_free()
        ctx.close()

    threads = [threading.Thread(target=rank_main, args=(g,)) for g in range(ranks)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert shared == [exchange == "shared"] * ranks, shared
    first = 0
    for g in range(ranks):
        k = len(both[g][0])
        assert result[g] is not None, f"rank {g} did not finish"
        assert result[g][0] == proof, f"rank {g}: messages differ from the oracle's"
        assert result[g][1] == point
        assert result[g][2] == finals[first:first + k]
        first += k
    print("equal")


if __name__ == "__main__":
    main(sys.argv[1], int(sys.argv[2]), sys.argv[3], sys.argv[4])
