"""Terms that share a cofactor run as one term over their tables' linear combination.  The combination needs memory of
its own; a call whose fold buffers alone still fit succeeds all the same."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes, importlib, sys
import numpy as np
sys.path.insert(0, {root!r})
from oracle import oracle as orc
from tests.conftest import load_package
dpb = load_package()
prover = importlib.import_module("deep_prove_b200.prover")
F, n, case = orc.FrField, 24, {case!r}
ctx, rng = dpb.Context(0), np.random.default_rng(31)
point = lambda: orc.scalars_to_array(F, [F.random_scalar(rng) for _ in range(n)])
column = lambda: ctx.upload_ints(rng.integers(-2**31, 2**31, size=1 << n, dtype=np.int64), dpb.FR_I32)
members = [ctx.eq_table(dpb.FR, point()) for _ in range(2)] if case == "begin" else [column() for _ in range(3)]
tabs = members + [column() if case == "begin" else ctx.eq_table(dpb.FR, point())]
terms = dpb.make_terms([(F.random_scalar(rng), [j, len(members)]) for j in range(len(members))], F.to_native)

def prove():
    st = prover.IOPProverState.prove(ctx, n, tabs, terms, prover.Blake3Transcript(dpb.FR))
    return [np.asarray(v).tobytes() for v in (st.proof, st.collect_raw_challenges(), st.get_mle_flatten_final_evaluations())]

want = prove()
table = 32 << n
# per table 3/4 of it for the fold buffers without the combination; with it, in table sizes: at the start 1 + 3/4 * 2, at
# the end 1 + 3/4 * 2 and 1 for the eq table the members are evaluated with
room = {{"begin": 3 * 0.75 * table, "finish": 4 * 0.75 * table}}[case] + (64 << 20)
assert room < {{"begin": 2.5, "finish": 3.5}}[case] * table
ctx.trim()
rt = ctypes.CDLL("libcudart.so.12")
free, total, filler = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_void_p()
assert rt.cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) == 0
assert rt.cudaMalloc(ctypes.byref(filler), ctypes.c_size_t(free.value - int(room))) == 0
assert prove() == want
rt.cudaFree(filler)
print("equal")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["begin", "finish"])
def test_room_for_the_fold_buffers_alone(case):
    env = dict(os.environ, DPB_ARENA="0")  # allocations of the size asked for
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, case=case)], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "equal", r.stdout[-1000:] + r.stderr[-2000:]
