"""The proving path's work as a user's program calls it: sumchecks, einsum layers, lookup layers, attention masks,
claim batching, commitments and embeddings, over the sizes of this repository's workload shapes and tests.

Every output is exact field arithmetic or bytes of a proof: whole numbers, compared for equality.  Tables live on the
GPU before the call (torch owns their memory); proofs come back on the host, as the prover's callers take them.
"""
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    # the package's directory name is not an identifier: it is loaded by path, as its own tests and benchmark do
    name = "deep_prove_b200"
    if name not in sys.modules:
        pkg = os.path.join(ROOT, "deep-prove_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _modules():
    dpb = _package()
    return dpb, importlib.import_module(dpb.__name__ + ".prover"), importlib.import_module(dpb.__name__ + ".workloads"), \
        importlib.import_module(dpb.__name__ + ".pcs")


_CTX = []


def _context():
    # one context per process and GPU, as a prover process keeps it
    if not _CTX:
        _CTX.append(_package().Context(torch.cuda.current_device()))
    return _CTX[0]


def lg(x):
    return max(int(x) - 1, 0).bit_length()


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the dense layer of the two-layer MLP: a short sumcheck, all latency
        dict(name="product_gl_2e10", kind="product", field="gl", ints=False, n=10, k=3),
        # the repository's benchmark: f * g * h over 2^28 base-field entries
        dict(name="product_gl_2e28", kind="product", field="gl", ints=False, n=28, k=3),
        # the same shape over the field the prover runs on, at an ordinary size
        dict(name="product_fr_2e22", kind="product", field="fr", ints=False, n=22, k=3),
        # a transformer's feed-forward projection (GPT-2-small, 512 tokens)
        dict(name="einsum_dense_fr", kind="einsum", form="dense", field="fr", heads=1, rows=512, inner=768, cols=3072),
        # attention scores over a ragged number of tokens
        dict(name="einsum_scores_gl_ragged", kind="einsum", form="scores", field="gl", heads=12, rows=197, inner=64, cols=197),
        # the activation of that feed-forward layer: witness, logup-GKR, linking, multiplicities
        dict(name="lookup_gelu_fr", kind="lookup", field="fr", table="gelu", bits=12, heads=1, rows=512, cols=3072),
        # the MLP's ReLU: the smallest lookup layer
        dict(name="lookup_relu_fr_small", kind="lookup", field="fr", table="relu", bits=12, heads=1, rows=1, cols=1024),
        # softmax over a ragged number of tokens: one instance per head
        dict(name="lookup_softmax_gl_ragged", kind="lookup", field="gl", table="exp", bits=12, heads=12, rows=197, cols=197),
        # the causal mask of one block: an expression over 16 tables of 2^18
        dict(name="mask_fr", kind="mask", field="fr", heads=12, seq=512),
        # the opening's claim batching over a few layers' weights, witness columns and small tables
        dict(name="claims_fr", kind="claims", field="fr", big=12, big_log2=20, mid=40, mid_log2=16, small=64, small_log2=12),
        # witness columns committed next to each other: small integers, one chunk of 2^20 each
        dict(name="commit_columns", kind="commit", scalars="int", columns=6, log2=20),
        # embeddings: bind the columns of a padded 50257 x 768 matrix, then the one-hot sumcheck
        dict(name="embeddings_fr", kind="embeddings", field="fr", vocab=50257, width=768),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    field = rng.choice(["fr", "gl"])
    kind = rng.choice(["product", "einsum", "lookup", "mask", "claims", "commit", "embeddings"])
    if kind == "product":
        ints = rng.random() < 0.3
        return dict(kind=kind, field=field, ints=ints, n=rng.randint(4, 23 if field == "fr" else 26), k=rng.choice([2, 3, 3, 4]))
    if kind == "einsum":
        form = rng.choice(["dense", "scores", "values"])
        if form == "dense":
            return dict(kind=kind, form=form, field=field, heads=1, rows=log_int(1, 1024), inner=log_int(16, 3072),
                        cols=log_int(10, 4096))
        t = log_int(8, 512)
        heads, dh = log_int(1, 16), rng.choice([16, 48, 64, 80, 128])
        return dict(kind=kind, form=form, field=field, heads=heads, rows=t, inner=dh if form == "scores" else t,
                    cols=t if form == "scores" else dh)
    if kind == "lookup":
        table = rng.choice(["gelu", "relu", "requant", "exp"])
        if table == "exp":
            t = log_int(8, 320)
            return dict(kind=kind, field=field, table=table, bits=rng.choice([8, 10, 12]), heads=log_int(1, 12), rows=t, cols=t)
        return dict(kind=kind, field=field, table=table, bits=rng.choice([8, 10, 12]), heads=1, rows=log_int(1, 512),
                    cols=log_int(64, 3072))
    if kind == "mask":
        return dict(kind=kind, field=field, heads=log_int(1, 12), seq=log_int(8, 512))
    if kind == "claims":
        return dict(kind=kind, field=field, big=log_int(1, 10), big_log2=rng.randint(14, 20), mid=log_int(1, 40),
                    mid_log2=rng.randint(10, 16), small=log_int(1, 64), small_log2=rng.randint(4, 12))
    if kind == "commit":
        scalars = rng.choice(["int", "field"])
        return dict(kind=kind, scalars=scalars, columns=log_int(1, 6) if scalars == "int" else 1,
                    log2=rng.randint(10, 20 if scalars == "int" else 19))
    return dict(kind=kind, field=field, vocab=log_int(100, 50257), width=log_int(24, 1024))


# ------------------------------------------------------------------------------------------------ inputs
class State:
    """What the program keeps: device tensors, library handles over them, points and challenges."""

    def __init__(self, field, seed):
        self.dpb, self.prover, self.workloads, self.pcs = _modules()
        self.ctx = _context()
        fr = field == "fr"
        dpb = self.dpb
        self.family, self.base, self.words = (dpb.FR, dpb.FR, 4) if fr else (dpb.GL_EXT, dpb.GL_BASE, 2)
        self.i32, self.i64 = (dpb.FR_I32, dpb.FR_I64) if fr else (dpb.GL_I32, dpb.GL_I64)
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.np = np.random.default_rng(seed)
        self.keep, self.handles, self.last = [], [], []
        self.one = np.frombuffer(dpb.one_bytes(self.family), dtype=np.uint64).copy()

    def __del__(self):
        try:
            for h in self.last + self.handles[::-1]:
                h.free()
        except Exception:
            pass  # interpreter shutdown

    def ints(self, lo, hi, shape):
        return torch.randint(lo, hi, shape, generator=self.gen, device="cuda", dtype=torch.int64)

    def wrap(self, t, dtype, n):
        self.keep.append(t)
        h = self.ctx.wrap_device(t.data_ptr(), dtype, n)
        self.handles.append(h)
        return h

    def int_table(self, t):
        """A table of integers, 4 bytes an entry, as quantised tensors are kept."""
        return self.wrap(t.reshape(-1).to(torch.int32), self.i32, t.numel())

    def field_table(self, n):
        """Uniform field elements (base field of Goldilocks; BN254 in the library's Montgomery layout)."""
        if self.family == self.dpb.FR:
            t = self.ints(-2**63, 2**63 - 1, (n, 4))
            t[:, 3] &= (1 << 60) - 1
        else:
            t = self.ints(-2**63, 2**63 - 1, (n,))
            t = torch.where(t >= -(2**32) + 1, torch.where(t < 0, t & (2**63 - 1), t), t)  # below the modulus
        return self.wrap(t, self.base, n)

    def tensor(self, t):
        """An int64 tensor in the padded device form that the axis fixing and the lookup witness take."""
        n = 1 << lg(t.numel())
        flat = torch.zeros(n, dtype=torch.int64, device="cuda")
        flat[:t.numel()] = t.reshape(-1)
        return self.wrap(flat, self.dpb.GL_BASE, n), tuple(t.shape)

    def point(self, m):
        p = self.np.integers(0, 2**62, size=(m, self.words), dtype=np.uint64)
        if self.words == 4:
            p[:, 3] &= np.uint64((1 << 60) - 1)
        return p

    def transcript(self):
        return self.prover.Blake3Transcript(self.family)

    def constant(self, x):
        """A small integer as a challenge element."""
        if self.words == 2:
            return np.array([x % (2**64 - 2**32 + 1), 0], dtype=np.uint64)
        v = (x << 256) % self.dpb.FR_MODULUS
        return np.frombuffer(v.to_bytes(32, "little"), dtype=np.uint64).copy()

    def terms(self, terms):
        return self.dpb.make_terms(terms, lambda c: np.ascontiguousarray(c, dtype=np.uint64).tobytes())


class _DeviceWords:
    def __init__(self, mle, words):
        self.__cuda_array_interface__ = {"shape": (words,), "typestr": "<i8", "data": (mle.device_ptr, False), "version": 3}


def _view(mle, words):
    """A device table's 64-bit words as a torch tensor, without a copy."""
    return torch.as_tensor(_DeviceWords(mle, words), device="cuda")


def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


VALUE_SHIFT = {"gelu": 1, "relu": 1, "requant": 1, "exp": -2}
VALUE_HEADROOM = {"gelu": 4, "relu": 4, "requant": 4, "exp": 10}


def prepare(case, seed):
    kind = case["kind"]
    s = State(case.get("field", "fr"), seed)
    dpb, P, W = s.dpb, s.prover, s.workloads
    if kind == "product":
        N = 1 << case["n"]
        s.tabs = [s.int_table(s.ints(-2**31, 2**31, (N,))) if case["ints"] else s.field_table(N) for _ in range(case["k"])]
        s.term_array = s.terms([(s.one, list(range(case["k"])))])
    elif kind == "einsum":
        h, r, c, q = case["heads"], case["rows"], case["inner"], case["cols"]
        O, C, S = dpb.AXIS_OUTER, dpb.AXIS_CONTRACTED, dpb.AXIS_STACKED
        if case["form"] == "dense":
            lhs, lk, lp = s.ints(-2**13, 2**13, (r, c)), (O, C), [s.point(lg(r)), None]
            rhs, rk, rp = s.ints(-2**11, 2**11, (c, q)), (C, O), [None, s.point(lg(q))]
        else:
            head = s.point(lg(h))
            lhs, lk, lp = s.ints(-2**13, 2**13, (h, r, c)), (S, O, C), [head, s.point(lg(r)), None]
            if case["form"] == "scores":
                rhs, rk, rp = s.ints(-2**13, 2**13, (h, q, c)), (S, O, C), [head, s.point(lg(q)), None]
            else:
                rhs, rk, rp = s.ints(-2**13, 2**13, (h, c, q)), (S, C, O), [head, None, s.point(lg(q))]
        s.lhs = P.EinsumOperand(None, lk, lp, device_tensor=s.tensor(lhs))
        s.rhs = P.EinsumOperand(None, rk, rp, device_tensor=s.tensor(rhs))
    elif kind == "lookup":
        bits, table = case["bits"], case["table"]
        s.sign, s.table_out, s.table_columns = W.value_table(table, bits)
        max_bits = 2 * bits + VALUE_HEADROOM[table]
        s.info = dpb.ChunkingInfo.new(bits + VALUE_SHIFT[table], bits, s.sign, max_bits, 1)
        shape = (case["heads"], case["rows"], case["cols"]) if case["heads"] > 1 else (case["rows"], case["cols"])
        # rescaled values: bell-shaped, a small share beyond the table's range, all within the declared size
        x = torch.randn(shape, generator=s.gen, device="cuda", dtype=torch.float64)
        x = (x * (1 << (2 * bits - 1 + (VALUE_SHIFT[table] > 0) - 1))).round().to(torch.int64)
        limit = (1 << (max_bits - 2)) - 1
        x = x.clamp(-limit, limit)
        if s.sign == dpb.SIGN_NEGATIVE:
            x = -x.abs()
        s.shape, s.tensor_dev = shape, s.tensor(x)
        s.table_dev = None
        if s.table_out is not None:
            s.table_dev = s.tensor(torch.from_numpy(s.table_out).cuda())
        s.chal = [s.point(2) for _ in range(4)]  # constant and column separation per table
        n2d = lg(shape[-2]) + lg(shape[-1])
        s.claim_point = s.point(n2d + (lg(shape[0]) if len(shape) > 2 else 0))
        s.logup_point = s.point(n2d)
        s.variant = P.VARIANT_SOFTMAX if table == "exp" else P.VARIANT_STANDARD
        if s.table_out is None:
            s.out_range = W.table_input_range(bits, s.sign)
        else:
            s.out_range = (int(s.table_out[0]), int(s.table_out[-1]))
    elif kind == "mask":
        h, seq = case["heads"], case["seq"]
        ps, s.n = 1 << lg(seq), 2 * lg(seq)
        i = torch.arange(ps, device="cuda")
        s.tabs = [s.int_table((i[None, :] <= i[:, None]).to(torch.int64)),
                  s.int_table((i < seq).to(torch.int64).repeat_interleave(ps)),
                  s.int_table((i < seq).to(torch.int64).repeat(ps))]
        s.tabs += [s.int_table(s.ints(-2**13, 2**13, (ps * ps,))) for _ in range(h)]
        s.eq_point, s.chi = s.point(s.n), s.point(h)
        X = P.Expression
        const = lambda v: X.Constant(s.constant(v).tobytes())
        zero = np.zeros(s.words, dtype=np.uint64).tobytes()
        s.expr = None
        for j in range(h):
            term = X.WitIn(0) * (X.WitIn(2) * X.WitIn(3)) * X.Challenge(j, 1, s.one.tobytes(), zero) * \
                (X.WitIn(1) * X.WitIn(4 + j) + const(-2**24) * (const(1) - X.WitIn(1)))
            s.expr = term if s.expr is None else s.expr + term
    elif kind == "claims":
        s.polys = []
        for name, lo, hi in (("big", -2**11, 2**11), ("mid", 0, 2**16), ("small", -2**13, 2**13)):
            for i in range(case[name]):
                m = case[name + "_log2"]
                chunks = 4 if name == "big" and i == 0 else 1  # the first weight is cut into four chunks
                tab = s.int_table(s.ints(lo, hi, (chunks << m,)))
                parts = [tab] if chunks == 1 else [tab.view(c << m, 1 << m) for c in range(chunks)]
                if chunks > 1:
                    s.handles += parts
                s.polys.append(P.CommittedPoly(parts, [(s.point(m + lg(chunks)), s.point(1)[0])]))
        s.polys.sort(key=lambda p: -p.chunks[0].len)
    elif kind == "commit":
        N = 1 << case["log2"]
        s.bases = s.pcs.G1Bases.synthetic(s.ctx, N, 1)
        s.handles.append(s.bases)
        s.tabs = []
        for j in range(case["columns"]):
            if case["scalars"] == "field":
                s.tabs.append(s.field_table(N))
            elif j % 3 == 2:  # a sign or zero-check column: almost all of one value
                s.tabs.append(s.int_table((s.ints(0, 100, (N,)) < 2).to(torch.int64)))
            else:             # a 16-bit chunk, a table input
                s.tabs.append(s.int_table(s.ints(0, 2**16, (N,)) if j % 3 == 0 else s.ints(-2**11, 2**11, (N,))))
    elif kind == "embeddings":
        V, e = case["vocab"], case["width"]
        pv, pe = 1 << lg(V), 1 << lg(e)
        m = torch.zeros((pv, pe), dtype=torch.int64, device="cuda")
        m[:V, :e] = s.ints(-2**11, 2**11, (V, e))
        s.n = lg(pv)
        s.matrix, s.one_hot = s.int_table(m), s.int_table(s.ints(0, 3, (pv,)))
        s.col_point = s.point(lg(e))
        s.term_array = s.terms([(s.one, [0, 1])])
    torch.cuda.synchronize()  # the library's stream reads what torch's stream wrote
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _sumcheck(s, n, tabs, terms):
    tr = s.transcript()
    st = s.prover.IOPProverState.prove(s.ctx, n, tabs, terms, tr)
    tr.free()
    return [st.proof, st.collect_raw_challenges(), st.get_mle_flatten_final_evaluations()]


def _lookup(s):
    dpb, P = s.dpb, s.prover
    bits = int(s.info.value_chunk_bits)
    counts = [dpb.LookupCounts(s.ctx, b) for b in (16, bits, 16, 16)]
    owner, ins, outs = dpb.lookup_witness(s.ctx, s.i64, s.info, 1, 0, None, s.table_out, s.table_columns, counts,
                                          device_tensor=s.tensor_dev, device_table=s.table_dev)
    n_sh, n_z = s.info.n_shifted_chunks, s.info.n_zeroing_chunks
    slices = s.shape[0] if len(s.shape) > 2 else 1
    value_in = 1 if s.table_columns != 1 else 0
    per_in, per_out = n_sh + value_in + n_z, 1 + n_z
    shift, value, zero, signed = [], [], [], []
    for c in range(slices):
        i0, o0 = c * per_in, c * per_out
        shift += ins[i0:i0 + n_sh]
        value += ([ins[i0 + n_sh]] if value_in else []) + [outs[o0]]
        for z in range(n_z):
            group = signed if s.sign == dpb.SIGN_MIXED and z == n_z - 1 else zero
            group += [ins[i0 + n_sh + value_in + z], outs[o0 + 1 + z]]
    inputs = [P.LogUpInput.new_lookup(cols, ch[0], ch[1], cpi)
              for cols, ch, cpi in zip((shift, value, zero, signed), s.chal, (1, s.table_columns, 2, 2)) if cols]
    tr = s.transcript()
    proof = P.new_batch_multiple_sizes_prove(s.ctx, inputs, tr)
    link = P.lookup_linking_prove(s.ctx, tr, s.variant, s.info, s.out_range[0], s.out_range[1], s.shape, list(outs),
                                  s.claim_point, s.logup_point)
    tr.free()
    mults = [c.multiplicities(s.family) for c in counts]
    s.ctx.sync()  # the tables below are read on another stream
    s.last = ins + outs + [owner] + mults + counts
    return [_bytes(proof), link["sumcheck"], link["point"], link["evaluations"], link["challenges"]] + \
        [_view(owner, (len(ins) + len(outs)) * ins[0].len)] + \
        [_view(h, h.len * dpb.elem_words(h.dtype)) for h in mults]  # the columns lie one after the other


def run(s):
    P = s.prover
    for h in s.last:  # the device tables that the last pass returned
        h.free()
    s.last = []
    if hasattr(s, "lhs"):
        tr = s.transcript()
        proof = P.einsum_prove(s.ctx, [s.lhs], [s.rhs], tr)
        tr.free()
        return _bytes(proof)
    if hasattr(s, "tensor_dev"):
        return _lookup(s)
    if hasattr(s, "expr"):
        eq = s.ctx.eq_table(s.family, s.eq_point)
        out = _sumcheck(s, s.n, [eq] + s.tabs, s.expr.to_terms(s.family, s.chi))
        eq.free()
        return out
    if hasattr(s, "polys"):
        tr = s.transcript()
        got = P.claims_batching_prove(s.ctx, tr, s.polys)
        tr.free()
        s.ctx.sync()
        s.last = [got["rlc"]]
        return [got["sumcheck"], got["point"], got["sumcheck_evals"], got["rlc_challenges"], _view(got["rlc"], got["rlc"].len * s.words)]
    if hasattr(s, "bases"):
        pts = s.pcs.batch_commit(s.ctx, s.bases, s.tabs)
        return _bytes(b"".join(int(x).to_bytes(32, "little") + int(y).to_bytes(32, "little") for x, y in pts))
    if hasattr(s, "matrix"):
        fixed = s.ctx.fix_low(s.matrix, s.col_point)
        out = _sumcheck(s, s.n, [s.one_hot, fixed], s.term_array)
        s.last = [fixed]
        s.ctx.sync()
        return out + [_view(fixed, fixed.len * s.words)]
    return _sumcheck(s, len_log2(s.tabs[0]), s.tabs, s.term_array)


def len_log2(table):
    return int(table.len).bit_length() - 1


# ------------------------------------------------------------------------------------------------ work
# multiplications and additions of 32-bit words that one field product takes, schoolbook with its reduction: 8 x 8
# words twice over for BN254; 2 x 2 words four times over (extension) and reductions for Goldilocks
PRODUCT_OPS = {"fr": 2 * 128, "gl": 2 * 20}


def work(case):
    kind, field = case["kind"], case.get("field", "fr")
    es, ops = (32 if field == "fr" else 16), PRODUCT_OPS[field]
    if kind == "product":
        N = 1 << case["n"]
        entry = 4 if case["ints"] else 32 if field == "fr" else 8
        k = case["k"]
        # (k + 1) points of k - 1 products a pair and one product a fold, over all rounds
        return {"bytes": k * N * entry, "flops": N * ((k - 1) * (k + 1) + k) * ops}
    if kind == "einsum":
        h, r, c, q = case["heads"], case["rows"], case["inner"], case["cols"]
        entries = h * (r * c + c * q)
        return {"bytes": 8 * entries, "flops": entries * 2 * 16}
    if kind == "lookup":
        pad = case["heads"] << (lg(case["rows"]) + lg(case["cols"]))
        entries = case["heads"] * case["rows"] * case["cols"]
        # five columns written; per instance and entry about 12 products in the layers' rounds and 3 in the tree
        return {"bytes": 8 * entries + 40 * pad, "flops": pad * 3 * 15 * ops}
    if kind == "mask":
        N = 1 << (2 * lg(case["seq"]))
        return {"bytes": 4 * N * (3 + case["heads"]), "flops": N * (case["heads"] * 5 + 15) * ops}
    if kind == "claims":
        N = sum(case[n] << case[n + "_log2"] for n in ("big", "mid", "small")) + (3 << case["big_log2"])
        return {"bytes": 4 * N + (es << case["big_log2"]), "flops": N * 6 * ops}
    if kind == "commit":
        N = 1 << case["log2"]
        # one mixed addition (about 11 products) per point and touched 16-bit window
        windows = case["columns"] if case["scalars"] == "int" else 16
        return {"bytes": N * 64 + case["columns"] * N * (4 if case["scalars"] == "int" else 32),
                "flops": N * windows * 11 * 2 * 128}
    N = 1 << (lg(case["vocab"]) + lg(case["width"]))
    return {"bytes": 4 * N, "flops": N * 2 * 8}


def tolerance(case):
    return "exact"


def exact(case, seed):
    # elements of finite fields and proof bytes: there is no rounding that a wider type would remove
    return None
