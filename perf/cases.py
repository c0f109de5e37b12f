"""Performance cases of the library: what users of vortexstark_b200 have it do, through its
public entry points (vortexstark_b200.api and the C ABI of include/vstark.h), from the
smallest calls to the benchmark's headline sizes.

Six kinds of work:

* commit:  api.commit_columns, the commitment-layer step: stwo LDE of every column and the
           row-packed Blake2s root (encoding and commitment of a trace);
* fri:     api.fri_fold_commit, the fold-and-commit chain over one QM31 vector;
* prove:   api.prove_fib, one Fibonacci proof from public inputs to proof bytes;
* batch:   api.Engine, a list of proofs of one size submitted at once and collected;
* cairo:   the Cairo chain: three column groups committed (vs_commit_group_cairo), then
           api.cairo_oods_fri from the AIR quotient to the last FRI layer;
* ntt:     the drop-in transforms of one column, interpolate then evaluate (decode, encode).

Every output is a whole number (field words, hashes, proof bytes) and every correct
implementation gives the same ones, so outputs are compared exactly; parity with the
reference is pinned by the repository's tests.
"""
import ctypes as C
import math

import numpy as np
import torch

import vortexstark_b200 as V
from vortexstark_b200 import api

P = V.P
CAIRO_TRACE, CAIRO_GROUPS = 34, ((0, 16), (16, 31), (31, 34))
COSTLIEST = 34 << 26  # committed words of the largest commitment


def listed():
    return [
        # the smallest commitment in use (a smoke-test trace): latency and launches count
        {"name": "commit 34x2^10", "kind": "commit", "n_cols": 34, "log_n": 10, "blowup": 2},
        # a ragged one: few columns, an odd count, the smallest blowup, below one wave of tiles
        {"name": "commit 7x2^17 x2", "kind": "commit", "n_cols": 7, "log_n": 17, "blowup": 1},
        # the middle size class of the serving mix
        {"name": "commit 34x2^20", "kind": "commit", "n_cols": 34, "log_n": 20, "blowup": 2},
        # the commitment benchmark's size
        {"name": "commit 34x2^24", "kind": "commit", "n_cols": 34, "log_n": 24, "blowup": 2},
        # FRI of a small proof, of an ordinary one (a 2^16-row trace) and of the benchmark
        {"name": "fri 2^10", "kind": "fri", "log_n": 10},
        {"name": "fri 2^18", "kind": "fri", "log_n": 18},
        {"name": "fri 2^26", "kind": "fri", "log_n": 26},
        # single proofs: the plain workload's size and a large one
        {"name": "prove 2^16", "kind": "prove", "log_n": 16},
        {"name": "prove 2^22", "kind": "prove", "log_n": 22},
        # the batched workload: 64 proofs of 2^16 rows
        {"name": "batch 64x2^16", "kind": "batch", "count": 64, "log_n": 16},
        # the Cairo chain at an ordinary trace size
        {"name": "cairo 2^18", "kind": "cairo", "log_n": 18, "n_inter": 12, "blind": True},
        # the reference's single-column transforms, as a caller of the drop-ins makes them
        {"name": "ntt 2^20", "kind": "ntt", "log_n": 20},
    ]


def draw(rng):
    kind = rng.choice(("commit", "commit", "commit", "fri", "fri", "prove", "prove", "batch", "cairo", "cairo", "ntt"))
    if kind == "commit":
        while True:
            c = {"kind": kind, "n_cols": rng.randint(1, 34), "log_n": rng.randint(8, 24), "blowup": rng.randint(1, 3)}
            if c["n_cols"] << (c["log_n"] + c["blowup"]) <= COSTLIEST:
                return c
    if kind == "fri":
        return {"kind": kind, "log_n": rng.randint(5, 26)}
    if kind == "prove":
        return {"kind": kind, "log_n": rng.randint(6, 24)}
    if kind == "batch":
        while True:
            c = {"kind": kind, "count": int(2 ** rng.uniform(0.5, 6)), "log_n": rng.randint(8, 18)}
            if c["count"] << c["log_n"] <= 64 << 16:
                return c
    if kind == "cairo":
        return {"kind": kind, "log_n": rng.randint(6, 21), "n_inter": rng.choice((4, 8, 12)), "blind": rng.random() < 0.5}
    return {"kind": kind, "log_n": rng.randint(6, 24)}


# ---------------------------------------------------------------- what a user's program holds
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _m31(g, *shape):
    return torch.randint(0, P, shape, dtype=torch.int32, device="cuda", generator=g)


def _empty(*shape):
    return torch.empty(shape, dtype=torch.int32, device="cuda")


class _Proofs:
    """A batching engine with its workspaces made, as a proving service keeps one."""

    def __init__(self, count, log_n, seed):
        rng = np.random.default_rng(seed)
        self.jobs = [api.fib_job(log_n, 1, int(b)) for b in rng.integers(1, P, count)]
        self.engine = api.Engine(8, 0)
        self.engine.prepare(self.jobs[0])

    def __del__(self):
        try:
            self.engine.close()
        except Exception:
            pass


def _point_mul(a, b):
    return (a[0] * b[0] - a[1] * b[1]) % P, (a[0] * b[1] + a[1] * b[0]) % P


def _point_double(p, times):
    for _ in range(times):
        p = _point_mul(p, p)
    return p


def _stwo_twiddles(log_n):
    """Flat stwo twiddle table of a 2^log_n transform and its inverse, built with the drop-ins:
    layer k holds the x-coordinates of the first half of half_odds(log_n - 1) doubled k times,
    bit-reversed; a final 1 fills the table to 2^(log_n - 1) words."""
    lib = V.lib()
    half = 1 << (log_n - 1)
    tw, itw = _empty(half), _empty(half)
    g = (2, 1268011823)
    init, step = _point_double(g, 30 - log_n), _point_double(g, 32 - log_n)
    off = 0
    for k in range(log_n - 1):
        m = log_n - 1 - k
        lib.cuda_compute_fold_twiddle_sources(*init, *step, tw[off:].data_ptr(), 1 << m, m, 0)
        off += 1 << (m - 1)
        init, step = _point_double(init, 1), _point_double(step, 1)
    tw[half - 1] = 1
    torch.cuda.synchronize()
    lib.cuda_batch_inverse_m31(tw.data_ptr(), itw.data_ptr(), half)
    torch.cuda.synchronize()
    return tw, itw


def _cairo(case, g):
    log_n = case["log_n"]
    n, N = 1 << log_n, 4 << log_n
    s = {"cols": _m31(g, CAIRO_TRACE, n), "coeffs": _empty(CAIRO_TRACE, n), "evals": _empty(CAIRO_TRACE, N),
         "evals_hc": _empty(CAIRO_TRACE, N), "roots": _empty(3, 8),
         "tiles": [_empty(max(1, N // 1024) * 8) for _ in CAIRO_GROUPS],
         # committed elsewhere in a Cairo proof: interaction columns and the AIR quotient
         "inter": _m31(g, case["n_inter"], N), "quotient": _m31(g, 4, N),
         "quotient_cn": _empty(4, N), "oods_quotient": _empty(4, N)}
    s["blind"] = [int(x) for x in _m31(g, CAIRO_TRACE).cpu()] if case["blind"] else None
    return s


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    api.init_memory_pool()  # once per device, as a program that uses the library does at start-up
    if kind == "commit":
        cols = _m31(g, case["n_cols"], 1 << case["log_n"])
        s = {"cols": cols, "lde": _empty(case["n_cols"], 1 << (case["log_n"] + case["blowup"])), "root": _empty(8)}
    elif kind == "fri":
        n = 1 << case["log_n"]
        rng = np.random.default_rng(seed)
        s = {"src": _m31(g, 4, n), "work": _empty(4 * n), "roots": _empty((case["log_n"] - 3) * 8), "last": _empty(32),
             "alphas": rng.integers(0, P, (case["log_n"] - 3, 4)).tolist()}
    elif kind == "prove":
        s = {"b": int(np.random.default_rng(seed).integers(1, P))}
    elif kind == "batch":
        s = {"proofs": _Proofs(case["count"], case["log_n"], seed)}
    elif kind == "cairo":
        s = _cairo(case, g)
    else:
        tw, itw = _stwo_twiddles(case["log_n"])
        s = {"evals": _m31(g, 1 << case["log_n"]), "coeffs": _empty(1 << case["log_n"]),
             "back": _empty(2 << case["log_n"]), "tw": tw, "itw": itw}
        s["tw2"], _ = _stwo_twiddles(case["log_n"] + 1)
    s["case"] = dict(case)
    return s


# ---------------------------------------------------------------- one pass
def _run_cairo(s):
    case = s["case"]
    log_n = case["log_n"]
    n, N = 1 << log_n, 4 << log_n
    st = torch.cuda.current_stream().cuda_stream
    for g, (a, b) in enumerate(CAIRO_GROUPS):
        blind = (C.c_uint32 * (b - a))(*s["blind"][a:b]) if s["blind"] else None
        V.check(V.lib().vs_commit_group_cairo(s["cols"][a].data_ptr(), n, b - a, log_n, blind, s["coeffs"][a].data_ptr(),
                                              s["evals"][a].data_ptr(), s["evals_hc"][a].data_ptr(),
                                              s["roots"][g].data_ptr(), s["tiles"][g].data_ptr(), st),
                "vs_commit_group_cairo")
    ch = api.Channel()
    for r in s["roots"].cpu().tolist():
        ch.mix_digest([x & 0xFFFFFFFF for x in r])
    out = api.cairo_oods_fri(ch, log_n, list(s["coeffs"]), list(s["evals"]), list(s["inter"]), list(s["quotient"]),
                             zk_scalars=s["blind"], quotient_cn=list(s["quotient_cn"]),
                             oods_quotient=list(s["oods_quotient"]))
    return {"tail": {k: np.array(v, dtype=np.int64) for k, v in out.items()},
            **{k: s[k] for k in ("coeffs", "evals", "evals_hc", "roots", "tiles", "quotient_cn", "oods_quotient")}}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "commit":
        api.commit_columns(s["cols"], case["log_n"], case["blowup"], s["lde"], s["root"])
        return s["lde"], s["root"]
    if kind == "fri":
        api.fri_fold_commit(s["src"], case["log_n"], s["alphas"], s["work"], s["roots"], s["last"])
        return s["roots"], s["last"]
    if kind == "prove":
        return np.frombuffer(api.prove_fib(1, s["b"], case["log_n"]), dtype=np.uint8)
    if kind == "batch":
        p = s["proofs"]
        return [np.frombuffer(p.engine.wait(t)[0], dtype=np.uint8) for t in p.engine.submit_many(p.jobs)]
    if kind == "cairo":
        return _run_cairo(s)
    # coefficients of a column, then its evaluation on the domain of twice the size
    n = 1 << case["log_n"]
    lib = V.lib()
    s["coeffs"].copy_(s["evals"])
    torch.cuda.current_stream().synchronize()
    lib.cuda_stwo_ntt_interpolate(s["coeffs"].data_ptr(), s["itw"].data_ptr(), n)
    lib.cuda_zero_pad(s["coeffs"].data_ptr(), s["back"].data_ptr(), n, 2 * n)
    lib.cuda_stwo_ntt_evaluate(s["back"].data_ptr(), s["tw2"].data_ptr(), 2 * n)
    return s["coeffs"], s["back"]


# ---------------------------------------------------------------- what a pass cannot do without
# Integer operations, counted as "flops": 3 per butterfly (a multiply, an add and a subtract
# mod p) and 1120 per Blake2s compression (10 rounds of 8 G functions, 14 operations each).
BUTTERFLY, BLAKE = 3, 10 * 8 * 14


def _lde_ops(cols, log_n, blowup):
    N = 1 << (log_n + blowup)  # the top `blowup` layers of a zero-padded input only copy
    return cols * BUTTERFLY * ((1 << log_n) // 2 * log_n + N // 2 * log_n)


def _tree_ops(leaves, words):
    return BLAKE * (leaves * max(1, math.ceil(words / 16)) + leaves - 1)


def _fri(log_n):
    n = 1 << log_n
    # per folded value: one QM31 product and one scaling (20 multiplies), its leaf and node hash
    ops = sum((20 * 2 + 2 * BLAKE) * (n >> k) for k in range(1, log_n - 2))
    return 16 * n, ops


def _prove(log_n):
    N = 4 << log_n
    ops = _lde_ops(1, log_n, 2) + _tree_ops(N, 1) + _tree_ops(N, 4) + _fri(log_n + 2)[1]
    proof = 80 * 2 * 32 * sum(range(4, log_n + 3)) + 80 * 2 * 32 * 2 * (log_n + 2)
    return proof, ops


def work(case):
    kind, log_n = case["kind"], case["log_n"]
    n = 1 << log_n
    if kind == "commit":
        c, N = case["n_cols"], n << case["blowup"]
        return {"bytes": 4 * c * (n + N) + 32, "flops": _lde_ops(c, log_n, case["blowup"]) + _tree_ops(N, c)}
    if kind == "fri":
        b, ops = _fri(log_n)
        return {"bytes": b + 32 * (log_n - 3) + 128, "flops": ops}
    if kind in ("prove", "batch"):
        b, ops = _prove(log_n)
        k = case.get("count", 1)
        return {"bytes": k * b, "flops": k * ops}
    if kind == "cairo":
        N = 4 * n
        cols = CAIRO_TRACE + case["n_inter"] + 4
        ops = _lde_ops(CAIRO_TRACE, log_n, 2) + sum(_tree_ops(N, b - a) for a, b in CAIRO_GROUPS) + 2 * _tree_ops(N, 4)
        ops += 2 * 2 * 4 * N * cols + _fri(log_n + 2)[1]  # OODS numerators of two points, then FRI
        # columns, coefficients, both evaluation orders; interaction columns; both quotients in and out
        return {"bytes": 4 * (CAIRO_TRACE * (2 * n + 2 * N) + case["n_inter"] * N + 3 * 4 * N), "flops": ops}
    return {"bytes": 4 * (n + n + 2 * n) + 4 * (n // 2 + n), "flops": BUTTERFLY * (n // 2 * log_n + n * (log_n + 1))}


def tolerance(case):
    return "exact"
