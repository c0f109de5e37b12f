"""GPU checks of the NTT launch-shape autotuner: every candidate plan gives the
oracle's LDE and NTT bit for bit (plans regroup layers into launches, nothing
else), and the tuner keeps one of the candidates and leaves results unchanged. Jobs
here have the columns that take them past the small-job passes, which no plan moves."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from gpu_util import captured, dev, empty, host, ptr, ptr_array, rand_m31, u32_host  # noqa: E402
import vortexstark_b200 as V  # noqa: E402
from vortexstark_b200 import api  # noqa: E402


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return V.lib()


@pytest.fixture(autouse=True)
def default_plans():
    yield
    if torch.cuda.is_available():
        for log_n in range(5, 31):
            api.set_ntt_plan(log_n)


def _lde(L, cols, log_n, native=False):
    n_cols = cols.shape[0]
    N = 1 << (log_n + 2)
    dst = empty(n_cols * N)
    fn = L.vs_lde_native if native else L.vs_lde_stwo
    V.check(fn(ptr(dev(cols.reshape(-1))), 1 << log_n, ptr(dst), N, n_cols, log_n, 2, None), "lde")
    return host(dst).reshape(n_cols, N)


@pytest.mark.parametrize("log_n,n_cols", [(14, 17), (16, 5), (18, 3)])
def test_every_candidate_plan_matches_oracle(L, log_n, n_cols):
    rng = np.random.default_rng(700 + log_n)
    cols = rand_m31(rng, n_cols, 1 << log_n)
    exp = O.stwo_lde_columns(cols, log_n, 2, threads=4)
    cands = api.ntt_plan_candidates(log_n)
    assert len(cands) >= 6
    for plan in cands:
        api.set_ntt_plan(log_n, *plan)
        assert api.ntt_plan(log_n) == tuple(plan)
        assert np.array_equal(_lde(L, cols, log_n), exp), plan


@pytest.mark.parametrize("log_n,n_cols", [(15, 17), (17, 5)])
def test_plans_native_lde_and_transforms(L, log_n, n_cols):
    rng = np.random.default_rng(800 + log_n)
    x = rand_m31(rng, n_cols, 1 << log_n)
    pad = np.zeros(3 << log_n, np.uint32)
    ref = np.stack([O.native_evaluate(np.concatenate([O.native_interpolate(c, log_n), pad]), log_n + 2) for c in x])
    exp_eval = [O.native_evaluate(c.copy(), log_n) for c in x]
    tw = O.native_twiddles(log_n)

    def batch(fn, cols, i=""):
        fn(ptr(ptr_array(cols)), ptr(dev(tw[i + "line"])), ptr(dev(tw[i + "circle"])), u32_host(tw["offsets"]),
           u32_host(tw["sizes"]), log_n - 1, 1 << log_n, n_cols)

    for plan in api.ntt_plan_candidates(log_n)[::5]:
        api.set_ntt_plan(log_n, *plan)
        assert np.array_equal(_lde(L, x, log_n, native=True), ref), plan
        cols = [dev(c) for c in x]
        batch(L.cuda_circle_ntt_evaluate_batch, cols)
        assert all(np.array_equal(host(d), e) for d, e in zip(cols, exp_eval)), plan
        batch(L.cuda_circle_ntt_interpolate_batch, cols, "i")
        assert all(np.array_equal(host(d), c) for d, c in zip(cols, x)), plan
    api.set_ntt_plan(log_n)
    assert np.array_equal(_lde(L, x, log_n, native=True), ref)


@pytest.mark.parametrize("log_n,n_cols,blowup", [(16, 1, 2), (14, 8, 1), (13, 34, 3), (8, 34, 2)])
def test_tuning_a_size_leaves_its_small_jobs_alone(L, tmp_path, log_n, n_cols, blowup):
    """A job of few words runs in the same launches after the size was tuned on 34 columns, and in
    a process that loads the tuning."""
    src, dst = empty(n_cols << log_n), empty(n_cols << (log_n + blowup))
    lde = lambda st: V.check(L.vs_lde_stwo(ptr(src), 1 << log_n, ptr(dst), 1 << (log_n + blowup), n_cols, log_n,
                                           blowup, st))
    lde(None)
    before = captured(lde)
    api.autotune_lde(log_n, n_cols=34, reps=1)
    assert captured(lde) == before
    api.save_tuning(tmp_path / "t.json", [log_n])
    api.set_ntt_plan(log_n)
    api.load_tuning(tmp_path / "t.json")
    assert captured(lde) == before


def test_autotune_keeps_a_candidate_and_results(L):
    log_n = 18
    res = api.autotune_lde(log_n, n_cols=4, reps=2)
    cands = api.ntt_plan_candidates(log_n)
    assert tuple(res["best"]) in [tuple(c) for c in cands]
    assert api.ntt_plan(log_n) == tuple(res["best"])
    times = [ms for _, ms in res["candidates"]]
    assert len(times) == len(cands) and all(t > 0 for t in times)
    assert dict((tuple(c), t) for c, t in res["candidates"])[tuple(res["best"])] == min(times)
    rng = np.random.default_rng(9)
    cols = rand_m31(rng, 2, 1 << log_n)
    assert np.array_equal(_lde(L, cols, log_n), O.stwo_lde_columns(cols, log_n, 2, threads=4))


# ------------------------------------------------------------------ Merkle split
@pytest.fixture
def default_split():
    yield
    if torch.cuda.is_available():
        api.set_merkle_split(0)


@pytest.mark.parametrize("log_n,n_cols,fri_log", [(15, 34, 15), (20, 18, 12), (21, 2, 22)])
def test_every_split_gives_the_oracle_roots(L, default_split, log_n, n_cols, fri_log):
    """The split shapes trees of 2^20 leaves and more and, up to 5, the large FRI layers (two of the
    chain of 2^22 values); smaller ones take no notice of it."""
    rng = np.random.default_rng(900 + log_n)
    cols = rand_m31(rng, n_cols, 1 << log_n)
    exp_rp = O.merkle_root_rowpacked(cols, threads=8)
    n_cap = min(16, n_cols)
    exp_cap = O.merkle_root_capped(cols[:n_cap], threads=8)
    src = rand_m31(rng, 4, 1 << fri_log)
    alphas = rand_m31(rng, fri_log - 3, 4)
    er = np.zeros((fri_log - 3, 8), np.uint32)
    el = np.zeros((8, 4), np.uint32)
    O.lib().oracle_bench_fri(O.ptr_array(list(src)), fri_log, O.ptr(alphas.reshape(-1).copy()), 8, O.ptr(er), O.ptr(el))
    d_cols, d_src = dev(cols.reshape(-1)), dev(src.reshape(-1))
    work, roots, last = empty(4 << fri_log), empty(8 * (fri_log - 3)), empty(32)
    for split in range(9):
        api.set_merkle_split(split)
        root = empty(8)
        V.check(L.vs_merkle_root_rowpacked(ptr(d_cols), 1 << log_n, n_cols, log_n, ptr(root), None), "rowpacked")
        assert np.array_equal(host(root), exp_rp), split
        V.check(L.vs_merkle_root_capped(ptr(d_cols), 1 << log_n, n_cap, log_n, ptr(root), None), "capped")
        assert np.array_equal(host(root), exp_cap), split
        V.check(L.vs_fri_fold_commit(ptr(d_src), fri_log, u32_host(alphas.reshape(-1)), ptr(work),
                                     ptr(roots), ptr(last), None), "vs_fri_fold_commit")
        assert np.array_equal(host(roots).reshape(-1, 8), er), split
        assert np.array_equal(host(last).reshape(8, 4), el), split


def test_autotune_merkle_keeps_a_split(L, default_split):
    res = api.autotune_merkle(21, n_cols=34, reps=2)
    assert 0 <= res["best"] <= 8 and api.merkle_split() == res["best"]
    assert all(t > 0 for t in res["ms"]) and res["ms"][res["best"]] == min(res["ms"])


@pytest.mark.parametrize("log_leaves", [11, 17, 18, 19])
def test_autotune_merkle_leaves_the_split_where_it_is_not_used(L, default_split, log_leaves):
    api.set_merkle_split(6)
    res = api.autotune_merkle(log_leaves, n_cols=3, reps=1)
    assert res["best"] == 6 == api.merkle_split()
    assert len(set(res["ms"])) == 1


def test_autotune_merkle_reports_the_split_that_runs(L, default_split):
    """Split 0 is the library's choice (7 here), timed as such: what is kept is what was measured."""
    for _ in range(3):
        api.set_merkle_split(0)
        res = api.autotune_merkle(21, n_cols=2, reps=3)
        assert res["ms"][0] == res["ms"][7]
        assert res["ms"][res["best"]] == min(res["ms"]) and api.merkle_split() == res["best"] != 7


@pytest.mark.parametrize("split", [1, 5, 8])
def test_prover_trees_with_split_match_oracle(L, default_split, split):
    """The graph prover's trees of 2^20 leaves (log_n 18) go through 2^min(split, 5) subtree
    roots per tile; the bytes stay the oracle's, as do those of vs_prove_fib, whose trees
    keep their lower levels and take no notice of the split."""
    import ctypes as C
    exp = O.prove(3, 77, 18)
    api.set_merkle_split(split)
    assert api.prove_fib(3, 77, 18) == exp
    h = C.c_void_p()
    V.check(L.vs_prover_create(18, C.byref(h)), "vs_prover_create")
    try:
        cap = 16 << 20
        buf = (C.c_uint8 * cap)()
        n = C.c_uint64()
        V.check(L.vs_prover_prove(h, 3, 77, buf, cap, C.byref(n)), "vs_prover_prove")
        assert bytes(buf[: n.value]) == exp
    finally:
        L.vs_prover_destroy(h)
