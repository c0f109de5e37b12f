"""LDEs and transforms in both conventions on either side of the rules that run jobs of few
words in the small-job passes, against the oracle."""
import numpy as np
import pytest

from gpu_util import captured, dev, empty, host, ptr, ptr_array, rand_m31, u32_host

pytestmark = pytest.mark.gpu

import oracle_lib as O  # noqa: E402
import vortexstark_b200 as V  # noqa: E402


def cases():
    for log_n in range(5, 14):
        for blowup in (0, 1, 3):
            yield log_n, blowup, 3
    for log_n, blowup, most in ((13, 3, 37), (13, 0, 148), (12, 2, 96), (10, 1, 592), (5, 2, 1184), (7, 3, 3072),
                                (14, 0, 40)):
        yield log_n, blowup, most      # on either side of the columns it takes
        yield log_n, blowup, most + 1
    yield 8, 4, 2     # more blocks than it takes
    yield 14, 2, 16   # 2^20 evaluation words: the most of a larger transform
    yield 14, 2, 17
    yield 16, 1, 3    # lower and upper passes, clusters of two
    yield 17, 3, 1    # and of eight
    yield 19, 1, 1
    yield 19, 0, 2


@pytest.mark.parametrize("log_n,blowup,n_cols", list(cases()))
def test_small_lde(log_n, blowup, n_cols):
    n, N = 1 << log_n, 1 << (log_n + blowup)
    cols = rand_m31(np.random.default_rng(log_n * 100 + blowup), n_cols, n)
    dst = empty(n_cols * N)
    V.check(V.lib().vs_lde_stwo(ptr(dev(cols.reshape(-1))), n, ptr(dst), N, n_cols, log_n, blowup, None), "vs_lde_stwo")
    assert np.array_equal(host(dst).reshape(n_cols, N), O.stwo_lde_columns(cols, log_n, blowup, threads=8))
    V.check(V.lib().vs_lde_native(ptr(dev(cols[0])), 0, ptr(dst), 0, 1, log_n, blowup, None), "vs_lde_native")
    coeffs = O.native_interpolate(cols[0], log_n)
    exp = O.native_evaluate(np.concatenate([coeffs, np.zeros(N - n, np.uint32)]), log_n + blowup)
    assert np.array_equal(host(dst)[:N], exp)


def _lde_launches(n_cols, log_n, blowup):
    src, dst = empty(n_cols << log_n), empty(n_cols << (log_n + blowup))
    lde = lambda st: V.check(V.lib().vs_lde_stwo(ptr(src), 1 << log_n, ptr(dst), 1 << (log_n + blowup), n_cols, log_n,
                                                 blowup, st))
    lde(None)  # tables are made outside a capture
    return captured(lde)[0]


def test_many_columns_run_in_word_rounds():
    """One CTA of 2^(log_n - 5) threads a column, where that fills the chip (128 columns x4 at 2^13
    rows: 26 us, and 45 in the small-job passes); eight words a thread and a CTA a block otherwise."""
    assert _lde_launches(128, 13, 2) == [((1, 128, 1), (256, 1, 1))]
    assert _lde_launches(34, 13, 2) == [((34, 4, 1), (1024, 1, 1))]
    assert _lde_launches(128, 12, 3) == [((1, 128, 1), (128, 1, 1))]
    assert _lde_launches(34, 12, 3) == [((34, 8, 1), (512, 1, 1))]


@pytest.mark.parametrize("log_n", list(range(5, 21)))
def test_small_transforms(log_n):
    """2^19 words and fewer take the small-job passes, in place, single and batched."""
    L = V.lib()
    x = rand_m31(np.random.default_rng(log_n), 1 << log_n)
    fwd, inv = O.stwo_twiddles(log_n)
    d, tf, ti = dev(x), dev(fwd), dev(inv)
    L.cuda_stwo_ntt_evaluate(ptr(d), ptr(tf), 1 << log_n)
    assert np.array_equal(host(d), O.stwo_evaluate(x, log_n))
    L.cuda_stwo_ntt_interpolate(ptr(d), ptr(ti), 1 << log_n)
    assert np.array_equal(host(d), x)
    cols = [dev(x), dev(x[::-1].copy())]
    tw = O.native_twiddles(log_n)
    arr, line, circle = ptr_array(cols), dev(tw["line"]), dev(tw["circle"])
    L.cuda_circle_ntt_evaluate_batch(ptr(arr), ptr(line), ptr(circle), u32_host(tw["offsets"]), u32_host(tw["sizes"]),
                                     log_n - 1, 1 << log_n, 2)
    for c, v in zip(cols, (x, x[::-1])):
        assert np.array_equal(host(c), O.native_evaluate(v.copy(), log_n))


EDGE = np.array([0, 1, 2**30 - 1, 2**30, 2**30 + 1, 2**31 - 2], dtype=np.uint32)


@pytest.mark.parametrize("forward", [True, False])
def test_butterfly_at_the_ends_of_its_ranges(forward):
    """One layer over every triple of edge values and twiddles."""
    v0, v1, t = (a.reshape(-1) for a in np.meshgrid(EDGE, EDGE, EDGE, indexing="ij"))
    n = 2 * len(t)
    d, tw = np.zeros(512, np.uint32), np.zeros(256, np.uint32)
    d[0:n:2], d[1:n:2], tw[:n // 2] = v0, v1, t
    g = dev(d)
    V.lib().cuda_circle_ntt_layer(ptr(g), ptr(dev(tw)), 0, 512, int(forward))
    assert np.array_equal(host(g), O.ntt_layer(d, tw, 0, forward))


@pytest.mark.parametrize("log_n", [5, 9, 13, 14, 17, 20, 22])
def test_edge_values_through_every_pass_form(log_n):
    """Words at the ends of [0, p) stay in range between layers, rounds and passes."""
    x = EDGE[np.random.default_rng(log_n).integers(0, len(EDGE), (2, 1 << log_n))]
    x[1] = 2**31 - 2
    fwd, inv = O.stwo_twiddles(log_n)
    for row in x:
        d = dev(row)
        V.lib().cuda_stwo_ntt_evaluate(ptr(d), ptr(dev(fwd)), 1 << log_n)
        assert np.array_equal(host(d), O.stwo_evaluate(row, log_n))
        V.lib().cuda_stwo_ntt_interpolate(ptr(d), ptr(dev(inv)), 1 << log_n)
        assert np.array_equal(host(d), row)
    dst = empty(2 << (log_n + 2))
    V.check(V.lib().vs_lde_stwo(ptr(dev(x.reshape(-1))), 1 << log_n, ptr(dst), 4 << log_n, 2, log_n, 2, None), "vs_lde_stwo")
    assert np.array_equal(host(dst).reshape(2, -1), O.stwo_lde_columns(x, log_n, 2, threads=8))


@pytest.mark.parametrize("log_n", list(range(5, 14)))
def test_word_round_lde(log_n):
    """Blowups above 8 run in word rounds, on plain words up to 12 layers and signed words at 13;
    words at the ends of [0, p), both conventions."""
    n, N = 1 << log_n, 16 << log_n
    x = EDGE[np.random.default_rng(log_n).integers(0, len(EDGE), (2, n))]
    dst = empty(2 * N)
    V.check(V.lib().vs_lde_stwo(ptr(dev(x.reshape(-1))), n, ptr(dst), N, 2, log_n, 4, None), "vs_lde_stwo")
    assert np.array_equal(host(dst).reshape(2, N), O.stwo_lde_columns(x, log_n, 4, threads=8))
    V.check(V.lib().vs_lde_native(ptr(dev(x.reshape(-1))), n, ptr(dst), N, 2, log_n, 4, None), "vs_lde_native")
    for got, row in zip(host(dst).reshape(2, N), x):
        coeffs = np.concatenate([O.native_interpolate(row, log_n), np.zeros(N - n, np.uint32)])
        assert np.array_equal(got, O.native_evaluate(coeffs, log_n + 4))
