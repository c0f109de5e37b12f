"""vs_fri_fold_commit at the sizes where its plan changes: one shared launch for all trees,
tiles of 256 to 1024 leaves, one and two fold launches, and the first large layers that take
the fused fold, against the oracle."""
import numpy as np
import pytest

from gpu_util import dev, empty, host, ptr, rand_m31, u32_host

pytestmark = pytest.mark.gpu

import oracle_lib as O  # noqa: E402
import vortexstark_b200 as V  # noqa: E402


@pytest.mark.parametrize("log_n", [4, 5, 7, 10, 11, 12, 13, 14, 16, 18, 19, 20, 21, 22, 23])
def test_fri_chain_at_plan_edges(log_n):
    rng = np.random.default_rng(7100 + log_n)
    src, alphas = rand_m31(rng, 4, 1 << log_n), rand_m31(rng, log_n - 3, 4)
    roots_o, last_o = np.zeros((log_n - 3, 8), np.uint32), np.zeros((8, 4), np.uint32)
    O.lib().oracle_bench_fri(O.ptr_array(list(src)), log_n, O.ptr(alphas.reshape(-1).copy()), 8, O.ptr(roots_o),
                             O.ptr(last_o))
    work, roots, last = empty(4 << log_n), empty(8 * (log_n - 3)), empty(32)
    V.check(V.lib().vs_fri_fold_commit(ptr(dev(src.reshape(-1))), log_n, u32_host(alphas.reshape(-1)), ptr(work),
                                       ptr(roots), ptr(last), None), "vs_fri_fold_commit")
    assert np.array_equal(host(roots).reshape(-1, 8), roots_o)
    assert np.array_equal(host(last).reshape(8, 4), last_o)
