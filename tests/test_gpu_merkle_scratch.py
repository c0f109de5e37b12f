"""What root-only trees take besides their input: nothing up to 1024 leaves where that matters
(a capture, the variant without allocations), and no more than there is."""
import numpy as np
import pytest

from gpu_util import captured, dev, host, ptr, small_pool, zeros

pytestmark = pytest.mark.gpu

import oracle_lib as O  # noqa: E402
import vortexstark_b200 as V  # noqa: E402


def _cols(log_leaves, n_cols=3):
    cols = O.seeded_m31(0x99 + log_leaves, n_cols << log_leaves).reshape(n_cols, -1)
    return cols, dev(cols)


@pytest.mark.parametrize("log_leaves", [8, 9, 10])
def test_noalloc_roots_up_to_1024_leaves_share_nothing(log_leaves):
    """One launch, so no hashes pass through the array that all calls share, and calls may overlap."""
    cols, d = _cols(log_leaves)
    root = zeros(8)
    kernels, memory = captured(lambda st: V.check(V.lib().vs_merkle_root_rowpacked_noalloc(
        ptr(d), 1 << log_leaves, 3, log_leaves, ptr(root), st)))
    assert len(kernels) == 1 and memory == 0
    V.check(V.lib().vs_merkle_root_rowpacked_noalloc(ptr(d), 1 << log_leaves, 3, log_leaves, ptr(root), None))
    assert np.array_equal(host(root), O.merkle_root_rowpacked(cols))


def _launches(call):
    before = V.lib().vs_launch_count()
    call()
    return V.lib().vs_launch_count() - before


def test_trees_that_one_launch_ends():
    """2^9 leaves, and 2^10 hashes: a second launch costs more than it saves."""
    L = V.lib()
    cols, d = _cols(9)
    root = zeros(8)
    assert _launches(lambda: V.check(L.vs_merkle_root_rowpacked(ptr(d), 1 << 9, 3, 9, ptr(root), None))) == 1
    assert np.array_equal(host(root), O.merkle_root_rowpacked(cols))
    q = O.seeded_m31(0x55, 4 << 9).reshape(4, -1)
    assert _launches(lambda: L.cuda_merkle_commit_small_soa4(*[ptr(dev(c)) for c in q], ptr(root), 1 << 9)) == 1
    assert np.array_equal(host(root), O.merkle_root_soa4(q))
    for log_n in (9, 10):
        nodes = O.seeded_m31(0x66 + log_n, 8 << log_n)
        assert _launches(lambda: L.cuda_merkle_reduce_to_root(ptr(dev(nodes)), ptr(root), 1 << log_n)) == 1
        assert np.array_equal(host(root), O.merkle_root_hashes(nodes.reshape(-1, 8)))


@pytest.mark.parametrize("log_leaves,held", [(24, 0), (10, 32 << 20)])
def test_roots_where_scratch_cannot_be_allocated(log_leaves, held):
    """The default split's 80 MB at 2^24 leaves, and any scratch at 2^10: the tree then leaves one
    root a tile, which takes 0.5 MB and none."""
    n = 1 << log_leaves
    d, root, less = zeros(n), zeros(8), zeros(8)
    V.check(V.lib().vs_fill_uniform_m31(ptr(d), n, 7, 0, None))
    V.check(V.lib().vs_merkle_root_rowpacked(ptr(d), n, 1, log_leaves, ptr(root), None))
    with small_pool(32 << 20) as pool:
        if held:
            pool.hold(held)
        V.check(V.lib().vs_merkle_root_rowpacked(ptr(d), n, 1, log_leaves, ptr(less), None))
    assert np.array_equal(host(less), host(root))


def test_captured_roots_up_to_1024_leaves_have_no_memory_nodes():
    cols, d = _cols(10)
    root = zeros(8)
    kernels, memory = captured(lambda st: V.check(V.lib().vs_merkle_root_rowpacked(ptr(d), 1 << 10, 3, 10, ptr(root), st)))
    assert len(kernels) == 1 and memory == 0
