"""What root-only trees take besides their input: nothing up to 1024 leaves where that matters
(a capture, the variant without allocations), and no more than there is."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import captured, dev, empty, host, ptr, small_pool, zeros

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
