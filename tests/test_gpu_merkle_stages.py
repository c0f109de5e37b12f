"""Root-only trees at the sizes where their plan changes (one tile; tiles of 128 to 1024
leaves; tiles that stop at 128 roots; one and two more reduction levels), with and without
an allocation, against the oracle."""
import numpy as np
import pytest

from gpu_util import dev, host, ptr, zeros

pytestmark = pytest.mark.gpu

import oracle_lib as O  # noqa: E402
import vortexstark_b200 as V  # noqa: E402


@pytest.mark.parametrize("log_leaves", [0, 1, 2, 4, 7, 8, 9, 10, 13, 14, 15, 16, 17, 18, 19, 20, 21, 22])
def test_roots_at_plan_edges(log_leaves):
    n_cols = 17 if log_leaves <= 16 else 2  # two compressions a leaf, or one
    cols = O.seeded_m31(0x77 + log_leaves, n_cols << log_leaves).reshape(n_cols, -1)
    d, exp = dev(cols), O.merkle_root_rowpacked(cols, threads=8)
    roots = [zeros(8) for _ in range(3)]
    for r, fn in zip(roots, ("", "", "_noalloc")):
        V.check(getattr(V.lib(), "vs_merkle_root_rowpacked" + fn)(ptr(d), 1 << log_leaves, n_cols, log_leaves, ptr(r), None))
    for r in roots:
        assert np.array_equal(host(r), exp)
