"""LDEs where the runtime refuses every launch in clusters: a child process loads a stand-in for
the library's one cluster launch that only counts, and the LDEs must come out of their other forms."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

STAND_IN = """
static int n;
extern "C" int vs_internal_cluster_launch(const void*, const void*, void**) { n++; return 801; /* not supported */ }
extern "C" int refused() { return n; }
"""
CHILD = """
import ctypes as C
import numpy as np
from gpu_util import dev, empty, host, ptr
import oracle_lib as O
import vortexstark_b200 as V
L, refused = V.lib(), C.CDLL(None).refused
for log_n, blowup, n_cols in [(5, 3, 2), (9, 2, 3), (13, 3, 2), (14, 2, 3), (16, 0, 2), (17, 3, 1), (19, 1, 1), (24, 1, 1)]:
    n, N = 1 << log_n, 1 << (log_n + blowup)
    cols = O.seeded_m31(log_n, n_cols * n).reshape(n_cols, n)
    exp, before = O.stwo_lde_columns(cols, log_n, blowup, threads=8), refused()
    src, dst = dev(cols.reshape(-1)), empty(n_cols * N)
    V.check(L.vs_lde_stwo(ptr(src), n, ptr(dst), N, n_cols, log_n, blowup, None), "vs_lde_stwo")
    assert np.array_equal(host(dst).reshape(n_cols, N), exp), log_n
    assert refused() == before + 1, log_n
    if n_cols == 1:  # in place
        dst[:n] = src
        V.check(L.vs_lde_stwo(ptr(dst), 0, ptr(dst), 0, 1, log_n, blowup, None), "vs_lde_stwo")
        assert np.array_equal(host(dst), exp[0]), log_n
for log_n in (10, 16):  # with coefficients
    cols = O.seeded_m31(log_n, 2 << log_n).reshape(2, -1)
    co, ev, root = empty(2 << log_n), empty(8 << log_n), empty(8)
    V.check(L.vs_commit_group_cairo(ptr(dev(cols.reshape(-1))), 1 << log_n, 2, log_n, None, ptr(co), ptr(ev), None,
                                    ptr(root), None, None), "vs_commit_group_cairo")
    exp = O.commit_group_cairo(cols, log_n)
    assert np.array_equal(host(co).reshape(2, -1), exp["coeffs"]) and np.array_equal(host(root), exp["root"]), log_n
print("ok", refused())
"""


def test_lde_where_clusters_are_refused(tmp_path):
    (tmp_path / "stand_in.cpp").write_text(STAND_IN)
    so = tmp_path / "stand_in.so"
    subprocess.run(["g++", "-shared", "-fPIC", str(tmp_path / "stand_in.cpp"), "-o", str(so)], check=True)
    root = Path(__file__).resolve().parents[1]
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=f"{root}{os.pathsep}{root / 'tests'}")
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["ok", "13"], r.stdout + r.stderr
