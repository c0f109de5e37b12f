"""vs_prove_fib at the trace sizes between those of test_gpu_prover.py (trees that end in one
launch or two, layers inside and above the last-layers kernel), and from several threads on
streams of their own, byte for byte against the oracle."""
import threading

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import oracle_lib as O  # noqa: E402
from gpu_util import ptr, small_pool, zeros  # noqa: E402
import vortexstark_b200 as V  # noqa: E402
from vortexstark_b200 import api  # noqa: E402


@pytest.mark.parametrize("log_n", [4, 7, 9, 13, 15, 17, 18])
def test_proof_bytes(log_n):
    assert api.prove_fib(3, 1000 + log_n, log_n) == O.prove(3, 1000 + log_n, log_n)


@pytest.mark.parametrize("log_n", [16, 18])
def test_proof_where_the_workspace_cannot_be_allocated(log_n):
    """180 bytes a row do not fit beside what is held, 96 do: trees keep fewer levels."""
    exp = O.prove(5, 50 + log_n, log_n)
    assert api.prove_fib(5, 50 + log_n, log_n) == exp  # tables of the size are cached from here on
    with small_pool(64 << 20) as pool:
        pool.hold((64 << 20) - (130 << log_n))
        assert api.prove_fib(5, 50 + log_n, log_n) == exp


def test_a_refused_workspace_does_not_fail_the_next_call():
    cols, root = zeros(3 << 8), zeros(8)
    with small_pool(32 << 20) as pool:
        pool.hold(32 << 20)
        with pytest.raises(V.VstarkError):
            api.prove_fib(1, 2, 12)
        V.check(V.lib().vs_merkle_root_rowpacked(ptr(cols), 1 << 8, 3, 8, ptr(root), None), "no scratch needed")


def test_threads_and_streams():
    sizes = (6, 9, 12, 14)
    exp = {k: O.prove(1, 7 + k, k) for k in sizes}
    got = {}

    def work(k):
        st = torch.cuda.Stream()
        got[k] = [api.prove_fib(1, 7 + k, k, stream=st) for _ in range(4)]

    th = [threading.Thread(target=work, args=(k,)) for k in sizes]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert all(got[k] == [exp[k]] * 4 for k in sizes)
