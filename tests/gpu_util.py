"""Device-buffer helpers for the GPU parity tests (torch owns the memory; the
library is called through its C ABI with raw device pointers)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

P = 0x7FFFFFFF


def dev(a) -> torch.Tensor:
    a = np.ascontiguousarray(a, dtype=np.uint32)
    return torch.from_numpy(a.view(np.int32).copy()).cuda()


def empty(n: int) -> torch.Tensor:
    return torch.empty(int(n), dtype=torch.int32, device="cuda")


def zeros(n: int) -> torch.Tensor:
    return torch.zeros(int(n), dtype=torch.int32, device="cuda")


def host(t: torch.Tensor) -> np.ndarray:
    torch.cuda.synchronize()
    return t.cpu().numpy().view(np.uint32)


# Every tensor whose raw pointer is handed to the library stays referenced here
# until the test has synchronised (tests/conftest.py clears it after each test):
# a temporary freed while a launch is queued would be recycled by torch's caching
# allocator and the kernel would read someone else's data.
KEEP: list = []


def ptr(t: torch.Tensor) -> int:
    KEEP.append(t)
    return t.data_ptr()


def ptr_array(ts) -> torch.Tensor:
    """Device array of device pointers (uint32_t**); keeps the columns alive too."""
    ts = list(ts)
    KEEP.extend(ts)
    arr = torch.tensor([t.data_ptr() for t in ts], dtype=torch.int64, device="cuda")
    KEEP.append(arr)
    return arr


def release() -> None:
    torch.cuda.synchronize()
    KEEP.clear()


def u32_host(vals) -> C.Array:
    vals = [int(v) for v in vals]
    return (C.c_uint32 * max(1, len(vals)))(*vals)


def rand_m31(rng: np.random.Generator, *shape) -> np.ndarray:
    return rng.integers(0, P, size=shape, dtype=np.uint64).astype(np.uint32)


# --- tiny exact QM31 helpers for small checks
def qm_mul(x, y):
    a, b, c, d = (int(v) for v in x)
    e, f, g, h = (int(v) for v in y)

    def cm(p, q, r, s):
        return ((p * r - q * s) % P, (p * s + q * r) % P)

    ac = cm(a, b, e, f)
    bd = cm(c, d, g, h)
    ad = cm(a, b, g, h)
    bc = cm(c, d, e, f)
    bdu = ((2 * bd[0] - bd[1]) % P, (bd[0] + 2 * bd[1]) % P)
    return [(ac[0] + bdu[0]) % P, (ac[1] + bdu[1]) % P, (ad[0] + bc[0]) % P, (ad[1] + bc[1]) % P]


def qm_add(x, y):
    return [(int(a) + int(b)) % P for a, b in zip(x, y)]


# --- driver calls of the tests on captured graphs and small memory pools
def _cu(name, *args):
    rc = getattr(C.CDLL("libcuda.so.1"), name)(*args)
    assert rc == 0, f"{name}: {rc}"


class _KernelNode(C.Structure):
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("smem", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def captured(call):
    """What call(stream handle) enqueues, as a capture sees it: the sorted (grid, block) of its
    kernels, and its number of memory nodes (stream-ordered allocations and frees)."""
    s = torch.cuda.Stream()
    st, graph, n = C.c_void_p(s.cuda_stream), C.c_void_p(), C.c_size_t()
    _cu("cuStreamBeginCapture_v2", st, 1)  # errors of this thread only
    try:
        call(s.cuda_stream)
    finally:
        _cu("cuStreamEndCapture", st, C.byref(graph))
    _cu("cuGraphGetNodes", graph, None, C.byref(n))
    nodes = (C.c_void_p * n.value)()
    _cu("cuGraphGetNodes", graph, nodes, C.byref(n))
    kernels, memory = [], 0
    for node in nodes:
        kind, k = C.c_int(), _KernelNode()
        _cu("cuGraphNodeGetType", C.c_void_p(node), C.byref(kind))
        memory += kind.value in (10, 11)  # CU_GRAPH_NODE_TYPE_MEM_ALLOC, _MEM_FREE
        if kind.value == 0:
            _cu("cuGraphKernelNodeGetParams_v2", C.c_void_p(node), C.byref(k))
            kernels.append((tuple(k.grid), tuple(k.block)))
    _cu("cuGraphDestroy", graph)
    return sorted(kernels), memory


class _PoolProps(C.Structure):
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location_type", C.c_int), ("device", C.c_int),
                ("win32", C.c_void_p), ("max_size", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


class small_pool:
    """Stream-ordered allocations come from a pool of at most max_bytes (in steps of 32 MB);
    what does not fit fails."""

    def __init__(self, max_bytes):
        self.props = _PoolProps(alloc_type=1, location_type=1, device=torch.cuda.current_device(), max_size=max_bytes)
        self.held = None

    def __enter__(self):
        torch.cuda.synchronize()
        self.dev, self.old, self.pool = self.props.device, C.c_void_p(), C.c_void_p()
        _cu("cuDeviceGetMemPool", C.byref(self.old), self.dev)
        _cu("cuMemPoolCreate", C.byref(self.pool), C.byref(self.props))
        _cu("cuDeviceSetMemPool", self.dev, self.pool)
        return self

    def hold(self, n_bytes):
        """Takes n_bytes of the pool until the end."""
        self.held = C.c_void_p()
        _cu("cuMemAllocAsync", C.byref(self.held), C.c_size_t(n_bytes), None)

    def __exit__(self, *exc):
        torch.cuda.synchronize()
        if self.held:
            _cu("cuMemFreeAsync", self.held, None)
            torch.cuda.synchronize()
        _cu("cuDeviceSetMemPool", self.dev, self.old)
        _cu("cuMemPoolDestroy", self.pool)
