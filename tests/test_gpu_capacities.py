"""Decode calls whose output capacity says nothing about the stream: none stated (-1) and
"no limit" (2^63 - 1), each with the stream's length stated and not."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O
from sleek_b200 import _capi, api

pytestmark = pytest.mark.gpu

NO_LIMIT = 2**63 - 1


def _decode(stream, dtype, n, cap, length):
    t = torch.frombuffer(bytearray(stream), dtype=torch.uint8).cuda()
    out = torch.full((n,), 7.0, dtype=torch.float32 if dtype == np.float32 else torch.float64, device="cuda")
    size = torch.zeros(1, dtype=torch.int64, device="cuda")
    f = getattr(_capi.lib(), f"sleek_decompress_f{8 * np.dtype(dtype).itemsize}")
    _capi.check(f(t.data_ptr(), length, out.data_ptr(), cap, size.data_ptr(), None, 0,
                  torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy(), int(size.item())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("cap", [-1, NO_LIMIT, NO_LIMIT - 16383, NO_LIMIT - 16382])
@pytest.mark.parametrize("chunks", [1, 40, 1000])
def test_capacities_without_meaning(cuda, dtype, cap, chunks):
    x = np.cumsum(np.random.default_rng(chunks).normal(0, 1, chunks * 16384 // np.dtype(dtype).itemsize - 3)).astype(dtype)
    s = O.encode(x)
    for length in (-1, len(s)):
        y, size = _decode(s, dtype, x.size, cap, length)
        assert size == x.nbytes and y.tobytes() == x.tobytes(), (cap, length)


@pytest.mark.parametrize("insize", [2**63 - 8, 2**63 - 16376, 2**62])
def test_headers_beyond_the_stream_are_corrupt(cuda, insize):
    s = insize.to_bytes(8, "little") + bytes(4096)
    for cap in (-1, NO_LIMIT):
        y, size = _decode(s, np.float64, 512, cap, len(s))
        assert size == -_capi.SLEEK_ERR_CORRUPT_STREAM
        assert np.all(y == 7.0)


class _KernelNode(C.Structure):  # CUDA_KERNEL_NODE_PARAMS of the driver API
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("smem", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _launched(call):
    """(CTAs, threads per CTA) of the one kernel that `call` launches."""
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
    cu = C.CDLL("libcuda.so.1")
    graph = C.c_void_p(g.raw_cuda_graph())
    n = C.c_size_t(0)
    assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0
    found = []
    for node in nodes:
        kind = C.c_int(-1)
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value == 0:  # a kernel
            p = _KernelNode()
            assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
            found.append((p.grid[0], p.block[0]))
    assert len(found) == 1, found
    return found[0]


def test_small_form_goes_by_the_output_not_by_the_stream(cuda):
    # 100 MB of zeros in 0.2 MB of stream: more chunks than SMs, a stream of a few chunks' length
    n = 6400 * 4096
    s = O.encode(np.zeros(n, np.float32))
    t = torch.frombuffer(bytearray(s), dtype=torch.uint8).cuda()
    out = torch.full((n,), 7.0, device="cuda")
    size = torch.zeros(1, dtype=torch.int64, device="cuda")
    L = _capi.lib()
    ws = torch.empty(L.sleek_decompress_workspace_size(), dtype=torch.uint8, device="cuda")

    def call(cap):
        _capi.check(L.sleek_decompress_f32(t.data_ptr(), t.numel(), out.data_ptr(), cap, size.data_ptr(), ws.data_ptr(),
                                           ws.numel(), torch.cuda.current_stream().cuda_stream))

    known = _launched(lambda: call(n * 4))
    assert _launched(lambda: call(-1)) == known
    small = _launched(lambda: call(40 * 16384))  # (captured only: the stream does not fit)
    assert small[1] != known[1]
    call(-1)
    assert int(size.item()) == n * 4 and not out.any()
