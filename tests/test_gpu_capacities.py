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
