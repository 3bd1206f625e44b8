"""Decoding into a view that is element- but not 16-byte aligned: about as fast as into an
aligned output (the stores are whole granules there too)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sleek_b200 import api

pytestmark = pytest.mark.gpu


def _us(call, n=20):
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    for _ in range(n):
        call()
    end.record()
    torch.cuda.synchronize()
    return start.elapsed_time(end) / n * 1e3


def test_a_view_at_element_one_costs_little_more(cuda):
    # 134 MB of f64 at
    # eb 1e-4: narrow codes, so that the stores are the larger part of the work
    n, eb = 1 << 24, 1e-4
    part = np.cumsum(np.random.default_rng(3).normal(0, 1e-3, 1 << 20))
    x = np.tile(part, 16)
    s = torch.frombuffer(bytearray(O.encode(x, eb)), dtype=torch.uint8).cuda()
    info = api.sleek_error_bound(eb, np.float64)
    buf = torch.empty(n + 2, dtype=torch.float64, device="cuda")
    size = torch.zeros(1, dtype=torch.int64, device="cuda")

    def decode(first):
        api.sleek_decompress_gpu(0, info, s, buf[first:first + n], size, encoded_bytes=s.numel())

    decode(0)
    aligned = buf[:n].clone()
    decode(1)
    assert int(size.item()) == x.nbytes and torch.equal(buf[1:n + 1], aligned)
    runs = [(_us(lambda: decode(0)), _us(lambda: decode(1))) for _ in range(7)]
    a, b = (sorted(r[k] for r in runs)[3] for k in (0, 1))
    assert b < 1.3 * a, (a, b)
