"""The decoder's unpacking and placing at the widths, alignments, launch shapes and
table sizes where its paths change: every code width, raw chunks among compressed
ones, outputs at every element offset, size tables of more than one window, and
batches whose streams hold fewer chunks than their outputs have room for."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sleek_b200 import _capi, api
from sleek_b200.batch import BatchPlan
from tests.test_gpu_encode_widths import CASES, _codes

pytestmark = pytest.mark.gpu


@pytest.fixture
def default_shapes():
    yield
    for w in (4, 8):
        for lossy in (0, 1):
            _capi.check(_capi.lib().sleek_set_launch_shape(1, w, lossy, -1, 0, 0))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("eb", [None, 0.5])
def test_widths_shapes_and_offsets(cuda, default_shapes, dt, case, eb):
    x = _codes(dt, case, 9)[:-3]
    stream = O.encode(x, eb)
    want = O.decode(stream, dt, eb).tobytes()
    t = torch.frombuffer(bytearray(stream), dtype=torch.uint8).cuda()
    buf = torch.empty(x.size + 8, dtype=torch.from_numpy(x).dtype, device="cuda")
    for shape in range(3):
        _capi.check(_capi.lib().sleek_set_launch_shape(1, x.itemsize, int(eb is not None), -1, shape, int(shape > 0)))
        for first in range(16 // x.itemsize):
            buf.fill_(7.0)
            y = api.decompress(t, dt, eb, out=buf[first:first + x.size])
            assert y.cpu().numpy().tobytes() == want, (shape, first)
            assert torch.all(buf[:first] == 7.0) and torch.all(buf[first + x.size:] == 7.0)


def test_size_table_of_two_windows(cuda):
    n = (24576 + 100) * 4096 + 5  # the last chunks' places follow from the first window's sum
    x = torch.zeros(n, device="cuda")
    x[:: 4096 * 997] = 3.25
    x[-5:] = torch.arange(5, device="cuda") + 0.5
    s = api.compress(x)
    assert torch.equal(api.decompress(s, np.float32), x)


def test_batch_outputs_larger_than_their_streams(cuda):
    arrays = [_codes(dt, case, 20 + k)[: 1 + 40000 * k]
              for k, (dt, case) in enumerate((d, c) for c in CASES for d in (np.float32, np.float64))]
    ebs = [None if k % 3 else 0.5 for k in range(len(arrays))]
    streams = [O.encode(x, eb) for x, eb in zip(arrays, ebs)]
    room = [x.size + (50000 if k % 2 else 0) for k, x in enumerate(arrays)]
    plan = BatchPlan.decompress([torch.frombuffer(bytearray(s), dtype=torch.uint8).cuda() for s in streams],
                                [x.dtype for x in arrays], ebs, room)
    plan.run()
    for x, eb, s, y in zip(arrays, ebs, streams, plan.arrays()):
        assert y.cpu().numpy().tobytes() == O.decode(s, x.dtype, eb).tobytes()
