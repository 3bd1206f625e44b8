"""sleek_set_ctas_per_sm limits the CTAs per SM of whatever form a call has: the forms for
small inputs stay in use where they keep within the limit."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sleek_b200 import _capi, api
from tests.test_gpu_capacities import _launched

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit():
    L = _capi.lib()

    def set_limit(decompress, ctas):
        _capi.check(L.sleek_set_ctas_per_sm(decompress, 4, 0, ctas))

    yield set_limit
    for dec in (0, 1):
        set_limit(dec, 0)
        _capi.check(L.sleek_set_launch_shape(dec, 4, 0, -1, 0, 0))


def test_small_forms_within_the_limit(cuda, limit):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = np.cumsum(np.random.default_rng(1).normal(0, 1, 5 * sms * 4096)).astype(np.float32)
    t = torch.from_numpy(x).cuda()
    out = torch.empty(api.sleek_upper_bound_size(x.nbytes), dtype=torch.uint8, device="cuda")
    y = torch.empty_like(t)
    size = torch.zeros(1, dtype=torch.int64, device="cuda")
    L = _capi.lib()
    ws = torch.empty(max(L.sleek_compress_workspace_size(x.nbytes), L.sleek_decompress_workspace_size()),
                     dtype=torch.uint8, device="cuda")

    def compress(chunks):
        api.sleek_compress_gpu(0, t[:chunks * 4096], chunks * 4096, out, size, workspace=ws)

    def decompress(chunks, s):
        api.sleek_decompress_gpu(0, s, y[:chunks * 4096], size, encoded_bytes=s.numel(), workspace=ws)

    small = _launched(lambda: compress(2))[1]
    large = _launched(lambda: compress(5 * sms))[1]
    assert small != large
    for ctas in (1, 2, 3, 4, 9):
        limit(0, ctas)
        for chunks in (1, 40, min(ctas, 4) * sms):  # one CTA per chunk
            assert _launched(lambda: compress(chunks)) == (chunks, small), (ctas, chunks)
        assert _launched(lambda: compress(min(ctas, 4) * sms + 1))[1] == large, ctas
        for chunks in (1, 40, 2 * sms):
            assert api.compress(t[:chunks * 4096]).cpu().numpy().tobytes() == O.encode(x[:chunks * 4096]), (ctas, chunks)
    s = api.compress(t[:40 * 4096])
    few = _launched(lambda: decompress(40, s))
    limit(1, 1)
    assert _launched(lambda: decompress(40, s)) == few
    # a shape asked for by its number is that shape, for any number of chunks
    _capi.check(L.sleek_set_launch_shape(0, 4, 0, -1, 0, 1))
    assert _launched(lambda: compress(2))[1] == large
