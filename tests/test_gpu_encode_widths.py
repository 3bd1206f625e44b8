"""The encoder's packing and placing at the widths, alignments and chunk mixes where
its paths change: every code width (whole and joined runs), chunks stored raw among
compressed ones (places at other alignments than expected), inputs at every element
offset, and more than two groups of 64 chunks, alone (one warp per chunk, and the
several warps per chunk of small inputs) and in a batch."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sleek_b200 import _capi, api
from sleek_b200.batch import compress_batch

pytestmark = pytest.mark.gpu


def _codes(dt, case, seed):
    """Values whose codes (bound 0.5: step 1) have chosen widths, chunk by chunk."""
    rng = np.random.default_rng(seed)
    vpc = 16384 // np.dtype(dt).itemsize
    top = 24 if dt == np.float32 else 53
    if case == "each width":  # one chunk per width
        parts = [rng.integers(0, 1 << w, vpc) for w in range(0, top)]
    elif case == "mixed widths":  # every subchunk its own width
        parts = [rng.integers(0, 1 << int(w), vpc // 32) for w in rng.integers(0, top, 32 * 40)]
    elif case == "around a word":  # runs of 14 to 34 bits side by side
        lo, hi = (3, 10) if dt == np.float32 else (7, 18)
        parts = [rng.integers(0, 1 << int(w), vpc // 32) for w in rng.integers(lo, hi, 32 * 40)]
    else:  # "raw among packed": noise chunks, which do not shrink, between small ones
        parts = []
        for k in range(150):
            if k % 7 in (2, 3) or k == 64:
                bits = rng.integers(0, 256, 16384, dtype=np.uint8).view(dt)
                parts.append(np.where(np.isfinite(bits), bits, dt(1)))
            else:
                parts.append(rng.integers(0, 1 << (k % 12 + 1), vpc))
    x = np.concatenate([np.asarray(p, dtype=dt) for p in parts])
    return x * rng.choice(np.array([-1, 1], dtype=dt), x.size)


CASES = ["each width", "mixed widths", "around a word", "raw among packed"]


@pytest.fixture
def default_shapes():
    yield
    for w in (4, 8):
        for lossy in (0, 1):
            _capi.check(_capi.lib().sleek_set_launch_shape(0, w, lossy, -1, 0, 0))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("eb", [None, 0.5])
def test_widths_and_places(cuda, default_shapes, dt, case, eb):
    x = _codes(dt, case, 5)[:-3]
    want = O.encode(x, eb)
    for ctas in (0, 1):  # by the number of chunks; one warp per chunk for any number
        _capi.check(_capi.lib().sleek_set_launch_shape(0, x.itemsize, int(eb is not None), -1, 0, ctas))
        for first in range(16 // x.itemsize):
            t = torch.from_numpy(np.concatenate([np.zeros(first, dt), x])).cuda()[first:]
            assert api.compress(t, eb).cpu().numpy().tobytes() == want, (ctas, first)


@pytest.mark.parametrize("chunks", [1, 2, 591, 592, 593])
def test_sizes_around_the_small_inputs(cuda, chunks):
    x = np.resize(_codes(np.float32, "mixed widths", 7), chunks * 4096 - 1)
    assert api.compress(torch.from_numpy(x).cuda(), 0.5).cpu().numpy().tobytes() == O.encode(x, 0.5)


def test_batch_places_over_groups(cuda):
    arrays, ebs = [], []
    rng = np.random.default_rng(6)
    for k, chunks in enumerate([1, 63, 64, 65, 3, 130, 1, 200, 5]):
        dt = np.float32 if k % 2 else np.float64
        x = _codes(dt, CASES[k % 4], k)
        x = np.tile(x, 1 + chunks * 16384 // x.nbytes)[: chunks * 16384 // x.itemsize - int(rng.integers(0, 9))]
        arrays.append(x)
        ebs.append(None if k % 3 == 0 else 0.5)
    got = compress_batch([torch.from_numpy(x).cuda() for x in arrays], ebs)
    for x, eb, s in zip(arrays, ebs, got):
        assert s.cpu().numpy().tobytes() == O.encode(x, eb)
