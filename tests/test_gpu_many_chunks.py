"""The single-buffer kernels with several chunks per team of warps: tickets, a second
chunk staged beside the first, every launch shape by its number (one CTA per SM, so that
shape 0 is not replaced by the forms for small inputs) and the automatic choice; valid
streams of every width at every output offset, and malformed ones, whose damage lies in
chunks between well compressed neighbours."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sleek_b200 import _capi, api, autotune
from tests.test_gpu_encode_widths import CASES, _codes

pytestmark = pytest.mark.gpu

CORRUPT, CAPACITY = _capi.SLEEK_ERR_CORRUPT_STREAM, _capi.SLEEK_ERR_CAPACITY
CHUNKS = 1700  # more than the teams of any decode shape with one CTA on each of 148 SMs


@pytest.fixture
def shape_of():
    def choose(decompress, w, lossy, shape, ctas):
        _capi.check(_capi.lib().sleek_set_launch_shape(decompress, w, int(lossy), -1, shape, ctas))

    yield choose
    for dec in (0, 1):
        for w in (4, 8):
            for lossy in (0, 1):
                choose(dec, w, lossy, 0, 0)


def _choices(decompress):
    return [(0, 0)] + [(s["shape"], 1) for s in autotune.shapes(bool(decompress))]


def _tiled(dt, case, seed):
    x = _codes(dt, case, seed)
    n = CHUNKS * 16384 // x.itemsize - 3
    return np.tile(x, 1 + n // x.size)[:n]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("eb", [None, 0.5])
def test_every_shape_with_chunks_for_many_turns(cuda, shape_of, dt, case, eb):
    x = _tiled(dt, case, 31)
    stream = O.encode(x, eb)
    want = torch.from_numpy(O.decode(stream, dt, eb)).cuda()
    t = torch.from_numpy(np.frombuffer(stream, np.uint8).copy()).cuda()
    words = torch.int32 if x.itemsize == 4 else torch.int64
    buf = torch.empty(x.size + 8, dtype=want.dtype, device="cuda")
    for shape, ctas in _choices(1):
        shape_of(1, x.itemsize, eb is not None, shape, ctas)
        for first in range(16 // x.itemsize):
            buf.fill_(7.0)
            y = api.decompress(t, dt, eb, out=buf[first:first + x.size])
            assert torch.equal(y.view(words), want.view(words)), (shape, first)
            assert torch.all(buf[:first] == 7.0) and torch.all(buf[first + x.size:] == 7.0), (shape, first)
    src = torch.from_numpy(x).cuda()
    for shape, ctas in _choices(0):
        shape_of(0, x.itemsize, eb is not None, shape, ctas)
        assert torch.equal(api.compress(src, eb), t), shape


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("eb", [None, 1e-3])
@pytest.mark.parametrize("chunks", [1, 40, 301])
def test_every_encode_shape_on_few_chunks(cuda, shape_of, dt, eb, chunks):
    w = np.dtype(dt).itemsize
    x = (np.cumsum(np.random.default_rng(chunks).normal(0, 1, chunks * 16384 // w - 5)) * 0.3).astype(dt)
    want = O.encode(x, eb)
    t = torch.from_numpy(x).cuda()
    for shape, ctas in _choices(0):
        shape_of(0, w, eb is not None, shape, ctas)
        assert api.compress(t, eb).cpu().numpy().tobytes() == want, shape


def _damaged(s, rng, count):
    """Streams with damage to the sizes, widths, trailers or bits of some middle chunks, to
    the header, or cut short."""
    insize = int.from_bytes(s[:8], "little")
    chunks = (insize + 16383) // 16384
    sizes = np.frombuffer(s, np.uint16, chunks, 8).astype(np.int64)
    places = 8 + 2 * chunks + np.concatenate([[0], np.cumsum(sizes)])
    for k in range(count):
        b = bytearray(s)
        kind = k % 8
        for c in rng.integers(chunks // 4, chunks, int(rng.integers(1, 4))):
            c = int(c)
            if kind == 0:    # any size
                b[8 + 2 * c:10 + 2 * c] = int(rng.integers(0, 65536)).to_bytes(2, "little")
            elif kind == 1:  # sizes at the limits
                b[8 + 2 * c:10 + 2 * c] = int(rng.choice([0, 1, 33, 34, 35, 16383, 16384, 16385, 65535])).to_bytes(2, "little")
            elif kind == 2:  # two sizes exchanged: the sum stays
                o = 8 + 2 * c
                b[o - 2:o + 2] = b[o:o + 2] + b[o - 2:o]
            elif kind == 3:  # a width
                b[int(places[c]) + int(rng.integers(0, 32))] = int(rng.integers(0, 256))
            elif kind == 4:  # a trailer
                b[int(places[c + 1]) - int(rng.integers(1, 3))] ^= int(rng.integers(1, 256))
            elif kind == 5:  # packed bits: another valid stream
                b[int(rng.integers(places[c] + 32, places[c + 1] - 2))] ^= int(rng.integers(1, 256))
            elif kind == 6:  # the header
                b[int(rng.integers(0, 8))] = int(rng.integers(0, 256))
        if kind == 7:
            b = b[:int(rng.integers(8, len(b)))]
        yield bytes(b)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("eb", [None, 1e-3])
def test_malformed_streams_of_many_chunks(cuda, shape_of, dt, eb):
    rng = np.random.default_rng(41 if eb is None else 42)
    w = np.dtype(dt).itemsize
    n = CHUNKS * 16384 // w - 3
    x = (np.cumsum(rng.normal(0, 1, n)) * 0.3).astype(dt)
    if eb is not None:
        x = np.round(x)
    # three chunks of four hold codes of a few bits: small denormals, small multiples of eb
    small = np.arange(n) * w // 16384 % 4 != 0
    few = rng.integers(0, 16, int(small.sum()))
    x[small] = few.astype(f"u{w}").view(dt) if eb is None else few * dt(eb)
    s = O.encode(x, eb)
    assert len(s) < x.nbytes / 2
    tdt = torch.float32 if w == 4 else torch.float64
    guard = 64
    buf = torch.empty(n + 2 * guard + 4, dtype=tdt, device="cuda")
    size = torch.empty(1, dtype=torch.int64, device="cuda")
    info = (api.sleek_error_bound(eb, dt),) if eb is not None else ()
    seen = {"valid": 0, "corrupt": 0, "capacity": 0}
    for k, b in enumerate(_damaged(s, rng, 48)):
        v = api.validate_stream(b, dt)
        fits = v["valid"] and v["insize"] <= x.nbytes
        want = torch.from_numpy(O.decode(b, dt, eb)).cuda() if fits else None
        enc = torch.frombuffer(bytearray(b), dtype=torch.uint8).cuda()
        for shape, ctas in _choices(1):
            shape_of(1, w, eb is not None, shape, ctas)
            first = guard + k % (16 // w)
            buf.fill_(7.0)
            view = buf[first:first + n]
            api.sleek_decompress_gpu(0, *info, enc, view, size, encoded_bytes=len(b))
            got = int(size.item())
            assert torch.all(buf[:first] == 7.0) and torch.all(buf[first + n:] == 7.0), (k, shape)
            if fits:
                assert got == v["insize"], (k, shape, got, v)
                assert view[:got // w].cpu().numpy().tobytes() == want.cpu().numpy().tobytes(), (k, shape)
            elif v["valid"]:
                assert got == -CAPACITY, (k, shape, got, v)
            else:
                assert got in (-CORRUPT, -CAPACITY), (k, shape, got, v)
                if v["insize"] <= x.nbytes and v["reason"] != 1:
                    assert got == -CORRUPT, (k, shape, got, v)
        seen["valid" if fits else "capacity" if v["valid"] else "corrupt"] += 1
    assert seen["valid"] >= 4 and seen["corrupt"] >= 16, seen
    shape_of(1, w, eb is not None, 0, 0)
    y = api.decompress(torch.frombuffer(bytearray(s), dtype=torch.uint8).cuda(), dt, eb)
    assert y.cpu().numpy().tobytes() == O.decode(s, dt, eb).tobytes()
