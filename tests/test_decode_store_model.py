"""CPU model of the decoder's stores into outputs that are not 16-byte aligned, and of a
stream's partial last chunk (unpack_unaligned and copy_raw in
sleek_b200/csrc/sleek_decode.cu): the kernel's index arithmetic, lane by lane, with the
chunk's own byte positions as the values.  Every byte of the chunk is written, with its
own value, nothing outside the chunk is written, and 16-byte stores are aligned."""
import pytest

CS, SC, G = 16384, 32, 4


class Out:
    def __init__(self, mis):
        self.mis, self.words = mis, {}

    def store16(self, at, v):
        assert (self.mis + at) % 16 == 0
        for k in range(4):
            self.word(at + 4 * k, v[k])

    def word(self, at, value):
        assert at not in self.words
        self.words[at] = value

    def value(self, at, width):
        for h in range(0, width, 4):
            assert self.words.get(at + h, at + h) == at + h  # (again with the same value, if at all)
            self.words[at + h] = at + h

    def check(self, osize):
        assert sorted(self.words) == list(range(0, osize, 4))
        assert all(a == v for a, v in self.words.items())


SIZES = [4, 8, 12, 16, 20, 24, 496, 504, 508, 512, 516, 2040, 2048, 2052, 2056, 9000, CS - 8, CS - 4, CS]


@pytest.mark.parametrize("width, mis", [(4, 0), (4, 4), (4, 8), (4, 12), (8, 0), (8, 8)])
def test_unpacked_chunks(width, mis):
    P, VPS = 16 // width, 512 // width
    m = mis // width
    for osize in SIZES:
        if osize % width:
            continue
        out = Out(mis)
        for i in range(SC):
            for lane in range(32):
                at = i * 512 + lane * 16 - mis
                first = lane * P - m  # the lane's values: those of the subchunk from here on
                mine = lane > 0 or mis == 0
                last = osize - 16 - lane * 16 + mis if mine else -1
                v = [i * 512 + first * width + 4 * k for k in range(4)]
                if i * 512 <= last:
                    assert 0 <= first and first + P <= VPS
                    out.store16(at, v)
        tail = (osize + mis) & 15
        if tail:
            i = (osize - width) // 512
            for lane in range(32):
                at = osize - tail + lane * width
                if i * 512 <= at < osize:
                    assert at < (i + 1) * 512
                    out.value(at, width)
        if mis:
            for i0 in range(0, SC, G):
                for lane in range(G * P):
                    u, t = lane // P, lane % P
                    k = t if t < P - m else VPS - P + t
                    at = (i0 + u) * 512 + k * width
                    if at < osize:
                        out.value(at, width)
        out.check(osize)


@pytest.mark.parametrize("width, mis", [(4, 0), (4, 4), (4, 8), (4, 12), (8, 0), (8, 8)])
@pytest.mark.parametrize("team", [1, 2, 8])
def test_raw_chunks(width, mis, team):
    for osize in SIZES:
        if osize % width:
            continue
        out = Out(mis)
        b = (16 - mis) & 15
        e = max(b, ((mis + osize) & ~15) - mis)
        for cw in range(team):
            for lane in range(32):
                for at in range(b + (cw * 32 + lane) * 16, e, team * 512):
                    assert at + 16 <= osize  # the staged bytes that are read
                    out.store16(at, [at + 4 * k for k in range(4)])
                if cw == 0:
                    at = 4 * lane if lane < 4 else e + 4 * (lane - 4)
                    if (at < min(b, osize)) if lane < 4 else (at < osize and lane < 8):
                        out.word(at, at)
        out.check(osize)
