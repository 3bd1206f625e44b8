"""A stream's header may state any 64-bit size: its chunks are counted without overflow,
and a size table that the stream has no room for is refused."""
import numpy as np
import pytest

from sleek_b200 import api


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("insize", [2**63 - 8, 2**63 - 16384, 2**63 - 16376, 2**62, 2**52])
def test_validator_refuses_sizes_the_stream_cannot_hold(dtype, insize):
    v = api.validate_stream(insize.to_bytes(8, "little") + bytes(64), dtype)
    assert not v["valid"] and v["insize"] == insize
    assert v["chunks"] == (insize + 16383) // 16384
    assert v["reason"] == 3, v  # size table past the end
