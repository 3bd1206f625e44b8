"""Host side of the Python API, no GPU needed."""
import numpy as np
import pytest

from sleek_b200 import api


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_the_callers_struct_of_a_bound_is_its_own(dtype):
    info = api.sleek_error_bound(1e-3, dtype)
    mine = info.c_struct()
    mine.eb_e, mine.thr_e, mine.offs_e = 0, 0, 0
    for again in (info.c_struct(), api.sleek_error_bound(1e-3, dtype).c_struct()):
        assert (again.eb_e, again.thr_e, again.offs_e) == (info.eb_e, info.thr_e, info.offs_e)
        assert type(again) is type(mine)
