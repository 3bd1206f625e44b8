"""What a device wait that gives up leads to, one wait at a time (sleek_selftest_wait):
nothing ever satisfies the wait, its limit is short, and the device stays usable."""
import ctypes as C

import pytest

from sleek_b200 import _capi

pytestmark = pytest.mark.gpu

LIMIT = 20_000_000  # ns


def run(what):
    res = (C.c_longlong * 3)(-9, -9, -9)
    _capi.check(_capi.lib().sleek_selftest_wait(what, LIMIT, res))
    return list(res)


@pytest.mark.parametrize("warp", [0, 1])
def test_every_warp_of_a_team_reports_its_own_timeout(cuda, warp):
    status, pos, ns = run(warp)
    assert (status, pos) == (_capi.SLEEK_ERR_TIMEOUT, 7)
    assert ns >= LIMIT


def test_a_warp_waits_once_more_for_its_copy_before_it_leaves(cuda):
    landed, _, ns = run(2)
    assert landed == 0
    assert ns >= 2 * LIMIT


@pytest.mark.parametrize("what, gives_up_with", [(3, -1), (4, -1), (5, 0)])
def test_waits_for_a_chunks_place_give_up(cuda, what, gives_up_with):
    got, _, ns = run(what)
    assert got == gives_up_with
    assert LIMIT <= ns < LIMIT + 2_000_000_000
