"""The ring of group prefixes that the encoder's scanner keeps: an entry that is said to
be held has not been overwritten, at any step of the scanner, and one that is said to be
lost may have been.  The scanner writes the entries of up to 32 groups after the ones it
knows before it says so."""
from sleek_b200 import _capi

RING = 128
STEP = 32


def test_ring_entries_are_held_until_they_can_be_overwritten():
    holds = _capi.lib().sleek_selftest_ring_holds
    for known in list(range(0, 3 * RING)) + [10**6, 2**40 + 5]:
        for own in range(max(1, known - 2 * RING), known + 1):
            # groups after `own` that use its slot, among those written or being written
            lost = own + RING <= known + STEP
            assert bool(holds(known, own)) == (not lost), (known, own)
