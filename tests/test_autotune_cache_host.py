"""The autotuner's cache file: a choice is found again by the library that it was made
with, and never by one whose table of launch shapes is another."""
import json

import pytest

from sleek_b200 import autotune


@pytest.fixture
def cache(tmp_path, monkeypatch):
    path = tmp_path / "tuning.json"
    monkeypatch.setenv("SLEEK_TUNING_CACHE", str(path))
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda: "a GPU")
    monkeypatch.setattr(autotune, "_time", lambda fn, reps=5: fn() or timed.append(1) or float(len(timed)))
    timed = []
    return path


@pytest.mark.parametrize("decompress", [False, True])
def test_choices_of_another_shape_table_are_not_used(cache, monkeypatch, decompress):
    # a file without the table in its keys, as written for another library: ignored
    old = f"a GPU|single|{'dec' if decompress else 'enc'}|4|0|2^22"
    cache.write_text(json.dumps({old: [0, 2]}))
    key = autotune.single_key(decompress, 4, False, 22)
    cands = autotune.single_candidates(decompress)
    r = autotune.tune(key, lambda c: None, cands)
    assert not r["cached"] and r["best"] == cands[0]
    r = autotune.tune(autotune.single_key(decompress, 4, False, 22), lambda c: None, cands)
    assert r["cached"] and r["best"] == cands[0]  # the same library finds its own choice
    # one more warp in the last shape: another library, another key
    table = autotune.shapes(decompress)
    table[-1]["warps"] += 1
    monkeypatch.setattr(autotune, "shapes", lambda dec: table)
    assert not autotune.tune(autotune.single_key(decompress, 4, False, 22), lambda c: None, cands)["cached"]


def test_keys_tell_the_kinds_apart():
    keys = {autotune.single_key(d, w, l, b) for d in (False, True) for w in (4, 8) for l in (False, True) for b in (3, 22)}
    assert len(keys) == 16
