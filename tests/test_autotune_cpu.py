"""Remembered tuning choices whose knob values have changed their meaning."""
import pytest

import compression_b200.autotune as at


@pytest.mark.parametrize("codec,entry,applies", [
    ("deflate", {"value": 12}, False),                  # before revisions were noted: a warp pair
    ("deflate", {"value": 4, "revision": 1}, False),
    ("deflate", {"value": 4, "revision": 2}, True),
    ("rlev1", {"value": 4}, True),                      # unchanged since
])
def test_apply(codec, entry, applies):
    t = at.Tuner.__new__(at.Tuner)
    t.name, t.results = "B200", {}
    t.results[t.key(codec, 1 << 20)] = entry
    knob = at.KNOBS[codec][0]
    prev = at.set_knob(knob, 0)
    try:
        assert t.apply(codec, 1 << 20) == applies
        assert at.get_knob(knob) == (entry["value"] if applies else 0)
    finally:
        at.set_knob(knob, prev)
