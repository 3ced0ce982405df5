"""The autotuner installs another launch shape than the library's own only when it is clearly faster: for calls whose
kernel ignores the shape, all candidates take the same time but for noise."""
import numpy as np
import pytest

from codag_b200 import tuning


def _search(native, monkeypatch, codec, seconds):
    stored = []
    monkeypatch.setattr(tuning, "store_cached", lambda codec, tag, shape: stored.append(tuple(shape)))
    shapes = iter(tuning.candidates(codec))
    monkeypatch.setattr(tuning, "time_call", lambda run: seconds(next(shapes)))
    old = native.get_tune(codec)
    try:
        best, _ = tuning.autotune(codec, lambda: None, use_cache=False)
        t = native.get_tune(codec)
    finally:
        native.set_tune(codec, old.warps_per_cta, old.ring_slots, old.lut_bits, old.cta_per_chunk)
    assert stored == [best] and best == (t.warps_per_cta, t.ring_slots, t.lut_bits, t.cta_per_chunk)
    return best


@pytest.mark.parametrize("codec", [0, 1, 2])
def test_noise_changes_nothing(native, monkeypatch, codec):
    for seed in range(20):
        rng = np.random.default_rng(seed)
        assert _search(native, monkeypatch, codec, lambda shape: 1e-4 * rng.uniform(0.985, 1.015)) == tuning.DEFAULT[codec]


def test_a_clear_winner_is_installed(native, monkeypatch):
    assert _search(native, monkeypatch, 1, lambda shape: 8e-5 if shape == (2, 8, 10, 0) else 1e-4) == (2, 8, 10, 0)


def test_default_is_the_library_s(native):
    for codec, shape in tuning.DEFAULT.items():
        t = native.get_tune(codec)
        assert shape == (t.warps_per_cta, t.ring_slots, t.lut_bits, t.cta_per_chunk)
        assert shape in tuning.candidates(codec)
