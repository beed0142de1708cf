"""The feature kernel at the sizes where it can go wrong, against the CPU
restatement (oracle/screen_ref.py) with that test's bar (1e-4 absolute; the
features are ratios and shares of order one, computed in 64 bits and rounded
to FP32): one curve on both sides of the middle of the time span, curves of
one to three points, 256 curves, a curve too long or too bright for 32-bit
limbs, curve counts around the warps, a single frequency.
"""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(lens, seed, span=2000.0, spread=0.3, amplitude=0.2):
    rng = np.random.default_rng(seed)
    tim, br = [], []
    for n in lens:
        t = rng.uniform(0, span) + np.sort(rng.uniform(0, spread, n))
        tim.append(t)
        br.append(1.0 + amplitude * np.sin(t * 23.0) + 0.02 * rng.standard_normal(n))
    return np.concatenate(tim), np.concatenate(br), np.asarray(lens, dtype=np.int32)


CASES = {
    "straddling": dict(lens=[300, 40, 55], spread=1500.0),
    "one curve": dict(lens=[90], spread=800.0),
    "tiny curves": dict(lens=[1, 2, 3, 1, 3, 2, 1]),
    "many curves": dict(lens=[3 + i % 5 for i in range(256)]),
    "seven": dict(lens=[31, 32, 33, 64, 65, 1, 96]),
    "eight": dict(lens=[31, 32, 33, 64, 65, 1, 96, 50]),
    "nine": dict(lens=[31, 32, 33, 64, 65, 1, 96, 50, 20]),
    "long": dict(lens=[5000, 60], spread=900.0),
    "bright": dict(lens=[70, 80], amplitude=0.9, scale=True),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("n_freq", [1, 37])
def test_features_at_the_edges(name, n_freq):
    from oracle import screen_ref
    from ps_claude_opt_b200 import screen

    kw = dict(CASES[name])
    scale = kw.pop("scale", False)
    tim, br, lens = _data(kw.pop("lens"), 5, **kw)
    if scale:  # a curve whose mean is near zero: relative brightness of several hundred
        br[:70] = br[:70] - br[:70].mean() + 0.001
    freqs = np.linspace(0.02, 0.4, n_freq)
    obj = types.SimpleNamespace(tim=tim, brightness=br, curve_len=lens, curve_rel=np.ones(len(lens), dtype=np.int32))
    got = screen.features(obj, freqs)
    ref = screen_ref.features(tim, br, lens, 24.0 * freqs)
    assert got.shape == ref.shape == (n_freq, 88)
    assert np.all(np.isfinite(got)) and np.max(np.abs(got - ref)) < 1e-4
    assert np.array_equal(screen.features(obj, freqs), got)
