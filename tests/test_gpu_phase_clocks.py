"""The phase clocks count the full evaluations of every fit, whether one CTA or a
team of 8, 4 or 2 runs it: at least one and at most one per iteration, and as
many in whole waves of a fit as waves times that fit alone."""
import numpy as np
import pytest

from conftest import prepared

pytestmark = pytest.mark.gpu


def _evals(eng, nf, pl):
    eng.phase_clocks()
    _, it, _ = eng.fit_items(nf, pl)
    return eng.phase_clocks(), it


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["tiny", "mixed", "lmax8"])
def test_evaluations_are_counted_alike(kind, precision):
    from ps_claude_opt_b200 import native

    if precision and kind == "lmax8":
        pytest.skip("mixed precision is built for n_coef <= 64")
    obj = prepared(kind)
    with native.Engine(obj) as eng:
        eng.set_precision(precision)
        eng.configure(stop_condition=6.0)
        per_sm, n_sm = eng.occupancy()
        wave = per_sm * n_sm
        one = np.ones(1, dtype=np.int32)
        clocks, it = _evals(eng, one, 3 * one)
        evals = clocks["evals"]
        assert 1 <= evals <= it[0] and clocks["sweep"] > 0 and clocks["trial"] > 0
        for n in (10, 30, 70, wave, wave + 13):
            clocks, _ = _evals(eng, np.ones(n, dtype=np.int32), np.full(n, 3, dtype=np.int32))
            assert clocks["evals"] == n * evals
