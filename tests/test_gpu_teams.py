"""Fits by a team of CTAs (a thread-block cluster per fit, used when few fits are
left) against fits by one CTA each: the same bits, at the sizes where the
dealing can go wrong -- fewer points than CTAs, partial tiles, curve counts
around the warps, both forms of the normal-matrix update, residuals in shared
memory and in the slab, facet counts that are no multiple of 4.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # points per curve, curves, lmax, nrows, facets dropped, calibrated points
    (5, 1, 3, 4, 0, 0),
    (33, 2, 3, 5, 1, 0),
    (60, 20, 3, 6, 0, 0),
    (40, 33, 6, 6, 3, 50),
    (47, 9, 7, 5, 0, 20),
    (45, 17, 8, 6, 2, 0),
    (100, 60, 3, 5, 0, 0),
    (70, 60, 8, 5, 0, 30),
]


def _object(pts, curves, lmax, nrows, drop, sparse):
    import oracle
    from ps_claude_opt_b200 import objects, synth

    cfg = synth.SynthConfig(l_max=lmax, m_max=lmax, nrows=nrows, n_dense=curves, dense_pts=(pts, pts), n_sparse=sparse,
                            sparse_curves=1, n_freq=20, truth_grid=(30, 60))
    obj = objects.parse_input(synth.generate(cfg, 31)[0], setup_fn=oracle.setup_shape)
    n = obj.n_fac - drop
    return dataclasses.replace(obj, n_fac=n, normal=obj.normal[:3 * n], d_area=obj.d_area[:n],
                               dsph=obj.dsph[:n * obj.n_coef])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", CASES)
def test_team_fits_equal_single_cta_fits(case, precision):
    from ps_claude_opt_b200 import native

    if precision and case[2] > 7:
        pytest.skip("mixed precision is built for n_coef <= 64")
    obj = _object(*case)
    with native.Engine(obj) as eng:
        eng.set_precision(precision)
        eng.configure(stop_condition=6.0)
        per_sm, n_sm = eng.occupancy()
        wave = per_sm * n_sm  # whole waves run one CTA per fit
        nf = 1 + np.arange(wave) // 10
        pl = np.arange(wave) % 10
        ref, it, st = eng.fit_items(nf, pl)
        for n in (10, 30, 70):  # teams of 8, 4 and 2
            g, gi, gs = eng.fit_items(nf[:n], pl[:n])
            assert np.array_equal(g, ref[:n], equal_nan=True)
            assert np.array_equal(gi, it[:n]) and np.array_equal(gs, st[:n])
        # whole wave and teams side by side
        g, gi, _ = eng.fit_items(np.concatenate([nf, nf[:13]]), np.concatenate([pl, pl[:13]]))
        assert np.array_equal(g, np.concatenate([ref, ref[:13]]), equal_nan=True)
        assert np.array_equal(gi, np.concatenate([it, it[:13]]))
