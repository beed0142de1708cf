"""Objects whose shared-memory layout ends within a few hundred bytes of what one
block may have: evaluations (a team of CTAs), a few fits (teams), a whole wave
with a few more (both kernels) and the allocation-free entry point, against
the oracle and one another.

Tolerances are those of the same checks at other sizes: FP64 evaluations
relative 1e-9, three-iteration fits relative 1e-7 in rms, period and chi^2 and
1e-6 degree; mixed precision 1e-4 (normwise, relative) and 1e-3 degree; one
kernel against another without tolerance.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMEM_LIMIT = 232448  # sm_100
CASES = [
    # lmax, rows, relative curves, calibrated points, precision
    (6, 8, 159, 0, 0),
    (6, 9, 146, 6, 0),
    (7, 8, 48, 0, 0),
    (7, 8, 45, 6, 0),
    (8, 11, 127, 6, 0),
    (6, 8, 101, 0, 1),
    (7, 8, 58, 0, 1),
    (7, 8, 5, 6, 1),
]


def _object(lmax, rows, curves, sparse):
    import oracle
    from ps_claude_opt_b200 import objects, synth

    cfg = synth.SynthConfig(l_max=lmax, m_max=lmax, nrows=rows, n_dense=curves,
                            dense_pts=(12, 20) if curves >= 100 else (60, 80), n_sparse=sparse, sparse_curves=1,
                            n_freq=20, truth_grid=(30, 60))
    return objects.parse_input(synth.generate(cfg, 31)[0], setup_fn=oracle.setup_shape)


def _smem(obj, mixed):
    """Shared memory of the layout that is chosen for the object."""
    from ps_claude_opt_b200 import native

    need = getattr(native.lib(), "_ZN3psb14fit_smem_bytesEiiiiiiii")
    need.restype = C.c_size_t
    nc = obj.n_coef
    sizes = [need(obj.n_fac, obj.mfit, (nc + 7) // 8 * 8, obj.n_curves, (nc + 10) & ~1, rows, cstat, mixed)
             for rows, cstat in ((32, 1), (32, 0), (16, 0))]
    return next(s for s in sizes if s <= SMEM_LIMIT)


@pytest.mark.parametrize("lmax,rows,curves,sparse,precision", CASES)
def test_layouts_at_the_limit(lmax, rows, curves, sparse, precision):
    import oracle
    from ps_claude_opt_b200 import native, objects

    obj = _object(lmax, rows, curves, sparse)
    assert SMEM_LIMIT - 768 < _smem(obj, precision) <= SMEM_LIMIT
    om = oracle.OracleModel(obj)
    rel_eval, rel_fit, deg = (1e-9, 1e-7, 1e-6) if precision == 0 else (1e-4, 1e-4, 1e-3)
    nf, pl = np.repeat([1], 10), np.arange(10)
    with native.Engine(obj) as eng:
        eng.set_precision(precision)
        eng.configure(stop_condition=3.0)
        a = objects.initial_params(obj, 2, 3)
        chi, alpha, beta, _ = eng.eval(a)
        chi_o, alpha_o, beta_o, _, _ = om.eval(a)
        assert abs(chi - chi_o) <= rel_eval * abs(chi_o)
        for g, o in ((alpha, alpha_o), (beta, beta_o)):
            assert np.abs(g - o).max() <= rel_eval * np.abs(o).max()
        g, gi, gs = eng.fit_items(nf, pl)
        om.m.n_iter_max = 3
        o, oi, _ = om.fit_batch(obj.grid.freq_start, obj.grid.freq_step, nf, pl)
        assert np.array_equal(gi, oi)
        for col in (0, 2, 5):
            assert np.allclose(g[:, col], o[:, col], rtol=rel_fit, atol=0)
        assert np.allclose(g[:, 3:5], o[:, 3:5], rtol=0, atol=deg)
        per_sm, n_sm = eng.occupancy()
        reps = (per_sm * n_sm + 9) // 10 + 1  # a wave of single CTAs, then teams
        w, wi, ws = eng.fit_items(np.tile(nf, reps), np.tile(pl, reps))
        assert np.array_equal(w, np.tile(g, (reps, 1)), equal_nan=True)
        assert np.array_equal(wi, np.tile(gi, reps)) and np.array_equal(ws, np.tile(gs, reps))
    if precision == 0:
        import dataclasses

        n, ni, ns = native.fit_items_noalloc(dataclasses.replace(obj, stop_condition=3.0), nf, pl)
        assert np.array_equal(n, g, equal_nan=True) and np.array_equal(ni, gi) and np.array_equal(ns, gs)
