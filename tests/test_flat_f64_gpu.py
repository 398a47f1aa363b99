"""The float64 fixed-point run with cells in flat order (rows that leave
threads of a 128-cell segment idle) and with CTAs of whole-warp divisors of
nz, against single steps (row segments of 128), bit for bit: pairs of rows in
a warp, one cell, fewer cells than a CTA and one more than a CTA's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 3), (1, 1, 127), (1, 43, 3), (7, 6, 33), (5, 9, 131), (4, 3, 100), (3, 5, 32), (4, 4, 96), (2, 5, 160),
          (3, 2, 192), (2, 3, 256), (2, 3, 255), (96, 96, 130)]


@pytest.mark.parametrize("shape", SHAPES)
def test_run_equals_single_steps(imex, shape):
    outs = []
    for steps in ([1] * 9, [9]):
        with imex.LBM(*shape, 0.02, 1.0, 0.05, engine=imex.IMEX_ENGINE_FIXED) as lat:
            lat.set_launch(0, 1, 1)
            lat.initialize_phase(0.4, 1.2, 2.1)
            for n in steps:
                lat.step(n)
            assert lat.fallback_cells() == 0
            outs.append(lat.get_f())
    assert np.array_equal(*outs)


def test_a_failed_run_in_flat_order_is_redone(imex, oracle):
    """A cell leaving the exact range stops the run and single steps redo it."""
    shape = (20, 11, 45)
    f = oracle.init(*shape, 1.0, 0.05)
    f[19, 7, 3, 44] = 1e-3        # below 2^-9
    want = f.copy()
    oracle.step(want, 0.05, 12)
    with imex.LBM(*shape, 0.05, 1.0, 0.05, engine=imex.IMEX_ENGINE_FIXED) as lat:
        lat.set_launch(0, 1, 1)
        lat.set_f(f)
        lat.step(12)
        got = lat.get_f()
    assert np.max(np.abs(got - want)) <= 1e-12
