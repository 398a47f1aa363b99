"""The fused step over flat cell pairs, against the row-staged and the
collide-then-stream forms of the same step: odd and even cell counts, pairs
across row and plane ends, one cell, fewer cells than a CTA and one more than
a CTA's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 1, 2), (3, 1, 1), (1, 1, 256), (1, 1, 257), (5, 7, 9), (2, 3, 43), (16, 5, 33), (4, 6, 31), (9, 8, 64)]


def run(imex, shape, prec, sr, single):
    with imex.LBM(*shape, 0.02, 1.0, 0.05, precision=prec) as lat:
        if prec == imex.IMEX_F16DEV:
            lat.set_rounding(imex.IMEX_ROUND_STOCHASTIC if sr else imex.IMEX_ROUND_NEAREST)
        lat.initialize_phase(0.2, 0.9, 1.7)
        for _ in range(5):
            if single:              # streaming alone, then a collision in place: one-cell kernels
                lat.Collision()
                lat.Streaming()
                lat.set_f(lat.get_f())
            else:
                lat.step(1)
        return lat.get_f()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec", ["f32", "f16 nearest", "f16 stochastic"])
def test_flat_pairs_equal_one_cell_kernels(imex, shape, prec):
    p = imex.IMEX_F32 if prec == "f32" else imex.IMEX_F16DEV
    sr = prec == "f16 stochastic"
    assert np.array_equal(run(imex, shape, p, sr, False), run(imex, shape, p, sr, True))


@pytest.mark.parametrize("shape", [(6, 5, 33), (12, 10, 17)])
def test_flat_pairs_in_a_batch(imex, shape):
    """Odd rows in a batch beside even ones, each as it ends alone."""
    specs = [(shape, imex.IMEX_F16DEV), (shape, imex.IMEX_F32), ((8, 9, 10), imex.IMEX_F16DEV), ((3, 3, 3), imex.IMEX_F32)]
    lats = []
    for s, p in specs:
        lats.append(imex.LBM(*s, 0.02, 1.0, 0.05, precision=p))
        lats[-1].initialize_phase(0.2, 0.9, 1.7)
    with imex.Batch(8) as b:
        b.set_launch(128, 0, 0)
        b.set_row_launch(-1)
        for lat in lats:
            b.add(lat)
        b.step(7)
        for lat, (s, p) in zip(lats, specs):
            with imex.LBM(*s, 0.02, 1.0, 0.05, precision=p) as one:
                one.initialize_phase(0.2, 0.9, 1.7)
                one.step(7)
                assert np.array_equal(lat.get_f(), one.get_f())
    for lat in lats:
        lat.close()
