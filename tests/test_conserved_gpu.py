"""Conserved sums in one launch: exact integer sums of the cells' fixed-point
moments.  Sizes around the kernel's rounds of 256 cells, more cells than one
round of every CTA, both buffer states, and cells outside the fixed-point
range, against the oracle's sums of the lattice's own f."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# float64: the parity tests' tolerances.  Reduced precision: a cell's moments
# are float32 sums of 27 deviations, every partial sum below 0.05, so each is
# off by less than 27 * 2^-25 * 0.05 = 4e-8; its kinetic energy, with |u| below
# 0.05, by less than 3 * 0.05 * 4e-8 = 6e-9.
MOMENT, ENERGY = 4e-8, 6e-9


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 255), (4, 1, 64), (257, 1, 1), (3, 5, 7), (64, 65, 67)])
@pytest.mark.parametrize("prec", ["f64", "f32", "f16"])
def test_conserved_sizes(imex, oracle, shape, prec):
    p = {"f64": imex.IMEX_F64, "f32": imex.IMEX_F32, "f16": imex.IMEX_F16DEV}[prec]
    cells = float(np.prod(shape))
    with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=p) as lat:
        lat.initialize_phase(0.3, 1.1, 0.7)
        for steps in (0, 3):
            lat.step(steps)
            got = lat.Conserved()
            assert got == lat.Conserved()
            want = oracle.conserved(lat.get_f())
            err = np.abs(np.subtract(got, want))
            if prec == "f64":
                assert err[0] <= 1e-12 * want[0] and err[4] <= 1e-12 * want[4] and np.all(err[1:4] <= 1e-10)
            else:
                assert np.all(err[:4] <= MOMENT * cells) and err[4] <= ENERGY * cells


@pytest.mark.parametrize("value", [-0.02, 1.7, 1e-6])
def test_cells_outside_the_fixed_point_range(imex, oracle, value):
    f = oracle.init(24, 20, 33, 1.0, 0.05)
    f[5, ::7, 3, 32] = value
    f[0, 23, 19, 1] = 1.25
    with imex.LBM(24, 20, 33, 0.05, 1.0, 0.05) as lat:
        lat.set_f(f)
        got, want = lat.Conserved(), oracle.conserved(f)
        assert np.allclose(got, want, rtol=1e-12, atol=1e-10)
        f[7, 1, 2, 3] = np.nan
        lat.set_f(f)
        assert np.isnan(lat.Conserved(allow_nonfinite=True)[0])
