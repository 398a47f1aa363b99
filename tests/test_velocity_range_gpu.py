"""Velocities of strongly diverged reduced-precision lattices: a component of
18 values just below 1/8 reaches 2.2 either way, so that the difference of two
lattices is above 4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def directions(imex, prec):
    """Velocity of each direction along x, read off a lattice: u of f = 1/16 in that direction alone."""
    with imex.LBM(1, 1, 27, 0.05, 1.0, 0.05, precision=prec) as lat:
        f = np.zeros((27, 1, 1, 27))
        for a in range(27):
            f[a, 0, 0, a] = 0.0625
        lat.set_f(f)
        u = lat.ComputeMacroscopic()[1]
        out = np.sign(np.round(np.asarray(u).reshape(27) * 16)).astype(int)
    assert sorted(out) == [-1] * 9 + [0] * 9 + [1] * 9
    return out


def weights(imex, prec):
    """f of a fluid at rest."""
    with imex.LBM(1, 1, 1, 0.05, 1.0, 0.0, precision=prec) as lat:
        lat.Initialize()
        return lat.get_f().reshape(27)


@pytest.mark.parametrize("pa", ["f32", "f16"])
@pytest.mark.parametrize("pb", ["f32", "f16"])
@pytest.mark.parametrize("value", [0.11, 0.112, 0.124])
def test_difference_of_opposite_extremes(imex, pa, pb, value):
    prec = {"f32": imex.IMEX_F32, "f16": imex.IMEX_F16DEV}
    shape = (3, 5, 37)
    lats = []
    for p, sign in ((prec[pa], 1), (prec[pb], -1)):
        e = directions(imex, p)
        lat = imex.LBM(*shape, 0.05, 1.0, 0.05, precision=p)
        lat.initialize_phase(0.3, 1.1, 0.7)
        f = lat.get_f()
        # what is stored is the value itself, or its deviation from the weight
        f[:, 2, 4, 36] = (0.0 if p == imex.IMEX_F32 else weights(imex, p)) + sign * value * e
        lat.set_f(f)
        lats.append(lat)
    a, b = lats
    for x, y in ((a, b), (b, a), (a, a)):
        ux, uy = x.ComputeMacroscopic()[1:], y.ComputeMacroscopic()[1:]
        want = (max(np.max(np.abs(s - t)) for s, t in zip(ux, uy)), max(np.max(np.abs(t)) for t in uy))
        # two roundings of sums below 8 each, and of their difference
        assert np.allclose(x.velocity_max_diff(y), want, rtol=0, atol=2e-13)
    assert a.velocity_max_diff(b)[0] > (4.4 if value == 0.124 else 3.9)
    for lat in lats:
        lat.close()
