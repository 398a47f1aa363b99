"""Conserved sums of reduced-precision lattices whose density puts every cell
outside the range of the ordinary integers, or some cells, or some beyond the wider
range too; and such a lattice's sums take no multiple of the time of one of
density 1."""
import math
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact(imex, lat, f):
    """Sums of the stored values: mass and momentum exact, the energy of exact velocities."""
    e = directions(imex)
    out = [math.fsum(f.ravel())]
    u = [np.tensordot(e[:, d].astype(np.longdouble), f.astype(np.longdouble), axes=(0, 0)) for d in range(3)]
    return out + [math.fsum(x.astype(np.float64).ravel()) for x in u] + [0.5 * float(sum((x * x).sum() for x in u))]


_dirs = []


def directions(imex):
    """(27, 3) velocities, read off a lattice: u of f = 1/16 in one direction a cell."""
    if not _dirs:
        with imex.LBM(1, 1, 27, 0.05, 1.0, 0.05) as lat:
            f = np.zeros((27, 1, 1, 27))
            f[np.arange(27), 0, 0, np.arange(27)] = 0.0625
            lat.set_f(f)
            _dirs.append(np.stack([np.round(np.asarray(c).reshape(27) * 16) for c in lat.ComputeMacroscopic()[1:]], axis=1))
    return _dirs[0]


@pytest.mark.parametrize("prec,rho0", [("f32", 2.5), ("f32", 1000.0), ("f32", 6000.0), ("f32", 1e5), ("f16", 2.5), ("f16", 30.0)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 7), (40, 41, 43)])
def test_density(imex, prec, rho0, shape):
    p = imex.IMEX_F32 if prec == "f32" else imex.IMEX_F16DEV
    with imex.LBM(*shape, 0.05, rho0, 0.05, precision=p) as lat:
        lat.initialize_phase(0.3, 1.1, 0.7)
        for pending in (False, True):
            if pending:
                lat.Streaming()
            got, f = lat.Conserved(), lat.get_f()
            want = exact(imex, lat, f)
            scale = abs(f).sum()
            # float64: 27 values a cell and the sums' own rounding; get_f's float16 values are rounded once each
            assert np.all(np.abs(np.subtract(got, want))[:4] <= 64 * 2.0 ** -53 * scale)
            assert abs(got[4] - want[4]) <= 64 * 2.0 ** -53 * max(want[4], float((abs(f).sum(axis=0) ** 2).sum()))


@pytest.mark.parametrize("prec", ["f32", "f16"])
def test_ranges_mixed_in_a_lattice(imex, prec):
    p = imex.IMEX_F32 if prec == "f32" else imex.IMEX_F16DEV
    shape = (24, 20, 33)
    rng = np.random.default_rng(8)
    with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=p) as lat:
        lat.initialize_phase(0.3, 1.1, 0.7)
        f = lat.get_f()
        g = f.reshape(27, -1)
        g[:, ::5] *= 9.0                                   # the wider range
        g[:, 1::7] *= rng.uniform(-1.5, 1.5, g[:, 1::7].shape)   # float16 deviations end at 16
        if prec == "f32":
            g[4, 2::9] = 1e-12                             # no multiple of its unit
            g[6, 3::11] = 3e5                              # and beyond it
        lat.set_f(f)
        got, f = lat.Conserved(), lat.get_f()
        want = exact(imex, lat, f)
        # cells in the ordinary range sum their deviations in float32, each partial sum below 2
        slack = 27 * 2.0 ** -24 * 2 * np.prod(shape)
        scale = 64 * 2.0 ** -53 * abs(f).sum()
        assert np.all(np.abs(np.subtract(got, want))[:4] <= slack + scale)
        assert abs(got[4] - want[4]) <= 3 * slack + 64 * 2.0 ** -53 * float((abs(f).sum(axis=0) ** 2).sum())
        g = f.reshape(27, -1)
        g[3, 17] = np.nan
        lat.set_f(f)
        assert np.isnan(lat.Conserved(allow_nonfinite=True)[0])


@pytest.mark.parametrize("prec,rho0", [("f32", 1000.0), ("f16", 3.0)])
@pytest.mark.parametrize("edge", [32, 192])
def test_no_multiple_of_the_time(imex, prec, rho0, edge):
    p = imex.IMEX_F32 if prec == "f32" else imex.IMEX_F16DEV

    def best(rho):
        with imex.LBM(edge, edge, edge, 0.05, rho, 0.05, precision=p) as lat:
            lat.Initialize()
            times = []
            for _ in range(20):
                t0 = time.perf_counter()
                lat.Conserved()
                times.append(time.perf_counter() - t0)
            return min(times)

    # the cells are read twice and summed in the integers twice; in float64 it was 5 to 11 times as long
    assert best(rho0) < 3.5 * best(1.0)
