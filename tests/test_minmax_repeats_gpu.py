"""Extremes of lattices whose cells repeat (a fluid at rest, blocks of equal cells
among others, whole planes) or lie outside the fixed-point range everywhere: a cell
with the values of the one summed before is not summed again, and the extremes are
those of the float64 sums of every cell, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def want(oracle, lat):
    p, u, v, w = oracle.macroscopic(lat.get_f())
    a = (u, v, w, p)
    return tuple(float(np.max(x)) for x in a) + tuple(float(np.min(x)) for x in a)


@pytest.mark.parametrize("prec", ["f64", "f32", "f16"])
@pytest.mark.parametrize("rho0", [1.0, 0.05, 12.0])
@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 5, 3), (20, 33, 31), (48, 40, 65)])
def test_repeating_cells(imex, oracle, prec, rho0, shape):
    p = {"f64": imex.IMEX_F64, "f32": imex.IMEX_F32, "f16": imex.IMEX_F16DEV}[prec]
    rng = np.random.default_rng(6)
    cells = int(np.prod(shape))
    with imex.LBM(*shape, 0.05, rho0, 0.0, precision=p) as lat:
        lat.Initialize()
        rest = lat.get_f()
        for kind in ("rest", "one", "few", "blocks", "rough"):
            f = rest.copy()
            g = f.reshape(27, cells)
            if kind == "one":
                g[rng.integers(27), rng.integers(cells)] *= 1.0 + 2.0 ** -9
            elif kind == "few":
                at = rng.integers(cells, size=max(1, cells // 100))
                g[:, at] *= 1.0 + 0.01 * rng.standard_normal((27, 1))
            elif kind == "blocks":
                g *= np.repeat(1.0 + 0.01 * rng.standard_normal((27, cells // 9 + 1)), 9, axis=1)[:, :cells]
            elif kind == "rough":
                g *= 1.0 + 0.02 * rng.standard_normal(g.shape)
                g[:, ::3] *= 2.5
            lat.set_f(f)
            for pending in (False, True):
                if pending:
                    lat.Streaming()
                assert lat.minmax_uvwp() == want(oracle, lat), (kind, pending)
