"""The extremes of u, v, w, p found with integers equal those of the float64
sums bit for bit: sizes around a chunk's 256 to 2048 cells, flows, fields
constant in a component (every cell a candidate) and values outside the
fixed-point range, NaN and infinities among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _extremes(oracle, f):
    """oracle.minmax_uvwp of the sums that skip a zero velocity (the oracle's own
    product with it makes NaN of an infinity)."""
    m = np.zeros((4,) + f.shape[1:])
    with np.errstate(invalid="ignore"):
        for a, e in enumerate(oracle.velocities()):
            m[3] += f[a]
            for d in range(3):
                if e[d] == 1:
                    m[d] += f[a]
                elif e[d] == -1:
                    m[d] -= f[a]
        m[3] *= 1.0 / 3.0
        big = np.finfo(np.float64).max
        hi = np.where(m > -big, m, -big).reshape(4, -1).max(1)
        lo = np.where(m < big, m, big).reshape(4, -1).min(1)
    return np.concatenate([hi, lo])


def _fields(lat, shape, rng):
    lat.initialize_phase(0.3, 1.1, 0.7)
    yield "flow", lat.get_f()
    lat.Initialize()
    yield "w constant", lat.get_f()
    f = lat.get_f()
    f[:] = f.reshape(27, -1)[:, :1].reshape(27, 1, 1, 1)
    yield "constant", f.copy()
    flat = f.reshape(27, -1)
    flat *= 1.0 + 1e-15 * rng.standard_normal(flat.shape)  # apart by the last bits
    yield "nearly constant", f.copy()
    flat[:, ::7] *= 1.0 + 0.05 * rng.standard_normal(flat[:, ::7].shape)
    flat[5, ::311] = -0.3
    flat[7, 1::401] = 2.5
    yield "outside", f.copy()
    flat[3, 2::503] = np.nan
    flat[9, -1] = np.inf
    flat[11, 0] = -np.inf
    yield "not finite", f.copy()
    flat[:] = np.nan
    yield "no number", f


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 255), (1, 2, 128), (257, 1, 1), (9, 9, 127), (61, 83, 129),
                                   (128, 200, 112)])
@pytest.mark.parametrize("prec", ["f64", "f32", "f16"])
def test_extremes_of_the_float64_sums(imex, oracle, shape, prec):
    p = {"f64": imex.IMEX_F64, "f32": imex.IMEX_F32, "f16": imex.IMEX_F16DEV}[prec]
    with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=p) as lat:
        for kind, f in list(_fields(lat, shape, np.random.default_rng(3))):
            lat.set_f(f)
            got = [lat.minmax_uvwp()]
            if shape[0] < 128:
                lat.Streaming()      # read through the pending streaming
                got.append(lat.minmax_uvwp())
            want = _extremes(oracle, lat.get_f())
            assert np.array_equal(np.array(got[-1]), want), (kind, got, want)
            if kind in ("flow", "w constant"):
                assert np.array_equal(want, oracle.minmax_uvwp(lat.get_f()))
