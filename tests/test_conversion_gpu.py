"""float64 f <-> float16 deviations: the integer conversions give the bits of
the float64 expressions they stand for, for every float16 value, for f around
and between them, and off the integer path's range (negative, tiny, huge, NaN,
Inf)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def weights(oracle):
    w = np.array([8.0 / 27.0, 2.0 / 27.0, 1.0 / 54.0, 1.0 / 216.0])
    return w[np.abs(oracle.velocities()).sum(1)]


@pytest.mark.parametrize("shape", [(16, 64, 64), (1, 257, 255)])
def test_float16_conversions_bit_for_bit(imex, oracle, shape):
    cells = int(np.prod(shape))
    w = weights(oracle)[:, None]
    bits = np.resize(np.arange(65536, dtype=np.uint16), cells)
    rng = np.random.default_rng(11)
    with np.errstate(all="ignore"):
        exact = w + bits.view(np.float16).astype(np.float64)[None] / 4096.0
        around = exact * (1.0 + 2.0 ** -12 * rng.standard_normal(exact.shape))
        spread = w * 10.0 ** rng.uniform(-4, 4, exact.shape) * np.where(rng.random(exact.shape) < 0.1, -1, 1)
        for f in (exact, around, spread):
            want = w + ((f - w).astype(np.float32) * np.float32(4096)).astype(np.float16).astype(np.float64) / 4096.0
            with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=imex.IMEX_F16DEV) as lat:
                lat.set_f(f.reshape((27,) + shape))
                assert np.array_equal(lat.get_f().reshape(27, cells), want, equal_nan=True)
                lat.Streaming()  # read back through the pending pull: the same values, moved
                moved = oracle.stream(np.ascontiguousarray(want.reshape((27,) + shape)))
                assert np.array_equal(lat.get_f(), moved, equal_nan=True)


def test_float32_conversion_bit_for_bit(imex):
    """float64 to float32 by integer rounding: ties, carries into the exponent, both
    ends of its range and what lies beyond them."""
    rng = np.random.default_rng(12)
    k = np.arange(1, 8193, 2)
    parts = [rng.standard_normal(40000) * 10.0 ** rng.integers(-44, 38, 40000),
             np.ldexp(1 + k * 2.0 ** -24, 5), -np.ldexp(1 + k * 2.0 ** -24, -100), np.ldexp(1 + k * 2.0 ** -24 + 2.0 ** -52, 0),
             np.ldexp(2 - k * 2.0 ** -25, 3), np.ldexp(1 + k * 2.0 ** -24, -127), np.ldexp(2 - k * 2.0 ** -40, 126),
             np.ldexp(2 - k * 2.0 ** -40, 127), [0.0, -0.0, np.inf, -np.inf, np.nan, 2.0 ** -126, 2.0 ** 127, 1e300, -1e-300]]
    v = np.concatenate(parts)
    shape = (5, 37, 64)
    f = np.resize(v, 27 * int(np.prod(shape))).reshape((27,) + shape)
    with np.errstate(over="ignore"):
        want = f.astype(np.float32).astype(np.float64)
    with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=imex.IMEX_F32) as lat:
        lat.set_f(f)
        got = lat.get_f()
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(np.signbit(got[~np.isnan(want)]), np.signbit(want[~np.isnan(want)]))
