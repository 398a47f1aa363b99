"""Pressure and velocity from exact fixed-point moments: sizes around a CTA's
128 cells, every storage precision, both buffer states, and cells outside the
fixed-point range (there the float64 sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 2, 64), (1, 1, 129), (5, 7, 11)])
@pytest.mark.parametrize("prec", ["f64", "f32", "f16"])
def test_macroscopic_of_the_stored_values(imex, oracle, shape, prec):
    p = {"f64": imex.IMEX_F64, "f32": imex.IMEX_F32, "f16": imex.IMEX_F16DEV}[prec]
    rng = np.random.default_rng(2)
    with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=p) as lat:
        for kind in ("flow", "rough"):
            lat.initialize_phase(0.3, 1.1, 0.7)
            if kind == "rough":
                f = lat.get_f() * (1.0 + 0.05 * rng.standard_normal((27,) + shape))
                f.reshape(27, -1)[5, ::3] = -0.3
                f.reshape(27, -1)[7, 1::4] = 2.5
                lat.set_f(f)
            for pending in (False, True):
                if pending:
                    lat.Streaming()
                # 27 values below 4, summed in float64: 27 * 27 / 2 * 2^-53 * 4
                for got, want in zip(lat.ComputeMacroscopic(), oracle.macroscopic(lat.get_f())):
                    assert np.max(np.abs(got - want)) <= 2e-13


@pytest.mark.parametrize("pa,pb", [("f64", "f64"), ("f32", "f64"), ("f16", "f64"), ("f64", "f32"), ("f16", "f32"), ("f32", "f16"),
                                   ("f32", "f32"), ("f16", "f16"), ("f64", "f16")])
def test_velocity_difference(imex, pa, pb):
    prec = {"f64": imex.IMEX_F64, "f32": imex.IMEX_F32, "f16": imex.IMEX_F16DEV}
    shape = (13, 9, 47)
    rng = np.random.default_rng(4)
    with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=prec[pa]) as a, imex.LBM(*shape, 0.03, 1.0, 0.06, precision=prec[pb]) as b:
        a.initialize_phase(0.3, 1.1, 0.7)
        b.initialize_phase(0.4, 1.0, 0.2)
        for round_ in range(3):
            ua, ub = a.ComputeMacroscopic()[1:], b.ComputeMacroscopic()[1:]
            want = (max(np.max(np.abs(x - y)) for x, y in zip(ua, ub)), max(np.max(np.abs(y)) for y in ub))
            assert np.allclose(a.velocity_max_diff(b), want, rtol=0, atol=2e-13)
            if round_ == 0:
                a.step(2)            # a streaming is pending
            else:                    # a cell outside the fixed-point range carries the maximum
                f = b.get_f()
                f[1, 12, 8, 46] = 3.0
                b.set_f(f)
