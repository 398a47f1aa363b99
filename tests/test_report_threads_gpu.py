"""Runs and sums read back through the shared page of pinned memory: many
threads at once, more than it has slots, each with a lattice of its own; and
a float64 run that leaves the fixed-point range, between others that do not."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _deck(imex, k, prec, out):
    with imex.LBM(8 + k % 5, 9, 12, 0.02, 1.0, 0.02 + 0.001 * (k % 40), precision=prec) as lat:
        lat.initialize_phase(0.1 * k, 1.1, 0.7)
        rows = []
        for _ in range(6):
            lat.step(5)
            rows.append(lat.Conserved())
        out[k] = (rows, lat.get_f())


@pytest.mark.parametrize("prec", ["f64", "f16"])
def test_many_threads(imex, prec):
    p = {"f64": imex.IMEX_F64, "f16": imex.IMEX_F16DEV}[prec]
    want, got = {}, {}
    for k in range(96):
        _deck(imex, k, p, want)
    threads = [threading.Thread(target=_deck, args=(imex, k, p, got)) for k in range(96)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(96):
        assert got[k][0] == want[k][0]
        assert np.array_equal(got[k][1], want[k][1])


def test_runs_around_a_failing_one(imex, oracle):
    """A cell outside the exact range stops a run; the runs before and after it
    are those of single steps."""
    shape, outs = (12, 10, 16), []
    for single in (False, True):
        with imex.LBM(*shape, 0.05, 1.0, 0.05) as lat:
            lat.Initialize()
            start = lat.get_f()
            res = []
            for bad in (False, True, False):
                f = start.copy()
                if bad:
                    f[1, 5, 5, 5] = 0.6   # above 1/8: the native path takes the cell
                lat.set_f(f)
                for _ in range(3):
                    if single:
                        for _ in range(4):
                            lat.step(1)
                    else:
                        lat.step(4)
                res.append((lat.get_f(), lat.Conserved()))
            outs.append(res)
    for a, b in zip(*outs):
        assert np.array_equal(a[0], b[0])
        assert a[1] == b[1]
