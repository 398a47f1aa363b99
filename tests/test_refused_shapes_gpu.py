"""A refused launch shape changes nothing: the members of a batch go on in
the kernels that the rule, or the shape pinned before, puts them in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REFUSED = [("set_launch", (64, 0, 0)), ("set_launch", (96, 1, 4)), ("set_launch", (128, 3, 4)), ("set_launch", (256, 1, 9)),
           ("set_row_launch", (9, 2, 1)), ("set_row_launch", (2, 3, 1)), ("set_row_launch", (2, 2, 5)),
           ("set_row_launch", (8, 4, 4))]


def make(imex, prec, q):
    lat = imex.LBM(96, 96, 96, 0.004, 1.0, 0.05, precision=prec)
    lat.initialize_phase(0.1 * q, 0.2, 0.3)
    return lat


def refused(imex, b, call):
    name, args = call
    with pytest.raises(imex.ImexError) as e:
        getattr(b, name)(*args)
    assert e.value.code == imex.IMEX_ERR_ARG


@pytest.mark.parametrize("call", REFUSED)
def test_refused_on_an_unpinned_batch(imex, call):
    lats = [make(imex, imex.IMEX_F32, q) for q in range(3)] + [make(imex, imex.IMEX_F16DEV, 3)]
    with imex.Batch(4) as b:
        refused(imex, b, call)           # before the rule has chosen anything
        for lat in lats:
            b.add(lat)
        b.step(1)
        assert b.get_row_launch()[0] > 0     # the float16 member's rows are staged
        rows, cells = b.get_row_launch(), b.get_launch()
        refused(imex, b, call)           # and after
        assert (b.get_row_launch(), b.get_launch()) == (rows, cells)
        before = b.kernel_launches()
        b.step(8)
        b.synchronize()
        assert b.kernel_launches() - before == 8 + 4   # float16: a launch a step, float32: one per two steps
        assert (b.get_row_launch(), b.get_launch()) == (rows, cells)
    for lat in lats:
        lat.close()


@pytest.mark.parametrize("call", REFUSED)
def test_refused_on_a_pinned_batch(imex, call):
    with make(imex, imex.IMEX_F32, 0) as lat, imex.Batch(4) as b:
        b.set_launch(256, 2, 4)
        b.set_row_launch(2, 2, 1, False)
        b.add(lat)
        refused(imex, b, call)
        assert b.get_launch() == (256, 2, 4)
        assert tuple(b.get_row_launch())[:3] == (2, 2, 1)
        b.step(1)
        before = b.kernel_launches()
        b.step(8)
        b.synchronize()
        assert b.kernel_launches() - before == 8
