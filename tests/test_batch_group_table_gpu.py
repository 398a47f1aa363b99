"""The segment kernel's member lookup table moves when a tick needs a larger
one, and a graph captured before holds its old address: it may not be launched
again even if the shapes, the members and the segment count are the ones it was
captured with."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 16 segments for the segment kernel while the float16 members are in the row
# kernel (one table entry, room for two); 848 with it switched off (four entries)
SPECS = [((16, 16, 16), "f32", 0.004), ((64, 64, 16), "f16", 0.02), ((96, 96, 16), "f16", 0.01)]


def make(imex, spec):
    shape, prec, tau = spec
    lat = imex.LBM(*shape, tau, 1.0, 0.05, precision=imex.IMEX_F32 if prec == "f32" else imex.IMEX_F16DEV)
    lat.initialize_phase(0.3, 1.1, 2.0)
    return lat


def test_graph_of_a_table_that_moved(imex):
    lats = [make(imex, s) for s in SPECS]
    with imex.Batch(4) as b:
        b.set_graph(4)
        b.set_row_launch(2, 2, 2, False)
        for lat in lats:
            b.add(lat)
        b.step(9)                    # the first collisions, then two ticks: captured
        before = b.kernel_launches()
        b.step(4)
        assert b.kernel_launches() - before == 4 * 2     # segment and row kernel
        b.set_row_launch(-1)
        b.step(3)                    # all in the segment kernel, no graph: the table moves
        assert b.kernel_launches() - before == 4 * 2 + 3
        b.set_row_launch(2, 2, 2, False)
        b.step(8)                    # the shapes and segments of the graph again
        b.synchronize()
        for lat, spec in zip(lats, SPECS):
            with make(imex, spec) as alone:
                alone.step(24)
                assert lat.steps_done() == 24
                assert np.array_equal(lat.get_f(), alone.get_f())
    for lat in lats:
        lat.close()
