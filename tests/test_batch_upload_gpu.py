"""A batch whose upload of the two-step members' tables failed goes on with
the right ones: the tensor maps laid out for the failed call never reached the
GPU, so the next call may not take them for uploaded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (128, 128, 128)


def make(imex, q):
    lat = imex.LBM(*SHAPE, 0.004 * (1 + q), 1.0, 0.05, precision=imex.IMEX_F32)
    lat.initialize_phase(0.1 * q, 0.2 * q, 0.3 * q)
    return lat


def alone(imex, q, steps):
    with make(imex, q) as lat:
        lat.set_launch(0, 1, 1)
        lat.step(steps)
        return lat.get_f()


@pytest.mark.parametrize("order", [(1, 0, 2), (2, 1, 0), (2, 0)])
@pytest.mark.parametrize("graph", [0, 4])
def test_members_in_another_order_after_a_failed_upload(imex, order, graph):
    L = imex.load()
    lats = [make(imex, q) for q in range(3)]
    with imex.Batch(4) as b:
        b.set_graph(graph)
        for lat in lats:
            b.add(lat)
        b.step(1)
        before = b.kernel_launches()
        b.step(4)
        assert b.kernel_launches() - before == 2      # all of them two steps a launch
        for lat in lats:
            b.remove(lat)
        for q in order:
            b.add(lats[q])
        try:
            assert L.imex_test_set_fault(imex.IMEX_TEST_FAULT_BATCH_UPLOAD, 0) == 0
            with pytest.raises(imex.ImexError) as e:
                b.step(4)
            assert e.value.code == imex.IMEX_ERR_CUDA
        finally:
            L.imex_test_set_fault(0, 0)
        b.step(4)
        b.synchronize()
        for q, lat in enumerate(lats):
            done = 9 if q in order else 5
            assert lat.steps_done() == done
            assert np.array_equal(lat.get_f(), alone(imex, q, done))
    for lat in lats:
        lat.close()
