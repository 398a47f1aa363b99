"""A batch's float32 members two steps per launch: enough of them to fill the
GPU go to the two-step kernel, and every member still ends where it ends
alone one step at a time - with odd and even step limits, odd and even graph
lengths, members joining and leaving, and members of the other kernels beside
them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TAU, U0 = 0.004, 0.05
SHAPES = [(96, 96, 96), (64, 101, 96), (128, 61, 64), (40, 160, 100), (112, 112, 112), (33, 90, 132), (80, 80, 80)]


def make(imex, shape, prec, q):
    lat = imex.LBM(*shape, TAU * (1 + q), 1.0, U0, precision=prec)
    lat.initialize_phase(0.1 * q, 0.2 * q, 0.3 * q)
    return lat


def alone(imex, shape, prec, q, steps):
    with make(imex, shape, prec, q) as lat:
        if prec == imex.IMEX_F32:
            lat.set_launch(0, 1, 1)     # one step per launch
        lat.step(steps)
        return lat.get_f()


@pytest.mark.parametrize("graph", [0, 4, 5, 16])
def test_pairs_in_a_batch_equal_alone(imex, graph):
    lats = [make(imex, s, imex.IMEX_F32, q) for q, s in enumerate(SHAPES)]
    with imex.Batch(16) as b:
        b.set_graph(graph)
        for lat in lats:
            b.add(lat)
        b.step(1)
        before = b.kernel_launches()
        b.step(8)
        b.synchronize()
        # 8 = 4 pairs, or with a graph of 5 steps 2 pairs + 1 single + 1 pair + 1 single
        assert b.kernel_launches() - before == (5 if graph == 5 else 4)
        b.step(13)
        for q, (lat, s) in enumerate(zip(lats, SHAPES)):
            assert lat.steps_done() == 22
            assert np.array_equal(lat.get_f(), alone(imex, s, imex.IMEX_F32, q, 22))
    for lat in lats:
        lat.close()


def test_pairs_with_limits_leavers_and_other_kernels(imex):
    f32, f16 = imex.IMEX_F32, imex.IMEX_F16DEV
    specs = [(s, f32) for s in SHAPES] + [((64, 64, 64), f16), ((48, 50, 33), f32), ((40, 30, 35), f16)]
    limits = [7, 12, 20, -1, 3, 15, -1, 9, -1, 14]
    lats = [make(imex, s, p, q) for q, (s, p) in enumerate(specs)]
    with imex.Batch(16) as b:
        b.set_graph(6)
        for lat, lim in list(zip(lats, limits))[2:]:
            b.add(lat, lim)
        b.step(5)
        for lat, lim in list(zip(lats, limits))[:2]:
            b.add(lat, lim)
        b.step(9)
        b.remove(lats[3])
        b.step(10)
        b.synchronize()
        for q, (lat, (s, p), lim) in enumerate(zip(lats, specs, limits)):
            done = lat.steps_done()
            assert done == (lim if lim >= 0 else 14 if q == 3 else 24)
            assert np.array_equal(lat.get_f(), alone(imex, s, p, q, done))
    for lat in lats:
        lat.close()


def test_pinned_shapes_keep_one_step_per_launch(imex):
    lats = [make(imex, (96, 96, 96), imex.IMEX_F32, q) for q in range(4)]
    with imex.Batch(4) as b:
        b.set_launch(128, 0, 0)
        b.set_row_launch(-1)
        for lat in lats:
            b.add(lat)
        b.step(1)
        before = b.kernel_launches()
        b.step(8)
        assert b.kernel_launches() - before == 8
        assert np.array_equal(lats[2].get_f(), alone(imex, (96, 96, 96), imex.IMEX_F32, 2, 9))
    for lat in lats:
        lat.close()
