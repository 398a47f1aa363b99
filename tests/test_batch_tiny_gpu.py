"""Many tiny members in one segment kernel: a CTA finds its member among more
than the 32 that a warp looks at together, with sizes that share segments' group
entries or span several, members that stop early, and both formats."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(imex, q, f16):
    shape = [(3, 2, 5), (8, 8, 8), (1, 7, 40), (6, 5, 4), (16, 9, 8)][q % 5] if q != 70 else (40, 41, 43)
    lat = imex.LBM(*shape, 0.01 + 0.001 * (q % 7), 1.0, 0.05, precision=imex.IMEX_F16DEV if f16 and q % 3 == 0 else imex.IMEX_F32)
    lat.initialize_phase(0.1 * q, 0.2, 0.3 * q)
    return lat


@pytest.mark.parametrize("members", [2, 33, 34, 66, 140])
@pytest.mark.parametrize("f16", [False, True])
def test_tiny_members(imex, members, f16):
    lats = [make(imex, q, f16) for q in range(members)]
    with imex.Batch(160) as b:
        b.set_launch(128, 0, 0)
        b.set_row_launch(-1)
        for q, lat in enumerate(lats):
            b.add(lat, -1 if q % 4 else 3)
        b.step(2)
        b.step(4)
        b.synchronize()
        for q, lat in enumerate(lats):
            steps = 6 if q % 4 else 3
            with make(imex, q, f16) as alone:
                alone.set_launch(0, 1, 1)
                alone.step(steps)
                assert lat.steps_done() == steps
                assert np.array_equal(lat.get_f(), alone.get_f()), q
    for lat in lats:
        lat.close()


@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("graph", [0, 4])
def test_shape_by_cells(imex, f16, graph):
    """By rule a batch of fewer cells than a CTA a SM has threads takes the persistent kernel, a
    larger one the segment kernel: members join and leave across the line."""
    torch = pytest.importorskip("torch")
    line = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    n = line // 1000                      # of 10^3: just below the line

    def tenth(q):
        lat = imex.LBM(10, 10, 10, 0.01 + 0.001 * q, 1.0, 0.05,
                       precision=imex.IMEX_F16DEV if f16 and q % 2 else imex.IMEX_F32)
        lat.initialize_phase(0.1 * q, 0.2, 0.3 * q)
        return lat

    lats = [tenth(q) for q in range(n + 1)]
    with imex.Batch(n + 1) as b:
        b.set_graph(graph)
        for lat in lats[:n]:
            b.add(lat)
        b.step(9)
        assert b.get_launch() == (128, 1, 8)
        b.add(lats[n])
        b.step(9)
        assert b.get_launch() == (128, 0, 0)
        b.remove(lats[0])
        b.step(8)
        assert b.get_launch() == (128, 1, 8)
        b.synchronize()
        for q, lat in enumerate(lats):
            steps = 18 if q == 0 else 17 if q == n else 26
            with tenth(q) as alone:
                alone.set_launch(0, 1, 1)
                alone.step(steps)
                assert lat.steps_done() == steps
                assert np.array_equal(lat.get_f(), alone.get_f()), q
    for lat in lats:
        lat.close()
