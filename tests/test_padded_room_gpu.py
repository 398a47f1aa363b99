"""Buffers large enough for the padded layout of odd rows: what lattices hold of
it without using it is bounded, and one created without it gets it at its first
run of its own - unless a graph of its steps reads the buffers it has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (1000, 200, 121)
ROWS = 1000 * 200
PLAIN, PADDED = (2 * 27 * 4 * ROWS * n for n in (121, 128))
MOST = 1 << 30                                  # unused, in the process


def make(imex):
    lat = imex.LBM(*SHAPE, 0.01, 1.0, 0.05, precision=imex.IMEX_F32)
    lat.initialize_phase(0.3, 1.1, 2.0)
    return lat


def room(lat):
    """Of a lattice's bytes; its scratch for the reports is below a value a cell."""
    extra = lat.device_bytes() - PLAIN
    has = extra >= PADDED - PLAIN
    assert 0 <= extra - has * (PADDED - PLAIN) < 4 * ROWS * 121 / 8
    return has


@pytest.fixture
def crowd(imex):
    """One lattice more than may have unused room."""
    n = MOST // (PADDED - PLAIN)
    lats = [make(imex) for _ in range(n + 1)]
    assert [room(lat) for lat in lats] == [True] * n + [False]
    yield lats
    for lat in lats:
        lat.close()


def same_as_single_steps(imex, lat, n):
    with make(imex) as want:
        want.set_launch(0, 1, 1)
        want.step(n)
        assert lat.velocity_max_diff(want)[0] == 0.0
        assert lat.Conserved() == want.Conserved()


def test_room_at_the_first_run(imex, crowd):
    lat = crowd[-1]
    with imex.Batch(2) as b:
        b.add(lat)
        b.step(3)
        b.synchronize()
        b.remove(lat)
    lat.Collision()
    lat.Streaming()
    lat.step(2)
    lat.set_launch(0, 1, 1)
    lat.step(6)
    assert not room(lat)
    lat.set_launch(-1)
    before = lat.kernel_launches()
    lat.step(10)
    assert lat.kernel_launches() - before == 1 + 4 + 1
    assert room(lat)
    same_as_single_steps(imex, lat, 22)
    lat.step(7)
    same_as_single_steps(imex, lat, 29)


def test_used_or_closed_room_counts_no_more(imex, crowd):
    crowd[0].step(9)                            # used now
    with make(imex) as lat:
        assert room(lat)
        crowd[1].close()
        with make(imex) as other:
            assert room(other)
            with make(imex) as third:
                assert not room(third)
    crowd[1] = make(imex)
    assert room(crowd[1])


def test_no_room_once_captured(imex, crowd):
    torch = pytest.importorskip("torch")
    lat = crowd[-1]
    lat.step(1)
    lat.fence()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    lat.set_stream(stream.cuda_stream)
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        lat.step(4)
    for _ in range(2):
        with torch.cuda.stream(stream):
            graph.replay()
        lat.step(6)
    assert not room(lat)
    lat.fence()
    lat.set_stream(None)
    same_as_single_steps(imex, lat, 1 + 2 * 10)
