"""Two float32 steps per launch: the results are those of single steps, bit
for bit, whatever the sizes do to the tiles (10 x 32 destinations at most):
rows and columns that just fit, one more, a single y tile, tiles one row
short, narrow last tiles, many and few x chunks, odd step counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(96, 96, 96), (700, 10, 128), (400, 19, 128), (650, 9, 160), (40, 160, 128), (90, 125, 124), (200, 59, 100),
          (33, 150, 256), (140, 88, 116), (260, 88, 60)]


def run(imex, shape, steps, pinned, restart=None):
    with imex.LBM(*shape, 0.003, 1.0, 0.06, precision=imex.IMEX_F32) as lat:
        if pinned:
            lat.set_launch(0, 1, 1)   # one step per launch
        lat.initialize_phase(0.3, 1.1, 2.0)
        if restart is not None:
            lat.set_f(restart)
        before = lat.kernel_launches()
        lat.step(steps)
        launches = lat.kernel_launches() - before
        return lat.get_f(), launches


@pytest.mark.parametrize("shape", SHAPES)
def test_pairs_equal_single_steps(imex, shape):
    want, _ = run(imex, shape, 9, True)
    got, launches = run(imex, shape, 9, False)
    assert launches == 1 + 4          # the collision in place, then two steps a launch
    assert np.array_equal(got, want)


def test_pairs_with_rough_state_and_odd_steps(imex):
    """Values far from equilibrium, so that every direction carries its own
    pattern; an odd number of steps left takes a single step at the end."""
    shape = (77, 100, 124)
    rng = np.random.default_rng(3)
    with imex.LBM(*shape, 0.1, 1.0, 0.05, precision=imex.IMEX_F32) as lat:
        lat.Initialize()
        f = lat.get_f() * (1.0 + 0.02 * rng.standard_normal((27,) + shape))
    for steps in (8, 11):
        want, _ = run(imex, shape, steps, True, f)
        got, _ = run(imex, shape, steps, False, f)
        assert np.array_equal(got, want)


def test_pairs_through_a_stream_and_single_calls(imex):
    """Collision / Streaming calls, short and long runs mixed."""
    shape = (96, 96, 96)
    outs = []
    for pinned in (True, False):
        with imex.LBM(*shape, 0.003, 1.0, 0.06, precision=imex.IMEX_F32) as lat:
            if pinned:
                lat.set_launch(0, 1, 1)
            lat.Initialize()
            for n in (1, 2, 4, 5):
                lat.step(n)
                lat.Collision()
                lat.Streaming()
            lat.step(7)
            assert lat.steps_done() == 23
            outs.append(lat.get_f())
    assert np.array_equal(*outs)


def test_starved_plane_is_reported_and_the_handle_recovers(imex):
    L = imex.load()
    shape = (96, 96, 96)
    want, _ = run(imex, shape, 9, True)
    with imex.LBM(*shape, 0.003, 1.0, 0.06, precision=imex.IMEX_F32) as lat:
        lat.initialize_phase(0.3, 1.1, 2.0)
        lat.step(3)
        try:
            assert L.imex_test_set_fault(imex.IMEX_TEST_FAULT_STARVE_STAGE, 200000) == 0
            lat.step(4)
            with pytest.raises(imex.ImexError) as e:
                lat.Conserved()
            assert e.value.code == imex.IMEX_ERR_CUDA
        finally:
            L.imex_test_set_fault(0, 0)
        lat.initialize_phase(0.3, 1.1, 2.0)
        lat.step(9)
        assert np.array_equal(lat.get_f(), want)


@pytest.mark.parametrize("steps", [4, 6])
def test_captured_run_replays(imex, steps):
    """A graph of an even number of steps, replayed, goes on from its own result."""
    torch = pytest.importorskip("torch")
    shape = (96, 96, 96)
    outs = []
    for captured in (False, True):
        with imex.LBM(*shape, 0.003, 1.0, 0.06, precision=imex.IMEX_F32) as lat:
            lat.initialize_phase(0.3, 1.1, 2.0)
            lat.step(1)
            if captured:
                stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
                lat.set_stream(stream.cuda_stream)
                with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
                    lat.step(steps)
                graph.replay()
                graph.replay()
                torch.cuda.synchronize()
            else:
                lat.step(2 * steps)
            outs.append(lat.get_f())
            lat.set_stream(None)
    assert np.array_equal(*outs)


@pytest.mark.parametrize("shape", [(121, 150, 98), (121, 150, 97), (90, 125, 131), (400, 19, 126), (650, 9, 157), (40, 160, 127),
                                   (200, 59, 101), (33, 150, 255), (260, 88, 62), (140, 88, 99)])
def test_rows_of_any_length(imex, shape):
    """Rows that are no multiple of 4 values go through the padded layout: last
    tiles of 1, 2, 3, 5, 29, 30 and 31 columns, odd and even, every number of
    steps left after the pairs, and a state far from equilibrium."""
    rng = np.random.default_rng(5)
    with imex.LBM(*shape, 0.1, 1.0, 0.05, precision=imex.IMEX_F32) as lat:
        lat.initialize_phase(0.3, 1.1, 2.0)
        f = lat.get_f() * (1.0 + 0.02 * rng.standard_normal((27,) + shape))
    for steps, launches in ((9, 1 + 2 + 3), (4, 1 + 3), (5, 1 + 2 + 1), (6, 1 + 2 + 1 + 1)):
        want, _ = run(imex, shape, steps, True, f)
        got, n = run(imex, shape, steps, False, f)
        assert n == launches
        assert np.array_equal(got, want)


def test_padded_room_is_counted(imex):
    """The larger buffers of a lattice with odd rows are at most 7 values a row more."""
    shape = (96, 128, 129)
    with imex.LBM(*shape, 0.05, 1.0, 0.05, precision=imex.IMEX_F32) as lat, \
            imex.LBM(96, 128, 128, 0.05, 1.0, 0.05, precision=imex.IMEX_F32) as even:
        per_value = lat.device_bytes() / (2 * 27 * 4 * 96 * 128)
        assert 129 < per_value < 129 + 8
        assert 128 <= even.device_bytes() / (2 * 27 * 4 * 96 * 128) < 129
