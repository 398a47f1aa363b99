"""A captured run reads the buffer that held the state when it was captured,
so whatever an even number of eager steps does in between must leave the state
in that buffer: float32 lattices that go two steps per launch, alone and in a
batch, in the plain and the padded layout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TAU, U0 = 0.003, 0.06


def make(imex, shape):
    lat = imex.LBM(*shape, TAU, 1.0, U0, precision=imex.IMEX_F32)
    lat.initialize_phase(0.3, 1.1, 2.0)
    return lat


def single_steps(imex, shape, n):
    with make(imex, shape) as lat:
        lat.set_launch(0, 1, 1)
        lat.step(n)
        return lat.get_f()


def captured(lat, steps, way):
    """The graph's replay, on the stream the lattice now works on."""
    torch = pytest.importorskip("torch")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    lat.fence()
    lat.set_stream(stream.cuda_stream)
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        if way == "step":
            lat.step(steps)
        else:
            for _ in range(steps):
                lat.Collision()
                lat.Streaming()

    def replay():
        with torch.cuda.stream(stream):
            graph.replay()
    return replay


@pytest.mark.parametrize("shape", [(96, 96, 96), (121, 150, 97)])
@pytest.mark.parametrize("eager", [4, 6, 8, 10, 14])
@pytest.mark.parametrize("way", ["step", "calls"])
def test_eager_steps_between_replays(imex, shape, eager, way):
    with make(imex, shape) as lat:
        lat.step(9)                     # pairs: rows of 97 values get their larger buffers here
        replay = captured(lat, 4, way)
        replay()
        lat.step(eager)
        replay()
        got = lat.get_f()
        lat.set_stream(None)
    assert np.array_equal(got, single_steps(imex, shape, 9 + 4 + eager + 4))


@pytest.mark.parametrize("eager", [6, 8])
def test_batch_steps_between_replays(imex, eager):
    shape = (128, 128, 128)
    with make(imex, shape) as lat, make(imex, shape) as other, imex.Batch(2) as b:
        lat.step(1)
        other.step(1)
        replay = captured(lat, 4, "step")
        replay()
        b.add(lat)
        b.add(other)
        b.step(eager)
        b.synchronize()
        b.remove(lat)
        replay()
        got = lat.get_f()
        lat.set_stream(None)
        assert np.array_equal(other.get_f(), single_steps(imex, shape, 1 + eager))
    assert np.array_equal(got, single_steps(imex, shape, 1 + 4 + eager + 4))


@pytest.mark.parametrize("shape", [(96, 96, 96), (121, 150, 97)])
def test_eager_steps_still_pair_once_captured(imex, shape):
    """Steps of a captured lattice go two per launch where that keeps the buffer."""
    with make(imex, shape) as lat:
        lat.step(9)
        captured(lat, 4, "step")
        before = lat.kernel_launches()
        lat.step(22)
        assert lat.kernel_launches() - before < 22
        got = lat.get_f()
        lat.set_stream(None)
        assert np.array_equal(got, single_steps(imex, shape, 31))
