"""Inputs and outputs on both sides of the sizes at which they go through the graph's page-locked memory, written and read
in every order a caller may use."""
import numpy as np
import pytest

import pyb2vx as B

pytestmark = pytest.mark.gpu


def relu(lib, dims):
    g = B.Graph(lib, 0)
    x = g.tensor(B.DT_UINT8, dims, B.ATTR_INPUT, scale=0.1, zero_point=10)
    y = g.tensor(B.DT_UINT8, dims, B.ATTR_OUTPUT, scale=0.1, zero_point=10)
    g.relu(x, y)
    g.compile()
    return g, x, y


# [W, H, C, N]: layouts that coincide and that do not; rows without pixels; tiny, small and large
SHAPES = [(1, 1, 5, 1), (1, 1, 16, 3), (1, 1, 1000, 7), (1, 1, 1001, 64), (1, 1, 1008, 64), (3, 3, 10, 2), (56, 56, 3, 1), (64, 64, 64, 1), (65, 64, 64, 1),
          (1, 1, 1000, 262), (1, 1, 1000, 263)]


@pytest.mark.parametrize("dims", SHAPES)
def test_round_trip(product_lib, dims):
    rng = np.random.default_rng(3)
    g, x, y = relu(product_lib, list(dims))
    a, b = (rng.integers(0, 256, size=dims[::-1]).astype(np.uint8) for _ in range(2))
    want = lambda v: np.maximum(v, 10)
    g.write(x, a)
    g.run()
    np.testing.assert_array_equal(g.read(y), want(a))
    np.testing.assert_array_equal(g.read(x), a)
    g.write(x, b)
    np.testing.assert_array_equal(g.read(y), want(a))   # not run yet
    g.run_async()
    g.write(x, a)                                       # waits for the run that reads b
    np.testing.assert_array_equal(g.read(y), want(b))
    g.run_async()
    np.testing.assert_array_equal(g.read(y), want(a))
    g.profile(2)
    np.testing.assert_array_equal(g.read(y), want(a))
    g.close()


# 10 bytes in one row, 48 bytes whose layouts coincide, 180 bytes that a kernel writes over the bus, 5 KB, and 300 KB (not staged)
@pytest.mark.parametrize("dims", [(1, 1, 10, 1), (1, 1, 16, 3), (3, 3, 10, 2), (8, 8, 80, 1), (64, 64, 74, 1)])
def test_written_output_is_read_back(product_lib, dims):
    rng = np.random.default_rng(4)
    a, b, c = (rng.integers(0, 256, size=dims[::-1]).astype(np.uint8) for _ in range(3))
    want = np.maximum(a, 10)
    g = B.Graph(product_lib, 0)
    x = g.tensor(B.DT_UINT8, list(dims), B.ATTR_INPUT, scale=0.1, zero_point=10)
    y = g.tensor(B.DT_UINT8, list(dims), B.ATTR_OUTPUT, scale=0.1, zero_point=10)
    g.relu(x, y)
    g.write(y, b)
    g.compile()
    np.testing.assert_array_equal(g.read(y), b)     # written before the graph was compiled
    g.write(x, a)
    g.run()
    np.testing.assert_array_equal(g.read(y), want)
    g.write(y, c)
    np.testing.assert_array_equal(g.read(y), c)     # and after a run
    g.run_async()
    g.write(y, b)                                   # waits for the run
    np.testing.assert_array_equal(g.read(y), b)
    g.run()
    np.testing.assert_array_equal(g.read(y), want)
    g.close()


# staged in one piece, by rows, over the bus, and not staged
@pytest.mark.parametrize("dims", [(8, 8, 80, 1), (1, 1, 1000, 7), (3, 3, 10, 2), (64, 64, 74, 1)])
def test_run_recorded_on_a_stream_of_the_caller(product_lib, dims):
    """The caller records the first run_async into a CUDA graph of its own and launches that without this library's
    knowing: what is written before a launch goes into it, and a read waits for it."""
    import torch
    rng = np.random.default_rng(5)
    data = [rng.integers(0, 256, size=dims[::-1]).astype(np.uint8) for _ in range(4)]
    g, x, y = relu(product_lib, list(dims))
    st = torch.cuda.Stream()
    g.set_stream(st.cuda_stream)
    recorded = torch.cuda.CUDAGraph()
    with torch.cuda.graph(recorded, stream=st, capture_error_mode="thread_local"):
        g.run_async()
    for a in data:
        g.write(x, a)
        with torch.cuda.stream(st):
            torch.cuda._sleep(20_000_000)   # about 10 ms: the launch behind it is still queued when the read begins
            recorded.replay()
        np.testing.assert_array_equal(g.read(y), np.maximum(a, 10))
    with torch.cuda.stream(st):
        torch.cuda._sleep(20_000_000)
        recorded.replay()
    g.write(x, data[0])                     # waits for that launch, which still reads the last one's bytes
    np.testing.assert_array_equal(g.read(y), np.maximum(data[-1], 10))
    torch.cuda.synchronize()
    recorded.reset()
    g.close()


def add(lib, n):
    """Two inputs of n elements each, one output: rows of one pixel where n is a multiple of 16, else 3 x 3 pixels."""
    dims = [1, 1, n, 1] if n % 16 == 0 else [3, 3, n // 9, 1]
    g = B.Graph(lib, 0)
    a, b = (g.tensor(B.DT_UINT8, dims, B.ATTR_INPUT, scale=0.1, zero_point=0) for _ in range(2))
    y = g.tensor(B.DT_UINT8, dims, B.ATTR_OUTPUT, scale=0.1, zero_point=0)
    g.add(a, b, y)
    return g, a, b, y, dims[::-1]


@pytest.mark.parametrize("n", [16, 90, 9009, 65536])
def test_one_of_two_inputs_changes(product_lib, n):
    """Runs that wait and runs that do not, in turn, with one input or none written in between."""
    rng = np.random.default_rng(6)
    g, a, b, y, shape = add(product_lib, n)
    g.compile()
    v = [np.zeros(shape, np.uint8), np.zeros(shape, np.uint8)]
    for step in range(24):
        which = (None, 0, None, 1, 0, 1)[step % 6]
        if which is not None:
            v[which] = rng.integers(0, 128, size=shape).astype(np.uint8)
            g.write((a, b)[which], v[which])
        if step % 5 < 2:
            g.run()
        elif step % 5 == 2:
            g.profile(1)
        else:
            for _ in range(step % 3 + 1):
                g.run_async()
        if step % 4:
            np.testing.assert_array_equal(g.read(y), v[0] + v[1])
    g.close()


@pytest.mark.parametrize("n", [16, 90, 9009, 65536])
def test_stream_handed_over_between_runs(product_lib, n):
    """What was written or computed before the graph gets a stream of the caller's is there afterwards."""
    import torch
    rng = np.random.default_rng(7)
    g, a, b, y, shape = add(product_lib, n)
    u, v, w = (rng.integers(0, 80, size=shape).astype(np.uint8) for _ in range(3))
    g.write(a, u)
    g.compile()
    g.write(b, v)
    g.run()
    st = torch.cuda.Stream()
    g.set_stream(st.cuda_stream)
    np.testing.assert_array_equal(g.read(y), u + v)
    g.write(a, w)
    g.run_async()
    np.testing.assert_array_equal(g.read(y), w + v)
    g.write(y, u)
    np.testing.assert_array_equal(g.read(y), u)
    g.set_stream(None)
    np.testing.assert_array_equal(g.read(y), u)
    g.run()
    np.testing.assert_array_equal(g.read(y), w + v)
    g.close()


@pytest.mark.parametrize("spec", ["gemm:16:4096:4096", "conv:3:64:64:56:1"])
def test_resident_data_is_not_moved_again(product_lib, spec):
    """run_async on data that is there launches the kernels of the plan and nothing else."""
    import torch
    import opworkloads
    g = B.Graph(product_lib, 0)
    work = opworkloads.build(spec, 1, g, np.random.default_rng(8))
    for t, a in work["inputs"]:
        g.write(t, a)
    g.run_async()
    g.sync()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        for _ in range(3):
            g.run_async()
        g.sync()
    launched = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    assert len(launched) == 3 * len(g.kernels()), launched
    g.close()
