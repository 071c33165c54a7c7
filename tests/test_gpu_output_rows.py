"""Graph outputs of one pixel per image that are too large to be staged on the host: rows lose their channel padding."""
import numpy as np
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels,rows", [(33, 9001), (17, 20000), (1000, 300), (1, 300001)])
def test_padded_rows(product_lib, oracle_lib, channels, rows):
    build = G.fc_q(48, channels, rows)
    want, _ = G.run_case(oracle_lib, build, 2)
    got, kernels = G.run_case(product_lib, build, 2)
    assert kernels[-1]["name"] == "cl_to_whcn"
    G.assert_same(want, got)


def test_float_rows_between_images(product_lib, oracle_lib):
    """Softmax to float32 behind a pool that leaves one pixel: rank 4, four bytes an element, not a multiple of four channels."""
    def build(g, rng):
        x = g.tensor(B.DT_UINT8, [3, 3, 27, 5000], B.ATTR_INPUT, scale=0.1, zero_point=3)
        p = g.tensor(B.DT_UINT8, [], B.ATTR_TRANSIENT, scale=0.1, zero_point=3)
        y = g.tensor(B.DT_FLOAT32, [1, 1, 27, 5000], B.ATTR_OUTPUT)
        g.pool2d(x, p, B.POOL_AVG, (3, 3), (1, 1))
        g.softmax(p, y, axis=2)
        return [(x, rng.integers(0, 256, size=(5000, 27, 3, 3)).astype(np.uint8))], [y]
    want, _ = G.run_case(oracle_lib, build, 2)
    got, _ = G.run_case(product_lib, build, 2)
    G.assert_same(want, got, float_tol=1e-5)


@pytest.mark.parametrize("outputs,batch", [(2, 1), (3, 300), (5, 7), (9, 2)])
def test_several_outputs_share_a_launch(product_lib, oracle_lib, outputs, batch):
    """Row counts equal, row lengths not (1 to 50 bytes); read after a run, after an asynchronous one, and after a second input."""
    def build(g, rng):
        x = g.tensor(B.DT_UINT8, [40, batch], B.ATTR_INPUT, scale=0.02, zero_point=128)
        ys = []
        for k in range(outputs):
            n = [10, 50, 1, 33, 17, 9, 47, 3, 21][k]
            w = g.tensor(B.DT_INT8, [40, n], B.ATTR_CONSTANT, scales=rng.uniform(0.001, 0.01, n).astype(np.float32), channel_dim=1,
                         data=rng.integers(-127, 128, size=(n, 40)).astype(np.int8))
            ys.append(g.tensor(B.DT_UINT8, [], B.ATTR_OUTPUT, scale=0.02, zero_point=100))
            g.fully_connected(x, w, None, ys[-1], axis=0, weights=n)
        return x, ys

    results = []
    for lib in (oracle_lib, product_lib):
        rng = np.random.default_rng(outputs)
        g = B.Graph(lib)
        x, ys = build(g, rng)
        g.compile()
        got = []
        for k in range(3):
            g.write(x, rng.integers(0, 256, size=(batch, 40)).astype(np.uint8))
            if k == 1 and hasattr(g, "run_async"):
                g.run_async()
                g.sync()
            else:
                g.run()
            got += [g.read(y) for y in ys]
        names = [k["name"] for k in g.kernels()]
        g.close()
        results.append(got)
    assert names.count("cl_to_whcn") == (outputs + 3) // 4, names
    G.assert_same(*results)
