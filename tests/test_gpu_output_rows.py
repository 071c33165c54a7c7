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
