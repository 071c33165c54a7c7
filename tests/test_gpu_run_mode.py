"""Narrow GEMM tiles of several 128-row pieces (layers with few output channels, a short K and very many pixels) against the
oracle on the first and the last images: whole and ragged last tiles, one and two column blocks, K of one and several blocks,
halved multipliers and int8 outputs, and a row count just below the rule's."""
import numpy as np
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu

# width, height, images (606208 pixels or more: eight tiles of 512 rows for each of 148 SMs), channels in and out, output quantization, type
CASES = {
    "whole_tiles": (112, 112, 64, 32, 16, (0.05, 0), B.DT_UINT8), "8_rows_left": (67, 29, 312, 16, 32, (0.05, 3), B.DT_UINT8),
    "129_rows_left": (173, 9, 421, 32, 16, (0.05, 0), B.DT_UINT8), "last_piece_partly": (128, 37, 129, 48, 32, (0.05, 0), B.DT_UINT8),
    "int8_k96": (67, 29, 314, 96, 24, (0.05, -5), B.DT_INT8), "halved": (67, 29, 313, 48, 17, (1.5e-4, 100), B.DT_UINT8),
    # two pieces a tile: 33 to 64 channels, from 303104 rows on
    "c64": (56, 56, 97, 64, 64, (0.05, 0), B.DT_UINT8), "c48_k192": (67, 29, 157, 192, 48, (0.05, 3), B.DT_UINT8), "c64_int8": (173, 9, 211, 144, 50, (0.05, -5), B.DT_INT8),
    "c64_halved": (128, 37, 65, 48, 64, (1.5e-4, 100), B.DT_UINT8), "c40": (1024, 1, 297, 256, 40, (0.05, 0), B.DT_UINT8), "k256": (112, 112, 49, 256, 32, (0.05, 0), B.DT_UINT8),
    "c64_below": (67, 29, 155, 16, 64, (0.05, 3), B.DT_UINT8), "one_tile_less": (67, 29, 311, 16, 32, (0.05, 3), B.DT_UINT8),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_1x1(product_lib, oracle_lib, name):
    w, h, n, cin, cout, out_q, dtype = CASES[name]
    x = np.random.default_rng(3).integers(0, 256, size=(n, cin, h, w)).astype(np.uint8)

    def layer(data):
        def build(g, rng):   # the weights are drawn before the input, so they do not depend on the number of images
            inputs, outputs = G.conv2d_q(w, h, cin, data.shape[0], 1, 1, cout, pad_type=B.PAD_VALID, out_q=out_q, out_dtype=dtype)(g, rng)
            return [(inputs[0][0], data)], outputs
        return build

    got, kernels = G.run_case(product_lib, layer(x), 5)
    assert any(k["name"] == "gemm_i8_tc" for k in kernels)
    for part in (slice(0, 3), slice(n - 3, n)):
        want, _ = G.run_case(oracle_lib, layer(np.ascontiguousarray(x[part])), 5)
        G.assert_same(want, [got[0][part]])
