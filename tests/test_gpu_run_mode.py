"""Narrow GEMM tiles of several 128-row pieces (layers with few output channels, a short K and very many pixels): every image against
the oracle, in that form and without it: whole and ragged last tiles, one and two column blocks, K of one and several blocks, halved
multipliers and int8 outputs, and row counts just below the rules'."""
import numpy as np
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu

# 128-row pieces of a tile; width, height, images, channels in and out, output quantization, type.  Four pieces from 606208 pixels on
# (eight tiles of 512 rows for each of 148 SMs) for up to 32 channels, two from 303104 on for 33 to 64.
CASES = {
    "whole_tiles": (4, 112, 112, 64, 32, 16, (0.05, 0), B.DT_UINT8), "8_rows_left": (4, 67, 29, 312, 16, 32, (0.05, 3), B.DT_UINT8),
    "129_rows_left": (4, 173, 9, 421, 32, 16, (0.05, 0), B.DT_UINT8), "last_piece_partly": (4, 128, 37, 129, 48, 32, (0.05, 0), B.DT_UINT8),
    "int8_k96": (4, 67, 29, 314, 96, 24, (0.05, -5), B.DT_INT8), "halved": (4, 67, 29, 313, 48, 17, (1.5e-4, 100), B.DT_UINT8),
    "k256": (4, 112, 112, 49, 256, 32, (0.05, 0), B.DT_UINT8), "one_tile_less": (1, 67, 29, 311, 16, 32, (0.05, 3), B.DT_UINT8),
    "c64": (2, 56, 56, 97, 64, 64, (0.05, 0), B.DT_UINT8), "c48_k192": (2, 67, 29, 157, 192, 48, (0.05, 3), B.DT_UINT8),
    "c64_int8": (2, 173, 9, 211, 144, 50, (0.05, -5), B.DT_INT8), "c64_halved": (2, 128, 37, 65, 48, 64, (1.5e-4, 100), B.DT_UINT8),
    "c40": (2, 1000, 1, 304, 256, 40, (0.05, 0), B.DT_UINT8), "c64_below": (1, 67, 29, 155, 16, 64, (0.05, 3), B.DT_UINT8),
}
IMAGES = 7   # different ones; a period of 7 images is no whole number of tiles, nor are the tiles of a round over all blocks


@pytest.mark.parametrize("name", sorted(CASES))
def test_1x1(product_lib, oracle_lib, monkeypatch, name):
    pieces, w, h, n, cin, cout, out_q, dtype = CASES[name]
    x = np.random.default_rng(3).integers(0, 256, size=(IMAGES, cin, h, w)).astype(np.uint8)
    period, step = IMAGES * w * h, 128 * pieces
    assert period % step and 148 * step % period

    def layer(data):
        def build(g, rng):   # the weights are drawn before the input, so they do not depend on the number of images
            inputs, outputs = G.conv2d_q(w, h, cin, data.shape[0], 1, 1, cout, pad_type=B.PAD_VALID, out_q=out_q, out_dtype=dtype)(g, rng)
            return [(inputs[0][0], data)], outputs
        return build

    (want,), _ = G.run_case(oracle_lib, layer(x), 5)
    which = np.arange(n) % IMAGES
    for switch, label in ((None, "gemm_i8_tc" if pieces == 1 else "gemm_i8_tc(x%d)" % pieces), ("0", "gemm_i8_tc")):
        if switch:
            monkeypatch.setenv("B2VX_TC_RUN", switch)
        (got,), kernels = G.run_case(product_lib, layer(x[which]), 5)
        assert label in [k["name"] for k in kernels], kernels
        G.assert_same([want[which]], [got])
