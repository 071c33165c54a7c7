"""The tensor-instruction depthwise kernel against the oracle at the edges of its tiles: every channel-slab width with and
without idle groups, output widths around the strip of eight, odd and even row counts, images that share a tile."""
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu


def dw(W, H, C, N, stride=1, in_zp=0, pad_type=B.PAD_SAME, x_dtype=B.DT_UINT8):
    return G.depthwise_q(W, H, C, N, 3, 3, stride=(stride, stride), in_q=(0.03, in_zp), w_kind="s8pc", pad_type=pad_type, x_dtype=x_dtype)


CASES = {
    # slabs of 16, 32, 48 and 64 channels; the last one partly idle; channels that are no multiple of 16
    "c16": dw(20, 11, 16, 9), "c32": dw(33, 16, 32, 5), "c48": dw(17, 9, 48, 3), "c64": dw(12, 12, 64, 2), "c80": dw(9, 9, 80, 2),
    "c144": dw(28, 28, 144, 2), "c21": dw(15, 8, 21, 3),
    # one pixel, one column, one row, a strip and its neighbours
    "w1h1": dw(1, 1, 64, 3), "w1": dw(1, 13, 32, 2), "h1": dw(23, 1, 32, 2), "w7": dw(7, 7, 960, 3), "w8": dw(8, 8, 96, 2), "w9": dw(9, 10, 96, 2),
    "w112": dw(112, 112, 32, 1),
    # stride 2, even and odd extents, both ends of the padding
    "s2_even": dw(56, 56, 144, 1, 2), "s2_odd": dw(15, 13, 48, 3, 2), "s2_tiny": dw(2, 2, 16, 4, 2), "s2_valid": dw(19, 12, 40, 2, 2, 7, B.PAD_VALID),
    # no padding: any input zero point; int8 inputs
    "valid_zp": dw(19, 11, 40, 2, 1, 133, B.PAD_VALID), "int8": dw(17, 17, 72, 2, 1, 0, B.PAD_SAME, B.DT_INT8),
    # more tiles than blocks
    "many": dw(40, 40, 64, 150),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_depthwise_mma(product_lib, oracle_lib, name):
    want, _ = G.run_case(oracle_lib, CASES[name], 5)
    got, kernels = G.run_case(product_lib, CASES[name], 5)
    assert any(k["name"] == "depthwise_mma" for k in kernels)
    G.assert_same(want, got)
