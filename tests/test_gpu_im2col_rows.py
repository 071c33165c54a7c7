"""First layers whose im2col blocks take several output rows, against the oracle: output heights that the block's rows do and do not
divide, both piece widths, strides 1 and 2, padding at every side, images from many (several rows a block) to one."""
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu

CASES = {
    "lenet_300": G.conv2d_q(28, 28, 1, 300, 5, 5, 20, pad_type=B.PAD_VALID), "lenet_1": G.conv2d_q(28, 28, 1, 1, 5, 5, 20, pad_type=B.PAD_VALID),
    "stem7_40": G.conv2d_q(64, 61, 3, 40, 7, 7, 24, stride=(2, 2), in_q=(0.02, 117)), "stem3_64": G.conv2d_q(60, 67, 3, 64, 3, 3, 32, stride=(2, 2), in_q=(0.02, 9)),
    "odd_heights": G.conv2d_q(30, 23, 2, 200, 3, 2, 16, in_q=(0.02, 200)), "tall": G.conv2d_q(9, 131, 3, 50, 4, 5, 16, in_q=(0.02, 1)),
    "one_row": G.conv2d_q(40, 3, 3, 900, 3, 3, 16, pad_type=B.PAD_VALID), "narrow": G.conv2d_q(4, 50, 5, 400, 3, 3, 40), "wide_k": G.conv2d_q(40, 33, 12, 120, 8, 6, 16),
    "stride_y3": G.conv2d_q(33, 50, 3, 90, 5, 5, 16, stride=(1, 3), in_q=(0.02, 77)), "unaligned": G.conv2d_q(35, 30, 3, 150, 3, 3, 16, stride=(2, 1)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_first_layer(product_lib, oracle_lib, name):
    want, _ = G.run_case(oracle_lib, CASES[name], 8)
    got, kernels = G.run_case(product_lib, CASES[name], 8)
    assert any(k["name"].startswith("im2col_whcn") for k in kernels), kernels
    G.assert_same(want, got)
