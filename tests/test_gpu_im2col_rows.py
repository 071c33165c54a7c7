"""First layers whose im2col blocks take several output rows, against the oracle: output heights that the block's rows do and do not
divide, both piece widths, strides 1 and 2, padding at every side, images from many (several rows a block) to one."""
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu

# width, height, channels in, images, filter width and height, channels out; strides, padding, zero point of the input
CASES = {
    "lenet_300": ((28, 28, 1, 300, 5, 5, 20), (1, 1), B.PAD_VALID, 128), "lenet_1": ((28, 28, 1, 1, 5, 5, 20), (1, 1), B.PAD_VALID, 128),
    "stem7_60": ((64, 61, 3, 60, 7, 7, 24), (2, 2), B.PAD_SAME, 117), "stem3_64": ((60, 67, 3, 64, 3, 3, 32), (2, 2), B.PAD_SAME, 9),
    "odd_heights": ((30, 23, 2, 200, 3, 2, 16), (1, 1), B.PAD_SAME, 200), "tall": ((9, 131, 3, 50, 4, 5, 16), (1, 1), B.PAD_SAME, 1),
    "one_row": ((40, 3, 3, 900, 3, 3, 16), (1, 1), B.PAD_VALID, 128), "narrow": ((4, 50, 5, 400, 3, 3, 40), (1, 1), B.PAD_SAME, 128),
    "wide_k": ((40, 33, 12, 120, 8, 6, 16), (1, 1), B.PAD_SAME, 128), "stride_y3": ((33, 50, 3, 110, 5, 5, 16), (1, 3), B.PAD_SAME, 77),
    "unaligned": ((35, 30, 3, 150, 3, 3, 16), (2, 1), B.PAD_SAME, 128),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_first_layer(product_lib, oracle_lib, launch_rules, name):
    sizes, stride, pad, zero = CASES[name]
    (w, h, c, n, kw, kh, _) = sizes
    ((block_rows, _, rows),) = launch_rules([("im2col", n, w, h, c, kw, kh) + stride + (int(pad == B.PAD_SAME), 148)])
    assert (block_rows > 1) == (name not in ("lenet_1", "one_row")), (block_rows, rows)
    case = G.conv2d_q(*sizes, stride=stride, pad_type=pad, in_q=(0.02, zero))
    want, _ = G.run_case(oracle_lib, case, 8)
    got, kernels = G.run_case(product_lib, case, 8)
    assert any(k["name"] == ("im2col_whcn4" if kw <= 4 else "im2col_whcn8") for k in kernels), kernels
    G.assert_same(want, got)


def test_blocks_of_several_rows_end_inside_an_image(launch_rules):
    """The cases above have both: output rows that the rows of a block divide, and a shorter last block."""
    answers = launch_rules([("im2col",) + (s[3], s[0], s[1], s[2], s[4], s[5]) + stride + (int(pad == B.PAD_SAME), 148) for s, stride, pad, _ in CASES.values()])
    left = [rows % block_rows for block_rows, _, rows in answers if block_rows > 1]
    assert 0 in left and any(left), answers
