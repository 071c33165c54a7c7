"""The tensor-instruction depthwise kernel against the oracle at the edges of its tiles: every channel-slab width with and
without idle groups, output widths around the strip of eight, odd and even row counts, images that share a tile."""
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu


def dw(W, H, C, N, stride=1, in_zp=0, pad_type=B.PAD_SAME, x_dtype=B.DT_UINT8):
    return G.depthwise_q(W, H, C, N, 3, 3, stride=(stride, stride), in_q=(0.03, in_zp), w_kind="s8pc", pad_type=pad_type, x_dtype=x_dtype)


def dw_u8(stride, in_scale, out_q, w_zp, w_range, in_zp=0, pad_type=B.PAD_SAME, x_dtype=B.DT_UINT8, out_dtype=B.DT_UINT8):
    """uint8 kernel of scale 0.02 with values in w_range; no Relu6 behind it."""
    return G.depthwise_q(27, 14, 48, 2, 3, 3, stride=(stride, stride), in_q=(in_scale, in_zp), w_kind="u8", w_zp=w_zp, w_range=w_range, out_q=out_q,
                         relu6=False, pad_type=pad_type, x_dtype=x_dtype, out_dtype=out_dtype)


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
    # accumulator scale above half the output scale (multipliers halved to fit 31 bits): both strides, both input types
    "ratio_1": dw_u8(1, 0.03, (6e-4, 3), 128, (127, 130)), "ratio_5_s2": dw_u8(2, 0.03, (1.2e-4, 100), 128, (127, 130)),
    "ratio_1_int8": dw_u8(1, 0.03, (6e-4, 3), 128, (127, 130), x_dtype=B.DT_INT8), "ratio_1_int8_s2": dw_u8(2, 0.03, (6e-4, 3), 128, (127, 130), x_dtype=B.DT_INT8),
    # int8 outputs
    "out_int8": dw_u8(1, 0.03, (0.3, -11), 128, (0, 256), out_dtype=B.DT_INT8), "out_int8_s2": dw_u8(2, 0.03, (0.3, -128), 128, (0, 256), out_dtype=B.DT_INT8),
    # a kernel whose centred values just fit int8; every second and every fourth accumulator on an exact half
    "u8_centred": dw_u8(1, 0.03, (0.3, 9), 110, (0, 238)), "halves": dw_u8(1, 0.5, (0.02, 20), 128, (126, 131)),
    "quarters": dw_u8(1, 0.25, (0.02, 20), 128, (126, 131)), "quarters_s2_int8": dw_u8(2, 0.25, (0.02, -20), 128, (126, 131), out_dtype=B.DT_INT8),
}

# Layers that are not this kernel's: centred weights that do not fit int8, padding with an input zero point, and the switch.
OTHERS = {"spread": dw_u8(1, 0.03, (0.3, 9), 20, (0, 256)), "padded_zp": dw(20, 11, 16, 9, 1, 3), "switch": dw(20, 11, 16, 9)}


@pytest.mark.parametrize("name", sorted(CASES))
def test_depthwise_mma(product_lib, oracle_lib, name):
    want, _ = G.run_case(oracle_lib, CASES[name], 5)
    got, kernels = G.run_case(product_lib, CASES[name], 5)
    assert any(k["name"] == "depthwise_mma" for k in kernels)
    G.assert_same(want, got)


@pytest.mark.parametrize("name", sorted(OTHERS))
def test_layers_of_the_other_kernels(product_lib, oracle_lib, monkeypatch, name):
    monkeypatch.setenv("B2VX_DW_STRIP", "1")   # the default: asks for nothing
    if name == "switch":
        G.assert_same(*(G.run_case(lib, OTHERS[name], 5)[0] for lib in (oracle_lib, product_lib)))
        assert any(k["name"] == "depthwise_mma" for k in G.run_case(product_lib, OTHERS[name], 5)[1])
        monkeypatch.setenv("B2VX_DW_MMA", "0")
    want, _ = G.run_case(oracle_lib, OTHERS[name], 5)
    got, kernels = G.run_case(product_lib, OTHERS[name], 5)
    assert not any(k["name"] == "depthwise_mma" for k in kernels)
    G.assert_same(want, got)
