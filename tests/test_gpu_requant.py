"""The tensor-core epilogue's fixed-point requantization against the oracle, where it can go wrong: ratios of accumulator
scale to output scale at both ends of the multiplier's range, ratios that put many accumulators on an exact half, every
column block width, and uint8 kernels on both sides of "the centred weights fit int8"."""
import numpy as np
import pytest

import graph_cases as G
import pyb2vx as B

pytestmark = pytest.mark.gpu


def conv1x1(C, Oc, N, W, out_scale, zp=0, w_scale=0.01, w_zp=None, spread=255, out_dtype=B.DT_UINT8, residual=False, bias=(-3000, 3001), odd_scale=None,
            odd_bias=None):
    """1x1 convolution on [W, W, C, N]; w_zp None: int8 kernel, per-tensor scale, or per channel with odd_scale in channel 5;
    else uint8 with `spread` values about w_zp.  odd_bias: of channel 20."""
    def build(g, rng):
        x = g.tensor(B.DT_UINT8, [W, W, C, N], B.ATTR_INPUT, scale=0.02, zero_point=7)
        if odd_scale is not None:
            scales = rng.uniform(0.5 * w_scale, 2 * w_scale, Oc).astype(np.float32)
            scales[5] = odd_scale
            w = g.tensor(B.DT_INT8, [1, 1, C, Oc], B.ATTR_CONSTANT, scales=scales, channel_dim=3,
                         data=rng.integers(-127, 128, size=(Oc, C, 1, 1)).astype(np.int8))
        elif w_zp is None:
            w = g.tensor(B.DT_INT8, [1, 1, C, Oc], B.ATTR_CONSTANT, scale=w_scale, zero_point=0,
                         data=rng.integers(-127, 128, size=(Oc, C, 1, 1)).astype(np.int8))
        else:
            lo, hi = max(0, w_zp - spread // 2), min(255, w_zp + spread // 2)
            w = g.tensor(B.DT_UINT8, [1, 1, C, Oc], B.ATTR_CONSTANT, scale=w_scale, zero_point=w_zp,
                         data=rng.integers(lo, hi + 1, size=(Oc, C, 1, 1)).astype(np.uint8))
        biases = rng.integers(bias[0], bias[1], size=Oc).astype(np.int32)
        if odd_bias is not None:
            biases[20] = odd_bias
        b = g.tensor(B.DT_INT32, [Oc], B.ATTR_CONSTANT, scale=float(np.float32(0.02) * np.float32(w_scale)), zero_point=0, data=biases)
        y = g.tensor(out_dtype, [], B.ATTR_TRANSIENT if residual else B.ATTR_OUTPUT, scale=out_scale, zero_point=zp)
        g.conv2d(x, w, b, y, pad_type=B.PAD_VALID)
        inputs = [(x, rng.integers(0, 256, size=(N, C, W, W)).astype(np.uint8))]
        if not residual:
            return inputs, [y]
        r = g.tensor(B.DT_UINT8, [W, W, Oc, N], B.ATTR_INPUT, scale=out_scale * 0.7, zero_point=3)
        s = g.tensor(B.DT_UINT8, [], B.ATTR_OUTPUT, scale=out_scale * 1.3, zero_point=11)
        g.add(y, r, s)
        return inputs + [(r, rng.integers(0, 256, size=(N, Oc, W, W)).astype(np.uint8))], [s]
    return build


CASES = {
    # scale ratio: well above 1 (the multiplier is halved until it fits), about 1/2, ordinary, tiny (wide windows), and so
    # small that every element takes the exact sequence
    "ratio_4": conv1x1(32, 48, 1, 13, 5e-5), "ratio_1_2": conv1x1(32, 48, 1, 13, 4e-4), "ratio_1e-3": conv1x1(64, 64, 1, 13, 0.2),
    "ratio_4e-7": conv1x1(64, 32, 1, 9, 500.0), "ratio_1e-10": conv1x1(64, 32, 1, 9, 2e6),
    # one accumulator in a hundred lies on an exact half
    "ties": conv1x1(32, 64, 2, 17, 0.02), "ties_int8": conv1x1(32, 80, 2, 17, 0.02, zp=-3, out_dtype=B.DT_INT8),
    # block widths 16, 32, 64; several blocks per warp group; a last N tile that is not full
    "oc16": conv1x1(48, 16, 1, 12, 0.05), "oc96": conv1x1(48, 96, 1, 12, 0.05, zp=128), "oc144": conv1x1(24, 144, 2, 28, 0.05),
    "oc240": conv1x1(32, 240, 1, 12, 0.05), "oc272": conv1x1(32, 272, 3, 40, 0.05), "oc512": conv1x1(64, 512, 1, 7, 0.05),
    # uint8 kernels: centred weights that fit int8 (no sum of the inputs needed), and ones that do not
    "u8_fits": conv1x1(96, 64, 2, 11, 0.3, w_zp=110, spread=200), "u8_spread": conv1x1(96, 64, 2, 11, 0.3, w_zp=60, spread=400),
    # residual Add in team mode (four residual buffers), more tiles than buffers; and on wide tiles
    "add_teams": conv1x1(64, 32, 4, 120, 0.05, residual=True), "add_wide": conv1x1(64, 256, 2, 60, 0.05, residual=True),
    "add_oc48_one_tile": conv1x1(64, 48, 1, 7, 0.05, residual=True),
    # one channel whose scale is far from the others': a dead one, ones whose outputs reach the next integer or a few, and one
    # that saturates; outputs that cannot reach the range at all; one channel of many that takes the exact sequence
    "dead_channel": conv1x1(64, 96, 1, 12, 0.05, odd_scale=1e-10), "nearly_dead": conv1x1(64, 96, 1, 12, 0.05, zp=100, odd_scale=3e-6),
    "half_dead": conv1x1(64, 96, 1, 12, 0.05, zp=100, odd_scale=2e-5), "wild_channel": conv1x1(64, 96, 1, 12, 0.05, zp=100, odd_scale=40.0),
    "below_range": conv1x1(32, 48, 1, 12, 2000.0, zp=-300), "above_range": conv1x1(32, 48, 1, 12, 2000.0, zp=700, odd_scale=1e-10),
    "exact_block": conv1x1(64, 192, 1, 12, 0.05, odd_scale=1e-9, odd_bias=2**31 - 5), "exact_block_teams": conv1x1(64, 64, 2, 30, 0.05, odd_bias=-2**31),
    # long K: on both sides of where the bound of a full-range kernel reaches 31 bits, with the bound from the weights' values,
    # and beyond that as well
    "k16448": G.fc_q(16448, 48, 20), "k16464": G.fc_q(16464, 48, 20), "k25088": G.fc_q(25088, 80, 130), "k65808": G.fc_q(65808, 32, 20),
    "k100352": G.fc_q(100352, 16, 17), "k140000": G.fc_q(140000, 16, 17), "k33040_u8": G.fc_q(33040, 32, 20, w_kind="u8"),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_fixed_point_requantization(product_lib, oracle_lib, name):
    want, _ = G.run_case(oracle_lib, CASES[name], 11)
    got, kernels = G.run_case(product_lib, CASES[name], 11)
    assert any(k["name"].startswith("gemm_i8_tc") for k in kernels)
    G.assert_same(want, got)


# The sum of accumulator and bias wraps in 32 bits for some elements of every channel and for others not: the wrapped sum
# counts, like in the reference's integer arithmetic, and 64-bit intermediates must not hide it.
NEAR_2_31 = (2**31 - 60000, 2**31)
WRAP = {
    "conv": conv1x1(32, 48, 1, 13, 4000.0, zp=128, bias=NEAR_2_31),
    "depthwise": G.depthwise_q(17, 9, 48, 2, 3, 3, w_kind="u8", in_q=(0.03, 0), out_q=(12000.0, 128), relu6=False, w_zp=128, bias=NEAR_2_31),
}


@pytest.mark.parametrize("name", sorted(WRAP))
def test_accumulator_and_bias_wrap(product_lib, oracle_lib, name):
    want, _ = G.run_case(oracle_lib, WRAP[name], 13)
    got, _ = G.run_case(product_lib, WRAP[name], 13)
    assert {int(v) for v in np.unique(want[0])} >= {128 - 107, 128 + 107}   # both sides of the wrap
    G.assert_same(want, got)


def test_one_dead_channel_does_not_slow_the_layer(product_lib):
    """A channel with a tiny scale among ordinary ones (a dead channel of a per-channel network) must not send the whole layer
    through the exact sequence, which takes 3.7 times as long here; twice is allowed."""
    us = {}
    for odd in (0.005, 1e-10):
        g = B.Graph(product_lib, 0)
        try:
            inputs, _ = conv1x1(256, 64, 64, 56, 0.5, odd_scale=odd)(g, np.random.default_rng(14))
            g.compile()
            for t, a in inputs:
                g.write(t, a)
            us[odd] = min(1e3 * k["ms"] for _ in range(3) for k in g.profile(5) if k["name"].startswith("gemm_i8_tc"))
        finally:
            g.close()
    assert us[1e-10] < 2 * us[0.005], us
